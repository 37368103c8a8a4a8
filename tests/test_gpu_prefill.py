"""The token-parallel prompt path against the decode kernel that steps through the same prompt.

The first layer's recurrent state sees no earlier bf16 rounding, so there the two must agree to fp32 sums; behind it
roundings of GEMV inputs flip, so logits and states are held to the bars the decode tests use.  Lengths: the shortest
this path takes, one row short of / past a 16-row tile and a 256-row tile, several passes, and a start behind a context.
Block-scaled FP8 with scales that are bf16 values and with others, in tiles with and without room for an accumulator per block."""

import pytest
import torch

pytestmark = pytest.mark.gpu

from megakernels_b200 import gemma26b, qwen27b, qwen35moe
from megakernels_b200.gemma26b.dims import FULL as FULL26
from megakernels_b200.qwen27b.dims import FULL as FULL27
from megakernels_b200.qwen35moe.dims import FULL as FULL35
from megakernels_b200.stage import runtime

SHAPES = {
    "27b": (qwen27b, FULL27.with_(hidden=1024, ffn=2048, vocab=4096, layers=4, nkh=4, nvh=12, nq=8, nkv=2)),
    "35b": (qwen35moe, FULL35.with_(hidden=1024, vocab=4096, layers=4, nkh=4, nvh=8, nq=8, nkv=2, fi=128, sfi=128)),
    "26b": (gemma26b, FULL26.with_(hidden=512, vocab=4096, layers=6, ffn=256, experts=128, eff=128, window=64)),
}
CASES = [("27b", {}, 1, 12, 0), ("27b", {}, 1, 258, 0), ("27b", {}, 3, 86, 37), ("27b", {"fmt": "bf16"}, 2, 41, 0),
         ("35b", {}, 1, 18, 0), ("35b", {}, 2, 129, 21), ("35b", {"fp32_scales": True}, 1, 18, 0), ("35b", {"fp32_scales": True}, 2, 129, 0), ("26b", {}, 1, 17, 0), ("26b", {}, 3, 150, 21)]


def rel(a, b):
    return float((a.double() - b.double()).norm() / b.double().norm())


@pytest.fixture(scope="module")
def packed():
    made = {}

    def get(model, fmt):
        key = (model, tuple(fmt.items()))
        if key not in made:
            pkg, shape = SHAPES[model]
            kw = dict(fmt)
            fp32_scales = kw.pop("fp32_scales", False)
            W = pkg.SynthWeights(shape, layers=shape.layers, init="realistic", device="cuda", **kw)
            if fp32_scales:                                  # block scales that are not bf16 values: just below the next one
                W.raw = {k: (q, sc.float() * 1.0037) for k, (q, sc) in W.raw.items()}
                W.exs = {k: sc.float() * 1.0037 for k, sc in W.exs.items()}
            made[key] = pkg.Packed(W, "cuda")
        return made[key]
    return get


@pytest.mark.parametrize("model,fmt,M,length,context", CASES)
def test_prompt_rows_equal_stepping(packed, monkeypatch, model, fmt, M, length, context):
    pkg, shape = SHAPES[model]
    prompts = [pkg.make_prompt(shape.vocab, context + length, seed=j) for j in range(M)]
    engines = []
    for rows in (True, False):
        eng = pkg.Engine(packed(model, fmt), M, maxlen=context + length + 64)
        for p in range(context):
            eng.step(torch.tensor([q[p] for q in prompts], device="cuda"))
        with monkeypatch.context() as mp:
            mp.setattr(runtime, "MAX_ROWS", 200)            # several passes for the longer prompts
            if not rows:
                mp.setattr(runtime, "MIN_ROWS_PATH", 1 << 30)
            launches = eng.rt.launches
            logits = eng.prefill([q[context:] for q in prompts]).clone()
            assert eng.rt.launches == launches + 1
            assert (eng.rt._workspace is not None) == rows           # one arm took the token-parallel path, the other stepped
        eng.check()
        engines.append((eng, logits))
    (a, la), (b, lb) = engines
    assert a.pos[:M].tolist() == b.pos[:M].tolist() == [context + length] * M
    assert rel(la, lb) < 3e-2
    if model == "26b":
        assert rel(a.ks[0], b.ks[0]) < 1e-3 and rel(a.vs[0], b.vs[0]) < 1e-3
        assert rel(a.kf, b.kf) < 3e-2 and rel(a.vf, b.vf) < 3e-2
    else:
        assert rel(a.ssm[0], b.ssm[0]) < 2e-4 and rel(a.ssm, b.ssm) < 1e-2 and rel(a.conv, b.conv) < 1e-2
        assert rel(a.k_cache, b.k_cache) < 2e-2 and rel(a.v_cache, b.v_cache) < 2e-2


def test_prompt_rows_see_no_key_before_their_window(packed):
    """What lies before the first row's window in its cache page may be anything: a page another sequence used, or never
    written.  The decode kernel does not touch it."""
    pkg, shape = SHAPES["26b"]
    prompt, got = pkg.make_prompt(shape.vocab, 40, seed=3), []
    for poisoned in (False, True):
        eng = pkg.Engine(packed("26b", {}), 1, maxlen=200)
        for t in (eng.ks, eng.vs):
            t.normal_(0.0, 0.5, generator=torch.Generator(device="cuda").manual_seed(5))
        if poisoned:
            bt = eng.bt[0].long()
            for p in range(100 - shape.window + 1):                   # positions 0 .. 36: the prompt starts at 100, the window is 64
                eng.ks[:, bt[p // 64], :, p % 64] = float("inf")
                eng.vs[:, bt[p // 64], :, p % 64] = float("nan")
        eng.pos[0] = 100
        got.append(eng.prefill([prompt]).clone())
        assert eng.rt._workspace is not None
        eng.check()
    assert torch.isfinite(got[0]).all() and torch.equal(*got)


def test_programs_without_the_row_path_step(packed):
    pkg, shape = SHAPES["35b"]
    eng = pkg.Engine(packed("35b", {}), 1, maxlen=64, exact_inputs=True)
    prompt = pkg.make_prompt(shape.vocab, 20, seed=3)
    got = eng.prefill([prompt]).clone()
    eng.reset()
    for t in prompt:
        want = eng.step(torch.tensor([t], device="cuda"))
    assert torch.equal(got, want)


# ---- the 0.8B model: fp32-exact, so ids are equal and states agree to fp32 sums -------------------------------------------
@pytest.fixture(scope="module")
def small():
    from megakernels_b200.config import qwen35_08b
    from megakernels_b200.synth import make_mtp_weights, make_weights
    cfg = qwen35_08b(n_layers=4, vocab=4096)
    return cfg, make_weights(cfg, 0, init="realistic"), make_mtp_weights(cfg, 0)


@pytest.mark.parametrize("quant,kv,length,context", [("bf16", "fp32", 17, 0), ("bf16", "fp32", 130, 5), ("int8", "fp32", 17, 3),
                                                     ("int8", "fp32", 300, 33), ("int8", "bf16", 90, 0)])
def test_small_model_prompt_equals_stepping(small, monkeypatch, quant, kv, length, context):
    from megakernels_b200 import engine as E
    from megakernels_b200.synth import make_prompt
    prompt, got = make_prompt(small[0], context + length), []
    for rows in (True, False):
        mk = E.Megakernel(small, max_seq=512, quant=quant, kv_dtype=kv, mtp=quant == "int8")
        with monkeypatch.context() as mp:
            mp.setattr(E, "MIN_PROMPT_ROWS", 1 << 30)
            if context:
                mk.run(prompt[:context])
            mp.setattr(E, "MIN_PROMPT_ROWS", 16 if rows else 1 << 30)
            mp.setattr(E, "EXACT_PROMPT", 0)                 # logits are asked for here
            mp.setattr(E, "MAX_PROMPT_ROWS", 120)            # several passes
            ids, logits = mk.run(prompt[context:], n_generate=6, return_logits=True, track_mtp=True)
        assert (mk._workspace is not None) == rows           # one arm took the prompt in at once, the other stepped
        got.append((mk, ids, logits))
    (a, ia, la), (b, ib, lb) = got
    tol = 2e-5 if kv == "fp32" else 2e-4                      # a bf16 cache rounds
    assert ia == ib and a.pos == b.pos and rel(la, lb) < tol
    for x, y in zip(a.bstate + a.conv_hist, b.bstate + b.conv_hist):
        assert rel(x, y) < tol
    assert rel(a.k_cache[0], b.k_cache[0]) < 50 * tol and rel(a.v_cache[0], b.v_cache[0]) < 50 * tol
    if a.mtp is not None:
        assert rel(a.mtp_k_cache, b.mtp_k_cache) < 50 * tol and a.mtp_h[0] == b.mtp_h[0]


@pytest.mark.parametrize("kv,context,length", [("fp32", 0, 130), ("fp32", 310, 20), ("fp32", 500, 17), ("bf16", 500, 17)])
def test_small_model_rows_share_their_keys(small, monkeypatch, kv, context, length):
    """Row blocks whose keys are shared by 2, 4 and 8 CTAs: whole shares, a last one that is short, and two empty ones."""
    from megakernels_b200 import engine as E
    from megakernels_b200.synth import make_prompt
    prompt, got = make_prompt(small[0], context + length), []
    for rows in (True, False):
        mk = E.Megakernel(small[:2], max_seq=576, quant="int8", kv_dtype=kv)
        with monkeypatch.context() as mp:
            mp.setattr(E, "MIN_PROMPT_ROWS", 1 << 30)
            if context:
                mk.run(prompt[:context])
            mp.setattr(E, "MIN_PROMPT_ROWS", 16 if rows else 1 << 30)
            mp.setattr(E, "EXACT_PROMPT", 0)
            got.append(mk.run(prompt[context:], n_generate=4, return_logits=True))
        assert (mk._workspace is not None) == rows
    (ia, la), (ib, lb) = got
    assert ia == ib and rel(la, lb) < (2e-5 if kv == "fp32" else 2e-4)              # a bf16 cache rounds


def test_small_model_batched_prompts_equal_stepping(small, monkeypatch):
    from megakernels_b200 import engine as E
    from megakernels_b200.synth import make_prompt
    prompts, got = [make_prompt(small[0], n, seed=n) for n in (60, 9, 17, 100)], []
    for rows in (16, 1 << 30):
        mk = E.Megakernel(small[:2], max_seq=256, quant="int8", batch=4)
        monkeypatch.setattr(E, "MIN_PROMPT_ROWS", rows)
        got.append((mk.run_batch(prompts, n_generate=8), mk))
        assert (mk._workspace is not None) == (rows == 16)
    (ia, a), (ib, b) = got
    assert ia == ib and a.bpos == b.bpos
    for x, y in zip(a.bstate + a.bconv_hist, b.bstate + b.bconv_hist):
        assert rel(x, y) < 2e-5


def test_small_model_refused_calls_leave_the_state_alone(small):
    """What a call refuses it refuses before the prompt goes in: bad arguments, formats and contexts the launch does not take."""
    from megakernels_b200 import _lib
    from megakernels_b200 import engine as E
    from megakernels_b200.synth import make_prompt
    prompt = make_prompt(small[0], 40)

    def untouched(mk):
        return mk.bpos == [0] * mk.batch and not any(bool(t.any()) for t in mk.bstate + mk.conv_hist + mk.bconv_hist + mk.k_cache)
    mk = E.Megakernel(small[:2], max_seq=256, quant="bf16")
    with pytest.raises((TypeError, ValueError)):
        mk.run(prompt, n_generate=2, stop_ids=["end"])
    assert untouched(mk)
    mk.reset()
    with pytest.raises(_lib.MkError, match="int8"):
        mk.run_batch([prompt], n_generate=2)
    assert untouched(mk)
    mk = E.Megakernel(small[:2], max_seq=4096, quant="int8", batch=8)
    with pytest.raises(_lib.MkError, match="too long"):
        mk.run_batch([make_prompt(small[0], 4060)] * 8, n_generate=8)
    assert untouched(mk)
    lv, _, g = mk._tables
    bare = dict(g, **dict.fromkeys(("xl", "projl", "mixl", "actl", "lml", "attn_part", "partl"), 0))
    gv = _lib.i64_array([bare[f] for f in _lib.GLOBAL_FIELDS])
    _lib.check(mk.lib.mk_set_params(mk._h, _lib.i64_array(lv), len(lv), None, 0, gv, len(gv)))
    mk.reset()
    with pytest.raises(_lib.MkError, match="hand-off"):
        mk.prefill(prompt)
    assert untouched(mk)


def test_small_model_prefill_reports_a_wait_that_ran_out(small):
    from megakernels_b200 import _lib
    from megakernels_b200 import engine as E
    from megakernels_b200.synth import make_prompt
    mk = E.Megakernel(small[:2], max_seq=256, quant="int8")
    mk.status[0] = _lib.MK_ERR_TIMEOUT                                # what a kernel leaves whose wait ran out
    with pytest.raises(_lib.MkError) as err:
        mk.prefill(make_prompt(small[0], 40))
    assert err.value.code == _lib.MK_ERR_TIMEOUT and mk.pos == 0
    mk.reset()
    mk.prefill(make_prompt(small[0], 40))
    assert mk.pos == 39


def test_small_model_without_a_deltanet_layer(lib_built):
    """A model of attention layers alone has no recurrent state to clear, keep or put back."""
    import dataclasses
    from megakernels_b200 import engine as E
    from megakernels_b200.config import qwen35_08b
    from megakernels_b200.synth import make_prompt, make_weights
    cfg = dataclasses.replace(qwen35_08b(n_layers=2, vocab=4096), layer_types=["full_attention"] * 2)
    mk = E.Megakernel((cfg, make_weights(cfg, 0, init="realistic")), max_seq=128, quant="bf16")
    prompt = make_prompt(cfg, 30)
    first = mk.run(prompt, n_generate=4)
    mk.reset()
    tail = mk.prefill(prompt)
    snap = mk.snapshot()
    assert mk.run([tail], n_generate=4) == first
    mk.restore(snap)
    assert mk.pos == 29 and mk.run([tail], n_generate=4) == first


def test_small_model_snapshots_kept_on_the_host(small):
    from megakernels_b200 import engine as E
    from megakernels_b200.synth import make_prompt
    mk = E.Megakernel(small[:2], max_seq=128, quant="int8")
    tail = mk.prefill(make_prompt(small[0], 30))
    tensors, pos, mode = mk.snapshot()
    first = mk.run([tail], n_generate=4)
    mk.restore(([t.cpu() for t in tensors], pos, mode))
    assert mk.run([tail], n_generate=4) == first


def test_prompts_step_where_no_memory_is_left(packed, small, monkeypatch):
    from megakernels_b200 import engine as E
    from megakernels_b200.synth import make_prompt
    pkg, shape = SHAPES["27b"]
    prompt, small_prompt = pkg.make_prompt(shape.vocab, 40, seed=3), make_prompt(small[0], 40)
    engines = [pkg.Engine(packed("27b", {}), 1, maxlen=128) for _ in range(2)]
    minis = [E.Megakernel(small[:2], max_seq=128, quant="int8") for _ in range(2)]
    real = torch.empty

    def full(*a, **k):
        if k.get("dtype") == torch.uint8:
            raise torch.cuda.OutOfMemoryError("no memory left")
        return real(*a, **k)
    got = []
    for eng, mk, arm in zip(engines, minis, ("full", "stepping")):
        with monkeypatch.context() as mp:
            if arm == "full":
                mp.setattr(torch, "empty", full)
            else:
                mp.setattr(runtime, "MIN_ROWS_PATH", 1 << 30)
                mp.setattr(E, "MIN_PROMPT_ROWS", 1 << 30)
            logits = eng.prefill([prompt]).clone()
            tail = mk.prefill(small_prompt)
            ids = mk.run([tail], n_generate=3)
            mk.reset()
            got.append((logits, ids, mk.run(small_prompt, n_generate=3), mk.bstate))
        assert eng.rt._workspace is None and mk._workspace is None
    (la, ia, ja, sa), (lb, ib, jb, sb) = got
    assert torch.equal(la, lb) and ia == ib and ja == jb and all(torch.equal(x, y) for x, y in zip(sa, sb))
    assert minis[0].run([1] * 30, n_generate=1) and minis[0]._workspace is not None     # memory again


@pytest.mark.parametrize("quant,length", [("bf16", 30), ("bf16", 150), ("bf16", 260), ("int8", 170), ("int8", 320)])
def test_small_model_prompts_are_as_exact_as_stepping(small, monkeypatch, quant, length):
    """Both paths against the decoder in 64 bits: sums in tensor memory round towards zero, so long ones drift (a single
    accumulator per product left a bf16 prompt five times as far from 64 bits as stepping).  Lengths: tiles of 32 and 80 to
    160 tokens, one to three of them."""
    from megakernels_b200 import engine as E
    from megakernels_b200.quant import dequantized_weights
    from megakernels_b200.synth import make_prompt
    from oracle import decoder

    def rms_norm(x, w, eps):
        return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps) * (w + 1.0)
    monkeypatch.setattr(decoder, "rms_norm", rms_norm)
    cfg, w = small[:2]
    prompt = make_prompt(cfg, length)
    d = decoder.Decoder(cfg, dequantized_weights(w, quant), max_seq=length)
    d.w, d.cos, d.sin = {k: v.double() for k, v in d.w.items()}, d.cos.double(), d.sin.double()
    for kept in (d.conv_hist, d.state, d.k_cache, d.v_cache):
        for k in kept:
            kept[k] = kept[k].double()
    for t in prompt[:-1]:
        d.hidden_step(t)
    off = []
    for rows in (16, 1 << 30):
        mk = E.Megakernel((cfg, w), max_seq=512, quant=quant)
        monkeypatch.setattr(E, "MIN_PROMPT_ROWS", rows)
        mk.prefill(prompt)
        assert (mk._workspace is not None) == (rows == 16)
        states = [rel(mk.deltanet_state(i).cpu(), s) for i, s in enumerate(d.state[i] for i in sorted(d.state))]
        off.append(sum(states) / len(states))
    assert off[0] < 1.5 * off[1] and off[0] < 5e-6, off


@pytest.mark.parametrize("model,M,length", [("26b", 5, 30), ("26b", 8, 50), ("26b", 8, 101), ("26b", 8, 200), ("35b", 8, 49), ("35b", 8, 101), ("35b", 8, 200)])
def test_prompt_rows_of_crowded_experts(model, M, length):
    """Routed products by the width of a work item (the mean load of 128 experts: 32, 64, 128 and 256 tokens; block-scaled ones up to a
    mean of 96 in items of 32, several an expert); 26b: 11 blocks of 64 columns in the down-projection, the last weight block past the matrix.
    Every position is compared: keys and values behind the first routed layers, row by row.  26b: a position whose last expert is another one
    for a flipped rounding is 0.08 to 0.1 off in the second layer, the others at most 5e-3; 35b: all at most 1.7e-2 in the fourth."""
    pkg, shape = SHAPES[model]
    shape = shape.with_(eff=704, hidden=576) if model == "26b" else shape.with_(experts=128)
    PK = pkg.Packed(pkg.SynthWeights(shape, layers=shape.layers, init="realistic", device="cuda"), "cuda")
    prompts = [pkg.make_prompt(shape.vocab, length, seed=j) for j in range(M)]
    out = []
    for rows in (True, False):
        eng = pkg.Engine(PK, M, maxlen=length + 64)
        with pytest.MonkeyPatch.context() as mp:
            if not rows:
                mp.setattr(runtime, "MIN_ROWS_PATH", 1 << 30)
            out.append((eng, eng.prefill(prompts).clone()))
        assert (eng.rt._workspace is not None) == rows
        eng.check()
    (a, la), (b, lb) = out
    assert rel(la, lb) < 3e-2

    def off(*layer):                                     # per sequence and position: keys and values of all heads
        x, y = (torch.stack([torch.cat(e.kv_rows(*layer, m, length)) for m in range(M)]).double() for e in (a, b))
        return ((x - y).norm(dim=(1, 3)) / y.norm(dim=(1, 3))).flatten()
    if model == "26b":
        assert rel(a.ks[0], b.ks[0]) < 1e-3 and rel(a.vs[0], b.vs[0]) < 1e-3
        assert rel(a.kf, b.kf) < 3e-2 and rel(a.vf, b.vf) < 3e-2
        second = off(False, 1)
        assert float(second.max()) < 0.15 and float((second > 0.02).double().mean()) < 0.02
    else:
        assert rel(a.ssm[0], b.ssm[0]) < 4e-4 and rel(a.ssm, b.ssm) < 1e-2 and rel(a.conv, b.conv) < 1e-2
        assert float(off(0).max()) < 5e-2


@pytest.mark.parametrize("fmt,M,length", [({}, 1, 258), ({}, 1, 386), ({}, 2, 386), ({"fmt": "bf16"}, 3, 130)])
def test_prompt_rows_in_wide_tiles(packed, fmt, M, length):
    """Tiles of more than 256 tokens (two MMAs per step): just over that, the widest one and a row past it, two of them.  The first
    layer's state sees no earlier bf16 rounding, so it agrees to fp32 sums."""
    pkg, shape = SHAPES["27b"]
    prompts, engines = [pkg.make_prompt(shape.vocab, length, seed=j) for j in range(M)], []
    for rows in (True, False):
        eng = pkg.Engine(packed("27b", fmt), M, maxlen=length + 64)
        with pytest.MonkeyPatch.context() as mp:
            if not rows:
                mp.setattr(runtime, "MIN_ROWS_PATH", 1 << 30)
            engines.append((eng, eng.prefill(prompts).clone()))
        assert (eng.rt._workspace is not None) == rows
        eng.check()
    (a, la), (b, lb) = engines
    assert rel(la, lb) < 3e-2 and rel(a.ssm[0], b.ssm[0]) < 2e-4 and rel(a.ssm, b.ssm) < 1e-2
