"""The work whose speed this library answers for, as cases that any build of it can be timed on.

`listed()` names them, `draw(rng)` gives another one of the same ranges, `prepare(case, seed)` makes what a program holds
before the call (an engine, a context, token ids), `run(state)` is one pass through the public entry points and returns
everything it computed, `work(case)` says what a pass cannot do without, `tolerance(case)` how far another correct
implementation may be off.

Two kinds of engine are measured:

* the 0.8B hybrid at full depth (`Megakernel`): a single call for one token, a short prompt with its reply, plain and batched
  generation, speculative cycles, and taking a long prompt in.  Its arithmetic is exact to fp32 rounding, so the chosen ids
  are part of the result;
* the 27B, 35B-A3B and 26B-A4B models (`Engine`) at their full widths and vocabularies, with one or two periods of the layer
  pattern as depth (every layer of a kind costs the same, and the weights of the shortest stack exceed the L2 several
  times): steps as a serving loop makes them, one call per token for all its sequences with the tokens given, and prompts.

Weights are seeded and synthetic; a program loads them once, so they are made once per process and shared by the states.
What a state holds apart from them (caches, recurrent state, token ids) comes from its own seed.
"""

import math

import torch

from megakernels_b200 import gemma26b, qwen27b, qwen35moe
from megakernels_b200.config import qwen35_08b
from megakernels_b200.engine import Megakernel

DEVICE = "cuda"
VOCAB_08B = 151936
LAYERS = {"27b": 8, "35b": 8, "26b": 6}
MODELS = {"27b": qwen27b, "35b": qwen35moe, "26b": gemma26b}
CONTEXT = {"27b": 2048, "35b": 4096, "26b": 8192}          # the prompt lengths of the benchmark's configurations


# ---------------------------------------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------------------------------------
def listed():
    return [
        # one token through the small model, as a loop that samples outside the engine asks for it: latency is everything
        {"name": "0.8b int8, one token", "model": "0.8b", "quant": "int8", "op": "generate", "context": 117, "steps": 1, "logits": True},
        # configuration 1: a 32-token prompt and its 128-token reply in one call
        {"name": "0.8b bf16, 32 + 128", "model": "0.8b", "quant": "bf16", "op": "chat", "prompt": 32, "steps": 128},
        # configuration 2, inside a reply: the stretch of tokens a streaming server asks for at a time
        {"name": "0.8b int8, generate", "model": "0.8b", "quant": "int8", "op": "generate", "context": 700, "steps": 48, "logits": False},
        # configuration 2 at batch 8, sequences at different positions
        {"name": "0.8b int8, generate x8", "model": "0.8b", "quant": "int8", "op": "batch", "batch": 8, "context": 640, "steps": 32},
        # configuration 2 with the draft head: speculative cycles
        {"name": "0.8b int8, speculative", "model": "0.8b", "quant": "int8", "op": "spec", "context": 530, "steps": 24},
        # configuration 2: a 512-token prompt up to its first token (what a chat user waits for)
        {"name": "0.8b int8, prompt of 512", "model": "0.8b", "quant": "int8", "op": "prompt", "prompt": 512},
        # configuration 3, one user and a full batch, at the benchmark's context
        {"name": "27b, steps x1", "model": "27b", "op": "step", "batch": 1, "context": 2048, "steps": 6},
        {"name": "27b, steps x8", "model": "27b", "op": "step", "batch": 8, "context": 2048, "steps": 6},
        # configuration 3: a prompt comes in
        {"name": "27b, prompt of 384", "model": "27b", "op": "prompt", "batch": 1, "prompt": 384},
        # configuration 4: routed experts at a full batch, and prompts of two users
        {"name": "35b, steps x8", "model": "35b", "op": "step", "batch": 8, "context": 4096, "steps": 6},
        {"name": "35b, prompts of 250 x2", "model": "35b", "op": "prompt", "batch": 2, "prompt": 250},
        # configuration 5: sliding-window layers, a few users with long contexts
        {"name": "26b, steps x4", "model": "26b", "op": "step", "batch": 4, "context": 8000, "steps": 6},
    ]


def _log(rng, lo, hi):
    """A whole number between lo and hi, spread over the logarithm."""
    return max(lo, min(hi, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def draw(rng):
    if rng.random() < 0.5:
        op = rng.choice(["generate", "chat", "batch", "spec", "prompt"])
        c = {"model": "0.8b", "quant": "int8" if op in ("batch", "spec") else rng.choice(["int8", "bf16"]), "op": op}
        if op == "generate":
            c.update(context=_log(rng, 16, 4000), steps=_log(rng, 1, 64), logits=rng.random() < 0.5)
        elif op == "chat":
            c.update(prompt=_log(rng, 4, 128), steps=_log(rng, 8, 128))
        elif op == "batch":
            c.update(batch=rng.randint(2, 8), context=_log(rng, 16, 2000), steps=_log(rng, 1, 48))
        elif op == "spec":
            c.update(context=_log(rng, 16, 2000), steps=_log(rng, 2, 32))
        else:
            c.update(prompt=_log(rng, 100, 700))
        return c
    model = rng.choice(sorted(MODELS))
    if rng.random() < 0.6:
        return {"model": model, "op": "step", "batch": rng.randint(1, 8), "context": _log(rng, 64, CONTEXT[model]), "steps": _log(rng, 1, 8)}
    batch = rng.randint(1, 4)
    return {"model": model, "op": "prompt", "batch": batch, "prompt": _log(rng, 40, 384)}


# ---------------------------------------------------------------------------------------------------------
# weights: one set per process and model
# ---------------------------------------------------------------------------------------------------------
_weights = {}


def _normal(gen, shape, mean=0.0, std=1.0, dtype=torch.bfloat16):
    return torch.empty(shape, device=DEVICE).normal_(mean, std, generator=gen).to(dtype)


def _small_weights():
    """The 0.8B model (matrices N(0, 0.02), a recurrent branch that carries signal) and its draft head."""
    if "0.8b" in _weights:
        return _weights["0.8b"]
    cfg = qwen35_08b(vocab=VOCAB_08B)
    gen = torch.Generator(device=DEVICE).manual_seed(0)
    H, D, nh = cfg.hidden, cfg.head_dim, cfg.lin_heads

    def n(*shape, mean=0.0, std=0.02):
        return _normal(gen, shape, mean, std)

    def attention(p, w):
        w[p + "q_proj.weight"], w[p + "k_proj.weight"] = n(2 * cfg.n_heads * D, H), n(cfg.n_kv_heads * D, H)
        w[p + "v_proj.weight"], w[p + "o_proj.weight"] = n(cfg.n_kv_heads * D, H), n(H, cfg.n_heads * D)
        w[p + "q_norm.weight"], w[p + "k_norm.weight"] = n(D), n(D)

    def around(p, w):
        w[p + "input_layernorm.weight"], w[p + "post_attention_layernorm.weight"] = n(H), n(H)
        w[p + "mlp.gate_proj.weight"], w[p + "mlp.up_proj.weight"] = n(cfg.intermediate, H), n(cfg.intermediate, H)
        w[p + "mlp.down_proj.weight"] = n(H, cfg.intermediate)

    w = {"embed_tokens.weight": n(cfg.vocab, H), "norm.weight": n(H)}
    for i, kind in enumerate(cfg.layer_types):
        p = f"layers.{i}."
        around(p, w)
        if kind == "linear_attention":
            q = p + "linear_attn."
            w[q + "in_proj_qkv.weight"], w[q + "in_proj_z.weight"] = n(cfg.conv_dim, H), n(nh * cfg.lin_v_dim, H)
            w[q + "in_proj_b.weight"], w[q + "in_proj_a.weight"] = n(nh, H), n(nh, H)
            w[q + "conv1d.weight"] = n(cfg.conv_dim, 1, cfg.conv_k, mean=0.5, std=0.2)
            w[q + "A_log"], w[q + "dt_bias"] = n(nh, mean=-1.0, std=1.0).float(), n(nh, std=1.0)
            w[q + "norm.weight"], w[q + "out_proj.weight"] = n(cfg.lin_v_dim, mean=1.0, std=0.1), n(H, nh * cfg.lin_v_dim)
        else:
            attention(p + "self_attn.", w)
    m = {"fc.weight": n(H, 2 * H), "pre_fc_norm_embedding.weight": n(H), "pre_fc_norm_hidden.weight": n(H), "norm.weight": n(H)}
    around("layers.0.", m)
    attention("layers.0.self_attn.", m)
    _weights["0.8b"] = cfg, w, m
    return _weights["0.8b"]


def _large_weights(model):
    if model not in _weights:
        pkg, layers = MODELS[model], LAYERS[model]
        kw = {"keep_dequant": False} if model == "27b" else ({"keep_dense": False} if model == "35b" else {})
        W = pkg.SynthWeights(layers=layers, seed=0, init="realistic", device=DEVICE, draw_device=DEVICE, **kw)
        _weights[model] = pkg.Packed(W, DEVICE)
    return _weights[model]


# ---------------------------------------------------------------------------------------------------------
# states
# ---------------------------------------------------------------------------------------------------------
def prepare(case, seed):
    gen = torch.Generator(device=DEVICE).manual_seed(seed)
    return (_prepare_small if case["model"] == "0.8b" else _prepare_large)(case, gen)


def _ids(gen, vocab, *shape):
    return torch.randint(0, vocab, shape, device=DEVICE, generator=gen, dtype=torch.int32)


def _fill(gen, tensors, std):
    for t in tensors:
        t.normal_(0.0, std, generator=gen)


def _prepare_small(case, gen):
    cfg, w, m = _small_weights()
    op, batch = case["op"], case.get("batch", 1)
    context, new = case.get("context", 0), case.get("prompt", 0) + case.get("steps", 1) * (2 if op == "spec" else 1)
    mk = Megakernel((cfg, w, m), max_seq=context + new + 64, quant=case["quant"], device=DEVICE, batch=batch, mtp=op == "spec")
    s = {"case": case, "mk": mk}
    if case.get("prompt"):
        s["prompt"] = _ids(gen, cfg.vocab, case["prompt"]).tolist()
        return s
    # a context as the tokens before it would have left it: normed keys, values and conv inputs of a projection's size
    _fill(gen, mk.k_cache + mk.v_cache, 1.0)
    if mk.mtp is not None:
        _fill(gen, [mk.mtp_k_cache, mk.mtp_v_cache], 1.0)
    _fill(gen, mk.bstate, 0.05)
    if op == "batch":
        _fill(gen, mk.bconv_hist, 0.6)
        s["pos"] = [max(1, context - 7 * j) for j in range(batch)]
        s["tokens"] = [[t] for t in _ids(gen, cfg.vocab, batch).tolist()]
    else:
        for i in range(len(mk.conv_hist)):
            mk.set_conv_window(i, torch.empty(cfg.conv_dim, 3, device=DEVICE).normal_(0.0, 0.6, generator=gen), context)
        s["token"], s["draft"] = _ids(gen, cfg.vocab, 2).tolist()
    return s


def _prepare_large(case, gen):
    PK = _large_weights(case["model"])
    batch = case["batch"]
    eng = MODELS[case["model"]].Engine(PK, batch, maxlen=case.get("context", 0) + case.get("prompt", 0) + case.get("steps", 0) + 64, device=DEVICE)
    s = {"case": case, "eng": eng}
    vocab = PK.shape.vocab
    if case["op"] == "prompt":
        s["prompts"] = _ids(gen, vocab, batch, case["prompt"]).tolist()
        return s
    if case["model"] == "26b":
        _fill(gen, [eng.ks, eng.kf], 0.25)
        _fill(gen, [eng.vs, eng.vf], 1.0)
    else:
        _fill(gen, [eng.k_cache, eng.v_cache], 1.0)
        _fill(gen, [eng.ssm], 0.05)
        _fill(gen, [eng.conv], 1.0)
    s["tokens"] = list(_ids(gen, vocab, case["steps"], batch))
    s["pos"] = torch.zeros(eng.pos.shape, dtype=torch.int32, device=DEVICE)
    s["pos"][:batch] = case["context"] - 5 * torch.arange(batch, dtype=torch.int32, device=DEVICE).clamp_max(case["context"] // 10)
    return s


# ---------------------------------------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------------------------------------
def run(state):
    return (_run_small if "mk" in state else _run_large)(state)


def _run_small(s):
    case, mk = s["case"], s["mk"]
    op = case["op"]
    if op == "chat":
        mk.reset()
        ids = mk.run(s["prompt"], n_generate=case["steps"])
    elif op == "prompt":
        mk.reset()
        ids = mk.run([mk.prefill(s["prompt"])], n_generate=1)
    elif op == "generate":
        mk.pos = case["context"]                       # every pass continues from the same context
        if case["logits"]:
            ids, logits = mk.run([s["token"]], n_generate=case["steps"], return_logits=True)
            return {"ids": torch.tensor(ids), "logits": logits, "state": mk.bstate}
        ids = mk.run([s["token"]], n_generate=case["steps"])
    elif op == "batch":
        mk.bpos = list(s["pos"])
        ids = mk.run_batch(s["tokens"], n_generate=case["steps"])
    else:
        mk.pos = case["context"]
        ids, draft = mk.run_spec(s["token"], s["draft"], case["steps"])
        return {"ids": torch.tensor(ids), "draft": draft, "state": mk.state, "keys": mk.k_cache, "values": mk.v_cache}
    return {"ids": torch.tensor(ids), "state": mk.bstate, "conv": mk.bconv_hist if op == "batch" else mk.conv_hist,
            "keys": mk.k_cache, "values": mk.v_cache}


def _run_large(s):
    case, eng = s["case"], s["eng"]
    if case["op"] == "prompt":
        eng.reset()
        logits = eng.prefill(s["prompts"])
    else:
        eng.pos.copy_(s["pos"])                        # every pass continues from the same context
        for tok in s["tokens"]:
            logits = eng.step(tok)
    out = {"logits": logits}
    if case["model"] == "26b":
        out.update(keys=[eng.ks, eng.kf], values=[eng.vs, eng.vf])
    else:
        out.update(keys=eng.k_cache, values=eng.v_cache, state=eng.ssm, conv=eng.conv)
    return out


# ---------------------------------------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------------------------------------
def _shape_costs(model, quant=None):
    """(bytes of the layers' dense weights, values of them, bytes of the LM head, values of it, recurrent state bytes per
    sequence, KV bytes per position and sequence, experts: (layers, experts, top-k, bytes of one, values of one))."""
    if model == "0.8b":
        c = qwen35_08b(vocab=VOCAB_08B)
        b = 1 if quant == "int8" else 2
        n_gdn = sum(k == "linear_attention" for k in c.layer_types)
        body = n_gdn * (c.gdn_in_rows + c.lin_heads * c.lin_v_dim) * c.hidden + 3 * c.n_layers * c.intermediate * c.hidden
        body += (c.n_layers - n_gdn) * (c.attn_in_rows + c.n_heads * c.head_dim) * c.hidden
        return body * b, body, c.vocab * c.hidden * b, c.vocab * c.hidden, n_gdn * c.lin_heads * 128 * 128 * 4, \
            (c.n_layers - n_gdn) * 2 * c.n_kv_heads * c.head_dim * 4, None
    s, L = MODELS[model].FULL, LAYERS[model]
    head = s.vocab * s.hidden
    if model == "26b":
        full = sum(s.is_full(i) for i in range(L))
        body = sum((s.qkv_n(i) + s.nq * s.attn_dims(i)[1]) * s.hidden for i in range(L)) + L * 3 * s.ffn * s.hidden
        router = L * s.experts * s.hidden
        return body + 2 * router, body + router, 2 * head, head, 0, full * 2 * s.nkv_f * s.hd_f * 2, \
            (L, s.experts, s.topk, 3 * s.eff * s.hidden, 3 * s.eff * s.hidden)
    att = sum(s.is_attn(i) for i in range(L))
    mixers = (L - att) * (s.inp_n + s.val_dim) * s.hidden + att * (s.qkv_n + s.nq * 256) * s.hidden
    state, kv = (L - att) * s.nvh * 128 * 128 * 4, att * 2 * s.nkv * 256 * 2
    if model == "27b":
        body = mixers + L * 3 * s.ffn * s.hidden
        return body * 17 // 32, body, 2 * head, head, state, kv, None
    body, router = mixers + L * 3 * s.sfi * s.hidden, L * (s.experts + 1) * s.hidden
    return body + 2 * router, body + router, 2 * head, head, state, kv, (L, s.experts, s.topk, 3 * s.fi * s.hidden, 3 * s.fi * s.hidden)


def work(case):
    body_b, body_n, head_b, head_n, state, kv, moe = _shape_costs(case["model"], case.get("quant"))
    batch, prompt, steps, context = case.get("batch", 1), case.get("prompt", 0), case.get("steps", 1), case.get("context", 0)
    if case["op"] == "prompt" and case["model"] != "0.8b":
        steps = 1

    def experts(tokens):
        if moe is None:
            return 0.0, 0.0
        layers, n, top, b, v = moe
        return layers * n * (1.0 - (1.0 - top / n) ** tokens) * b, layers * top * v * tokens

    nbytes = flops = 0.0
    if prompt:                                          # the weights once, the state and the caches written
        eb, ev = experts(batch * prompt)
        nbytes += body_b + eb + batch * (state + kv * prompt)
        flops += 2 * (body_n * batch * prompt + ev) + 2 * head_n * batch
        nbytes += head_b
        steps = steps - 1
    if case["model"] == "26b" and not prompt:           # sliding layers read at most their window
        s = MODELS["26b"].FULL
        window = sum(not s.is_full(i) for i in range(LAYERS["26b"])) * 2 * s.nkv_s * s.hd_s * 2 * min(context, s.window)
    else:
        window = 0
    for i in range(steps):                              # a step depends on the one before: the weights pass once per step
        eb, ev = experts(batch)
        nbytes += body_b + eb + head_b + batch * (2 * state + kv * (context + prompt + i) + window)
        flops += 2 * (body_n + head_n) * batch + 2 * ev
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    if case["model"] == "0.8b":
        # exact products, fp32 sums over two dozen layers
        return {"rel": 1e-4, "differ": 0.0}
    # GEMV inputs, keys and values are rounded to bf16 in every layer: sums in another order flip such roundings (a change
    # of 1e-6 in the norm weights moves the logits behind a prompt by 8e-3 of their norm); where experts are routed, now and
    # then they also swap the last chosen expert with the next one
    return {"rel": 1.5e-2 if case["model"] == "27b" else 3e-2}
