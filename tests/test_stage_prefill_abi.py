"""Which programs `mk_stage_prefill` takes (no GPU needed: the check follows the host records and touches no device).

A program it refuses (MK_ERR_UNSUPPORTED) steps through its prompts, so a record that it would read differently from the
decode kernel must be refused: the cases change one record of an accepted program at a time."""

import ctypes

import pytest

from megakernels_b200 import _lib
from megakernels_b200.stage import desc as D

H, Y, FFN, E = 256, 2048, 128, 128


def _gemv(x, out, n, K, *, x_stride, out_stride, fmt=D.MKS_FMT_BF16, tiles=None, **kw):
    i = dict(FMT=fmt, TILES=tiles or -(-n // 16), SPLITS=1, GROUPS=1, UNIT_STEPS=K // 16, CHUNK_STEPS=8, CHUNK_BYTES=4096, KC=K, PROLOGUE=D.MKS_P_PLAIN,
             EPILOGUE=D.MKS_E_STORE, N_VALID=n, X_STRIDE=x_stride, OUT_STRIDE=out_stride, K_TOTAL=K, PIECES=1)
    p = dict(W=0x1000, X=x, OUT=out)
    for k, v in kw.items():
        (p if k in ("X_SSQ", "NORM_W", "OUT_SSQ", "KEYS", "CNT", "PART", "W_SHARED") else i)[k] = v
    return D.desc(D.MKS_OP_GEMV, 0, i=i, p=p)


def _program():
    """Every kind of record once; addresses stand for buffers [2 sequences][width] of fp32."""
    h, ssq, y, y2, act, rt, ex = 0x100000, 0x200000, 0x300000, 0x400000, 0x500000, 0x600000, 0x700000
    a, assq = 0x800000, 0x900000
    norm = dict(PROLOGUE=D.MKS_P_NORM, X_SSQ=ssq, NORM_W=0x10)
    resid = dict(EPILOGUE=D.MKS_E_RESID, OUT_SSQ=ssq)
    return dict(
        embed=D.desc(D.MKS_OP_EMBED, 0, i=dict(HIDDEN=H, VOCAB=100), p=dict(TABLE=0x10, H=h, H_SSQ=ssq)),
        inp=_gemv(h, y, 1024, H, x_stride=H, out_stride=Y, **norm),
        ba=_gemv(h, y + 1024 * 4, 4, H, x_stride=H, out_stride=Y, **norm),
        gdn=D.desc(D.MKS_OP_GDN, 0, i=dict(NKH=1, NVH=2, Q_OFF=0, K_OFF=128, V_OFF=256, Z_OFF=512, B_OFF=1024, A_OFF=1026, CONV_DIM=512, Y_STRIDE=Y, Y2_STRIDE=512),
                   p=dict(Y=y, Y2=y2)),
        out=_gemv(y2, h, H, 256, x_stride=512, out_stride=H, **resid),
        qkv=_gemv(h, y, 1536, H, x_stride=H, out_stride=Y, **norm),
        attn=D.desc(D.MKS_OP_ATTN, 0, i=dict(NQ=2, NKV=1, HD=256, ROT=64, ROPE_PAIRS=32, A_Q_OFF=0, A_Q_HSTRIDE=512, A_GATE_OFF=256, A_K_OFF=1024, A_V_OFF=1280,
                                             A_Y_STRIDE=Y, A_Y2_STRIDE=512, CHUNK_POS=64, MAX_PAGES=4, MAX_CHUNKS=16, Q_BF16=1), p=dict(A_Y=y, A_Y2=y2)),
        o=_gemv(y2, h, H, 512, x_stride=512, out_stride=H, **resid),
        gu=_gemv(h, act, FFN, H, x_stride=H, out_stride=FFN, tiles=16, EPILOGUE=D.MKS_E_GLU, **norm),
        down=_gemv(act, a, H, FFN, x_stride=FFN, out_stride=H, OUT_SSQ=assq),
        vec=D.desc(D.MKS_OP_VEC, 0, i=dict(VEC_N=H), p=dict(VEC_BASE=h, VEC_A=a, VEC_A_SSQ=assq, VEC_A_W=0x10, VEC_OUT=h, VEC_OUT_SSQ=ssq)),
        router=_gemv(h, rt, E + 1, H, x_stride=H, out_stride=144, **norm),
        route=D.desc(D.MKS_OP_ROUTE, 0, i=dict(EXPERTS=E, TOPK=8, LOGIT_STRIDE=144, ROUTE_KIND=0), p=dict(LOGITS=rt)),
        ex_gu=_gemv(h, ex, FFN, H, x_stride=H, out_stride=FFN, tiles=16, EPILOGUE=D.MKS_E_GLU, GROUPS=-1, OUT_GSTRIDE=2 * FFN, W_SHARED=0x20, **norm),
        ex_down=_gemv(ex, h, H, FFN, x_stride=FFN, out_stride=H, GROUPS=-1, X_GSTRIDE=2 * FFN, REDUCE_GROUPS=1, CNT=0x10, PART=0x10, W_SHARED=0x20, **resid),
        lm=_gemv(h, 0xA00000, 100, H, x_stride=H, out_stride=100, EPILOGUE=D.MKS_E_LOGITS, KEYS=0x10, **norm),
    )


def _answer(stages, positions=64):
    arr = (D.StageDesc * len(stages))(*stages)
    return D.lib().mk_stage_prefill_bytes(arr, len(stages), 2, positions, 0)


def test_the_program_is_taken(lib_built):
    got = _answer(list(_program().values()))
    assert got > 0 or got == _lib.MK_ERR_CUDA, D.lib().mk_last_error()       # (no device here: it got as far as asking for one)
    for less in (["lm"], ["router", "route", "ex_gu", "ex_down"], ["vec", "down", "gu"]):
        got = _answer([d for k, d in _program().items() if k not in less])
        assert got > 0 or got == _lib.MK_ERR_CUDA, (less, D.lib().mk_last_error())


I, P = True, False
CASES = [
    # (record, index kind, field, value) -> refused
    ("inp", I, "PIECES", 2), ("inp", I, "ALLREDUCE", 1), ("inp", I, "GROUPS", 2), ("inp", I, "K_TOTAL", 512), ("inp", I, "X_STRIDE", 128),
    ("inp", P, "X", 0xB00000), ("inp", P, "X_SSQ", 0xB00000), ("inp", I, "N_VALID", 512),                     # (z is then unwritten)
    ("ba", P, "OUT", 0x300000 + 1030 * 4), ("ba", I, "OUT_STRIDE", 1024), ("ba", P, "OUT", 0x300000 + 8192 + 64),       # the last: inside the second row
    ("gdn", I, "Z_OFF", 1032), ("gdn", I, "K_OFF", 130), ("gdn", I, "CONV_DIM", 640), ("gdn", P, "Y", 0xB00000), ("gdn", P, "Y2", 0x100000),
    ("out", I, "PROLOGUE", 1), ("out", I, "X_STRIDE", 256), ("out", P, "OUT", 0xB00000), ("o", I, "REDUCE_GROUPS", 1),
    ("attn", I, "KV_F32", 1), ("attn", I, "Q_BF16", 0), ("attn", I, "ROT", 32), ("attn", I, "ROPE_PAIRS", 64), ("attn", I, "NKV", 2), ("attn", I, "A_V_OFF", 1284),
    ("attn", P, "A_Y2", 0x400000 + 64),
    ("gu", P, "OUT", 0x100000), ("gu", I, "N_VALID", 96), ("down", P, "X", 0x500010), ("down", P, "OUT_SSQ", 0),
    ("vec", P, "VEC_A", 0x300000), ("vec", P, "VEC_BASE", 0xB00000), ("vec", P, "VEC_B", 0xB00000), ("vec", I, "VEC_N", 128),
    ("route", P, "LOGITS", 0xB00000), ("route", I, "LOGIT_STRIDE", 128), ("route", I, "ROUTE_KIND", 1), ("router", I, "N_VALID", 128),
    ("ex_gu", I, "X_GSTRIDE", 512), ("ex_gu", P, "W_SHARED", 0), ("ex_down", P, "X", 0x500000), ("ex_down", I, "REDUCE_GROUPS", 0), ("ex_down", I, "X_GSTRIDE", 512),
    ("lm", P, "X", 0x800000), ("lm", P, "X_SSQ", 0x900000),
]


@pytest.mark.parametrize("name,integer,field,value", CASES, ids=[f"{c[0]}-{c[2]}-{c[3]:x}" for c in CASES])
def test_records_of_another_form_are_refused(lib_built, name, integer, field, value):
    prog = _program()
    d = prog[name]
    if integer:
        d.i[D.K["MKS_I_" + field]] = value
    else:
        d.p[D.K["MKS_P_" + field]] = value
    for needs, *pointers in (("VEC_B", "VEC_B_SSQ", "VEC_B_W"), ("PROLOGUE", "X_SSQ", "NORM_W"), ("REDUCE_GROUPS", "CNT", "PART")):
        if field == needs:
            for p in pointers:
                d.p[D.K["MKS_P_" + p]] = 0x10
    assert D.lib().mk_stage_validate((D.StageDesc * len(prog))(*prog.values()), len(prog), 2) == _lib.MK_OK      # the decode kernel takes it
    assert _answer(list(prog.values())) == _lib.MK_ERR_UNSUPPORTED, D.lib().mk_last_error()


@pytest.mark.parametrize("order", [["ba", "inp"], ["ex_gu", "route"], ["lm", "o"]])
def test_records_in_another_order_are_refused(lib_built, order):
    prog = _program()
    names = list(prog)
    a, b = (names.index(n) for n in order)
    names[a], names[b] = names[b], names[a]
    assert _answer([prog[n] for n in names]) == _lib.MK_ERR_UNSUPPORTED, D.lib().mk_last_error()


def test_malformed_programs_and_sizes_are_errors(lib_built):
    prog = _program()
    stages = list(prog.values())
    assert _answer(stages, positions=40000) == _lib.MK_ERR_BADARG           # 80000 rows
    assert _answer(stages[1:]) == _lib.MK_ERR_BADARG
    prog["inp"].i[D.K["MKS_I_CHUNK_STEPS"]] = 3
    assert _answer(stages) == _lib.MK_ERR_BADARG
    a = D.PrefillArgs(program=ctypes.addressof((D.StageDesc * 1)(prog["embed"])), n_stages=1, batch=2, positions=40000, tokens=16, pos=16, status=16, workspace=1024)
    assert D.lib().mk_stage_prefill(ctypes.byref(a), None) == _lib.MK_ERR_BADARG


def test_prompt_kernels_own_tensor_memory_before_the_next_one_starts():
    """Read in the source: every kernel of the chain waits for the one before, and one that allocates tensor memory lets the next kernel's CTAs
    come up only behind the barrier that follows the allocation.  (What breaks the rule would hang a GPU, so no run can show it.)"""
    import os
    import re
    csrc = os.path.join(os.path.dirname(_lib.__file__), "csrc")
    text = open(os.path.join(csrc, "mk_prefill.cuh")).read() + open(os.path.join(csrc, "mk_prefill_08b.cu")).read()
    heads = [m.start() for m in re.finditer(r"__global__ void", text)]
    allocating = 0
    for at, end in zip(heads, heads[1:] + [len(text)]):
        body = text[at: re.compile(r"^}", re.M).search(text, at).end()]
        name = re.search(r"(\w+)\(", body[body.index(")") if "__launch_bounds__" in body.split("\n")[0] else 0:]).group(1)
        if name.startswith("slabs_from"):                    # lays the weights out once, not a kernel of a pass
            continue
        assert re.search(r"chain_(wait|acquire)\(\)", body), name
        alloc = body.find("tcgen05.alloc")
        if alloc < 0:
            continue
        allocating += 1
        owned = body.index("__syncthreads()", alloc)
        assert all(m.start() > owned for m in re.finditer(r"chain_(wait|release)\(\)", body)), name
    assert allocating == 1
