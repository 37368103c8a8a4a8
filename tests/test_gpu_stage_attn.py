"""The attention stage alone, through the C ABI, against attention in fp64 over the same rounded queries, keys and values:
tasks of one to several sub-chunks of 256 positions (a task is a chunk of one sequence and KV head; a CTA gets about one, so
eight sequences of eight KV heads leave two chunks each), ragged lengths, a window, both head dims, heads that do not fill
the MMA columns."""

import pytest
import torch

pytestmark = pytest.mark.gpu

from megakernels_b200.stage import desc as D
from megakernels_b200.stage.runtime import Program, Runtime

EPS = 1e-6


def _bf(x):
    return x.to(torch.bfloat16).float()


def _head(x, w, cos, sin):
    """RMS norm with 1 + w, rotation of the first 2 * cos.shape[-1] dims, rounding to bf16."""
    n = x * torch.rsqrt((x * x).mean(-1, keepdim=True) + EPS) * (1.0 + w)
    h = cos.shape[-1]
    a, b = n[..., :h], n[..., h: 2 * h]
    return _bf(torch.cat([a * cos - b * sin, b * cos + a * sin, n[..., 2 * h:]], -1))


def _run(M, nkv, qpk, HD, lengths, window=0, seed=0, exact=False):
    """`exact`: queries and new keys of +-1 and no rotation, so that nothing but the attention itself rounds."""
    dev = torch.device("cuda", 0)
    grid = torch.cuda.get_device_properties(dev).multi_processor_count
    g = torch.Generator(device=dev).manual_seed(seed)
    rnd = lambda *s: torch.randn(*s, device=dev, generator=g)      # noqa: E731
    nq, rot, maxlen = nkv * qpk, 64, max(lengths) + 1
    nb = -(-maxlen // 64)
    pr = Program(dev, M, grid)
    pr.embed(pr.zeros(4, 256, dtype=torch.bfloat16), pr.zeros(M, 256), pr.zeros(M, 16), None, 256, 4, keys_valid=False)
    width = nq * HD + 2 * nkv * HD
    y, y2 = rnd(M, width), pr.zeros(M, nq * HD)
    qn, kn = pr.hold(0.1 * rnd(HD)), pr.hold(0.1 * rnd(HD))
    if exact:
        y[:, : nq * HD + nkv * HD].sign_()
        qn.zero_(), kn.zero_()
    y = pr.hold(y)
    ang = torch.arange(maxlen, device=dev)[:, None] * (0.01 ** (torch.arange(rot // 2, device=dev) / (rot // 2)))[None]
    cos, sin = (pr.hold((ang * (not exact)).cos()), pr.hold((ang * (not exact)).sin()))
    kc, vc = (pr.hold(rnd(M * nb, nkv, 64, HD).to(torch.bfloat16)) for _ in range(2))
    bt = pr.hold(torch.randperm(M * nb, device=dev, generator=g).reshape(M, nb).to(torch.int32))
    rec = -(-qpk * (HD + 2) // 4) * 4
    part, cnt = pr.zeros(M * nkv * 64 * rec), pr.zeros(M * nkv, dtype=torch.int32)
    pr.add(D.desc(D.MKS_OP_ATTN, 0,
                  i=dict(NQ=nq, NKV=nkv, HD=HD, ROT=rot, A_Q_OFF=0, A_Q_HSTRIDE=HD, A_GATE_OFF=-1, A_K_OFF=nq * HD, A_V_OFF=nq * HD + nkv * HD,
                         A_Y_STRIDE=width, A_Y2_STRIDE=nq * HD, WINDOW=window, CHUNK_POS=256, MAX_PAGES=nb, ROPE_PAIRS=rot // 2, Q_BF16=1, MAX_CHUNKS=64),
                  f=dict(EPS=EPS, SCALE=HD ** -0.5),
                  p=dict(A_Y=y.data_ptr(), A_Y2=y2.data_ptr(), Q_NORM=qn.data_ptr(), K_NORM=kn.data_ptr(), K_CACHE=kc.data_ptr(), V_CACHE=vc.data_ptr(),
                         BLOCK_TABLE=bt.data_ptr(), ROPE_COS=cos.data_ptr(), ROPE_SIN=sin.data_ptr(), A_PART=part.data_ptr(), A_CNT=cnt.data_ptr())))
    rt = Runtime(pr, spin_limit_ms=1000)
    rt.pos[:M] = torch.tensor(lengths, dtype=torch.int32)
    want = torch.zeros(M, nq * HD, device=dev, dtype=torch.float64)
    for m, n in enumerate(lengths):
        p = torch.arange(n, device=dev)
        k, v = (c[bt[m].long()[p // 64], :, p % 64].transpose(0, 1).double() for c in (kc, vc))          # [nkv, n, HD]
        q = _head(y[m, : nq * HD].view(nkv, qpk, HD), qn, cos[n], sin[n]).double()
        nk = _head(y[m, nq * HD: nq * HD + nkv * HD].view(nkv, 1, HD), kn, cos[n], sin[n]).double()
        nv = _bf(y[m, nq * HD + nkv * HD:].view(nkv, 1, HD)).double()
        lo = max(0, n + 1 - window) if window else 0
        k, v = torch.cat([k, nk], 1)[:, lo:], torch.cat([v, nv], 1)[:, lo:]
        want[m] = (torch.softmax(q @ k.transpose(1, 2) * HD ** -0.5, -1) @ v).reshape(-1)
    for _ in range(3):                                             # (the same position again: the appended row is the same)
        rt.pos[:M] = torch.tensor(lengths, dtype=torch.int32)
        rt.launch(1)
        torch.cuda.synchronize()
        rt.check()
        err = float((y2.double() - want).norm() / want.norm())
        # a norm and a rotation in fp32 may round a query or key dim to the neighbouring bf16: 2^-9 of one of HD terms
        assert err < 1e-3, err
    return err


@pytest.mark.parametrize("M,nkv,qpk,HD,lengths,window", [
    (8, 8, 6, 256, [1100, 1600, 513, 255, 256, 1299, 1024, 1537], 0),       # up to four sub-chunks per task
    (8, 8, 8, 512, [1100, 1600, 513, 255, 256, 1299, 1024, 1537], 0),
    (8, 8, 3, 256, [1900, 1800, 700, 1300, 16, 2000, 15, 1], 1333),         # three sub-chunks inside a window
    (1, 4, 6, 256, [900], 0),
    (2, 1, 1, 256, [17, 3000], 0),
])
def test_attention_stage_matches_fp64(M, nkv, qpk, HD, lengths, window):
    _run(M, nkv, qpk, HD, lengths, window)


@pytest.mark.parametrize("M,nkv,qpk,HD,n,bound", [(8, 4, 6, 256, 1000, 1.6e-7), (8, 8, 6, 256, 1600, 3e-7), (8, 8, 8, 512, 1600, 6e-7)])
def test_attention_sums_round_towards_zero_in_short_chains(M, nkv, qpk, HD, n, bound):
    """250, 800 and 800 positions per task: 1.2e-7, 2.1e-7 and 4.2e-7 measured; chains twice as long gave 1.9e-7, 4.6e-7 and
    9.0e-7."""
    assert _run(M, nkv, qpk, HD, [n] * M, seed=4, exact=True) < bound
