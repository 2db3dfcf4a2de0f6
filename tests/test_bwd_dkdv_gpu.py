"""dK, dV and dQ where the dK/dV kernel's rings and buffers turn over: items of one tile up to more than the stages of Q and dO hold,
several query heads a key block, ragged ends and blocks without a tile, for each head width and type, against 64-bit torch."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


# results are rounded once to the input type, P and dS on the way: 2^-8 relative in bf16, 2^-11 in fp16, of values up to about 4
@pytest.mark.parametrize("dtype,tol", [(torch.bfloat16, 2e-2), (torch.float16, 4e-3)])
@pytest.mark.parametrize("D", [32, 64, 128])
@pytest.mark.parametrize("B,H,Hk,M,N,causal,docs", [
    (1, 1, 1, 1, 1, False, 0),         # one entry
    (1, 2, 1, 129, 129, True, 0),      # items of two tiles and of one, two heads each
    (1, 3, 1, 385, 513, True, 0),      # three heads, a gap, four tiles a head
    (2, 2, 2, 700, 300, False, 0),     # more queries than keys, six tiles
    (1, 2, 2, 900, 900, True, 5),      # documents: tiles left out
    (1, 4, 2, 640, 1000, False, 300),  # ids no query has: key blocks without a tile
])
def test_gradients(B, H, Hk, M, N, causal, docs, D, dtype, tol):
    import flash_b200
    g = torch.Generator().manual_seed(M + D)
    q, k, v, do = (torch.randn(s, generator=g).to(dtype) for s in ((B, H, M, D), (B, Hk, N, D), (B, Hk, N, D), (B, H, M, D)))
    eq = ek = None
    if docs:
        ids = -1 - np.sort(np.random.default_rng(D).integers(0, docs, N))
        if docs > N // 4:
            ids[:N - M] = -docs - 2  # in no query
        ek = torch.from_numpy(ids)[None].repeat(B, 1)
        eq = ek[:, N - M:]
    t = [x.cuda().requires_grad_() for x in (q, k, v)]
    ids = [None if e is None else e.cuda()[:, None].expand(B, H, e.shape[1]) for e in (eq, ek)]
    mode = flash_b200.SCORE_FUNC_MODE1_DOC if docs else flash_b200.SCORE_FUNC_MODE0_NOPE
    o = flash_b200.attention(*t, causal, None, ids[0], ids[1], mode)
    got = torch.autograd.grad(o, t, do.cuda())
    x = [y.double().requires_grad_() for y in (q, k, v)]
    kr, vr = (y.repeat_interleave(H // Hk, 1) for y in x[1:])
    s = x[0] @ kr.transpose(2, 3) / D ** 0.5
    keep = torch.ones(B, 1, M, N, dtype=torch.bool)
    if causal:
        keep &= torch.arange(N)[None] <= torch.arange(M)[:, None] + max(0, N - M)
    if docs:
        keep = keep & ((eq[:, None, :, None] >= 0) | (eq[:, None, :, None] == ek[:, None, None, :]))
    p = torch.softmax(s.masked_fill(~keep, -1e30), -1) * keep
    want = torch.autograd.grad(p @ vr, x, do.double())
    for name, a, b in zip(("dQ", "dK", "dV"), got, want):
        a = a.double().cpu()
        err = (a - b).abs()
        assert (err <= tol + tol / 2 * b.abs()).all(), (name, float(err.max()))
