"""Kernels that set themselves up while the one before them ends still find what it wrote and overwrite nothing that it reads: passes
whose inputs are written directly before them in the stream, and overwritten directly behind them, give the bits of lone ones."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("captured", [False, True])
@pytest.mark.parametrize("dtype,mode,causal,M,N", [
    (torch.bfloat16, 0, True, 300, 300),     # no plan
    (torch.float16, 0, True, 3, 2000),       # a split forward and its merge
    (torch.bfloat16, 0, False, 2500, 2500),  # more blocks than SMs: counters
    (torch.bfloat16, 1, True, 700, 700),     # one plan kernel
    (torch.float16, 1, True, 4500, 4500),    # three
    (torch.float16, 1, False, 300, 900),     # rows sorted and permuted
    (torch.float32, 1, True, 300, 300),
])
def test_inputs_change_around_every_pass(dtype, mode, causal, M, N, captured):
    import flash_b200 as fb
    B, H, D = 1, 8, 64
    g = torch.Generator(device="cuda").manual_seed(M)
    sets = [[torch.randn(B, H, n, D, generator=g, device="cuda").to(dtype) for n in (M, N, N, M)] for _ in range(3)]
    ids = [(-1 - (torch.arange(N, device="cuda") + 37 * i) // 150) for i in range(3)]
    bufs = [torch.zeros_like(t).requires_grad_(i < 3) for i, t in enumerate(sets[0])]
    ek = torch.empty_like(ids[0])
    eq_full, ek_full = ek[N - M:].expand(B, H, M), ek.expand(B, H, N)

    def one(i, out):
        with torch.no_grad():
            for b, t in zip(bufs, sets[i]):
                b.copy_(t)
            ek.copy_(ids[i])
        o = fb.attention(*bufs[:3], causal, None, eq_full if mode else None, ek_full if mode else None, mode)
        res = (o.detach(), *torch.autograd.grad(o, bufs[:3], bufs[3]))
        for a, r in zip(out, res):
            a.copy_(r)
        with torch.no_grad():  # what a late reader would find
            for b in bufs:
                b.fill_(float("nan"))
            ek.fill_(-(1 << 20))

    def outputs():
        return [[torch.empty_like(t) for t in (bufs[0], *bufs[:3])] for _ in range(3)]

    want = outputs()
    for i in range(3):
        one(i, want[i])
        torch.cuda.synchronize()
    got = outputs()
    if captured:
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            for i in range(3):
                one(i, got[i])
    for _ in range(5):
        if captured:
            graph.replay()
        else:
            for i in range(3):
                one(i, got[i])
    torch.cuda.synchronize()
    fb.check_status()
    for a, b in zip(got, want):
        assert all(torch.equal(x, y) and not x.isnan().any() for x, y in zip(a, b))
