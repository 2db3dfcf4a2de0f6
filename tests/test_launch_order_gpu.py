"""Kernels that set themselves up while the one before them ends still find what it wrote and overwrite nothing that it reads. Passes
whose inputs torch writes directly before them in the stream, and overwrites directly behind them, give the bits of lone ones; torch's
kernels begin when all that is older has ended, so that this shows the order inside a pass. From one pass to the next the library's kernels
follow each other directly in the other tests here: through one's results, and through memory that both use."""
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


def _queued(run, captured):
    """`run()` with its launches back to back: from a graph, or queued up behind a kernel of a millisecond or two."""
    if captured:
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            run()
        graph.replay()
    else:
        torch.cuda._sleep(3_000_000)
        run()
    torch.cuda.synchronize()


@pytest.mark.parametrize("captured", [False, True])
@pytest.mark.parametrize("dtype,mode,causal,M,N,D", [
    (torch.bfloat16, 0, True, 300, 300, 64),
    (torch.bfloat16, 0, True, 300, 300, 128),
    (torch.float16, 0, True, 3, 2000, 128),      # a split forward and its merge
    (torch.bfloat16, 0, False, 2500, 2500, 128),
    (torch.bfloat16, 1, True, 700, 700, 128),    # a plan in front of each
    (torch.float16, 1, True, 4500, 4500, 64),
    (torch.float16, 1, False, 300, 900, 64),     # rows sorted and permuted
    (torch.float32, 1, True, 300, 300, 64),
])
def test_forwards_of_the_previous_result(dtype, mode, causal, M, N, D, captured):
    import flash_b200 as fb
    B, H, n = 1, 8, 6
    g = torch.Generator(device="cuda").manual_seed(N + D)
    x0, k, v = (torch.randn(B, H, L, D, generator=g, device="cuda").to(dtype) for L in (M, N, N))
    ids = -1 - torch.arange(N, device="cuda") // 150
    eq, ek = (ids[N - M:].expand(B, H, M), ids.expand(B, H, N)) if mode else (None, None)
    fb.attention(x0, k, v, causal, None, eq, ek, mode)

    def run(out, wait):
        x = x0
        for _ in range(n):
            x = fb.attention(x, *((x, x) if M == N else (k, v)), causal, None, eq, ek, mode)
            out.append(x)
            if wait:
                torch.cuda.synchronize()

    want, got = [], []
    run(want, True)
    _queued(lambda: run(got, False), captured)
    fb.check_status()
    for a, b in zip(got, want, strict=True):
        assert torch.equal(a, b) and not a.isnan().any()


@pytest.mark.parametrize("captured", [False, True])
@pytest.mark.parametrize("dtype,mode,L,D", [
    (torch.bfloat16, 0, 300, 64), (torch.bfloat16, 0, 300, 128),
    (torch.bfloat16, 1, 700, 64), (torch.bfloat16, 1, 700, 128),
    (torch.bfloat16, 1, 4500, 128),  # a plan by three kernels
    (torch.float32, 1, 300, 64),
])
def test_steps_that_share_all_scratch_memory(dtype, mode, L, D, captured):
    """Steps through the C ABI with one plan, o, LSE and delta for all of them, other ids each, and with the gradients of one among the
    inputs of the next."""
    import flash_b200 as fb
    from flash_b200 import _lib, ops
    import ctypes
    lib = _lib.load()
    B, H, n = 1, 8, 3
    g = torch.Generator(device="cuda").manual_seed(L + D)
    q, k, v, do = (torch.randn(B, H, L, D, generator=g, device="cuda").to(dtype) for _ in range(4))
    prob = ops._problem(B, H, H, L, L, D, dtype, True, mode, 1, D ** -0.5)
    ids = [-1 - (torch.arange(L, device="cuda") + 61 * i) // (90 + 40 * i) for i in range(n)]
    o, status = torch.empty_like(q), torch.zeros(1, dtype=torch.int32, device="cuda")
    lse, delta = (torch.empty(B, H, lib.fa_padded_rows(L), device="cuda") for _ in range(2))
    size = ctypes.c_size_t()
    _lib.check(lib.fa_plan_bytes(prob, size), "fa_plan_bytes")
    plan = torch.empty(size.value // 4, dtype=torch.int32, device="cuda")

    def run(out, wait):
        tens, ptr, s = ops._tensor, torch.Tensor.data_ptr, ops._stream()
        vi, doi = v, do
        for i in range(n):
            grads = out[i]
            e = ops._ids(ids[i].expand(B, H, L)) if mode else None
            _lib.check(lib.fa_plan_build(prob, e, e, ptr(plan), size.value, ptr(status), s), "fa_plan_build")
            t = [tens(x) for x in (q, k, vi, o)]
            _lib.check(lib.fa_fwd(prob, *t, ptr(lse), ptr(plan), ptr(status), s), "fa_fwd")
            _lib.check(lib.fa_bwd(prob, *t, tens(doi), ptr(lse), ptr(delta), *(tens(x) for x in grads), ptr(plan), ptr(status), s), "fa_bwd")
            vi, doi = grads[1], grads[0]
            if wait:
                torch.cuda.synchronize()

    want, got = ([[torch.empty_like(q) for _ in range(3)] for _ in range(n)] for _ in range(2))
    run(want, True)
    _queued(lambda: run(got, False), captured)
    assert int(status.item()) == 0
    for a, b in zip(got, want):
        assert all(torch.equal(x, y) and not x.isnan().any() and x.any() for x, y in zip(a, b))
