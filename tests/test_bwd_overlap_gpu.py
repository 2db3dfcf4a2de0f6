"""fa_bwd, whose dQ kernel may overlap the dK/dV kernel, gives the bits of the three separate calls: with fewer items
than SMs, with a tail of items, with more than one round; eagerly, back to back, and replayed from a graph."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,H,Hk,L,D,mode", [(1, 2, 2, 100, 64, 0), (2, 8, 2, 1100, 128, 0), (4, 12, 12, 600, 64, 1), (1, 4, 2, 300, 64, 1)])
def test_overlapped_backward(B, H, Hk, L, D, mode, monkeypatch):
    import flash_b200 as fb
    from flash_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(L)
    q, k, v = [torch.randn(B, h, L, D, generator=g, device="cuda").bfloat16().requires_grad_() for h in (H, Hk, Hk)]
    do = torch.randn(B, H, L, D, generator=g, device="cuda").bfloat16()
    ids = (-1 - torch.arange(L, device="cuda") // 70).expand(B, H, L) if mode else None

    def step():
        return torch.autograd.grad(fb.attention(q, k, v, True, None, ids, ids, mode), (q, k, v), do)

    monkeypatch.setattr(ops, "PROFILE", [])  # timed kernel by kernel: the separate calls
    want = [t.clone() for t in step()]
    monkeypatch.setattr(ops, "PROFILE", None)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        several = [[t.sum(dtype=torch.float64) for t in step()] + list(step()) for _ in range(5)]
    torch.cuda.current_stream().wait_stream(side)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        replayed = step()
    for _ in range(3):
        graph.replay()
    torch.cuda.synchronize()
    fb.check_status()
    for a, *got in zip(want, replayed, *[s[3:] for s in several]):
        assert all(torch.equal(a, x) for x in got)
    for s in several:  # a consumer right behind the backward sees complete gradients
        assert all(torch.equal(a.sum(dtype=torch.float64), x) for a, x in zip(want, s[:3]))


@pytest.mark.parametrize("counters", [False, True])
def test_dq_of_blocks_that_start_after_a_time_out(counters):
    """Blocks of one dQ launch that find the status word set while others found it clear: every tile is either computed
    or NaN, none is left as it was. Another launch keeps some SMs busy, so that some blocks start when the first
    ones leave; the word is set, as by a kernel that gave up, while the first ones work."""
    import ctypes
    import time
    import flash_b200 as fb
    from flash_b200 import _lib, ops
    lib = _lib.load()
    B, H, Hk, M, N, D = 1, 16, 1, 1200, 65536, 128  # 160 items of 512 tiles each, about half a millisecond
    g = torch.Generator(device="cuda").manual_seed(1)
    q, k, v, do = [torch.randn(B, h, n, D, generator=g, device="cuda").bfloat16() for h, n in ((H, M), (Hk, N), (Hk, N), (H, M))]
    qr, kr, vr = [t.clone().requires_grad_() for t in (q, k, v)]
    o = fb.attention(qr, kr, vr)
    want = torch.autograd.grad(o, qr, do)[0]
    lse, delta = torch.empty(B, H, 1280, device="cuda"), torch.empty(B, H, 1280, device="cuda")
    prob = ops._problem(B, H, Hk, M, N, D, q.dtype, False, 0, 1, D ** -0.5)
    status, other = [torch.zeros(1, dtype=torch.int32, device="cuda") for _ in range(2)]
    plan = ops.build_plan(prob, None, None, status) if counters else None
    tq, tk, tv, tdo, to = [ops._tensor(t) for t in (q, k, v, do, o.detach())]
    stream = ops._stream()
    assert lib.fa_fwd(prob, tq, tk, tv, ops._tensor(torch.empty_like(q)), lse.data_ptr(), None, other.data_ptr(), stream) == 0
    assert lib.fa_bwd_delta(prob, to, tdo, delta.data_ptr(), stream) == 0
    # 40 blocks of the fp32 kernel, whose shared memory leaves no room for a block of dQ, with 1024 tiles each: six milliseconds
    busy_q, busy_k = torch.randn(1, 40, 32, D, device="cuda"), torch.randn(1, 40, 65536, D, device="cuda")
    busy = ops._problem(1, 40, 40, 32, 65536, D, busy_q.dtype, False, 0, 1, D ** -0.5)
    busy_o, busy_lse = torch.empty_like(busy_q), torch.empty(1, 40, 128, device="cuda")
    gave_up = torch.full((1,), 107, dtype=torch.int32).pin_memory()
    s1, s2 = torch.cuda.Stream(), torch.cuda.Stream()

    def dq_launch(dq):
        assert lib.fa_bwd_dq(prob, tq, tk, tv, tdo, lse.data_ptr(), delta.data_ptr(), ops._tensor(dq),
                             plan.data_ptr() if counters else None, status.data_ptr(), stream) == 0

    for _ in range(3):
        dq = torch.full_like(q, 12345.0)
        torch.cuda.synchronize()
        with torch.cuda.stream(s1):
            assert lib.fa_fwd(busy, ops._tensor(busy_q), ops._tensor(busy_k), ops._tensor(busy_k), ops._tensor(busy_o),
                              busy_lse.data_ptr(), None, other.data_ptr(), ctypes.c_void_p(s1.cuda_stream)) == 0
        time.sleep(5e-5)
        dq_launch(dq)
        with torch.cuda.stream(s2):
            status.copy_(gave_up, non_blocking=True)  # by a copy engine: a kernel would queue behind the waiting blocks
        torch.cuda.synchronize()
        lost = torch.isnan(dq)
        assert torch.equal(dq[~lost], want[~lost])
        status.zero_()
    dq = torch.full_like(q, 12345.0)
    dq_launch(dq)  # the counters are clear again
    assert torch.equal(dq, want) and int(status.item()) == 0
    fb.check_status()
