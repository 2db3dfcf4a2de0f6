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
