"""Regular calls get a native autograd node: the same bits, gradients, launches and refusals as with the node in Python."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def inputs(dtype, mode, B=2, H=4, Hk=2, L=300, D=64):
    g = torch.Generator(device="cuda").manual_seed(3)
    q, k, v, do = (torch.randn(B, h, L, D, generator=g, device="cuda").to(dtype) for h in (H, Hk, Hk, H))
    ids = (-1 - torch.arange(L, device="cuda") // 70).expand(B, H, L) if mode else None
    return q, k, v, do, ids


@pytest.mark.parametrize("causal", [True, False])
@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
def test_same_as_the_python_node(dtype, mode, causal, monkeypatch):
    import flash_b200 as fb
    from flash_b200 import ops
    monkeypatch.setattr(ops, "GROUP_QUERIES", False)  # (grouped calls have nodes of their own around this one)
    q, k, v, do, ids = inputs(dtype, mode)
    fb.attention(q, k, v, True)  # (the first call on a device makes its status word on the general path)

    def step(call, which=(True, True, True), do=do):
        x = [t.detach().requires_grad_(w) for t, w in zip((q, k, v), which)]
        before = ops.LAUNCHES
        o = call(*x, causal, None, ids, ids, mode)
        g = torch.autograd.grad(o, [t for t, w in zip(x, which) if w], do)
        return o, g, ops.LAUNCHES - before

    for which in ((True, True, True), (False, True, False), (True, False, False)):
        (o, g, n), (o2, g2, n2) = step(fb.attention, which), step(fb.FlashAttention.apply, which)
        assert type(o.grad_fn).__name__ != type(o2.grad_fn).__name__ and n == n2
        assert torch.equal(o, o2) and all(torch.equal(a, b) for a, b in zip(g, g2))
    # gradients that the kernels do not take as they are: expanded, of rows that are not 16-byte aligned, of another type, negated
    wide = torch.cat([do, do[..., :4]], 3)[..., :64]
    one = torch.ones((), dtype=dtype, device="cuda").expand_as(do)
    for d in (one, wide, do.to(torch.float64), torch._neg_view(do)):
        assert all(torch.equal(a, b) for a, b in zip(step(fb.attention, do=d)[1], step(fb.FlashAttention.apply, do=d)[1]))


def test_graph_forms():
    import flash_b200 as fb
    q, k, v, do, ids = inputs(torch.bfloat16, 1)
    fb.attention(q, k, v, True)
    x = [t.requires_grad_() for t in (q, k, v)]
    o = fb.attention(*x, True, None, ids, ids, 1)
    first = torch.autograd.grad(o, x, do, retain_graph=True)
    assert all(torch.equal(a, b) for a, b in zip(first, torch.autograd.grad(o, x, do)))
    with pytest.raises(RuntimeError, match="second time"):
        torch.autograd.grad(o, x, do)
    o = fb.attention(*x, True, None, ids, ids, 1)
    second = torch.autograd.grad(o, x, do, create_graph=True)
    assert not any(t.requires_grad for t in second)  # as from the node in Python
    o = fb.attention(*x, True, None, ids, ids, 1)
    with torch.no_grad():
        k.mul_(2)
    with pytest.raises(RuntimeError, match="modified by an inplace operation"):
        torch.autograd.grad(o, x, do)
    # a saved-tensor hook sees what the node in Python saves
    names = []
    with torch.autograd.graph.saved_tensors_hooks(lambda t: names.append(tuple(t.shape)) or t, lambda t: t):
        o = fb.attention(*x, True, None, ids, ids, 1)
    assert len(names) == 7 and o.grad_fn.name() == "FlashAttentionBackward"
    with torch.no_grad():
        assert fb.attention(*x, True, None, ids, ids, 1).grad_fn is None


def test_on_a_side_stream_and_in_another_thread():
    import threading
    import flash_b200 as fb
    q, k, v, do, ids = inputs(torch.bfloat16, 1, L=1000)
    fb.attention(q, k, v, True)

    def step():
        x = [t.detach().requires_grad_() for t in (q, k, v)]
        o = fb.attention(*x, True, None, ids, ids, 1)
        return o.detach(), *torch.autograd.grad(o, x, do)

    want, got = step(), []
    torch.cuda.synchronize()

    def work():
        s = torch.cuda.Stream()
        with torch.cuda.stream(s):
            for _ in range(5):
                got.append(step())
        s.synchronize()

    threads = [threading.Thread(target=work) for _ in range(3)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert len(got) == 15 and all(torch.equal(a, b) for r in got for a, b in zip(r, want))
