"""The native host call takes regular calls; every other form takes the general path to the same kernels and the same bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def layouts(x):
    B, H, L, D = x.shape
    yield "contiguous", x.clone()
    yield "transposed", x.transpose(1, 2).contiguous().transpose(1, 2)
    wide = torch.zeros(B, H, L, 2 * D, dtype=x.dtype, device=x.device)
    wide[..., ::2] = x
    yield "last stride 2", wide[..., ::2]
    odd = torch.zeros(x.numel() + 1, dtype=x.dtype, device=x.device)
    odd[1:] = x.reshape(-1)
    yield "odd rows", torch.cat([x, x[..., :4]], 3)[..., :D]
    if x.dtype == torch.float32:  # 16-bit tensors of this kind are refused by the library, as before
        yield "odd base", odd[1:].view(B, H, L, D)


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_layouts_give_the_same_bits(dtype, mode):
    import flash_b200 as fb
    B, H, Hk, L, D = 2, 4, 2, 200, 64
    g = torch.Generator(device="cuda").manual_seed(1)
    q, k, v, do = (torch.randn(B, h, L, D, generator=g, device="cuda").to(dtype) for h in (H, Hk, Hk, H))
    ids = (-1 - torch.arange(L, device="cuda") // 70).expand(B, H, L) if mode else None

    def step(q, k, v, do):
        q, k, v = (x.detach().requires_grad_() for x in (q, k, v))
        o = fb.attention(q, k, v, True, None, ids, ids, mode)
        return (o.detach(), *torch.autograd.grad(o, (q, k, v), do))

    want = step(q, k, v, do)
    for (name, a), (_, b), (_, c), (_, d) in zip(*(layouts(x) for x in (q, k, v, do))):
        for args in ((a, b, c, do), (q, k, v, d)):
            for x, y in zip(step(*args), want):
                assert torch.equal(x, y), name
    # an expanded gradient
    one = torch.ones((), dtype=dtype, device="cuda").expand(B, H, L, D)
    assert all(torch.equal(x, y) for x, y in zip(step(q, k, v, one), step(q, k, v, one.contiguous())))


def test_autograd_forms():
    import flash_b200 as fb
    q, k, v = (torch.randn(1, 2, 64, 64, device="cuda", dtype=torch.bfloat16, requires_grad=True) for _ in range(3))
    packed = []
    with torch.autograd.graph.saved_tensors_hooks(lambda t: packed.append(t.shape) or t, lambda t: t):
        o = fb.attention(q, k, v, True)
    assert len(packed) == 5 and o.grad_fn.name() == "FlashAttentionBackward"
    o.sum().backward()
    with pytest.raises(RuntimeError):  # buffers freed
        o.sum().backward()
    with torch.no_grad():
        assert not fb.attention(q, k, v, True).requires_grad
    with pytest.raises(RuntimeError):  # no vmap rule
        torch.vmap(lambda x: fb.attention(x, x, x, True))(torch.randn(2, 1, 2, 64, 64, device="cuda", dtype=torch.bfloat16))
    with pytest.raises(NotImplementedError):
        fb.attention(q, k, v, True, 0.0)
    with pytest.raises(AssertionError):
        fb.attention(q, k[:, :, :32], v[:, :, :32], True)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_a_negative_number_of_runs_is_refused(dtype):
    import flash_b200 as fb
    q, k, v = (torch.randn(1, 4, 300, 64, device="cuda").to(dtype) for _ in range(3))
    o = fb.attention(q, k, v, True)
    for x in (q, torch.cat([q, q[..., :4]], 3)[..., :64]):  # the native call, the general code
        for runs in (-1, -3):
            with pytest.raises(RuntimeError, match="bad argument"):
                fb.attention_in_runs(x, k, v, runs, True)
        assert torch.equal(fb.attention_in_runs(x, k, v, 0, True), o)  # 0: as `attention` chooses


@pytest.mark.parametrize("kind", [float, bool, torch.tensor])
def test_the_mode_may_be_any_number(kind):
    import flash_b200 as fb
    q, k, v, do = (torch.randn(1, 4, 300, 64, device="cuda").bfloat16() for _ in range(4))
    ids = (-1 - torch.arange(300, device="cuda") // 70).expand(1, 4, 300)

    def step(e, mode):
        x = [t.clone().requires_grad_() for t in (q, k, v)]
        o = fb.attention(*x, True, None, e, e, mode)
        return (o.detach(), *torch.autograd.grad(o, x, do))

    for e, mode in ((None, 0), (ids, 0), (ids, 1)):
        assert all(torch.equal(a, b) for a, b in zip(step(e, kind(mode)), step(e, mode)))


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_longer_keys_and_values_are_read_as_far_as_the_call_goes(dtype):
    import flash_b200 as fb
    B, H, Hk, M, N, D = 2, 4, 2, 200, 230, 64
    q, k, v, do = (torch.randn(b, h, n, D, device="cuda").to(dtype) for b, h, n in ((B, H, M), (B + 1, Hk, N), (B + 2, Hk, N + 10), (B, H, M)))

    def step(k, v):
        x = q.clone().requires_grad_()
        o = fb.attention(x, k, v, True)
        return o.detach(), *torch.autograd.grad(o, x, do)

    assert all(torch.equal(a, b) for a, b in zip(step(k, v), step(k[:B], v[:B, :, :N])))
    for x in (k, v):  # a gradient of theirs would have the wrong shape
        with pytest.raises(RuntimeError, match="invalid gradient"):
            x.requires_grad_()
            fb.attention(q, k, v, True).backward(do)
        x.requires_grad_(False)
    for a, b in ((k[:1], v), (k, v[:1]), (k, v[:, :, :N - 1])):
        with pytest.raises(RuntimeError):
            fb.attention(q, a, b, True)


class _Tagged(torch.Tensor):
    pass


@pytest.mark.parametrize("mode", [0, 1])
def test_a_tensor_subclass_gives_one(mode):
    import flash_b200 as fb
    q, k, v = (torch.randn(2, 4, 200, 64, device="cuda").bfloat16() for _ in range(3))
    ids = (-1 - torch.arange(200, device="cuda") // 70).expand(2, 4, 200) if mode else None
    want = fb.attention(q, k, v, True, None, ids, ids, mode)
    for x in (q, q.transpose(1, 2).contiguous().transpose(1, 2), torch.cat([q, q[..., :4]], 3)[..., :64]):
        o = fb.attention(x.as_subclass(_Tagged), k, v, True, None, ids, ids, mode)
        assert type(o) is _Tagged and torch.equal(o.as_subclass(torch.Tensor), want)
    assert type(fb.attention(torch.nn.Parameter(q), k, v, True, None, ids, ids, mode)) is torch.Tensor


def test_tracing_is_refused():
    """A trace would hold the allocation of the result and not the kernel that fills it."""
    import flash_b200 as fb
    x = torch.randn(1, 4, 200, 64, device="cuda").bfloat16()
    fb.attention(x, x, x, True)
    with pytest.raises(AssertionError):
        torch.jit.trace(lambda q: fb.attention(q, q, q, True), x, check_trace=False)


def test_negated_views():
    import flash_b200 as fb
    q, k, v, do = (torch.randn(1, 4, 200, 64, device="cuda").bfloat16() for _ in range(4))

    def step(q, do):
        q = q.detach().requires_grad_()
        o = fb.attention(q, k, v, True)
        return o.detach(), *torch.autograd.grad(o, q, do)

    want = step(-q, -do)
    assert all(torch.equal(a, b) for a, b in zip(step(torch._neg_view(q), torch._neg_view(do)), want))


class _Recorder:
    """The native host calls, with what each was asked and whether it took the call: (direction, prepared, taken)."""

    def __init__(self, host):
        self.host, self.calls = host, []

    def forward(self, *args):
        done = self.host.forward(*args)
        self.calls.append(("forward", args[3], done is not None))
        return done

    def backward(self, *args):
        done = self.host.backward(*args)
        self.calls.append(("backward", args[6], done is not None))
        return done


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_which_calls_take_the_native_route(monkeypatch, dtype):
    """Regular calls are taken as they are, in both directions; the others are declined once and taken when they have
    been prepared."""
    import flash_b200 as fb
    from flash_b200 import ops
    B, H, L, D = 2, 4, 200, 64
    q, k, v, do = (torch.randn(B, H, L, D, device="cuda").to(dtype) for _ in range(4))
    fb.attention(q, k, v, True)  # (the first call on a device makes its status word on the general path)
    recorder = _Recorder(ops._host())
    monkeypatch.setattr(ops, "_HOST", recorder)

    def route(q, k, v, do):
        recorder.calls.clear()
        x = [t.detach().requires_grad_() for t in (q, k, v)]
        fb.attention(*x, True).backward(do)
        return list(recorder.calls)

    forward, backward = [("forward", False, True)], [("backward", False, True)]
    general_forward = [("forward", False, False), ("forward", True, True)]
    general_backward = [("backward", False, False), ("backward", True, True)]
    regular = ("contiguous", "transposed")
    for (name, a), (_, b), (_, c), (_, d) in zip(*(layouts(x) for x in (q, k, v, do))):
        assert route(a, b, c, do) == (forward if name in regular else general_forward) + backward, name
        assert route(q, k, v, d) == forward + (backward if name in regular else general_backward), name
    assert route(q, k, v, torch.ones((), dtype=dtype, device="cuda").expand(B, H, L, D)) == forward + general_backward
    assert route(q, k, v, do.to(torch.float64)) == forward + backward  # (autograd casts it first)
    with torch.no_grad():
        recorder.calls.clear()
        fb.attention(q, k, v, True)
        assert recorder.calls == forward
        ids = (-1 - torch.arange(L, device="cuda") // 70).expand(B, H, L)
        recorder.calls.clear()
        fb.attention(q, k, v, True, None, ids, ids, fb.SCORE_FUNC_MODE1_DOC)  # ids: a plan is built first
        assert recorder.calls == [("forward", True, True)]


def test_no_autograd_node_changes_nothing():
    """Calls that need no gradient go without a node: the same bits, messages and refusals as with one."""
    import flash_b200 as fb
    import torch.autograd.forward_ad as fwad
    q, k, v = (torch.randn(2, 4, 200, 64, device="cuda").bfloat16() for _ in range(3))
    want = fb.attention(q.clone().requires_grad_(), k, v, True)
    assert want.requires_grad
    with torch.no_grad():
        got = fb.attention(q.clone().requires_grad_(), k, v, True)
    with torch.inference_mode():
        frozen = fb.attention(q, k, v, True)
    for o in (got, frozen, fb.attention(q, k, v, True)):
        assert not o.requires_grad and o.grad_fn is None and torch.equal(o, want)
    assert frozen.is_inference()
    for bad, error in (((q, k[:, :, :32], v[:, :, :32]), AssertionError), ((q, k.half(), v), ValueError), ((q, k.cpu(), v), ValueError)):
        with pytest.raises(error):
            fb.attention(*bad, True)
    with pytest.raises(RuntimeError):
        torch.vmap(lambda x: fb.attention(x, x, x, True))(torch.randn(2, 1, 2, 64, 64, device="cuda").bfloat16())
    with torch.no_grad(), fwad.dual_level(), pytest.raises(Exception, match="jvp"):
        fb.attention(fwad.make_dual(q, q), k, v, True)
    with pytest.raises(Exception):
        torch.func.jvp(lambda x: fb.attention(x, k, v, True), (q,), (q,))


@pytest.mark.parametrize("dtype", [torch.int32, torch.int64, torch.int16])
def test_ids_of_any_form_give_the_same_bits(dtype):
    """Broadcast over the heads or not, strided or not, of a type that the library takes or one that is converted first."""
    import flash_b200 as fb
    B, H, L = 2, 4, 200
    q, k, v = (torch.randn(B, H, L, 64, device="cuda").bfloat16() for _ in range(3))
    ids = (-1 - torch.arange(L, device="cuda") // 70).to(dtype)
    want = fb.attention(q, k, v, True, None, ids.long().expand(B, H, L), ids.long().expand(B, H, L), 1)
    full = ids.expand(B, H, L).contiguous()
    for e in (ids.expand(B, H, L), full, full.transpose(0, 2).contiguous().transpose(0, 2), torch.stack([full, full], -1)[..., 0]):
        assert torch.equal(fb.attention(q, k, v, True, None, e, e, 1), want)
    for bad in (ids.expand(B, 1, L), ids[:-1].expand(B, H, L - 1), ids.expand(B, H, L).float()):
        with pytest.raises(AssertionError):
            fb.attention(q, k, v, True, None, ids.expand(B, H, L), bad, 1)
