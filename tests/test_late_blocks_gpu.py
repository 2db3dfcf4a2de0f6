"""Blocks of one launch that find the status word set while others found it clear: every tile of a result is either computed or NaN, and
so is every row's LSE; none is left as it was."""
import ctypes
import time

import pytest
import torch

pytestmark = pytest.mark.gpu

UNTOUCHED = 12345.0


@pytest.fixture()
def busy():
    """Keeps some SMs for six milliseconds: fp32 blocks, whose shared memory leaves no room for one of the 16-bit kernels."""
    from flash_b200 import _lib, ops
    lib = _lib.load()
    q, k = torch.randn(1, 40, 32, 128, device="cuda"), torch.randn(1, 40, 65536, 128, device="cuda")
    o, lse, status = torch.empty_like(q), torch.empty(1, 40, 128, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
    prob = ops._problem(1, 40, 40, 32, 65536, 128, q.dtype, False, 0, 1, 128 ** -0.5)

    def launch(stream):
        assert lib.fa_fwd(prob, ops._tensor(q), ops._tensor(k), ops._tensor(k), ops._tensor(o), lse.data_ptr(), None, status.data_ptr(),
                          ctypes.c_void_p(stream.cuda_stream)) == 0
    return launch


def late_blocks(busy, launch, outputs, want, status):
    """`launch` starts while `busy` holds some SMs; its last blocks begin when its first ones leave, after the status word has changed."""
    s1, s2 = torch.cuda.Stream(), torch.cuda.Stream()
    gave_up = torch.full((1,), 107, dtype=torch.int32).pin_memory()
    for _ in range(3):
        for x in outputs:
            x.fill_(UNTOUCHED)
        torch.cuda.synchronize()
        busy(s1)
        time.sleep(5e-5)
        launch()
        time.sleep(2e-4)
        with torch.cuda.stream(s2):
            status.copy_(gave_up, non_blocking=True)  # by a copy engine: a kernel would queue behind the waiting blocks
        torch.cuda.synchronize()
        for x, w in zip(outputs, want):
            lost = torch.isnan(x)
            assert torch.equal(x[~lost], w[~lost])
        status.zero_()
    for x in outputs:
        x.fill_(UNTOUCHED)
    launch()  # the counters are clear again
    assert all(torch.equal(x, w) for x, w in zip(outputs, want)) and int(status.item()) == 0


# one query block of one head a tile; the four query heads of one kv head a tile; with ids. Each block works for half a millisecond.
@pytest.mark.parametrize("form,counters", [("blocks", False), ("blocks", True), ("packed", False), ("packed", True), ("ids", True)])
def test_forward(busy, form, counters):
    from flash_b200 import _lib, ops
    lib = _lib.load()
    B, H, Hk, M, N, D = {"blocks": (1, 16, 1, 1200, 65536, 128), "packed": (40, 32, 8, 1, 32768, 128), "ids": (2, 10, 1, 1200, 32768, 64)}[form]
    g = torch.Generator(device="cuda").manual_seed(1)
    q, k, v = (torch.randn(B, h, n, D, generator=g, device="cuda").bfloat16() for h, n in ((H, M), (Hk, N), (Hk, N)))
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    prob = ops._problem(B, H, Hk, M, N, D, q.dtype, False, int(form == "ids"), 1, D ** -0.5)
    eq, ek = (torch.full((B, H, n), -1, device="cuda") for n in (M, N))
    plan = ops.build_plan(prob, *((eq, ek) if form == "ids" else (None, None)), status) if counters else None
    o, lse = torch.empty_like(q), torch.empty(B, H, lib.fa_padded_rows(M), device="cuda")

    def launch():
        assert lib.fa_fwd(prob, ops._tensor(q), ops._tensor(k), ops._tensor(v), ops._tensor(o), lse.data_ptr(),
                          plan.data_ptr() if counters else None, status.data_ptr(), ops._stream()) == 0

    launch()
    late_blocks(busy, launch, (o, lse[..., :M]), (o.clone(), lse[..., :M].clone()), status)


@pytest.mark.parametrize("counters", [False, True])
def test_dkdv(busy, counters):
    from flash_b200 import _lib, ops
    lib = _lib.load()
    B, H, Hk, M, N, D = 1, 16, 16, 32768, 1200, 128
    g = torch.Generator(device="cuda").manual_seed(1)
    q, k, v, do = (torch.randn(B, h, n, D, generator=g, device="cuda").bfloat16() for h, n in ((H, M), (Hk, N), (Hk, N), (H, M)))
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    prob = ops._problem(B, H, Hk, M, N, D, q.dtype, False, 0, 1, D ** -0.5)
    plan = ops.build_plan(prob, None, None, status) if counters else None
    o, dk, dv = torch.empty_like(q), torch.empty_like(k), torch.empty_like(v)
    lse, delta = (torch.empty(B, H, lib.fa_padded_rows(M), device="cuda") for _ in range(2))
    tq, tk, tv, to, tdo = [ops._tensor(t) for t in (q, k, v, o, do)]
    assert lib.fa_fwd(prob, tq, tk, tv, to, lse.data_ptr(), None, status.data_ptr(), ops._stream()) == 0
    assert lib.fa_bwd_delta(prob, to, tdo, delta.data_ptr(), ops._stream()) == 0

    def launch():
        assert lib.fa_bwd_dkdv(prob, tq, tk, tv, tdo, lse.data_ptr(), delta.data_ptr(), ops._tensor(dk), ops._tensor(dv),
                               plan.data_ptr() if counters else None, status.data_ptr(), ops._stream()) == 0

    launch()
    late_blocks(busy, launch, (dk, dv), (dk.clone(), dv.clone()), status)
