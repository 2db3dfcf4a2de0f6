"""Row sums of O and dO: blocks of several rows a thread, at the edges of rows, blocks and the padding."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("layout", ["bhld", "blhd"])
@pytest.mark.parametrize("M", [1, 63, 64, 65, 127, 128, 129, 300])
@pytest.mark.parametrize("D", [16, 32, 64, 128])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_delta(dtype, D, M, layout):
    import flash_b200 as fb
    from flash_b200 import _lib, ops
    B, H, pad = 2, 3, (M + 127) // 128 * 128
    g = torch.Generator(device="cuda").manual_seed(M)
    o, do = (torch.randn((B, H, M, D) if layout == "bhld" else (B, M, H, D), generator=g, device="cuda").to(dtype) for _ in range(2))
    if layout == "blhd":
        o, do = o.transpose(1, 2), do.transpose(1, 2)
    guard = 64  # floats behind the buffer that nothing may touch
    buf = torch.full((B * H * pad + guard,), 7.0, device="cuda")
    prob = ops._problem(B, H, H, M, M, D, dtype, False, 0, 1, 1.0)
    _lib.check(_lib.load().fa_bwd_delta(ctypes.byref(prob), ops._tensor(o), ops._tensor(do), buf.data_ptr(), ops._stream()), "fa_bwd_delta")
    delta = buf[:B * H * pad].view(B, H, pad)
    prod = o.double() * do.double()
    # D products rounded and summed in fp32
    assert bool(((delta[..., :M].double() - prod.sum(3)).abs() <= D * 2.0 ** -24 * prod.abs().sum(3)).all())
    assert bool((delta[..., M:] == 0).all()) and bool((buf[B * H * pad:] == 7.0).all())
    fb.check_status()
