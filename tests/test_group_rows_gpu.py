"""Grouping of the queries: both ways of sorting against a stable sort, and the row permutation, at the edges of their blocks."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.int32, torch.int64])
@pytest.mark.parametrize("M", [1, 15, 16, 17, 63, 64, 65, 1000, 1024, 4095, 4096, 4097, 16384])
@pytest.mark.parametrize("B,He", [(1, 1), (3, 2), (1, 13)])  # thirteen rows of 4096 are more than counting is taken for
def test_stable_sort(B, He, M, dtype):
    import flash_b200 as fb
    from flash_b200 import _lib, ops
    g = torch.Generator(device="cuda").manual_seed(M + He)
    for ids in (-torch.randint(1, 9, (B, He, M), generator=g, device="cuda"), torch.randint(-5, 3, (B, He, M), generator=g, device="cuda"),
                -torch.randint(1, 2 ** 31, (B, He, M), generator=g, device="cuda"), torch.full((B, He, M), 7, device="cuda")):
        ids = ids.to(dtype)
        wide = torch.zeros(B, He, M, 2, dtype=dtype, device="cuda")
        wide[..., 1] = ids
        out = torch.full((3, B, He, M), -1, dtype=torch.int32, device="cuda")
        status = torch.zeros(1, dtype=torch.int32, device="cuda")
        H = max(He, 2)
        prob = ops._problem(B, H if He == 1 else He, H if He == 1 else He, M, M, 64, torch.bfloat16, False, 1, He, 1.0)
        _lib.check(_lib.load().fa_group_rows(ctypes.byref(prob), ops._ids(wide[..., 1]), out[0].data_ptr(), out[1].data_ptr(), out[2].data_ptr(),
                                             status.data_ptr(), ops._stream()), "fa_group_rows")
        code = torch.where(ids >= 0, torch.full_like(ids, 2 ** 31 - 1), ids)
        want = code.sort(dim=2, stable=True)
        assert torch.equal(out[0].long(), want.indices) and torch.equal(out[2].to(dtype), want.values)
        assert torch.equal(out[1].long(), want.indices.argsort(2)) and int(status) == 0


@pytest.mark.parametrize("D", [16, 32, 64, 128])
@pytest.mark.parametrize("M", [1, 31, 33, 127, 129, 515])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_permute(dtype, M, D):
    from flash_b200 import _lib, ops
    B, H = 2, 3
    g = torch.Generator(device="cuda").manual_seed(M)
    x = torch.randn(B, M, H, D, generator=g, device="cuda").to(dtype).transpose(1, 2)
    for He in (1, H):
        index = torch.stack([torch.randperm(M, generator=g, device="cuda") for _ in range(B * He)]).view(B, He, M)
        out = torch.full((B, H, M + 1, D), 7.0, device="cuda").to(dtype)
        prob = ops._problem(B, H, H, M, M, D, dtype, False, 1, He, 1.0)
        _lib.check(_lib.load().fa_permute_rows(ctypes.byref(prob), ops._tensor(x), ops._tensor(out[:, :, :M]), index.int().data_ptr(), ops._stream()),
                   "fa_permute_rows")
        assert torch.equal(out[:, :, :M], x.gather(2, index.expand(B, H, M)[..., None].expand(B, H, M, D)))
        assert bool((out[:, :, M:] == 7.0).all())
