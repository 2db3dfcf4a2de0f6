"""fa_group_rows with one of its outputs in the place of the ids: as with outputs of their own."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [64, 65, 1000, 4096, 4097])
@pytest.mark.parametrize("B,He", [(1, 1), (3, 2)])
@pytest.mark.parametrize("which", [0, 1, 2])  # order, inverse, grouped ids
def test_in_place(which, B, He, M):
    from flash_b200 import _lib, ops
    lib = _lib.load()
    g = torch.Generator(device="cuda").manual_seed(M)
    H = max(He, 2)
    prob = ops._problem(B, H, H, M, M, 64, torch.bfloat16, False, 1, He, 1.0)
    for ids in (-torch.randint(1, 9, (B, He, M), generator=g, device="cuda"), -torch.randint(1, 2 ** 31, (B, He, M), generator=g, device="cuda")):
        want = ids.sort(dim=2, stable=True)
        results = want.indices, want.indices.argsort(2), want.values
        for _ in range(3):
            out = torch.full((3, B, He, M), -1, dtype=torch.int32, device="cuda")
            status = torch.zeros(1, dtype=torch.int32, device="cuda")
            out[which] = ids
            assert lib.fa_group_rows(ctypes.byref(prob), ops._ids(out[which]), out[0].data_ptr(), out[1].data_ptr(), out[2].data_ptr(),
                                     status.data_ptr(), ops._stream()) == 0
            assert all(torch.equal(a.long(), b) for a, b in zip(out, results)) and int(status) == 0
