"""Calls in a second CUDA context of the same device, after the first has used every kernel: what a launch needs is set
up per context, not per device. In a process of its own, which it leaves with the second context current."""
import subprocess
import sys

import pytest

from conftest import PKG

pytestmark = pytest.mark.gpu

SCRIPT = """
import ctypes, sys
sys.path.insert(0, sys.argv[1])
import torch
import flash_b200 as fb
from flash_b200 import ops, _lib
lib = _lib.load()
B, H, L = 1, 2, 300
KINDS = [(torch.bfloat16, 64), (torch.float16, 128), (torch.float32, 32), (torch.float32, 128)]
ids = (-1 - torch.arange(L, device="cuda") // 100).expand(B, H, L)
for dt, D in KINDS:
    x = [torch.randn(B, H, L, D, device="cuda").to(dt).requires_grad_() for _ in range(3)]
    fb.attention(*x, False, None, ids, ids, 1).sum().backward()
fb.check_status()

def static_plan(p, q, k, v, o, lse, ids, status):
    return lib.fa_fwd_static_plan(p, q, k, v, o, lse, ids, ids, status, None)

x, st = [torch.randn(B, H, L, 64, device="cuda").bfloat16() for _ in range(4)], torch.zeros(1, dtype=torch.int32, device="cuda")
assert static_plan(ops._problem(B, H, H, L, L, 64, torch.bfloat16, False, 1, 1, 1.0), *[ops._tensor(t) for t in x],
                   torch.empty(B, H, 384, device="cuda").data_ptr(), ops._ids(ids), st.data_ptr()) == 0
torch.cuda.synchronize()
cu = ctypes.CDLL("libcuda.so.1")
assert cu.cuCtxCreate_v2(ctypes.byref(ctypes.c_void_p()), 0, 0) == 0

def alloc(data):
    p = ctypes.c_uint64()
    assert cu.cuMemAlloc_v2(ctypes.byref(p), ctypes.c_size_t(len(data))) == 0
    assert cu.cuMemcpyHtoD_v2(p, data, ctypes.c_size_t(len(data))) == 0
    return p.value

for dt, D in KINDS:
    size = 4 if dt == torch.float32 else 2
    t = [_lib.Tensor(alloc(bytes(B * H * L * D * size)), (H * L * D, L * D, D, 1)) for _ in range(8)]
    q, k, v, o, do, dq, dk, dv = t
    lse, delta, status = alloc(bytes(B * H * 384 * 4)), alloc(bytes(B * H * 384 * 4)), alloc(bytes(4))
    rows = [alloc(bytes(4 * B * L)) for _ in range(3)]
    ek = _lib.Ids(alloc(b"\\xff" * (8 * B * L)), (L, 0, 1), _lib.FA_ID_INT64)
    p = ops._problem(B, H, H, L, L, D, dt, False, 1, 1, 1.0)
    n = ctypes.c_size_t(0)
    assert lib.fa_plan_bytes(p, ctypes.byref(n)) == 0
    plan = alloc(bytes(n.value))
    rc = [lib.fa_group_rows(p, ek, *rows, status, None), lib.fa_plan_build(p, ek, ek, plan, n.value, status, None),
          lib.fa_fwd(p, q, k, v, o, lse, plan, status, None),
          lib.fa_bwd(p, q, k, v, o, do, lse, delta, dq, dk, dv, plan, status, None),
          static_plan(p, q, k, v, o, lse, ek, status), cu.cuCtxSynchronize()]
    got = ctypes.c_int32(-1)
    assert cu.cuMemcpyDtoH_v2(ctypes.byref(got), ctypes.c_uint64(status), ctypes.c_size_t(4)) == 0
    assert rc == [0] * 6 and got.value == 0, (dt, D, rc, got.value)
print("served")
"""


def test_second_context_of_a_device():
    r = subprocess.run([sys.executable, "-c", SCRIPT, PKG], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "served" in r.stdout, r.stderr[-2000:]
