"""The native autograd node shows what the node in Python shows, on the first call of a process as on every other."""
import os
import subprocess
import sys

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("which", [(True, True, True), (False, True, False)])
def test_attributes(mode, which, monkeypatch):
    import flash_b200 as fb
    from flash_b200 import ops
    monkeypatch.setattr(ops, "GROUP_QUERIES", False)
    B, H, L, D = 2, 4, 300, 128
    q, k, v, do = (torch.randn(B, H, L, D, device="cuda").bfloat16() for _ in range(4))
    ids = (-1 - torch.arange(L, device="cuda") // 70).expand(B, H, L) if mode else None
    x = [t.requires_grad_(w) for t, w in zip((q, k, v), which)]
    native, python = (call(*x, bool(mode), None, ids, ids, mode) for call in (fb.attention, fb.FlashAttention.apply))
    a, b = native.grad_fn, python.grad_fn
    assert type(a) is not type(b)
    assert a.name() == b.name() == "FlashAttentionBackward"
    for name in ("needs_input_grad", "sm_scale", "causal", "score_func_info", "id_heads"):
        assert getattr(a, name) == getattr(b, name) and type(getattr(a, name)) is type(getattr(b, name)), name
    assert (a.plan is None) == (b.plan is None) and (a.plan is None or a.plan.shape == b.plan.shape)
    assert type(a.saved_tensors) is tuple and len(a.saved_tensors) == len(b.saved_tensors) == (7 if mode else 5)
    for i, (s, t) in enumerate(zip(a.saved_tensors, b.saved_tensors)):
        if i == 4:  # what pads the rows of the LSE is not used
            s, t = s[..., :L], t[..., :L]
        assert torch.equal(s, t) and s.requires_grad == t.requires_grad
    assert a.saved_tensors[0].data_ptr() == q.data_ptr() and a.saved_tensors[3].data_ptr() == native.data_ptr()
    assert [f is None for f, _ in a.next_functions[:3]] == [f is None for f, _ in b.next_functions[:3]]
    seen = []
    a.register_hook(lambda grads, outs: seen.append((len(grads), len(outs))))
    a.register_prehook(lambda outs: seen.append(len(outs)))
    a.metadata["key"] = 1
    assert native.grad_fn.metadata == {"key": 1}
    wanted = [t for t in x if t.requires_grad]
    assert all(torch.equal(s, t) for s, t in zip(torch.autograd.grad(native, wanted, do), torch.autograd.grad(python, wanted, do)))
    assert seen[0] == 1 and len(seen) == 2
    for node in (a, b):
        with pytest.raises(RuntimeError, match="second time"):
            node.saved_tensors


def test_the_first_call_gets_the_same_node(repo_root):
    code = """
import torch, flash_b200 as fb
x = [torch.randn(1, 2, 200, 64, device="cuda").bfloat16().requires_grad_() for _ in range(3)]
first, second = fb.attention(*x, True), fb.attention(*x, True)
assert type(first.grad_fn) is type(second.grad_fn) and torch.equal(first, second)
"""
    path = os.path.join(repo_root, "triton-flash-attention-with-flexible-masks_b200")
    env = dict(os.environ, PYTHONPATH=path + os.pathsep + os.environ.get("PYTHONPATH", ""))
    r = subprocess.run([sys.executable, "-c", code], env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]


def test_saved_tensors_while_another_thread_frees_them():
    import threading
    import flash_b200 as fb
    x = [torch.randn(1, 2, 200, 64, device="cuda").bfloat16().requires_grad_() for _ in range(3)]
    do = torch.randn_like(x[0])
    for _ in range(50):
        o = fb.attention(*x, True)
        node, wrong, begun = o.grad_fn, [], threading.Event()

        def look():
            begun.set()
            while True:
                try:
                    if len(node.saved_tensors) != 5:
                        wrong.append("tensors missing")
                except RuntimeError as e:
                    if "second time" not in str(e):
                        wrong.append(str(e))
                    return

        threads = [threading.Thread(target=look) for _ in range(3)]
        for t in threads:
            t.start()
        begun.wait()
        torch.autograd.grad(o, x, do)
        for t in threads:
            t.join()
        assert not wrong
