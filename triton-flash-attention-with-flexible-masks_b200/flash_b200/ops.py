"""Host-side mirror of the reference operator (flash_triton.py:506-641).

`attention(q, k, v, causal, sm_scale, eq, ek, score_func_mode)` keeps the reference's
signature, defaults, assertions, saved-tensor contract and return convention; the four Triton
launches are replaced by calls into libfa_b200.so (hand-written sm_100a kernels). There is no
Triton, no dispatch over back-ends and no CPU path: CPU tensors raise.
"""
import contextlib
import ctypes
import math
import os

import torch

from . import _lib

# scoring function modes (flash_triton.py:18-22)
SCORE_FUNC_MODE0_NOPE = 0  # no extra mask
SCORE_FUNC_MODE1_DOC = 1   # query id < 0: attend only to keys with the same id; id >= 0: attend to all

# bf16 / fp16 run on the tensor-core kernels; fp32 (accepted by the reference, flash_triton.py:512 and
# testing.py:158) on fp32 FMA kernels that are exact to fp32 rounding but not fast
_DTYPES = {torch.bfloat16: _lib.FA_BF16, torch.float16: _lib.FA_FP16, torch.float32: _lib.FA_FP32}
_STATUS = {}  # device index -> int32[1] status word
_SYNC_STATUS = os.environ.get("FA_B200_SYNC_STATUS", "0") not in ("", "0")
# When set to a list, every kernel launch appends (name, start_event, end_event) recorded on the
# launching stream. LAUNCHES (below) counts the library's kernels. Used by the benchmark only.
PROFILE = None
_launches = 0


def __getattr__(name):
    if name == "LAUNCHES":
        return _launches + (_HOST.launched() if _HOST is not None else 0)
    raise AttributeError(f"module {__name__!r} has no attribute {name!r}")


class _Timed:
    """Brackets one C-ABI call with CUDA events on the current stream when PROFILE is a list (`_timed`)."""

    def __init__(self, name):
        self.name = name

    def __enter__(self):
        # inside a CUDA graph capture the events become record nodes of the graph, re-recorded by
        # every replay and readable after it
        ext = torch.cuda.is_current_stream_capturing()
        self.e0 = torch.cuda.Event(enable_timing=True, external=ext)
        self.e1 = torch.cuda.Event(enable_timing=True, external=ext)
        self.e0.record()
        return self

    def __exit__(self, *exc):
        self.e1.record()
        if PROFILE is not None:
            PROFILE.append((self.name, self.e0, self.e1))
        return False


_UNTIMED = contextlib.nullcontext()


def _timed(name, kernels=1):
    global _launches
    _launches += kernels
    return _UNTIMED if PROFILE is None else _Timed(name)


def _count(kernels):
    global _launches
    _launches += kernels


def _current(device):
    """A context in which `device` is the current one; nothing to do, and nothing paid, if it is already."""
    return _UNTIMED if torch.cuda.current_device() == device.index else torch.cuda.device(device)


def _status_word(device):
    idx = device.index if device.index is not None else torch.cuda.current_device()
    st = _STATUS.get(idx)
    if st is None:
        st = torch.zeros(1, dtype=torch.int32, device=device)
        _STATUS[idx] = st
    return st


def check_status(device=None):
    """Synchronises `device` (default: every device used so far) and raises if a kernel recorded an
    error since the last check. A device given without an index means the current device.

    The status word of a device is sticky: once a bounded wait inside a kernel has run out, every
    later attention kernel on that device returns at once and fills its outputs with NaN, until this
    function has been called (it clears the word). Call it once per step, or set
    FA_B200_SYNC_STATUS=1 to have every forward and backward call do so."""
    if device is None:
        devs = list(_STATUS)
    else:
        idx = torch.device(device).index
        devs = [torch.cuda.current_device() if idx is None else idx]
    for idx in devs:
        st = _STATUS.get(idx)
        if st is None:
            continue
        code = int(st.item())
        if code != 0:
            st.zero_()
            if 100 <= code < 200:
                raise RuntimeError(f"flash_b200: a bounded wait inside a kernel ran out (role {code - 100}); "
                                   "results of that call are invalid")
            if code == 200:
                raise RuntimeError("flash_b200: a negative query id does not fit in int32")
            raise RuntimeError(f"flash_b200: kernel status {code}")


def maybe_contiguous(x):
    """flash_triton.py:435-437, extended by the TMA rules: last stride 1, 16-byte aligned base,
    other strides positive multiples of 8 elements, no pending negation."""
    x = x.resolve_neg()
    ok = x.data_ptr() % 16 == 0
    if ok and x.is_contiguous() and x.shape[-1] % 8 == 0:
        return x
    ok = ok and x.stride(-1) == 1
    if ok:
        for size, stride in zip(x.shape[:-1], x.stride()[:-1]):
            if size > 1 and (stride <= 0 or stride % 8 != 0):
                ok = False
    return x if ok else x.contiguous()


def _same_device(ref, **tensors):
    """Every pointer handed to the library is dereferenced on ref's device: a tensor that lives elsewhere
    (host memory, another GPU) must be refused here, before any launch."""
    for name, t in tensors.items():
        if t is not None and t.device != ref.device:
            raise ValueError(f"flash_b200: {name} is on {t.device}, but q is on {ref.device}; all tensors of a call "
                             "must be on the same CUDA device")


def _tensor(x):
    return _lib.Tensor(x.data_ptr(), x.stride())


def _ids(x):
    return _lib.Ids(x.data_ptr(), x.stride(), _lib.FA_ID_INT32 if x.dtype == torch.int32 else _lib.FA_ID_INT64)


def _id_tensor(e, B, H, L, name):
    assert e.dim() == 3 and e.shape[0] == B and e.shape[1] == H and e.shape[2] == L, \
        f"{name} must have shape [bs, H, L] = {[B, H, L]}, got {list(e.shape)}"
    assert not e.dtype.is_floating_point and not e.dtype.is_complex, f"{name} must hold integer ids"
    if e.dtype not in (torch.int32, torch.int64):
        e = e.to(torch.int64)
    return e


def _problem(B, H, Hk, M, N, D, dtype, causal, mode, id_heads, sm_scale):
    if dtype not in _DTYPES:
        raise NotImplementedError(f"flash_b200 supports bf16, fp16 and fp32 inputs, got {dtype}")
    return _lib.Problem(B, H, Hk, M, N, D, _DTYPES[dtype], 1 if causal else 0, int(mode), id_heads, float(sm_scale))


def _stream():
    """The current stream of the current device, as the library takes it."""
    return torch._C._cuda_getCurrentRawStream(torch.cuda.current_device())


def forward_splits(B, H, Hk, M, N, D, dtype, causal, mode):
    """Into how many runs the forward of this call cuts the keys of a query block (fa_fwd_splits): `attention_in_runs`
    takes it for a part of a call that is to give the bits of the whole one."""
    return _lib.load().fa_fwd_splits(ctypes.byref(_problem(B, H, Hk, M, N, D, dtype, causal, mode, 1, 1.0)))


def _plan_kernels(M, N):
    return 1 if (M + 127) // 128 + (N + 127) // 128 <= _lib.FA_PLAN_ONE_KERNEL_BLOCKS else 3


def build_plan(prob, eq, ek, status):
    """Mask plan: int32 device buffer consumed by the forward and backward kernels. With ids it
    holds their codes and block statistics; without (eq is None) only the kernels' work counters."""
    make = _PLAN or _host().plan
    if eq is None:
        _count(1)
        return make(ctypes.addressof(prob), None, None, status)
    with _timed("plan", _plan_kernels(prob.M, prob.N)):
        return make(ctypes.addressof(prob), eq, ek, status)


_own_build_plan = build_plan


def _host():
    """The native host calls (csrc/host.cpp); no call runs without them."""
    global _HOST, _PLAN, _AS_IS, _ID_HEADS
    if _HOST is None:
        _lib.load()
        from . import _host as module
        _HOST, _PLAN, _AS_IS, _ID_HEADS = module, module.plan, module.as_is, module.id_heads
    return _HOST


_HOST = _PLAN = _AS_IS = _ID_HEADS = None


def _like_subclass(q):
    """The result's tensor for a q of a subclass of torch.Tensor, so that it is one of them, too; else None."""
    return None if type(q) in _PLAIN else torch.empty_like(q)


# looked up once: a short call's host time is what bounds it
_TENSOR, _PLAIN, _tracing_state = torch.Tensor, (torch.Tensor, torch.nn.Parameter), torch._C._get_tracing_state
_transforms, _forward_ad = torch._C._functorch.peek_interpreter_stack, torch.autograd.forward_ad


def _native_forward(host, q, k, v, causal, sm_scale, needs_grad, key_runs):
    """One native call for a regular call without ids and without need of a plan; None for any other."""
    if (PROFILE is not None or _SYNC_STATUS or not (sm_scale is None or type(sm_scale) is float)
            or _tracing_state() is not None):  # (a trace would hold no kernel: the general code's checks refuse it)
        return None
    status = _STATUS.get(q.get_device())
    if status is None:
        return None
    return host.forward(q, k, v, False, bool(causal), sm_scale, SCORE_FUNC_MODE0_NOPE, 1, None, needs_grad, key_runs, status, _like_subclass(q))


class FlashAttention(torch.autograd.Function):
    """The autograd node of every call that `attend` (csrc/host.cpp) does not take."""

    @staticmethod
    def forward(ctx, q, k, v, causal, sm_scale, eq, ek, score_func_mode, key_runs=None):
        host = _HOST or _host()
        needs_grad = any(ctx.needs_input_grad[:3])
        done, plan, id_heads = None, None, 1
        if (eq is None and ek is None and score_func_mode == SCORE_FUNC_MODE0_NOPE and isinstance(q, _TENSOR) and isinstance(k, _TENSOR)
                and isinstance(v, _TENSOR)):
            done = _native_forward(host, q, k, v, causal, sm_scale, needs_grad, key_runs or 0)
        if done is None:
            # checks of flash_triton.py:510-520
            q_shape, k_shape, v_shape = q.shape, k.shape, v.shape
            Dq, Dk, Dv = q_shape[-1], k_shape[-1], v_shape[-1]
            assert Dq == Dk and Dk == Dv, "feature size of q, k, v should be equal"
            assert Dk in {16, 32, 64, 128}
            B, H, M, D = q_shape
            N = k_shape[2]
            Hk, Hv = k_shape[1], v_shape[1]
            assert Hk == Hv, "num of heads in k and v should be equal"
            assert H % Hk == 0, "number of heads in q must be a multiple of that in k & v"
            assert (N >= M) or (not causal), "KV length should be larger than M length in causal mode!"
            # score mode (flash_triton.py:527-530)
            assert (eq is None) == (ek is None)
            if eq is None:
                assert score_func_mode == SCORE_FUNC_MODE0_NOPE
            assert score_func_mode in (SCORE_FUNC_MODE0_NOPE, SCORE_FUNC_MODE1_DOC)
            score_func_mode = int(score_func_mode)
            if not q.is_cuda:
                raise RuntimeError("flash_b200 runs on CUDA tensors only (there is no CPU implementation)")
            device = q.device
            if k.device != device or v.device != device or (eq is not None and (eq.device != device or ek.device != device)):
                _same_device(q, k=k, v=v, eq=eq, ek=ek)
            if k.dtype != q.dtype or v.dtype != q.dtype:
                raise ValueError(f"flash_b200: q, k, v must share one dtype, got {q.dtype}, {k.dtype}, {v.dtype}")
            if sm_scale is None:
                sm_scale = 1. / math.sqrt(D)
            if not sm_scale > 0:
                raise NotImplementedError("flash_b200 needs sm_scale > 0")
            if not _AS_IS(q, k, v):
                q, k, v = maybe_contiguous(q), maybe_contiguous(k), maybe_contiguous(v)
            if score_func_mode == SCORE_FUNC_MODE1_DOC:
                id_heads = _ID_HEADS(eq, ek, B, H, M, N)
                if not id_heads:
                    eq = _id_tensor(eq, B, H, M, "eq")
                    ek = _id_tensor(ek, B, H, N, "ek")
                    broadcast = (H == 1) or (eq.stride(1) == 0 and ek.stride(1) == 0)
                    id_heads = 1 if broadcast else H
            with _current(device):
                prob = _problem(B, H, Hk, M, N, D, q.dtype, causal, score_func_mode, id_heads, sm_scale)
                status = _status_word(device)
                if score_func_mode == SCORE_FUNC_MODE1_DOC:
                    plan = build_plan(prob, eq, ek, status)
                elif not _lib.load().fa_plan_optional(prob, needs_grad):  # else so few items that counters would not pay
                    plan = build_plan(prob, None, None, status)
                with _timed("fwd", 0):
                    done = host.forward(q, k, v, True, bool(causal), float(sm_scale), score_func_mode, id_heads, plan, needs_grad,
                                        key_runs or 0, status, _like_subclass(q))
                if done is None:
                    raise RuntimeError("flash_b200: q, k, v are not plain [bs, H, L, D] CUDA tensors of matching shapes")
                if _SYNC_STATUS:
                    check_status(q.device)
        Out, L, ctx.sm_scale, launched = done
        _count(launched)
        # autograd context (flash_triton.py:558-562); eq/ek are kept for the saved-tensor contract,
        # the plan built from them is reused by backward
        if eq is None:
            ctx.save_for_backward(q, k, v, Out, L)
        else:
            ctx.save_for_backward(q, k, v, Out, L, eq, ek)
        ctx.plan = plan
        ctx.id_heads = id_heads
        ctx.causal = causal
        ctx.score_func_info = (int(score_func_mode), )
        ctx.n_other = 5 if key_runs is None else 6  # inputs that are not q, k, v
        return Out

    @staticmethod
    def backward(ctx, do):
        host = _HOST or _host()
        q, k, v, o, L = ctx.saved_tensors[:5]
        score_func_mode, = ctx.score_func_info
        device, plan = q.device, ctx.plan
        rest = (bool(ctx.causal), ctx.sm_scale, score_func_mode, ctx.id_heads, plan, _status_word(device))
        grads = None
        if PROFILE is None:  # the three kernels in one call
            grads = host.backward(do, q, k, v, o, L, False, *rest)
        if grads is None:
            if do.device != device:
                _same_device(q, do=do)
            if do.dtype != q.dtype:
                do = do.to(q.dtype)
            do = maybe_contiguous(do)
            with _current(device):
                grads = host.backward(do, q, k, v, o, L, True, *rest) if PROFILE is None else _backward_timed(do, q, k, v, o, L, *rest)
                if grads is None:
                    raise RuntimeError("flash_b200: the gradient is not a plain [bs, H, M, D] CUDA tensor")
        if PROFILE is None:
            _count(3)
        if _SYNC_STATUS:
            check_status(device)
        return grads + (None,) * ctx.n_other


def _backward_timed(do, q, k, v, o, L, causal, sm_scale, score_func_mode, id_heads, plan, status):
    """The backward with its kernels launched, and timed, one by one."""
    lib = _lib.load()
    (B, H, M, D), (Hk, N) = q.shape, k.shape[1:3]
    prob = _problem(B, H, Hk, M, N, D, q.dtype, causal, score_func_mode, id_heads, sm_scale)
    stream = _stream()
    plan_ptr = plan.data_ptr() if plan is not None else None
    delta = torch.empty_like(L)
    dk = torch.empty((B, Hk, N, D), dtype=k.dtype, device=q.device)
    dv = torch.empty((B, Hk, N, D), dtype=v.dtype, device=q.device)
    dq = torch.empty(q.shape, dtype=q.dtype, device=q.device)
    tq, tk, tv, to, tdo = _tensor(q), _tensor(k), _tensor(v), _tensor(o), _tensor(do)
    tdq, tdk, tdv = _tensor(dq), _tensor(dk), _tensor(dv)
    lp, dp, sp = L.data_ptr(), delta.data_ptr(), status.data_ptr()
    # delta = rowsum(o * do) (flash_triton.py:584-592)
    with _timed("delta"):
        _lib.check(lib.fa_bwd_delta(prob, to, tdo, dp, stream), "fa_bwd_delta")
    # dk, dv (flash_triton.py:594-614, group sum of :635-637 done inside the kernel)
    with _timed("dkdv"):
        _lib.check(lib.fa_bwd_dkdv(prob, tq, tk, tv, tdo, lp, dp, tdk, tdv, plan_ptr, sp, stream), "fa_bwd_dkdv")
    # dq (flash_triton.py:616-634); every row is written by the kernel
    with _timed("dq"):
        _lib.check(lib.fa_bwd_dq(prob, tq, tk, tv, tdo, lp, dp, tdq, plan_ptr, sp, stream), "fa_bwd_dq")
    return dq, dk, dv


# Without a causal mask the order of the queries is free. When the query ids are not grouped (every
# block of 128 queries holds every document) no tile can be skipped and every tile needs the id check.
# Calls in document mode without a causal mask therefore first sort the query rows by id inside the
# library (fa_group_rows: a stable sort, so ids that are grouped already keep their places), run the
# kernels on the grouped rows, whose blocks are (nearly) uniform again, and put o back in the caller's
# order; backward does the same with dO and dQ. The cost is one sort of the ids and two row permutations
# per pass. GROUP_QUERIES = False (or FA_B200_GROUP_QUERIES=0 in the environment) runs such calls in the
# caller's order. Longer rows than the library sorts (FA_GROUP_MAX_ROWS) always run in the caller's order.
GROUP_QUERIES = os.environ.get("FA_B200_GROUP_QUERIES", "1") not in ("", "0")


def _permute_rows(x, index, id_heads):
    """out[b, h, i, :] = x[b, h, index[b, he, i], :] by the library's row-permutation kernel."""
    lib = _lib.load()
    x = maybe_contiguous(x)
    B, H, M, D = x.shape
    out = torch.empty((B, H, M, D), dtype=x.dtype, device=x.device)
    with _current(x.device):
        prob = _problem(B, H, H, M, M, D, x.dtype, False, SCORE_FUNC_MODE1_DOC, id_heads, 1.0)
        tx, to = _tensor(x), _tensor(out)
        with _timed("permute"):
            _lib.check(lib.fa_permute_rows(prob, tx, to, index.data_ptr(),
                                           _stream()), "fa_permute_rows")
    return out


class _PermuteRows(torch.autograd.Function):
    """y[..., i, :] = x[..., index[i], :]; the gradient moves through the inverse permutation."""

    @staticmethod
    def forward(ctx, x, index, inverse, id_heads):
        ctx.save_for_backward(inverse)
        ctx.id_heads = id_heads
        return _permute_rows(x, index, id_heads)

    @staticmethod
    def backward(ctx, g):
        inverse, = ctx.saved_tensors
        return _permute_rows(g, inverse, ctx.id_heads), None, None, None


def group_rows(eq, B, H, M):
    """(order, inverse, grouped_ids, id_heads): the stable sort of each id row of eq [B, H, M] by the mask's
    id code, as int32 tensors [B, id_heads, M] (id_heads is 1 when eq is broadcast over the heads)."""
    lib = _lib.load()
    eq = _id_tensor(eq, B, H, M, "eq")
    id_heads = 1 if (H == 1 or eq.stride(1) == 0) else H
    with _current(eq.device):
        out = torch.empty((3, B, id_heads, M), dtype=torch.int32, device=eq.device)
        prob = _problem(B, H, H, M, M, 64, torch.bfloat16, False, SCORE_FUNC_MODE1_DOC, id_heads, 1.0)
        ieq = _ids(eq)
        status = _status_word(eq.device)
        with _timed("group"):
            _lib.check(lib.fa_group_rows(prob, ieq, out[0].data_ptr(), out[1].data_ptr(),
                                         out[2].data_ptr(), status.data_ptr(), _stream()), "fa_group_rows")
    return out[0], out[1], out[2], id_heads


def _attention_grouped(q, k, v, sm_scale, eq, ek):
    B, H, M, D = q.shape
    _same_device(q, eq=eq)
    order, inverse, grouped, id_heads = group_rows(eq, B, H, M)
    q_g = _PermuteRows.apply(q, order, inverse, id_heads)
    o_g = FlashAttention.apply(q_g, k, v, False, sm_scale, grouped.expand(B, H, M), ek, SCORE_FUNC_MODE1_DOC)
    return _PermuteRows.apply(o_g, inverse, order, id_heads)


def attention(q, k, v, causal=False, sm_scale=None, eq=None, ek=None, score_func_mode=SCORE_FUNC_MODE0_NOPE):
    """Drop-in for flash_triton.py:640-641.

    The tensor-core kernels are built for head dims 64 and 128. For 16-bit inputs the reference's smaller
    head dims (16 and 32, flash_triton.py:512) run on the 64-wide kernels without any padded copy: the library
    describes the tensors to the TMA unit with their real head dim, the loads fill the missing columns of a
    tile with zeros (zero columns add nothing to q k^T and give zero output columns) and the stores write the
    real columns only."""
    if (GROUP_QUERIES and score_func_mode == SCORE_FUNC_MODE1_DOC and not causal and eq is not None and ek is not None
            and q.is_cuda and q.dim() == 4 and 128 < q.shape[2] <= _lib.FA_GROUP_MAX_ROWS):
        return _attention_grouped(q, k, v, sm_scale, eq, ek)
    # Regular calls go to the library in one native call, with a native autograd node where a gradient is needed. A small training step is
    # bound by its host time: 4 x 12 heads x 1000 x 64 in documents, some 70 us of kernels, 122 us a step with the node of this module (its backward waits for
    # the interpreter in the engine's thread), 92 with the native one. Transforms of torch.func and forward-mode gradients need
    # the node of this module for their messages, subclasses for their hooks, and a trace for its refusal.
    # Without a gradient there is no node at all: 8 heads of 200 queries took 13.6 us a call with the one of this module, 7.5 now.
    if (type(q) in _PLAIN and type(k) in _PLAIN and type(v) in _PLAIN and type(score_func_mode) is int and (eq is None or type(eq) in _PLAIN)
            and (ek is None or type(ek) in _PLAIN) and (sm_scale is None or type(sm_scale) is float) and PROFILE is None and not _SYNC_STATUS
            and build_plan is _own_build_plan  # (not somebody's own)
            and _transforms() is None and _forward_ad._current_level < 0 and _tracing_state() is None):
        host, status = _HOST, _STATUS.get(q.get_device())
        if status is None and q.is_cuda:  # the first call on a device gets the same node as the others
            host, status = host or _host(), _status_word(q.device)
        attend = getattr(host, "attend", None)
        if attend is not None and status is not None:
            done = attend(q, k, v, bool(causal), sm_scale, eq, ek, score_func_mode, status)
            if done is not None:
                return done
    return FlashAttention.apply(q, k, v, causal, sm_scale, eq, ek, score_func_mode)


def attention_in_runs(q, k, v, key_runs, causal=False, sm_scale=None):
    """`attention` without ids, with the keys cut into `key_runs` runs in the forward.

    `attention` chooses a number where a call cannot fill the GPU (few queries) from its sizes, the batch and the SM count
    among them (`forward_splits`), so that a sequence's result can differ in its last bits with what it is batched with.
    1 computes every sequence in one run, whatever lies beside it; another number, at most one per 128 keys (fp32: 1),
    is for callers that fix it by the sequence alone or, for the shards of a call, by the whole call."""
    return FlashAttention.apply(q, k, v, causal, sm_scale, None, None, SCORE_FUNC_MODE0_NOPE, int(key_runs))


def debug_mask(B, H, M, N, causal, eq=None, ek=None, score_func_mode=SCORE_FUNC_MODE0_NOPE, device="cuda"):
    """Materialises the kernels' keep / tile-class decisions: returns (keep [B,He,M,N] bool,
    tile_class [B,He,nQ,nK] uint8) computed on the device by the attention kernels' own predicate."""
    lib = _lib.load()
    device = torch.device(device)
    if device.type != "cuda":
        raise RuntimeError("flash_b200 runs on CUDA devices only (there is no CPU implementation)")
    if device.index is None:
        device = torch.device("cuda", torch.cuda.current_device())
    for name, t in (("eq", eq), ("ek", ek)):
        if t is not None and t.device != device:
            raise ValueError(f"flash_b200: {name} is on {t.device}, but the mask is evaluated on {device}")
    id_heads = 1
    with torch.cuda.device(device):
        status = _status_word(device)
        if score_func_mode == SCORE_FUNC_MODE1_DOC:
            eq = _id_tensor(eq, B, H, M, "eq")
            ek = _id_tensor(ek, B, H, N, "ek")
            id_heads = 1 if (H == 1 or (eq.stride(1) == 0 and ek.stride(1) == 0)) else H
        prob = _problem(B, H, H, M, N, 64, torch.bfloat16, causal, score_func_mode, id_heads, 1.0)
        plan = build_plan(prob, eq, ek, status) if score_func_mode == SCORE_FUNC_MODE1_DOC else None
        He = id_heads if score_func_mode == SCORE_FUNC_MODE1_DOC else 1
        nQ, nK = (M + 127) // 128, (N + 127) // 128
        keep = torch.zeros((B, He, M, N), dtype=torch.uint8, device=device)
        cls = torch.zeros((B, He, nQ, nK), dtype=torch.uint8, device=device)
        _lib.check(lib.fa_debug_mask(prob, plan.data_ptr() if plan is not None else None,
                                     keep.data_ptr(), cls.data_ptr(), _stream()), "fa_debug_mask")
    return keep.bool(), cls
