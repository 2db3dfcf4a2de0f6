// The host side of a regular `attention()` call in one native call each way: allocations, the problem and tensor
// descriptors, and the launches of fa_b200.h. The autograd node stays in Python (ops.py), and so do all messages: a
// call that is not regular (another layout, device, shape or type than the kernels take as they are) is declined with
// None, and ops.py's general code copies, asks or raises. Bound by per-call overhead: a forward of 8 heads of 200
// queries took 27 us of host time around 8 us of kernel through ctypes.
#include <c10/cuda/CUDAStream.h>
#include <c10/cuda/CUDAFunctions.h>
#include <torch/csrc/utils/pybind.h>
#include <torch/types.h>
#include <cmath>
#include "../../include/fa_b200.h"

namespace {

using at::Tensor;

int dtype_of(const Tensor& t) {
    switch (t.scalar_type()) {
        case at::kBFloat16: return FA_BF16;
        case at::kHalf: return FA_FP16;
        case at::kFloat: return FA_FP32;
        default: return -1;
    }
}

// what ops.maybe_contiguous leaves as it is
bool taken_as_is(const Tensor& t) {
    if (reinterpret_cast<uintptr_t>(t.const_data_ptr()) % 16 != 0) return false;
    if (t.is_contiguous() && t.size(3) % 8 == 0) return true;
    if (t.stride(3) != 1) return false;
    for (int i = 0; i < 3; ++i)
        if (t.size(i) > 1 && (t.stride(i) <= 0 || t.stride(i) % 8 != 0)) return false;
    return true;
}

fa_tensor view(const Tensor& t) {
    return fa_tensor{t.data_ptr(), {t.stride(0), t.stride(1), t.stride(2), t.stride(3)}};
}

void check(int rc, const char* what) {
    TORCH_CHECK(rc == FA_OK, what, " failed with code ", rc, ": ", fa_error_string(rc));
}

bool plain_cuda(const Tensor& t) {
    return t.is_cuda() && t.layout() == at::kStrided && t.dim() == 4 && !t.is_conj() && !t.is_neg();
}

// Fills `p`, or says that the call is not a regular one on the current device. `prepared`: ops.maybe_contiguous has seen the
// tensors already, and what the library does not take of what it returned the library refuses. There k and v may have more
// batches, and v more keys, than q and k ask for: the first ones are read.
bool regular(const Tensor& q, const Tensor& k, const Tensor& v, bool prepared, bool causal, double sm_scale, int mode, int id_heads,
             fa_problem& p) {
    if (!plain_cuda(q) || !plain_cuda(k) || !plain_cuda(v)) return false;
    const int dt = dtype_of(q);
    if (dt < 0 || k.scalar_type() != q.scalar_type() || v.scalar_type() != q.scalar_type()) return false;
    if (k.device() != q.device() || v.device() != q.device() || q.get_device() != c10::cuda::current_device()) return false;
    const int64_t B = q.size(0), H = q.size(1), M = q.size(2), D = q.size(3), Hk = k.size(1), N = k.size(2);
    if (D != 16 && D != 32 && D != 64 && D != 128) return false;
    if (k.size(3) != D || v.size(1) != Hk || v.size(3) != D) return false;
    if (prepared ? k.size(0) < B || v.size(0) < B || v.size(2) < N : k.size(0) != B || v.size(0) != B || v.size(2) != N) return false;
    if (B < 1 || H < 1 || M < 1 || Hk < 1 || N < 1 || B > 65535 || H > 65535 || M > INT32_MAX || N > INT32_MAX) return false;
    if (H % Hk != 0 || (causal && N < M) || !(sm_scale > 0)) return false;
    if (!prepared && (!taken_as_is(q) || !taken_as_is(k) || !taken_as_is(v))) return false;
    p = fa_problem{int(B), int(H), int(Hk), int(M), int(N), int(D), dt, causal ? 1 : 0, mode, id_heads, float(sm_scale)};
    return true;
}

void* current_stream(const Tensor& t) { return c10::cuda::getCurrentCUDAStream(t.get_device()).stream(); }

// Would ops.maybe_contiguous return all three as they are? (Where this says no, ops.py goes by that.)
bool as_is(const Tensor& q, const Tensor& k, const Tensor& v) {
    return plain_cuda(q) && plain_cuda(k) && plain_cuda(v) && taken_as_is(q) && taken_as_is(k) && taken_as_is(v);
}

// How many heads the ids of a call have, 1 or H, where they are as the library takes them; 0: ops.py looks, converts or refuses.
int64_t id_heads(const Tensor& eq, const Tensor& ek, int64_t B, int64_t H, int64_t M, int64_t N) {
    for (const Tensor* t : {&eq, &ek})
        if (!t->is_cuda() || t->layout() != at::kStrided || t->dim() != 3 || t->is_neg() || t->size(0) != B || t->size(1) != H ||
            t->size(2) != (t == &eq ? M : N) || (t->scalar_type() != at::kInt && t->scalar_type() != at::kLong))
            return 0;
    return H == 1 || (eq.stride(1) == 0 && ek.stride(1) == 0) ? 1 : H;
}

// The plan of a call (ops.build_plan): its memory and the launches that fill it. `problem` is the address of an fa_problem; the
// ids, if any, are int32 or int64 tensors [B, H, M] and [B, H, N] that ops.py has checked.
Tensor plan(uintptr_t problem, const std::optional<Tensor>& eq, const std::optional<Tensor>& ek, const Tensor& status) {
    const fa_problem* p = reinterpret_cast<const fa_problem*>(problem);
    auto ids = [](const Tensor& t) {
        return fa_ids{t.const_data_ptr(), {t.stride(0), t.stride(1), t.stride(2)}, t.scalar_type() == at::kInt ? FA_ID_INT32 : FA_ID_INT64};
    };
    py::gil_scoped_release free;
    size_t bytes = 0;
    check(fa_plan_bytes(p, &bytes), "fa_plan_bytes");
    Tensor plan = at::empty({int64_t(bytes / 4)}, status.options());
    const fa_ids q = eq ? ids(*eq) : fa_ids{}, k = ek ? ids(*ek) : fa_ids{};
    check(fa_plan_build(p, eq ? &q : nullptr, ek ? &k : nullptr, plan.data_ptr(), bytes, status.data_ptr<int>(), current_stream(status)),
          "fa_plan_build");
    return plan;
}

// (o, lse, scale, kernels launched), or None. Unprepared calls without a plan are taken only if it would gain nothing. `out`: a
// tensor like q for the result, given where q is of a subclass of torch.Tensor.
py::object forward(const Tensor& q, const Tensor& k, const Tensor& v, bool prepared, bool causal, std::optional<double> scale, int mode,
                   int id_heads, const std::optional<Tensor>& plan, bool backward, int key_runs, const Tensor& status,
                   const std::optional<Tensor>& out) {
    fa_problem p;
    const double sm_scale = scale ? *scale : 1.0 / std::sqrt(double(q.dim() == 4 ? q.size(3) : 1));
    if (!regular(q, k, v, prepared, causal, sm_scale, mode, id_heads, p)) return py::none();
    if (!plan && (mode != FA_MODE0_NOPE || (!prepared && !fa_plan_optional(&p, backward)))) return py::none();
    Tensor o, lse;
    int splits = 1;
    {
        py::gil_scoped_release free;
        o = out ? *out : at::empty_like(q);
        if (!taken_as_is(o)) o = at::empty(q.sizes(), q.options());
        const auto f32 = q.options().dtype(at::kFloat);
        lse = at::empty({p.B, p.H, fa_padded_rows(p.M)}, f32);
        splits = key_runs != 0 ? key_runs : fa_fwd_splits(&p);  // (a number below 1 is the library's to refuse)
        Tensor work;
        size_t bytes = 0;
        if (splits > 1) {
            check(fa_fwd_workspace_bytes(&p, splits, &bytes), "fa_fwd_workspace_bytes");
            work = at::empty({int64_t(bytes / 4)}, f32);
        }
        const fa_tensor tq = view(q), tk = view(k), tv = view(v), to = view(o);
        check(fa_fwd_split(&p, &tq, &tk, &tv, &to, lse.data_ptr<float>(), plan ? plan->data_ptr() : nullptr, splits,
                           work.defined() ? work.data_ptr() : nullptr, bytes, status.data_ptr<int>(), current_stream(q)),
              "fa_fwd_split");
    }
    return py::make_tuple(std::move(o), std::move(lse), sm_scale, splits > 1 ? 2 : 1);
}

// (dq, dk, dv), or None. q, k, v, o, lse and the numbers are those of a forward.
py::object backward(const Tensor& d_o, const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& o, const Tensor& lse,
                    bool prepared, bool causal, double sm_scale, int mode, int id_heads, const std::optional<Tensor>& plan,
                    const Tensor& status) {
    fa_problem p;
    if (!regular(q, k, v, true, causal, sm_scale, mode, id_heads, p) || !plain_cuda(d_o) || d_o.scalar_type() != q.scalar_type() ||
        d_o.device() != q.device() || d_o.sizes() != q.sizes() || (!prepared && !taken_as_is(d_o)))
        return py::none();
    Tensor dq, dk, dv;
    {
        py::gil_scoped_release free;
        Tensor delta = at::empty_like(lse);
        dk = at::empty({p.B, p.Hk, p.N, p.D}, k.options());
        dv = at::empty({p.B, p.Hk, p.N, p.D}, v.options());
        dq = at::empty(q.sizes(), q.options());
        const fa_tensor tq = view(q), tk = view(k), tv = view(v), to = view(o), tdo = view(d_o), tdq = view(dq), tdk = view(dk),
                        tdv = view(dv);
        check(fa_bwd(&p, &tq, &tk, &tv, &to, &tdo, lse.data_ptr<float>(), delta.data_ptr<float>(), &tdq, &tdk, &tdv,
                     plan ? plan->data_ptr() : nullptr, status.data_ptr<int>(), current_stream(q)),
              "fa_bwd");
    }
    return py::make_tuple(std::move(dq), std::move(dk), std::move(dv));
}

}  // namespace

PYBIND11_MODULE(_host, m) {
    m.def("as_is", &as_is);
    m.def("id_heads", &id_heads);
    m.def("plan", &plan);
    m.def("forward", &forward);
    m.def("backward", &backward);
}
