// The host side of a regular `attention()` call in one native call each way: allocations, the problem and tensor
// descriptors, the launches of fa_b200.h and the autograd node. The general code and its node stay in Python (ops.py), and so do all
// messages: a call that is not regular (another layout, device, shape or type than the kernels take as they are) is declined with
// None, and ops.py copies, asks or raises. Bound by per-call overhead: a forward of 8 heads of 200
// queries took 27 us of host time around 8 us of kernel through ctypes; a training step of 4 x 12
// heads x 1000 x 64 in documents 122 us with the node in Python, 92 with the one below, around some 70 of kernels.
#include <ATen/SavedTensorHooks.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/custom_function.h>
#include <torch/csrc/autograd/python_cpp_function.h>
#include <torch/csrc/utils/pybind.h>
#include <torch/types.h>
#include <atomic>
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

fa_ids id_view(const Tensor& t) {
    return fa_ids{t.const_data_ptr(), {t.stride(0), t.stride(1), t.stride(2)}, t.scalar_type() == at::kInt ? FA_ID_INT32 : FA_ID_INT64};
}

// The plan of a call: its memory and the launches that fill it. eq and ek, if any, are int32 or int64 tensors [B, H, M] and [B, H, N].
Tensor build_plan(const fa_problem& p, const Tensor* eq, const Tensor* ek, const Tensor& status) {
    size_t bytes = 0;
    check(fa_plan_bytes(&p, &bytes), "fa_plan_bytes");
    Tensor plan = at::empty({int64_t(bytes / 4)}, status.options());
    const fa_ids q = eq ? id_view(*eq) : fa_ids{}, k = ek ? id_view(*ek) : fa_ids{};
    check(fa_plan_build(&p, eq ? &q : nullptr, ek ? &k : nullptr, plan.data_ptr(), bytes, status.data_ptr<int>(), current_stream(status)),
          "fa_plan_build");
    return plan;
}

// ops.build_plan. `problem` is the address of an fa_problem; ops.py has checked the ids.
Tensor plan(uintptr_t problem, const std::optional<Tensor>& eq, const std::optional<Tensor>& ek, const Tensor& status) {
    py::gil_scoped_release free;
    return build_plan(*reinterpret_cast<const fa_problem*>(problem), eq ? &*eq : nullptr, ek ? &*ek : nullptr, status);
}

struct Outputs {
    Tensor o, lse;
    int splits;
};

// The forward's allocations and launches for a problem that `regular` has filled.
Outputs launch_forward(const fa_problem& p, const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& plan, int key_runs,
                       const Tensor& status, const std::optional<Tensor>& out) {
    Outputs r;
    r.o = out ? *out : at::empty_like(q);
    if (!taken_as_is(r.o)) r.o = at::empty(q.sizes(), q.options());
    const auto f32 = q.options().dtype(at::kFloat);
    r.lse = at::empty({p.B, p.H, fa_padded_rows(p.M)}, f32);
    r.splits = key_runs != 0 ? key_runs : fa_fwd_splits(&p);  // (a number below 1 is the library's to refuse)
    Tensor work;
    size_t bytes = 0;
    if (r.splits > 1) {
        check(fa_fwd_workspace_bytes(&p, r.splits, &bytes), "fa_fwd_workspace_bytes");
        work = at::empty({int64_t(bytes / 4)}, f32);
    }
    const fa_tensor tq = view(q), tk = view(k), tv = view(v), to = view(r.o);
    check(fa_fwd_split(&p, &tq, &tk, &tv, &to, r.lse.data_ptr<float>(), plan.defined() ? plan.data_ptr() : nullptr, r.splits,
                       work.defined() ? work.data_ptr() : nullptr, bytes, status.data_ptr<int>(), current_stream(q)),
          "fa_fwd_split");
    return r;
}

// dq, dk, dv. q, k, v, o, lse and the problem are those of a forward, d_o is like q.
std::array<Tensor, 3> launch_backward(const fa_problem& p, const Tensor& d_o, const Tensor& q, const Tensor& k, const Tensor& v,
                                      const Tensor& o, const Tensor& lse, const Tensor& plan, const Tensor& status) {
    Tensor delta = at::empty_like(lse);
    Tensor dk = at::empty({p.B, p.Hk, p.N, p.D}, k.options()), dv = at::empty({p.B, p.Hk, p.N, p.D}, v.options());
    Tensor dq = at::empty(q.sizes(), q.options());
    const fa_tensor tq = view(q), tk = view(k), tv = view(v), to = view(o), tdo = view(d_o), tdq = view(dq), tdk = view(dk), tdv = view(dv);
    check(fa_bwd(&p, &tq, &tk, &tv, &to, &tdo, lse.data_ptr<float>(), delta.data_ptr<float>(), &tdq, &tdk, &tdv,
                 plan.defined() ? plan.data_ptr() : nullptr, status.data_ptr<int>(), current_stream(q)),
          "fa_bwd");
    return {std::move(dq), std::move(dk), std::move(dv)};
}

bool like_query(const Tensor& d_o, const Tensor& q) {
    return plain_cuda(d_o) && d_o.scalar_type() == q.scalar_type() && d_o.device() == q.device() && d_o.sizes() == q.sizes();
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
    Outputs r;
    {
        py::gil_scoped_release free;
        r = launch_forward(p, q, k, v, plan ? *plan : Tensor(), key_runs, status, out);
    }
    return py::make_tuple(std::move(r.o), std::move(r.lse), sm_scale, r.splits > 1 ? 2 : 1);
}

// (dq, dk, dv), or None. q, k, v, o, lse and the numbers are those of a forward.
py::object backward(const Tensor& d_o, const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& o, const Tensor& lse,
                    bool prepared, bool causal, double sm_scale, int mode, int id_heads, const std::optional<Tensor>& plan,
                    const Tensor& status) {
    fa_problem p;
    if (!regular(q, k, v, true, causal, sm_scale, mode, id_heads, p) || !like_query(d_o, q) || (!prepared && !taken_as_is(d_o)))
        return py::none();
    std::array<Tensor, 3> g;
    {
        py::gil_scoped_release free;
        g = launch_backward(p, d_o, q, k, v, o, lse, plan ? *plan : Tensor(), status);
    }
    return py::make_tuple(std::move(g[0]), std::move(g[1]), std::move(g[2]));
}

// Kernels launched by `attend` and its gradients (ops.LAUNCHES).
std::atomic<int64_t> n_launched{0};

// What a regular call is, besides q, k and v.
struct Call {
    fa_problem p;
    double sm_scale;
    const Tensor *eq, *ek;  // null without ids
    const Tensor& status;
    bool needs_grad;
    int plan_kernels;
};

// The autograd node of a regular call: what ops.FlashAttention does, without Python on the way of the gradients, whose thread would
// have to be given the interpreter first. Saves the same tensors; the plan is the node's own.
struct FlashAttention : torch::autograd::Function<FlashAttention> {
    static Tensor forward(torch::autograd::AutogradContext* ctx, const Tensor& q, const Tensor& k, const Tensor& v, const Call& c) {
        Tensor plan;
        Outputs r = launch(q, k, v, c, plan);
        torch::autograd::variable_list saved{q, k, v, r.o, r.lse};
        if (c.eq) {
            saved.push_back(*c.eq);
            saved.push_back(*c.ek);
        }
        ctx->save_for_backward(std::move(saved));
        ctx->saved_data["plan"] = plan;
        ctx->saved_data["status"] = c.status;
        ctx->saved_data["causal"] = int64_t(c.p.causal);
        ctx->saved_data["mode"] = int64_t(c.p.mode);
        ctx->saved_data["id_heads"] = int64_t(c.p.id_heads);
        ctx->saved_data["scale"] = c.sm_scale;
        return r.o;
    }

    // The plan, where the call needs one, and the forward.
    static Outputs launch(const Tensor& q, const Tensor& k, const Tensor& v, const Call& c, Tensor& plan) {
        py::gil_scoped_release free;
        if (c.eq || !fa_plan_optional(&c.p, c.needs_grad)) plan = build_plan(c.p, c.eq, c.ek, c.status);
        Outputs r = launch_forward(c.p, q, k, v, plan, 0, c.status, std::nullopt);
        n_launched += (plan.defined() ? c.plan_kernels : 0) + (r.splits > 1 ? 2 : 1);
        return r;
    }

    static torch::autograd::variable_list backward(torch::autograd::AutogradContext* ctx, torch::autograd::variable_list grads) {
        const auto saved = ctx->get_saved_variables();
        const Tensor &q = saved[0], &k = saved[1], &v = saved[2];
        const c10::cuda::CUDAGuard device(q.device());
        auto& data = ctx->saved_data;
        fa_problem p;
        TORCH_CHECK(regular(q, k, v, true, data["causal"].toInt() != 0, data["scale"].toDouble(), int(data["mode"].toInt()),
                            int(data["id_heads"].toInt()), p),
                    "flash_b200: the saved q, k, v are not plain [bs, H, L, D] CUDA tensors of matching shapes");
        Tensor d_o = grads[0];
        if (d_o.scalar_type() != q.scalar_type()) d_o = d_o.to(q.scalar_type());
        d_o = d_o.resolve_neg();
        TORCH_CHECK(like_query(d_o, q), "flash_b200: the gradient is not a plain [bs, H, M, D] CUDA tensor");
        if (!taken_as_is(d_o)) d_o = d_o.contiguous();  // (ops.maybe_contiguous)
        auto g = launch_backward(p, d_o, q, k, v, saved[3], saved[4], data["plan"].toTensor(), data["status"].toTensor());
        n_launched += 3;
        return {std::move(g[0]), std::move(g[1]), std::move(g[2]), Tensor()};
    }
};

// The whole of a regular call, its gradients included; None: ops.py takes it another way. Saved-tensor hooks count what is saved and by whom, so
// that their calls take ops.FlashAttention.
py::object attend(const Tensor& q, const Tensor& k, const Tensor& v, bool causal, std::optional<double> scale, const std::optional<Tensor>& eq,
                  const std::optional<Tensor>& ek, const py::int_& score_mode, const Tensor& status) {
    fa_problem p;
    int beyond = 0;  // (a number of any size: what no mode has is for ops.py to refuse)
    const long mode = PyLong_AsLongAndOverflow(score_mode.ptr(), &beyond);
    const double sm_scale = scale ? *scale : 1.0 / std::sqrt(double(q.dim() == 4 ? q.size(3) : 1));
    if (beyond != 0 || eq.has_value() != ek.has_value() || mode != (eq ? FA_MODE1_DOC : FA_MODE0_NOPE)) return py::none();
    if (!regular(q, k, v, false, causal, sm_scale, int(mode), 1, p)) return py::none();
    if (eq) {
        if (eq->device() != q.device() || ek->device() != q.device()) return py::none();
        p.id_heads = int(id_heads(*eq, *ek, p.B, p.H, p.M, p.N));
        if (p.id_heads == 0) return py::none();
    }
    const bool needs_grad = at::GradMode::is_enabled() && (q.requires_grad() || k.requires_grad() || v.requires_grad());
    if (needs_grad && at::SavedTensorDefaultHooks::get_hooks()) return py::none();
    const int plan_kernels = !eq || (p.M + 127) / 128 + (p.N + 127) / 128 <= FA_PLAN_ONE_KERNEL_BLOCKS ? 1 : 3;
    const Call call{p, sm_scale, eq ? &*eq : nullptr, ek ? &*ek : nullptr, status, needs_grad, plan_kernels};
    if (needs_grad) return py::cast(FlashAttention::apply(q, k, v, call));
    Tensor plan;
    return py::cast(FlashAttention::launch(q, k, v, call, plan).o);
}

int64_t launched() { return n_launched; }

// What `grad_fn` of a regular call shows to Python: what it shows of ops.FlashAttention (the reference's contract, flash_triton.py:558-562).
using Node = torch::autograd::CppNode<FlashAttention>;

Node& node_of(PyObject* self) { return static_cast<Node&>(*reinterpret_cast<torch::autograd::THPCppFunction*>(self)->cdata); }

// The engine's thread gives the saved tensors up, behind the node's lock, without the interpreter: so they are asked for.
torch::autograd::variable_list saved_tensors(Node& n) {
    struct Open : torch::autograd::Node {
        static std::mutex& lock_of(torch::autograd::Node& n) { return n.*(&Open::mutex_); }
    };
    py::gil_scoped_release free;
    const std::lock_guard<std::mutex> lock(Open::lock_of(n));
    return n.ctx_.get_saved_variables();
}

using Shown = py::object (*)(Node&);

PyObject* show(PyObject* self, void* get) {
    HANDLE_TH_ERRORS
    return reinterpret_cast<Shown>(get)(node_of(self)).release().ptr();
    END_HANDLE_TH_ERRORS
}

PyGetSetDef property(const char* name, Shown get) { return {name, show, nullptr, nullptr, reinterpret_cast<void*>(get)}; }

PyObject* node_name(PyObject*, PyObject*) { return PyUnicode_FromString("FlashAttentionBackward"); }

void register_node() {
    using namespace torch::autograd;
    static PyGetSetDef properties[] = {
        {"next_functions", THPCppFunction_next_functions, nullptr, nullptr, nullptr},
        {"requires_grad", THPCppFunction_requires_grad, nullptr, nullptr, nullptr},
        {"metadata", THPCppFunction_metadata, nullptr, nullptr, nullptr},
        {"_input_metadata", THPCppFunction_input_metadata, nullptr, nullptr, nullptr},
        property("saved_tensors", [](Node& n) -> py::object { return py::tuple(py::cast(saved_tensors(n))); }),
        property("needs_input_grad", [](Node& n) -> py::object {
            py::tuple t(8);  // of attention()'s arguments
            for (size_t i = 0; i < 8; ++i) t[i] = py::bool_(i < 3 && n.should_compute_output(i));
            return t;
        }),
        property("sm_scale", [](Node& n) -> py::object { return py::cast(n.ctx_.saved_data["scale"].toDouble()); }),
        property("causal", [](Node& n) -> py::object { return py::cast(n.ctx_.saved_data["causal"].toInt() != 0); }),
        property("score_func_info", [](Node& n) -> py::object { return py::make_tuple(n.ctx_.saved_data["mode"].toInt()); }),
        property("id_heads", [](Node& n) -> py::object { return py::cast(n.ctx_.saved_data["id_heads"].toInt()); }),
        property("plan", [](Node& n) -> py::object { return py::cast(n.ctx_.saved_data["plan"].toTensor()); }),  // (None where there is none)
        {nullptr, nullptr, nullptr, nullptr, nullptr},
    };
    static PyMethodDef methods[] = {
        {"name", node_name, METH_NOARGS, nullptr},
        {"register_hook", THPCppFunction_register_hook, METH_O, nullptr},
        {"register_prehook", THPCppFunction_register_prehook, METH_O, nullptr},
        {"_register_hook_dict", THPCppFunction_register_hook_dict, METH_O, nullptr},
        {"_sequence_nr", THPCppFunction_sequence_nr, METH_NOARGS, nullptr},
        {nullptr, nullptr, 0, nullptr},
    };
    static PyTypeObject type{PyVarObject_HEAD_INIT(nullptr, 0)};
    registerCppFunction(typeid(Node), _initFunctionPyTypeObject(type, "flash_b200._host.FlashAttentionNode", properties, methods));
}

}  // namespace

PYBIND11_MODULE(_host, m) {
    m.def("as_is", &as_is);
    m.def("id_heads", &id_heads);
    m.def("plan", &plan);
    m.def("forward", &forward);
    m.def("backward", &backward);
    m.def("attend", &attend);
    m.def("launched", &launched);
    register_node();
}
