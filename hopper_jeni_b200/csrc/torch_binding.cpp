// Tensor-level host path in native code: argument checks, output allocation, the current stream and the autograd
// nodes around the C ABI, as one CPython module (`hopper_jeni_b200._gqa_torch`).
//
// Why it exists: a call's host work bounds every small problem.  Checked, allocated and marshalled in Python a forward
// cost 21 us of host time, a backward 56 us and an autograd step 163 us, against 5 to 40 us of GPU time at up to 256
// tokens.  Nothing here computes: the library does, through the function addresses that capi.py hands to bind() (so
// that a library chosen by GQA_B200_LIB is the one that runs).
#include <Python.h>

#include <ATen/ATen.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/custom_function.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/utils/pybind.h>

#include <cmath>
#include <optional>

#include "../../include/gqa.h"

namespace {

using at::Tensor;
using OptTensor = std::optional<Tensor>;

struct Api {
    decltype(&gqa_fwd_ex) fwd_ex = nullptr;
    decltype(&gqa_bwd_ex) bwd_ex = nullptr;
    decltype(&gqa_bwd_workspace_bytes_ex) bwd_workspace_bytes_ex = nullptr;
    decltype(&gqa_fwd_varlen) fwd_varlen = nullptr;
    decltype(&gqa_bwd_varlen) bwd_varlen = nullptr;
    decltype(&gqa_bwd_varlen_workspace_bytes) bwd_varlen_workspace_bytes = nullptr;
    PyObject* check = nullptr;  // capi.check: raises GqaError for a non-zero status
} api;

// A non-zero status of the library becomes the package's GqaError, in whatever thread the call was made (the
// autograd engine runs backward nodes in its own).
void check_status(const char* fn, int rc) {
    if (rc == GQA_OK) return;
    pybind11::gil_scoped_acquire gil;
    PyObject* r = PyObject_CallFunction(api.check, "si", fn, rc);
    Py_XDECREF(r);
    python_error e;
    e.persist();
    throw std::move(e);
}

void require(const Tensor& t, const char* name, at::ScalarType dtype) {
    TORCH_CHECK_VALUE(t.is_cuda(), name, " must be a CUDA tensor (this library has no CPU path)");
    TORCH_CHECK_VALUE(t.scalar_type() == dtype, name, " must be ", dtype, ", got ", t.scalar_type());
    TORCH_CHECK_VALUE(t.is_contiguous(), name, " must be contiguous");
}

// `t` lives on `like`'s device, is contiguous and has exactly the given shape and dtype: the library receives raw
// pointers, so a wrong-sized or wrong-device tensor would become an out-of-bounds access.
void require_like(const Tensor& t, const char* name, const Tensor& like, at::IntArrayRef shape, at::ScalarType dtype) {
    require(t, name, dtype);
    TORCH_CHECK_VALUE(t.device() == like.device(), name, " is on ", t.device(), ", expected ", like.device());
    TORCH_CHECK_VALUE(t.sizes() == shape, name, " has shape ", t.sizes(), ", expected ", shape);
}
void require_like(const Tensor& t, const char* name, const Tensor& like) {
    require_like(t, name, like, like.sizes(), like.scalar_type());
}

struct Dims {
    int B, Hq, Hkv, S, D;
};

int as_int(int64_t v) {
    TORCH_CHECK_VALUE(v >= INT_MIN && v <= INT_MAX, "dimension ", v, " is too large");
    return static_cast<int>(v);
}

// K against Q (V, dK and dV are compared with K, everything else with Q): nothing of a call is on another device.
void require_same_device(const Tensor& q, const Tensor& k) {
    TORCH_CHECK_VALUE(k.device() == q.device(), "K is on ", k.device(), ", expected ", q.device());
}

Dims dims(const Tensor& q, const Tensor& k, bool bshd) {
    TORCH_CHECK_VALUE(q.dim() == 4 && k.dim() == 4, "Q and K/V must be 4-dimensional");
    require_same_device(q, k);
    const int seq = bshd ? 1 : 2, head = bshd ? 2 : 1;
    TORCH_CHECK_VALUE(k.size(0) == q.size(0) && k.size(seq) == q.size(seq) && k.size(3) == q.size(3), "K/V shape ",
                      k.sizes(), " does not match Q ", q.sizes());
    return {as_int(q.size(0)), as_int(q.size(head)), as_int(k.size(head)), as_int(q.size(seq)), as_int(q.size(3))};
}

Dims packed_dims(const Tensor& q, const Tensor& k, const Tensor& cu) {
    TORCH_CHECK_VALUE(q.dim() == 3 && k.dim() == 3, "packed batches are [total_tokens, H, D]");
    require_same_device(q, k);
    TORCH_CHECK_VALUE(k.size(0) == q.size(0) && k.size(2) == q.size(2), "K ", k.sizes(), " does not match Q ", q.sizes());
    TORCH_CHECK_VALUE(cu.scalar_type() == at::kInt && cu.dim() == 1 && cu.numel() >= 2 && cu.is_cuda() &&
                          cu.device() == q.device() && cu.is_contiguous(),
                      "cu_seqlens must be a contiguous int32 vector of n_seqs + 1 entries on ", q.device());
    return {1, as_int(q.size(1)), as_int(k.size(1)), as_int(q.size(0)), as_int(q.size(2))};
}

float scale_or_default(double scale, int D) {  // NaN: not given
    return static_cast<float>(std::isnan(scale) ? 1.0 / std::sqrt(static_cast<double>(D)) : scale);
}

struct CallArgs {
    bool causal = false, bshd = false;
    double scale = std::nan("");
    unsigned bwd_flags = 0;                 // GQA_BWD_* of a backward call
    std::optional<uintptr_t> stream;
    bool subclass = false;                  // Q, K or V is of a subclass of torch.Tensor
};

// No autograd bookkeeping for the outputs, they are plain memory; not around what a subclass overrides.
struct PlainMemory {
    explicit PlainMemory(const CallArgs& a) {
        if (!a.subclass) below_.emplace();
    }
    std::optional<at::AutoDispatchBelowADInplaceOrView> below_;
};

// For a subclass of torch.Tensor: outputs are made through torch.empty_like (and contiguous copies through the method),
// so that they are of the subclass and its overrides are heard.  C++ knows neither.
Tensor unpack_result(PyObject* r) {
    if (!r) {
        python_error e;
        e.persist();
        throw std::move(e);
    }
    const auto owned = pybind11::reinterpret_steal<pybind11::object>(r);
    TORCH_CHECK_TYPE(THPVariable_Check(r), "expected a torch.Tensor, got ", Py_TYPE(r)->tp_name);
    return THPVariable_Unpack(r);
}
Tensor py_empty_like(const Tensor& t) {
    pybind11::gil_scoped_acquire gil;
    const auto self = pybind11::reinterpret_steal<pybind11::object>(THPVariable_Wrap(t));
    const auto torch = pybind11::reinterpret_steal<pybind11::object>(PyImport_ImportModule("torch"));
    return unpack_result(torch ? PyObject_CallMethod(torch.ptr(), "empty_like", "O", self.ptr()) : nullptr);
}
Tensor contiguous(const Tensor& t, const CallArgs& a) {
    if (!a.subclass || t.is_contiguous()) return t.contiguous();
    pybind11::gil_scoped_acquire gil;
    const auto self = pybind11::reinterpret_steal<pybind11::object>(THPVariable_Wrap(t));
    return unpack_result(PyObject_CallMethod(self.ptr(), "contiguous", nullptr));
}

// The device and the stream of one call, current for as long as this lives.  A stream that was given and is not the
// caller's current one owns what the call allocates: torch's allocator orders the reuse of a block by its stream, so a
// workspace taken from the current stream's pool could be handed out again, and an output could be memory that the
// current stream still uses, while the kernels run on the given one.
class CallStream {
public:
    CallStream(const Tensor& q, const CallArgs& a)
        : device_(q.device()),
          caller_(c10::cuda::getCurrentCUDAStream(q.get_device())),
          handle_(caller_.stream()),
          subclass_(a.subclass) {
        if (!a.stream || reinterpret_cast<cudaStream_t>(*a.stream) == caller_.stream()) return;
        const auto run = c10::cuda::getStreamFromExternal(reinterpret_cast<cudaStream_t>(*a.stream), q.get_device());
        handle_ = run.stream();
        given_.emplace(run);
    }
    gqa_stream_t handle() const { return handle_; }
    // A tensor that goes back to the caller: its block is not reused before the caller's stream is done with it, either.
    Tensor returned(Tensor t) const {
        if (given_) t.record_stream(caller_.unwrap());
        return t;
    }
    Tensor empty_like(const Tensor& t, const char* name) const {
        if (!subclass_) return returned(at::empty_like(t));
        Tensor r = py_empty_like(t);
        require_like(r, name, t);  // an override may have returned anything
        return returned(std::move(r));
    }
    Tensor empty_f32(const Tensor& like, at::IntArrayRef shape) const {
        return returned(at::empty(shape, like.options().dtype(at::kFloat)));
    }

private:
    const c10::cuda::CUDAGuard device_;
    const c10::cuda::CUDAStream caller_;
    gqa_stream_t handle_;
    const bool subclass_;
    std::optional<c10::cuda::CUDAStreamGuard> given_;
};

void check_qkv(const Tensor& q, const Tensor& k, const Tensor& v) {
    require(q, "Q", at::kBFloat16);
    require(k, "K", at::kBFloat16);
    require(v, "V", at::kBFloat16);
}

std::tuple<Tensor, Tensor> forward(const Tensor& q, const Tensor& k, const Tensor& v, const CallArgs& a, OptTensor out,
                                   OptTensor lse) {
    const PlainMemory below(a);
    check_qkv(q, k, v);
    const Dims d = dims(q, k, a.bshd);
    require_like(v, "V", k);
    const int64_t lse_shape[3] = {d.B, d.Hq, d.S};
    if (out) require_like(*out, "O", q);
    if (lse) require_like(*lse, "LSE", q, lse_shape, at::kFloat);
    const CallStream stream(q, a);
    if (!out) out = stream.empty_like(q, "O");
    if (!lse) lse = stream.empty_f32(q, lse_shape);
    check_status("gqa_fwd_ex", api.fwd_ex(q.data_ptr(), k.data_ptr(), v.data_ptr(), out->data_ptr(),
                                          static_cast<float*>(lse->data_ptr()), d.B, d.Hq, d.Hkv, d.S, d.D, a.causal,
                                          scale_or_default(a.scale, d.D), stream.handle(),
                                          a.bshd ? GQA_LAYOUT_BSHD : 0u));
    return {std::move(*out), std::move(*lse)};
}

std::tuple<Tensor, Tensor> forward_varlen(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& cu,
                                          int64_t max_seqlen, const CallArgs& a, OptTensor out, OptTensor lse) {
    const PlainMemory below(a);
    check_qkv(q, k, v);
    const Dims d = packed_dims(q, k, cu);
    require_like(v, "V", k);
    const int64_t lse_shape[2] = {d.Hq, d.S};
    if (out) require_like(*out, "O", q);
    if (lse) require_like(*lse, "LSE", q, lse_shape, at::kFloat);
    const CallStream stream(q, a);
    if (!out) out = stream.empty_like(q, "O");
    if (!lse) lse = stream.empty_f32(q, lse_shape);
    check_status("gqa_fwd_varlen",
                 api.fwd_varlen(q.data_ptr(), k.data_ptr(), v.data_ptr(), out->data_ptr(),
                                static_cast<float*>(lse->data_ptr()), static_cast<const int*>(cu.data_ptr()),
                                as_int(cu.numel()) - 1, d.S, as_int(max_seqlen), d.Hq, d.Hkv, d.D, a.causal,
                                scale_or_default(a.scale, d.D), stream.handle()));
    return {std::move(*out), std::move(*lse)};
}

struct Grads {
    Tensor dq, dk, dv;
};

// Everything of a backward call that does not depend on the layout; `lse_shape` is the LSE's.
struct BwdTensors {
    const Tensor &q, &k, &v, &o, &dout, &lse;
    OptTensor workspace, dq, dk, dv;

    void check_inputs() const {
        check_qkv(q, k, v);
        require(o, "O", at::kBFloat16);
        require(dout, "dO", at::kBFloat16);
        require(lse, "LSE", at::kFloat);
    }
    void check_all(at::IntArrayRef lse_shape) const {
        require_like(v, "V", k);
        require_like(o, "O", q);
        require_like(dout, "dO", q);
        if (dq) require_like(*dq, "dQ", q);
        if (dk) require_like(*dk, "dK", k);
        if (dv) require_like(*dv, "dV", k);
        require_like(lse, "LSE", q, lse_shape, at::kFloat);
        // its size is checked by the library (GQA_ERR_WORKSPACE, with the needed size in the error text)
        if (workspace)
            TORCH_CHECK_VALUE(workspace->is_cuda() && workspace->device() == q.device() && workspace->is_contiguous(),
                              "workspace must be contiguous memory on ", q.device());
    }
    void allocate(size_t need, const CallStream& stream) {
        if (!workspace) workspace = at::empty({static_cast<int64_t>(need)}, q.options().dtype(at::kByte));
        if (!dq) dq = stream.empty_like(q, "dQ");
        if (!dk) dk = stream.empty_like(k, "dK");
        if (!dv) dv = stream.empty_like(v, "dV");
    }
};

Grads backward(BwdTensors t, const CallArgs& a) {
    const PlainMemory below(a);
    t.check_inputs();
    const Dims d = dims(t.q, t.k, a.bshd);
    const size_t need = t.workspace ? 1
                                    : api.bwd_workspace_bytes_ex(d.B, d.Hq, d.Hkv, d.S, d.D, a.causal,
                                                                 a.bwd_flags & GQA_BWD_SPLIT_HEADS);
    if (need == 0) check_status("gqa_bwd_workspace_bytes", GQA_ERR_UNSUPPORTED);
    const int64_t lse_shape[3] = {d.B, d.Hq, d.S};
    t.check_all(lse_shape);
    const CallStream stream(t.q, a);
    t.allocate(need, stream);
    const unsigned flags = a.bwd_flags | (a.bshd ? GQA_LAYOUT_BSHD : 0u);
    check_status("gqa_bwd_ex",
                 api.bwd_ex(t.q.data_ptr(), t.k.data_ptr(), t.v.data_ptr(), t.o.data_ptr(), t.dout.data_ptr(),
                            static_cast<const float*>(t.lse.data_ptr()), t.dq->data_ptr(), t.dk->data_ptr(),
                            t.dv->data_ptr(), d.B, d.Hq, d.Hkv, d.S, d.D, a.causal, scale_or_default(a.scale, d.D),
                            t.workspace->data_ptr(), t.workspace->nbytes(), stream.handle(), flags));
    return {std::move(*t.dq), std::move(*t.dk), std::move(*t.dv)};
}

Grads backward_varlen(BwdTensors t, const Tensor& cu, int64_t max_seqlen, const CallArgs& a) {
    const PlainMemory below(a);
    t.check_inputs();
    const Dims d = packed_dims(t.q, t.k, cu);
    const size_t need = t.workspace ? 1 : api.bwd_varlen_workspace_bytes(d.S, d.Hq, d.Hkv, d.D);
    if (need == 0) check_status("gqa_bwd_varlen_workspace_bytes", GQA_ERR_UNSUPPORTED);
    const int64_t lse_shape[2] = {d.Hq, d.S};
    t.check_all(lse_shape);
    const CallStream stream(t.q, a);
    t.allocate(need, stream);
    check_status("gqa_bwd_varlen",
                 api.bwd_varlen(t.q.data_ptr(), t.k.data_ptr(), t.v.data_ptr(), t.o.data_ptr(), t.dout.data_ptr(),
                                static_cast<const float*>(t.lse.data_ptr()), t.dq->data_ptr(), t.dk->data_ptr(),
                                t.dv->data_ptr(), static_cast<const int*>(cu.data_ptr()), as_int(cu.numel()) - 1, d.S,
                                as_int(max_seqlen), d.Hq, d.Hkv, d.D, a.causal, scale_or_default(a.scale, d.D),
                                t.workspace->data_ptr(), t.workspace->nbytes(), stream.handle()));
    return {std::move(*t.dq), std::move(*t.dk), std::move(*t.dv)};
}

// ---- autograd nodes: the forward keeps O and LSE for the backward -----------------------------------------------
using torch::autograd::AutogradContext;
using torch::autograd::variable_list;

struct Attention : torch::autograd::Function<Attention> {
    static Tensor forward(AutogradContext* ctx, Tensor q, Tensor k, Tensor v, const CallArgs& a) {
        q = contiguous(q, a);
        k = contiguous(k, a);
        v = contiguous(v, a);
        auto [o, lse] = ::forward(q, k, v, a, std::nullopt, std::nullopt);
        ctx->save_for_backward({q, k, v, o, lse});
        ctx->saved_data["causal"] = a.causal;
        ctx->saved_data["bshd"] = a.bshd;
        ctx->saved_data["scale"] = a.scale;
        ctx->saved_data["subclass"] = a.subclass;
        ctx->saved_data["flags"] = static_cast<int64_t>(a.bwd_flags);
        return o;
    }
    static variable_list backward(AutogradContext* ctx, variable_list grads) {
        const variable_list s = ctx->get_saved_variables();
        CallArgs a;
        a.causal = ctx->saved_data["causal"].toBool();
        a.bshd = ctx->saved_data["bshd"].toBool();
        a.scale = ctx->saved_data["scale"].toDouble();
        a.subclass = ctx->saved_data["subclass"].toBool();
        a.bwd_flags = static_cast<unsigned>(ctx->saved_data["flags"].toInt());
        const Tensor dout = grads[0].contiguous();
        Grads g = ::backward({s[0], s[1], s[2], s[3], dout, s[4], {}, {}, {}, {}}, a);
        return {std::move(g.dq), std::move(g.dk), std::move(g.dv), Tensor()};
    }
};

struct AttentionVarlen : torch::autograd::Function<AttentionVarlen> {
    static Tensor forward(AutogradContext* ctx, Tensor q, Tensor k, Tensor v, const Tensor& cu, int64_t max_seqlen,
                          const CallArgs& a) {
        q = contiguous(q, a);
        k = contiguous(k, a);
        v = contiguous(v, a);
        auto [o, lse] = ::forward_varlen(q, k, v, cu, max_seqlen, a, std::nullopt, std::nullopt);
        ctx->save_for_backward({q, k, v, o, lse, cu});
        ctx->saved_data["causal"] = a.causal;
        ctx->saved_data["scale"] = a.scale;
        ctx->saved_data["subclass"] = a.subclass;
        ctx->saved_data["max_seqlen"] = max_seqlen;
        return o;
    }
    static variable_list backward(AutogradContext* ctx, variable_list grads) {
        const variable_list s = ctx->get_saved_variables();
        CallArgs a;
        a.causal = ctx->saved_data["causal"].toBool();
        a.scale = ctx->saved_data["scale"].toDouble();
        a.subclass = ctx->saved_data["subclass"].toBool();
        const Tensor dout = grads[0].contiguous();
        Grads g = ::backward_varlen({s[0], s[1], s[2], s[3], dout, s[4], {}, {}, {}, {}}, s[5],
                                    ctx->saved_data["max_seqlen"].toInt(), a);
        return {std::move(g.dq), std::move(g.dk), std::move(g.dv), Tensor(), Tensor(), Tensor()};
    }
};

// ---- CPython entry points (positional arguments only: the Python wrappers in ops.py and autograd.py name them) ----
const Tensor& tensor_arg(PyObject* o, const char* name) {
    TORCH_CHECK_TYPE(THPVariable_Check(o), name, " must be a torch.Tensor, got ", Py_TYPE(o)->tp_name);
    return THPVariable_Unpack(o);
}
OptTensor opt_tensor_arg(PyObject* o, const char* name) {
    if (o == Py_None) return std::nullopt;
    return tensor_arg(o, name);
}
bool subclass_arg(PyObject* q, PyObject* k, PyObject* v) {  // (a Parameter counts as a plain tensor)
    return !(THPVariable_CheckTypeExact(Py_TYPE(q)) && THPVariable_CheckTypeExact(Py_TYPE(k)) &&
             THPVariable_CheckTypeExact(Py_TYPE(v)));
}
bool bool_arg(PyObject* o) {
    const int r = PyObject_IsTrue(o);
    if (r < 0) throw python_error();
    return r != 0;
}
double scale_arg(PyObject* o) {
    if (o == Py_None) return std::nan("");
    const auto f = pybind11::reinterpret_steal<pybind11::object>(PyNumber_Float(o));  // whatever float() takes
    if (!f) throw python_error();
    const double v = PyFloat_AS_DOUBLE(f.ptr());
    return std::isnan(v) ? 0.0 : v;  // NaN marks "not given" above; the library refuses both
}
int64_t int_arg(PyObject* o) {
    const long long v = PyLong_AsLongLong(o);
    if (v == -1 && PyErr_Occurred()) throw python_error();
    return v;
}
std::optional<uintptr_t> stream_arg(PyObject* o) {  // None or a cudaStream_t as an integer
    if (o == Py_None) return std::nullopt;
    const unsigned long long v = PyLong_AsUnsignedLongLong(o);
    if (v == static_cast<unsigned long long>(-1) && PyErr_Occurred()) throw python_error();
    return static_cast<uintptr_t>(v);
}
bool layout_arg(PyObject* o) {  // true: [B,S,H,D]
    if (PyUnicode_Check(o)) {
        if (PyUnicode_CompareWithASCIIString(o, "bhsd") == 0) return false;
        if (PyUnicode_CompareWithASCIIString(o, "bshd") == 0) return true;
    }
    PyErr_Format(PyExc_ValueError, "layout must be 'bhsd' or 'bshd', got %R", o);
    throw python_error();
}
void count_args(Py_ssize_t n, Py_ssize_t want) {
    TORCH_CHECK_TYPE(n == want, "expected ", want, " arguments, got ", n);
    TORCH_CHECK_TYPE(api.check, "the module has not been bound to the library");
}
template <class... T>
PyObject* wrap(const T&... t) {
    PyObject* r = PyTuple_New(sizeof...(T));
    if (!r) throw python_error();
    Py_ssize_t i = 0;
    (PyTuple_SET_ITEM(r, i++, THPVariable_Wrap(t)), ...);
    return r;
}

// forward(q, k, v, causal, scale, out, lse, stream, layout)
PyObject* py_forward(PyObject*, PyObject* const* x, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    count_args(n, 9);
    CallArgs a;
    a.subclass = subclass_arg(x[0], x[1], x[2]);
    a.causal = bool_arg(x[3]);
    a.scale = scale_arg(x[4]);
    a.stream = stream_arg(x[7]);
    a.bshd = layout_arg(x[8]);
    const Tensor &q = tensor_arg(x[0], "Q"), &k = tensor_arg(x[1], "K"), &v = tensor_arg(x[2], "V");
    OptTensor out = opt_tensor_arg(x[5], "O"), lse = opt_tensor_arg(x[6], "LSE");
    std::tuple<Tensor, Tensor> r;
    {
        pybind11::gil_scoped_release release;
        r = forward(q, k, v, a, std::move(out), std::move(lse));
    }
    return wrap(std::get<0>(r), std::get<1>(r));
    END_HANDLE_TH_ERRORS
}

// backward(q, k, v, o, do, lse, causal, scale, workspace, dq, dk, dv, stream, layout, flags)
PyObject* py_backward(PyObject*, PyObject* const* x, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    count_args(n, 15);
    CallArgs a;
    a.subclass = subclass_arg(x[0], x[1], x[2]);
    a.causal = bool_arg(x[6]);
    a.scale = scale_arg(x[7]);
    a.stream = stream_arg(x[12]);
    a.bshd = layout_arg(x[13]);
    a.bwd_flags = static_cast<unsigned>(int_arg(x[14]));
    BwdTensors t{tensor_arg(x[0], "Q"),  tensor_arg(x[1], "K"),   tensor_arg(x[2], "V"), tensor_arg(x[3], "O"),
                 tensor_arg(x[4], "dO"), tensor_arg(x[5], "LSE"), opt_tensor_arg(x[8], "workspace"),
                 opt_tensor_arg(x[9], "dQ"), opt_tensor_arg(x[10], "dK"), opt_tensor_arg(x[11], "dV")};
    Grads g;
    {
        pybind11::gil_scoped_release release;
        g = backward(std::move(t), a);
    }
    return wrap(g.dq, g.dk, g.dv);
    END_HANDLE_TH_ERRORS
}

// forward_varlen(q, k, v, cu_seqlens, max_seqlen, causal, scale, out, lse, stream)
PyObject* py_forward_varlen(PyObject*, PyObject* const* x, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    count_args(n, 10);
    CallArgs a;
    a.subclass = subclass_arg(x[0], x[1], x[2]);
    a.causal = bool_arg(x[5]);
    a.scale = scale_arg(x[6]);
    a.stream = stream_arg(x[9]);
    const Tensor &q = tensor_arg(x[0], "Q"), &k = tensor_arg(x[1], "K"), &v = tensor_arg(x[2], "V"),
                 &cu = tensor_arg(x[3], "cu_seqlens");
    const int64_t max_seqlen = int_arg(x[4]);
    OptTensor out = opt_tensor_arg(x[7], "O"), lse = opt_tensor_arg(x[8], "LSE");
    std::tuple<Tensor, Tensor> r;
    {
        pybind11::gil_scoped_release release;
        r = forward_varlen(q, k, v, cu, max_seqlen, a, std::move(out), std::move(lse));
    }
    return wrap(std::get<0>(r), std::get<1>(r));
    END_HANDLE_TH_ERRORS
}

// backward_varlen(q, k, v, o, do, lse, cu_seqlens, max_seqlen, causal, scale, workspace, dq, dk, dv, stream)
PyObject* py_backward_varlen(PyObject*, PyObject* const* x, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    count_args(n, 15);
    CallArgs a;
    a.subclass = subclass_arg(x[0], x[1], x[2]);
    a.causal = bool_arg(x[8]);
    a.scale = scale_arg(x[9]);
    a.stream = stream_arg(x[14]);
    BwdTensors t{tensor_arg(x[0], "Q"),  tensor_arg(x[1], "K"),   tensor_arg(x[2], "V"), tensor_arg(x[3], "O"),
                 tensor_arg(x[4], "dO"), tensor_arg(x[5], "LSE"), opt_tensor_arg(x[10], "workspace"),
                 opt_tensor_arg(x[11], "dQ"), opt_tensor_arg(x[12], "dK"), opt_tensor_arg(x[13], "dV")};
    const Tensor& cu = tensor_arg(x[6], "cu_seqlens");
    const int64_t max_seqlen = int_arg(x[7]);
    Grads g;
    {
        pybind11::gil_scoped_release release;
        g = backward_varlen(std::move(t), cu, max_seqlen, a);
    }
    return wrap(g.dq, g.dk, g.dv);
    END_HANDLE_TH_ERRORS
}

// attention(q, k, v, causal, scale, layout, deterministic)
PyObject* py_attention(PyObject*, PyObject* const* x, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    count_args(n, 7);
    CallArgs a;
    a.subclass = subclass_arg(x[0], x[1], x[2]);
    a.causal = bool_arg(x[3]);
    a.scale = scale_arg(x[4]);
    a.bshd = layout_arg(x[5]);
    a.bwd_flags = bool_arg(x[6]) ? GQA_BWD_DETERMINISTIC : 0u;
    const Tensor &q = tensor_arg(x[0], "Q"), &k = tensor_arg(x[1], "K"), &v = tensor_arg(x[2], "V");
    Tensor o;
    {
        pybind11::gil_scoped_release release;
        o = Attention::apply(q, k, v, a);
    }
    return THPVariable_Wrap(o);
    END_HANDLE_TH_ERRORS
}

// attention_varlen(q, k, v, cu_seqlens, max_seqlen, causal, scale)
PyObject* py_attention_varlen(PyObject*, PyObject* const* x, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    count_args(n, 7);
    CallArgs a;
    a.subclass = subclass_arg(x[0], x[1], x[2]);
    a.causal = bool_arg(x[5]);
    a.scale = scale_arg(x[6]);
    const Tensor &q = tensor_arg(x[0], "Q"), &k = tensor_arg(x[1], "K"), &v = tensor_arg(x[2], "V"),
                 &cu = tensor_arg(x[3], "cu_seqlens");
    const int64_t max_seqlen = int_arg(x[4]);
    Tensor o;
    {
        pybind11::gil_scoped_release release;
        o = AttentionVarlen::apply(q, k, v, cu, max_seqlen, a);
    }
    return THPVariable_Wrap(o);
    END_HANDLE_TH_ERRORS
}

// bind(check, addresses of fwd_ex, bwd_ex, bwd_workspace_bytes_ex, fwd_varlen, bwd_varlen, bwd_varlen_workspace_bytes)
PyObject* py_bind(PyObject*, PyObject* const* x, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    TORCH_CHECK_TYPE(n == 7, "expected 7 arguments, got ", n);
    api.fwd_ex = reinterpret_cast<decltype(api.fwd_ex)>(int_arg(x[1]));
    api.bwd_ex = reinterpret_cast<decltype(api.bwd_ex)>(int_arg(x[2]));
    api.bwd_workspace_bytes_ex = reinterpret_cast<decltype(api.bwd_workspace_bytes_ex)>(int_arg(x[3]));
    api.fwd_varlen = reinterpret_cast<decltype(api.fwd_varlen)>(int_arg(x[4]));
    api.bwd_varlen = reinterpret_cast<decltype(api.bwd_varlen)>(int_arg(x[5]));
    api.bwd_varlen_workspace_bytes = reinterpret_cast<decltype(api.bwd_varlen_workspace_bytes)>(int_arg(x[6]));
    Py_INCREF(x[0]);
    api.check = x[0];
    Py_RETURN_NONE;
    END_HANDLE_TH_ERRORS
}

#define GQA_METHOD(name) \
    { #name, reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(py_##name)), METH_FASTCALL, nullptr }
PyMethodDef methods[] = {GQA_METHOD(bind),           GQA_METHOD(forward),         GQA_METHOD(backward),
                         GQA_METHOD(forward_varlen), GQA_METHOD(backward_varlen), GQA_METHOD(attention),
                         GQA_METHOD(attention_varlen), {nullptr, nullptr, 0, nullptr}};
PyModuleDef module_def = {PyModuleDef_HEAD_INIT, "_gqa_torch", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__gqa_torch(void) { return PyModule_Create(&module_def); }
