// The per-call host path between PyTorch tensors and the C ABI: layout tests, output allocation, the
// argument struct and the call itself, in one native step per direction.  In Python the same steps take
// longer than the kernels of a small call.  The layout rules live here (functional.py calls them for row
// views).  Argument checks with their error texts, and the autograd functions, live in functional.py; an ordinary
// differentiable call takes the native autograd functions below.
#include <torch/csrc/utils/pybind.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/custom_function.h>
#include <torch/csrc/autograd/python_cpp_function.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/jit/frontend/tracer.h>
#include <ATen/ATen.h>
#include <ATen/PythonTorchFunctionTLS.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAStream.h>

#include <cstring>
#include <optional>
#include <tuple>

#include "../../include/na2d.h"

namespace {

using at::Tensor;
using MaybeTensor = std::optional<Tensor>;

// The library functions, as loaded by _lib.py (which may have been pointed at another build of them).
struct Abi {
    int (*forward)(const na2d_args*) = nullptr;
    int (*backward)(const na2d_args*) = nullptr;
    size_t (*backward_workspace)(const na2d_args*) = nullptr;
    int (*poll)(int, void*) = nullptr;
} abi;

void bind_abi(uintptr_t forward, uintptr_t backward, uintptr_t backward_workspace, uintptr_t poll) {
    abi.forward = reinterpret_cast<int (*)(const na2d_args*)>(forward);
    abi.backward = reinterpret_cast<int (*)(const na2d_args*)>(backward);
    abi.backward_workspace = reinterpret_cast<size_t (*)(const na2d_args*)>(backward_workspace);
    abi.poll = reinterpret_cast<int (*)(int, void*)>(poll);
}

int poll_device(int device) { return abi.poll(device, nullptr); }
uintptr_t current_stream(int device) { return reinterpret_cast<uintptr_t>(c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)device).stream()); }

// Whether the kernels can read t in place: contiguous channels, no broadcast dimension, and for 16-bit types (the
// tensor-core path's TMA tensor maps) a base and strides on 16-byte boundaries.
bool kernel_ready(const Tensor& t) {
    if (t.numel() == 0) return true;
    if (t.dim() == 0) return false;
    const auto sizes = t.sizes();
    const auto strides = t.strides();
    const int64_t last = t.dim() - 1;
    if (strides[last] != 1 && sizes[last] != 1) return false;
    const bool half = t.element_size() == 2;
    if (half && reinterpret_cast<uintptr_t>(t.data_ptr()) % 16) return false;
    for (int64_t i = 0; i < last; ++i) {
        if (sizes[i] <= 1) continue;
        if (strides[i] <= 0 || (half && strides[i] % 8)) return false;
    }
    return true;
}
Tensor in_place_or_copy(const Tensor& t) { return kernel_ready(t) ? t : t.contiguous(); }

// A dimension of extent 1 may report any stride; the library ignores it, but all-zero means dense.
int64_t at_least_one(int64_t stride) { return stride < 1 ? 1 : stride; }
na2d_tensor describe(const Tensor& t) {
    TORCH_CHECK_VALUE(t.dim() == 5 || t.dim() == 4, "expected (B, heads, H, W, C) or (B, heads, T, C); got ", t.dim(), " dimensions");
    const auto s = t.strides();
    if (t.dim() == 5)
        return {t.data_ptr(), at_least_one(s[0]), at_least_one(s[1]), at_least_one(s[2]), at_least_one(s[3])};
    return {t.data_ptr(), at_least_one(s[0]), at_least_one(s[1]), 0, at_least_one(s[2])};
}

na2d_args arguments(const Tensor& q, int64_t kernel_size, int path, double scale) {
    na2d_args a;
    std::memset(&a, 0, sizeof(a));
    a.struct_size = sizeof(a);
    const bool one_d = q.dim() == 4;
    a.op = one_d ? NA2D_OP_1D : NA2D_OP_2D;
    a.B = (int)q.size(0);
    a.N = (int)q.size(1);
    a.H = one_d ? 1 : (int)q.size(2);
    a.W = (int)q.size(one_d ? 2 : 3);
    a.C = (int)q.size(one_d ? 3 : 4);
    a.kernel_size = (int)kernel_size;
    a.dtype = q.scalar_type() == at::kFloat ? NA2D_F32 : q.scalar_type() == at::kBFloat16 ? NA2D_BF16 : NA2D_F16;
    a.path = path;
    a.device = q.device().index();
    a.scale = (float)scale;
    a.stream = c10::cuda::getCurrentCUDAStream(q.device().index()).stream();
    return a;
}

at::DimVector rows_of(const Tensor& q) { return at::DimVector(q.sizes().begin(), q.sizes().end() - 1); }

// Checked q, k, v -> (status, o, lse).
std::tuple<int, Tensor, Tensor> forward(const Tensor& q_in, const Tensor& k_in, const Tensor& v_in, int64_t kernel_size,
                                        int path, double scale) {
    const Tensor q = in_place_or_copy(q_in), k = in_place_or_copy(k_in), v = in_place_or_copy(v_in);
    Tensor o = at::empty(q.sizes(), q.options());
    Tensor lse = at::empty(rows_of(q), q.options().dtype(at::kFloat));
    int status = NA2D_OK;
    if (q.numel() != 0) {
        na2d_args a = arguments(q, kernel_size, path, scale);
        a.q = describe(q); a.k = describe(k); a.v = describe(v); a.o = describe(o);
        a.lse = lse.data_ptr<float>();
        status = abi.forward(&a);
    }
    return {status, o, lse};
}

// Operands of whole images, the differentiated ones checked -> (status, dQ, dK, dV), None for a half that is not wanted.
std::tuple<int, MaybeTensor, MaybeTensor, MaybeTensor> backward(const Tensor& q_in, const Tensor& k_in, const Tensor& v_in,
                                                                const MaybeTensor& o_in, const Tensor& lse_in,
                                                                const Tensor& d_o_in, int64_t kernel_size, int path,
                                                                double scale, bool need_dq, bool need_dkdv) {
    // (saved-tensor hooks may hand back anything for these two as well)
    TORCH_CHECK_VALUE(!o_in || (o_in->sizes().equals(q_in.sizes()) && o_in->scalar_type() == q_in.scalar_type() && o_in->device() == q_in.device()),
                      "o must match q in shape, dtype and device");
    TORCH_CHECK_VALUE(lse_in.sizes().equals(rows_of(q_in)) && lse_in.scalar_type() == at::kFloat && lse_in.device() == q_in.device(),
                      "lse must hold a float32 for each row of q, on its device");
    const Tensor lse = lse_in.contiguous(), q = in_place_or_copy(q_in), k = in_place_or_copy(k_in), v = in_place_or_copy(v_in);
    const Tensor d_o = in_place_or_copy(d_o_in);
    MaybeTensor o, d_q, d_k, d_v;
    if (o_in) o = in_place_or_copy(*o_in);
    if (need_dq) d_q = at::empty(q.sizes(), q.options());
    if (need_dkdv) {
        d_k = at::empty(k.sizes(), q.options());
        d_v = at::empty(k.sizes(), q.options());
    }
    int status = NA2D_OK;
    if (q.numel() != 0 && (need_dq || need_dkdv)) {
        Tensor delta = at::empty(rows_of(q), q.options().dtype(at::kFloat)), workspace;
        na2d_args a = arguments(q, kernel_size, path, scale);
        a.q = describe(q); a.k = describe(k); a.v = describe(v); a.d_o = describe(d_o);
        if (o) a.o = describe(*o);
        if (d_q) a.d_q = describe(*d_q);
        if (d_k) { a.d_k = describe(*d_k); a.d_v = describe(*d_v); }
        a.lse = lse.data_ptr<float>();
        a.delta = delta.data_ptr<float>();
        // Where memory is short, the halves take more turns with a smaller workspace; without any, the key half forms
        // the weights again.
        constexpr size_t kLeast = 1 << 20;
        for (size_t bytes = d_k ? abi.backward_workspace(&a) : 0; bytes != 0; bytes = bytes / 2 < kLeast ? 0 : bytes / 2) {
            try {
                workspace = at::empty({(int64_t)bytes}, q.options().dtype(at::kByte));
                a.workspace = workspace.data_ptr();
                a.workspace_bytes = bytes;
                break;
            } catch (const c10::OutOfMemoryError&) {
            }
        }
        status = abi.backward(&a);
    }
    return {status, d_q, d_k, d_v};
}

// ---- native autograd functions -----------------------------------------------------------------------------------
// Natten2d.apply(...)[0] and Natten1d.apply(...) of functional.py without the interpreter between autograd and the calls above:
// a step of 1 x 2 x 16 x 16 x 32, window 5, fp32, whose kernels took 43 us (39 now), took 85 us instead of 114 (the poll without a copy is
// part of that), one of 4 x 4 x 32 x 32 x 128, bf16, 81 instead of 113.  They save the same tensors in the same order and
// return the same gradients.

// Raises what _lib.check raises for a status.
void check(int status) {
    if (status == NA2D_OK) return;
    pybind11::gil_scoped_acquire gil;
    pybind11::module_::import("e_natten_b200._lib").attr("check")(status);
}

namespace ag = torch::autograd;

// What the operator takes; everything else is for functional.py, to serve or to refuse.
template <bool ONE_D>
bool takes(const Tensor& q, const Tensor& k, const Tensor& v, int64_t kernel_size) {
    const auto dtype = q.scalar_type();
    return q.is_cuda() && q.dim() == (ONE_D ? 4 : 5) && q.numel() != 0 && k.device() == q.device() && v.device() == q.device() &&
           k.scalar_type() == dtype && v.scalar_type() == dtype &&
           (dtype == at::kFloat || dtype == at::kBFloat16 || dtype == at::kHalf) && k.sizes().equals(q.sizes()) &&
           v.sizes().equals(q.sizes()) && q.size(2) >= kernel_size && (ONE_D || q.size(3) >= kernel_size);
}

template <bool ONE_D>
struct Attention : ag::Function<Attention<ONE_D>> {
    // A wait that gave up in a kernel of an earlier call surfaces here, without a sync.
    static void poll(const Tensor& q) {
        if constexpr (!ONE_D) check(poll_device(q.device().index()));
    }
    static Tensor forward(ag::AutogradContext* ctx, const Tensor& q, const Tensor& k, const Tensor& v, int64_t kernel_size,
                          double scale) {
        poll(q);
        auto [status, o, lse] = ::forward(q, k, v, kernel_size, NA2D_PATH_AUTO, scale);
        check(status);
        ctx->save_for_backward({q, k, v, o, lse});
        ctx->saved_data["kernel_size"] = kernel_size;
        ctx->saved_data["scale"] = scale;
        ctx->set_materialize_grads(false);
        return o;
    }
    static ag::variable_list backward(ag::AutogradContext* ctx, const ag::variable_list& grads) {
        const auto saved = ctx->get_saved_variables();
        const Tensor &q = saved[0], &k = saved[1], &v = saved[2];
        // an undefined gradient (a node above returned none) counts as zeros
        const Tensor d_o = grads[0].defined() ? grads[0] : at::zeros(q.sizes(), q.options());
        const bool need_dk = ctx->needs_input_grad(1), need_dv = ctx->needs_input_grad(2);
        const int64_t kernel_size = ctx->saved_data["kernel_size"].toInt();
        const double scale = ctx->saved_data["scale"].toDouble();
        MaybeTensor o, d_q, d_k, d_v;
        int status = NA2D_OK;
        // saved-tensor hooks may hand back other tensors than were saved: what the checks of functional.py say of them
        if (!takes<ONE_D>(q, k, v, kernel_size) || !d_o.sizes().equals(q.sizes()) || d_o.scalar_type() != q.scalar_type() ||
            d_o.device() != q.device()) {
            pybind11::gil_scoped_acquire gil;
            const auto functional = pybind11::module_::import("e_natten_b200.functional");
            using namespace pybind11::literals;
            const auto call = functional.attr(ONE_D ? "natten1d_backward" : "natten2d_backward");
            std::tie(d_q, d_k, d_v) = call(q, k, v, saved[3], saved[4], d_o, kernel_size, "need_dq"_a = ctx->needs_input_grad(0),
                                           "need_dkdv"_a = need_dk || need_dv, "scale"_a = scale)
                                          .template cast<std::tuple<MaybeTensor, MaybeTensor, MaybeTensor>>();
        } else {
            poll(q);
            if constexpr (!ONE_D) o = saved[3];
            std::tie(status, d_q, d_k, d_v) = ::backward(q, k, v, o, saved[4], d_o, kernel_size, NA2D_PATH_AUTO, scale,
                                                         ctx->needs_input_grad(0), need_dk || need_dv);
        }
        check(status);
        return {d_q.value_or(Tensor()), need_dk ? *d_k : Tensor(), need_dv ? *d_v : Tensor(), Tensor(), Tensor()};
    }
};

// What the graph node of a call shows in Python: the name and the attributes that the nodes of functional.py have.
template <bool ONE_D>
struct AttentionNode {
    static constexpr const char* kName = ONE_D ? "Natten1dBackward" : "Natten2dBackward";
    static ag::AutogradContext& context(PyObject* self) {
        return static_cast<ag::CppNode<Attention<ONE_D>>*>(reinterpret_cast<ag::THPCppFunction*>(self)->cdata.get())->ctx_;
    }
    static PyObject* name(PyObject*, PyObject*) { return PyUnicode_FromString(kName); }
    static PyObject* saved_tensors(PyObject* self, void*) {
        HANDLE_TH_ERRORS
        const auto saved = context(self).get_saved_variables();
        pybind11::tuple tensors(saved.size());
        for (size_t i = 0; i < saved.size(); ++i) tensors[i] = pybind11::cast(saved[i]);
        return tensors.release().ptr();
        END_HANDLE_TH_ERRORS
    }
    static PyObject* kernel_size(PyObject* self, void*) {
        HANDLE_TH_ERRORS
        return PyLong_FromLongLong(context(self).saved_data["kernel_size"].toInt());
        END_HANDLE_TH_ERRORS
    }
    static PyObject* scale(PyObject* self, void*) {
        HANDLE_TH_ERRORS
        return PyFloat_FromDouble(context(self).saved_data["scale"].toDouble());
        END_HANDLE_TH_ERRORS
    }
    static PyObject* set_sequence_nr(PyObject* self, PyObject* number) {
        HANDLE_TH_ERRORS
        const auto n = PyLong_AsUnsignedLongLong(number);
        if (PyErr_Occurred()) return nullptr;
        reinterpret_cast<ag::THPCppFunction*>(self)->cdata->set_sequence_nr(n);
        Py_RETURN_NONE;
        END_HANDLE_TH_ERRORS
    }
    static void add() {
        using namespace torch::autograd;
        // (those of every node, which PyTorch adds only where a type has none of its own, and the ones above)
        static PyMethodDef methods[] = {{"_register_hook_dict", THPCppFunction_register_hook_dict, METH_O, nullptr},
                                        {"register_hook", THPCppFunction_register_hook, METH_O, nullptr},
                                        {"register_prehook", THPCppFunction_register_prehook, METH_O, nullptr},
                                        {"_sequence_nr", THPCppFunction_sequence_nr, METH_NOARGS, nullptr},
                                        {"_set_sequence_nr", set_sequence_nr, METH_O, nullptr},
                                        {"name", name, METH_NOARGS, nullptr},
                                        {nullptr}};
        static PyGetSetDef properties[] = {THP_FUNCTION_DEFAULT_PROPERTIES,
                                           {"saved_tensors", saved_tensors, nullptr, nullptr, nullptr},
                                           {"kernel_size", kernel_size, nullptr, nullptr, nullptr},
                                           {"scale", scale, nullptr, nullptr, nullptr},
                                           {nullptr}};
        static PyTypeObject type;
        ag::registerCppFunction(typeid(ag::CppNode<Attention<ONE_D>>), ag::_initFunctionPyTypeObject(type, kName, properties, methods));
    }
};

// Whether anything looks into the call that the functions of functional.py serve and the native ones do not: a functional
// transform, forward-mode gradients, a trace, a function or dispatch mode.
bool looked_into() {
    const auto tls = c10::impl::tls_local_dispatch_key_set();
    return tls.included_.has(c10::DispatchKey::FuncTorchDynamicLayerFrontMode) || tls.included_.has(c10::DispatchKey::Functionalize) ||
           tls.included_.has(c10::DispatchKey::Python) || c10::impl::TorchDispatchModeTLS::any_modes_set() ||
           at::impl::torch_function_mode_enabled() || torch::jit::tracer::isTracing();
}
bool ordinary(const Tensor& t) {
    return t.is_cuda() && t.layout() == at::kStrided && !t.unsafeGetTensorImpl()->is_python_dispatch() && !t.is_neg() && !t.is_conj() &&
           !t._is_zerotensor() && !t.key_set().has(c10::DispatchKey::FuncTorchBatched) &&
           !t.key_set().has(c10::DispatchKey::FuncTorchGradWrapper) && !t.key_set().has(c10::DispatchKey::Functionalize) &&
           !t._fw_grad(0).defined();
}

// The operator on (q, k, v, kernel_size, scale) as the caller passed them; None where the call is not an ordinary one or an
// argument is not what the operator takes: functional.py serves it, or says what is wrong.
template <bool ONE_D>
pybind11::object attention(const pybind11::object& q_in, const pybind11::object& k_in, const pybind11::object& v_in,
                           const pybind11::object& kernel_size_in, const pybind11::object& scale_in) {
    for (const pybind11::object* t : {&q_in, &k_in, &v_in})
        if (!THPVariable_CheckExact(t->ptr())) return pybind11::none();
    if (!PyLong_CheckExact(kernel_size_in.ptr())) return pybind11::none();
    int overflow = 0;
    const long kernel_size = PyLong_AsLongAndOverflow(kernel_size_in.ptr(), &overflow);
    if (overflow != 0 || kernel_size <= 0 || kernel_size % 2 == 0) return pybind11::none();
    double scale = 1.0;
    if (PyFloat_CheckExact(scale_in.ptr())) scale = PyFloat_AS_DOUBLE(scale_in.ptr());
    else if (!scale_in.is_none()) return pybind11::none();
    const Tensor &q = THPVariable_Unpack(q_in.ptr()), &k = THPVariable_Unpack(k_in.ptr()), &v = THPVariable_Unpack(v_in.ptr());
    if (looked_into() || !ordinary(q) || !ordinary(k) || !ordinary(v) || !takes<ONE_D>(q, k, v, kernel_size)) return pybind11::none();
    Tensor o;
    {
        pybind11::gil_scoped_release no_gil;
        o = Attention<ONE_D>::apply(q, k, v, (int64_t)kernel_size, scale);
    }
    return pybind11::reinterpret_steal<pybind11::object>(THPVariable_Wrap(std::move(o)));
}

}  // namespace

PYBIND11_MODULE(_na2d_torch, m) {
    m.attr("built_for") = NA2D_EXT_TAG;         // looked for in the file by build.py
    m.def("bind_abi", &bind_abi);
    m.def("poll", &poll_device);
    m.def("stream", &current_stream);
    m.def("kernel_ready", &kernel_ready);
    m.def("strides", [](const Tensor& t) {      // (batch, heads, row, column), as they go into na2d_tensor
        const na2d_tensor d = describe(t);
        return std::make_tuple(d.stride_b, d.stride_n, d.stride_h, d.stride_w);
    });
    AttentionNode<false>::add();
    AttentionNode<true>::add();
    m.def("attention_2d", &attention<false>);
    m.def("attention_1d", &attention<true>);
    m.def("forward", &forward, pybind11::call_guard<pybind11::gil_scoped_release>());
    m.def("backward", &backward, pybind11::call_guard<pybind11::gil_scoped_release>());
}
