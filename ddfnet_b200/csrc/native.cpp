// The operator's (and the stem pooling's) host path in C++: argument checks, output allocation, autograd node and the call
// into libddf_b200.so.  A call of `ddf` through torch.autograd.Function and ctypes cost 28 us of
// host time (forward) and 140 us (forward + backward through autograd) -- more than the GPU needs
// for most shapes up to a few hundred microseconds of device work; the same call here costs a few
// microseconds, most of it the launch itself.
//
// Semantics are those of the reference's autograd function (ddf/ddf.py:27-122).  This path takes the
// ordinary call: arguments that pass the checks below, plain tensors, nothing that watches or
// transforms the program.  Every other call goes to the Python function `general` (op.py), the same
// operator as a torch.autograd.Function: it raises the reference's assertions and this framework's
// errors, and torch handles it under jit tracing (a node past the tracer would leave the traced
// batch's output in the graph as a constant), functorch transforms, dispatch modes and forward mode.
//
// The library's entry points are bound by address (bind()), so DDF_B200_LIB keeps working.
#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/SequenceNumber.h>
#include <ATen/cuda/CUDAGraphsUtils.cuh>
#include <ATen/cuda/EmptyTensor.h>
#include <ATen/record_function.h>
#include <c10/core/impl/LocalDispatchKeySet.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/function.h>
#include <torch/csrc/autograd/functions/utils.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/autograd/saved_variable.h>

#include <cstring>
#include <string>

#include "../../include/ddf_b200.h"

namespace {

using at::Tensor;

// ------------------------------------------------------------------ bound entry points
struct Library {
    decltype(&ddf_b200_forward) forward = nullptr;
    decltype(&ddf_b200_forward_sfnorm) forward_sfnorm = nullptr;
    decltype(&ddf_b200_backward_workspace) backward_workspace = nullptr;
    decltype(&ddf_b200_backward) backward = nullptr;
    decltype(&ddf_b200_sfnorm) sfnorm = nullptr;
    decltype(&ddf_b200_sfnorm_backward) sfnorm_backward = nullptr;
    decltype(&ddf_b200_maxpool_nhwc) maxpool_nhwc = nullptr;
    decltype(&ddf_b200_take_fault) take_fault = nullptr;
} lib;
PyObject* g_error_class = nullptr;  // _lib.DDFError
PyObject* g_general = nullptr;      // op._general
PyObject* g_load = nullptr;         // op._bind_native: loads the library and calls bind()
bool g_debug = false;

[[noreturn]] void raise_python() {
    python_error e;
    e.persist();
    throw e;
}

// A non-zero status becomes _lib.DDFError(status); with DDF_B200_DEBUG=1 the fault word is read
// after every call.  Called without the GIL.
void check(int status) {
    if (C10_LIKELY(status == 0 && !g_debug)) return;
    if (status != 0) {
        pybind11::gil_scoped_acquire gil;
        PyObject* v = PyLong_FromLong(status);
        PyErr_SetObject(g_error_class, v);
        Py_XDECREF(v);
        raise_python();
    }
    if (at::cuda::currentStreamCaptureStatusMayInitCtx() != at::cuda::CaptureStatus::None) return;
    const int fault = lib.take_fault();
    if (fault != 0)
        throw std::runtime_error("ddf_b200: a kernel's bounded wait ran out (fault code " + std::to_string(fault) +
                                 "); the output of the last call is incomplete");
}

int dtype_code(at::ScalarType t) {
    switch (t) {
        case at::kFloat: return DDF_B200_F32;
        case at::kHalf: return DDF_B200_F16;
        case at::kBFloat16: return DDF_B200_BF16;
        case at::kDouble: return DDF_B200_F64;
        default: return -1;
    }
}

Tensor empty_like_on(at::IntArrayRef sizes, at::ScalarType dt, const at::Device& dev) {
    return at::detail::empty_cuda(sizes, dt, dev, std::nullopt);
}

void* ptr(const Tensor& t) { return t.defined() ? t.data_ptr() : nullptr; }

// ------------------------------------------------------------------ one call's parameters
struct Params {
    int k = 3, d = 1, s = 1, combine = DDF_B200_MUL;
    int variant = DDF_B200_VARIANT_AUTO;
    bool norm = false;    // spatial FilterNorm inside the kernel (ddf_sfnorm)
    double scale = 1.0;
};

// ------------------------------------------------------------------ autograd node
struct DDFBackward : public torch::autograd::Node {
    std::string name() const override { return p.norm ? "DDFSpatialNormFunctionBackward" : "DDFFunctionBackward"; }

    void release_variables() override {
        std::lock_guard<std::mutex> lock(mutex_);
        x_.reset_data();
        cf_.reset_data();
        sf_.reset_data();
        released = true;
    }

    torch::autograd::variable_list apply(torch::autograd::variable_list&& grads) override {
        torch::autograd::variable_list out(3);
        std::lock_guard<std::mutex> lock(mutex_);
        TORCH_CHECK(!released, torch::autograd::ERR_BACKWARD_TWICE);
        const bool need_x = task_should_compute_output(0), need_cf = task_should_compute_output(1),
                   need_sf = task_should_compute_output(2);
        const Tensor x = x_.unpack(), cf = cf_.unpack(), sf = sf_.unpack();
        at::NoGradGuard no_grad;
        const at::ScalarType dt = x.scalar_type();
        // a gradient that never reached the output is zero, as torch.autograd.Function has it
        Tensor go = grads[0].defined() ? grads[0]
                                       : at::zeros({x.size(0), x.size(1), x.size(2) / p.s, x.size(3) / p.s}, x.options());
        TORCH_CHECK(go.is_cuda(), "the gradient of the op's output must be a CUDA tensor");
        if (go.scalar_type() != dt) go = go.to(dt);
        go = go.contiguous();

        const int B = (int)x.size(0), C = (int)x.size(1), H = (int)x.size(2), W = (int)x.size(3);
        const int dtc = dtype_code(dt);
        const at::Device dev = x.device();
        c10::cuda::CUDAGuard guard(dev);
        void* stream = c10::cuda::getCurrentCUDAStream(dev.index()).stream();
        // 'f' selects a forward kernel only, as in the reference (ddf/ddf.py:71,103,114)
        const int variant = p.variant == DDF_B200_VARIANT_GENERIC ? DDF_B200_VARIANT_GENERIC : DDF_B200_VARIANT_AUTO;

        Tensor filter = sf;
        if (p.norm) {  // the normalised filter, recomputed once for the gradient kernels
            filter = empty_like_on(sf.sizes(), dt, dev);
            check(lib.sfnorm(sf.data_ptr(), filter.data_ptr(), B, p.k, (int)sf.size(2), (int)sf.size(3), dtc, p.scale,
                             stream));
        }
        Tensor gx, gcf, gsf, ws;
        if (need_x) gx = empty_like_on(x.sizes(), dt, dev);
        if (need_cf) gcf = empty_like_on(cf.sizes(), dt, dev);
        if (need_sf) gsf = empty_like_on(sf.sizes(), dt, dev);
        const size_t bytes = lib.backward_workspace(B, C, H, W, p.k, p.d, p.s, p.combine, dtc, variant);
        if (bytes) ws = empty_like_on({(int64_t)bytes}, at::kByte, dev);
        check(lib.backward(go.data_ptr(), x.data_ptr(), cf.data_ptr(), filter.data_ptr(), ptr(gx), ptr(gcf), ptr(gsf),
                           ptr(ws), bytes, B, C, H, W, p.k, p.d, p.s, p.combine, dtc, variant, stream));
        if (p.norm && need_sf) {  // ... and the filter gradient carried back through the normalisation
            Tensor raw = empty_like_on(sf.sizes(), dt, dev);
            check(lib.sfnorm_backward(sf.data_ptr(), gsf.data_ptr(), raw.data_ptr(), B, p.k, (int)sf.size(2),
                                      (int)sf.size(3), dtc, p.scale, stream));
            gsf = raw;
        }
        if (need_x) out[0] = types[0] == dt ? gx : gx.to(types[0]);
        if (need_cf) out[1] = types[1] == dt ? gcf : gcf.to(types[1]);
        if (need_sf) out[2] = types[2] == dt ? gsf : gsf.to(types[2]);
        return out;
    }

    Params p;
    at::ScalarType types[3];  // of the inputs as given: 2-byte and float inputs may be mixed
    torch::autograd::SavedVariable x_, cf_, sf_;
    bool released = false;
};

// ------------------------------------------------------------------ forward
bool plain_int(PyObject* o, int& v) {
    long n = -1;
    if (PyLong_CheckExact(o)) {
        n = PyLong_AsLong(o);
    } else if (PyObject* i = PyNumber_Index(o)) {
        n = PyLong_AsLong(i);
        Py_DECREF(i);
    }
    if (PyErr_Occurred()) { PyErr_Clear(); return false; }
    if (n < 1 || n > (1 << 20)) return false;
    v = (int)n;
    return true;
}

bool text_is(PyObject* o, const char* s) { return PyUnicode_Check(o) && PyUnicode_CompareWithASCIIString(o, s) == 0; }

// The reference's argument checks (ddf/ddf.py:32-65); false: `general` finds out which one failed.
bool parse(PyObject* const* args, Py_ssize_t n, bool norm, Params& p, const Tensor*& x, const Tensor*& cf,
           const Tensor*& sf, at::ScalarType& dt) {
    if (n < 3 || n > (norm ? 9 : 8)) return false;
    for (int i = 0; i < 3; ++i)
        if (!THPVariable_Check(args[i])) return false;
    x = &THPVariable_Unpack(args[0]);
    cf = &THPVariable_Unpack(args[1]);
    sf = &THPVariable_Unpack(args[2]);
    p.norm = norm;
    if (n > 3 && !plain_int(args[3], p.k)) return false;
    if (n > 4 && !plain_int(args[4], p.d)) return false;
    if (n > 5 && !plain_int(args[5], p.s)) return false;
    if (n > 6) {
        if (text_is(args[6], "mul")) p.combine = DDF_B200_MUL;
        else if (text_is(args[6], "add")) p.combine = DDF_B200_ADD;
        else return false;
    }
    const int at_version = norm ? 8 : 7;
    if (norm && n > 7) {
        p.scale = PyFloat_AsDouble(args[7]);
        if (p.scale == -1.0 && PyErr_Occurred()) { PyErr_Clear(); return false; }
    }
    if (n > at_version) {
        if (text_is(args[at_version], "")) p.variant = DDF_B200_VARIANT_AUTO;
        else if (text_is(args[at_version], "o")) p.variant = DDF_B200_VARIANT_GENERIC;
        else if (text_is(args[at_version], "f")) p.variant = DDF_B200_VARIANT_STREAM;
        else return false;
    }
    if (p.k % 2 != 1 || (norm && p.k < 3)) return false;
    if (!x->is_cuda() || cf->device() != x->device() || sf->device() != x->device()) return false;
    if (x->dim() != 4 || cf->dim() != 4 || sf->dim() != 4) return false;
    const auto xs = x->sizes(), cs = cf->sizes(), ss = sf->sizes();
    if (cs[0] != xs[0] || cs[1] != xs[1] || cs[2] != p.k || cs[3] != p.k) return false;
    if (ss[0] != xs[0] || ss[1] != (int64_t)p.k * p.k || ss[2] != xs[2] / p.s || ss[3] != xs[3] / p.s) return false;
    for (int i = 0; i < 4; ++i)
        if (xs[i] > INT32_MAX) return false;
    if (!x->is_contiguous() || !cf->is_contiguous() || !sf->is_contiguous()) return false;
    dt = x->scalar_type();
    if (cf->scalar_type() != dt || sf->scalar_type() != dt)
        dt = at::promoteTypes(at::promoteTypes(dt, cf->scalar_type()), sf->scalar_type());
    return dtype_code(dt) >= 0;
}

// Nothing watches or transforms the program (see the head of this file).
bool ordinary(std::initializer_list<const Tensor*> tensors) {
    using c10::DispatchKey;
    // set while a thread traces, has a dispatch mode, is inside a functorch transform
    constexpr c10::DispatchKeySet watching({DispatchKey::Tracer, DispatchKey::Python,
                                            DispatchKey::FuncTorchDynamicLayerFrontMode});
    if (c10::impl::tls_local_dispatch_key_set().included_.has_any(watching)) return false;
    for (const Tensor* t : tensors)  // wrappers hold no storage of their own
        if (!t->has_storage() || torch::autograd::isFwGradDefined(*t)) return false;
    return true;
}

// Loads and binds the library on the first call; false: a Python error is set.
bool loaded() {
    if (C10_LIKELY(lib.forward != nullptr)) return true;
    PyObject* r = PyObject_CallNoArgs(g_load);
    Py_XDECREF(r);
    return r != nullptr;
}

PyObject* call(PyObject* const* args, Py_ssize_t n, bool norm) {
    HANDLE_TH_ERRORS
    Params p;
    const Tensor *x, *cf, *sf;
    at::ScalarType dt;
    if (!parse(args, n, norm, p, x, cf, sf, dt) || !ordinary({x, cf, sf})) {
        PyObject* list = PyTuple_New(n + 1);
        if (!list) return nullptr;
        PyTuple_SET_ITEM(list, 0, PyBool_FromLong(norm));
        for (Py_ssize_t i = 0; i < n; ++i) PyTuple_SET_ITEM(list, i + 1, Py_NewRef(args[i]));
        PyObject* r = PyObject_CallObject(g_general, list);
        Py_DECREF(list);
        return r;
    }
    if (!loaded()) return nullptr;
    const bool grad = at::GradMode::is_enabled() && (x->requires_grad() || cf->requires_grad() || sf->requires_grad());
    // the range that a profiler shows for an autograd function's forward
    at::RecordFunction range(at::RecordScope::FUNCTION);
    if (C10_UNLIKELY(range.isActive())) {
        const char* name = norm ? "DDFSpatialNormFunction" : "DDFFunction";
        const c10::IValue inputs[] = {*x, *cf, *sf};
        if (range.needsInputs())
            range.before(name, c10::ArrayRef<const c10::IValue>(inputs), at::sequence_number::peek());
        else
            range.before(name, at::sequence_number::peek());
    }
    Tensor out;
    {
        pybind11::gil_scoped_release no_gil;
        Tensor kept[3];
        auto as_type = [&](const Tensor* t, int i) -> const Tensor* {
            if (t->scalar_type() == dt) return t;
            at::NoGradGuard no_grad;
            kept[i] = t->to(dt);
            return &kept[i];
        };
        const Tensor *xd = as_type(x, 0), *cfd = as_type(cf, 1), *sfd = as_type(sf, 2);
        const int B = (int)x->size(0), C = (int)x->size(1), H = (int)x->size(2), W = (int)x->size(3);
        const at::Device dev = x->device();
        c10::cuda::CUDAGuard guard(dev);
        void* stream = c10::cuda::getCurrentCUDAStream(dev.index()).stream();
        out = empty_like_on({B, C, H / p.s, W / p.s}, dt, dev);
        check(norm ? lib.forward_sfnorm(xd->data_ptr(), cfd->data_ptr(), sfd->data_ptr(), out.data_ptr(), B, C, H, W,
                                        p.k, p.d, p.s, p.combine, dtype_code(dt), p.variant, p.scale, stream)
                   : lib.forward(xd->data_ptr(), cfd->data_ptr(), sfd->data_ptr(), out.data_ptr(), B, C, H, W, p.k,
                                 p.d, p.s, p.combine, dtype_code(dt), p.variant, stream));
        if (grad) {
            std::shared_ptr<DDFBackward> node(new DDFBackward(), torch::autograd::deleteNode);
            node->set_next_edges(torch::autograd::collect_next_edges(*x, *cf, *sf));
            node->p = p;
            node->types[0] = x->scalar_type();
            node->types[1] = cf->scalar_type();
            node->types[2] = sf->scalar_type();
            node->x_ = torch::autograd::SavedVariable(*xd, false);
            node->cf_ = torch::autograd::SavedVariable(*cfd, false);
            node->sf_ = torch::autograd::SavedVariable(*sfd, false);
            torch::autograd::set_history(out, node);
        }
    }
    return THPVariable_Wrap(std::move(out));
    END_HANDLE_TH_ERRORS
}

PyObject* py_ddf(PyObject*, PyObject* const* args, Py_ssize_t n) { return call(args, n, false); }
PyObject* py_ddf_sfnorm(PyObject*, PyObject* const* args, Py_ssize_t n) { return call(args, n, true); }

// stem_maxpool(x): the stem's 3 x 3 / stride 2 pooling of a plain channels_last CUDA tensor that records no
// gradient; None where torch's has to be taken.  Host time 5.8 us (as Python and ctypes 18.5; torch's own
// operator 11), and the call is the faster one at the smallest size too, so there is no lower limit:
// (1,64,80x80) f16 8.2 us against 22, f32 10.2 against 20.5, (16,64,112x112) f16 10.3 against 57.
PyObject* py_stem_maxpool(PyObject*, PyObject* arg) {
    HANDLE_TH_ERRORS
    if (!THPVariable_CheckExact(arg)) Py_RETURN_NONE;
    const Tensor& x = THPVariable_Unpack(arg);
    const int dtc = x.is_cuda() ? dtype_code(x.scalar_type()) : -1;
    if (dtc < 0 || dtc == DDF_B200_F64 || x.dim() != 4 || (at::GradMode::is_enabled() && x.requires_grad()) ||
        !ordinary({&x}))
        Py_RETURN_NONE;
    const auto s = x.sizes();
    if (x.numel() == 0 || s[0] > INT32_MAX || s[1] > INT32_MAX || s[2] * s[3] > (1ll << 30) ||
        s[1] * (int64_t)x.element_size() % 16 != 0 || reinterpret_cast<uintptr_t>(x.data_ptr()) % 16 != 0 ||
        !x.is_contiguous(at::MemoryFormat::ChannelsLast) || x.is_contiguous())
        Py_RETURN_NONE;
    if (!loaded()) return nullptr;
    Tensor out;
    {
        pybind11::gil_scoped_release no_gil;
        const at::Device dev = x.device();
        c10::cuda::CUDAGuard guard(dev);
        out = at::detail::empty_cuda({s[0], s[1], (s[2] - 1) / 2 + 1, (s[3] - 1) / 2 + 1}, x.scalar_type(), dev,
                                     at::MemoryFormat::ChannelsLast);
        check(lib.maxpool_nhwc(x.data_ptr(), out.data_ptr(), (int)s[0], (int)s[1], (int)s[2], (int)s[3], dtc,
                               c10::cuda::getCurrentCUDAStream(dev.index()).stream()));
    }
    return THPVariable_Wrap(std::move(out));
    END_HANDLE_TH_ERRORS
}

// hooks(error_class, general, load): the Python side's callables, set when the package is imported.
PyObject* py_hooks(PyObject*, PyObject* args) {
    PyObject *e, *x, *l;
    if (!PyArg_ParseTuple(args, "OOO", &e, &x, &l)) return nullptr;
    Py_XSETREF(g_error_class, Py_NewRef(e));
    Py_XSETREF(g_general, Py_NewRef(x));
    Py_XSETREF(g_load, Py_NewRef(l));
    Py_RETURN_NONE;
}

// bind(addresses, debug): addresses of the library's entry points by name.
PyObject* py_bind(PyObject*, PyObject* args) {
    PyObject* d;
    int debug;
    if (!PyArg_ParseTuple(args, "O!p", &PyDict_Type, &d, &debug)) return nullptr;
    Library l;
    auto get = [&](const char* name, auto& f) {
        PyObject* v = PyDict_GetItemString(d, name);
        f = reinterpret_cast<std::decay_t<decltype(f)>>(v ? PyLong_AsVoidPtr(v) : nullptr);
        return f != nullptr;
    };
    if (!get("ddf_b200_forward", l.forward) || !get("ddf_b200_forward_sfnorm", l.forward_sfnorm) ||
        !get("ddf_b200_backward_workspace", l.backward_workspace) || !get("ddf_b200_backward", l.backward) ||
        !get("ddf_b200_sfnorm", l.sfnorm) || !get("ddf_b200_sfnorm_backward", l.sfnorm_backward) ||
        !get("ddf_b200_take_fault", l.take_fault) || !get("ddf_b200_maxpool_nhwc", l.maxpool_nhwc)) {
        PyErr_SetString(PyExc_KeyError, "bind: an entry point is missing");
        return nullptr;
    }
    lib = l;
    g_debug = debug != 0;
    Py_RETURN_NONE;
}

PyMethodDef methods[] = {
    {"ddf", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_ddf)), METH_FASTCALL,
     "ddf(features, channel_filter, spatial_filter, kernel_size=3, dilation=1, stride=1, kernel_combine='mul', "
     "version='') -- positional only"},
    {"ddf_sfnorm", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_ddf_sfnorm)), METH_FASTCALL,
     "ddf_sfnorm(features, channel_filter, spatial_raw, kernel_size=3, dilation=1, stride=1, kernel_combine='mul', "
     "scale=1.0, version='') -- positional only"},
    {"stem_maxpool", py_stem_maxpool, METH_O, "stem_maxpool(x) -> the pooled tensor, or None"},
    {"hooks", py_hooks, METH_VARARGS, nullptr},
    {"bind", py_bind, METH_VARARGS, nullptr},
    {nullptr, nullptr, 0, nullptr}};

PyModuleDef module = {PyModuleDef_HEAD_INIT, "_native", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__native(void) { return PyModule_Create(&module); }
