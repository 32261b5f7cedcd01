// Autograd nodes of the training path in native code: one node per LogicLayer and one for GroupSum.
//
// What a training step of a small network costs is the host: a Python autograd function with its views, checks and ctypes calls took
// 40 us forward and 60 us backward per layer, for kernels of 3 to 10 us.  These nodes do the same -- same kernels, same
// launches, same saved tensors -- without the interpreter: a step of 784 -> 4 x 8000, batch 100, in a plain loop
// 626 -> 340 us (forward 206 -> 102, backward 312 -> 164; what is left is mostly PyTorch's modules, loss, engine and optimizer hooks).
//
// A call that does not have the ordinary form returns None, and the Python functions of difflogic.py take it, with their checks and
// messages: other tensor types, dtypes and layouts, functorch transforms, tensor and function modes, forward mode, tracing.  So does a
// backward pass that has more to do than the layer's gradients (an optimizer that steps inside it, an exchange between GPUs,
// backward_w on a stream of its own): those are asked for when it runs, since they may be switched on after the forward pass.
#include <Python.h>

#include <ATen/PythonTorchFunctionTLS.h>
#include <ATen/core/Tensor.h>
#include <ATen/ops/empty.h>
#include <ATen/ops/empty_strided.h>
#include <c10/core/impl/LocalDispatchKeySet.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/custom_function.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/jit/frontend/tracer.h>
#include <torch/csrc/utils/object_ptr.h>

#include <atomic>

#include "difflogic_b200.h"

namespace {

using at::Tensor;
using torch::autograd::AutogradContext;
using torch::autograd::variable_list;

struct WithGil {  // for the engine's threads
    PyGILState_STATE state = PyGILState_Ensure();
    ~WithGil() { PyGILState_Release(state); }
};
struct WithoutGil {
    PyThreadState *state = PyEval_SaveThread();
    ~WithoutGil() { PyEval_RestoreThread(state); }
};

std::atomic<long long> g_launches{0};  // kernels launched from here, as _native.launch_count() counts
PyObject *g_module_dict = nullptr;     // difflogic.py's: `_backward_w_stream` and `_backward_of_node`

void check(int status) {
    TORCH_CHECK(status == DL_OK, "difflogic_b200 (status ", status, "): ", dl_last_error_string());
    ++g_launches;
}

bool ordinary(PyObject *o) { return THPVariable_CheckExact(o); }
bool plain(const Tensor &t, at::ScalarType type, int64_t dim, const c10::Device &device) {
    return t.defined() && t.layout() == at::kStrided && t.is_cuda() && t.device() == device && t.scalar_type() == type && t.dim() == dim;
}
bool vector_of(const Tensor &t, at::ScalarType type, int64_t n, const c10::Device &device) {
    return plain(t, type, 1, device) && t.size(0) == n && t.is_contiguous();
}
bool matrix_of(const Tensor &t, at::ScalarType type, int64_t rows, int64_t cols, const c10::Device &device) {
    return plain(t, type, 2, device) && t.size(0) == rows && t.size(1) == cols && t.is_contiguous();
}
// Whether something wants to see every operation, which these nodes would pass by.
bool observed() {
    return c10::impl::tls_is_dispatch_key_included(at::DispatchKey::FuncTorchDynamicLayerFrontMode) || c10::impl::TorchDispatchModeTLS::any_modes_set() ||
           at::impl::torch_function_mode_enabled() || torch::jit::tracer::isTracing();
}
bool aligned16(const Tensor &t) { return reinterpret_cast<uintptr_t>(t.data_ptr()) % 16 == 0; }
void *stream_of(const Tensor &t) { return c10::cuda::getCurrentCUDAStream(t.device().index()).stream(); }
// A [batch][features] tensor as it is stored between layers: feature-major, and no view.
Tensor feature_major(int64_t batch, int64_t features, const Tensor &like) {
    return at::empty_strided({batch, features}, {1, batch}, like.options().requires_grad(false));
}

struct Layer {
    Tensor a, b, start, plan, grad_out, walk;  // grad_out, walk: may be undefined
    double grad_factor;
    bool complete;
    bool transposed;  // x is batch-major: the library transposes it
};

PyObject *wrap(const Tensor &t) {
    if (t.defined()) return THPVariable_Wrap(t);
    Py_RETURN_NONE;
}

struct LayerNode : torch::autograd::Function<LayerNode> {
    static Tensor forward(AutogradContext *ctx, const Tensor &input, const Tensor &weights, const Layer &l) {
        const int64_t batch = input.size(0), n_in = input.size(1), n_out = weights.size(0);
        Tensor x = input.t();
        void *stream = stream_of(input);
        if (l.transposed) {
            x = at::empty({n_in, batch}, input.options().requires_grad(false));
            check(dl_transpose_f32(input.data_ptr<float>(), x.data_ptr<float>(), batch, n_in, stream));
        } else if (!x.is_contiguous()) {
            x = x.contiguous();
        }
        Tensor y = feature_major(batch, n_out, input), coef = at::empty({n_out, 4}, input.options().requires_grad(false));
        if (l.walk.defined())
            check(dl_forward_walk_f32(x.data_ptr<float>(), weights.data_ptr<float>(), DL_W_LOGITS, y.data_ptr<float>(), coef.data_ptr<float>(),
                                      l.walk.data_ptr<int32_t>(), l.walk.size(0), n_in, n_out, batch, DL_LAUNCH_OVERLAP_SETUP, stream));
        else
            check(dl_forward_f32(x.data_ptr<float>(), l.a.data_ptr<int64_t>(), l.b.data_ptr<int64_t>(), weights.data_ptr<float>(), DL_W_LOGITS,
                                 y.data_ptr<float>(), coef.data_ptr<float>(), n_in, n_out, batch, DL_LAUNCH_OVERLAP_SETUP, stream));
        ctx->save_for_backward({x, weights, l.a, l.b, l.start, l.plan, coef});
        ctx->saved_data["grad_factor"] = l.grad_factor;
        ctx->saved_data["complete"] = l.complete;
        if (l.grad_out.defined()) ctx->saved_data["grad_out"] = l.grad_out;
        if (l.walk.defined()) ctx->saved_data["walk"] = l.walk;
        return y;
    }

    // Whether the weights' gradient is somebody's business beside autograd's, or a stream is set for it.
    static bool managed(const Tensor &weights) {
        PyObject *stream = PyDict_GetItemString(g_module_dict, "_backward_w_stream");
        if (stream != nullptr && stream != Py_None) return true;
        PyObject *w = THPVariable_Wrap(weights);
        if (w == nullptr) throw python_error();
        PyObject *dict = PyObject_GenericGetDict(w, nullptr);
        const bool found = dict != nullptr && (PyDict_GetItemString(dict, "_dl_adam") != nullptr || PyDict_GetItemString(dict, "_dl_exchange") != nullptr);
        if (dict == nullptr) PyErr_Clear();
        Py_XDECREF(dict);
        Py_DECREF(w);
        return found;
    }

    static variable_list in_python(AutogradContext *ctx, const variable_list &saved, const Tensor &grad_y, const Tensor &grad_out, const Tensor &walk,
                                   bool want_x, bool want_w) {
        PyObject *run = PyDict_GetItemString(g_module_dict, "_backward_of_node");
        TORCH_CHECK(run != nullptr, "difflogic_b200: difflogic._backward_of_node is missing");
        THPObjectPtr args(PyTuple_New(13));
        if (!args) throw python_error();
        for (int i = 0; i < 7; ++i) PyTuple_SET_ITEM(args.get(), i, wrap(saved[i]));
        PyTuple_SET_ITEM(args.get(), 7, wrap(grad_y));
        PyTuple_SET_ITEM(args.get(), 8, PyFloat_FromDouble(ctx->saved_data["grad_factor"].toDouble()));
        PyTuple_SET_ITEM(args.get(), 9, wrap(grad_out));
        PyTuple_SET_ITEM(args.get(), 10, walk.defined() ? Py_BuildValue("(NO)", wrap(walk), ctx->saved_data["complete"].toBool() ? Py_True : Py_False)
                                                       : Py_NewRef(Py_None));
        PyTuple_SET_ITEM(args.get(), 11, PyBool_FromLong(want_x));
        PyTuple_SET_ITEM(args.get(), 12, PyBool_FromLong(want_w));
        THPObjectPtr got(PyObject_CallObject(run, args.get()));
        if (!got) throw python_error();
        variable_list out(3);
        for (int i = 0; i < 2; ++i) {
            PyObject *t = PyTuple_GET_ITEM(got.get(), i);
            if (t != Py_None) out[i] = THPVariable_Unpack(t);
        }
        return out;
    }

    static variable_list backward(AutogradContext *ctx, variable_list grads) {
        const bool want_x = ctx->needs_input_grad(0), want_w = ctx->needs_input_grad(1);
        const variable_list saved = ctx->get_saved_variables();
        const Tensor &x = saved[0], &weights = saved[1], &start = saved[4], &plan = saved[5], &coef = saved[6];
        const int64_t n_in = x.size(0), batch = x.size(1), n_out = weights.size(0);
        auto kept = [&](const char *name) {
            auto it = ctx->saved_data.find(name);
            return it == ctx->saved_data.end() ? Tensor() : it->second.toTensor();
        };
        const Tensor grad_out = kept("grad_out"), walk = kept("walk");
        const c10::cuda::CUDAGuard guard(x.device());
        Tensor gy = grads[0].t();
        if (!gy.is_contiguous()) gy = gy.contiguous();
        variable_list out(3);
        {
            const WithGil gil;
            if (managed(weights)) {
                out = in_python(ctx, saved, gy, grad_out, walk, want_x, want_w);
                if (out[0].defined()) out[0] = out[0].t();
                return out;
            }
        }
        // what the hooks for saved tensors handed back, and the gradient, are what the kernels take
        const c10::Device device = x.device();
        TORCH_CHECK(matrix_of(x, at::kFloat, n_in, batch, device) && matrix_of(weights, at::kFloat, n_out, 16, device) &&
                        matrix_of(coef, at::kFloat, n_out, 4, device) && matrix_of(gy, at::kFloat, n_out, batch, device) &&
                        vector_of(saved[2], at::kLong, n_out, device) && vector_of(saved[3], at::kLong, n_out, device) &&
                        vector_of(start, at::kLong, n_in + 1, device) && matrix_of(plan, at::kInt, 2 * n_out, 2, device),
                    "difflogic_b200: the backward pass of a LogicLayer got tensors of other types, sizes or layouts than its forward pass");
        const float *xp = x.data_ptr<float>(), *gp = gy.data_ptr<float>(), *cp = coef.data_ptr<float>();
        const float scale = (float)ctx->saved_data["grad_factor"].toDouble();
        void *stream = stream_of(x);
        Tensor gx, gw;
        if (want_x) gx = at::empty({n_in, batch}, x.options().requires_grad(false));
        if (want_w) gw = grad_out.defined() ? grad_out.view(grad_out.sizes()) : at::empty({n_out, 16}, x.options().requires_grad(false));
        float *gxp = want_x ? gx.data_ptr<float>() : nullptr, *gwp = want_w ? gw.data_ptr<float>() : nullptr;
        if (walk.defined() && want_w && (!want_x || ctx->saved_data["complete"].toBool()) && aligned16(weights) && aligned16(gw)) {
            check(dl_backward_walk_f32(xp, gp, cp, weights.data_ptr<float>(), gwp, gxp, scale, walk.data_ptr<int32_t>(), walk.size(0),
                                       ctx->saved_data["complete"].toBool() ? 1 : 0, n_in, n_out, batch, 1, nullptr, nullptr, 0.f, 0.f, 0.f, 0.f, 1.f,
                                       nullptr, DL_LAUNCH_OVERLAP_SETUP, stream));
        } else {
            if (want_x)
                check(dl_backward_x_f32(xp, cp, gp, start.data_ptr<int64_t>(), plan.data_ptr<int32_t>(), scale, gxp, n_in, n_out, batch,
                                        DL_LAUNCH_OVERLAP_SETUP, stream));
            if (want_w)
                check(dl_backward_w_f32(xp, saved[2].data_ptr<int64_t>(), saved[3].data_ptr<int64_t>(), gp, weights.data_ptr<float>(), DL_W_LOGITS, gwp,
                                        n_in, n_out, batch, DL_LAUNCH_OVERLAP_SETUP, stream));
        }
        if (want_x) out[0] = gx.t();
        if (want_w) out[1] = gw;
        return out;
    }
};

struct GroupSumNode : torch::autograd::Function<GroupSumNode> {
    static Tensor forward(AutogradContext *ctx, const Tensor &input, const Tensor &workspace, int64_t k, double tau) {
        const int64_t batch = input.size(0), n = input.size(1);
        Tensor x = input.t();
        if (!x.is_contiguous()) x = x.contiguous();
        Tensor out = at::empty({batch, k}, input.options().requires_grad(false));
        check(dl_groupsum_f32(x.data_ptr<float>(), out.data_ptr<float>(), workspace.data_ptr(), n, batch, k, (float)tau, stream_of(input)));
        ctx->saved_data["n"] = n;
        ctx->saved_data["tau"] = tau;
        return out;
    }

    static variable_list backward(AutogradContext *ctx, variable_list grads) {
        const Tensor grad = grads[0].contiguous();
        const int64_t n = ctx->saved_data["n"].toInt(), batch = grad.size(0), k = grad.size(1);
        TORCH_CHECK(matrix_of(grad, at::kFloat, batch, k, grad.device()), "difflogic_b200: the gradient of a GroupSum must be float32 on a CUDA device");
        const c10::cuda::CUDAGuard guard(grad.device());
        Tensor gx = at::empty({n, batch}, grad.options().requires_grad(false));
        check(dl_groupsum_backward_f32(grad.data_ptr<float>(), gx.data_ptr<float>(), n, batch, k, (float)ctx->saved_data["tau"].toDouble(), stream_of(grad)));
        return {gx.t(), Tensor(), Tensor(), Tensor()};
    }
};

// layer(x, weights, a, b, start, plan, grad_factor, grad_out | None, walk entries | None, walk gives grad_x) -> output, or None
PyObject *layer(PyObject *, PyObject *const *args, Py_ssize_t count) {
    HANDLE_TH_ERRORS
    if (count != 10) {
        PyErr_SetString(PyExc_TypeError, "layer: ten arguments");
        return nullptr;
    }
    for (int i = 0; i < 6; ++i)
        if (!ordinary(args[i])) Py_RETURN_NONE;
    const Tensor &x = THPVariable_Unpack(args[0]), &w = THPVariable_Unpack(args[1]);
    const c10::Device device = x.device();
    if (!plain(x, at::kFloat, 2, device) || x.size(0) == 0 || x.size(1) == 0 || w.dim() != 2 || w.size(0) == 0 ||
        !matrix_of(w, at::kFloat, w.size(0), 16, device))
        Py_RETURN_NONE;
    const int64_t n_in = x.size(1), n_out = w.size(0);
    Layer l = {THPVariable_Unpack(args[2]), THPVariable_Unpack(args[3]), THPVariable_Unpack(args[4]), THPVariable_Unpack(args[5])};
    if (!vector_of(l.a, at::kLong, n_out, device) || !vector_of(l.b, at::kLong, n_out, device) || !vector_of(l.start, at::kLong, n_in + 1, device) ||
        !matrix_of(l.plan, at::kInt, 2 * n_out, 2, device))
        Py_RETURN_NONE;
    l.grad_factor = PyFloat_AsDouble(args[6]);
    if (l.grad_factor == -1. && PyErr_Occurred()) return nullptr;
    if (args[7] != Py_None) {
        if (!ordinary(args[7])) Py_RETURN_NONE;
        l.grad_out = THPVariable_Unpack(args[7]);
        if (!matrix_of(l.grad_out, at::kFloat, n_out, 16, device)) Py_RETURN_NONE;
    }
    if (args[8] != Py_None) {
        if (!ordinary(args[8])) Py_RETURN_NONE;
        l.walk = THPVariable_Unpack(args[8]);
        if (!matrix_of(l.walk, at::kInt, l.walk.size(0), 2, device)) Py_RETURN_NONE;
    }
    l.complete = args[9] == Py_True;
    if (observed() || x._fw_grad(0).defined() || w._fw_grad(0).defined()) Py_RETURN_NONE;
    l.transposed = !x.t().is_contiguous() && x.is_contiguous();
    Tensor y;
    {
        const WithoutGil nogil;
        const c10::cuda::CUDAGuard guard(device);
        y = LayerNode::apply(x, w, l);
    }
    return THPVariable_Wrap(y);
    END_HANDLE_TH_ERRORS
}

// group_sum(x, workspace, k, tau) -> output, or None
PyObject *group_sum(PyObject *, PyObject *const *args, Py_ssize_t count) {
    HANDLE_TH_ERRORS
    if (count != 4) {
        PyErr_SetString(PyExc_TypeError, "group_sum: four arguments");
        return nullptr;
    }
    if (!ordinary(args[0]) || !ordinary(args[1])) Py_RETURN_NONE;
    const Tensor &x = THPVariable_Unpack(args[0]), &workspace = THPVariable_Unpack(args[1]);
    const long long k = PyLong_AsLongLong(args[2]);
    const double tau = PyFloat_AsDouble(args[3]);
    if (PyErr_Occurred()) return nullptr;
    if (!plain(x, at::kFloat, 2, x.device()) || x.numel() == 0 || k <= 0 || x.size(1) % k != 0 || observed() || x._fw_grad(0).defined()) Py_RETURN_NONE;
    Tensor y;
    {
        const WithoutGil nogil;
        const c10::cuda::CUDAGuard guard(x.device());
        y = GroupSumNode::apply(x, workspace, (int64_t)k, tau);
    }
    return THPVariable_Wrap(y);
    END_HANDLE_TH_ERRORS
}

PyObject *launches(PyObject *, PyObject *) { return PyLong_FromLongLong(g_launches.load()); }

// connect(dict of difflogic.py)
PyObject *connect(PyObject *, PyObject *dict) {
    if (!PyDict_Check(dict)) {
        PyErr_SetString(PyExc_TypeError, "connect: a dict");
        return nullptr;
    }
    Py_XDECREF(g_module_dict);
    g_module_dict = Py_NewRef(dict);
    Py_RETURN_NONE;
}

PyMethodDef kMethods[] = {{"layer", (PyCFunction)(void *)layer, METH_FASTCALL, nullptr},
                          {"group_sum", (PyCFunction)(void *)group_sum, METH_FASTCALL, nullptr},
                          {"launches", launches, METH_NOARGS, nullptr},
                          {"connect", connect, METH_O, nullptr},
                          {nullptr, nullptr, 0, nullptr}};
PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "dl_autograd", nullptr, -1, kMethods};

}  // namespace

extern "C" __attribute__((visibility("default"))) PyObject *PyInit_dl_autograd(void) { return PyModule_Create(&kModule); }
