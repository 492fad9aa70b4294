// The host side of QuantizedLinear's forward where no gradient is recorded, in one native call: checks, output
// allocation and bw_qmatmul on the current stream.  A decode step is launches of a few microseconds each, and in Python
// the autograd function (7.5 us), the checks, torch.empty and the foreign call took 21 us a layer.
//
// forward(x, qweight, scale, zero_point, bias, bits, group_size) returns the fp16 output, or None for every call that
// is not plain: the caller then goes through QuantizedLinearFunction, which converts, records, or raises.  Plain means
// exact torch tensors on the current CUDA device, contiguous and of their final types, no input that gradients are
// recorded for, no forward-mode tangent, and no tracing, dispatch or function mode and no function transform in force.
// The outcome depends on this call's arguments, torch's thread-local modes and the stream's scratch; nothing is kept.
#define PY_SSIZE_T_CLEAN
#include <ATen/ATen.h>
#include <ATen/PythonTorchFunctionTLS.h>
#include <Python.h>
#include <c10/core/GradMode.h>
#include <c10/core/impl/LocalDispatchKeySet.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAGraphsC10Utils.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/jit/frontend/tracer.h>
#include <torch/csrc/utils/pybind.h>

#include "bitween_b200.h"

namespace {

// The tensor of a Python argument; null unless it is exactly a torch tensor (or parameter).
const at::Tensor *tensor_of(PyObject *o) { return THPVariable_CheckExact(o) ? &THPVariable_Unpack(o) : nullptr; }

using QMatmul = int (*)(const void *, int, int64_t, int64_t, int64_t, const int32_t *, const void *, const void *, const void *,
                        void *, int, int, int, void *, size_t, void *);
QMatmul g_qmatmul = nullptr;      // of the library that the Python binding has loaded; set once, at import
PyObject *g_workspaces = nullptr; // the binding's dict (device index, stream handle) -> scratch tensor; kept by the binding too

// The stream's scratch, as the Python binding's current_workspace returns it; null inside a capture and before the
// binding has made one.  Called with the GIL held; the tensor stays in the dict, or is replaced by a larger one.
const at::Tensor *workspace_of(int device, cudaStream_t stream) {
    if (stream != nullptr && c10::cuda::currentStreamCaptureStatusMayInitCtx() != c10::cuda::CaptureStatus::None) return nullptr;
    PyObject *key = Py_BuildValue("(iK)", device, (unsigned long long)reinterpret_cast<uintptr_t>(stream));
    if (!key) { PyErr_Clear(); return nullptr; }
    PyObject *t = PyDict_GetItemWithError(g_workspaces, key);       // borrowed
    Py_DECREF(key);
    if (!t) { PyErr_Clear(); return nullptr; }
    return tensor_of(t);
}

// A plain tensor: strided, on `device`, contiguous, without tangents or lazy views, and of no interest to autograd.
bool plain(const at::Tensor &t, const c10::Device &device, bool recording) {
    if (!t.defined() || t.layout() != c10::kStrided || !t.is_cuda() || t.device() != device || !t.is_contiguous()) return false;
    if (t.is_neg() || t._is_zerotensor() || t.key_set().has(c10::DispatchKey::Python)) return false;
    if (recording && t.requires_grad()) return false;
    return !t._fw_grad(/*level=*/0).defined();
}

bool modes_active() {
    return c10::impl::TorchDispatchModeTLS::any_modes_set() || at::impl::torch_function_mode_enabled() || torch::jit::tracer::isTracing() ||
           c10::impl::tls_is_dispatch_key_included(c10::DispatchKey::FuncTorchDynamicLayerFrontMode);
}

PyObject *forward(PyObject *, PyObject *const *args, Py_ssize_t nargs) {
    HANDLE_TH_ERRORS
    if (nargs != 7) {
        PyErr_SetString(PyExc_TypeError, "forward(x, qweight, scale, zero_point, bias, bits, group_size)");
        return nullptr;
    }
    const at::Tensor *x = tensor_of(args[0]), *q = tensor_of(args[1]), *s = tensor_of(args[2]), *z = tensor_of(args[3]), *b = nullptr;
    if (!x || !q || !s || !z || !g_qmatmul || !PyLong_CheckExact(args[5]) || !PyLong_CheckExact(args[6])) Py_RETURN_NONE;
    if (args[4] != Py_None && !(b = tensor_of(args[4]))) Py_RETURN_NONE;
    const long bits = PyLong_AsLong(args[5]), group = PyLong_AsLong(args[6]);
    if (PyErr_Occurred()) { PyErr_Clear(); Py_RETURN_NONE; }
    if ((bits != 2 && bits != 4 && bits != 8) || group < 1 || group > 1 << 30 || modes_active()) Py_RETURN_NONE;

    const c10::Device device = x->device();
    if (!device.is_cuda() || device.index() != c10::cuda::current_device()) Py_RETURN_NONE;
    const bool recording = c10::GradMode::is_enabled();
    if (!plain(*x, device, recording) || !plain(*q, device, recording) || !plain(*s, device, recording) || !plain(*z, device, recording) ||
        (b && !plain(*b, device, recording)))
        Py_RETURN_NONE;
    const auto xt = x->scalar_type();
    const int x_code = xt == at::kHalf ? BW_F16 : xt == at::kBFloat16 ? BW_BF16 : xt == at::kFloat ? BW_F32 : -1;
    if (x_code < 0 || q->scalar_type() != at::kInt || s->scalar_type() != at::kHalf || z->scalar_type() != at::kHalf) Py_RETURN_NONE;
    if (x->dim() < 1 || q->dim() != 2 || s->dim() != 2 || z->dim() != 2) Py_RETURN_NONE;
    const int64_t K = x->size(-1), N = q->size(0);
    if (K < 1 || N < 1 || x->numel() < 1 || q->size(1) * (32 / bits) != K || K % group) Py_RETURN_NONE;
    if (s->size(0) != N || s->size(1) != K / group || z->size(0) != N || z->size(1) != K / group) Py_RETURN_NONE;
    if (b && (b->scalar_type() != at::kHalf || b->numel() != N)) Py_RETURN_NONE;

    const int64_t M = x->numel() / K;
    const cudaStream_t stream = c10::cuda::getCurrentCUDAStream(device.index()).stream();
    const at::Tensor *ws = workspace_of(device.index(), stream);
    // (9 to 32 tokens would run without scratch, on a slower kernel)
    if (M > 8 && M <= 32 && (!ws || ws->numel() < 64 * (K + 256))) Py_RETURN_NONE;
    const at::Tensor scratch = ws ? *ws : at::Tensor();              // (held: another thread may replace it in the dict)
    at::Tensor out;
    int rc;
    {
        pybind11::gil_scoped_release no_gil;
        c10::SmallVector<int64_t, 5> sizes(x->sizes().begin(), x->sizes().end());
        sizes.back() = N;
        out = at::empty(sizes, at::TensorOptions().dtype(at::kHalf).device(device));
        rc = g_qmatmul(x->const_data_ptr(), x_code, M, N, K, static_cast<const int32_t *>(q->const_data_ptr()),
                       s->const_data_ptr(), z->const_data_ptr(), b ? b->const_data_ptr() : nullptr, out.mutable_data_ptr(), BW_F16,
                       (int)bits, (int)group, scratch.defined() ? scratch.mutable_data_ptr() : nullptr,
                       scratch.defined() ? (size_t)scratch.numel() : 0, stream);
    }
    // (a kernel that needs more scratch, or an error: nothing has been launched, the Python path supplies it or raises)
    if (rc != BW_OK) Py_RETURN_NONE;
    return THPVariable_Wrap(std::move(out));
    END_HANDLE_TH_ERRORS
}

// set_entry(address of bw_qmatmul, the binding's dict of workspaces)
PyObject *set_entry(PyObject *, PyObject *const *args, Py_ssize_t nargs) {
    if (nargs != 2 || !PyDict_CheckExact(args[1])) {
        PyErr_SetString(PyExc_TypeError, "set_entry(address, workspaces)");
        return nullptr;
    }
    void *p = PyLong_AsVoidPtr(args[0]);
    if (!p && PyErr_Occurred()) return nullptr;
    Py_INCREF(args[1]);
    Py_XSETREF(g_workspaces, args[1]);
    g_qmatmul = reinterpret_cast<QMatmul>(p);
    Py_RETURN_NONE;
}

PyMethodDef methods[] = {
    {"forward", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(forward)), METH_FASTCALL, nullptr},
    {"set_entry", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(set_entry)), METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr},
};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_host_forward", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__host_forward() { return PyModule_Create(&module); }
