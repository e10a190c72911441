// The common form of three operators of flexllm_b200/ops.py without the interpreter's share of a call: tensors are checked, outputs allocated and the
// library's entry point called here. With ctypes a call of the linear layer took 9.2 us of host time, of which the launch is 3.4
// (torch.empty from Python 2.4, five pointers 0.9, the foreign call 0.9), longer than its kernel at 128 x 2048 x 2048, and the MLP block
// of one token 20 us for 14 us of kernels.
//
// Each function returns the output tensor, a status other than 0 as an integer, or None where the arguments are not plain contiguous CUDA
// tensors of the expected types: the caller then takes its general path, which decides what to do with them. The entry points are
// handed over as addresses (bind), so that the library that is called is the one that Python has loaded.
#include <Python.h>

#include <ATen/PythonTorchFunctionTLS.h>
#include <ATen/TensorSubclassLikeUtils.h>
#include <ATen/core/Tensor.h>
#include <ATen/ops/empty.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include "../../include/flexllm_b200.h"

namespace {

decltype(&flexllm_linear_prefill_i8) g_prefill = nullptr;
decltype(&flexllm_linear_decode_i8) g_decode = nullptr;
decltype(&flexllm_mlp_block_workspace) g_mlp_workspace = nullptr;
decltype(&flexllm_mlp_block_decode) g_mlp = nullptr;

// A plain contiguous CUDA tensor of `dim` dimensions and type `dtype`, or nullptr.
const at::Tensor* plain(PyObject* o, at::ScalarType dtype, int64_t dim) {
    if (!THPVariable_CheckExact(o)) return nullptr;
    const at::Tensor& t = THPVariable_Unpack(o);
    if (!t.defined() || !t.is_cuda() || t.scalar_type() != dtype || t.dim() != dim || at::isTensorSubclassLike(t) || !t.is_contiguous()) return nullptr;
    return &t;
}
at::Tensor empty_like_device(at::IntArrayRef size, at::ScalarType dtype, const at::Tensor& like) {
    return at::empty(size, at::TensorOptions().dtype(dtype).device(like.device()));
}
PyObject* general() { Py_RETURN_NONE; }
bool modes() { return c10::impl::dispatch_mode_enabled() || at::impl::torch_function_mode_enabled(); }        // someone wants to see the calls
PyObject* result(int status, at::Tensor&& y) { return status != 0 ? PyLong_FromLong(status) : THPVariable_Wrap(std::move(y)); }
bool fits(int64_t v) { return v >= 0 && v <= INT32_MAX; }

template <class F> PyObject* guarded(F f) {          // C++ exceptions as torch's own functions raise them (torch.OutOfMemoryError, torch.AcceleratorError, ...)
    try {
        return f();
    } catch (...) {
        torch::translate_exception_to_python(std::current_exception());
        return nullptr;
    }
}

// bind(prefill, decode, mlp_workspace, mlp)
PyObject* bind(PyObject*, PyObject* args) {
    unsigned long long a, b, c, d;
    if (!PyArg_ParseTuple(args, "KKKK", &a, &b, &c, &d)) return nullptr;
    g_prefill = (decltype(g_prefill))a; g_decode = (decltype(g_decode))b;
    g_mlp_workspace = (decltype(g_mlp_workspace))c; g_mlp = (decltype(g_mlp))d;
    Py_RETURN_NONE;
}

// linear(decode, a [M,K] int8, s_tok [M], w [N,K] int8, s_ch [N]) -> y [M,N]
PyObject* linear(PyObject*, PyObject* const* v, Py_ssize_t n) {
    return guarded([&]() -> PyObject* {
        if (n != 5 || !g_prefill || modes()) return general();
        const at::Tensor *a = plain(v[1], at::kChar, 2), *s = plain(v[2], at::kFloat, 1), *w = plain(v[3], at::kChar, 2), *c = plain(v[4], at::kFloat, 1);
        if (!a || !s || !w || !c) return general();
        const int64_t M = a->size(0), K = a->size(1), N = w->size(0);
        if (!fits(M) || !fits(K) || !fits(N)) return general();
        at::Tensor y = empty_like_device({M, N}, at::kFloat, *a);
        auto fn = v[0] == Py_True ? g_decode : g_prefill;
        const int8_t *ap = (const int8_t*)a->data_ptr(), *wp = (const int8_t*)w->data_ptr();
        const float *sp = (const float*)s->data_ptr(), *cp = (const float*)c->data_ptr();
        float* yp = (float*)y.data_ptr();
        void* stream = c10::cuda::getCurrentCUDAStream().stream();
        int status;
        Py_BEGIN_ALLOW_THREADS
        status = fn(ap, sp, wp, cp, (int)M, (int)N, (int)K, nullptr, yp, stream);
        Py_END_ALLOW_THREADS
        return result(status, std::move(y));
    });
}

// mlp_block(x [M,D], gamma [D], w_gu [2F,D] int8, s_gu [2F], w_d [D,F] int8, s_d [D], eps, order, fht_scale) -> y [M,D]
PyObject* mlp_block(PyObject*, PyObject* const* v, Py_ssize_t n) {
    return guarded([&]() -> PyObject* {
        if (n != 9 || !g_mlp || modes()) return general();
        const at::Tensor *x = plain(v[0], at::kFloat, 2), *g = plain(v[1], at::kFloat, 1), *wgu = plain(v[2], at::kChar, 2), *sgu = plain(v[3], at::kFloat, 1),
                         *wd = plain(v[4], at::kChar, 2), *sd = plain(v[5], at::kFloat, 1);
        if (!x || !g || !wgu || !sgu || !wd || !sd || !PyFloat_Check(v[6]) || !PyLong_Check(v[7]) || !PyFloat_Check(v[8])) return general();
        const float eps = (float)PyFloat_AS_DOUBLE(v[6]), scale = (float)PyFloat_AS_DOUBLE(v[8]);
        const long order = PyLong_AsLong(v[7]);
        if (order == -1 && PyErr_Occurred()) { PyErr_Clear(); return general(); }
        const int64_t M = x->size(0), D = x->size(1), F = wd->size(1);
        if (!fits(M) || !fits(D) || !fits(F) || !fits(order)) return general();
        const size_t bytes = g_mlp_workspace((int)M, (int)D, (int)F);
        at::Tensor ws = empty_like_device({(int64_t)bytes}, at::kByte, *x), y = empty_like_device({M, D}, at::kFloat, *x);
        const float *xp = (const float*)x->data_ptr(), *gp = (const float*)g->data_ptr(), *sgp = (const float*)sgu->data_ptr(), *sdp = (const float*)sd->data_ptr();
        const int8_t *wgp = (const int8_t*)wgu->data_ptr(), *wdp = (const int8_t*)wd->data_ptr();
        float* yp = (float*)y.data_ptr();
        void *wsp = ws.data_ptr(), *stream = c10::cuda::getCurrentCUDAStream().stream();
        int status;
        Py_BEGIN_ALLOW_THREADS
        status = g_mlp(xp, gp, wgp, sgp, wdp, sdp, (int)M, (int)D, (int)F, eps, (int)order, scale, yp, wsp, bytes, stream);
        Py_END_ALLOW_THREADS
        return result(status, std::move(y));
    });
}

PyMethodDef methods[] = {{"bind", bind, METH_VARARGS, "addresses of the library's entry points"},
                         {"linear", (PyCFunction)(void*)linear, METH_FASTCALL, "W8A8 linear layer, output fp32"},
                         {"mlp_block", (PyCFunction)(void*)mlp_block, METH_FASTCALL, "decode MLP block"},
                         {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_front_end", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__front_end() { return PyModule_Create(&module); }
