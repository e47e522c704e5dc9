// PyTorch face of the C ABI (include/gla_b200.h) for the calls a program makes once per layer or once per token.
//
// At those rates the host path is the call: checking six tensors, filling the argument structure and asking for stream
// and device through Python and ctypes took 26 us per operator call and 43 us per one-token call, several times what the
// GPU needs.  The functions here do the same checks on the tensor objects themselves and call the library through the
// addresses bind() was given, so there is one library and one ABI.  A call whose arguments are not all as the fast path
// wants them is answered with kSlow, and the Python code in ops.py, which knows how to say what is wrong, takes over.
#include <ATen/ATen.h>
#include <ATen/core/grad_mode.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/python_variable.h>

#include <cmath>
#include <cstring>

#include "gla_b200.h"

namespace {

constexpr int kSlow = 1;               // arguments for the Python path
constexpr int64_t kV = GLA_B200_HEAD_V;

decltype(&gla_b200_forward) g_forward = nullptr;
decltype(&gla_b200_workspace_bytes) g_workspace_bytes = nullptr;

// The tensor inside a Python object, or null when it is not a plain torch.Tensor / Parameter.
const at::Tensor* tensor(PyObject* o) {
    if (!THPVariable_CheckExact(o)) return nullptr;
    return &THPVariable_Unpack(o);
}

bool number(PyObject* o, double* out) {
    if (PyFloat_CheckExact(o)) { *out = PyFloat_AS_DOUBLE(o); return true; }
    if (PyLong_CheckExact(o)) {
        *out = PyLong_AsDouble(o);
        if (*out == -1.0 && PyErr_Occurred()) { PyErr_Clear(); return false; }
        return true;
    }
    return false;
}
bool integer(PyObject* o, long* out) {
    if (!PyLong_CheckExact(o)) return false;
    *out = PyLong_AsLong(o);
    if (*out == -1 && PyErr_Occurred()) { PyErr_Clear(); return false; }
    return *out >= INT32_MIN && *out <= INT32_MAX;
}
bool grid_pair(PyObject* o, int32_t* h, int32_t* w) {
    if (o == Py_None) { *h = *w = 0; return true; }
    if (!PyTuple_CheckExact(o) || PyTuple_GET_SIZE(o) != 2) return false;
    long a, b;
    if (!integer(PyTuple_GET_ITEM(o, 0), &a) || !integer(PyTuple_GET_ITEM(o, 1), &b)) return false;
    *h = static_cast<int32_t>(a); *w = static_cast<int32_t>(b);
    return true;
}
// "row", "row_rev", ... take the Python path
bool scan_order(PyObject* o, int32_t* d) {
    long x;
    if (!integer(o, &x)) return false;
    *d = static_cast<int32_t>(x);
    return true;
}

// A [B, T, H, last] fp16 CUDA operand with a dense innermost dimension, on q's device.
bool operand(const at::Tensor& x, const at::Tensor& q, int64_t last, const void** ptr, int64_t strides[3]) {
    if (!x.is_cuda() || x.scalar_type() != at::kHalf || x.dim() != 4 || x.layout() != at::kStrided) return false;
    const auto s = x.sizes(), n = q.sizes(), t = x.strides();
    if (s[3] != last || s[0] != n[0] || s[1] != n[1] || s[2] != n[2] || x.device() != q.device()) return false;
    if (x.numel() == 0 || t[3] != 1) return false;
    *ptr = x.data_ptr();
    strides[0] = t[0]; strides[1] = t[1]; strides[2] = t[2];
    return true;
}
bool state(const at::Tensor& s, const at::Tensor& q) {
    const auto n = q.sizes(), m = s.sizes();
    return s.is_cuda() && s.scalar_type() == at::kFloat && s.dim() == 4 && m[0] == n[0] && m[1] == n[2] && m[2] == n[3] &&
           m[3] == kV && s.is_contiguous() && s.device() == q.device();
}

// q, k, v, g and everything that follows from their shape; false: the Python path
bool operands(gla_b200_args& a, const at::Tensor& q, const at::Tensor& k, const at::Tensor& v, const at::Tensor& g) {
    if (q.dim() != 4) return false;
    const auto n = q.sizes();
    if ((n[3] != 32 && n[3] != 64) || n[0] > INT32_MAX || n[1] > INT32_MAX || n[2] > INT32_MAX) return false;
    if (!operand(q, q, n[3], &a.q, a.q_stride) || !operand(k, q, n[3], &a.k, a.k_stride) ||
        !operand(g, q, n[3], &a.g, a.g_stride) || !operand(v, q, kV, &a.v, a.v_stride))
        return false;
    a.B = static_cast<int32_t>(n[0]); a.T = static_cast<int32_t>(n[1]); a.H = static_cast<int32_t>(n[2]);
    a.K = static_cast<int32_t>(n[3]); a.V = static_cast<int32_t>(kV);
    return true;
}

// run(q, k, v, gk, o, ws, scale, gk_normalizer, direction, grid_hw, initial_state, final_state, out_gate, rms_w, eps,
//     segments, wait_limit) -> 0, a library error, or kSlow.  The operator on caller-owned output and workspace.
PyObject* run(PyObject*, PyObject* const* v, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    if (n != 17) return PyLong_FromLong(kSlow);
    const at::Tensor* t[6];
    for (int i = 0; i < 6; ++i)
        if (!(t[i] = tensor(v[i]))) return PyLong_FromLong(kSlow);
    const at::Tensor& q = *t[0];
    gla_b200_args a;
    std::memset(&a, 0, sizeof(a));
    double scale, norm, eps;
    long segments, limit;
    const void* optr = nullptr;
    if (!operands(a, q, *t[1], *t[2], *t[3]) || !operand(*t[4], q, kV, &optr, a.o_stride) || !number(v[6], &scale) ||
        !number(v[7], &norm) || !scan_order(v[8], &a.direction) || !grid_pair(v[9], &a.grid_h, &a.grid_w) ||
        !number(v[14], &eps) || !integer(v[15], &segments) || !integer(v[16], &limit) || limit < 0)
        return PyLong_FromLong(kSlow);
    a.o = const_cast<void*>(optr);
    for (int i = 0; i < 2; ++i) {
        if (v[10 + i] == Py_None) continue;
        const at::Tensor* s = tensor(v[10 + i]);
        if (!s || !state(*s, q)) return PyLong_FromLong(kSlow);
        if (i == 0) a.initial_state = static_cast<const float*>(s->data_ptr());
        else a.final_state = static_cast<float*>(s->data_ptr());
    }
    if (v[12] != Py_None || v[13] != Py_None) {
        const at::Tensor *gate = tensor(v[12]), *w = tensor(v[13]);
        if (!gate || !w || !operand(*gate, q, kV, &a.out_gate, a.gate_stride) || w->scalar_type() != at::kHalf ||
            w->numel() != kV || !w->is_contiguous() || w->device() != q.device())
            return PyLong_FromLong(kSlow);
        a.rms_weight = w->data_ptr();
        a.rms_eps = static_cast<float>(eps);
    }
    const at::Tensor& ws = *t[5];
    if (!ws.is_cuda() || ws.device() != q.device() || !ws.is_contiguous()) return PyLong_FromLong(kSlow);
    a.workspace = ws.data_ptr();
    a.workspace_bytes = ws.nbytes();
    a.segments = static_cast<int32_t>(segments);
    a.scale = static_cast<float>(scale);
    a.gk_normalizer = static_cast<float>(norm);
    a.wait_limit = static_cast<uint32_t>(limit);
    const c10::cuda::CUDAGuard guard(q.device());
    return PyLong_FromLong(g_forward(&a, c10::cuda::getCurrentCUDAStream(q.device().index()).stream()));
    END_HANDLE_TH_ERRORS
}

// gla(q, k, v, g, scale, initial_state, output_final_state, direction, grid_hw, gk_normalizer, segments) ->
// (o, final_state or None), a library error, or kSlow.  The FLA-style call outside autograd: allocates output, scratch and
// final state.  The scratch need not be cleared (the launch clears what must be).
PyObject* gla(PyObject*, PyObject* const* v, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    if (n != 11) return PyLong_FromLong(kSlow);
    const at::Tensor* t[4];
    for (int i = 0; i < 4; ++i)
        if (!(t[i] = tensor(v[i]))) return PyLong_FromLong(kSlow);
    const at::Tensor& q = *t[0];
    const at::Tensor* s0 = v[5] == Py_None ? nullptr : tensor(v[5]);
    if (v[5] != Py_None && !s0) return PyLong_FromLong(kSlow);
    if (at::GradMode::is_enabled()) {
        bool wanted = s0 && s0->requires_grad();
        for (const at::Tensor* x : t) wanted = wanted || x->requires_grad();
        if (wanted) return PyLong_FromLong(kSlow);
    }
    gla_b200_args a;
    std::memset(&a, 0, sizeof(a));
    double scale, norm;
    long segments;
    if (!operands(a, q, *t[1], *t[2], *t[3]) || !scan_order(v[7], &a.direction) || !grid_pair(v[8], &a.grid_h, &a.grid_w) ||
        !number(v[9], &norm) || !integer(v[10], &segments) || (s0 && !state(*s0, q)))
        return PyLong_FromLong(kSlow);
    if (v[4] == Py_None) scale = 1.0 / std::sqrt(static_cast<double>(a.K));
    else if (!number(v[4], &scale)) return PyLong_FromLong(kSlow);
    const int final_wanted = PyObject_IsTrue(v[6]);
    if (final_wanted < 0) return nullptr;
    if (s0) a.initial_state = static_cast<const float*>(s0->data_ptr());
    a.segments = static_cast<int32_t>(segments);
    a.scale = static_cast<float>(scale);
    a.gk_normalizer = static_cast<float>(norm);

    const c10::cuda::CUDAGuard guard(q.device());
    const auto opts = at::TensorOptions().device(q.device());
    at::Tensor o = at::empty({a.B, a.T, a.H, kV}, opts.dtype(at::kHalf)), final_state;
    if (final_wanted) {
        final_state = at::empty({a.B, a.H, a.K, kV}, opts.dtype(at::kFloat));
        a.final_state = static_cast<float*>(final_state.data_ptr());
    }
    a.o = o.data_ptr();
    a.workspace_bytes = g_workspace_bytes(a.B, a.T, a.H, a.K, a.V);
    const at::Tensor ws = at::empty({static_cast<int64_t>(a.workspace_bytes)}, opts.dtype(at::kByte));
    a.workspace = ws.data_ptr();
    const int rc = g_forward(&a, c10::cuda::getCurrentCUDAStream(q.device().index()).stream());
    if (rc != GLA_B200_OK) return PyLong_FromLong(rc);
    PyObject* po = THPVariable_Wrap(o);
    if (!po) return nullptr;
    PyObject* pf = final_wanted ? THPVariable_Wrap(final_state) : Py_NewRef(Py_None);
    if (!pf) { Py_DECREF(po); return nullptr; }
    PyObject* out = PyTuple_Pack(2, po, pf);
    Py_DECREF(po);
    Py_DECREF(pf);
    return out;
    END_HANDLE_TH_ERRORS
}

// bind(address of gla_b200_forward, address of gla_b200_workspace_bytes)
PyObject* bind(PyObject*, PyObject* const* v, Py_ssize_t n) {
    if (n != 2) { PyErr_SetString(PyExc_TypeError, "bind takes 2 addresses"); return nullptr; }
    void* p[2];
    for (int i = 0; i < 2; ++i)
        if (!(p[i] = PyLong_AsVoidPtr(v[i]))) {
            if (!PyErr_Occurred()) PyErr_SetString(PyExc_ValueError, "null address");
            return nullptr;
        }
    g_forward = reinterpret_cast<decltype(g_forward)>(p[0]);
    g_workspace_bytes = reinterpret_cast<decltype(g_workspace_bytes)>(p[1]);
    Py_RETURN_NONE;
}

PyMethodDef methods[] = {
    {"bind", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(bind)), METH_FASTCALL, nullptr},
    {"run", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(run)), METH_FASTCALL, nullptr},
    {"gla", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(gla)), METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_front", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__front() { return PyModule_Create(&module); }
