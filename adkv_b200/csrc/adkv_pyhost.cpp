// Host side of adkv_b200.gemv.decode_attn in native code: argument checks, output allocation and the call into the C ABI
// of libadkv_b200.so for the form that a decode loop uses -- plain contiguous CUDA tensors on the current device, no mask,
// no checkpoints.  Whatever is not of that form, an argument error included, is left to the Python code: `decode` then
// returns None and has done nothing.
//
// A step of one short sequence is bound by this path: the device needs 9.4 us of it (batch 1, 128 tokens), the checks,
// attribute look-ups and 30-argument ctypes call of the Python path took 24 us.
#include <torch/csrc/autograd/python_variable.h>
#include <ATen/ops/empty.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>

#include <climits>

#include "../../include/adkv_b200.h"

namespace {

using decode_fn = decltype(&adkv_decode_attn);
decode_fn g_decode = nullptr;   // the entry point of the library that _lib.py loaded

// A tensor whose memory is what its metadata says: no subclass, no wrapper of a transform, no lazy conjugate or negative.
const at::Tensor *plain(PyObject *o)
{
    if (!THPVariable_CheckExact(o)) return nullptr;
    const at::Tensor &t = THPVariable_Unpack(o);
    constexpr c10::DispatchKeySet odd({c10::DispatchKey::Conjugate, c10::DispatchKey::Negative, c10::DispatchKey::ZeroTensor,
                                       c10::DispatchKey::Python, c10::DispatchKey::Functionalize,
                                       c10::DispatchKey::FuncTorchGradWrapper, c10::DispatchKey::FuncTorchBatched,
                                       c10::DispatchKey::BatchedNestedTensor, c10::DispatchKey::NestedTensor});
    if (!t.defined() || t.layout() != at::kStrided || t.key_set().has_any(odd) || !t.has_storage()) return nullptr;
    return &t;
}

struct Device {
    c10::DeviceIndex index;
    const at::Tensor *tensor(PyObject *o, at::ScalarType type) const
    {
        const at::Tensor *t = plain(o);
        if (!t || !t->is_cuda() || t->get_device() != index || t->scalar_type() != type || !t->is_contiguous()) return nullptr;
        return t;
    }
    const void *data(PyObject *o, at::ScalarType type, int64_t numel) const
    {
        const at::Tensor *t = tensor(o, type);
        return t && t->numel() == numel ? t->data_ptr() : nullptr;
    }
    bool params(PyObject *o, int64_t numel, adkv_params &p) const
    {
        if (!PyTuple_Check(o) && !PyList_Check(o)) return false;
        if (PySequence_Fast_GET_SIZE(o) != 5) return false;
        const void **at[5] = {&p.zp_init, &p.scale_init, &p.alpha, &p.beta, &p.target};
        for (int i = 0; i < 5; ++i)
            if (!(*at[i] = data(PySequence_Fast_GET_ITEM(o, i), at::kHalf, numel))) return false;
        return true;
    }
};

bool as_int(PyObject *o, int &v)
{
    if (!PyLong_CheckExact(o)) return false;
    int overflow = 0;
    const long n = PyLong_AsLongAndOverflow(o, &overflow);
    if (overflow || n < 0 || n >= INT_MAX) return false;
    v = int(n);
    return true;
}

bool as_float(PyObject *o, float &v)
{
    if (PyFloat_CheckExact(o)) v = float(PyFloat_AS_DOUBLE(o));
    else return false;
    return true;
}

// decode(q, k_cache, v_cache, k_new, v_new, k_params, v_params, T, scaling, scale_min, scale_max, bits, out, k_tail, v_tail,
// flags) -> the output tensor, an error code of the library, or None
PyObject *decode(PyObject *, PyObject *const *a, Py_ssize_t n)
{
    if (n != 16 || !g_decode) Py_RETURN_NONE;
    try {
        const at::Tensor *kc = plain(a[1]), *vc = plain(a[2]);
        if (!kc || !vc || !kc->is_cuda() || kc->dim() != 6 || kc->size(4) != 4 || kc->size(5) != 4) Py_RETURN_NONE;
        const Device dev{kc->get_device()};
        if (dev.index != c10::cuda::current_device()) Py_RETURN_NONE;
        if (!dev.tensor(a[1], at::kByte) || !dev.tensor(a[2], at::kByte) || vc->sizes() != kc->sizes()) Py_RETURN_NONE;
        const int64_t B = kc->size(0), Hkv = kc->size(1), cap = kc->size(2), D = 4 * kc->size(3);
        const at::Tensor *q = dev.tensor(a[0], at::kHalf);
        if (!q || q->dim() != 4 || q->size(2) != 1 || q->size(0) != B || q->size(3) != D) Py_RETURN_NONE;
        const int64_t Hq = q->size(1);
        if (B <= 0 || Hkv <= 0 || Hq <= 0 || Hq % Hkv != 0 || B > INT_MAX || Hq > INT_MAX || cap > INT_MAX || D > 512) Py_RETURN_NONE;
        const void *kn = dev.data(a[3], at::kHalf, B * Hkv * D), *vn = dev.data(a[4], at::kHalf, B * Hkv * D);
        adkv_params kp, vp;
        int T, bits, flags;
        float scaling, smin, smax;
        if (!kn || !vn || !dev.params(a[5], Hkv * D, kp) || !dev.params(a[6], Hkv * D, vp) || !as_int(a[7], T) ||
            !as_float(a[8], scaling) || !as_float(a[9], smin) || !as_float(a[10], smax) || !as_int(a[11], bits) ||
            (bits != 2 && bits != 4) || T / (32 / bits) >= cap || !as_int(a[15], flags))
            Py_RETURN_NONE;
        void *tail[2] = {nullptr, nullptr};
        if ((a[13] == Py_None) != (a[14] == Py_None)) Py_RETURN_NONE;
        if (a[13] != Py_None) {
            if (flags & ADKV_FLAG_HALF_STATE) Py_RETURN_NONE;
            for (int i = 0; i < 2; ++i) {
                const at::Tensor *t = dev.tensor(a[13 + i], at::kFloat);
                if (!t || t->dim() != 4 || t->size(0) != B || t->size(1) != Hkv || t->size(2) != 2 || t->size(3) != D) Py_RETURN_NONE;
                tail[i] = t->data_ptr();
            }
        }
        void *const stream = c10::cuda::getCurrentCUDAStream(dev.index).stream();
        const void *const qp = q->data_ptr();
        void *const kcp = kc->data_ptr(), *const vcp = vc->data_ptr();
        // Everything that may fail comes before the launch, the Python object of the result too: a step that has been
        // launched must not be left to the Python code, which would launch it again.
        void *op;
        PyObject *result;
        if (a[12] == Py_None) {
            const at::Tensor out = at::empty({B, Hq, D}, kc->options().dtype(at::kHalf));
            if (!out.is_cuda() || !out.has_storage()) Py_RETURN_NONE;
            op = out.data_ptr();
            result = THPVariable_Wrap(out);
            if (!result) {
                PyErr_Clear();
                Py_RETURN_NONE;
            }
        } else {
            const at::Tensor *t = dev.tensor(a[12], at::kHalf);
            if (!t || t->dim() != 3 || t->size(0) != B || t->size(1) != Hq || t->size(2) != D) Py_RETURN_NONE;
            op = t->data_ptr();
            result = a[12];
            Py_INCREF(result);
        }
        int rc;
        Py_BEGIN_ALLOW_THREADS
        rc = g_decode(qp, kcp, vcp, kn, vn, &kp, &vp, tail[0], tail[1], nullptr, 0, op, int(B), int(Hq), int(Hkv), T, int(D),
                      int(cap), bits, scaling, smin, smax, unsigned(flags), stream);
        Py_END_ALLOW_THREADS
        if (!rc) return result;
        Py_DECREF(result);
        return PyLong_FromLong(rc);
    } catch (...) {   // out of memory and the like: the Python code meets it again and raises what it raises
        PyErr_Clear();
        Py_RETURN_NONE;
    }
}

PyObject *bind(PyObject *, PyObject *addr)
{
    g_decode = reinterpret_cast<decode_fn>(PyLong_AsVoidPtr(addr));
    if (PyErr_Occurred()) return nullptr;
    Py_RETURN_NONE;
}

PyMethodDef methods[] = {
    {"decode", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(decode)), METH_FASTCALL, nullptr},
    {"bind", bind, METH_O, nullptr},
    {nullptr, nullptr, 0, nullptr},
};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_adkv_pyhost", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__adkv_pyhost(void) { return PyModule_Create(&module); }
