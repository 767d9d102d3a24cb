// CPython binding of the forward calls: what W4a16Dec's Python methods did per call -- spec lookup, tensor checks, the
// output allocation, the current stream, the C ABI call -- in one native function each.
//
// Why: a decode linear runs 4 to 20 us on the GPU, and a host that drives a layer call by call (no captured graph) spent
// 13 us in Python and ctypes around each of them (10 with the caller's output): 4 us for torch.cuda.current_stream(), 2.5 for
// torch.empty, 1.3 for a ctypes lin_spec, 1 for the ctypes call itself.  Here the same steps and the launch take 3.4 us (2.4
// with the caller's output), so eager decode is bound by the launches again.
//
// The library itself keeps its plain C ABI; this module reaches it through the addresses that the ctypes loader resolved
// (bind()), so that both go to the same build of it.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/cuda/EmptyTensor.h>
#include <ATen/record_function.h>
#include <c10/core/impl/LocalDispatchKeySet.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/python_variable.h>

#include <cstdint>

#include "../../include/w4a16_b200.h"

namespace {

decltype(&w4a16_last_error) p_last_error;
decltype(&w4a16_lin_spec) p_lin_spec;
decltype(&w4a16_sk_multi_dev) p_sk_multi_dev;
decltype(&w4a16_moe_ffn) p_moe_ffn;
decltype(&w4a16_head_spec) p_head_spec;
decltype(&w4a16_head_forward) p_head_forward;
// entry points with the signature of w4a16_lin_forward, by the index that the caller passes
typedef decltype(&w4a16_lin_forward) lin_fn;
constexpr int N_LIN = 5;
lin_fn p_lin[N_LIN];
const char* const lin_symbol[N_LIN] = {"w4a16_lin_forward", "w4a16_sk_single_dev", "w4a16_sk_single_static",
                                       "w4a16_sk_single_allreduce", "w4a16_lin_forward_x32"};
const char* const lin_method[N_LIN] = {"lin_forward", "sk_single_dev", "sk_single_static", "sk_single_allreduce",
                                       "lin_forward_x32"};
constexpr int LIN_X32 = 4;

PyObject* error_type = nullptr;   // W4a16Error

PyObject* raise_last(w4a16_dec* dec) {
    PyErr_SetString(error_type, p_last_error(dec));
    return nullptr;
}

const char* type_name(at::ScalarType st) { return st == at::kHalf ? "torch.float16" : "torch.float32"; }

// The tensor behind `o` if it is a contiguous CUDA tensor of that type on that device; else null with W4a16Error set.
const at::Tensor* checked(PyObject* o, at::ScalarType st, int device, const char* what) {
    if (!THPVariable_Check(o)) {
        PyErr_Format(PyExc_TypeError, "%s: expected a torch.Tensor", what);
        return nullptr;
    }
    const at::Tensor& v = THPVariable_Unpack(o);
    if (!(v.is_cuda() && v.is_contiguous() && v.scalar_type() == st && v.get_device() == device)) {
        PyErr_Format(error_type, "%s: need a contiguous %s CUDA tensor on device %d", what, type_name(st), device);
        return nullptr;
    }
    return &v;
}

// Nothing stands between torch.empty and its allocator: no dispatch mode or function transform, no profiler, no deterministic
// fill.  Then the allocator may be called directly (3.4 us of host time per call against 4.4 through the dispatcher).
bool plain_empty() {
    const at::Context& ctx = at::globalContext();
    return c10::impl::tls_local_dispatch_key_set().included_ == c10::default_included_set && !at::hasCallbacks() &&
           !(ctx.deterministicAlgorithms() && ctx.deterministicFillUninitializedMemory());
}

// A [t, n] output: the caller's buffer, checked, or a new tensor.
bool output(PyObject* dst, int64_t t, int64_t n, bool f16, int device, at::Tensor* out) {
    const at::ScalarType st = f16 ? at::kHalf : at::kFloat;
    if (dst == Py_None) {
        const c10::Device where(c10::kCUDA, (c10::DeviceIndex)device);
        *out = plain_empty() ? at::detail::empty_cuda({t, n}, st, where, std::nullopt)
                             : at::empty({t, n}, at::TensorOptions().dtype(st).device(where));
        return true;
    }
    const at::Tensor* d = checked(dst, st, device, "dst");
    if (!d) {
        return false;
    }
    if (d->numel() != t * n) {
        PyErr_Format(error_type, "dst has %lld elements, need %lldx%lld", (long long)d->numel(), (long long)t, (long long)n);
        return false;
    }
    *out = *d;
    return true;
}

// torch's current stream.  Its default stream has the handle 0, which the C ABI reads as "the decoder's own stream";
// 1 is cudaStreamLegacy, the explicit name of that same stream.
void* current_stream(int device) {
    void* s = (void*)c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)device).stream();
    return s ? s : (void*)1;
}

struct Args {
    w4a16_dec* dec;
    int device;
};
bool head_args(PyObject* const* a, Args* r) {
    r->dec = (w4a16_dec*)PyLong_AsVoidPtr(a[0]);
    if (!r->dec) {
        if (!PyErr_Occurred()) {
            PyErr_SetString(error_type, "the decoder is closed");
        }
        return false;
    }
    r->device = (int)PyLong_AsLong(a[1]);
    return !PyErr_Occurred();
}

bool want_args(Py_ssize_t n, Py_ssize_t want) {
    if (n != want) {
        PyErr_Format(PyExc_TypeError, "expected %zd arguments, got %zd", want, n);
        return false;
    }
    return true;
}

template <class F>
PyObject* guarded(F f) {
    try {
        return f();
    } catch (const std::exception& e) {   // an allocation that failed
        PyErr_SetString(PyExc_RuntimeError, e.what());
        return nullptr;
    }
}

// linear(handle, device, entry, name, x, t, dst, out_f16) -> dst
PyObject* linear(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
    return guarded([&]() -> PyObject* {
        Args r;
        if (!want_args(nargs, 8) || !head_args(a, &r)) {
            return nullptr;
        }
        const long entry = PyLong_AsLong(a[2]);
        const char* name = PyUnicode_AsUTF8(a[3]);
        const long long t = PyLong_AsLongLong(a[5]);
        const int f16 = PyObject_IsTrue(a[7]);
        if (PyErr_Occurred() || !name || entry < 0 || entry >= N_LIN) {
            return nullptr;
        }
        int n, k, g;
        if (p_lin_spec(r.dec, name, &n, &k, &g)) {
            return raise_last(r.dec);
        }
        const bool x32 = entry == LIN_X32;
        const at::Tensor* x = checked(a[4], x32 ? at::kFloat : at::kHalf, r.device, x32 ? "x32" : "x16");
        if (!x) {
            return nullptr;
        }
        if (x->numel() != t * k) {
            PyErr_Format(error_type, "%s %s: x has %lld elements, need %lldx%d", lin_method[entry], name, (long long)x->numel(),
                         t, k);
            return nullptr;
        }
        at::Tensor out;
        if (!output(a[6], t, n, f16, r.device, &out)) {
            return nullptr;
        }
        void *xp = x->data_ptr(), *yp = out.data_ptr(), *st = current_stream(r.device);
        int rc;
        Py_BEGIN_ALLOW_THREADS
        rc = p_lin[entry](r.dec, name, xp, yp, (int)t, f16 ? W4A16_OUT_F16 : W4A16_OUT_F32, st);
        Py_END_ALLOW_THREADS
        if (rc) {
            return raise_last(r.dec);
        }
        return THPVariable_Wrap(out);
    });
}

// multi(handle, device, names, x, outs, t, out_f16) -> list of outputs
PyObject* multi(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
    return guarded([&]() -> PyObject* {
        Args r;
        if (!want_args(nargs, 7) || !head_args(a, &r)) {
            return nullptr;
        }
        constexpr Py_ssize_t MAXSEG = 64;   // the library refuses more than it supports with its own message
        // tuples of their own: the library reads the names without the interpreter lock, while the caller's lists may change
        PyObject* names = PySequence_Tuple(a[2]);
        if (!names) {
            return nullptr;
        }
        PyObject* outs = a[4] == Py_None ? nullptr : PySequence_Tuple(a[4]);
        PyObject* result = nullptr;
        [&] {
            if (a[4] != Py_None && !outs) {
                return;
            }
            const Py_ssize_t ns = PyTuple_GET_SIZE(names);
            const long long t = PyLong_AsLongLong(a[5]);
            const int f16 = PyObject_IsTrue(a[6]);
            if (PyErr_Occurred()) {
                return;
            }
            if (ns < 1 || ns > MAXSEG) {
                PyErr_Format(error_type, "w4a16 sk_multi: %zd segments", ns);
                return;
            }
            const char* nm[MAXSEG];
            int n[MAXSEG], k = 0;
            for (Py_ssize_t i = 0; i < ns; ++i) {
                nm[i] = PyUnicode_AsUTF8(PyTuple_GET_ITEM(names, i));
                if (!nm[i]) {
                    return;
                }
                int ki, g;
                if (p_lin_spec(r.dec, nm[i], &n[i], &ki, &g)) {
                    raise_last(r.dec);
                    return;
                }
                k = i == 0 ? ki : k;
            }
            const at::Tensor* x = checked(a[3], at::kHalf, r.device, "x16");
            if (!x) {
                return;
            }
            if (x->numel() != t * k) {
                PyErr_SetString(error_type, "sk_multi_dev: x size does not match t*k");
                return;
            }
            // outputs beyond the names are left alone, a name without an output is refused
            const Py_ssize_t no = outs ? PyTuple_GET_SIZE(outs) : ns;
            if (no < ns) {
                PyErr_Format(error_type, "sk_multi_dev: %zd outputs for %zd names", no, ns);
                return;
            }
            at::Tensor y[MAXSEG];
            void* yp[MAXSEG];
            for (Py_ssize_t i = 0; i < ns; ++i) {
                if (!output(outs ? PyTuple_GET_ITEM(outs, i) : Py_None, t, n[i], f16, r.device, &y[i])) {
                    return;
                }
                yp[i] = y[i].data_ptr();
            }
            void *xp = x->data_ptr(), *st = current_stream(r.device);
            int rc;
            Py_BEGIN_ALLOW_THREADS
            rc = p_sk_multi_dev(r.dec, nm, (int)ns, xp, yp, (int)t, f16 ? W4A16_OUT_F16 : W4A16_OUT_F32, st);
            Py_END_ALLOW_THREADS
            if (rc) {
                raise_last(r.dec);
                return;
            }
            result = PyList_New(ns);
            for (Py_ssize_t i = 0; result && i < ns; ++i) {
                PyList_SET_ITEM(result, i, THPVariable_Wrap(y[i]));
            }
        }();
        Py_DECREF(names);
        Py_XDECREF(outs);
        return result;
    });
}

// moe(handle, device, layer, logits, x, t, n_experts, hidden, out, out_f16) -> out
PyObject* moe(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
    return guarded([&]() -> PyObject* {
        Args r;
        if (!want_args(nargs, 10) || !head_args(a, &r)) {
            return nullptr;
        }
        const int layer = (int)PyLong_AsLong(a[2]);
        const long long t = PyLong_AsLongLong(a[5]), ne = PyLong_AsLongLong(a[6]), h = PyLong_AsLongLong(a[7]);
        const int f16 = PyObject_IsTrue(a[9]);
        if (PyErr_Occurred()) {
            return nullptr;
        }
        const at::Tensor* lg = checked(a[3], at::kFloat, r.device, "logits");
        const at::Tensor* x = lg ? checked(a[4], at::kHalf, r.device, "x16") : nullptr;
        if (!x) {
            return nullptr;
        }
        if (lg->numel() != t * ne || x->numel() != t * h) {
            PyErr_SetString(error_type, "moe_ffn_dev_t: logits/x sizes do not match t");
            return nullptr;
        }
        at::Tensor out;
        if (!output(a[8], t, h, f16, r.device, &out)) {
            return nullptr;
        }
        const float* lp = (const float*)lg->data_ptr();
        void *xp = x->data_ptr(), *yp = out.data_ptr(), *st = current_stream(r.device);
        int rc;
        Py_BEGIN_ALLOW_THREADS
        rc = p_moe_ffn(r.dec, layer, lp, xp, yp, (int)t, f16 ? W4A16_OUT_F16 : W4A16_OUT_F32, st);
        Py_END_ALLOW_THREADS
        if (rc) {
            return raise_last(r.dec);
        }
        return THPVariable_Wrap(out);
    });
}

// head(handle, device, x, t, out) -> out
PyObject* head(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
    return guarded([&]() -> PyObject* {
        Args r;
        if (!want_args(nargs, 5) || !head_args(a, &r)) {
            return nullptr;
        }
        const long long t = PyLong_AsLongLong(a[3]);
        if (PyErr_Occurred()) {
            return nullptr;
        }
        int n, k;
        if (p_head_spec(r.dec, &n, &k)) {
            return raise_last(r.dec);
        }
        const at::Tensor* x = checked(a[2], at::kFloat, r.device, "x32");
        if (!x) {
            return nullptr;
        }
        if (x->numel() != t * k) {
            PyErr_Format(error_type, "head_forward: x has %lld elements, need %lldx%d", (long long)x->numel(), t, k);
            return nullptr;
        }
        at::Tensor out;
        if (!output(a[4], t, n, false, r.device, &out)) {
            return nullptr;
        }
        const float* xp = (const float*)x->data_ptr();
        float* yp = (float*)out.data_ptr();
        void* st = current_stream(r.device);
        int rc;
        Py_BEGIN_ALLOW_THREADS
        rc = p_head_forward(r.dec, xp, yp, (int)t, st);
        Py_END_ALLOW_THREADS
        if (rc) {
            return raise_last(r.dec);
        }
        return THPVariable_Wrap(out);
    });
}

// bind(error_type, address_of): `address_of(symbol)` gives the address of a library function
PyObject* bind(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
    if (!want_args(nargs, 2)) {
        return nullptr;
    }
    auto resolve = [&](const char* symbol, auto* to) {
        PyObject* v = PyObject_CallFunction(a[1], "s", symbol);
        if (!v) {
            return false;
        }
        *(void**)to = PyLong_AsVoidPtr(v);
        Py_DECREF(v);
        return !PyErr_Occurred();
    };
    bool ok = resolve("w4a16_last_error", &p_last_error) && resolve("w4a16_lin_spec", &p_lin_spec) &&
              resolve("w4a16_sk_multi_dev", &p_sk_multi_dev) && resolve("w4a16_moe_ffn", &p_moe_ffn) &&
              resolve("w4a16_head_spec", &p_head_spec) && resolve("w4a16_head_forward", &p_head_forward);
    for (int i = 0; ok && i < N_LIN; ++i) {
        ok = resolve(lin_symbol[i], &p_lin[i]);
    }
    if (!ok) {
        return nullptr;
    }
    Py_INCREF(a[0]);
    Py_XSETREF(error_type, a[0]);
    Py_RETURN_NONE;
}

PyMethodDef methods[] = {
    {"bind", (PyCFunction)(void (*)(void))bind, METH_FASTCALL, nullptr},
    {"linear", (PyCFunction)(void (*)(void))linear, METH_FASTCALL, nullptr},
    {"multi", (PyCFunction)(void (*)(void))multi, METH_FASTCALL, nullptr},
    {"moe", (PyCFunction)(void (*)(void))moe, METH_FASTCALL, nullptr},
    {"head", (PyCFunction)(void (*)(void))head, METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr},
};
PyModuleDef module_def = {PyModuleDef_HEAD_INIT, "_native", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__native(void) { return PyModule_Create(&module_def); }
