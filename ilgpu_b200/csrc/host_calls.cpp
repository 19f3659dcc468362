// The host path of the Python mirror (algorithms.py) for calls that need nothing special: argument
// checks, temp sizing, the current stream and the call into the native library in one step.
//
// A pass over a few thousand elements takes the GPU a few microseconds; the same checks written in
// Python, with ctypes for the call, took ten to twenty on the host, which then was what small and
// ordinary calls cost.  Each function below returns True (or the result) when it has done the work,
// and False (or None) for whatever it does not cover: a view that fails a check, an accelerator
// whose device is not current, a status other than success.  The caller then goes through the
// Python code, which raises the reference's exceptions in the reference's order.
#include <Python.h>

#include <ATen/ATen.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>
#include <cuda_runtime.h>
#include <torch/csrc/autograd/python_variable.h>

#include <cmath>
#include <cstring>

#include "../../include/b200alg.h"

namespace {

// Entry points of the library that the package has loaded (addresses handed over by bind(), in the
// order of ENTRY_POINTS).
#define B200ALG_ENTRY_POINTS(X) \
    X(radix_sort_temp_bytes) \
    X(radix_sort_keys) \
    X(radix_sort_pairs) \
    X(radix_sort_pairs_sequence) \
    X(scan_temp_bytes) \
    X(scan_carry) \
    X(reduce) \
    X(reduce_to_host) \
    X(histogram) \
    X(initialize) \
    X(unique_temp_bytes) \
    X(unique_to_host)
struct Library {
#define B200ALG_MEMBER(name) decltype(&b200alg_##name) name;
    B200ALG_ENTRY_POINTS(B200ALG_MEMBER)
} lib;
#define B200ALG_NAME(name) "b200alg_" #name,
constexpr const char *kEntryPoints[] = {B200ALG_ENTRY_POINTS(B200ALG_NAME)};

constexpr int64_t kMaxLength = (1ll << 31) - 1;  // the reference's int.MaxValue

// element type codes of include/b200alg.h
int code_of(at::ScalarType t) {
    switch (t) {
    case at::kChar: return B200ALG_I8;
    case at::kByte: return B200ALG_U8;
    case at::kShort: return B200ALG_I16;
    case at::kUInt16: return B200ALG_U16;
    case at::kInt: return B200ALG_I32;
    case at::kUInt32: return B200ALG_U32;
    case at::kLong: return B200ALG_I64;
    case at::kUInt64: return B200ALG_U64;
    case at::kHalf: return B200ALG_F16;
    case at::kFloat: return B200ALG_F32;
    case at::kDouble: return B200ALG_F64;
    default: return -1;
    }
}

struct View {
    void *data = nullptr;
    int64_t n = 0, stride = 1;
    int code = -1, bytes = 0;
};

// A one-dimensional CUDA view on `device` (element type `code` unless that is negative).
bool view_of(PyObject *o, int device, int code, View &v) {
    if (!THPVariable_Check(o)) return false;
    const at::Tensor &t = THPVariable_Unpack(o);
    if (t.dim() != 1 || !t.is_cuda() || t.get_device() != device) return false;
    v.code = code_of(t.scalar_type());
    if (v.code < 0 || (code >= 0 && v.code != code)) return false;
    v.n = t.numel();
    v.stride = v.n > 1 ? t.stride(0) : 1;
    if (v.stride < 1 || v.n > kMaxLength) return false;
    v.data = t.data_ptr();
    v.bytes = (int)t.element_size();
    return true;
}

// A dense int view that starts on 256 bytes and holds at least `need` bytes.
bool temp_of(PyObject *o, int device, int64_t need, View &v) {
    return view_of(o, device, B200ALG_I32, v) && v.stride == 1 && v.n >= (need + 3) / 4 && (uintptr_t)v.data % 256 == 0;
}

// The accelerator's device when it is the current one (-1: whichever is current), else -1.
int device_of(PyObject *o) {
    const long wanted = PyLong_AsLong(o);
    const int current = (int)c10::cuda::current_device();
    return wanted < 0 || wanted == current ? current : -1;
}

bool stream_of(PyObject *o, int device, void *&stream) {
    if (o == Py_None) {
        stream = c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)device).stream();
        return true;
    }
    PyObject *handle = PyObject_GetAttrString(o, "cuda_stream");
    if (handle) {
        stream = PyLong_AsVoidPtr(handle);
        Py_DECREF(handle);
    }
    if (PyErr_Occurred()) {
        PyErr_Clear();
        return false;
    }
    return true;
}

int int_of(PyObject *o) { return (int)PyLong_AsLong(o); }

// Runs `call` (a status) with the interpreter lock released.
template <typename Call> int released(Call call) {
    int status;
    Py_BEGIN_ALLOW_THREADS;
    status = call();
    Py_END_ALLOW_THREADS;
    return status;
}

// What every function below does around its own work: no C++ exception leaves, and a Python error
// from a conversion means "not covered".
template <typename Body> PyObject *guarded(Body body) {
    bool done = false;
    try {
        done = body();
    } catch (...) {
        done = false;
    }
    if (PyErr_Occurred()) {
        PyErr_Clear();
        done = false;
    }
    return PyBool_FromLong(done);
}

// A few bytes of host memory that a kernel can write, one for each host thread that asks for a
// scalar result; given back when the thread ends.
struct HostSlot {
    void *p = nullptr;
    void *get() {
        if (!p && cudaHostAlloc(&p, 64, cudaHostAllocPortable | cudaHostAllocMapped) != cudaSuccess) {
            (void)cudaGetLastError();
            p = nullptr;
        }
        return p;
    }
    ~HostSlot() {
        if (p) cudaFreeHost(p);
    }
};
thread_local HostSlot host_slot;

// sort_keys(device, code, order, stream, view, temp)
PyObject *sort_keys(PyObject *, PyObject *const *a, Py_ssize_t count) {
    return guarded([&] {
        const int device = count == 6 ? device_of(a[0]) : -1;
        const int code = int_of(a[1]), order = int_of(a[2]);
        View keys, temp;
        void *stream;
        int64_t need = 0;
        if (device < 0 || !view_of(a[4], device, code, keys)) return false;
        if (lib.radix_sort_temp_bytes(code, keys.n, 0, &need) != B200ALG_OK || !temp_of(a[5], device, need, temp)) return false;
        if (!stream_of(a[3], device, stream)) return false;
        return released([&] {
                   return lib.radix_sort_keys(stream, keys.data, keys.n, keys.stride, code, order, temp.data, temp.n * 4);
               }) == B200ALG_OK;
    });
}

// sort_pairs(device, code, order, value_code or -1, stream, keys, values, temp); with a value code the
// values are made by that type's sequencer
PyObject *sort_pairs(PyObject *, PyObject *const *a, Py_ssize_t count) {
    return guarded([&] {
        const int device = count == 8 ? device_of(a[0]) : -1;
        const int code = int_of(a[1]), order = int_of(a[2]), sequence = int_of(a[3]);
        View keys, values, temp;
        void *stream;
        int64_t need = 0;
        if (device < 0 || !view_of(a[5], device, code, keys) || !view_of(a[6], device, sequence, values)) return false;
        if (keys.stride != 1 || values.stride != 1 || (sequence >= 0 ? values.n != keys.n : values.n < keys.n)) return false;
        if (lib.radix_sort_temp_bytes(code, keys.n, values.bytes, &need) != B200ALG_OK || !temp_of(a[7], device, need, temp)) return false;
        if (!stream_of(a[4], device, stream)) return false;
        return released([&] {
                   if (sequence >= 0)
                       return lib.radix_sort_pairs_sequence(stream, keys.data, values.data, keys.n, code, sequence, order, temp.data, temp.n * 4);
                   return lib.radix_sort_pairs(stream, keys.data, values.data, keys.n, code, values.bytes, order, temp.data, temp.n * 4);
               }) == B200ALG_OK;
    });
}

// scan(device, code, op, inclusive, stream, input, output, temp)
PyObject *scan(PyObject *, PyObject *const *a, Py_ssize_t count) {
    return guarded([&] {
        const int device = count == 8 ? device_of(a[0]) : -1;
        const int code = int_of(a[1]), op = int_of(a[2]), inclusive = int_of(a[3]);
        View in, out, temp;
        void *stream;
        int64_t need = 0;
        if (device < 0 || !view_of(a[5], device, code, in) || !view_of(a[6], device, code, out) || out.n < in.n) return false;
        if (lib.scan_temp_bytes(code, in.n, &need) != B200ALG_OK || !temp_of(a[7], device, need, temp)) return false;
        if (!stream_of(a[4], device, stream)) return false;
        return released([&] {
                   return lib.scan_carry(stream, in.data, in.stride, out.data, out.stride, in.n, code, op, inclusive, nullptr, temp.data,
                                         temp.n * 4);
               }) == B200ALG_OK;
    });
}

// reduce(device, code, op, stream, input, output)
PyObject *reduce(PyObject *, PyObject *const *a, Py_ssize_t count) {
    return guarded([&] {
        const int device = count == 6 ? device_of(a[0]) : -1;
        const int code = int_of(a[1]), op = int_of(a[2]);
        View in, out;
        void *stream;
        if (device < 0 || !view_of(a[4], device, code, in) || !view_of(a[5], device, code, out) || in.n < 1 || out.n < 1) return false;
        if (!stream_of(a[3], device, stream)) return false;
        return released([&] { return lib.reduce(stream, in.data, in.stride, in.n, code, op, out.data); }) == B200ALG_OK;
    });
}

PyObject *number_of(const void *p, int code) {
    switch (code) {
    case B200ALG_I32: { int32_t v; memcpy(&v, p, 4); return PyLong_FromLong(v); }
    case B200ALG_U32: { uint32_t v; memcpy(&v, p, 4); return PyLong_FromUnsignedLong(v); }
    case B200ALG_I64: { int64_t v; memcpy(&v, p, 8); return PyLong_FromLongLong(v); }
    case B200ALG_U64: { uint64_t v; memcpy(&v, p, 8); return PyLong_FromUnsignedLongLong(v); }
    case B200ALG_F32: { float v; memcpy(&v, p, 4); return PyFloat_FromDouble(v); }
    case B200ALG_F64: { double v; memcpy(&v, p, 8); return PyFloat_FromDouble(v); }
    }
    return nullptr;
}

// reduce_value(device, code, op, stream, input): the value, once the GPU has it; None: not covered
PyObject *reduce_value(PyObject *, PyObject *const *a, Py_ssize_t count) {
    PyObject *value = nullptr;
    PyObject *ok = guarded([&] {
        const int device = count == 5 ? device_of(a[0]) : -1;
        const int code = int_of(a[1]), op = int_of(a[2]);
        View in;
        void *stream;
        if (device < 0 || !view_of(a[4], device, code, in) || in.n < 1 || !stream_of(a[3], device, stream)) return false;
        void *slot = host_slot.get();
        if (!slot) return false;
        const at::Tensor out = at::empty({8}, at::TensorOptions().dtype(at::kByte).device(at::kCUDA, device));
        void *result = out.data_ptr();
        const int status = released([&]() -> int {
            const int rc = lib.reduce_to_host(stream, in.data, in.stride, in.n, code, op, result, slot);
            if (rc != B200ALG_OK) return rc;
            return cudaStreamSynchronize((cudaStream_t)stream) == cudaSuccess ? B200ALG_OK : B200ALG_CUDA_ERROR;
        });
        if (status != B200ALG_OK) return false;
        value = number_of(slot, code);
        return value != nullptr;
    });
    if (ok != Py_True) {
        Py_XDECREF(value);
        value = Py_None;
        Py_INCREF(value);
    }
    Py_DECREF(ok);
    return value;
}

// histogram(device, locator, lo, hi, stream, view, bins, overflow or None)
PyObject *histogram(PyObject *, PyObject *const *a, Py_ssize_t count) {
    return guarded([&] {
        const int device = count == 8 ? device_of(a[0]) : -1;
        const int locator = int_of(a[1]);
        const double lo = PyFloat_AsDouble(a[2]), hi = PyFloat_AsDouble(a[3]);
        View in, bins, overflow;
        void *stream;
        if (device < 0 || !view_of(a[5], device, -1, in) || !view_of(a[6], device, -1, bins) || bins.n < 1 || bins.stride != 1) return false;
        if (a[7] != Py_None && (!view_of(a[7], device, B200ALG_I32, overflow) || overflow.n < 1)) return false;
        if (!stream_of(a[4], device, stream) || PyErr_Occurred()) return false;
        return released([&] {
                   return lib.histogram(stream, in.data, in.stride, in.n, in.code, locator, lo, hi, bins.data, bins.n, bins.code,
                                        overflow.data);
               }) == B200ALG_OK;
    });
}

// unique(device, code, stream, data): the new length, once the GPU has it; a status other than success
// that the GPU reports, as a negative number (the data has changed, the call cannot be made again);
// None: not covered
PyObject *unique(PyObject *, PyObject *const *a, Py_ssize_t count) {
    PyObject *value = nullptr;
    PyObject *ok = guarded([&] {
        const int device = count == 4 ? device_of(a[0]) : -1;
        const int code = int_of(a[1]);
        View data;
        void *stream;
        int64_t need = 0;
        if (device < 0 || !view_of(a[3], device, code, data) || data.stride != 1 || !stream_of(a[2], device, stream)) return false;
        if (lib.unique_temp_bytes(code, data.n, &need) != B200ALG_OK) return false;
        int64_t *slot = (int64_t *)host_slot.get();
        if (!slot || data.n < 1) return false;
        slot[1] = B200ALG_OK;
        const at::Tensor temp = at::empty({need}, at::TensorOptions().dtype(at::kByte).device(at::kCUDA, device));
        void *t = temp.data_ptr();
        // the kernel stores the count, and a wait that ran out, straight into the host slot
        const int status = released([&]() -> int {
            const int rc = lib.unique_to_host(stream, data.data, data.n, code, slot, t, need);
            if (rc != B200ALG_OK) return rc;
            return cudaStreamSynchronize((cudaStream_t)stream) == cudaSuccess ? B200ALG_OK : B200ALG_CUDA_ERROR;
        });
        if (status != B200ALG_OK) return false;
        value = PyLong_FromLongLong(slot[1] == B200ALG_OK ? slot[0] : -slot[1]);
        return value != nullptr;
    });
    if (ok != Py_True) {
        Py_XDECREF(value);
        value = Py_None;
        Py_INCREF(value);
    }
    Py_DECREF(ok);
    return value;
}

// initialize(device, stream, view, value)
PyObject *initialize(PyObject *, PyObject *const *a, Py_ssize_t count) {
    return guarded([&] {
        const int device = count == 4 ? device_of(a[0]) : -1;
        View view;
        void *stream;
        if (device < 0 || !view_of(a[2], device, -1, view) || !stream_of(a[1], device, stream)) return false;
        alignas(8) unsigned char value[8];
        if (view.code == B200ALG_F32 || view.code == B200ALG_F64) {
            const double d = PyFloat_Check(a[3]) || PyLong_Check(a[3]) ? PyFloat_AsDouble(a[3]) : NAN;
            const float f = (float)d;
            if (!std::isfinite(d) || !std::isfinite(f)) return false;
            if (view.code == B200ALG_F32) memcpy(value, &f, 4);
            else memcpy(value, &d, 8);
        } else if (view.code == B200ALG_I32 || view.code == B200ALG_I64 || view.code == B200ALG_U32) {
            if (!PyLong_Check(a[3])) return false;
            const long long i = PyLong_AsLongLong(a[3]);
            if (PyErr_Occurred()) return false;
            if (view.code == B200ALG_I32 && i != (int32_t)i) return false;
            if (view.code == B200ALG_U32 && i != (long long)(uint32_t)i) return false;
            memcpy(value, &i, 8);
        } else {
            return false;
        }
        return released([&] { return lib.initialize(stream, view.data, view.stride, view.n, view.bytes, value); }) == B200ALG_OK;
    });
}

// bind(addresses): one address per name in ENTRY_POINTS
PyObject *bind(PyObject *, PyObject *addresses) {
    constexpr Py_ssize_t kCount = sizeof(Library) / sizeof(void *);
    void *p[kCount];
    if (!PyTuple_Check(addresses) || PyTuple_GET_SIZE(addresses) != kCount) {
        PyErr_SetString(PyExc_ValueError, "bind: wrong number of addresses");
        return nullptr;
    }
    for (Py_ssize_t i = 0; i < kCount; ++i) p[i] = PyLong_AsVoidPtr(PyTuple_GET_ITEM(addresses, i));
    if (PyErr_Occurred()) return nullptr;
    memcpy(&lib, p, sizeof(lib));
    Py_RETURN_NONE;
}

#define FAST(name) {#name, (PyCFunction)(void (*)(void))name, METH_FASTCALL, nullptr}
PyMethodDef methods[] = {{"bind", bind, METH_O, nullptr}, FAST(sort_keys), FAST(sort_pairs), FAST(scan), FAST(reduce), FAST(reduce_value),
                         FAST(histogram), FAST(unique), FAST(initialize), {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_host", "Host path of the algorithm calls.", -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__host(void) {
    PyObject *m = PyModule_Create(&module);
    constexpr Py_ssize_t kCount = sizeof(kEntryPoints) / sizeof(kEntryPoints[0]);
    PyObject *names = m ? PyTuple_New(kCount) : nullptr;
    for (Py_ssize_t i = 0; names && i < kCount; ++i) {
        PyObject *name = PyUnicode_FromString(kEntryPoints[i]);
        if (!name) Py_CLEAR(names);
        else PyTuple_SET_ITEM(names, i, name);
    }
    if (!names || PyModule_AddObject(m, "ENTRY_POINTS", names) < 0) {
        Py_XDECREF(names);
        Py_XDECREF(m);
        return nullptr;
    }
    return m;
}
