// Host side of the layer classes in native code: the calls into libaether_b200.so with tensors, numbers and None as
// arguments, and the allocation of output arrays.
//
// A training step of the reference's small networks is some fifty kernels of two to five microseconds; through ctypes
// every call cost ten to forty microseconds of Python (argument objects, conversions, stream and device queries,
// torch.empty), so the GPU waited for the host.  Here a call converts its arguments by the C prototype (include/
// aether_b200.h is the single source of the signatures), takes the current stream, releases the GIL around the library
// call and raises on a non-zero return code: about a microsecond plus the kernel launches.
//
// The library itself is not linked: bind(path) resolves the entry points in the copy _lib.py has loaded.
#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDACachingAllocator.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>
#include <dlfcn.h>
#include <string.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <tuple>
#include <type_traits>
#include <utility>
#include <vector>

#include "../../include/aether_b200.h"

namespace {

PyObject* g_error = nullptr;                      // AetherError, handed in by bind()
const char* (*g_last_error)() = nullptr;

// ---------------------------------------------------------------------------------- arguments
template <typename T>
struct Arg;                                       // from(object, value): false with a Python error set on failure

template <typename T>
struct Arg<T*> {                                  // device array: a tensor, None, or an address
    static bool from(PyObject* o, T*& v) {
        if (o == Py_None) { v = nullptr; return true; }
        if (THPVariable_Check(o)) { v = static_cast<T*>(const_cast<void*>(THPVariable_Unpack(o).const_data_ptr())); return true; }
        void* p = PyLong_AsVoidPtr(o);
        if (p == nullptr && PyErr_Occurred()) return false;
        v = static_cast<T*>(p);
        return true;
    }
};
template <>
struct Arg<const AetherConvDesc*> {               // the bytes of an AetherConvDesc
    static bool from(PyObject* o, const AetherConvDesc*& v) {
        if (!PyBytes_Check(o) || PyBytes_GET_SIZE(o) != (Py_ssize_t)sizeof(AetherConvDesc)) {
            PyErr_SetString(PyExc_TypeError, "expected the bytes of an AetherConvDesc");
            return false;
        }
        v = reinterpret_cast<const AetherConvDesc*>(PyBytes_AS_STRING(o));
        return true;
    }
};
template <>
struct Arg<float> {
    static bool from(PyObject* o, float& v) {
        const double d = PyFloat_AsDouble(o);
        if (d == -1.0 && PyErr_Occurred()) return false;
        v = (float)d;
        return true;
    }
};
template <typename T>
bool integer(PyObject* o, T& v) {
    const long long n = PyLong_AsLongLong(o);
    if (n == -1 && PyErr_Occurred()) return false;
    v = (T)n;
    return true;
}
template <>
struct Arg<int> {
    static bool from(PyObject* o, int& v) { return integer(o, v); }
};
template <>
struct Arg<int64_t> {
    static bool from(PyObject* o, int64_t& v) { return integer(o, v); }
};
template <>
struct Arg<uint64_t> {                            // (also size_t)
    static bool from(PyObject* o, uint64_t& v) {
        v = PyLong_AsUnsignedLongLongMask(o);
        return !(v == (uint64_t)-1 && PyErr_Occurred());
    }
};

PyObject* fail(int rc, const char* what) {
    const char* said = g_last_error ? g_last_error() : "";
    if (rc == AETHER_E_BAD_ARG) PyErr_Format(PyExc_ValueError, "%s: %s", what, said);
    else PyErr_Format(g_error, "%s failed (%d): %s", what, rc, said);
    return nullptr;
}

void* current_stream() { return static_cast<void*>(c10::cuda::getCurrentCUDAStream().stream()); }

// ---------------------------------------------------------------------------------- entry points
// Every entry point ends in `void* stream`, which is not an argument of the Python function.
template <typename Sig>
struct Entry;
template <typename... A>
struct Entry<int (*)(A...)> {
    using Fn = int (*)(A...);
    using Args = std::tuple<A...>;
    static constexpr size_t N = sizeof...(A) - 1;

    template <size_t... I>
    static PyObject* call(Fn fn, const char* name, PyObject* const* args, std::index_sequence<I...>) {
        Args a;
        if (!(Arg<std::tuple_element_t<I, Args>>::from(args[I], std::get<I>(a)) && ...)) return nullptr;
        std::get<N>(a) = current_stream();
        int rc;
        Py_BEGIN_ALLOW_THREADS
        rc = std::apply(fn, a);
        Py_END_ALLOW_THREADS
        if (rc != 0) return fail(rc, name);
        Py_RETURN_NONE;
    }
    static PyObject* run(void* fn, const char* name, PyObject* const* args, Py_ssize_t n) {
        if (fn == nullptr) {
            PyErr_Format(g_error ? g_error : PyExc_RuntimeError, "%s: the library has not been bound", name);
            return nullptr;
        }
        if (n != (Py_ssize_t)N) {
            PyErr_Format(PyExc_TypeError, "%s takes %zd arguments (%zd given)", name, (Py_ssize_t)N, n);
            return nullptr;
        }
        HANDLE_TH_ERRORS                          // (the stream query throws on a machine without a device)
        return call(reinterpret_cast<Fn>(fn), name, args, std::make_index_sequence<N>{});
        END_HANDLE_TH_ERRORS
    }
};

#define ENTRY_POINTS(X)                                                                                                \
    X(aether_conv2d_fwd_ex) X(aether_conv2d_bwd_ex) X(aether_conv2d_filter_copies) X(aether_conv2d_pool_fwd) X(aether_bn_fwd_train) X(aether_bn_fwd_train_partials)             \
    X(aether_bn_fwd_eval) X(aether_bn_bwd) X(aether_bn_act_fwd_train) X(aether_bn_act_fwd_eval) X(aether_bn_act_bwd)   \
    X(aether_bn_act_pool_fwd_copy) X(aether_chain_fwd) X(aether_pool_fwd) X(aether_pool_bwd) X(aether_leaky_relu_fwd)                      \
    X(aether_leaky_relu_bwd) X(aether_leaky_relu_fwd_mask) X(aether_leaky_relu_bwd_mask) X(aether_channel_scale) X(aether_dropout_fwd) X(aether_mul) X(aether_adam_step)           \
    X(aether_adam_step_dev) X(aether_dropout_fwd_dev) X(aether_channel_mask_dev) X(aether_regularizer_grad)            \
    X(aether_regularizer_loss) X(aether_copy) X(aether_conv2d_act_fwd) X(aether_act_bwd_copy) X(aether_head_softmax_fwd) X(aether_head_cce_bwd_ex) X(aether_softmax_cce) X(aether_softmax_cce_i64) X(aether_softmax_bwd) X(aether_softmax_cce_targets)

#define DECLARE(name)                                                                                                  \
    void* fn_##name = nullptr;                                                                                         \
    PyObject* py_##name(PyObject*, PyObject* const* args, Py_ssize_t n) {                                              \
        return Entry<decltype(&name)>::run(fn_##name, #name, args, n);                                                 \
    }
ENTRY_POINTS(DECLARE)

// Entry points that report a number through an `int*` argument (the rows of column sums a backward pass wrote): the Python
// function does not have that argument and returns the number.
template <typename Sig>
struct EntryOut;
template <typename... A>
struct EntryOut<int (*)(A...)> {
    using Fn = int (*)(A...);
    using Args = std::tuple<A...>;
    static constexpr size_t N = sizeof...(A) - 1;

    template <size_t I>
    static bool get(Args& a, PyObject* const* args, int& next, int* out) {
        if constexpr (std::is_same_v<std::tuple_element_t<I, Args>, int*>) {
            std::get<I>(a) = out;
            return true;
        } else {
            return Arg<std::tuple_element_t<I, Args>>::from(args[next++], std::get<I>(a));
        }
    }
    template <size_t... I>
    static PyObject* call(Fn fn, const char* name, PyObject* const* args, std::index_sequence<I...>) {
        Args a;
        int next = 0, out = 0, rc;
        if (!(get<I>(a, args, next, &out) && ...)) return nullptr;
        std::get<N>(a) = current_stream();
        Py_BEGIN_ALLOW_THREADS
        rc = std::apply(fn, a);
        Py_END_ALLOW_THREADS
        return rc != 0 ? fail(rc, name) : PyLong_FromLong(out);
    }
    static PyObject* run(void* fn, const char* name, PyObject* const* args, Py_ssize_t n) {
        if (fn == nullptr || n != (Py_ssize_t)N - 1) {
            PyErr_Format(PyExc_TypeError, "%s takes %zd arguments (%zd given) and a bound library", name, (Py_ssize_t)N - 1, n);
            return nullptr;
        }
        HANDLE_TH_ERRORS
        return call(reinterpret_cast<Fn>(fn), name, args, std::make_index_sequence<N>{});
        END_HANDLE_TH_ERRORS
    }
};
#define ENTRY_POINTS_OUT(X) X(aether_bn_act_pool_bwd_copy) X(aether_chain_bwd)
#define DECLARE_OUT(name)                                                                                              \
    void* fn_##name = nullptr;                                                                                         \
    PyObject* py_##name(PyObject*, PyObject* const* args, Py_ssize_t n) {                                              \
        return EntryOut<decltype(&name)>::run(fn_##name, #name, args, n);                                              \
    }
ENTRY_POINTS_OUT(DECLARE_OUT)

// aether_adam_steps(arrays, lr, beta1, beta2, eps, bias_corr1, bias_corr2, grad_scale): `arrays` is a flat list of
// (parameters, gradients, momentums, cache) per tensor.
void* fn_adam_steps = nullptr;
void* fn_upload = nullptr;
PyObject* py_adam_steps(PyObject*, PyObject* const* args, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    static const char* name = "aether_adam_steps";
    if (fn_adam_steps == nullptr || n != 8 || !PyList_Check(args[0]) || PyList_GET_SIZE(args[0]) % 4 != 0) {
        PyErr_Format(PyExc_TypeError, "%s takes a list of (p, g, m, v) arrays, seven numbers and a bound library", name);
        return nullptr;
    }
    const Py_ssize_t count = PyList_GET_SIZE(args[0]) / 4;
    std::vector<AetherAdamTensor> t((size_t)count);
    for (Py_ssize_t i = 0; i < count; ++i) {
        PyObject* p = PyList_GET_ITEM(args[0], 4 * i);
        if (!THPVariable_Check(p)) {
            PyErr_Format(PyExc_TypeError, "%s: parameters must be tensors", name);
            return nullptr;
        }
        t[i].n = THPVariable_Unpack(p).numel();
        if (!Arg<float*>::from(p, t[i].p) || !Arg<const float*>::from(PyList_GET_ITEM(args[0], 4 * i + 1), t[i].g) ||
            !Arg<float*>::from(PyList_GET_ITEM(args[0], 4 * i + 2), t[i].m) || !Arg<float*>::from(PyList_GET_ITEM(args[0], 4 * i + 3), t[i].v))
            return nullptr;
    }
    float f[7];
    for (int i = 0; i < 7; ++i)
        if (!Arg<float>::from(args[1 + i], f[i])) return nullptr;
    void* st = current_stream();
    int rc;
    Py_BEGIN_ALLOW_THREADS
    rc = reinterpret_cast<decltype(&aether_adam_steps)>(fn_adam_steps)(t.data(), (int)count, f[0], f[1], f[2], f[3], f[4], f[5], f[6], st);
    Py_END_ALLOW_THREADS
    if (rc != 0) return fail(rc, name);
    Py_RETURN_NONE;
    END_HANDLE_TH_ERRORS
}

PyObject* py_bind(PyObject*, PyObject* args) {
    const char* path;
    PyObject* error;
    if (!PyArg_ParseTuple(args, "sO", &path, &error)) return nullptr;
    void* h = dlopen(path, RTLD_NOW | RTLD_LOCAL);
    if (h == nullptr) {
        PyErr_Format(PyExc_OSError, "%s: %s", path, dlerror());
        return nullptr;
    }
#define RESOLVE(name)                                                                          \
    if ((fn_##name = dlsym(h, #name)) == nullptr) {                                            \
        PyErr_Format(error, "%s does not export %s: rebuild it with `python -m aether_ml_b200.build`", path, #name); \
        return nullptr;                                                                        \
    }
    ENTRY_POINTS(RESOLVE)
    ENTRY_POINTS_OUT(RESOLVE)
    fn_adam_steps = dlsym(h, "aether_adam_steps");
    fn_upload = dlsym(h, "aether_upload");
    g_last_error = reinterpret_cast<const char* (*)()>(dlsym(h, "aether_last_error"));
    Py_XDECREF(g_error);
    Py_INCREF(error);
    g_error = error;
    Py_RETURN_NONE;
}

// ---------------------------------------------------------------------------------- arrays
// Every function below translates what torch may throw (a tensor of inference mode has no version counter, a sparse one no
// contiguity, a wrapped one no address): an exception that left a C callback would end the process.  The ones that every
// layer calls several times set the translation up only where something is thrown.
PyObject* translated() {                          // (from a catch block)
    HANDLE_TH_ERRORS
    throw;
    END_HANDLE_TH_ERRORS
}

// The argument itself when it is a contiguous fp32 CUDA tensor, else None.
PyObject* py_ready(PyObject*, PyObject* o) try {
    if (THPVariable_Check(o)) {
        const at::Tensor& t = THPVariable_Unpack(o);
        if (t.is_cuda() && t.scalar_type() == at::kFloat && t.is_contiguous()) {
            Py_INCREF(o);
            return o;
        }
    }
    Py_RETURN_NONE;
} catch (...) {
    return translated();
}

PyObject* py_device(PyObject*, PyObject*) {
    HANDLE_TH_ERRORS
    return PyLong_FromLong(c10::cuda::current_device());
    END_HANDLE_TH_ERRORS
}

PyObject* new_array(at::IntArrayRef sizes, at::ScalarType type) {
    HANDLE_TH_ERRORS
    return THPVariable_Wrap(at::detail::empty_cuda(sizes, type, c10::Device(c10::DeviceType::CUDA, c10::cuda::current_device()), std::nullopt));
    END_HANDLE_TH_ERRORS
}

template <at::ScalarType TYPE>
PyObject* py_empty(PyObject*, PyObject* shape) {
    if (!PyTuple_Check(shape) || PyTuple_GET_SIZE(shape) > 8) {
        PyErr_SetString(PyExc_TypeError, "expected a shape of at most eight dimensions");
        return nullptr;
    }
    int64_t d[8];
    const Py_ssize_t n = PyTuple_GET_SIZE(shape);
    for (Py_ssize_t i = 0; i < n; ++i)
        if (!integer(PyTuple_GET_ITEM(shape, i), d[i])) return nullptr;
    return new_array(at::IntArrayRef(d, (size_t)n), TYPE);
}

PyObject* py_empty_like(PyObject*, PyObject* o) {
    HANDLE_TH_ERRORS
    if (!THPVariable_Check(o)) {
        PyErr_SetString(PyExc_TypeError, "expected a tensor");
        return nullptr;
    }
    const at::Tensor& t = THPVariable_Unpack(o);
    return new_array(t.sizes(), t.scalar_type());
    END_HANDLE_TH_ERRORS
}

// upload(values, like_shape): a new array of that shape with the fp32 values of a contiguous host buffer.
PyObject* py_upload(PyObject*, PyObject* const* args, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    if (fn_upload == nullptr || n != 2) {
        PyErr_SetString(PyExc_TypeError, "upload takes a host array and a shape, and needs a bound library");
        return nullptr;
    }
    void* const stream = current_stream();        // (nothing throws while the buffer is held)
    Py_buffer b;
    if (PyObject_GetBuffer(args[0], &b, PyBUF_C_CONTIGUOUS | PyBUF_FORMAT) != 0) return nullptr;
    PyObject* t = nullptr;
    if (b.format == nullptr || strcmp(b.format, "f") != 0) {
        PyErr_SetString(PyExc_TypeError, "upload: expected fp32 values");
    } else if ((t = py_empty<at::kFloat>(nullptr, args[1])) != nullptr) {
        const at::Tensor& a = THPVariable_Unpack(t);
        int rc = AETHER_E_BAD_ARG;
        if (a.numel() == b.len / 4 && a.numel() < (1 << 30))
            rc = reinterpret_cast<decltype(&aether_upload)>(fn_upload)(static_cast<const float*>(b.buf), static_cast<float*>(a.mutable_data_ptr()),
                                                                       (int)a.numel(), stream);
        if (rc != 0) {
            Py_DECREF(t);
            t = fail(rc, "aether_upload");
        }
    }
    PyBuffer_Release(&b);
    return t;
    END_HANDLE_TH_ERRORS
}

// Identity of an array's contents as far as the host can tell: address, elements, in-place changes so far, row length.
PyObject* py_tag(PyObject*, PyObject* o) try {
    if (!THPVariable_Check(o)) {
        PyErr_SetString(PyExc_TypeError, "expected a tensor");
        return nullptr;
    }
    const at::Tensor& t = THPVariable_Unpack(o);
    return Py_BuildValue("(nLLL)", (Py_ssize_t) reinterpret_cast<intptr_t>(t.const_data_ptr()), (long long)t.numel(),
                         (long long)t._version(), (long long)(t.dim() > 0 ? t.size(-1) : 1));
} catch (...) {
    return translated();
}

// same(tensor, tag): whether tag(tensor) starts with the values of `tag`, without building a tuple to compare.
PyObject* py_same(PyObject*, PyObject* const* args, Py_ssize_t n) try {
    if (n != 2 || !THPVariable_Check(args[0]) || !PyTuple_Check(args[1]) || PyTuple_GET_SIZE(args[1]) > 4) {
        PyErr_SetString(PyExc_TypeError, "expected a tensor and a tag");
        return nullptr;
    }
    const at::Tensor& t = THPVariable_Unpack(args[0]);
    const long long now[4] = {(long long)reinterpret_cast<intptr_t>(t.const_data_ptr()), (long long)t.numel(), (long long)t._version(),
                              (long long)(t.dim() > 0 ? t.size(-1) : 1)};
    for (Py_ssize_t i = 0; i < PyTuple_GET_SIZE(args[1]); ++i) {
        long long v;
        if (!integer(PyTuple_GET_ITEM(args[1], i), v)) return nullptr;
        if (v != now[i]) Py_RETURN_FALSE;
    }
    Py_RETURN_TRUE;
} catch (...) {
    return translated();
}

// In-place changes so far of a tensor whose every writer counts them, else -1: inference mode counts none, and memory that another library owns (an array
// handed in by its address) is changed by that library's kernels.
PyObject* py_counted(PyObject*, PyObject* o) try {
    if (!THPVariable_Check(o)) {
        PyErr_SetString(PyExc_TypeError, "expected a tensor");
        return nullptr;
    }
    const at::Tensor& t = THPVariable_Unpack(o);
    const bool own = !t.is_inference() && t.has_storage() && t.storage().data_ptr().get_deleter() == c10::cuda::CUDACachingAllocator::get()->raw_deleter();
    return PyLong_FromLongLong(own ? (long long)t._version() : -1);
} catch (...) {
    return translated();
}

#define METHOD(name) {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_##name)), METH_FASTCALL, nullptr},
PyMethodDef methods[] = {
    ENTRY_POINTS(METHOD)
    ENTRY_POINTS_OUT(METHOD)
    {"aether_adam_steps", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_adam_steps)), METH_FASTCALL, nullptr},
    {"upload", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_upload)), METH_FASTCALL, "upload(host fp32 buffer, shape): a new array with those values"},
    {"device", py_device, METH_NOARGS, "index of the current device"},
    {"bind", py_bind, METH_VARARGS, "bind(path, AetherError): resolve the entry points in the library at `path`"},
    {"ready", py_ready, METH_O, "the argument when it is a contiguous fp32 CUDA tensor, else None"},
    {"empty", py_empty<at::kFloat>, METH_O, "uninitialised fp32 array on the current device"},
    {"empty_u8", py_empty<at::kByte>, METH_O, "uninitialised uint8 array on the current device"},
    {"empty_i32", py_empty<at::kInt>, METH_O, "uninitialised int32 array on the current device"},
    {"empty_like", py_empty_like, METH_O, "uninitialised contiguous array of the argument's shape and type on the current device"},
    {"tag", py_tag, METH_O, "(address, elements, version, row length) of a tensor"},
    {"counted", py_counted, METH_O, "in-place changes of a tensor so far, -1 where not every writer counts them"},
    {"same", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_same)), METH_FASTCALL, "whether a tensor still has the values of a tag"},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_host", "native host path of aether_ml_b200", -1, methods};

}  // namespace

PyMODINIT_FUNC PyInit__host(void) { return PyModule_Create(&module); }
