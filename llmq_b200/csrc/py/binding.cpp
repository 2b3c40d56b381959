// Typed Python entry points of the kernels that are launched most often, and the argument check of the custom ops.
//
// ctypes builds an object per argument (0.16 us each, a GEMM has thirty) and the check of the custom ops reads six attributes of every tensor: for a
// GEMM call 9.6 us of Python around 4.5 us of launch, which is longer than many of these kernels run.  Here a call unpacks tensors and numbers by
// the types of the C function, appends the current stream and calls it with the GIL released (a launch may wait for room in the queue, and
// another thread of the process may have to launch what makes that room).  The shapes, types and refusals of a call stay in ops/kernels.py.
//
// us of host time, one x86 core, through ctypes and checks in Python / with this module: matmul 14.1 / 8.1, rope_forward 8.5 / 4.4, attention_backward 14.0 / 7.5.
#include <Python.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/python_variable.h>
#include <climits>
#include <string>
#include <utility>
#include <vector>

namespace {

typedef void* P;               // tensor, address or None
typedef long long LL;

// get(): the C value; with an exception set, ok becomes false
template <typename T> struct Arg;
template <> struct Arg<P> {
    static constexpr char code = 'p';
    static P get(PyObject* o, bool& ok) {
        if (o == Py_None) return nullptr;
        if (THPVariable_Check(o)) return THPVariable_Unpack(o).data_ptr();
        if (PyLong_Check(o)) {
            P v = PyLong_AsVoidPtr(o);
            ok = v || !PyErr_Occurred();
            return v;
        }
        ok = false;
        PyErr_Format(PyExc_TypeError, "expected a tensor, an address or None, got %s", Py_TYPE(o)->tp_name);
        return nullptr;
    }
};
template <> struct Arg<int> {
    static constexpr char code = 'i';
    static int get(PyObject* o, bool& ok) {
        const long v = PyLong_AsLong(o);
        if (v == -1) ok = !PyErr_Occurred();
        if (v < INT_MIN || v > INT_MAX) { ok = false; PyErr_SetString(PyExc_OverflowError, "size does not fit a C int"); }
        return static_cast<int>(v);
    }
};
template <> struct Arg<unsigned int> {
    static constexpr char code = 'u';
    static unsigned int get(PyObject* o, bool& ok) {
        const unsigned long v = PyLong_AsUnsignedLong(o);
        if (v > UINT_MAX) {                                  // also where the conversion failed
            ok = false;
            if (!PyErr_Occurred()) PyErr_SetString(PyExc_OverflowError, "value does not fit an unsigned C int");
        }
        return static_cast<unsigned int>(v);
    }
};
template <> struct Arg<LL> {
    static constexpr char code = 'l';
    static LL get(PyObject* o, bool& ok) {
        const LL v = PyLong_AsLongLong(o);
        if (v == -1) ok = !PyErr_Occurred();
        return v;
    }
};
template <> struct Arg<double> {
    static constexpr char code = 'd';
    static double get(PyObject* o, bool& ok) {
        const double v = PyFloat_AsDouble(o);
        if (v == -1.) ok = !PyErr_Occurred();
        return v;
    }
};
template <> struct Arg<float> {
    static constexpr char code = 'f';
    static float get(PyObject* o, bool& ok) { return static_cast<float>(Arg<double>::get(o, ok)); }
};

template <int Id, typename... A>
struct Entry {
    typedef int (*Fn)(A..., cudaStream_t);
    static inline Fn fn = nullptr;

    static PyObject* call(PyObject*, PyObject* const* args, Py_ssize_t n) {
        if (!fn || n != static_cast<Py_ssize_t>(sizeof...(A))) {
            PyErr_Format(PyExc_TypeError, fn ? "expected %d arguments, got %zd" : "not bound (%d arguments, got %zd)", static_cast<int>(sizeof...(A)), n);
            return nullptr;
        }
        return invoke(args, std::index_sequence_for<A...>{});
    }
    template <size_t... I>
    static PyObject* invoke(PyObject* const* args, std::index_sequence<I...>) {
        try {
            bool ok = true;
            std::tuple<A...> v{(ok ? Arg<A>::get(args[I], ok) : A())...};      // in order, up to the first that fails
            if (!ok) return nullptr;
            const cudaStream_t stream = c10::cuda::getCurrentCUDAStream().stream();
            int rc;
            Py_BEGIN_ALLOW_THREADS
            rc = fn(std::get<I>(v)..., stream);
            Py_END_ALLOW_THREADS
            return PyLong_FromLong(rc);
        } catch (const std::exception& e) {
            if (!PyErr_Occurred()) PyErr_SetString(PyExc_RuntimeError, e.what());
            return nullptr;
        }
    }
    static std::string codes() { return std::string{Arg<A>::code...}; }
};

// name, types of the arguments without the stream, which is the last one of every function
#define LLMQ_ENTRIES(X)                                                                                                              \
    X(llmq_gemm_ready, P, P, P, P, int, int, int, int, int, int, int, LL, LL, LL, int, int, int, P, P, float, P, P, int, P, unsigned int, int, double, P, LL) \
    X(llmq_gemm_split_mode, P, int, int, int, int, LL, int, int)                                                                    \
    X(llmq_rmsnorm_forward, P, P, P, P, P, P, P, float, int, int, int, P, P, P)                                                      \
    X(llmq_rmsnorm_backward, P, P, P, P, P, P, P, int, int, int, P, int, int, P)                                                     \
    X(llmq_swiglu_forward, P, P, P, LL, int, int, P, P, P, int)                                                                      \
    X(llmq_swiglu_backward, P, P, P, LL, int, int, P, int)                                                                           \
    X(llmq_rope, P, P, P, int, int, int, int, int, int, int, P, int)                                                                 \
    X(llmq_attention_forward, P, P, P, int, int, int, int, int, P, P)                                                                \
    X(llmq_attention_backward, P, P, P, P, P, P, int, int, int, int, int, P)                                                         \
    X(llmq_bias_backward, P, P, P, LL, int, int, P, P, int, int, int)                                                                \
    X(llmq_abs_max, P, P, LL, int, int)                                                                                              \
    X(llmq_quantize, P, P, P, P, LL, int, int, int)                                                                                  \
    X(llmq_quantize_transpose, P, P, P, P, P, int, int, int, int)                                                                    \
    X(llmq_transpose, P, P, P, P, int, int, int, int)                                                                                \
    X(llmq_fused_classifier, P, P, P, P, float, float, int, int, LL, int, int)                                                       \
    X(llmq_norm_squared, P, P, LL, int, int)                                                                                         \
    X(llmq_deterministic_sum, P, P, int)                                                                                             \
    X(llmq_norm_sum_finish, P, P, int, float, P)                                                                                     \
    X(llmq_norm_finish, P, float, P)                                                                                                 \
    X(llmq_adamw_hyper, P, P, P, P, P, LL, float, float, float, int, float, float, P, P, unsigned int, LL, int, int, int, int, int, P)

enum {
#define X(name, ...) k_##name,
    LLMQ_ENTRIES(X)
#undef X
};
#define X(name, ...) typedef Entry<k_##name, __VA_ARGS__> E_##name;
LLMQ_ENTRIES(X)
#undef X

// bind(name, address): the C function behind an entry
PyObject* bind(PyObject*, PyObject* const* args, Py_ssize_t n) {
    const char* name = n == 2 ? PyUnicode_AsUTF8(args[0]) : nullptr;
    void* address = name ? PyLong_AsVoidPtr(args[1]) : nullptr;
    if (!name || PyErr_Occurred()) {
        if (!PyErr_Occurred()) PyErr_SetString(PyExc_TypeError, "bind(name, address)");
        return nullptr;
    }
#define X(f, ...) if (std::string(name) == #f) { E_##f::fn = reinterpret_cast<E_##f::Fn>(address); Py_RETURN_NONE; }
    LLMQ_ENTRIES(X)
#undef X
    PyErr_Format(PyExc_KeyError, "%s", name);
    return nullptr;
}

// signatures(): name -> a letter per argument (p pointer, i int, u unsigned, l long long, f float, d double)
PyObject* signatures(PyObject*, PyObject*) {
    PyObject* d = PyDict_New();
    if (!d) return nullptr;
#define X(f, ...) { PyObject* v = PyUnicode_FromString(E_##f::codes().c_str()); if (!v || PyDict_SetItemString(d, #f, v) < 0) { Py_XDECREF(v); Py_DECREF(d); return nullptr; } Py_DECREF(v); }
    LLMQ_ENTRIES(X)
#undef X
    return d;
}

// What a custom op wants of its arguments
struct Spec {
    std::vector<PyObject*> kinds;       // nullptr: tensor, else the exact type (referenced for good: specs live as long as the process)
    std::vector<char> optional;
    std::vector<Py_ssize_t> mutated;
    Py_ssize_t required;
};

Spec* spec_of(PyObject* capsule) { return static_cast<Spec*>(PyCapsule_GetPointer(capsule, "llmq_spec")); }

// spec(kinds, optional, required, mutated)
PyObject* make_spec(PyObject*, PyObject* const* args, Py_ssize_t n) {
    if (n != 4 || !PyTuple_Check(args[0]) || !PyTuple_Check(args[1]) || !PyTuple_Check(args[3]) || PyTuple_GET_SIZE(args[0]) != PyTuple_GET_SIZE(args[1])) {
        PyErr_SetString(PyExc_TypeError, "spec(kinds, optional, required, mutated)");
        return nullptr;
    }
    Spec* s = new Spec;
    for (Py_ssize_t i = 0; i < PyTuple_GET_SIZE(args[0]); ++i) {
        PyObject* k = PyTuple_GET_ITEM(args[0], i);
        Py_INCREF(k);
        s->kinds.push_back(k == Py_None ? nullptr : k);
        s->optional.push_back(PyObject_IsTrue(PyTuple_GET_ITEM(args[1], i)) == 1);
    }
    for (Py_ssize_t i = 0; i < PyTuple_GET_SIZE(args[3]); ++i) s->mutated.push_back(PyLong_AsSsize_t(PyTuple_GET_ITEM(args[3], i)));
    s->required = PyLong_AsSsize_t(args[2]);
    if (PyErr_Occurred()) { delete s; return nullptr; }
    return PyCapsule_New(s, "llmq_spec", nullptr);
}

// plain(spec, args): every argument is of exactly the schema's type, and every tensor one that nothing but its own kernel has to see: CPU or CUDA,
// strided, no subclass, gradient, inference or lazy bit, and not a zero tensor, which has no memory until the dispatcher gives it some
PyObject* plain(PyObject*, PyObject* const* args, Py_ssize_t n) {
    const Spec* s = n == 2 && PyTuple_Check(args[1]) ? spec_of(args[0]) : nullptr;
    if (!s) {
        if (!PyErr_Occurred()) PyErr_SetString(PyExc_TypeError, "plain(spec, args)");
        return nullptr;
    }
    const Py_ssize_t given = PyTuple_GET_SIZE(args[1]);
    if (given < s->required || given > static_cast<Py_ssize_t>(s->kinds.size())) Py_RETURN_FALSE;
    try {
        for (Py_ssize_t i = 0; i < given; ++i) {
            PyObject* v = PyTuple_GET_ITEM(args[1], i);
            if (s->kinds[i]) {
                if (reinterpret_cast<PyObject*>(Py_TYPE(v)) != s->kinds[i]) Py_RETURN_FALSE;
                continue;
            }
            if (v == Py_None && s->optional[i]) continue;
            if (reinterpret_cast<PyObject*>(Py_TYPE(v)) != THPVariableClass) Py_RETURN_FALSE;
            const at::Tensor& t = THPVariable_Unpack(v);
            if (!t.defined() || t.requires_grad() || t.layout() != at::kStrided || t.is_inference() || t.is_neg() || t._is_zerotensor() || !(t.is_cuda() || t.is_cpu()))
                Py_RETURN_FALSE;
        }
    } catch (const std::exception&) {
        PyErr_Clear();
        Py_RETURN_FALSE;               // the dispatcher says what is wrong
    }
    Py_RETURN_TRUE;
}

// bump(spec, args): raises the version of every tensor that the op writes, for arguments that were plain
PyObject* bump(PyObject*, PyObject* const* args, Py_ssize_t n) {
    const Spec* s = n == 2 && PyTuple_Check(args[1]) ? spec_of(args[0]) : nullptr;
    if (!s) {
        if (!PyErr_Occurred()) PyErr_SetString(PyExc_TypeError, "bump(spec, args)");
        return nullptr;
    }
    const Py_ssize_t given = PyTuple_GET_SIZE(args[1]);
    try {
        for (const Py_ssize_t i : s->mutated) {
            if (i >= given) continue;
            PyObject* v = PyTuple_GET_ITEM(args[1], i);
            if (THPVariable_Check(v)) THPVariable_Unpack(v).unsafeGetTensorImpl()->bump_version();
        }
    } catch (const std::exception& e) {
        if (!PyErr_Occurred()) PyErr_SetString(PyExc_RuntimeError, e.what());
        return nullptr;
    }
    Py_RETURN_NONE;
}

#define FAST(f) reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)(void)>(f))
PyMethodDef methods[] = {
    {"bind", FAST(bind), METH_FASTCALL, nullptr}, {"signatures", signatures, METH_NOARGS, nullptr}, {"spec", FAST(make_spec), METH_FASTCALL, nullptr},
    {"plain", FAST(plain), METH_FASTCALL, nullptr}, {"bump", FAST(bump), METH_FASTCALL, nullptr},
#define X(name, ...) {#name, FAST(E_##name::call), METH_FASTCALL, nullptr},
    LLMQ_ENTRIES(X)
#undef X
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "llmq_b200_binding", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

// torch_version: the one that this file was compiled against, which the loader compares with the one at hand
PyMODINIT_FUNC PyInit_llmq_b200_binding() {
    PyObject* m = PyModule_Create(&module);
    if (m && PyModule_AddStringConstant(m, "torch_version", LLMQ_TORCH_VERSION) < 0) Py_CLEAR(m);
    return m;
}
