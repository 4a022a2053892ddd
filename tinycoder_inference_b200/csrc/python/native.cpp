// native.cpp -- the Python front's way into the C ABI: CPython functions that take torch tensors,
// read their device addresses and the current stream, and make the call.
//
// What bounds it: an eager decode step is a handful of launches of a few microseconds each, so what the
// host spends in front of a launch is on the critical path.  Through ctypes an attend call of nine
// arguments cost 7 us before its first launch (tensor attribute look-ups, c_void_p objects, a Stream object,
// argument conversion); here the conversion of a call is a fraction of a microsecond.
//
// Every wrapper returns the C function's code as an int; ops.py turns a non-zero one into an exception.
// Integers wrap like ctypes' unsigned types do, None is a null pointer, a tensor has to be
// contiguous and on a CUDA device.  The interpreter lock is not held during a call that may block (a launch into a full
// queue, the synchronise at the end of `clear`): other Python threads go on, and a stream that waits for one of them
// gets there.  What torch throws on the way (a tensor without storage, no device) becomes the
// Python exception that torch itself would raise.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <cstring>
#include <type_traits>
#include <utility>

#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include "../../../include/tc_attn.h"

namespace {

tc_stream currentStream() { return c10::cuda::getCurrentCUDAStream().stream(); }

// ---- one argument ---------------------------------------------------------------------------
bool toPointer(PyObject *o, void **out) {
    if (o == Py_None) {
        *out = nullptr;
        return true;
    }
    if (!THPVariable_Check(o)) {
        PyErr_Format(PyExc_TypeError, "tensor or None expected, got %s", Py_TYPE(o)->tp_name);
        return false;
    }
    const at::Tensor &t = THPVariable_Unpack(o);
    if (!t.is_cuda() || !t.is_contiguous()) {
        PyErr_SetString(PyExc_AssertionError, "device-resident contiguous tensor required");
        return false;
    }
    *out = t.data_ptr();
    return true;
}
// the address alone (the batch descriptor's fields: layout is the caller's business there)
bool toAddress(PyObject *o, const void **out) {
    *out = nullptr;
    if (o == Py_None) return true;
    if (!THPVariable_Check(o)) {
        PyErr_Format(PyExc_TypeError, "tensor or None expected, got %s", Py_TYPE(o)->tp_name);
        return false;
    }
    *out = THPVariable_Unpack(o).data_ptr();
    return true;
}
template <typename T>
bool toArg(PyObject *o, T *out) {
    if constexpr (std::is_same_v<T, tc_kv_session *> || std::is_same_v<T, const tc_kv_session *>) {
        *out = static_cast<tc_kv_session *>(PyLong_AsVoidPtr(o));
    } else if constexpr (std::is_pointer_v<T>) {
        void *p = nullptr;
        if (!toPointer(o, &p)) return false;
        *out = static_cast<T>(p);
    } else if constexpr (std::is_floating_point_v<T>) {
        *out = static_cast<T>(PyFloat_AsDouble(o));
    } else {
        *out = static_cast<T>(PyLong_AsUnsignedLongLongMask(o));
    }
    return PyErr_Occurred() == nullptr;
}

// The C call itself, without the interpreter lock.
template <typename F>
auto unlocked(F &&call) {
    PyThreadState *const state = PyEval_SaveThread();
    const auto rc = call();
    PyEval_RestoreThread(state);
    return rc;
}

// ---- a C function int f(args..., tc_stream) as a Python function f(args...) -------------------
template <auto Fn>
struct Wrap;
template <typename... A, int (*Fn)(A...)>
struct Wrap<Fn> {
    static constexpr size_t kArgs = sizeof...(A) - 1;  // the stream is the current one
    template <size_t... I>
    static PyObject *call(PyObject *const *args, std::index_sequence<I...>) {
        std::tuple<A...> v;
        if (!(toArg(args[I], &std::get<I>(v)) && ...)) return nullptr;
        std::get<kArgs>(v) = currentStream();
        return PyLong_FromLong(unlocked([&] { return std::apply(Fn, v); }));
    }
    static PyObject *py(PyObject *, PyObject *const *args, Py_ssize_t n) {
        HANDLE_TH_ERRORS
        if (static_cast<size_t>(n) != kArgs) {
            PyErr_Format(PyExc_TypeError, "%zu arguments expected, got %zd", kArgs, n);
            return nullptr;
        }
        return call(args, std::make_index_sequence<kArgs>());
        END_HANDLE_TH_ERRORS
    }
};

// ---- the calls that need more than that -----------------------------------------------------------

// attend(session, slot, q, k, v, out, pos, dev_pos, graph_capture): the rows of the call are q's
PyObject *attend(PyObject *, PyObject *const *a, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    if (n != 9) {
        PyErr_SetString(PyExc_TypeError, "attend: 9 arguments expected");
        return nullptr;
    }
    tc_kv_session *s;
    uint32_t slot, pos;
    float *q, *out;
    const float *k, *v;
    const uint32_t *dev;
    int graph;
    if (!toArg(a[0], &s) || !toArg(a[1], &slot) || !toArg(a[2], &q) || !toArg(a[3], &k) || !toArg(a[4], &v) ||
        !toArg(a[5], &out) || !toArg(a[6], &pos) || !toArg(a[7], &dev))
        return nullptr;
    graph = PyObject_IsTrue(a[8]);
    if (graph < 0) return nullptr;
    if (a[2] == Py_None) {
        PyErr_SetString(PyExc_TypeError, "attend: q is required");
        return nullptr;
    }
    const uint32_t rows = static_cast<uint32_t>(THPVariable_Unpack(a[2]).size(0));
    const tc_stream st = currentStream();
    return PyLong_FromLong(unlocked([&] { return tc_kv_session_attend(s, slot, q, k, v, out, rows, pos, dev, graph, st); }));
    END_HANDLE_TH_ERRORS
}

// begin(session, n) -> position, or -code
PyObject *begin(PyObject *, PyObject *const *a, Py_ssize_t n) {
    tc_kv_session *s;
    uint32_t rows, pos = 0;
    if (n != 2) {
        PyErr_SetString(PyExc_TypeError, "begin: 2 arguments expected");
        return nullptr;
    }
    if (!toArg(a[0], &s) || !toArg(a[1], &rows)) return nullptr;
    const int rc = tc_kv_session_begin(s, rows, &pos);
    return PyLong_FromLongLong(rc == TC_OK ? static_cast<long long>(pos) : -static_cast<long long>(rc));
}

// decode_i8_batch(q, k8, v8, ks, vs, out, pAcc, pM, pL, lens, rowBase, nextK8, nextV8, tickets, appendK,
//                 appendV, rowsPerSeq, totalRows, batch, nHeads, nKV, hd, maxLen, numChunks, invSqrt,
//                 partialsOnly, flags, prefetchRows) -> chunk slots used, or -code
PyObject *decodeI8Batch(PyObject *, PyObject *const *a, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    if (n != 28) {
        PyErr_SetString(PyExc_TypeError, "decode_i8_batch: 28 arguments expected");
        return nullptr;
    }
    const void *p[16];
    for (int i = 0; i < 16; ++i)
        if (!toAddress(a[i], &p[i])) return nullptr;
    tc_decode_i8_batch d;
    memset(&d, 0, sizeof(d));
    uint32_t used = 0;
    auto f = [&](int i) { return const_cast<float *>(static_cast<const float *>(p[i])); };
    d.q = f(0);
    d.k8 = static_cast<const int8_t *>(p[1]), d.v8 = static_cast<const int8_t *>(p[2]);
    d.ks = f(3), d.vs = f(4);
    d.out = f(5);
    d.pAcc = f(6), d.pM = f(7), d.pL = f(8);
    d.lens = static_cast<const uint32_t *>(p[9]);
    d.rowBase = static_cast<const uint64_t *>(p[10]);
    d.nextK8 = static_cast<const int8_t *>(p[11]), d.nextV8 = static_cast<const int8_t *>(p[12]);
    d.mergeTickets = const_cast<uint32_t *>(static_cast<const uint32_t *>(p[13]));
    d.appendK = f(14), d.appendV = f(15);
    if (!toArg(a[16], &d.rowsPerSeq) || !toArg(a[17], &d.totalRows) || !toArg(a[18], &d.batch) ||
        !toArg(a[19], &d.nHeads) || !toArg(a[20], &d.nKV) || !toArg(a[21], &d.hd) || !toArg(a[22], &d.maxLen) ||
        !toArg(a[23], &d.numChunks) || !toArg(a[24], &d.invSqrt) || !toArg(a[25], &d.partialsOnly) ||
        !toArg(a[26], &d.flags) || !toArg(a[27], &d.prefetchRows))
        return nullptr;
    d.chunksUsed = &used;
    const tc_stream st = currentStream();
    const int rc = unlocked([&] { return tc_attn_decode_i8_batch(&d, st); });
    return PyLong_FromLongLong(rc == TC_OK ? static_cast<long long>(used) : -static_cast<long long>(rc));
    END_HANDLE_TH_ERRORS
}

#define TC_FAST(name, fn) {name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(fn)), METH_FASTCALL, nullptr}
#define TC_WRAP(name, fn) TC_FAST(name, Wrap<fn>::py)
PyMethodDef kMethods[] = {
        TC_FAST("attend", attend),
        TC_FAST("begin", begin),
        TC_FAST("decode_i8_batch", decodeI8Batch),
        TC_WRAP("clear", tc_kv_session_clear),
        TC_WRAP("kv_append", tc_kv_append),
        TC_WRAP("kv_append_rope", tc_kv_append_rope),
        TC_WRAP("rope_q", tc_rope_q),
        TC_WRAP("kv_quantize_i8", tc_kv_quantize_i8),
        TC_WRAP("kv_quantize_i8_batch", tc_kv_quantize_i8_batch),
        TC_WRAP("decode_i8", tc_attn_decode_i8),
        TC_WRAP("decode_i8_noalloc", tc_attn_decode_i8_noalloc),
        TC_WRAP("decode_kv", tc_attn_decode_kv),
        TC_WRAP("merge_partials", tc_attn_merge_partials),
        TC_WRAP("merge_gathered", tc_attn_merge_gathered),
        TC_WRAP("prefill_f16", tc_attn_prefill_f16),
        TC_WRAP("prefill_f16_kv8", tc_attn_prefill_f16_kv8),
        TC_WRAP("prefill_f16_kvhalf", tc_attn_prefill_f16_kvhalf),
        TC_WRAP("prefill_f16_i8", tc_attn_prefill_f16_i8),
        TC_WRAP("prefill_kv", tc_attn_prefill_kv),
        TC_WRAP("prefill_i8", tc_attn_prefill_i8),
        TC_WRAP("qk_norm_rope", tc_qk_norm_rope),
        TC_WRAP("sigmoid_gate", tc_attn_sigmoid_gate),
        {nullptr, nullptr, 0, nullptr},
};

PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_native", "Calls into libtc_attn.so with torch tensors.", -1, kMethods,
                       nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__native(void) { return PyModule_Create(&kModule); }
