// fsb_python.cpp - the hot calls of the Python binding in native code (module ferro_b200.lib._fsb_native).
//
// A decode step through Python used to spend 9 us (one row) to 70 us (64 rows of 512-id histories) before it reached
// the C ABI: packing the histories row by row with numpy, and one ctypes pointer object per argument.  Here the
// arrays' own memory is handed to the C ABI directly.  Every function returns its result, or the negative status as
// an int, which the caller turns into an exception.  The GIL is released while the C ABI runs.
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#define NPY_NO_DEPRECATED_API NPY_1_7_API_VERSION
#include <numpy/arrayobject.h>

#include <cstdint>
#include <cstring>
#include <vector>

#include "../../include/ferro_sampler_b200.h"
#include "fsb_internal.h"

namespace {

// An int32 C-contiguous array for `o` (itself, if it is one already); null with an exception set on failure.
PyArrayObject* as_i32(PyObject* o) {
    return reinterpret_cast<PyArrayObject*>(PyArray_FROM_OTF(o, NPY_INT32, NPY_ARRAY_C_CONTIGUOUS | NPY_ARRAY_ALIGNED | NPY_ARRAY_FORCECAST));
}
int32_t* i32(PyArrayObject* a) { return static_cast<int32_t*>(PyArray_DATA(a)); }
PyArrayObject* new_i32(npy_intp n) { return reinterpret_cast<PyArrayObject*>(PyArray_SimpleNew(1, &n, NPY_INT32)); }
fsb_handle* handle(unsigned long long v) { return reinterpret_cast<fsb_handle*>(static_cast<uintptr_t>(v)); }
fsb_batch* batch(unsigned long long v) { return reinterpret_cast<fsb_batch*>(static_cast<uintptr_t>(v)); }

// References held for the duration of a call.
struct Refs {
    std::vector<PyObject*> v;
    ~Refs() {
        for (PyObject* o : v) Py_XDECREF(o);
    }
    template <class T>
    T* keep(T* o) {
        v.push_back(reinterpret_cast<PyObject*>(o));
        return o;
    }
};

// A sequence of integer sequences as pointers and lengths.  False with an exception set on failure.
struct Lists {
    std::vector<const int32_t*> ptr;
    std::vector<int64_t> len;
    int64_t total = 0;
};
bool take_lists(PyObject* seq, Refs& refs, Lists& out) {
    PyObject* fast = refs.keep(PySequence_Fast(seq, "a sequence of integer sequences is expected"));
    if (!fast) return false;
    const Py_ssize_t n = PySequence_Fast_GET_SIZE(fast);
    out.ptr.resize((size_t)n);
    out.len.resize((size_t)n);
    refs.v.reserve(refs.v.size() + (size_t)n + 4);
    for (Py_ssize_t i = 0; i < n; ++i) {
        PyArrayObject* a = refs.keep(as_i32(PySequence_Fast_GET_ITEM(fast, i)));
        if (!a) return false;
        out.ptr[(size_t)i] = i32(a);
        out.len[(size_t)i] = (int64_t)PyArray_SIZE(a);
        out.total += out.len[(size_t)i];
    }
    return true;
}

// sample_batch(handle, stream_ids, logits pointer, ld, n_vocab, histories, flags) -> tokens
PyObject* sample_batch(PyObject*, PyObject* args) {
    unsigned long long h, logits;
    long long ld;
    int n_vocab;
    unsigned flags;
    PyObject *sids_o, *hist_o;
    if (!PyArg_ParseTuple(args, "KOKLiOI", &h, &sids_o, &logits, &ld, &n_vocab, &hist_o, &flags)) return nullptr;
    Refs refs;
    PyArrayObject* sids = refs.keep(as_i32(sids_o));
    if (!sids) return nullptr;
    const npy_intp n = PyArray_SIZE(sids);
    Lists hist;
    if (!take_lists(hist_o, refs, hist)) return nullptr;
    if ((npy_intp)hist.ptr.size() < n) {
        PyErr_SetString(PyExc_ValueError, "one history per row is expected");
        return nullptr;
    }
    PyArrayObject* tokens = refs.keep(new_i32(n));
    if (!tokens) return nullptr;
    std::memset(i32(tokens), 0, sizeof(int32_t) * (size_t)n);
    int rc;
    Py_BEGIN_ALLOW_THREADS
    rc = fsb_sample_batch_lists(handle(h), (int)n, i32(sids), reinterpret_cast<const float*>((uintptr_t)logits), ld, n_vocab, hist.ptr.data(),
                                hist.len.data(), i32(tokens), flags);
    Py_END_ALLOW_THREADS
    if (rc) return PyLong_FromLong(rc);
    Py_INCREF(tokens);
    return reinterpret_cast<PyObject*>(tokens);
}

// sample_batch_resident(handle, stream_ids, logits pointer, ld, n_vocab, flags) -> tokens
PyObject* sample_batch_resident(PyObject*, PyObject* args) {
    unsigned long long h, logits;
    long long ld;
    int n_vocab;
    unsigned flags;
    PyObject* sids_o;
    if (!PyArg_ParseTuple(args, "KOKLiI", &h, &sids_o, &logits, &ld, &n_vocab, &flags)) return nullptr;
    Refs refs;
    PyArrayObject* sids = refs.keep(as_i32(sids_o));
    if (!sids) return nullptr;
    const npy_intp n = PyArray_SIZE(sids);
    PyArrayObject* tokens = refs.keep(new_i32(n));
    if (!tokens) return nullptr;
    std::memset(i32(tokens), 0, sizeof(int32_t) * (size_t)n);
    int rc;
    Py_BEGIN_ALLOW_THREADS
    rc = fsb_sample_batch_resident(handle(h), (int)n, i32(sids), reinterpret_cast<const float*>((uintptr_t)logits), ld, n_vocab, i32(tokens), flags);
    Py_END_ALLOW_THREADS
    if (rc) return PyLong_FromLong(rc);
    Py_INCREF(tokens);
    return reinterpret_cast<PyObject*>(tokens);
}

// verify_windows(handle, stream_ids, rows, logits pointer, ld, n_vocab, histories or None, max_accept or None, flags)
//   -> (tokens per stream, accepted, confirmed); None for the histories: the streams' resident ones
PyObject* verify_windows(PyObject*, PyObject* args) {
    unsigned long long h, logits;
    long long ld;
    int n_vocab;
    unsigned flags;
    PyObject *sids_o, *rows_o, *hist_o, *ma_o;
    if (!PyArg_ParseTuple(args, "KOOKLiOOI", &h, &sids_o, &rows_o, &logits, &ld, &n_vocab, &hist_o, &ma_o, &flags)) return nullptr;
    Refs refs;
    PyArrayObject* sids = refs.keep(as_i32(sids_o));
    if (!sids) return nullptr;
    const npy_intp n = PyArray_SIZE(sids);
    Lists rows, hist;
    if (!take_lists(rows_o, refs, rows)) return nullptr;
    if ((npy_intp)rows.ptr.size() != n) {
        PyErr_SetString(PyExc_ValueError, "one window per stream is expected");
        return nullptr;
    }
    const bool resident = hist_o == Py_None;
    if (!resident) {
        if (!take_lists(hist_o, refs, hist)) return nullptr;
        if ((npy_intp)hist.ptr.size() < n) {
            PyErr_SetString(PyExc_ValueError, "one history per stream is expected");
            return nullptr;
        }
    }
    PyArrayObject* ma = ma_o == Py_None ? nullptr : refs.keep(as_i32(ma_o));
    if (ma_o != Py_None && !ma) return nullptr;
    std::vector<int> off((size_t)n + 1, 0);
    std::vector<int32_t> flat((size_t)rows.total);
    for (npy_intp i = 0; i < n; ++i) {
        const size_t m = (size_t)rows.len[(size_t)i];
        if (m) std::memcpy(flat.data() + off[(size_t)i], rows.ptr[(size_t)i], m * sizeof(int32_t));
        off[(size_t)i + 1] = off[(size_t)i] + (int)m;
    }
    PyArrayObject *tokens = refs.keep(new_i32((npy_intp)rows.total)), *acc = refs.keep(new_i32(n)), *conf = refs.keep(new_i32(n));
    PyObject* parts = refs.keep(PyList_New(n));
    if (!tokens || !acc || !conf || !parts) return nullptr;
    std::memset(i32(tokens), 0, sizeof(int32_t) * (size_t)rows.total);
    std::memset(i32(acc), 0, sizeof(int32_t) * (size_t)n);
    std::memset(i32(conf), 0, sizeof(int32_t) * (size_t)n);
    const float* lg = reinterpret_cast<const float*>((uintptr_t)logits);
    int rc;
    Py_BEGIN_ALLOW_THREADS
    if (resident)
        rc = fsb_verify_windows_resident(handle(h), (int)n, i32(sids), off.data(), flat.data(), lg, ld, n_vocab, ma ? i32(ma) : nullptr, i32(tokens),
                                         i32(acc), i32(conf), flags);
    else
        rc = fsb_verify_windows_lists(handle(h), (int)n, i32(sids), off.data(), flat.data(), lg, ld, n_vocab, hist.ptr.data(), hist.len.data(),
                                      ma ? i32(ma) : nullptr, i32(tokens), i32(acc), i32(conf), flags);
    Py_END_ALLOW_THREADS
    if (rc) return PyLong_FromLong(rc);
    for (npy_intp i = 0; i < n; ++i) {   // views of the one token array
        npy_intp m = off[(size_t)i + 1] - off[(size_t)i];
        PyArray_Descr* dt = PyArray_DescrFromType(NPY_INT32);
        PyObject* v = PyArray_NewFromDescr(&PyArray_Type, dt, 1, &m, nullptr, i32(tokens) + off[(size_t)i], NPY_ARRAY_CARRAY, nullptr);
        if (!v) return nullptr;
        Py_INCREF(tokens);
        if (PyArray_SetBaseObject(reinterpret_cast<PyArrayObject*>(v), reinterpret_cast<PyObject*>(tokens)) < 0) {
            Py_DECREF(v);
            return nullptr;
        }
        PyList_SET_ITEM(parts, i, v);
    }
    return PyTuple_Pack(3, parts, reinterpret_cast<PyObject*>(acc), reinterpret_cast<PyObject*>(conf));
}

// A scalar (the same for all) or one value per stream.
bool per_stream(PyObject* o, npy_intp n, Refs& refs, std::vector<int>& out) {
    PyArrayObject* a = refs.keep(as_i32(o));
    if (!a) return false;
    const npy_intp m = PyArray_SIZE(a);
    if (m != n && m != 1) {
        PyErr_SetString(PyExc_ValueError, "one value, or one per stream, is expected");
        return false;
    }
    out.resize((size_t)n);
    for (npy_intp i = 0; i < n; ++i) out[(size_t)i] = i32(a)[m == 1 ? 0 : i];
    return true;
}

// lookup_drafts(handle, stream_ids, kmax, min_n, eos) -> a list of int32 arrays
PyObject* lookup_drafts(PyObject*, PyObject* args) {
    unsigned long long h;
    int eos;
    PyObject *sids_o, *k_o, *m_o;
    if (!PyArg_ParseTuple(args, "KOOOi", &h, &sids_o, &k_o, &m_o, &eos)) return nullptr;
    Refs refs;
    PyArrayObject* sids = refs.keep(as_i32(sids_o));
    if (!sids) return nullptr;
    const npy_intp n = PyArray_SIZE(sids);
    std::vector<int> km, mn;
    if (!per_stream(k_o, n, refs, km) || !per_stream(m_o, n, refs, mn)) return nullptr;
    int stride = 1;
    for (int k : km) stride = k > stride ? k : stride;
    std::vector<int32_t> drafts((size_t)n * (size_t)stride + 1);
    std::vector<int> cnt((size_t)n + 1, 0);
    int rc;
    Py_BEGIN_ALLOW_THREADS
    rc = fsb_lookup_drafts_resident(handle(h), (int)n, i32(sids), km.data(), mn.data(), eos, drafts.data(), stride, cnt.data());
    Py_END_ALLOW_THREADS
    if (rc) return PyLong_FromLong(rc);
    PyObject* parts = refs.keep(PyList_New(n));
    if (!parts) return nullptr;
    for (npy_intp i = 0; i < n; ++i) {
        PyArrayObject* a = new_i32(cnt[(size_t)i]);
        if (!a) return nullptr;
        if (cnt[(size_t)i] > 0) std::memcpy(i32(a), drafts.data() + (size_t)i * (size_t)stride, sizeof(int32_t) * (size_t)cnt[(size_t)i]);
        PyList_SET_ITEM(parts, i, reinterpret_cast<PyObject*>(a));
    }
    Py_INCREF(parts);
    return parts;
}

// history_set / history_append(handle, stream id, ids) -> status
PyObject* history_op(PyObject* args, bool append) {
    unsigned long long h;
    int sid;
    PyObject* ids_o;
    if (!PyArg_ParseTuple(args, "KiO", &h, &sid, &ids_o)) return nullptr;
    Refs refs;
    PyArrayObject* ids = refs.keep(as_i32(ids_o));
    if (!ids) return nullptr;
    const npy_intp n = PyArray_SIZE(ids);
    int rc;
    Py_BEGIN_ALLOW_THREADS
    rc = append ? fsb_stream_history_append(handle(h), sid, i32(ids), (int)n) : fsb_stream_history_set(handle(h), sid, i32(ids), (int64_t)n);
    Py_END_ALLOW_THREADS
    return PyLong_FromLong(rc);
}
PyObject* history_set(PyObject*, PyObject* args) { return history_op(args, false); }
PyObject* history_append(PyObject*, PyObject* args) { return history_op(args, true); }

// open_stream(handle, buffer of one parameter record) -> (status, stream id)
PyObject* open_stream(PyObject*, PyObject* args) {
    unsigned long long h;
    Py_buffer b;
    if (!PyArg_ParseTuple(args, "Ky*", &h, &b)) return nullptr;
    int sid = -1, rc = FSB_ERR_INVALID;
    if (b.len >= (Py_ssize_t)sizeof(ferro_sampler_params)) {
        ferro_sampler_params p;
        std::memcpy(&p, b.buf, sizeof p);
        rc = fsb_stream_open(handle(h), &p, &sid);
    }
    PyBuffer_Release(&b);
    return Py_BuildValue("(ii)", rc, sid);
}
PyObject* close_stream(PyObject*, PyObject* args) {
    unsigned long long h;
    int sid;
    if (!PyArg_ParseTuple(args, "Ki", &h, &sid)) return nullptr;
    return PyLong_FromLong(fsb_stream_close(handle(h), sid));
}

// batch_*(handle, batch, ...) -> status
PyObject* batch_launch(PyObject*, PyObject* args) {
    unsigned long long h, b, logits;
    if (!PyArg_ParseTuple(args, "KKK", &h, &b, &logits)) return nullptr;
    int rc;
    Py_BEGIN_ALLOW_THREADS
    rc = fsb_batch_launch(handle(h), batch(b), reinterpret_cast<const float*>((uintptr_t)logits));
    Py_END_ALLOW_THREADS
    return PyLong_FromLong(rc);
}
PyObject* batch_redraw(PyObject*, PyObject* args) {
    unsigned long long h, b;
    if (!PyArg_ParseTuple(args, "KK", &h, &b)) return nullptr;
    int rc;
    Py_BEGIN_ALLOW_THREADS
    rc = fsb_batch_redraw(handle(h), batch(b));
    Py_END_ALLOW_THREADS
    return PyLong_FromLong(rc);
}
PyObject* batch_check(PyObject*, PyObject* args) {
    unsigned long long h, b;
    if (!PyArg_ParseTuple(args, "KK", &h, &b)) return nullptr;
    int rc;
    Py_BEGIN_ALLOW_THREADS
    rc = fsb_batch_check(handle(h), batch(b));
    Py_END_ALLOW_THREADS
    return PyLong_FromLong(rc);
}
PyObject* batch_shard_launch_packed(PyObject*, PyObject* args) {
    unsigned long long h, b, logits, out;
    int stride;
    if (!PyArg_ParseTuple(args, "KKKKi", &h, &b, &logits, &out, &stride)) return nullptr;
    int rc;
    Py_BEGIN_ALLOW_THREADS
    rc = fsb_batch_shard_launch_packed(handle(h), batch(b), reinterpret_cast<const float*>((uintptr_t)logits), reinterpret_cast<uint64_t*>((uintptr_t)out),
                                       stride);
    Py_END_ALLOW_THREADS
    return PyLong_FromLong(rc);
}
PyObject* batch_merge_launch_packed(PyObject*, PyObject* args) {
    unsigned long long h, b, lists;
    int stride, n_lists, row_begin, n_rows;
    if (!PyArg_ParseTuple(args, "KKKiiii", &h, &b, &lists, &stride, &n_lists, &row_begin, &n_rows)) return nullptr;
    int rc;
    Py_BEGIN_ALLOW_THREADS
    rc = fsb_batch_merge_launch_packed(handle(h), batch(b), reinterpret_cast<const uint64_t*>((uintptr_t)lists), stride, n_lists, row_begin, n_rows);
    Py_END_ALLOW_THREADS
    return PyLong_FromLong(rc);
}

PyMethodDef methods[] = {
    {"sample_batch", sample_batch, METH_VARARGS, nullptr},
    {"sample_batch_resident", sample_batch_resident, METH_VARARGS, nullptr},
    {"verify_windows", verify_windows, METH_VARARGS, nullptr},
    {"lookup_drafts", lookup_drafts, METH_VARARGS, nullptr},
    {"history_set", history_set, METH_VARARGS, nullptr},
    {"history_append", history_append, METH_VARARGS, nullptr},
    {"open_stream", open_stream, METH_VARARGS, nullptr},
    {"close_stream", close_stream, METH_VARARGS, nullptr},
    {"batch_launch", batch_launch, METH_VARARGS, nullptr},
    {"batch_redraw", batch_redraw, METH_VARARGS, nullptr},
    {"batch_check", batch_check, METH_VARARGS, nullptr},
    {"batch_shard_launch_packed", batch_shard_launch_packed, METH_VARARGS, nullptr},
    {"batch_merge_launch_packed", batch_merge_launch_packed, METH_VARARGS, nullptr},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_fsb_native", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__fsb_native() {
    import_array();
    return PyModule_Create(&module);
}
