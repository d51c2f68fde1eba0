// CPython front end of the C ABI for torch tensors: reads the tensors' addresses, shapes and strides,
// allocates the result and calls libws_tp.so, all natively.
//
// Filling a ctypes struct, torch.empty, torch.cuda.current_stream() and the ctypes call itself cost
// ~12 us of host time per step (B200 host, measured), more than a decode step of a tensor-parallel shard
// takes on the device (6 us).  A function here returns None for arguments outside the plain form
// (non-CUDA tensors, unexpected types or layouts); tp.py then takes its own path, which explains what is
// wrong.  A negative status of the C ABI is returned as an int.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/ATen.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/python_variable.h>

#include <vector>

#include "../../include/ws_tp.h"

namespace {

const at::Tensor *tensor(PyObject *o) {
    if (!THPVariable_Check(o)) return nullptr;
    const at::Tensor &t = THPVariable_Unpack(o);
    return t.is_cuda() ? &t : nullptr;
}

bool act_dtype(const at::Tensor &t, int32_t *out) {
    if (t.scalar_type() == at::kBFloat16) *out = WS_ACT_BF16;
    else if (t.scalar_type() == at::kFloat) *out = WS_ACT_F32;
    else return false;
    return true;
}

// What a kernel reads or writes has to be there: all rows of scale blocks, a result of m x n floats.  (Block shapes and
// offsets that make no sense are the C ABI's to refuse.)
bool covers(const at::Tensor &scales, int64_t row0, int64_t n, int64_t bn) {
    return bn <= 0 || row0 < 0 || n < 1 || (row0 + n - 1) / bn < scales.size(0);
}
bool holds(const at::Tensor &out, int64_t m, int64_t n) {
    return out.scalar_type() == at::kFloat && out.is_contiguous() && out.numel() >= m * n;
}

// Everything of a step but its result; false: not the plain form.
bool fill_fp8(ws_fp8_gemm_args_t &a, PyObject *ox, PyObject *ow, PyObject *os, int32_t bn, int32_t bk, int64_t row0, int64_t k0) {
    const at::Tensor *x = tensor(ox), *w = tensor(ow), *s = tensor(os);
    if (!x || !w || !s || x->dim() != 2 || w->dim() != 2 || s->dim() != 2) return false;
    if (w->scalar_type() != at::kByte && w->scalar_type() != at::kFloat8_e4m3fn) return false;
    if (s->scalar_type() == at::kFloat) a.scale_kind = WS_SCALE_F32;
    else if (s->scalar_type() == at::kByte) a.scale_kind = WS_SCALE_UE8M0;
    else return false;
    if (!act_dtype(*x, &a.x_dtype) || x->stride(1) != 1 || w->stride(1) != 1 || !s->is_contiguous() || w->size(1) != x->size(1)) return false;
    const int64_t m = x->size(0), n = w->size(0), k = x->size(1);
    if (m > INT32_MAX || n > INT32_MAX || k > INT32_MAX || !covers(*s, row0, n, bn)) return false;
    a.m = (int32_t)m; a.n = (int32_t)n; a.k = (int32_t)k;
    a.x = x->data_ptr(); a.ldx = m > 1 ? x->stride(0) : k;
    a.w = static_cast<const uint8_t *>(w->data_ptr()); a.ldw = w->stride(0);
    a.scales = s->data_ptr(); a.scale_ld = s->size(1);
    a.block_n = bn; a.block_k = bk; a.row0 = row0; a.k0 = k0;
    return true;
}

bool fill_moe(ws_moe_down_args_t &a, PyObject *oh, PyObject *oids, PyObject *orw, PyObject *ow, PyObject *os, int32_t e_start) {
    const at::Tensor *h = tensor(oh), *ids = tensor(oids), *rw = tensor(orw), *w = tensor(ow), *s = tensor(os);
    if (!h || !ids || !rw || !w || !s || w->dim() != 3 || s->dim() != 3 || ids->dim() != 2 || h->dim() != 2) return false;
    if (!w->is_contiguous() || !s->is_contiguous() || !ids->is_contiguous() || !rw->is_contiguous()) return false;
    if (ids->scalar_type() != at::kInt || rw->scalar_type() != at::kFloat || !act_dtype(*h, &a.h_dtype)) return false;
    const int64_t k = w->size(2) * 2, routes = ids->numel();
    if (w->element_size() != 1 || s->element_size() != 1 || s->numel() * 16 < w->numel()) return false;
    if (h->size(0) < routes || h->size(1) < k || h->stride(1) != 1 || rw->numel() < routes) return false;
    a.h = h->data_ptr(); a.ldh = h->size(0) > 1 ? h->stride(0) : k;
    a.m = (int32_t)ids->size(0); a.top_k = (int32_t)ids->size(1); a.n = (int32_t)w->size(1); a.k = (int32_t)k;
    a.route_ids = ids->data_ptr<int32_t>(); a.route_w = rw->data_ptr<float>();
    a.w2 = static_cast<const uint8_t *>(w->data_ptr()); a.s2 = static_cast<const uint8_t *>(s->data_ptr());
    a.e_start = e_start; a.e_len = (int32_t)w->size(0);
    return true;
}

at::Tensor new_f32(const at::Tensor &like, int64_t m, int64_t n) { return at::empty({m, n}, like.options().dtype(at::kFloat).requires_grad(false)); }

bool stream_of(PyObject *o, void **out) {  // None: torch's current stream of the current device
    if (o == Py_None) {
        *out = c10::cuda::getCurrentCUDAStream().stream();
        return true;
    }
    *out = PyLong_AsVoidPtr(o);
    return !PyErr_Occurred();
}

// A status, or the result: `result` is the caller's `out` or a tensor made here.
PyObject *answer(ws_status_t st, PyObject *result) {
    if (st == WS_OK) return result;
    Py_XDECREF(result);
    return PyLong_FromLong(st);
}

#define WS_CALL(st, expr)            \
    ws_status_t st;                  \
    Py_BEGIN_ALLOW_THREADS           \
    st = expr;                       \
    Py_END_ALLOW_THREADS

// fp8(handle, x, w, scales, block_n, block_k, row0, k0, out, stream)
PyObject *py_fp8(PyObject *, PyObject *const *v, Py_ssize_t nargs) {
    HANDLE_TH_ERRORS
    if (nargs != 10) { PyErr_SetString(PyExc_TypeError, "fp8 takes 10 arguments"); return nullptr; }
    ws_fp8_gemm_args_t a{};
    ws_tp_t *const tp = static_cast<ws_tp_t *>(PyLong_AsVoidPtr(v[0]));
    const long bn = PyLong_AsLong(v[4]), bk = PyLong_AsLong(v[5]);
    const int64_t row0 = PyLong_AsLongLong(v[6]), k0 = PyLong_AsLongLong(v[7]);
    void *stream;
    if (PyErr_Occurred() || !stream_of(v[9], &stream)) return nullptr;
    if (!fill_fp8(a, v[1], v[2], v[3], (int32_t)bn, (int32_t)bk, row0, k0)) Py_RETURN_NONE;
    PyObject *res;
    if (v[8] == Py_None) {
        at::Tensor out = new_f32(THPVariable_Unpack(v[1]), a.m, a.n);
        a.out = out.data_ptr<float>();
        res = THPVariable_Wrap(std::move(out));
    } else {
        const at::Tensor *out = tensor(v[8]);
        if (!out || !holds(*out, a.m, a.n)) Py_RETURN_NONE;
        a.out = static_cast<float *>(out->data_ptr());
        Py_INCREF(v[8]);
        res = v[8];
    }
    WS_CALL(st, ws_fp8_rowpar_gemm_allreduce(tp, &a, stream))
    return answer(st, res);
    END_HANDLE_TH_ERRORS
}

// fp8_host(handle, x_host, w, scales, block_n, block_k, row0, k0, x_dtype, out_host) -> status: x_host and out_host are
// C-contiguous buffers (numpy arrays) of at least m * k activations and m * n floats.
PyObject *py_fp8_host(PyObject *, PyObject *const *v, Py_ssize_t nargs) {
    HANDLE_TH_ERRORS
    if (nargs != 10) { PyErr_SetString(PyExc_TypeError, "fp8_host takes 10 arguments"); return nullptr; }
    ws_tp_t *const tp = static_cast<ws_tp_t *>(PyLong_AsVoidPtr(v[0]));
    const at::Tensor *w = tensor(v[2]), *s = tensor(v[3]);
    ws_fp8_gemm_args_t a{};
    a.block_n = (int32_t)PyLong_AsLong(v[4]); a.block_k = (int32_t)PyLong_AsLong(v[5]);
    a.row0 = PyLong_AsLongLong(v[6]); a.k0 = PyLong_AsLongLong(v[7]); a.x_dtype = (int32_t)PyLong_AsLong(v[8]);
    if (PyErr_Occurred()) return nullptr;
    if (!w || !s || w->dim() != 2 || s->dim() != 2 || w->stride(1) != 1 || w->element_size() != 1) Py_RETURN_NONE;
    if (!s->is_contiguous() || !covers(*s, a.row0, w->size(0), a.block_n)) Py_RETURN_NONE;
    if (s->scalar_type() == at::kFloat) a.scale_kind = WS_SCALE_F32;
    else if (s->scalar_type() == at::kByte) a.scale_kind = WS_SCALE_UE8M0;
    else Py_RETURN_NONE;
    Py_buffer x, out;
    if (PyObject_GetBuffer(v[1], &x, PyBUF_ND) != 0) { PyErr_Clear(); Py_RETURN_NONE; }
    if (PyObject_GetBuffer(v[9], &out, PyBUF_ND | PyBUF_WRITABLE) != 0) { PyBuffer_Release(&x); PyErr_Clear(); Py_RETURN_NONE; }
    a.n = (int32_t)w->size(0); a.k = (int32_t)w->size(1);
    a.m = x.ndim > 0 ? (int32_t)x.shape[0] : 0;
    a.ldx = a.k; a.w = static_cast<const uint8_t *>(w->data_ptr()); a.ldw = w->stride(0);
    a.scales = s->data_ptr(); a.scale_ld = s->size(1);
    const int64_t es = a.x_dtype == WS_ACT_BF16 ? 2 : 4;
    const bool fits = x.len >= es * a.m * a.k && out.len >= (int64_t)4 * a.m * a.n;
    ws_status_t st = WS_OK;
    if (fits) {
        Py_BEGIN_ALLOW_THREADS
        st = ws_fp8_rowpar_gemm_allreduce_host(tp, &a, x.buf, static_cast<float *>(out.buf));
        Py_END_ALLOW_THREADS
    }
    PyBuffer_Release(&x);
    PyBuffer_Release(&out);
    if (!fits) Py_RETURN_NONE;
    return PyLong_FromLong(st);
    END_HANDLE_TH_ERRORS
}

// moe(handle, h, route_ids, route_w, w2, s2, e_start, out, stream)
PyObject *py_moe(PyObject *, PyObject *const *v, Py_ssize_t nargs) {
    HANDLE_TH_ERRORS
    if (nargs != 9) { PyErr_SetString(PyExc_TypeError, "moe takes 9 arguments"); return nullptr; }
    ws_moe_down_args_t a{};
    ws_tp_t *const tp = static_cast<ws_tp_t *>(PyLong_AsVoidPtr(v[0]));
    const long e_start = PyLong_AsLong(v[6]);
    void *stream;
    if (PyErr_Occurred() || !stream_of(v[8], &stream)) return nullptr;
    if (!fill_moe(a, v[1], v[2], v[3], v[4], v[5], (int32_t)e_start)) Py_RETURN_NONE;
    PyObject *res;
    if (v[7] == Py_None) {
        at::Tensor out = new_f32(THPVariable_Unpack(v[1]), a.m, a.n);
        a.out = out.data_ptr<float>();
        res = THPVariable_Wrap(std::move(out));
    } else {
        const at::Tensor *out = tensor(v[7]);
        if (!out || !holds(*out, a.m, a.n)) Py_RETURN_NONE;
        a.out = static_cast<float *>(out->data_ptr());
        Py_INCREF(v[7]);
        res = v[7];
    }
    WS_CALL(st, ws_moe_down_combine_allreduce(tp, &a, stream))
    return answer(st, res);
    END_HANDLE_TH_ERRORS
}

// head(handle, x, w, scales, block_n, block_k, row0, vocab_row0, vocab, want_logits, stream) -> (logits | None, argmax)
PyObject *py_head(PyObject *, PyObject *const *v, Py_ssize_t nargs) {
    HANDLE_TH_ERRORS
    if (nargs != 11) { PyErr_SetString(PyExc_TypeError, "head takes 11 arguments"); return nullptr; }
    ws_lm_head_args_t a{};
    ws_tp_t *const tp = static_cast<ws_tp_t *>(PyLong_AsVoidPtr(v[0]));
    const long bn = PyLong_AsLong(v[4]), bk = PyLong_AsLong(v[5]), vocab = PyLong_AsLong(v[8]);
    const int64_t row0 = PyLong_AsLongLong(v[6]);
    a.vocab_row0 = PyLong_AsLongLong(v[7]);
    a.vocab = (int32_t)vocab;
    const int want = PyObject_IsTrue(v[9]);
    void *stream;
    if (PyErr_Occurred() || !stream_of(v[10], &stream)) return nullptr;
    if (vocab < 0 || vocab > INT32_MAX || !fill_fp8(a.g, v[1], v[2], v[3], (int32_t)bn, (int32_t)bk, row0, 0)) Py_RETURN_NONE;
    const at::Tensor &x = THPVariable_Unpack(v[1]);
    at::Tensor logits, arg = at::empty({a.g.m}, x.options().dtype(at::kInt).requires_grad(false));
    a.argmax = reinterpret_cast<uint32_t *>(arg.data_ptr<int32_t>());
    if (want) {
        logits = new_f32(x, a.g.m, vocab);
        a.logits = logits.data_ptr<float>();
    }
    WS_CALL(st, ws_lm_head_allgather_argmax(tp, &a, stream))
    if (st != WS_OK) return PyLong_FromLong(st);
    PyObject *first = Py_None;
    if (want) first = THPVariable_Wrap(std::move(logits));
    else Py_INCREF(Py_None);
    PyObject *second = THPVariable_Wrap(std::move(arg));
    PyObject *pair = PyTuple_Pack(2, first, second);
    Py_DECREF(first);
    Py_DECREF(second);
    return pair;
    END_HANDLE_TH_ERRORS
}

// fp8_group(handles, devices, xs, ws, scales, block_n, block_k, row0s | None, k0s | None) -> [out of every rank]
PyObject *py_fp8_group(PyObject *, PyObject *const *v, Py_ssize_t nargs) {
    HANDLE_TH_ERRORS
    if (nargs != 9) { PyErr_SetString(PyExc_TypeError, "fp8_group takes 9 arguments"); return nullptr; }
    if (!PyTuple_Check(v[0]) || !PyTuple_Check(v[1])) Py_RETURN_NONE;
    const Py_ssize_t world = PyTuple_GET_SIZE(v[0]);
    for (int i = 2; i < 5; ++i)
        if (!PyList_Check(v[i]) || PyList_GET_SIZE(v[i]) != world) Py_RETURN_NONE;
    for (int i = 7; i < 9; ++i)
        if (v[i] != Py_None && (!PyList_Check(v[i]) || PyList_GET_SIZE(v[i]) != world)) Py_RETURN_NONE;
    if (world < 1 || world > WS_MAX_WORLD) Py_RETURN_NONE;
    const long bn = PyLong_AsLong(v[5]), bk = PyLong_AsLong(v[6]);
    ws_fp8_gemm_args_t a[WS_MAX_WORLD] = {};
    ws_tp_t *tps[WS_MAX_WORLD];
    void *streams[WS_MAX_WORLD];
    at::Tensor outs[WS_MAX_WORLD];
    for (Py_ssize_t r = 0; r < world; ++r) {
        tps[r] = static_cast<ws_tp_t *>(PyLong_AsVoidPtr(PyTuple_GET_ITEM(v[0], r)));
        const int64_t row0 = v[7] == Py_None ? 0 : PyLong_AsLongLong(PyList_GET_ITEM(v[7], r));
        const int64_t k0 = v[8] == Py_None ? 0 : PyLong_AsLongLong(PyList_GET_ITEM(v[8], r));
        const long dev = PyLong_AsLong(PyTuple_GET_ITEM(v[1], r));
        if (PyErr_Occurred()) return nullptr;
        if (!fill_fp8(a[r], PyList_GET_ITEM(v[2], r), PyList_GET_ITEM(v[3], r), PyList_GET_ITEM(v[4], r), (int32_t)bn, (int32_t)bk, row0, k0))
            Py_RETURN_NONE;
        streams[r] = c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)dev).stream();
        outs[r] = new_f32(THPVariable_Unpack(PyList_GET_ITEM(v[2], r)), a[r].m, a[r].n);
        a[r].out = outs[r].data_ptr<float>();
    }
    WS_CALL(st, ws_fp8_rowpar_gemm_allreduce_group(tps, (int32_t)world, a, streams))
    if (st != WS_OK) return PyLong_FromLong(st);
    PyObject *list = PyList_New(world);
    for (Py_ssize_t r = 0; list && r < world; ++r) PyList_SET_ITEM(list, r, THPVariable_Wrap(std::move(outs[r])));
    return list;
    END_HANDLE_TH_ERRORS
}

#define WS_METHOD(name) {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)(void)>(py_##name)), METH_FASTCALL, nullptr}
PyMethodDef methods[] = {WS_METHOD(fp8), WS_METHOD(fp8_host), WS_METHOD(moe), WS_METHOD(head), WS_METHOD(fp8_group), {nullptr, nullptr, 0, nullptr}};
PyModuleDef module_def = {PyModuleDef_HEAD_INIT, "_ws_torch", "torch tensors -> libws_tp.so", -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__ws_torch(void) { return PyModule_Create(&module_def); }
