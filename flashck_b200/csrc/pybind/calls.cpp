// The plain calls of flashck_b200.ops in native code: argument checks, output and workspace allocation and the C-ABI call.
//
// Around a short attention call the Python of ops/fmha.py (checks, torch.empty, argument conversion) takes two to four times as
// long as its kernels: 2 x 128 tokens 24 us a call with 7 us on the GPU, a decode step of one sequence (two launches) 45 us with
// 10 us on the GPU.  Here the same calls take 7.0 and 11.6 us.  A function takes only what the host can check completely -- exact
// torch.Tensor objects that are dense, contiguous, on one CUDA device, of the expected types and of sizes that fit one another (what
// lies in device memory, lengths and page ids, is the caller's), Python bools, ints and floats -- and returns None for everything else (subclasses, functorch wrappers, active modes or tracing, other argument
// types, shapes that do not fit); the caller then goes on in Python, which converts, or raises what it always raised.
// Otherwise it returns the result, or the non-zero status of the C call.
#include <ATen/ATen.h>
#include <ATen/PythonTorchFunctionTLS.h>
#include <ATen/cuda/CUDAContext.h>
#include <c10/core/impl/LocalDispatchKeySet.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAGuard.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/jit/frontend/tracer.h>
#include <torch/extension.h>

#include "flashck_b200.h"

namespace flashck {
namespace calls {

namespace {

// Everything is ordinary: no mode, transform or tracer that would have to see the operations of the call.
bool plain_state() {
    return !at::impl::torch_function_mode_enabled() && !c10::impl::TorchDispatchModeTLS::any_modes_set() &&
           !c10::impl::tls_is_dispatch_key_included(c10::DispatchKey::FuncTorchDynamicLayerFrontMode) &&
           !c10::impl::tls_is_dispatch_key_included(c10::DispatchKey::Functionalize) && !torch::jit::tracer::isTracing();
}

// A dense contiguous CUDA tensor of a Python object that is exactly torch.Tensor.
const at::Tensor* tensor(PyObject* o) {
    if (!THPVariable_CheckExact(o)) return nullptr;
    const at::Tensor& t = THPVariable_Unpack(o);
    if (!t.defined() || !t.is_cuda() || t.layout() != at::kStrided || t.is_neg() || t.is_conj()) return nullptr;
    const c10::DispatchKeySet backend = t.key_set() - c10::autograd_dispatch_keyset_with_ADInplaceOrView -
                                        c10::autocast_dispatch_keyset;
    if (backend != c10::DispatchKeySet(c10::DispatchKey::CUDA)) return nullptr;
    return t.is_contiguous() ? &t : nullptr;
}
// The arguments of one call, read in order; `ok` turns false with the first one that is not plain.
struct Reader {
    PyObject* const* args;
    Py_ssize_t n, i = 0;
    bool ok = true;
    c10::Device device{c10::kCPU};

    PyObject* next() {
        if (i >= n) { ok = false; return Py_None; }
        return args[i++];
    }
    const at::Tensor* need(at::ScalarType type, int64_t dim = -1) {
        PyObject* o = next();
        const at::Tensor* t = ok ? tensor(o) : nullptr;
        if (!t || (type != at::ScalarType::Undefined && t->scalar_type() != type) || (dim >= 0 && t->dim() != dim)) { ok = false; return nullptr; }
        if (device.is_cpu()) device = t->device();
        else if (device != t->device()) ok = false;
        return t;
    }
    const at::Tensor* maybe(at::ScalarType type, int64_t dim = -1) {
        if (i < n && args[i] == Py_None) { ++i; return nullptr; }
        return need(type, dim);
    }
    bool flag() {
        PyObject* o = next();
        if (o != Py_True && o != Py_False) ok = false;
        return o == Py_True;
    }
    int64_t integer(PyObject* o) {
        if (!PyLong_CheckExact(o)) { ok = false; return 0; }
        int overflow = 0;
        const long long v = PyLong_AsLongLongAndOverflow(o, &overflow);
        if (overflow) ok = false;
        return v;
    }
    int64_t integer() { return integer(next()); }
    double real(bool none_is_zero) {
        PyObject* o = next();
        if (none_is_zero && o == Py_None) return 0.0;
        if (!PyFloat_CheckExact(o)) { ok = false; return 0.0; }
        return PyFloat_AS_DOUBLE(o);
    }
    // causal, window_size, mask_type -> the C ABI's (mask_type, left, right), as ops.fmha._mask has it
    void mask(uint32_t& type, int64_t& left, int64_t& right) {
        const bool causal = flag();
        PyObject* w = next();
        PyObject* mt = next();
        left = right = -1;
        type = 0;
        if (!ok) return;
        if (PyTuple_CheckExact(w) && PyTuple_GET_SIZE(w) == 2) {
            left = integer(PyTuple_GET_ITEM(w, 0));
            right = integer(PyTuple_GET_ITEM(w, 1));
        } else {
            ok = false;
            return;
        }
        if (mt != Py_None) {
            const int64_t v = integer(mt);
            if (v < 0 || v > 3) ok = false;
            type = (uint32_t)v;
            if (causal) right = 0;
        } else if (causal) {
            type = 2;
            right = 0;
        } else if (left >= 0 || right >= 0) {
            type = 2;
        } else {
            left = right = -1;
        }
    }
};

bool holds(const at::Tensor* t, int64_t entries) { return !t || t->numel() >= entries; }
// K and its V: the same sizes in all dimensions but the last, and V may go on behind K's first one.  (The kernels are given K's.)
bool rows_fit(const at::Tensor& k, const at::Tensor& v) {
    return k.dim() == v.dim() && k.size(0) <= v.size(0) && k.sizes().slice(1, k.dim() - 2) == v.sizes().slice(1, v.dim() - 2);
}
void* ptr(const at::Tensor* t) { return t ? t->data_ptr() : nullptr; }
void* ptr(const at::Tensor& t) { return t.defined() ? t.data_ptr() : nullptr; }
int dtype_code(const at::Tensor& t) { return t.scalar_type() == at::kHalf ? FLASHCK_DTYPE_FLOAT16 : FLASHCK_DTYPE_BFLOAT16; }
bool elem16(const at::Tensor* t) { return t && (t->scalar_type() == at::kHalf || t->scalar_type() == at::kBFloat16); }
at::Tensor empty(at::IntArrayRef shape, at::ScalarType type, c10::Device dev) {
    return at::empty(shape, at::TensorOptions().dtype(type).device(dev));
}
void* stream_of(c10::Device dev) { return (void*)at::cuda::getCurrentCUDAStream(dev.index()).stream(); }

// o, (o, lse) or the status of the call
PyObject* result(int rc, const at::Tensor& o, const at::Tensor& lse) {
    if (rc != 0) return PyLong_FromLong(rc);
    if (!lse.defined()) return THPVariable_Wrap(o);
    PyObject* a = THPVariable_Wrap(o);
    PyObject* b = a ? THPVariable_Wrap(lse) : nullptr;
    PyObject* r = b ? PyTuple_Pack(2, a, b) : nullptr;
    Py_XDECREF(a);
    Py_XDECREF(b);
    return r;
}

// (q, k, v, cu_seqlens_q | None, cu_seqlens_k | None, max_seqlen_q, scale, causal, window_size, mask_type, return_lse, cap)
PyObject* call_forward(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
    HANDLE_TH_ERRORS
    if (!plain_state()) Py_RETURN_NONE;
    Reader r{args, nargs};
    const at::Tensor* q = r.need(at::ScalarType::Undefined);
    if (!r.ok || !elem16(q)) Py_RETURN_NONE;
    const at::ScalarType elem = q->scalar_type();
    const at::Tensor *k = r.need(elem, q->dim()), *v = r.need(elem, q->dim());
    const at::Tensor *cu_q = r.maybe(at::kLong), *cu_k = r.maybe(at::kLong);
    int64_t max_q = r.integer();
    const double scale = r.real(true);
    uint32_t mt;
    int64_t wl, wr;
    r.mask(mt, wl, wr);
    const bool with_lse = r.flag();
    const double cap = r.real(false);
    if (!r.ok || r.i != nargs) Py_RETURN_NONE;
    const bool group = cu_q != nullptr;
    if (q->dim() != (group ? 3 : 4) || group != (cu_k != nullptr)) Py_RETURN_NONE;
    const int64_t hq = q->size(-2), d = q->size(-1), hkv = k->size(-2), dv = v->size(-1);
    if (k->size(-1) != d || v->size(-2) != hkv) Py_RETURN_NONE;
    int64_t batch, sq, sk;
    if (group) {
        if (cu_q->numel() != cu_k->numel() || cu_q->numel() < 2 || v->size(0) != k->size(0)) Py_RETURN_NONE;
        batch = cu_q->numel() - 1;
        sq = q->size(0);
        sk = k->size(0);
    } else {
        batch = q->size(0);
        sq = max_q = q->size(1);
        sk = k->size(1);
        if (k->size(0) != batch || v->size(0) != batch || v->size(1) != sk) Py_RETURN_NONE;
    }
    at::Tensor o, lse;
    int rc;
    {
        pybind11::gil_scoped_release no_gil;
        const c10::cuda::CUDAGuard guard(r.device);
        o = group ? empty({sq, hq, dv}, elem, r.device) : empty({batch, sq, hq, dv}, elem, r.device);
        if (with_lse) lse = group ? empty({hq, sq}, at::kFloat, r.device) : empty({batch, hq, sq}, at::kFloat, r.device);
        rc = FmhaFwdBias(ptr(q), ptr(k), ptr(v), nullptr, ptr(o), (int64_t*)ptr(cu_q), (int64_t*)ptr(cu_k), nullptr, batch, sq,
                         sk, hq, hkv, d, dv, max_q, (float)scale, wl, wr, mt, stream_of(r.device), ptr(lse), dtype_code(*q), 0,
                         0, (float)cap);
    }
    return result(rc, o, lse);
    END_HANDLE_TH_ERRORS
}

// (q, k_pool, v_pool, block_table, seqlen_k, cu_seqlens_q | None, max_seqlen_q, scale, causal, window_size, mask_type, return_lse)
PyObject* call_paged_prefill(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
    HANDLE_TH_ERRORS
    if (!plain_state()) Py_RETURN_NONE;
    Reader r{args, nargs};
    const at::Tensor* q = r.need(at::ScalarType::Undefined);
    if (!r.ok || !elem16(q)) Py_RETURN_NONE;
    const at::ScalarType elem = q->scalar_type();
    const at::Tensor *k = r.need(elem, 4), *v = r.need(elem, 4), *bt = r.need(at::kInt, 2), *sl = r.need(at::kInt);
    const at::Tensor* cu_q = r.maybe(at::kLong);
    int64_t max_q = r.integer();
    const double scale = r.real(true);
    uint32_t mt;
    int64_t wl, wr;
    r.mask(mt, wl, wr);
    const bool with_lse = r.flag();
    if (!r.ok || r.i != nargs) Py_RETURN_NONE;
    const bool group = cu_q != nullptr;
    if (q->dim() != (group ? 3 : 4) || (!group && q->size(0) != bt->size(0))) Py_RETURN_NONE;
    const int64_t batch = bt->size(0), hq = q->size(-2), d = q->size(-1), dv = v->size(3);
    const int64_t sq = group ? q->size(0) : q->size(1);
    if (k->size(3) != d || !rows_fit(*k, *v) || !holds(sl, batch) || !holds(cu_q, batch + 1)) Py_RETURN_NONE;
    if (!group || max_q == 0) max_q = sq;
    at::Tensor o, lse;
    int rc;
    {
        pybind11::gil_scoped_release no_gil;
        const c10::cuda::CUDAGuard guard(r.device);
        o = group ? empty({sq, hq, dv}, elem, r.device) : empty({batch, sq, hq, dv}, elem, r.device);
        if (with_lse) lse = group ? empty({hq, sq}, at::kFloat, r.device) : empty({batch, hq, sq}, at::kFloat, r.device);
        rc = FmhaFwdPagedKVPrefillEx(ptr(q), ptr(k), ptr(v), nullptr, ptr(o), (int64_t*)ptr(cu_q), ptr(sl), ptr(bt), nullptr,
                                     batch, sq, hq, k->size(2), d, dv, max_q, batch * bt->size(1), k->size(1), (float)scale, wl,
                                     wr, mt, stream_of(r.device), ptr(lse), dtype_code(*q), 0, 0, k->size(0));
    }
    return result(rc, o, lse);
    END_HANDLE_TH_ERRORS
}

// ops.fmha.default_num_splits with its default arguments
int64_t num_splits_for(int64_t batch, int64_t rows_per_kv_head) {
    if (rows_per_kv_head > 16) return 16;
    const int64_t b = std::max<int64_t>(batch, 1);
    return std::max<int64_t>(2, std::min<int64_t>(128, (2 * 148 + b - 1) / b + 1));
}

// (q, k_cache, v_cache, seqlen_k | None, block_table | None, cu_seqlens_q | None, max_seqlen_q, num_splits, scale, causal,
//  window_size, mask_type, return_lse)
PyObject* call_splitkv(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
    HANDLE_TH_ERRORS
    if (!plain_state()) Py_RETURN_NONE;
    Reader r{args, nargs};
    const at::Tensor* q = r.need(at::ScalarType::Undefined);
    if (!r.ok || !elem16(q)) Py_RETURN_NONE;
    const at::ScalarType elem = q->scalar_type();
    const at::Tensor *k = r.need(elem, 4), *v = r.need(elem, 4), *sl = r.maybe(at::kInt), *bt = r.maybe(at::kInt, 2);
    const at::Tensor* cu_q = r.maybe(at::kLong);
    int64_t max_q = r.integer(), splits = r.integer();
    const double scale = r.real(true);
    uint32_t mt;
    int64_t wl, wr;
    r.mask(mt, wl, wr);
    const bool with_lse = r.flag();
    if (!r.ok || r.i != nargs) Py_RETURN_NONE;
    const bool group = cu_q != nullptr;
    if (q->dim() != (group ? 3 : 4) || (bt && !sl)) Py_RETURN_NONE;
    const int64_t hq = q->size(-2), d = q->size(-1), hkv = k->size(2), dv = v->size(3);
    const int64_t batch = group ? cu_q->numel() - 1 : q->size(0), sq = group ? q->size(0) : q->size(1);
    if (batch < 1 || k->size(3) != d || !rows_fit(*k, *v) || !holds(sl, batch)) Py_RETURN_NONE;
    if (bt ? bt->size(0) != batch : k->size(0) < batch) Py_RETURN_NONE;
    if (!group || max_q == 0) max_q = sq;
    if (splits <= 0) splits = num_splits_for(batch, max_q * (hq / std::max<int64_t>(hkv, 1)));
    const int64_t page = bt ? k->size(1) : 0, bs = group ? 1 : batch;
    at::Tensor o, lse, work;
    int rc;
    {
        pybind11::gil_scoped_release no_gil;
        const c10::cuda::CUDAGuard guard(r.device);
        void* stream = stream_of(r.device);
        // one workspace: the partial rows, then their LSEs
        const int64_t rows = bs * hq * splits * sq;
        work = empty({rows * (dv + 1)}, at::kFloat, r.device);
        float* o_acc = (float*)work.data_ptr();
        float* lse_acc = o_acc + rows * dv;
        rc = FmhaFwdSplitKVEx(ptr(q), ptr(k), ptr(v), nullptr, lse_acc, o_acc, (int64_t*)ptr(cu_q), nullptr, ptr(sl), ptr(bt),
                              nullptr, batch, sq, bt ? 0 : k->size(1), hq, hkv, d, dv, max_q, splits,
                              bt ? batch * bt->size(1) : 0, page, (float)scale, wl, wr, mt, stream, dtype_code(*q), 0, 0,
                              k->size(0));
        if (rc == 0) {
            o = group ? empty({sq, hq, dv}, elem, r.device) : empty({batch, sq, hq, dv}, elem, r.device);
            if (with_lse) lse = group ? empty({hq, sq}, at::kFloat, r.device) : empty({batch, hq, sq}, at::kFloat, r.device);
            rc = FmhaFwdSplitKVCombine(lse_acc, o_acc, ptr(o), nullptr, bs, sq, hq, dv, sq, splits, stream, ptr(lse),
                                       dtype_code(*q));
            if (rc != 0) rc = -rc;  // (which of the two calls it was)
        }
    }
    return result(rc, o, lse);
    END_HANDLE_TH_ERRORS
}

// (q | None, k_cache, v_cache, knew, vnew, seqlen_k, rotary_cos | None, rotary_sin | None, rope, rotary_dim | None,
//  block_table | None, cu_seqlens_q | None, cu_seqlens_knew | None) -> status
PyObject* call_append_kv(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
    HANDLE_TH_ERRORS
    if (!plain_state()) Py_RETURN_NONE;
    Reader r{args, nargs};
    const at::Tensor* q = r.maybe(at::ScalarType::Undefined);
    const at::Tensor* k = r.need(at::ScalarType::Undefined, 4);
    if (!r.ok || !elem16(k)) Py_RETURN_NONE;
    const at::ScalarType elem = k->scalar_type();
    const at::Tensor *v = r.need(elem, 4), *knew = r.need(elem), *vnew = r.need(elem), *sl = r.need(at::kInt);
    const at::Tensor *cos = r.maybe(elem, 2), *sin = r.maybe(elem, 2);
    const int64_t rope = r.integer();
    PyObject* width = r.next();  // rotary_dim: None is the tables' width; a number goes to the C call as it is, which refuses a bad one
    int64_t rotary_dim = width == Py_None ? 0 : r.integer(width);
    const at::Tensor *bt = r.maybe(at::kInt, 2), *cu_q = r.maybe(at::kLong), *cu_n = r.maybe(at::kLong);
    if (!r.ok || r.i != nargs || (q && q->scalar_type() != elem) || (cu_q != nullptr) != (cu_n != nullptr)) Py_RETURN_NONE;
    const int64_t dim = cu_n ? 3 : 4;
    if (knew->dim() != dim || vnew->dim() != dim || (q && q->dim() != dim) || (rope != 0 && (!cos || !sin))) Py_RETURN_NONE;
    const int64_t batch = sl->numel(), hkv = knew->size(-2), d = knew->size(-1), dv = vnew->size(-1);
    const int64_t n_new = cu_n ? knew->size(0) : knew->size(1), sq = !q ? 0 : cu_n ? q->size(0) : q->size(1);
    if (!rows_fit(*knew, *vnew) || !rows_fit(*k, *v) || k->size(2) != hkv || k->size(3) != d || v->size(3) != dv) Py_RETURN_NONE;
    if (cu_n ? !holds(cu_n, batch + 1) || !holds(cu_q, batch + 1) : knew->size(0) < batch) Py_RETURN_NONE;
    if ((bt ? bt->size(0) : k->size(0)) < batch) Py_RETURN_NONE;
    if (rope != 0 && (sin->size(1) != cos->size(1) || (width != Py_None && 2 * cos->size(1) < rotary_dim && rotary_dim <= d) ||
                      (q && (q->size(-1) != d || (!cu_n && q->size(0) < batch)))))
        Py_RETURN_NONE;
    if (width == Py_None && rope != 0) rotary_dim = 2 * cos->size(1);
    int rc;
    {
        pybind11::gil_scoped_release no_gil;
        const c10::cuda::CUDAGuard guard(r.device);
        rc = FmhaFwdAppendKV(ptr(q), ptr(k), ptr(knew), ptr(v), ptr(vnew), ptr(sl), (int64_t*)ptr(cu_q), (int64_t*)ptr(cu_n),
                             ptr(cos), ptr(sin), ptr(bt), nullptr, batch, sq, bt ? 0 : k->size(1), n_new,
                             q ? q->size(-2) : hkv, hkv, d, dv, rotary_dim, (int)rope, bt ? batch * bt->size(1) : 0,
                             bt ? k->size(1) : 0, stream_of(r.device), dtype_code(*k));
    }
    return PyLong_FromLong(rc);
    END_HANDLE_TH_ERRORS
}

PyObject* num_splits(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
    Reader r{args, nargs};
    const int64_t b = r.integer(), rows = r.integer();
    if (!r.ok) Py_RETURN_NONE;
    return PyLong_FromLongLong(num_splits_for(b, rows));
}

PyMethodDef methods[] = {
    {"_call_forward", (PyCFunction)(void (*)(void))call_forward, METH_FASTCALL, nullptr},
    {"_call_paged_prefill", (PyCFunction)(void (*)(void))call_paged_prefill, METH_FASTCALL, nullptr},
    {"_call_splitkv", (PyCFunction)(void (*)(void))call_splitkv, METH_FASTCALL, nullptr},
    {"_call_append_kv", (PyCFunction)(void (*)(void))call_append_kv, METH_FASTCALL, nullptr},
    {"_num_splits", (PyCFunction)(void (*)(void))num_splits, METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr},
};

}  // namespace

void add_calls(PyObject* module) {
    if (PyModule_AddFunctions(module, methods) != 0) throw pybind11::error_already_set();
}

}  // namespace calls
}  // namespace flashck
