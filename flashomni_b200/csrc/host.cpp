// Host part of the usual calls: argument checks, output allocation and the C ABI calls of an op in one native function.
//
// Every function takes what the Python function of the same op takes and either does the whole call or returns None, and
// then the Python code goes through its own checks, conversions and error messages: only calls whose arguments are as the
// kernels take them are done here (plain strided CUDA tensors of the current device, no dispatch modes, contiguous int32
// indptrs, ...). An int is the error code of the C ABI. What it replaces is one Python expression per argument and ctypes
// conversions of up to 45 of them, which took longer than the kernels of small calls. Host time to issue a call, us, before ->
// here: attention of a short request 48 -> 14, of the image layer 40 -> 9, GEMM-Q 31 -> 11, GEMM-O 34 -> 10, a layer step 141-157 ->
// 59, block selection 26 -> 11, packing of both masks (two calls, each waiting for its bytes) 72 -> 31.
#include <Python.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>
#include <cuda_runtime_api.h>
#include <dlfcn.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/extension.h>

#include <cmath>
#include <cstdlib>

#include "../../include/flashomni_b200.h"

namespace {

struct Api {
  decltype(&fo_attn_run) attn_run;
  decltype(&fo_gemm_q) gemm_q;
  decltype(&fo_gemm_o) gemm_o;
  decltype(&fo_gemm_q_prepared) gemm_q_prepared;
  decltype(&fo_gemm_o_prepared) gemm_o_prepared;
  decltype(&fo_gemm_workspace_bytes) gemm_workspace_bytes;
  decltype(&fo_segment_packbits_polled) segment_packbits_polled;
  decltype(&fo_select_blocks_uniform) select_blocks_uniform;
  decltype(&fo_select_blocks_scratch_bytes) select_scratch_bytes;
};
Api g_api;
PyObject *s_kind, *s_key, *s_ws, *s_event, *s_cuda_event;

// A tensor as the kernels take it, or null: exactly torch.Tensor, strided, with storage, on device `dev` (< 0: any CUDA
// device), and not a wrapper that some mode or transform has put in its place.
const c10::DispatchKeySet kWrapped({c10::DispatchKey::Python, c10::DispatchKey::FuncTorchBatched, c10::DispatchKey::FuncTorchGradWrapper,
                                    c10::DispatchKey::Batched, c10::DispatchKey::Functionalize, c10::DispatchKey::Conjugate,
                                    c10::DispatchKey::Negative, c10::DispatchKey::ZeroTensor});
const at::Tensor* plain(PyObject* o, int dev) {
  if (!THPVariable_CheckExact(o)) return nullptr;
  const at::Tensor& t = THPVariable_Unpack(o);
  if (!t.defined() || !t.is_cuda() || t.layout() != at::kStrided) return nullptr;
  const c10::TensorImpl* impl = t.unsafeGetTensorImpl();
  if (!impl->has_storage() || impl->key_set().has_any(kWrapped)) return nullptr;
  if (dev >= 0 && t.get_device() != dev) return nullptr;
  return &t;
}
bool modes_active() { return c10::impl::TorchDispatchModeTLS::any_modes_set(); }
bool debug_checks() {  // then the Python path, which checks after the call
  const char* e = std::getenv("FLASHOMNI_B200_CHECK");
  return e != nullptr && e[0] != '\0' && !(e[0] == '0' && e[1] == '\0');
}
bool dense16(const at::Tensor& t) { return t.scalar_type() == at::kBFloat16 || t.scalar_type() == at::kHalf; }
int dtype_code(const at::Tensor& t) { return t.scalar_type() == at::kBFloat16 ? FO_DTYPE_BF16 : FO_DTYPE_F16; }
void* current_stream(int dev) { return c10::cuda::getCurrentCUDAStream(static_cast<c10::DeviceIndex>(dev)).stream(); }
bool contiguous_i32(const at::Tensor* t, int64_t n) {
  return t != nullptr && t->scalar_type() == at::kInt && t->dim() == 1 && t->size(0) == n && t->is_contiguous();
}
bool bytes(const at::Tensor* t) { return t != nullptr && t->scalar_type() == at::kByte && t->is_contiguous(); }
bool as_i64(PyObject* o, int64_t& v) {  // a plain int (bool included), as ctypes would take it
  if (!PyLong_Check(o)) return false;
  v = PyLong_AsLongLong(o);
  if (v == -1 && PyErr_Occurred()) { PyErr_Clear(); return false; }
  return v >= INT32_MIN && v <= INT32_MAX;
}
// Orders `stream` after a torch.cuda.Event (nothing if it has not been recorded, as Stream.wait_event does).
bool wait_event(void* stream, PyObject* event) {
  PyObject* h = PyObject_GetAttr(event, s_cuda_event);
  if (h == nullptr) { PyErr_Clear(); return false; }
  void* ev = PyLong_Check(h) ? PyLong_AsVoidPtr(h) : nullptr;
  Py_DECREF(h);
  if (ev == nullptr) { PyErr_Clear(); return true; }
  return cudaStreamWaitEvent(static_cast<cudaStream_t>(stream), static_cast<cudaEvent_t>(ev), 0) == cudaSuccess;
}

#define NOT_HERE Py_RETURN_NONE

// ------------------------------------------------------------------------------------------------ attention
struct AttnPlan {
  int64_t dev, is_bf16, fp8_kind /* -1: k and v have the type of q */, total_q, hq, hkv, d, total_kv, batch, nhd, fresh_out,
      lists[27] /* the plan array of fo_layer_lists */, status, partials;
};
constexpr int kPlanWords = sizeof(AttnPlan) / sizeof(int64_t);

void free_plan(PyObject* c) { delete static_cast<AttnPlan*>(PyCapsule_GetPointer(c, "fo.attn_plan")); }

PyObject* attn_plan(PyObject*, PyObject* const* args, Py_ssize_t n) {
  if (n != kPlanWords) return PyErr_Format(PyExc_TypeError, "attn_plan takes %d words", kPlanWords);
  int64_t w[kPlanWords];
  for (int i = 0; i < kPlanWords; ++i) {
    w[i] = args[i] == Py_None ? 0 : static_cast<int64_t>(PyLong_AsUnsignedLongLongMask(args[i]));
    if (PyErr_Occurred()) return nullptr;
  }
  AttnPlan* p = new AttnPlan;
  memcpy(p, w, sizeof(w));
  PyObject* c = PyCapsule_New(p, "fo.attn_plan", free_plan);
  if (c == nullptr) delete p;
  return c;
}

template <class T>
T* ptr(int64_t v) { return reinterpret_cast<T*>(v); }
int32_t i32(int64_t v) { return static_cast<int32_t>(v); }

// (plan, q, k, v, sparse_info, sparse_kv_info, info_indptr, kv_info_indptr, is_full, out, lse, return_lse, sm_scale, soft cap,
// event behind prepared lists or None)
PyObject* attn_run(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  if (nargs != 15) return PyErr_Format(PyExc_TypeError, "attn_run takes 15 arguments");
  const AttnPlan* p = static_cast<const AttnPlan*>(PyCapsule_GetPointer(args[0], "fo.attn_plan"));
  if (p == nullptr) return nullptr;
  const int dev = i32(p->dev);
  if (modes_active() || debug_checks() || plain(args[1], dev) == nullptr || c10::cuda::current_device() != dev) NOT_HERE;
  const at::Tensor *q = plain(args[1], dev), *k = plain(args[2], dev), *v = plain(args[3], dev);
  if (q == nullptr || k == nullptr || v == nullptr || q->dim() != 3 || k->dim() != 3 || v->dim() != 3) NOT_HERE;
  const auto qt = p->is_bf16 ? at::kBFloat16 : at::kHalf;
  const auto kvt = p->fp8_kind < 0 ? qt : (p->fp8_kind == 0 ? at::kFloat8_e4m3fn : at::kFloat8_e5m2);
  if (q->scalar_type() != qt || k->scalar_type() != kvt || v->scalar_type() != kvt) NOT_HERE;
  if (q->size(0) != p->total_q || q->size(1) != p->hq || q->size(2) != p->d) NOT_HERE;
  const int tok = p->nhd ? 0 : 1, hd = 1 - tok;
  if (k->size(tok) != p->total_kv || k->size(hd) != p->hkv || k->size(2) != p->d || !v->sizes().equals(k->sizes())) NOT_HERE;
  if (q->stride(2) != 1 || k->stride(2) != 1 || v->stride(2) != 1) NOT_HERE;
  const int full = PyObject_IsTrue(args[8]), return_lse = PyObject_IsTrue(args[11]);
  if (full < 0 || return_lse < 0) return nullptr;
  const at::Tensor *si = nullptr, *skv = nullptr, *ip = nullptr, *kp = nullptr;
  const bool prepared = args[14] != Py_None;
  if (!full) {
    si = plain(args[4], dev); skv = plain(args[5], dev); ip = plain(args[6], dev); kp = plain(args[7], dev);
    if (!bytes(si) || !bytes(skv) || !contiguous_i32(ip, p->batch + 1) || !contiguous_i32(kp, p->batch + 1)) NOT_HERE;
  } else if (args[4] != Py_None || args[5] != Py_None || args[6] != Py_None || args[7] != Py_None) {
    NOT_HERE;
  }
  const bool fresh = args[9] == Py_None;
  const at::Tensor* out_in = nullptr;
  if (fresh) {
    if (!p->fresh_out || prepared) NOT_HERE;
  } else {
    out_in = plain(args[9], dev);
    if (out_in == nullptr || out_in->scalar_type() != qt || !out_in->sizes().equals(q->sizes()) || out_in->stride(2) != 1 ||
        out_in->stride(0) % 8 != 0 || out_in->stride(1) % 8 != 0) NOT_HERE;
  }
  const at::Tensor* lse_in = nullptr;
  if (args[10] != Py_None) {
    lse_in = plain(args[10], dev);
    if (!return_lse || lse_in == nullptr || lse_in->scalar_type() != at::kFloat || lse_in->dim() != 2 ||
        lse_in->size(0) != p->total_q || lse_in->size(1) != p->hq || !lse_in->is_contiguous()) NOT_HERE;
  }
  double scale = 0.0, cap = 0.0;
  if (args[12] == Py_None) scale = 1.0 / std::sqrt(static_cast<double>(q->size(2)));
  else if (PyFloat_Check(args[12])) scale = PyFloat_AS_DOUBLE(args[12]);
  else NOT_HERE;
  if (args[13] != Py_None) {
    if (!PyFloat_Check(args[13])) NOT_HERE;
    cap = PyFloat_AS_DOUBLE(args[13]);
    if (!(cap >= 0.0)) NOT_HERE;
  }
  if (p->fp8_kind >= 0 && (k->numel() % 8 != 0 || k->numel() == 0 || !k->is_contiguous() || !v->is_contiguous())) NOT_HERE;

  void* stream = current_stream(dev);
  at::Tensor kv16, lse;
  fo_attn_call c;
  memset(&c, 0, sizeof(c));
  c.fp8_kind = i32(p->fp8_kind);
  if (p->fp8_kind >= 0) {  // both copies in one allocation
    kv16 = at::empty({2, k->size(0), k->size(1), k->size(2)}, q->options());
    c.kv_values = k->numel();
    c.k16 = kv16.data_ptr();
    c.v16 = static_cast<char*>(c.k16) + 2 * k->numel();
  }
  if (return_lse) lse = lse_in != nullptr ? *lse_in : at::empty({q->size(0), q->size(1)}, q->options().dtype(at::kFloat));
  const at::Tensor out = fresh ? at::empty(q->sizes(), q->options()) : *out_in;
  c.plan = p->lists;
  if (!full) {
    c.sparse_info = si->data_ptr<uint8_t>();
    c.sparse_info_bytes = si->numel();
    c.sparse_kv_info = skv->data_ptr<uint8_t>();
    c.sparse_kv_info_bytes = skv->numel();
    c.sparse_info_indptr = ip->data_ptr<int32_t>();
    c.sparse_kv_info_indptr = kp->data_ptr<int32_t>();
  }
  c.is_full = full;
  c.lists_ready = prepared ? 1 : 0;
  c.zero_inactive = fresh ? 1 : 0;   // an output allocated here reads as zero in q-blocks that are not computed
  c.dtype = dtype_code(*q);
  c.q = q->data_ptr();
  c.k = k->data_ptr();
  c.v = v->data_ptr();
  c.o = out.data_ptr();
  c.lse = return_lse ? lse.data_ptr<float>() : nullptr;
  c.total_q = p->total_q;
  c.total_kv = p->total_kv;
  c.num_qo_heads = i32(p->hq);
  c.num_kv_heads = i32(p->hkv);
  c.head_dim = i32(p->d);
  c.q_stride_n = q->stride(0);
  c.q_stride_h = q->stride(1);
  c.k_stride_n = k->stride(tok);   // (fp8: contiguous, and the copies are laid out alike)
  c.k_stride_h = k->stride(hd);
  c.v_stride_n = v->stride(tok);
  c.v_stride_h = v->stride(hd);
  c.o_stride_n = out.stride(0);
  c.o_stride_h = out.stride(1);
  c.partials = ptr<float>(p->partials);
  c.sm_scale = static_cast<float>(scale);
  c.logits_soft_cap = static_cast<float>(cap);
  c.status = ptr<int32_t>(p->status);
  if (prepared && !wait_event(stream, args[14])) return PyErr_Format(PyExc_RuntimeError, "waiting for the prepared work lists failed");
  int rc;
  {
    pybind11::gil_scoped_release no_gil;
    rc = g_api.attn_run(&c, stream);
  }
  if (rc != FO_OK) return PyLong_FromLong(rc);
  PyObject* o = fresh ? THPVariable_Wrap(out) : (Py_INCREF(args[9]), args[9]);
  if (!return_lse || o == nullptr) return o;
  PyObject* l = lse_in != nullptr ? (Py_INCREF(args[10]), args[10]) : THPVariable_Wrap(lse);
  if (l == nullptr) { Py_DECREF(o); return nullptr; }
  PyObject* t = PyTuple_New(2);
  if (t == nullptr) { Py_DECREF(o); Py_DECREF(l); return nullptr; }
  PyTuple_SET_ITEM(t, 0, o);
  PyTuple_SET_ITEM(t, 1, l);
  return t;
  END_HANDLE_TH_ERRORS
}

// ------------------------------------------------------------------------------------------------ GEMMs
struct GemmCall {
  const at::Tensor *a, *b;
  int64_t batch, m, n, k, num_heads, head_begin, head_dim, ntt, sq;
  int dev;
};
// the checks that both ops share; `head_dim` None: n / num_heads
bool gemm_args(GemmCall& g, PyObject* A, PyObject* B, PyObject* heads, PyObject* ntt, PyObject* sq, PyObject* head_begin, PyObject* head_dim) {
  if (modes_active() || debug_checks()) return false;
  g.a = plain(A, -1);
  if (g.a == nullptr) return false;   // (before the first look at CUDA)
  g.dev = c10::cuda::current_device();
  g.b = plain(B, g.dev);
  if (g.a->get_device() != g.dev || g.b == nullptr || g.a->dim() != 3 || g.b->dim() != 2 || !dense16(*g.a) || g.a->scalar_type() != g.b->scalar_type() ||
      !g.a->is_contiguous() || !g.b->is_contiguous()) return false;
  g.batch = g.a->size(0); g.m = g.a->size(1); g.k = g.a->size(2); g.n = g.b->size(0);
  if (g.b->size(1) != g.k || g.m % 128 != 0 || g.n % 128 != 0 || g.k % 32 != 0 || g.batch > INT32_MAX || g.m > INT32_MAX || g.n > INT32_MAX ||
      g.k > INT32_MAX) return false;
  if (!as_i64(heads, g.num_heads) || !as_i64(ntt, g.ntt) || !as_i64(sq, g.sq) || !as_i64(head_begin, g.head_begin)) return false;
  if (head_dim == Py_None) {
    if (g.num_heads <= 0) return false;
    g.head_dim = g.n / g.num_heads;
    return true;
  }
  return as_i64(head_dim, g.head_dim);
}
// The workspace of the current stream from the Python layer's table, or an undefined tensor.
at::Tensor workspace(PyObject* table, const GemmCall& g, void* stream) {
  PyObject* key = Py_BuildValue("(siK)", "cuda", g.dev, static_cast<unsigned long long>(reinterpret_cast<uintptr_t>(stream)));
  if (key == nullptr) { PyErr_Clear(); return {}; }
  PyObject* o = PyDict_GetItem(table, key);
  Py_DECREF(key);
  if (o == nullptr) return {};
  const at::Tensor* t = plain(o, g.dev);
  const size_t need = g_api.gemm_workspace_bytes(i32(g.batch), i32(g.m), i32(g.n), i32(g.k), i32(g.head_dim));
  return t != nullptr && static_cast<size_t>(t->numel()) >= need ? *t : at::Tensor();
}
// A prepared list (flashomni_b200.gemm.GemmWorklist) for this op and shape: its workspace, after ordering `stream` behind it.
at::Tensor worklist(PyObject* wl, const char* kind, int64_t batch, int64_t m, int64_t n_or_k, int64_t head_dim, int for_cache, int dev,
                    void* stream) {
  at::Tensor ws;
  PyObject *k = PyObject_GetAttr(wl, s_kind), *key = PyObject_GetAttr(wl, s_key), *w = PyObject_GetAttr(wl, s_ws),
           *ev = PyObject_GetAttr(wl, s_event);
  PyErr_Clear();
  if (k != nullptr && key != nullptr && w != nullptr && ev != nullptr && PyUnicode_Check(k) && PyUnicode_CompareWithASCIIString(k, kind) == 0 &&
      PyTuple_Check(key) && PyTuple_GET_SIZE(key) == 5) {
    const int64_t want[5] = {batch, m, n_or_k, head_dim, for_cache};
    bool same = true;
    for (int i = 0; i < 5 && same; ++i) {
      int64_t x = 0;
      same = as_i64(PyTuple_GET_ITEM(key, i), x) && x == want[i];
    }
    const at::Tensor* t = same ? plain(w, dev) : nullptr;
    if (t != nullptr && (ev == Py_None || wait_event(stream, ev))) ws = *t;
  }
  Py_XDECREF(k); Py_XDECREF(key); Py_XDECREF(w); Py_XDECREF(ev);
  return ws;
}

// (A, B, num_qo_heads, sparse_info, indptr, num_text_tokens, bias, out, sparse_q_size, is_full, head_begin, head_dim, worklist,
// workspaces)
PyObject* gemm_q(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  if (nargs != 14) return PyErr_Format(PyExc_TypeError, "gemm_q takes 14 arguments");
  GemmCall g;
  if (!gemm_args(g, args[0], args[1], args[2], args[5], args[8], args[10], args[11])) NOT_HERE;
  const int full = PyObject_IsTrue(args[9]);
  if (full < 0) return nullptr;
  const at::Tensor* bias = nullptr;
  if (args[6] != Py_None) {
    bias = plain(args[6], g.dev);
    if (bias == nullptr || bias->scalar_type() != g.a->scalar_type() || !bias->is_contiguous() || bias->numel() != g.n) NOT_HERE;
  }
  const at::Tensor* out = plain(args[7], g.dev);   // (None: the Python path, which zeroes a new one)
  if (out == nullptr || out->scalar_type() != g.a->scalar_type() || out->dim() != 3 || out->size(0) != g.batch || out->size(1) != g.m ||
      out->size(2) != g.n || !out->is_contiguous()) NOT_HERE;
  void* stream = current_stream(g.dev);
  int rc;
  if (args[12] != Py_None && !full) {
    const at::Tensor ws = worklist(args[12], "q", g.batch, g.m, g.n, g.head_dim, 0, g.dev, stream);
    if (!ws.defined()) NOT_HERE;
    pybind11::gil_scoped_release no_gil;
    rc = g_api.gemm_q_prepared(g.a->data_ptr(), g.b->data_ptr(), out->data_ptr(), bias != nullptr ? bias->data_ptr() : nullptr,
                               dtype_code(*g.a), i32(g.batch), i32(g.m), i32(g.n), i32(g.k), i32(g.head_dim), ws.data_ptr(),
                               static_cast<size_t>(ws.numel()), stream);
  } else {
    const at::Tensor *si = nullptr, *ip = nullptr;
    if (args[3] != Py_None && !bytes(si = plain(args[3], g.dev))) NOT_HERE;
    if (args[4] != Py_None && !contiguous_i32(ip = plain(args[4], g.dev), g.batch + 1)) NOT_HERE;
    if (!full && (si == nullptr || ip == nullptr)) NOT_HERE;
    const at::Tensor ws = workspace(args[13], g, stream);
    if (!ws.defined()) NOT_HERE;
    pybind11::gil_scoped_release no_gil;
    rc = g_api.gemm_q(g.a->data_ptr(), g.b->data_ptr(), out->data_ptr(), bias != nullptr ? bias->data_ptr() : nullptr, dtype_code(*g.a),
                      i32(g.batch), i32(g.m), i32(g.n), i32(g.k), i32(g.num_heads), i32(g.head_begin), i32(g.head_dim), i32(g.sq),
                      i32(g.ntt), full, si != nullptr ? si->data_ptr<uint8_t>() : nullptr, si != nullptr ? si->numel() : 0,
                      ip != nullptr ? ip->data_ptr<int32_t>() : nullptr, ws.data_ptr(), static_cast<size_t>(ws.numel()), stream);
  }
  if (rc != FO_OK) return PyLong_FromLong(rc);
  Py_INCREF(args[7]);
  return args[7];
  END_HANDLE_TH_ERRORS
}

// (A, B, num_qo_heads, sparse_info, indptr, num_text_tokens, bias, is_for_cache, sparse_q_size, head_begin, head_dim, out,
// worklist, workspaces)
PyObject* gemm_o(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  if (nargs != 14) return PyErr_Format(PyExc_TypeError, "gemm_o takes 14 arguments");
  GemmCall g;
  if (!gemm_args(g, args[0], args[1], args[2], args[5], args[8], args[9], args[10])) NOT_HERE;
  const int cache = PyObject_IsTrue(args[7]);
  if (cache < 0) return nullptr;
  const at::Tensor* init = nullptr;
  if (args[6] != Py_None) {
    init = plain(args[6], g.dev);
    if (init == nullptr || init->scalar_type() != g.a->scalar_type() || !init->is_contiguous() ||
        init->numel() != (cache ? g.n : g.batch * g.m * g.n)) NOT_HERE;
  }
  const int init_full = init != nullptr && !cache ? 1 : 0;
  const bool fresh = args[11] == Py_None;
  const at::Tensor* out_in = nullptr;
  if (!fresh) {
    out_in = plain(args[11], g.dev);
    if (out_in == nullptr || out_in->scalar_type() != g.a->scalar_type() || out_in->dim() != 3 || out_in->size(0) != g.batch ||
        out_in->size(1) != g.m || out_in->size(2) != g.n || !out_in->is_contiguous()) NOT_HERE;
  }
  void* stream = current_stream(g.dev);
  at::Tensor ws;
  const at::Tensor *si = nullptr, *ip = nullptr;
  const bool listed = args[12] != Py_None;
  if (listed) {
    ws = worklist(args[12], "o", g.batch, g.m, g.k, g.head_dim, cache, g.dev, stream);
  } else {
    if (!bytes(si = plain(args[3], g.dev)) || !contiguous_i32(ip = plain(args[4], g.dev), g.batch + 1)) NOT_HERE;
    ws = workspace(args[13], g, stream);
  }
  if (!ws.defined()) NOT_HERE;
  const at::Tensor out = fresh ? at::empty({g.batch, g.m, g.n}, g.a->options()) : *out_in;
  int rc;
  {
    pybind11::gil_scoped_release no_gil;
    const void* c = init != nullptr ? init->data_ptr() : nullptr;
    rc = listed ? g_api.gemm_o_prepared(g.a->data_ptr(), g.b->data_ptr(), out.data_ptr(), c, init_full, dtype_code(*g.a), i32(g.batch),
                                        i32(g.m), i32(g.n), i32(g.k), i32(g.head_dim), ws.data_ptr(),
                                        static_cast<size_t>(ws.numel()), stream)
                : g_api.gemm_o(g.a->data_ptr(), g.b->data_ptr(), out.data_ptr(), c, init_full, dtype_code(*g.a), i32(g.batch), i32(g.m),
                               i32(g.n), i32(g.k), i32(g.num_heads), i32(g.head_begin), i32(g.head_dim), i32(g.sq), i32(g.ntt), cache,
                               si->data_ptr<uint8_t>(), si->numel(), ip->data_ptr<int32_t>(), ws.data_ptr(),
                               static_cast<size_t>(ws.numel()), stream);
  }
  if (rc != FO_OK) return PyLong_FromLong(rc);
  if (fresh) return THPVariable_Wrap(out);
  Py_INCREF(args[11]);
  return args[11];
  END_HANDLE_TH_ERRORS
}

// ------------------------------------------------------------------------------------------------ masks
// (x, indptr, little)
PyObject* segment_packbits(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  if (nargs != 3) return PyErr_Format(PyExc_TypeError, "segment_packbits takes 3 arguments");
  if (modes_active() || plain(args[0], -1) == nullptr) NOT_HERE;
  const int dev = c10::cuda::current_device();
  const at::Tensor *x = plain(args[0], dev), *ip = plain(args[1], dev);
  const int little = PyObject_IsTrue(args[2]);
  if (little < 0) return nullptr;
  if (x == nullptr || ip == nullptr || !x->is_contiguous() || !ip->is_contiguous() || ip->dim() != 1) NOT_HERE;
  const auto xt = x->scalar_type(), it = ip->scalar_type();
  if ((xt != at::kBool && xt != at::kByte && xt != at::kChar) || (it != at::kInt && it != at::kLong)) NOT_HERE;
  const int64_t n = x->numel(), nseg = ip->size(0) - 1;
  if (nseg < 1 || nseg > 1024 || n <= 0 || n >= (1ll << 33)) NOT_HERE;
  const int64_t capacity = (n + 7 * nseg) / 8;
  at::Tensor y = at::empty({capacity}, x->options().dtype(at::kByte));
  at::Tensor bytes_indptr = at::empty({nseg + 1}, x->options().dtype(at::kInt));
  constexpr int kWords = 148;   // (one block per SM: beyond that the wait for the stream is a small part of the call)
  const at::Tensor words = at::empty({kWords}, at::TensorOptions().dtype(at::kLong).pinned_memory(true));
  void* stream = current_stream(dev);
  int rc;
  {
    pybind11::gil_scoped_release no_gil;   // (this call waits)
    rc = g_api.segment_packbits_polled(static_cast<const uint8_t*>(x->data_ptr()), n, ip->data_ptr(), it == at::kLong ? 1 : 0, i32(nseg),
                                       capacity, little, y.data_ptr<uint8_t>(), bytes_indptr.data_ptr<int32_t>(),
                                       words.data_ptr<int64_t>(), kWords, stream);
  }
  if (rc != FO_OK) return PyLong_FromLong(rc);
  const int64_t nbytes = *words.data_ptr<int64_t>();
  if (nbytes < 0) NOT_HERE;   // (refused: the Python code finds the reason)
  at::Tensor packed = y.narrow(0, 0, nbytes);
  // segments that cover little of x: the result does not keep the rest of the allocation alive (below a megabyte, the
  // allocator's own granularity, the copy would cost more than it frees)
  if (capacity - nbytes > (nbytes > (1 << 20) ? nbytes : (1 << 20))) {
    pybind11::gil_scoped_release no_gil;
    packed = packed.clone();
    c10::cuda::getCurrentCUDAStream(static_cast<c10::DeviceIndex>(dev)).synchronize();
  }
  PyObject* a = THPVariable_Wrap(packed);
  PyObject* b = THPVariable_Wrap(bytes_indptr);
  PyObject* t = a != nullptr && b != nullptr ? PyTuple_New(2) : nullptr;
  if (t == nullptr) { Py_XDECREF(a); Py_XDECREF(b); return nullptr; }
  PyTuple_SET_ITEM(t, 0, a);
  PyTuple_SET_ITEM(t, 1, b);
  return t;
  END_HANDLE_TH_ERRORS
}

// (pooled_score, num_text_blocks, q_threshold, kv_threshold, zero_inactive)
PyObject* select_blocks(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  if (nargs != 5) return PyErr_Format(PyExc_TypeError, "select_blocks takes 5 arguments");
  if (modes_active() || plain(args[0], -1) == nullptr) NOT_HERE;
  const int dev = c10::cuda::current_device();
  const at::Tensor* s = plain(args[0], dev);
  int64_t t2t = 0;
  if (s == nullptr || s->dim() != 4 || s->scalar_type() != at::kFloat || !s->is_contiguous() || s->size(2) != s->size(3) || s->numel() == 0 ||
      !as_i64(args[1], t2t) || !PyFloat_Check(args[2]) || !PyFloat_Check(args[3])) NOT_HERE;
  const int64_t B = s->size(0), H = s->size(1), n = s->size(2);
  const double qt = PyFloat_AS_DOUBLE(args[2]), kt = PyFloat_AS_DOUBLE(args[3]);
  if (t2t < 0 || t2t > n || B > INT32_MAX || H > INT32_MAX || n > INT32_MAX || !(std::fabs(qt) <= 1e30) || !(std::fabs(kt) <= 1e30)) NOT_HERE;
  const int zero = PyObject_IsTrue(args[4]);
  if (zero < 0) return nullptr;
  const int64_t info_seg = (n * H + 7) / 8, kv_seg = (n * H * n + 7) / 8, kv_alloc = (B * kv_seg + 3) / 4 * 4;
  const auto u8 = s->options().dtype(at::kByte), i4 = s->options().dtype(at::kInt);
  at::Tensor si = at::empty({B * info_seg}, u8), skv = at::empty({kv_alloc}, u8), ip = at::empty({B + 1}, i4), kp = at::empty({B + 1}, i4);
  const at::Tensor scratch = at::empty({static_cast<int64_t>(g_api.select_scratch_bytes(i32(B), i32(n)))}, u8);
  int rc;
  {
    void* stream = current_stream(dev);
    pybind11::gil_scoped_release no_gil;
    rc = g_api.select_blocks_uniform(s->data_ptr<float>(), i32(B), i32(H), i32(n), i32(t2t), static_cast<float>(qt), static_cast<float>(kt),
                                     zero, si.data_ptr<uint8_t>(), si.numel(), skv.data_ptr<uint8_t>(), skv.numel(),
                                     ip.data_ptr<int32_t>(), kp.data_ptr<int32_t>(), scratch.data_ptr(), static_cast<size_t>(scratch.numel()),
                                     stream);
  }
  if (rc != FO_OK) return PyLong_FromLong(rc);
  PyObject* r[4] = {THPVariable_Wrap(si), THPVariable_Wrap(kv_alloc == B * kv_seg ? skv : skv.narrow(0, 0, B * kv_seg)), THPVariable_Wrap(ip),
                    THPVariable_Wrap(kp)};
  PyObject* t = r[0] && r[1] && r[2] && r[3] ? PyTuple_New(4) : nullptr;
  for (int i = 0; i < 4; ++i) {
    if (t != nullptr) PyTuple_SET_ITEM(t, i, r[i]); else Py_XDECREF(r[i]);
  }
  return t;
  END_HANDLE_TH_ERRORS
}

// ------------------------------------------------------------------------------------------------ module
// bind(handle of the CUDA library as ctypes holds it)
PyObject* bind(PyObject*, PyObject* arg) {
  void* h = PyLong_AsVoidPtr(arg);
  if (PyErr_Occurred()) return nullptr;
  Api a;
  const char* missing = nullptr;
  auto get = [&](auto& fn, const char* name) {
    fn = reinterpret_cast<std::decay_t<decltype(fn)>>(dlsym(h, name));
    if (fn == nullptr) missing = name;
  };
  get(a.attn_run, "fo_attn_run");
  get(a.gemm_q, "fo_gemm_q");
  get(a.gemm_o, "fo_gemm_o");
  get(a.gemm_q_prepared, "fo_gemm_q_prepared");
  get(a.gemm_o_prepared, "fo_gemm_o_prepared");
  get(a.gemm_workspace_bytes, "fo_gemm_workspace_bytes");
  get(a.segment_packbits_polled, "fo_segment_packbits_polled");
  get(a.select_blocks_uniform, "fo_select_blocks_uniform");
  get(a.select_scratch_bytes, "fo_select_blocks_scratch_bytes");
  if (missing != nullptr) return PyErr_Format(PyExc_RuntimeError, "flashomni_b200: the native library has no %s", missing);
  g_api = a;
  Py_RETURN_NONE;
}

// What it was compiled for, as flashomni_b200._native.host_abi() names it: the caller compares before any other function is used.
PyObject* abi(PyObject*, PyObject*) { return PyUnicode_FromString(FO_HOST_ABI); }

#define FAST(f) {#f, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(f)), METH_FASTCALL, nullptr}
PyMethodDef kMethods[] = {FAST(attn_plan), FAST(attn_run), FAST(gemm_q), FAST(gemm_o), FAST(segment_packbits), FAST(select_blocks),
                          {"bind", bind, METH_O, nullptr}, {"abi", abi, METH_NOARGS, nullptr}, {nullptr, nullptr, 0, nullptr}};
PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_fo_host", nullptr, -1, kMethods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__fo_host() {
  s_kind = PyUnicode_InternFromString("kind");
  s_key = PyUnicode_InternFromString("key");
  s_ws = PyUnicode_InternFromString("ws");
  s_event = PyUnicode_InternFromString("event");
  s_cuda_event = PyUnicode_InternFromString("cuda_event");
  return PyModule_Create(&kModule);
}
