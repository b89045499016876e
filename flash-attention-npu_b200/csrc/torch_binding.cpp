// CPython / libtorch host path of the public attention calls: argument checks, output and workspace allocation, autograd
// and the launch without a line of Python in between.
//
// The Python front ends (flash_attn_npu_v2 / v3 interface.py) try these functions first.  A function takes over when every
// argument is of the ordinary kind -- plain CUDA tensors of one device with a contiguous last dimension, a head dim that
// needs no padding, no dispatch mode, no functorch transform -- and returns NotImplemented otherwise, also for every
// invalid argument: the Python path then serves the call or raises its own message.  So nothing here repeats an error text.
//
// Why: a small call is bound by its host work.  Dense forward of 2 x 128 tokens, 4 heads, head dim 64: 6 us of kernel
// behind 80 us of autograd.Function, torch.library dispatch and ctypes field stores in Python; its training step 350 us.
//
// The structure of the differentiable calls is that of the reference's autograd Functions
// (flash_attn_npu_v2/interface_arch22.py:774-900).
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/TracerMode.h>
#include <ATen/cuda/CUDAContext.h>
#include <c10/core/impl/LocalDispatchKeySet.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAGuard.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/custom_function.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/autograd/variable.h>

#include <cstring>
#include <exception>

#include "fa_b200.h"

namespace {

using at::Tensor;

// ------------------------------------------------------------------------------------------------ argument access
bool as_tensor(PyObject* o, const Tensor*& t) {
  if (o == Py_None) { t = nullptr; return true; }
  if (!THPVariable_CheckExact(o)) return false;
  t = &THPVariable_Unpack(o);
  return true;
}
bool as_int(PyObject* o, int64_t& v) {
  v = PyLong_AsLongLong(o);
  if (v == -1 && PyErr_Occurred()) { PyErr_Clear(); return false; }
  return true;
}
bool as_float(PyObject* o, double& v) {
  v = PyFloat_AsDouble(o);
  if (v == -1.0 && PyErr_Occurred()) { PyErr_Clear(); return false; }
  return true;
}
bool as_bool(PyObject* o, bool& v) {
  const int r = PyObject_IsTrue(o);
  if (r < 0) { PyErr_Clear(); return false; }
  v = r != 0;
  return true;
}
PyObject* not_implemented() { Py_RETURN_NOTIMPLEMENTED; }

// No dispatch mode (FakeTensorMode, make_fx, ...), no functorch transform and no torch.jit.trace is active: they record
// or replace operators, and a launch from here is none (a trace would keep the allocation of the outputs alone).
bool plain_eager() {
  return c10::impl::TorchDispatchModeTLS::stack_len() == 0 && !at::tracer::impl::is_dispatch_enabled() &&
         !c10::impl::tls_is_dispatch_key_included(c10::DispatchKey::FuncTorchDynamicLayerFrontMode);
}
bool plain(const Tensor& t) {
  static constexpr c10::DispatchKeySet special({c10::DispatchKey::Python, c10::DispatchKey::Conjugate, c10::DispatchKey::Negative,
                                                c10::DispatchKey::ZeroTensor, c10::DispatchKey::FuncTorchBatched,
                                                c10::DispatchKey::FuncTorchGradWrapper, c10::DispatchKey::Functionalize});
  return t.defined() && t.is_cuda() && t.layout() == at::kStrided && !t.key_set().has_any(special);
}
bool data_tensor(const Tensor* t, const Tensor& q, int64_t dim) {  // a 16-bit operand beside q
  return t && plain(*t) && t->scalar_type() == q.scalar_type() && t->device() == q.device() && t->dim() == dim && t->stride(-1) == 1;
}
bool index_tensor(const Tensor* t, const Tensor& q, int64_t numel) {  // optional contiguous int32 vector
  return !t || (plain(*t) && t->scalar_type() == at::kInt && t->device() == q.device() && t->dim() == 1 && t->numel() == numel &&
                t->is_contiguous());
}
const void* ptr(const Tensor* t) { return t ? t->const_data_ptr() : nullptr; }

// ------------------------------------------------------------------------------------------------ forward
struct FwdArgs {
  const Tensor *q, *k, *v, *k_new = nullptr, *v_new = nullptr, *cu_q = nullptr, *cu_k = nullptr, *seqused_k = nullptr,
               *batch_idx = nullptr, *table = nullptr, *cos = nullptr, *sin = nullptr, *alibi = nullptr;
  int64_t max_q = 0, max_k = 0, wl = -1, wr = -1, num_splits = 0;
  bool causal = false, interleaved = true;
  double scale = 1.0, softcap = 0.0;
  const char* plan = nullptr;  // bytes of a plan made ahead of the call
  Py_ssize_t plan_bytes = 0;
};

// Checks the arguments and fills everything of the parameter block but the outputs; false: not an ordinary call.
bool fill_params(const FwdArgs& a, fa_fwd_params& p) {
  std::memset(&p, 0, sizeof(p));
  if (!a.q || !plain(*a.q) || a.q->stride(-1) != 1) return false;
  const Tensor &q = *a.q;
  const bool packed_q = a.cu_q != nullptr, packed_k = a.cu_k != nullptr;
  if (q.scalar_type() != at::kHalf && q.scalar_type() != at::kBFloat16) return false;
  if (q.dim() != (packed_q ? 3 : 4) || !data_tensor(a.k, q, packed_k ? 3 : 4) || !data_tensor(a.v, q, packed_k ? 3 : 4)) return false;
  const Tensor &k = *a.k, &v = *a.v;
  if (k.sizes() != v.sizes() || k.size(-1) != q.size(-1)) return false;
  const int64_t d = q.size(-1), h = q.size(-2), h_k = k.size(-2);
  if (d % 8 != 0 || q.numel() == 0 || k.numel() == 0) return false;
  int64_t b = q.size(0);
  if (packed_q) {
    if (a.cu_q->dim() != 1) return false;
    b = a.cu_q->numel() - 1;
    if (b <= 0 || !index_tensor(a.cu_q, q, b + 1)) return false;
  }
  if (packed_k && (!packed_q || !index_tensor(a.cu_k, q, b + 1))) return false;
  if (!packed_k && !a.table && !a.batch_idx && k.size(0) != b) return false;
  if (!index_tensor(a.seqused_k, q, b) || !index_tensor(a.batch_idx, q, b)) return false;
  if (a.table && (!plain(*a.table) || a.table->scalar_type() != at::kInt || a.table->device() != q.device() || a.table->dim() != 2 ||
                  a.table->size(0) != b || a.table->stride(1) != 1))
    return false;
  p.q = ptr(a.q); p.k = ptr(a.k); p.v = ptr(a.v);
  p.dtype = q.scalar_type() == at::kBFloat16 ? FA_BF16 : FA_FP16;
  if (packed_q) {
    p.q_row_stride = q.stride(0); p.q_head_stride = q.stride(1);
    p.seqlen_q = (int32_t)a.max_q; p.total_q = (int32_t)q.size(0);
  } else {
    p.q_batch_stride = q.stride(0); p.q_row_stride = q.stride(1); p.q_head_stride = q.stride(2);
    p.seqlen_q = (int32_t)q.size(1); p.total_q = (int32_t)(b * q.size(1));
  }
  if (packed_k) {
    p.k_row_stride = k.stride(0); p.k_head_stride = k.stride(1);
    p.v_row_stride = v.stride(0); p.v_head_stride = v.stride(1);
    p.seqlen_k = (int32_t)a.max_k; p.total_k = (int32_t)k.size(0);
  } else {
    p.k_batch_stride = k.stride(0); p.k_row_stride = k.stride(1); p.k_head_stride = k.stride(2);
    p.v_batch_stride = v.stride(0); p.v_row_stride = v.stride(1); p.v_head_stride = v.stride(2);
    if (a.table || a.batch_idx) p.kv_outer = (int32_t)k.size(0);
    p.seqlen_k = (int32_t)k.size(1);
    if (a.table) {
      p.page_size = (int32_t)k.size(1);
      p.seqlen_k = (int32_t)(a.table->size(1) * k.size(1));
      p.block_table_batch_stride = a.table->stride(0);
    }
  }
  p.b = (int32_t)b; p.h = (int32_t)h; p.h_k = (int32_t)h_k; p.d = (int32_t)d;
  if ((a.k_new != nullptr) != (a.v_new != nullptr)) return false;
  if (a.k_new) {
    if (!data_tensor(a.k_new, q, 4) || !data_tensor(a.v_new, q, 4) || a.k_new->sizes() != a.v_new->sizes() ||
        a.k_new->size(0) != b || a.k_new->size(2) != h_k || a.k_new->size(3) != d)
      return false;
    p.k_new = ptr(a.k_new); p.v_new = ptr(a.v_new);
    p.seqlen_new = (int32_t)a.k_new->size(1);
    p.knew_batch_stride = a.k_new->stride(0); p.knew_row_stride = a.k_new->stride(1); p.knew_head_stride = a.k_new->stride(2);
    p.vnew_batch_stride = a.v_new->stride(0); p.vnew_row_stride = a.v_new->stride(1); p.vnew_head_stride = a.v_new->stride(2);
  }
  p.cu_seqlens_q = (const int32_t*)ptr(a.cu_q); p.cu_seqlens_k = (const int32_t*)ptr(a.cu_k);
  p.seqused_k = (const int32_t*)ptr(a.seqused_k); p.cache_batch_idx = (const int32_t*)ptr(a.batch_idx);
  p.block_table = (const int32_t*)ptr(a.table);
  if ((a.cos != nullptr) != (a.sin != nullptr)) return false;
  if (a.cos) {
    if (!data_tensor(a.cos, q, 2) || !data_tensor(a.sin, q, 2) || !a.cos->is_contiguous() || !a.sin->is_contiguous() ||
        a.cos->sizes() != a.sin->sizes())
      return false;
    p.rotary_cos = ptr(a.cos); p.rotary_sin = ptr(a.sin);
    p.rotary_seqlen = (int32_t)a.cos->size(0); p.rotary_dim = (int32_t)a.cos->size(1) * 2;
    p.rotary_interleaved = a.interleaved;
  }
  if (a.alibi) {
    const Tensor& s = *a.alibi;
    if (!plain(s) || s.scalar_type() != at::kFloat || s.device() != q.device() || s.stride(-1) != 1) return false;
    const bool per_head = s.dim() == 1 && s.size(0) == h, per_batch = s.dim() == 2 && s.size(0) == b && s.size(1) == h;
    if (!per_head && !per_batch) return false;
    p.alibi_slopes = (const float*)ptr(a.alibi);
    p.alibi_batch_stride = per_batch ? s.stride(0) : 0;
  }
  p.causal = a.causal; p.window_left = (int32_t)a.wl; p.window_right = (int32_t)a.wr;
  p.max_seqlen_k_known = -1;
  p.num_splits = (int32_t)a.num_splits;
  p.num_sm = at::cuda::getDeviceProperties(q.device().index())->multiProcessorCount;
  p.softmax_scale = (float)a.scale; p.softcap = (float)a.softcap;
  return true;
}

struct NoGil {  // a launch blocks when the queue is full: other Python threads go on meanwhile
  PyThreadState* state = PyGILState_Check() ? PyEval_SaveThread() : nullptr;
  ~NoGil() {
    if (state) PyEval_RestoreThread(state);
  }
};

struct Scratch {
  c10::Device device;
  Tensor tensor;
  std::exception_ptr error;  // out of memory: kept out of the C entry point the callback runs under
};
void* alloc_workspace(size_t bytes, void* ctx) {  // from torch's caching allocator, in the order of the current stream
  auto* s = static_cast<Scratch*>(ctx);
  try {
    s->tensor = at::empty({(int64_t)bytes}, at::TensorOptions().dtype(at::kByte).device(s->device));
    return s->tensor.data_ptr();
  } catch (...) {
    s->error = std::current_exception();
    return nullptr;
  }
}

// Allocates the outputs and launches; false: the library refused the call (the Python path repeats it for the message).
bool launch_forward(const FwdArgs& a, fa_fwd_params& p, Tensor& out, Tensor& lse) {
  const Tensor& q = *a.q;
  c10::cuda::CUDAGuard guard(q.device());
  out = at::empty(q.sizes(), q.options().requires_grad(false));
  const auto f32 = at::TensorOptions().dtype(at::kFloat).device(q.device());
  if (a.cu_q) {
    lse = at::empty({p.h, p.total_q}, f32);
    p.o_row_stride = out.stride(0); p.o_head_stride = out.stride(1);
    p.lse_head_stride = p.total_q;
  } else {
    lse = at::empty({p.b, p.h, p.seqlen_q}, f32);
    p.o_batch_stride = out.stride(0); p.o_row_stride = out.stride(1); p.o_head_stride = out.stride(2);
    p.lse_batch_stride = (int64_t)p.h * p.seqlen_q; p.lse_head_stride = p.seqlen_q;
  }
  p.o = out.data_ptr();
  p.lse = (float*)lse.data_ptr();
  Scratch ws{q.device(), Tensor(), nullptr};
  void* stream = at::cuda::getCurrentCUDAStream(q.device().index()).stream();
  NoGil nogil;
  const int rc = fa_b200_fwd_alloc(&p, a.plan, (size_t)a.plan_bytes, alloc_workspace, &ws, stream);
  if (ws.error) std::rethrow_exception(ws.error);
  return rc == FA_OK;
}

// ------------------------------------------------------------------------------------------------ backward
void run_backward(const Tensor& dout_in, const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& out, const Tensor& lse,
                  const Tensor& cu_q, const Tensor& cu_k, int64_t max_q, int64_t max_k, double scale, bool causal, int64_t wl,
                  int64_t wr, double softcap, Tensor& dq, Tensor& dk, Tensor& dv) {
  TORCH_CHECK(dout_in.is_cuda() && dout_in.scalar_type() == q.scalar_type(), "dout, q, k, v and out must have the same dtype");
  TORCH_CHECK(dout_in.sizes() == out.sizes(), "dout must have the shape of out");
  c10::cuda::CUDAGuard guard(q.device());
  const Tensor dout = dout_in.stride(-1) == 1 ? dout_in : dout_in.contiguous();
  dq = at::empty_like(q); dk = at::empty_like(k); dv = at::empty_like(v);
  fa_bwd_params p;
  std::memset(&p, 0, sizeof(p));
  p.q = q.const_data_ptr(); p.k = k.const_data_ptr(); p.v = v.const_data_ptr(); p.o = out.const_data_ptr();
  p.dout = dout.const_data_ptr(); p.lse = (const float*)lse.const_data_ptr();
  p.dq = dq.data_ptr(); p.dk = dk.data_ptr(); p.dv = dv.data_ptr();
  const bool packed = cu_q.defined();
  auto strides = [&](const Tensor& t, int64_t& bs, int64_t& rs, int64_t& hs) {
    bs = packed ? 0 : t.stride(0);
    rs = t.stride(-3);
    hs = t.stride(-2);
  };
  strides(q, p.q_batch_stride, p.q_row_stride, p.q_head_stride);
  strides(k, p.k_batch_stride, p.k_row_stride, p.k_head_stride);
  strides(v, p.v_batch_stride, p.v_row_stride, p.v_head_stride);
  strides(out, p.o_batch_stride, p.o_row_stride, p.o_head_stride);
  strides(dout, p.do_batch_stride, p.do_row_stride, p.do_head_stride);
  strides(dq, p.dq_batch_stride, p.dq_row_stride, p.dq_head_stride);
  strides(dk, p.dk_batch_stride, p.dk_row_stride, p.dk_head_stride);
  strides(dv, p.dv_batch_stride, p.dv_row_stride, p.dv_head_stride);
  if (packed) {
    p.cu_seqlens_q = (const int32_t*)cu_q.const_data_ptr(); p.cu_seqlens_k = (const int32_t*)cu_k.const_data_ptr();
    p.b = (int32_t)cu_q.numel() - 1; p.seqlen_q = (int32_t)max_q; p.seqlen_k = (int32_t)max_k;
    p.total_q = (int32_t)q.size(0); p.total_k = (int32_t)k.size(0);
    p.lse_head_stride = lse.stride(0);
  } else {
    p.b = (int32_t)q.size(0); p.seqlen_q = (int32_t)q.size(1); p.seqlen_k = (int32_t)k.size(1);
    p.total_q = p.b * p.seqlen_q;
    p.lse_batch_stride = lse.stride(0); p.lse_head_stride = lse.stride(1);
  }
  p.h = (int32_t)q.size(-2); p.h_k = (int32_t)k.size(-2); p.d = (int32_t)q.size(-1);
  p.dtype = q.scalar_type() == at::kBFloat16 ? FA_BF16 : FA_FP16;
  p.causal = causal; p.window_left = (int32_t)wl; p.window_right = (int32_t)wr;
  p.softmax_scale = (float)scale; p.softcap = (float)softcap;
  const size_t bytes = fa_b200_bwd_workspace_bytes(&p);
  const Tensor ws = at::empty({(int64_t)std::max<size_t>(bytes, 16)}, at::TensorOptions().dtype(at::kByte).device(q.device()));
  const int rc = fa_b200_bwd(&p, ws.data_ptr(), bytes, at::cuda::getCurrentCUDAStream(q.device().index()).stream());
  TORCH_CHECK(rc == FA_OK, fa_b200_last_error());
}

struct Refused : std::exception {};  // launch_forward said no inside the autograd function

struct Attention : public torch::autograd::Function<Attention> {
  static torch::autograd::variable_list forward(torch::autograd::AutogradContext* ctx, const Tensor& q, const Tensor& k,
                                                const Tensor& v, const FwdArgs* a, fa_fwd_params* p) {
    Tensor out, lse;
    if (!launch_forward(*a, *p, out, lse)) throw Refused();
    ctx->save_for_backward({q, k, v, out, lse, a->cu_q ? *a->cu_q : Tensor(), a->cu_k ? *a->cu_k : Tensor()});
    auto& d = ctx->saved_data;
    d["max_q"] = a->max_q; d["max_k"] = a->max_k; d["scale"] = a->scale; d["causal"] = a->causal;
    d["wl"] = a->wl; d["wr"] = a->wr; d["softcap"] = a->softcap;
    ctx->mark_non_differentiable({lse});
    ctx->set_materialize_grads(false);
    return {out, lse};
  }
  static torch::autograd::variable_list backward(torch::autograd::AutogradContext* ctx, torch::autograd::variable_list grads) {
    torch::autograd::variable_list g(5);
    if (!grads[0].defined()) return g;
    const auto s = ctx->get_saved_variables();
    auto& d = ctx->saved_data;
    run_backward(grads[0], s[0], s[1], s[2], s[3], s[4], s[5], s[6], d["max_q"].toInt(), d["max_k"].toInt(), d["scale"].toDouble(),
                 d["causal"].toBool(), d["wl"].toInt(), d["wr"].toInt(), d["softcap"].toDouble(), g[0], g[1], g[2]);
    return g;
  }
};

PyObject* two(Tensor out, Tensor lse) {
  PyObject* t = PyTuple_New(2);
  if (!t) return nullptr;
  PyTuple_SET_ITEM(t, 0, THPVariable_Wrap(std::move(out)));
  PyTuple_SET_ITEM(t, 1, THPVariable_Wrap(std::move(lse)));
  return t;
}

// attention(q, k, v, cu_seqlens_q, cu_seqlens_k, max_seqlen_q, max_seqlen_k, alibi_slopes, softmax_scale, causal, window_left,
//           window_right, softcap, num_splits) -> (out, lse), differentiable in q, k, v; or NotImplemented
PyObject* attention(PyObject*, PyObject* const* o, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  FwdArgs a;
  fa_fwd_params p;
  if (n != 14 || !plain_eager()) return not_implemented();
  if (!as_tensor(o[0], a.q) || !as_tensor(o[1], a.k) || !as_tensor(o[2], a.v) || !as_tensor(o[3], a.cu_q) || !as_tensor(o[4], a.cu_k) ||
      (a.cu_q && (!as_int(o[5], a.max_q) || !as_int(o[6], a.max_k))) || !as_tensor(o[7], a.alibi) || !as_float(o[8], a.scale) ||
      !as_bool(o[9], a.causal) || !as_int(o[10], a.wl) || !as_int(o[11], a.wr) || !as_float(o[12], a.softcap) || !as_int(o[13], a.num_splits))
    return not_implemented();
  if ((a.cu_q != nullptr) != (a.cu_k != nullptr) || !fill_params(a, p)) return not_implemented();
  for (const Tensor* t : {a.q, a.k, a.v})
    if (t->_fw_grad(/*level=*/0).defined()) return not_implemented();  // forward-mode differentiation: refused there
  Tensor out, lse;
  if (at::GradMode::is_enabled() && (a.q->requires_grad() || a.k->requires_grad() || a.v->requires_grad())) {
    if (a.alibi) return not_implemented();  // the backward says why not
    try {
      auto r = Attention::apply(*a.q, *a.k, *a.v, (const FwdArgs*)&a, &p);
      return two(std::move(r[0]), std::move(r[1]));
    } catch (const Refused&) {
      return not_implemented();
    }
  }
  if (!launch_forward(a, p, out, lse)) return not_implemented();
  return two(std::move(out), std::move(lse));
  END_HANDLE_TH_ERRORS
}

// kvcache(q, k_cache, v_cache, k, v, cu_seqlens_q, max_seqlen_q, cache_seqlens, cache_batch_idx, block_table, rotary_cos,
//         rotary_sin, rotary_interleaved, alibi_slopes, softmax_scale, causal, window_left, window_right, softcap, num_splits,
//         plan bytes or None, refuse_grad) -> (out, lse), or NotImplemented; neither is differentiable.  refuse_grad: also
//         NotImplemented when an input requires a gradient
PyObject* kvcache(PyObject*, PyObject* const* o, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  FwdArgs a;
  fa_fwd_params p;
  bool refuse_grad = false;
  if (n != 22 || !plain_eager()) return not_implemented();
  if (!as_tensor(o[0], a.q) || !as_tensor(o[1], a.k) || !as_tensor(o[2], a.v) || !as_tensor(o[3], a.k_new) || !as_tensor(o[4], a.v_new) ||
      !as_tensor(o[5], a.cu_q) || (a.cu_q && !as_int(o[6], a.max_q)) || !as_tensor(o[7], a.seqused_k) || !as_tensor(o[8], a.batch_idx) ||
      !as_tensor(o[9], a.table) || !as_tensor(o[10], a.cos) || !as_tensor(o[11], a.sin) || !as_bool(o[12], a.interleaved) ||
      !as_tensor(o[13], a.alibi) || !as_float(o[14], a.scale) || !as_bool(o[15], a.causal) || !as_int(o[16], a.wl) ||
      !as_int(o[17], a.wr) || !as_float(o[18], a.softcap) || !as_int(o[19], a.num_splits) || !as_bool(o[21], refuse_grad))
    return not_implemented();
  if (o[20] != Py_None && PyBytes_AsStringAndSize(o[20], const_cast<char**>(&a.plan), &a.plan_bytes) < 0) {
    PyErr_Clear();
    return not_implemented();
  }
  if (!fill_params(a, p)) return not_implemented();
  if (refuse_grad && at::GradMode::is_enabled())
    for (const Tensor* t : {a.q, a.k, a.v, a.k_new, a.v_new, a.cos, a.sin})
      if (t && t->requires_grad()) return not_implemented();
  if (a.k_new && (a.k->is_inference() || a.v->is_inference())) return not_implemented();
  Tensor out, lse;
  if (!launch_forward(a, p, out, lse)) return not_implemented();
  if (a.k_new) {  // the cache has been written to
    torch::autograd::impl::bump_version(*a.k);
    torch::autograd::impl::bump_version(*a.v);
  }
  return two(std::move(out), std::move(lse));
  END_HANDLE_TH_ERRORS
}

// plain_eager() -> bool: no mode, transform or trace is active that every function here would decline for
PyObject* py_plain_eager(PyObject*, PyObject*) { return PyBool_FromLong(plain_eager()); }

PyMethodDef methods[] = {
    {"attention", (PyCFunction)(void (*)(void))attention, METH_FASTCALL, "dense or packed attention; NotImplemented: use the Python path"},
    {"kvcache", (PyCFunction)(void (*)(void))kvcache, METH_FASTCALL, "attention over a KV cache; NotImplemented: use the Python path"},
    {"plain_eager", py_plain_eager, METH_NOARGS, "False: a mode, transform or trace is active and every function here declines"},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_native", "Native host path of the public attention calls.", -1, methods};

}  // namespace

PyMODINIT_FUNC PyInit__native() { return PyModule_Create(&module); }
