// The five entry points of flash_attn_2_cuda for the calls that need nothing but their outputs allocated: plain tensors whose
// shapes, types and alignment the kernels take as they are.  Each function returns None for any other call (dropout, padding,
// copies, given outputs, every error): flash_attn_2_cuda/__init__.py does those, with the same C ABI underneath.
//
// Why native: filling the argument struct and checking the operands took 26 us (forward) and 47 us (backward) of interpreter
// time per call, next to kernels of 10 to 30 us for a short prompt, a small training step or a decode step.
#include <ATen/ATen.h>
#include <ATen/cuda/CUDAContext.h>
#include <torch/csrc/utils/pybind.h>

#include <cstdlib>
#include <initializer_list>
#include <limits>
#include <optional>

#include "fa_b200.h"

namespace {

using at::Tensor;
using MaybeTensor = std::optional<Tensor>;

// An ordinary dense CUDA tensor on device `dev` (no subclass, no tracing or functorch wrapper)
bool ordinary(const Tensor& t, c10::Device dev) {
  return t.defined() && t.is_cuda() && t.device() == dev && t.layout() == at::kStrided &&
         !t.key_set().has_any(c10::DispatchKeySet({c10::DispatchKey::Python, c10::DispatchKey::FuncTorchGradWrapper,
                                                   c10::DispatchKey::FuncTorchBatched, c10::DispatchKey::Functionalize}));
}

bool has_shape(const Tensor& t, std::initializer_list<int64_t> shape) { return t.sizes() == c10::IntArrayRef(shape); }

// What the kernels take without a copy: 16-byte pieces everywhere, and no dim that repeats its elements
bool direct(const Tensor& t, bool may_repeat = false) {
  if (t.stride(-1) != 1 || (reinterpret_cast<uintptr_t>(t.data_ptr()) & 15)) return false;
  for (int64_t i = 0; i + 1 < t.dim(); ++i)
    if (t.stride(i) % 8 || (t.stride(i) == 0 && !may_repeat)) return false;
  return true;
}

FaTensor view(const Tensor& t) {  // (batch, seq, head, dim), or packed (total, head, dim)
  if (t.dim() == 3) return FaTensor{t.data_ptr(), 0, t.stride(0), t.stride(1)};
  return FaTensor{t.data_ptr(), t.stride(0), t.stride(1), t.stride(2)};
}

bool takes(const Tensor& q) {
  if (!q.defined() || !q.is_cuda()) return false;
  if (q.scalar_type() != at::kHalf && q.scalar_type() != at::kBFloat16) return false;
  return q.device().index() == c10::cuda::current_device() && ordinary(q, q.device());
}

int32_t code(const Tensor& q) { return q.scalar_type() == at::kBFloat16 ? FA_DTYPE_BF16 : FA_DTYPE_FP16; }

// csrc/flash_attn/flash_api.cpp:113-114, 297: a window open on one side gets seqlen_k there
void windows(bool causal, int64_t seqlen_k, int64_t& wl, int64_t& wr) {
  if (causal) wr = 0;
  if (wl < 0 && wr >= 0) wl = seqlen_k;
  if (wl >= 0 && wr < 0) wr = seqlen_k;
}

bool fits(std::initializer_list<int64_t> values) {
  for (int64_t v : values)
    if (v < std::numeric_limits<int32_t>::min() || v > std::numeric_limits<int32_t>::max()) return false;
  return true;
}

int sm_count(c10::Device) { return at::cuda::getCurrentDeviceProperties()->multiProcessorCount; }

fa_stream_t stream_of(const Tensor& q) { return reinterpret_cast<fa_stream_t>(at::cuda::getCurrentCUDAStream(q.device().index()).stream()); }

void check(int status, const char* what) {
  if (status) throw std::runtime_error(std::string(what) + ": " + fa_last_error());
}

bool int32_vector(const Tensor& t, c10::Device dev, int64_t n) {
  return ordinary(t, dev) && t.scalar_type() == at::kInt && t.dim() == 1 && t.numel() == n && t.is_contiguous();
}

// fwd / varlen_fwd: [out, q, k, v, out, softmax_lse, None, rng_state]
// varlen: which of the two was called; packed operands without their offsets are an error, not a padded batch
py::object fwd(bool varlen, const Tensor& q, const Tensor& k, const Tensor& v, const MaybeTensor& cu_q, const MaybeTensor& cu_k, int64_t max_q,
               int64_t max_k, double scale, bool causal, int64_t wl, int64_t wr) {
  if (cu_q.has_value() != varlen || cu_k.has_value() != varlen) return py::none();
  if (!takes(q) || q.dim() != (varlen ? 3 : 4) || getenv("FA_B200_FWD_SPLITS")) return py::none();
  const c10::Device dev = q.device();
  for (const Tensor* t : {&k, &v})
    if (!ordinary(*t, dev) || t->scalar_type() != q.scalar_type() || t->dim() != q.dim()) return py::none();
  const int64_t heads = q.size(-2), heads_k = k.size(-2), d = q.size(-1);
  int64_t batch, sq, sk, total_q = 0, total_k = 0;
  if (varlen) {
    total_q = q.size(0), total_k = k.size(0);
    batch = cu_q->numel() - 1, sq = max_q, sk = max_k;
    if (!int32_vector(*cu_q, dev, batch + 1) || !int32_vector(*cu_k, dev, batch + 1) || total_q <= 0 || total_k <= 0) return py::none();
    if (!has_shape(k, {total_k, heads_k, d}) || !has_shape(v, {total_k, heads_k, d})) return py::none();
  } else {
    batch = q.size(0), sq = q.size(1), sk = k.size(1);
    if (!has_shape(k, {batch, sk, heads_k, d}) || !has_shape(v, {batch, sk, heads_k, d})) return py::none();
    if (sq == 1) return py::none();  // (may change places with the heads of a group)
  }
  if (batch <= 0 || sq <= 0 || sk <= 0 || d <= 0 || d > 256 || d % 8 || heads_k <= 0 || heads <= 0 || heads % heads_k) return py::none();
  if (!direct(q) || !direct(k) || !direct(v)) return py::none();
  windows(causal, sk, wl, wr);
  if (!fits({batch, sq, sk, heads, wl, wr, total_q, total_k, heads / heads_k * sq})) return py::none();

  const auto f32 = q.options().dtype(at::kFloat).requires_grad(false);
  Tensor out = at::empty(q.sizes(), q.options().requires_grad(false));
  Tensor lse = at::empty({batch, heads, sq}, f32);
  Tensor rng = at::empty({2}, f32.dtype(at::kLong));
  FaFwdArgs a = {};
  a.q = view(q), a.k = view(k), a.v = view(v), a.out = view(out);
  a.softmax_lse = static_cast<float*>(lse.data_ptr());
  a.lse_seqlen = a.seqlen_q = sq;
  a.batch = batch, a.seqlen_k = sk, a.heads = heads, a.heads_k = heads_k, a.head_dim = d;
  a.dtype = code(q), a.softmax_scale = scale;
  a.window_left = wl, a.window_right = wr;
  a.num_splits = 1;
  Tensor lse_acc, out_acc;
  if (varlen) {
    a.cu_seqlens_q = static_cast<int32_t*>(cu_q->data_ptr()), a.cu_seqlens_k = static_cast<int32_t*>(cu_k->data_ptr());
    a.total_q = total_q, a.total_k = total_k;
  } else {
    // the heads of a group share the kernel's 128-row tiles
    const int n = fa_fwd_num_splits(batch, heads_k, sq * (heads / heads_k), sk, d, sm_count(dev));
    if (n > 1) {
      lse_acc = at::empty({n, batch, heads, sq}, f32);
      out_acc = at::empty({n, batch, heads, sq, d}, f32);
      a.num_splits = n, a.lse_accum = static_cast<float*>(lse_acc.data_ptr()), a.out_accum = static_cast<float*>(out_acc.data_ptr());
    }
  }
  int status;
  {
    const fa_stream_t st = stream_of(q);
    py::gil_scoped_release unlocked;
    status = fa_fwd(&a, st);
  }
  check(status, varlen ? "flash_attn_2_cuda.varlen_fwd" : "flash_attn_2_cuda.fwd");
  py::list r(8);
  r[0] = out, r[1] = q, r[2] = k, r[3] = v, r[4] = out, r[5] = lse, r[6] = py::none(), r[7] = rng;
  return r;
}

// bwd / varlen_bwd: [dq, dk, dv, softmax_d]
py::object bwd(bool varlen, const Tensor& dout, const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& out, const Tensor& lse,
               const MaybeTensor& dq_, const MaybeTensor& dk_, const MaybeTensor& dv_, const MaybeTensor& cu_q, const MaybeTensor& cu_k,
               int64_t max_q, int64_t max_k, double scale, bool causal, int64_t wl, int64_t wr, bool deterministic) {
  if (cu_q.has_value() != varlen || cu_k.has_value() != varlen) return py::none();
  if (!takes(q) || q.dim() != (varlen ? 3 : 4) || !dq_ || !dk_ || !dv_) return py::none();
  const c10::Device dev = q.device();
  const Tensor &dq = *dq_, &dk = *dk_, &dv = *dv_;
  for (const Tensor* t : {&dout, &k, &v, &out, &dq, &dk, &dv})
    if (!ordinary(*t, dev) || t->scalar_type() != q.scalar_type() || t->dim() != q.dim()) return py::none();
  const int64_t heads = q.size(-2), heads_k = k.size(-2), d = q.size(-1);
  int64_t batch, sq, sk, total_q = 0, total_k = 0;
  if (varlen) {
    total_q = q.size(0), total_k = k.size(0);
    batch = cu_q->numel() - 1, sq = max_q, sk = max_k;
    if (!int32_vector(*cu_q, dev, batch + 1) || !int32_vector(*cu_k, dev, batch + 1) || total_q <= 0 || total_k <= 0) return py::none();
    if (!has_shape(k, {total_k, heads_k, d})) return py::none();
  } else {
    batch = q.size(0), sq = q.size(1), sk = k.size(1);
    if (!has_shape(k, {batch, sk, heads_k, d})) return py::none();
  }
  if (v.sizes() != k.sizes() || dk.sizes() != k.sizes() || dv.sizes() != k.sizes() || dout.sizes() != q.sizes() || out.sizes() != q.sizes() ||
      dq.sizes() != q.sizes())
    return py::none();
  if (batch <= 0 || sq <= 0 || sk <= 0 || d <= 0 || d > 256 || d % 8 || heads_k <= 0 || heads <= 0 || heads % heads_k) return py::none();
  for (const Tensor* t : {&dout, &q, &k, &v, &out, &dq, &dk, &dv})
    if (!direct(*t)) return py::none();
  if (!ordinary(lse, dev) || lse.scalar_type() != at::kFloat || lse.dim() != 3) return py::none();
  windows(causal, sk, wl, wr);
  const int64_t d_seqlen = (sq + 127) / 128 * 128;
  if (!fits({batch, d_seqlen, sk, heads, wl, wr, total_q, total_k, lse.size(-1)})) return py::none();

  const auto f32 = q.options().dtype(at::kFloat).requires_grad(false);
  Tensor softmax_d = at::empty({batch, heads, d_seqlen}, f32);
  Tensor dq_accum = at::empty({fa_bwd_workspace_bytes(batch, sq, heads, d, total_q, varlen) / 4}, f32);
  FaBwdArgs a = {};
  a.q = view(q), a.k = view(k), a.v = view(v), a.out = view(out), a.dout = view(dout);
  a.dq = view(dq), a.dk = view(dk), a.dv = view(dv);
  a.softmax_lse = static_cast<float*>(lse.data_ptr()), a.lse_seqlen = lse.size(-1);
  a.softmax_d = static_cast<float*>(softmax_d.data_ptr()), a.d_seqlen = d_seqlen;
  a.dq_accum = static_cast<float*>(dq_accum.data_ptr());
  a.batch = batch, a.seqlen_q = sq, a.seqlen_k = sk, a.heads = heads, a.heads_k = heads_k, a.head_dim = d;
  a.dtype = code(q), a.softmax_scale = scale;
  a.window_left = wl, a.window_right = wr;
  if (varlen) {
    a.cu_seqlens_q = static_cast<int32_t*>(cu_q->data_ptr()), a.cu_seqlens_k = static_cast<int32_t*>(cu_k->data_ptr());
    a.total_q = total_q, a.total_k = total_k;
  }
  a.deterministic = deterministic;
  int status;
  {
    const fa_stream_t st = stream_of(q);
    py::gil_scoped_release unlocked;
    status = fa_bwd(&a, st);
  }
  check(status, varlen ? "flash_attn_2_cuda.varlen_bwd" : "flash_attn_2_cuda.bwd");
  py::list r(4);
  r[0] = dq, r[1] = dk, r[2] = dv, r[3] = softmax_d;
  return r;
}

// fwd_kvcache: [out, softmax_lse]
py::object fwd_kvcache(const Tensor& q_in, const Tensor& kc, const Tensor& vc, const MaybeTensor& k, const MaybeTensor& v,
                       const MaybeTensor& lens, const MaybeTensor& cos, const MaybeTensor& sin, const MaybeTensor& batch_idx, double scale,
                       bool causal, int64_t wl, int64_t wr, bool interleaved, int64_t num_splits, const MaybeTensor& table) {
  if (!takes(q_in) || q_in.dim() != 4) return py::none();
  const c10::Device dev = q_in.device();
  const auto dtype = q_in.scalar_type();
  for (const Tensor* t : {&kc, &vc})
    if (!ordinary(*t, dev) || t->scalar_type() != dtype || t->dim() != 4 || !direct(*t, /*may_repeat=*/true)) return py::none();
  Tensor q = q_in;
  const int64_t batch = q.size(0), batch_c = kc.size(0), heads_k = kc.size(2), d = q.size(3);
  int64_t sq = q.size(1), heads = q.size(2), cap = kc.size(1), page = 0;
  if (vc.sizes() != kc.sizes() || kc.size(3) != d) return py::none();
  if (batch <= 0 || batch_c <= 0 || sq <= 0 || cap <= 0 || d <= 0 || d > 256 || d % 8 || heads_k <= 0 || heads <= 0 || heads % heads_k) return py::none();
  if (table) {
    if (!ordinary(*table, dev) || table->scalar_type() != at::kInt || table->dim() != 2 || table->size(0) != batch || table->stride(1) != 1 ||
        batch_idx || cap % 64)
      return py::none();
    page = cap;
    cap = table->size(1) * page;
    if (cap <= 0) return py::none();
  } else if (!batch_idx && batch_c < batch) {
    return py::none();
  }
  if (sq == 1) causal = false;
  windows(causal, cap, wl, wr);
  if (!direct(q)) return py::none();
  // one token: the heads of a group are the rows of a call (csrc/flash_attn/flash_api.cpp:299-307)
  const bool swapped = sq == 1 && heads > heads_k && wl < 0 && wr < 0;
  if (swapped) {
    if (!q.is_contiguous()) return py::none();
    sq = heads / heads_k, heads = heads_k;
    q = q.view({batch, heads, sq, d}).transpose(1, 2);
  }
  FaKvcacheArgs a = {};
  int64_t sn = 0;
  if (k) {
    if (!v || !lens || (sq > cap && !swapped)) return py::none();
    sn = k->size(1);
    for (const Tensor* t : {&*k, &*v})
      if (!ordinary(*t, dev) || t->scalar_type() != dtype || !has_shape(*t, {batch, sn, heads_k, d}) || !direct(*t, true)) return py::none();
    a.knew = view(*k), a.vnew = view(*v);
  }
  if (lens) {
    if (!int32_vector(*lens, dev, batch)) return py::none();
    a.cache_seqlens = static_cast<int32_t*>(lens->data_ptr());
  }
  if (batch_idx) {
    if (!int32_vector(*batch_idx, dev, batch)) return py::none();
    a.cache_batch_idx = static_cast<int32_t*>(batch_idx->data_ptr());
  }
  if (cos) {
    if (!k || !sin || cos->dim() != 2 || sin->sizes() != cos->sizes()) return py::none();
    for (const Tensor* t : {&*cos, &*sin})
      if (!ordinary(*t, dev) || t->scalar_type() != dtype || !t->is_contiguous()) return py::none();
    a.rotary_dim = cos->size(1) * 2, a.seqlen_ro = cos->size(0), a.rotary_interleaved = interleaved;
    if (a.rotary_dim <= 0 || a.rotary_dim > d || a.rotary_dim % 16 || cos->size(0) < cap) return py::none();
    a.rotary_cos = cos->data_ptr(), a.rotary_sin = sin->data_ptr();
  }
  if (num_splits < 0 || num_splits > 128 || !fits({batch, batch_c, cap, sq, heads, sn, wl, wr})) return py::none();

  const auto f32 = q.options().dtype(at::kFloat).requires_grad(false);
  const auto same = q.options().requires_grad(false);
  // (swapped: laid out as the caller sees it, so that no copy follows)
  Tensor out = swapped ? at::empty({batch, heads, sq, d}, same).transpose(1, 2) : at::empty({batch, sq, heads, d}, same);
  Tensor lse = at::empty({batch, heads, sq}, f32);
  a.q = view(q), a.kcache = view(kc), a.vcache = view(vc), a.out = view(out);
  a.softmax_lse = static_cast<float*>(lse.data_ptr());
  a.batch = batch, a.batch_cache = batch_c, a.seqlen_q = sq, a.seqlen_cache = cap, a.seqlen_new = sn;
  a.heads = heads, a.heads_k = heads_k, a.head_dim = d;
  a.dtype = code(q), a.softmax_scale = scale;
  a.window_left = wl, a.window_right = wr;
  a.q_rows_share_position = swapped;
  a.num_splits = num_splits;
  if (table) a.block_table = static_cast<int32_t*>(table->data_ptr()), a.block_table_stride = table->stride(0), a.page_block_size = page;
  int64_t lse_bytes = 0, out_bytes = 0;
  const int n = fa_kvcache_plan(&a, sm_count(dev), &lse_bytes, &out_bytes);
  if (n < 0) check(1, "flash_attn_2_cuda.fwd_kvcache");
  a.num_splits = n;  // what the workspaces are sized for
  Tensor lse_acc, out_acc, q_rot;
  if (n > 1) {
    lse_acc = at::empty({lse_bytes / 4}, f32);
    out_acc = at::empty({out_bytes / 4}, f32);
    a.lse_accum = static_cast<float*>(lse_acc.data_ptr()), a.out_accum = static_cast<float*>(out_acc.data_ptr());
  }
  if (cos) {
    q_rot = at::empty({batch, sq, heads, d}, same);
    a.q_rotated = q_rot.data_ptr();
  }
  int status;
  {
    const fa_stream_t st = stream_of(q);
    py::gil_scoped_release unlocked;
    status = fa_fwd_kvcache(&a, st);
  }
  check(status, "flash_attn_2_cuda.fwd_kvcache");
  if (swapped) {
    out = out.transpose(1, 2).view({batch, 1, heads * sq, d});
    lse = lse.view({batch, heads * sq, 1});
  }
  py::list r(2);
  r[0] = out, r[1] = lse;
  return r;
}

}  // namespace

PYBIND11_MODULE(_torch_glue, m) {
  m.def("fwd", &fwd);
  m.def("bwd", &bwd);
  m.def("fwd_kvcache", &fwd_kvcache);
}
