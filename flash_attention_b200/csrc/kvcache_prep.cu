// KV-cache append + rotary embedding as a stand-alone launch, used when a decode call does not fit
// the fused single-token kernel (several new tokens, long query blocks, odd head dims).
// Same effect as the prologue of compute_attn_1rowblock_splitkv
// (csrc/flash_attn/src/flash_fwd_kernel.h:768-891): new K rows are rotated at absolute position
// cache_seqlens[b] + i and written with the new V rows into the cache at batch slot
// cache_batch_idx[b]; q is rotated at cache_seqlens[b] + i when the mask is causal/local and at
// cache_seqlens[b] for every row otherwise.  Rotary math is fp32, rounded once
// (csrc/flash_attn/src/utils.h:391-517).
#include "fa_common.cuh"

namespace fa {

template <typename T>
__device__ __forceinline__ void rotate_row(const T* src, T* dst, const T* cosr, const T* sinr, int D, int rdim,
                                           bool interleaved, int lane_step, int lane0) {
  // cosr/sinr: row of rdim/2 values, or nullptr for a plain copy
  const int half = rdim / 2;
  for (int d = lane0; d < D; d += lane_step) {
    float x = Pack<T>::one(src[d]);
    float y = x;
    if (cosr && d < rdim) {
      int i, partner;
      bool first;
      if (interleaved) {
        i = d >> 1;
        first = (d & 1) == 0;
        partner = first ? d + 1 : d - 1;
      } else {
        first = d < half;
        i = first ? d : d - half;
        partner = first ? d + half : d - half;
      }
      float c = Pack<T>::one(cosr[i]), s = Pack<T>::one(sinr[i]);
      float xp = Pack<T>::one(src[partner]);
      y = first ? x * c - xp * s : x * c + xp * s;
    }
    dst[d] = Pack<T>::from(y);
  }
}

// grid: (seqlen_new + seqlen_q, max(heads, heads_k), batch); block 128
template <typename T>
__global__ void __launch_bounds__(128) kvcache_prep_kernel(const __grid_constant__ FaKvcacheArgs p, int q_follows_rows) {
  const int b = blockIdx.z, hh = blockIdx.y;
  const int L = p.cache_seqlens ? p.cache_seqlens[b] : p.seqlen_cache;
  const T* cosb = reinterpret_cast<const T*>(p.rotary_cos);
  const T* sinb = reinterpret_cast<const T*>(p.rotary_sin);
  const int half = p.rotary_dim / 2;
  const int D = p.head_dim;
  int r = blockIdx.x;
  if (r < p.seqlen_new) {
    if (hh >= p.heads_k || !p.knew.ptr) return;
    const int pos = L + r;
    if (pos >= p.seqlen_cache) return;
    int64_t cb = p.cache_batch_idx ? p.cache_batch_idx[b] : b;
    int row = pos;
    if (p.block_table) {  // paged cache: the table names the page, the row is the position inside it
      cb = p.block_table[(int64_t)b * p.block_table_stride + pos / p.page_block_size];
      row = pos % p.page_block_size;
    }
    const T* ks = reinterpret_cast<const T*>(p.knew.ptr) + b * p.knew.stride_b + r * p.knew.stride_s + hh * p.knew.stride_h;
    const T* vs = reinterpret_cast<const T*>(p.vnew.ptr) + b * p.vnew.stride_b + r * p.vnew.stride_s + hh * p.vnew.stride_h;
    T* kd = reinterpret_cast<T*>(p.kcache.ptr) + cb * p.kcache.stride_b + (int64_t)row * p.kcache.stride_s + hh * p.kcache.stride_h;
    T* vd = reinterpret_cast<T*>(p.vcache.ptr) + cb * p.vcache.stride_b + (int64_t)row * p.vcache.stride_s + hh * p.vcache.stride_h;
    const bool rot = cosb != nullptr && pos < p.seqlen_ro;
    rotate_row<T>(ks, kd, rot ? cosb + (int64_t)pos * half : nullptr, rot ? sinb + (int64_t)pos * half : nullptr, D,
                  p.rotary_dim, p.rotary_interleaved != 0, blockDim.x, threadIdx.x);
    for (int d = threadIdx.x; d < D; d += blockDim.x) vd[d] = vs[d];
  } else {
    r -= p.seqlen_new;
    if (hh >= p.heads || !p.q_rotated || r >= p.seqlen_q) return;
    const int pos = L + (q_follows_rows ? r : 0);
    const T* qs = reinterpret_cast<const T*>(p.q.ptr) + b * p.q.stride_b + r * p.q.stride_s + hh * p.q.stride_h;
    // q_rotated is contiguous (batch, seqlen_q, heads, D)
    T* qd = reinterpret_cast<T*>(p.q_rotated) + (((int64_t)b * p.seqlen_q + r) * p.heads + hh) * D;
    const bool rot = cosb != nullptr && pos < p.seqlen_ro;
    rotate_row<T>(qs, qd, rot ? cosb + (int64_t)pos * half : nullptr, rot ? sinb + (int64_t)pos * half : nullptr, D,
                  p.rotary_dim, p.rotary_interleaved != 0, blockDim.x, threadIdx.x);
  }
}

// Bound by memory latency and launch (4 x 128 tokens, 32/8 heads of 128: 24 us a byte pair at a time, 5 us here).
// The same work in 16-byte pieces: a thread takes one piece of a row and, where the halves are turned against each
// other, its partner piece.  The scalar kernel above moves 2 bytes a thread in 128-thread blocks that live for one row.
// Items of a row: K and Q rows have rotary_dim / 16 pairs of pieces (NeoX) or rotary_dim / 8 pieces (interleaved) to
// turn and (head_dim - rotary_dim) / 8 to copy, V rows head_dim / 8 to copy.
template <typename T>
__device__ __forceinline__ uint4 turn8(const uint4& x, const uint4& other, const uint4& c, const uint4& s, bool first) {
  const uint32_t xs[4] = {x.x, x.y, x.z, x.w}, os[4] = {other.x, other.y, other.z, other.w}, cs[4] = {c.x, c.y, c.z, c.w},
                 ss[4] = {s.x, s.y, s.z, s.w};
  uint32_t y[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float a = Pack<T>::lo(xs[i]), b = Pack<T>::hi(xs[i]), oa = Pack<T>::lo(os[i]), ob = Pack<T>::hi(os[i]);
    const float ca = Pack<T>::lo(cs[i]), cb = Pack<T>::hi(cs[i]), sa = Pack<T>::lo(ss[i]), sb = Pack<T>::hi(ss[i]);
    y[i] = first ? Pack<T>::two(a * ca - oa * sa, b * cb - ob * sb) : Pack<T>::two(a * ca + oa * sa, b * cb + ob * sb);
  }
  return make_uint4(y[0], y[1], y[2], y[3]);
}

template <typename T>
__global__ void __launch_bounds__(256) kvcache_prep_vec_kernel(const __grid_constant__ FaKvcacheArgs p, int q_follows_rows) {
  const int b = blockIdx.y;
  const int L = p.cache_seqlens ? p.cache_seqlens[b] : p.seqlen_cache;
  const int D = p.head_dim, half = p.rotary_dim / 2;
  const bool rotary = p.rotary_cos != nullptr;
  const int turns = !rotary ? 0 : (p.rotary_interleaved ? p.rotary_dim / 8 : half / 8);
  const int turned = rotary ? p.rotary_dim : 0;                 // elements of a row that the turns cover
  const int per_row = turns + (D - turned) / 8, per_v = D / 8;  // items of a K or Q row, of a V row
  const int k_items = p.seqlen_new * p.heads_k * per_row, v_items = p.seqlen_new * p.heads_k * per_v;
  const int q_items = p.q_rotated ? p.seqlen_q * p.heads * per_row : 0;
  int i = blockIdx.x * 256 + threadIdx.x;
  if (i >= k_items + v_items + q_items) return;
  const bool is_q = i >= k_items + v_items, is_v = !is_q && i >= k_items;
  i -= is_q ? k_items + v_items : is_v ? k_items : 0;
  const int per = is_v ? per_v : per_row, heads = is_q ? p.heads : p.heads_k;
  const int item = i % per, hh = (i / per) % heads, r = i / per / heads;
  const int pos = L + (!is_q || q_follows_rows ? r : 0);
  const FaTensor& st = is_q ? p.q : is_v ? p.vnew : p.knew;
  const T* src = reinterpret_cast<const T*>(st.ptr) + b * st.stride_b + r * st.stride_s + hh * st.stride_h;
  T* dst;
  if (is_q) {
    dst = reinterpret_cast<T*>(p.q_rotated) + (((int64_t)b * p.seqlen_q + r) * p.heads + hh) * D;
  } else {
    if (pos >= p.seqlen_cache) return;
    int64_t cb = p.cache_batch_idx ? p.cache_batch_idx[b] : b;
    int row = pos;
    if (p.block_table) {
      cb = p.block_table[(int64_t)b * p.block_table_stride + pos / p.page_block_size];
      row = pos % p.page_block_size;
    }
    const FaTensor& ct = is_v ? p.vcache : p.kcache;
    dst = reinterpret_cast<T*>(ct.ptr) + cb * ct.stride_b + (int64_t)row * ct.stride_s + hh * ct.stride_h;
  }
  const uint4* s16 = reinterpret_cast<const uint4*>(src);
  uint4* d16 = reinterpret_cast<uint4*>(dst);
  if (is_v || item >= turns) {
    const int c = is_v ? item : turned / 8 + item - turns;
    d16[c] = s16[c];
    return;
  }
  const bool turn = pos < p.seqlen_ro;
  const T* cosr = reinterpret_cast<const T*>(p.rotary_cos) + (int64_t)pos * half;
  const T* sinr = reinterpret_cast<const T*>(p.rotary_sin) + (int64_t)pos * half;
  if (p.rotary_interleaved) {
    uint4 x = s16[item];
    if (turn) {
      const uint2 c = reinterpret_cast<const uint2*>(cosr)[item], s = reinterpret_cast<const uint2*>(sinr)[item];
      uint32_t xs[4] = {x.x, x.y, x.z, x.w};
      const uint32_t cs[2] = {c.x, c.y}, ss[2] = {s.x, s.y};
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float ce = e & 1 ? Pack<T>::hi(cs[e >> 1]) : Pack<T>::lo(cs[e >> 1]);
        const float se = e & 1 ? Pack<T>::hi(ss[e >> 1]) : Pack<T>::lo(ss[e >> 1]);
        const float a = Pack<T>::lo(xs[e]), o = Pack<T>::hi(xs[e]);
        xs[e] = Pack<T>::two(a * ce - o * se, o * ce + a * se);
      }
      x = make_uint4(xs[0], xs[1], xs[2], xs[3]);
    }
    d16[item] = x;
  } else {
    const int h8 = half / 8;
    uint4 x = s16[item], y = s16[item + h8];
    if (turn) {
      const uint4 c = reinterpret_cast<const uint4*>(cosr)[item], s = reinterpret_cast<const uint4*>(sinr)[item];
      const uint4 x1 = turn8<T>(x, y, c, s, true);
      y = turn8<T>(y, x, c, s, false);
      x = x1;
    }
    d16[item] = x;
    d16[item + h8] = y;
  }
}

static bool pieces_aligned(const FaTensor& t) {
  return (reinterpret_cast<uintptr_t>(t.ptr) & 15) == 0 && t.stride_s % 8 == 0 && t.stride_h % 8 == 0 && t.stride_b % 8 == 0;
}

// 16-byte pieces need 16-byte rows everywhere (the tables included) and an item count that fits an int
static bool prep_in_pieces(const FaKvcacheArgs& a) {
  if (a.head_dim % 8 || (a.rotary_cos && a.rotary_dim % 16)) return false;
  if (a.knew.ptr && !(pieces_aligned(a.knew) && pieces_aligned(a.vnew) && pieces_aligned(a.kcache) && pieces_aligned(a.vcache)))
    return false;
  if (a.q_rotated && (!pieces_aligned(a.q) || (reinterpret_cast<uintptr_t>(a.q_rotated) & 15))) return false;
  if ((reinterpret_cast<uintptr_t>(a.rotary_cos) & 15) || (reinterpret_cast<uintptr_t>(a.rotary_sin) & 15)) return false;
  return ((int64_t)a.seqlen_new * 2 * a.heads_k + (int64_t)a.seqlen_q * a.heads) * (a.head_dim / 8) < (1ll << 30) && a.batch <= 65535;
}

int kvcache_prep(const FaKvcacheArgs& a, int q_follows_rows, cudaStream_t st) {
  int rows = (a.knew.ptr ? a.seqlen_new : 0);
  FaKvcacheArgs c = a;
  if (!a.knew.ptr) c.seqlen_new = 0;
  if (a.q_rotated) rows += a.seqlen_q;
  if (rows == 0) return 0;
  if (prep_in_pieces(c)) {
    const int64_t items = ((int64_t)c.seqlen_new * 2 * c.heads_k + (c.q_rotated ? (int64_t)c.seqlen_q * c.heads : 0)) * (c.head_dim / 8);
    const dim3 vgrid((unsigned)((items + 255) / 256), c.batch);
    if (a.dtype == FA_DTYPE_BF16)
      kvcache_prep_vec_kernel<__nv_bfloat16><<<vgrid, 256, 0, st>>>(c, q_follows_rows);
    else
      kvcache_prep_vec_kernel<__half><<<vgrid, 256, 0, st>>>(c, q_follows_rows);
    return fa_host::check_launch("kvcache_prep_vec_kernel");
  }
  dim3 grid(rows, a.heads > a.heads_k ? a.heads : a.heads_k, a.batch);
  if (a.dtype == FA_DTYPE_BF16)
    kvcache_prep_kernel<__nv_bfloat16><<<grid, 128, 0, st>>>(c, q_follows_rows);
  else
    kvcache_prep_kernel<__half><<<grid, 128, 0, st>>>(c, q_follows_rows);
  return fa_host::check_launch("kvcache_prep_kernel");
}

}  // namespace fa
