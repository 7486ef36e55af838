// Merge of partial attention results by log-sum-exp.  Same math as combine_attn_seqk_parallel
// (csrc/flash_attn/src/flash_fwd_kernel.h:1169-1327): LSE = logsumexp_s(LSE_s),
// O = sum_s exp(LSE_s - LSE) * O_s; a row whose parts are all empty (-inf) gets O = 0, LSE = +inf, a row with a part whose
// LSE is NaN (a NaN score) gets what one pass gives: O = NaN, LSE = +inf.
#include "fa_common.cuh"

namespace fa {

struct CombineParams {
  const float* out_parts;  // (n_parts, rows, D)
  const float* lse_parts;  // (n_parts, rows)
  void* out;
  float* lse;  // may be NULL
  int64_t out_sb, out_ss, out_sh;
  int32_t n_parts, B, H, S, D, lse_pitch;
  FastDiv by_s, by_h;  // rows of a head, heads
};

// G: groups of 32 parts, one part per lane.  One group is an instance of its own, without the choice among groups and with two
// steps of the walk in flight, four with more groups (before PRE: 16384 rows of 128 in 5 parts 10.9 us, 11.6 with four groups for
// all; 2048 rows in 64 parts 12.6 us, 16.6 with two steps in flight).
// PRE: the rows of the first four parts are on their way before it is known which of them have keys (32 rows in 18 parts: 4.0 -> 3.0
// us, 1024 in 8: 3.0 -> 2.5, 16384 in 5: 10.2 -> 9.9; with fewer parts and many rows the registers cost more than the wait: 16384 in
// 2 parts 7.0 without, 7.7 with).
template <typename T, int G, bool PRE>
__global__ void __launch_bounds__(128) combine_kernel(const CombineParams p) {
  const int lane = threadIdx.x & 31;
  const int64_t rows = (int64_t)p.B * p.H * p.S;
  const int64_t row = (int64_t)blockIdx.x * 4 + (threadIdx.x >> 5);
  if (row >= rows) return;
  auto load = [&](int s, float4(&x)[2]) {
    const float* src = p.out_parts + ((int64_t)s * rows + row) * p.D;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int c = lane * 4 + i * 128;
      x[i] = s < p.n_parts && c < p.D ? *reinterpret_cast<const float4*>(src + c) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
  };
  float4 pre[4][2];  // (an empty part's row, which nobody may have written, is dropped below)
  if constexpr (PRE)
#pragma unroll
    for (int k = 0; k < 4; ++k) load(k, pre[k]);
  float l[G];
  uint32_t live[G];  // parts with keys (+inf is not an LSE of theirs)
  float mx = -INFINITY;
#pragma unroll
  for (int i = 0; i < G; ++i) {
    int s = lane + 32 * i;
    l[i] = s < p.n_parts ? p.lse_parts[(int64_t)s * rows + row] : -INFINITY;
    live[i] = __ballot_sync(0xffffffffu, l[i] != -INFINITY && l[i] != INFINITY);
    mx = fmaxf(mx, l[i]);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  float sum = 0.f;
  const float msafe = mx == -INFINITY ? 0.f : mx;
#pragma unroll
  for (int i = 0; i < G; ++i) sum += __expf(l[i] - msafe);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
  // (fmaxf drops a NaN, the sum does not; an LSE of +inf makes it NaN as well)
  const bool nan = sum != sum && mx != INFINITY;
  const bool empty = !nan && (!(sum > 0.f) || mx == -INFINITY);
  const float lse = empty || nan ? INFINITY : logf(sum) + mx;
  // (two 64-bit divisions per row were a third of its instructions; combine() checks that a row's number has 32 bits)
  const uint32_t bh = p.by_s.div((uint32_t)row), b = p.by_h.div(bh);
  const int s_idx = (int)((uint32_t)row - bh * p.S), h = (int)(bh - b * p.H);
  if (lane == 0 && p.lse) p.lse[(int64_t)bh * p.lse_pitch + s_idx] = lse;
  T* o = reinterpret_cast<T*>(p.out) + b * p.out_sb + s_idx * p.out_ss + h * p.out_sh;
  // head_dim <= 256: at most two 4-column groups per lane
  float4 acc[2] = {make_float4(0.f, 0.f, 0.f, 0.f), make_float4(0.f, 0.f, 0.f, 0.f)};
  float wgt[G];
#pragma unroll
  for (int i = 0; i < G; ++i) wgt[i] = nan ? sum : empty ? 0.f : __expf(l[i] - lse);
  // Bound by the latency of the loads: four parts are in flight at a time (16 parts of 2048 x 128: 9.4 us, 11.5 us with one
  // at a time).  Empty parts, those past the last one among them, are not read, or dropped where PRE has read them: nobody
  // may have written them.  The walk ends behind the last part with keys (2048 rows of 128, 64 parts, 4 of them with keys: 8.9 -> 3.5 us; a test of every four parts
  // in the loop instead: 4.6, and 16.2 where all have keys).
  constexpr int kSteps = G == 1 ? 2 : 4;
  int end = 0;
#pragma unroll
  for (int i = 0; i < G; ++i)
    if (live[i]) end = 32 * (i + 1) - __clz(live[i]);
#pragma unroll kSteps
  for (int s0 = 0; s0 < end; s0 += 4) {  // uniform trip count: every lane takes part in the shuffles
    float wsel = wgt[0];
    uint32_t lsel = live[0];
    if constexpr (G > 1) {
      wsel = (s0 >> 5) == 0 ? wgt[0] : (s0 >> 5) == 1 ? wgt[1] : (s0 >> 5) == 2 ? wgt[2] : wgt[3];
      lsel = (s0 >> 5) == 0 ? live[0] : (s0 >> 5) == 1 ? live[1] : (s0 >> 5) == 2 ? live[2] : live[3];
    }
    lsel >>= s0 & 31;
    float w[4];
    float4 x[4][2];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      w[k] = __shfl_sync(0xffffffffu, wsel, (s0 + k) & 31);
      const bool on = lsel >> k & 1;
      if (PRE && s0 == 0) {
#pragma unroll
        for (int i = 0; i < 2; ++i) x[k][i] = on ? pre[k][i] : make_float4(0.f, 0.f, 0.f, 0.f);
      } else if (PRE || G > 1) {  // (a branch is the faster form here, a select below)
        if (on)
          load(s0 + k, x[k]);
        else
          x[k][0] = x[k][1] = make_float4(0.f, 0.f, 0.f, 0.f);
      } else {
        const float* src = p.out_parts + ((int64_t)(s0 + k) * rows + row) * p.D;
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const int c = lane * 4 + i * 128;
          x[k][i] = on && c < p.D ? *reinterpret_cast<const float4*>(src + c) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
      }
    }
#pragma unroll
    for (int k = 0; k < 4; ++k)
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        acc[i].x += w[k] * x[k][i].x;
        acc[i].y += w[k] * x[k][i].y;
        acc[i].z += w[k] * x[k][i].z;
        acc[i].w += w[k] * x[k][i].w;
      }
  }
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    int c = lane * 4 + i * 128;
    if (c < p.D) {
      uint2 pk;
      pk.x = Pack<T>::two(acc[i].x, acc[i].y);
      pk.y = Pack<T>::two(acc[i].z, acc[i].w);
      *reinterpret_cast<uint2*>(o + c) = pk;
    }
  }
}

int combine(const float* out_parts, const float* lse_parts, const FaTensor& out, float* lse, int lse_pitch, int n_parts,
            int B, int H, int S, int D, int dtype, cudaStream_t st) {
  CombineParams p{out_parts, lse_parts, out.ptr, lse, out.stride_b, out.stride_s, out.stride_h, n_parts, B, H, S, D, lse_pitch, fast_div(S), fast_div(H)};
  int64_t rows = (int64_t)B * H * S;
  FA_REQUIRE(rows < (1ll << 32), "too many rows");
  unsigned grid = (unsigned)((rows + 3) / 4);
  const bool bf = dtype == FA_DTYPE_BF16, pre = n_parts >= 4 || rows <= 4096;
  auto kern = n_parts > 32 ? (bf ? combine_kernel<__nv_bfloat16, 4, false> : combine_kernel<__half, 4, false>)
              : pre        ? (bf ? combine_kernel<__nv_bfloat16, 1, true> : combine_kernel<__half, 1, true>)
                           : (bf ? combine_kernel<__nv_bfloat16, 1, false> : combine_kernel<__half, 1, false>);
  kern<<<grid, 128, 0, st>>>(p);
  return fa_host::check_launch("combine_kernel");
}

// ---------------------------------------------------------------------------------------------
// In-place merge of one more partial result into a running fp32 accumulator (the per-step update of
// context-parallel ring attention): acc <- acc * exp(la - l) + part * exp(lb - l), la <- l, with
// l = logaddexp(la, lb).  An LSE of +inf (the kernels' "row saw no key") or -inf means empty.
struct MergeParams {
  float* acc;
  float* lse_acc;
  const void* part;
  const float* lse_part;
  int64_t acc_sb, acc_ss, acc_sh, part_sb, part_ss, part_sh;
  int64_t lacc_sb, lacc_sh, lpart_sb, lpart_sh;
  int32_t B, S, H, D;
};

template <typename T>
__global__ void __launch_bounds__(256) merge_partial_kernel(const MergeParams p) {
  const int lane = threadIdx.x & 31;
  const int64_t rows = (int64_t)p.B * p.S * p.H;
  const int64_t row = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
  if (row >= rows) return;
  const int h = (int)(row % p.H);
  const int s = (int)((row / p.H) % p.S);
  const int b = (int)(row / ((int64_t)p.H * p.S));
  float* la_p = p.lse_acc + b * p.lacc_sb + h * p.lacc_sh + s;
  float la = *la_p, lb = p.lse_part[b * p.lpart_sb + h * p.lpart_sh + s];
  if (la == INFINITY) la = -INFINITY;
  if (lb == INFINITY) lb = -INFINITY;
  const float mx = fmaxf(la, lb);
  float wa = 0.f, wb = 0.f, l = -INFINITY;
  if (mx != -INFINITY) {
    const float ea = __expf(la - mx), eb = __expf(lb - mx);
    const float inv = 1.f / (ea + eb);
    wa = ea * inv;
    wb = eb * inv;
    l = mx + __logf(ea + eb);
  }
  float* a = p.acc + b * p.acc_sb + s * p.acc_ss + h * p.acc_sh;
  const T* o = reinterpret_cast<const T*>(p.part) + b * p.part_sb + s * p.part_ss + h * p.part_sh;
  for (int c = lane * 4; c < p.D; c += 128) {
    float4 x = *reinterpret_cast<float4*>(a + c);
    const uint2 y = *reinterpret_cast<const uint2*>(o + c);
    x.x = wa * x.x + wb * Pack<T>::lo(y.x);
    x.y = wa * x.y + wb * Pack<T>::hi(y.x);
    x.z = wa * x.z + wb * Pack<T>::lo(y.y);
    x.w = wa * x.w + wb * Pack<T>::hi(y.y);
    *reinterpret_cast<float4*>(a + c) = x;
  }
  if (lane == 0) *la_p = l;
}

int merge_partial(const FaTensor& acc, float* lse_acc, int64_t lacc_sb, int64_t lacc_sh, const FaTensor& part,
                  const float* lse_part, int64_t lpart_sb, int64_t lpart_sh, int B, int S, int H, int D, int dtype,
                  cudaStream_t st) {
  MergeParams p{reinterpret_cast<float*>(acc.ptr), lse_acc, part.ptr, lse_part, acc.stride_b, acc.stride_s, acc.stride_h,
                part.stride_b, part.stride_s, part.stride_h, lacc_sb, lacc_sh, lpart_sb, lpart_sh, B, S, H, D};
  const int64_t rows = (int64_t)p.B * p.S * p.H;
  if (rows == 0) return 0;
  const unsigned grid = (unsigned)((rows + 7) / 8);
  if (dtype == FA_DTYPE_BF16)
    merge_partial_kernel<__nv_bfloat16><<<grid, 256, 0, st>>>(p);
  else
    merge_partial_kernel<__half><<<grid, 256, 0, st>>>(p);
  return fa_host::check_launch("merge_partial_kernel");
}

}  // namespace fa
