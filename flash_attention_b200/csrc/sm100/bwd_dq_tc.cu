// Backward attention on tcgen05 tensor cores (head dim <= 128), part 2 of 2: dQ.
//
// One CTA owns 128 query rows of one (batch, query head), keeps Q and dO in shared memory and dQ in
// tensor memory, and walks every block of 64 (or 128) keys those rows can see (bwd_tc.cu holds part 1, dK / dV,
// and says why the pass is split).  Same math as the dQ half of compute_dq_dk_dv_1colblock
// (csrc/flash_attn/src/flash_bwd_kernel.h:425-1112):
//   S   = Q K^T           (lanes = queries, columns = keys)             SS MMA  -> TMEM tS
//   dP  = dO V^T                                                         SS MMA  -> TMEM tdP
//   P   = exp2(S*scale*log2e - LSE*log2e)             one thread per query row, stays in registers
//   dS  = P o (dP - D)                                                   -> TMEM (16-bit)
//   dQ += dS K            A = dS from TMEM, B = K tile (MN-major)        -> TMEM tdQ
// It also computes D = rowsum(dO o O) of its rows, for itself and for bwd_tc.cu.
//
// What bounds it: the chain S -> P, dP -> dS -> dQ through the barriers (one CTA alone keeps the tensor pipe half busy), and
// per CTA what comes before the first and after the last block.  Hence blocks of 64 keys, 256 tensor-memory columns
// and at most 113 KiB: two CTAs share an SM, and one's waits, start and end run under the other's blocks.  An N = 64 SS MMA
// takes 48 cycles against 32 of math (it reads its A slice for half the columns); on long sequences that eats what
// the second CTA gives.  16 x 2048 tokens, with D: 16 heads of 128 causal 455 + 47 -> 440 us, 32 heads of 64 full
// 1186 + 47 -> 906 us (two buffers of dS of its own, so that dP(j+1) need not wait for dQ(j): 948); 32768 tokens causal unchanged.
// Where the grid leaves every CTA an SM of its own, nothing runs under its waits: blocks of 128 keys halve them (bwd_dq_tc_main).
// Registers: 80 a thread in the 64-key form, with 4 to 28 bytes spilled, none in the 128-key one.
//
// Warps: 0-7 compute (warpgroup w handles the half w of a block's key columns; in the epilogue,
// head-dim columns [D/2*w, ...)), 8 = TMA producer, 9 = MMA issuer, 10 = TMEM owner, 11 = issuer of dQ.
#include <cstdlib>

#include "../fa_common.cuh"
#include "ptx.cuh"
#include "tma_host.cuh"

namespace fa {

using namespace ptx;

StatusRef status_ref(bool may_allocate);

namespace {

constexpr int kM = 128;                  // query rows per CTA
constexpr int kChunkM = kM * 128;        // [128 rows][64 x 16-bit]
constexpr int kCompute = 8;              // compute warps
constexpr int kThreads = 32 * kCompute + 128;
constexpr int kWarpProducer = kCompute, kWarpMma = kCompute + 1, kWarpTmem = kCompute + 2, kWarpMmaDq = kCompute + 3;

enum DqWait { W_Q_ALIGN = 40, W_Q_QDO = 41, W_Q_KV_FULL = 42, W_Q_KV_EMPTY = 43, W_Q_S = 44, W_Q_DP = 45, W_Q_DS = 46,
              W_Q_DONE = 47 };

// KN: keys per block
template <int DH, int KN>
struct QCfg {
  static constexpr int CTAS = KN > 64 ? 1 : 2;  // per SM
  static constexpr int NCHUNK = DH / 64;
  static constexpr int CHUNK_N = KN * 128;  // [KN rows][64 x 16-bit]
  static constexpr int TILE_M = NCHUNK * kChunkM, TILE_N = NCHUNK * CHUNK_N;  // Q / dO tile, K / V tile
  // K(j) is needed from S(j) (issued a block early) to dQ(j), V(j) only by dP(j): K gets the deeper ring
  static constexpr int NSK = DH > 64 ? 2 : 4;
  static constexpr int NSV = DH > 64 ? (KN > 64 ? 2 : 1) : 3;
  static constexpr int OFF_Q = 0;
  static constexpr int OFF_DO = TILE_M;
  static constexpr int OFF_K = 2 * TILE_M;
  static constexpr int OFF_V = OFF_K + NSK * TILE_N;
  static constexpr int OFF_BAR = OFF_V + NSV * TILE_N;
  static constexpr int NBAR = 2 * NSK + 2 * NSV + 8;
  static constexpr int OFF_D = OFF_BAR + NBAR * 8 + 32;  // D of the 128 rows, fp32
  static constexpr int SMEM_BYTES = OFF_D + kM * 4;
  static constexpr int COL_S = 0, COL_DP = KN, COL_DQ = 2 * KN;  // dS (16-bit) goes over dP
  static constexpr int TMEM_COLS = KN > 64 ? 512 : 256;
  static_assert(CTAS * (SMEM_BYTES + 1024) <= 228 * 1024 && COL_DQ + DH <= TMEM_COLS, "what the CTAs of an SM share");
};

struct DqTcParams {
  CUtensorMap tq, tk, tv, tdo;
  FaBwdArgs a;
  StatusRef status;
  CtaOrder order;
  FastDiv group;  // query heads per KV head
};

template <typename T>
struct QFmt;
template <>
struct QFmt<__half> {
  static constexpr int kIdesc = 0;
};
template <>
struct QFmt<__nv_bfloat16> {
  static constexpr int kIdesc = 1;
};


// UNEVEN: CTAs in the order of cta_item.  (An instance of its own: with the block and head worked out instead of read from
// blockIdx the even case took 4 % longer at head dim 64.)
template <typename T, int DH, int KN, bool UNEVEN, bool TRIM>
__global__ void __launch_bounds__(kThreads, QCfg<DH, KN>::CTAS) bwd_dq_tc_kernel(const __grid_constant__ DqTcParams P) {
  using C = QCfg<DH, KN>;
  constexpr int NSK = C::NSK, NSV = C::NSV;
  const FaBwdArgs& a = P.a;
  extern __shared__ __align__(1024) unsigned char smem[];
  const uint32_t s_base = smem_addr(smem);
  const uint32_t sQ = s_base + C::OFF_Q, sDO = s_base + C::OFF_DO;
  auto sK = [&](int st) { return s_base + C::OFF_K + st * C::TILE_N; };
  auto sV = [&](int st) { return s_base + C::OFF_V + st * C::TILE_N; };
  const uint32_t bar0 = s_base + C::OFF_BAR;
  auto bar_k_full = [&](int st) { return bar0 + 8 * st; };
  auto bar_k_empty = [&](int st) { return bar0 + 8 * (NSK + st); };
  auto bar_v_full = [&](int st) { return bar0 + 8 * (2 * NSK + st); };
  auto bar_v_empty = [&](int st) { return bar0 + 8 * (2 * NSK + NSV + st); };
  constexpr int kB0 = 2 * NSK + 2 * NSV;
  const uint32_t bar_s = bar0 + 8 * kB0, bar_sread = bar0 + 8 * (kB0 + 1), bar_q = bar0 + 8 * (kB0 + 2), bar_do = bar0 + 8 * (kB0 + 6),
                 bar_dp = bar0 + 8 * (kB0 + 3), bar_ds = bar0 + 8 * (kB0 + 4), bar_done = bar0 + 8 * (kB0 + 5);
  volatile uint32_t* tmem_ptr_smem = reinterpret_cast<volatile uint32_t*>(smem + C::OFF_BAR + C::NBAR * 8);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + C::OFF_BAR + C::NBAR * 8 + 4);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 32) {  // the TMA unit fetches the descriptors while the CTA sets itself up
    prefetch_tensormap(&P.tq);
    prefetch_tensormap(&P.tk);
    prefetch_tensormap(&P.tdo);
    prefetch_tensormap(&P.tv);
  }
  const CtaItem item = UNEVEN ? cta_item(P.order) : CtaItem{(int)blockIdx.x, (int)blockIdx.y, (int)blockIdx.z};
  const int hq = item.head, b = item.batch;
  const int hk = (int)P.group.div(hq);
  const SeqInfo si = seq_info(a.cu_seqlens_q, a.cu_seqlens_k, nullptr, nullptr, a.seqlen_q, a.seqlen_k,
                              a.use_mask_shift, a.mask_shift, b);
  // heavy query blocks (bottom rows of a causal mask see the most keys) are scheduled first
  const int mblk = (int)gridDim.x - 1 - item.block;
  const int m0 = mblk * kM;
  float* d_out = a.softmax_d + ((int64_t)b * a.heads + hq) * a.d_seqlen + m0;
  if (m0 >= si.sq) {  // a shorter sequence of a packed batch: only its padding rows of D
    if (threadIdx.x < kM && m0 + (int)threadIdx.x < a.d_seqlen) d_out[threadIdx.x] = 0.f;
    return;
  }
  int n_lo, n_hi;
  key_block_range(m0, kM, KN, si.sk, si.shift, a.window_left, a.window_right, n_lo, n_hi);
  const int iters = n_hi - n_lo;

  if (threadIdx.x == 64) {  // reads global memory: not in front of the first loads
    abort_init(abort_flag, P.status);
    if (s_base & 1023u) abort_raise(abort_flag, W_Q_ALIGN);  // the swizzled tiles need a 1024-byte aligned base
  }
  if (threadIdx.x == 0) {
    for (int s = 0; s < NSK; ++s) {
      mbar_init(bar_k_full(s), 1);
      mbar_init(bar_k_empty(s), 1);
    }
    for (int s = 0; s < NSV; ++s) {
      mbar_init(bar_v_full(s), 1);
      mbar_init(bar_v_empty(s), 1);
    }
    mbar_init(bar_s, 1);
    mbar_init(bar_sread, kCompute);
    mbar_init(bar_q, 1);
    mbar_init(bar_do, 1);
    mbar_init(bar_dp, 1);
    mbar_init(bar_ds, kCompute);
    mbar_init(bar_done, 1);
    fence_barrier_init();
    fence_proxy_async();
    if (iters > 0) {
      // This thread has made the barriers, so it can start the first block's loads while the CTA still sets itself up:
      // Q and K first, which S(0) needs
      auto load = [&](uint32_t dst, const CUtensorMap* tm, uint32_t bar, int chunk, int64_t row, int head, int64_t batch) {
        mbar_expect_tx(bar, C::NCHUNK * chunk);
        for (int c = 0; c < C::NCHUNK; ++c) tma_load_4d(dst + c * chunk, tm, bar, c * 64, (int)row, head, (int)batch);
      };
      load(sQ, &P.tq, bar_q, kChunkM, si.q_row0 + m0, hq, si.q_batch);
      load(sK(0), &P.tk, bar_k_full(0), C::CHUNK_N, si.k_row0 + n_lo * KN, hk, si.k_batch);
      load(sDO, &P.tdo, bar_do, kChunkM, si.q_row0 + m0, hq, si.q_batch);
      load(sV(0), &P.tv, bar_v_full(0), C::CHUNK_N, si.k_row0 + n_lo * KN, hk, si.k_batch);
    }
  }
  if (warp == kWarpTmem) {
    tmem_alloc(smem_addr(const_cast<uint32_t*>(tmem_ptr_smem)), C::TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_ptr_smem;
  const bool run = (*abort_flag == 0) && iters > 0;
  const float scale_log2 = a.softmax_scale * kLog2e;

  if (warp < kCompute) {
    // ---------------------------------------------------------------- compute warpgroups
    constexpr int KW = KN / 2;                  // key columns of a warpgroup
    const int w = warp >> 2;                    // key-column half / head-dim half
    const int r = (warp & 3) * 32 + lane;       // query row of this thread within the CTA tile
    const int qrow = m0 + r;
    const uint32_t lane_off = (uint32_t)((warp & 3) * 32) << 16;
    const uint32_t tdP = tmem + lane_off + C::COL_DP + w * KW;
    bool ok = (*abort_flag == 0);  // with iters == 0 the loop is skipped and the epilogue writes zeros
    // D = rowsum(dO o O) of the CTA's rows, while the first tiles and S(0) are on their way: DH / 8 threads share a row.
    // bwd_tc.cu, launched after this kernel, reads D.  (A launch of its own took 47 us next to 1050 us of both kernels on
    // 16 x 2048 x 16 x 128, and read dO once more.)
    float* sD = reinterpret_cast<float*>(smem + C::OFF_D);
    {
      constexpr int TPR = DH / 8, RPP = 32 * kCompute / TPR;  // threads per row, rows per pass
      const int piece = threadIdx.x % TPR, row0 = threadIdx.x / TPR;
      const T* og = reinterpret_cast<const T*>(a.out.ptr) + si.q_batch * a.out.stride_b + (si.q_row0 + m0) * a.out.stride_s +
                    (int64_t)hq * a.out.stride_h + piece * 8;
      const T* dg = reinterpret_cast<const T*>(a.dout.ptr) + si.q_batch * a.dout.stride_b + (si.q_row0 + m0) * a.dout.stride_s +
                    (int64_t)hq * a.dout.stride_h + piece * 8;
      const int rows = min(kM, si.sq - m0);
#pragma unroll 1
      for (int base = 0; base < kM; base += 4 * RPP) {
        uint4 o4[4], d4[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int row = base + u * RPP + row0;
          o4[u] = d4[u] = make_uint4(0u, 0u, 0u, 0u);
          if (row < rows && piece * 8 < a.head_dim) {
            o4[u] = *reinterpret_cast<const uint4*>(og + row * a.out.stride_s);
            d4[u] = *reinterpret_cast<const uint4*>(dg + row * a.dout.stride_s);
          }
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const uint32_t ow[4] = {o4[u].x, o4[u].y, o4[u].z, o4[u].w}, dw[4] = {d4[u].x, d4[u].y, d4[u].z, d4[u].w};
          float acc = 0.f;
#pragma unroll
          for (int e = 0; e < 4; ++e) acc += Pack<T>::lo(ow[e]) * Pack<T>::lo(dw[e]) + Pack<T>::hi(ow[e]) * Pack<T>::hi(dw[e]);
#pragma unroll
          for (int x = TPR / 2; x > 0; x >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, x);
          const int row = base + u * RPP + row0;
          if (piece == 0) {
            sD[row] = acc;
            if (m0 + row < a.d_seqlen) d_out[row] = acc;
          }
        }
      }
    }
    named_bar_sync(1, 32 * kCompute);
    // per-row statistics; +inf LSE (rows past the end or without keys) gives P = 0
    const float dsum = sD[r];
    const float lse2 = qrow < si.sq ? a.softmax_lse[((int64_t)b * a.heads + hq) * a.lse_seqlen + qrow] * kLog2e : INFINITY;
    // keys this row can see: [k_lo, k_hi]
    int k_lo = 0, k_hi = si.sk - 1;
    if (a.window_right >= 0) k_hi = min(k_hi, qrow + si.shift + a.window_right);
    if (a.window_left >= 0) k_lo = max(k_lo, qrow + si.shift - a.window_left);
    const uint64_t scale2 = pack2(scale_log2, scale_log2), neg_lse2 = pack2(-lse2, -lse2), neg_d2 = pack2(-dsum, -dsum);
    for (int j = 0; j < iters && ok; ++j) {
      const int n0 = (n_lo + j) * KN;
      const uint32_t tS = tmem + lane_off + C::COL_S + w * KW;
      const bool need_mask = (n0 + KN > si.sk) ||
                             (a.window_right >= 0 && n0 + KN - 1 > m0 + si.shift + a.window_right) ||
                             (a.window_left >= 0 && n0 < m0 + kM - 1 + si.shift - a.window_left);
      // ---- P = exp2(S * scale - LSE), KW key columns per thread, kept in registers
      ok = mbar_wait(bar_s, j & 1, W_Q_S, abort_flag);
      if (!ok) break;
      tc_fence_after();
      float p[KW];
      {
        uint32_t s[KW / 32][32];
#pragma unroll
        for (int h = 0; h < KW / 32; ++h) tmem_ld32(tS + h * 32, s[h]);
        tmem_wait_ld();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(bar_sread);  // S(j) is in registers: S(j+1) may overwrite it
#pragma unroll
        for (int c = 0; c < KW; c += 2) {
          float x0, x1;
          unpack2(fma2(pack2u(s[c / 32][c % 32], s[c / 32][c % 32 + 1]), scale2, neg_lse2), x0, x1);
          p[c] = ex2(x0);
          p[c + 1] = ex2(x1);
        }
      }
      if (need_mask) {
        const int c_lo = k_lo - n0 - w * KW, c_hi = k_hi - n0 - w * KW;
#pragma unroll
        for (int c = 0; c < KW; ++c) p[c] = (c >= c_lo && c <= c_hi) ? p[c] : 0.f;
      }
      // ---- dS = P o (dP - D), 16-bit, over this warp's own, now read, columns of dP
      ok = mbar_wait(bar_dp, j & 1, W_Q_DP, abort_flag);
      if (!ok) break;
      tc_fence_after();
      {
        uint32_t d[KW / 32][32], pk[KW / 2];
#pragma unroll
        for (int h = 0; h < KW / 32; ++h) tmem_ld32(tdP + h * 32, d[h]);
        tmem_wait_ld();
#pragma unroll
        for (int c = 0; c < KW; c += 2) {
          float x0, x1;
          unpack2(mul2(pack2(p[c], p[c + 1]), add2(pack2u(d[c / 32][c % 32], d[c / 32][c % 32 + 1]), neg_d2)), x0, x1);
          pk[c >> 1] = Pack<T>::two(x0, x1);
        }
        if constexpr (KW == 64)
          tmem_st32(tdP, pk);
        else
          tmem_st16(tdP, pk);
      }
      tmem_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar_ds);
    }
    // ---- epilogue: dQ * softmax_scale
    if (ok && iters > 0) ok = mbar_wait(bar_done, 0, W_Q_DONE, abort_flag);
    tc_fence_after();
    ok = __all_sync(0xffffffffu, ok && *abort_flag == 0);  // the TMEM loads below are warp-wide instructions
    if (ok) {
      const uint32_t tdQ = tmem + lane_off + C::COL_DQ + w * (DH / 2);
      const float sc = a.softmax_scale;
#pragma unroll
      for (int c0 = 0; c0 < DH / 2; c0 += 32) {
        uint32_t o[32];
        if (iters > 0) {
          tmem_ld32(tdQ + c0, o);
          tmem_wait_ld();
        } else {
#pragma unroll
          for (int i = 0; i < 32; ++i) o[i] = 0u;
        }
        // 16-bit rows over the Q tile (every MMA is done), 16-byte pieces swizzled
#pragma unroll
        for (int i = 0; i < 32; i += 8) {
          uint4 v;
          v.x = Pack<T>::two(__uint_as_float(o[i]) * sc, __uint_as_float(o[i + 1]) * sc);
          v.y = Pack<T>::two(__uint_as_float(o[i + 2]) * sc, __uint_as_float(o[i + 3]) * sc);
          v.z = Pack<T>::two(__uint_as_float(o[i + 4]) * sc, __uint_as_float(o[i + 5]) * sc);
          v.w = Pack<T>::two(__uint_as_float(o[i + 6]) * sc, __uint_as_float(o[i + 7]) * sc);
          *reinterpret_cast<uint4*>(smem + C::OFF_Q + r * (DH * 2) + ((((w * (DH / 2) + c0 + i) / 8) ^ (r & 7)) << 4)) = v;
        }
      }
    }
    named_bar_sync(1, 32 * kCompute);
    if (ok) {  // whole rows by neighbouring threads
      constexpr int CPR = DH / 8;  // 16-byte pieces per row
      T* g = reinterpret_cast<T*>(a.dq.ptr) + si.q_batch * a.dq.stride_b + (si.q_row0 + m0) * a.dq.stride_s + (int64_t)hq * a.dq.stride_h;
      const int rows = min(kM, si.sq - m0), col = (int)threadIdx.x % CPR;
      if (col * 8 < a.head_dim)
        for (int row = threadIdx.x / CPR; row < rows; row += 32 * kCompute / CPR)
          *reinterpret_cast<uint4*>(g + row * a.dq.stride_s + col * 8) =
              *reinterpret_cast<const uint4*>(smem + C::OFF_Q + row * (DH * 2) + ((col ^ (row & 7)) << 4));
    }
  } else {
    if (warp == kWarpProducer) {
      // -------------------------------------------------------------- TMA producer
      if (lane == 0 && run) {
        const int kb = (int)si.k_batch;
        bool ok = true;
        for (int j = 1; j < iters && ok; ++j) {  // block 0 is on its way
          const int ks = j % NSK, vs = j % NSV;
          const int row = (int)si.k_row0 + (n_lo + j) * KN;
          ok = mbar_wait(bar_k_empty(ks), ((j / NSK) & 1) ^ 1, W_Q_KV_EMPTY, abort_flag);
          if (!ok) break;
          mbar_expect_tx(bar_k_full(ks), C::TILE_N);
          for (int c = 0; c < C::NCHUNK; ++c) tma_load_4d(sK(ks) + c * C::CHUNK_N, &P.tk, bar_k_full(ks), c * 64, row, hk, kb);
          ok = mbar_wait(bar_v_empty(vs), ((j / NSV) & 1) ^ 1, W_Q_KV_EMPTY, abort_flag);
          if (!ok) break;
          mbar_expect_tx(bar_v_full(vs), C::TILE_N);
          for (int c = 0; c < C::NCHUNK; ++c) tma_load_4d(sV(vs) + c * C::CHUNK_N, &P.tv, bar_v_full(vs), c * 64, row, hk, kb);
        }
      }
    } else if (warp == kWarpMma || warp == kWarpMmaDq) {
      // -------------------------------------------------------------- MMA issuer
      // Warp 9 issues S(j+1) as soon as the compute warps hold S(j) in registers; warp 11 issues the chain
      // dQ(j) | dP(j+1): dS(j) sits over dP(j), and the MMAs of one thread execute in order.  MMAs of the two threads are
      // not ordered among themselves and need not be.
      if (run) with_head_steps<DH, TRIM>(a.head_dim, [&](auto steps) {  // the whole warp runs the loops (see mma_ss_w); one elected lane issues
        constexpr int F = QFmt<T>::kIdesc;
        constexpr uint32_t idesc_s = make_idesc(kM, KN, F, 0, 0);   // S, dP: K-major x K-major, N = KN keys
        constexpr int KS = decltype(steps)::value;
        constexpr uint32_t idesc_dq = make_idesc(kM, KS * 16, F, 0, 1);  // dQ: A in TMEM, B MN-major, N = head dim
        // One descriptor is built (Q tile, K-major); every other operand differs from it only in the
        // low word: the address field (+ byte offset >> 4) and, for MN-major reads, the LBO field.
        const uint64_t d_base = smem_desc_sw128(sQ, 16, 1024);
        const uint32_t d_lo = (uint32_t)d_base, d_hi = (uint32_t)(d_base >> 32);
        auto dsc = [&](uint32_t lo_add) { return ((uint64_t)d_hi << 32) | (uint64_t)(d_lo + lo_add); };
        constexpr uint32_t kMn = (uint32_t)((C::CHUNK_N - 16) >> 4) << 16;  // K-major -> MN-major (LBO = chunk stride)
        constexpr uint32_t oQ = 0, oDO = C::TILE_M >> 4, oK = (C::OFF_K - C::OFF_Q) >> 4, oV = (C::OFF_V - C::OFF_Q) >> 4,
                           kTile16 = C::TILE_N >> 4;
        auto koff_m = [](int kk) { return (uint32_t)(((kk >> 2) * kChunkM + (kk & 3) * 32) >> 4); };  // K-major k-step
        auto koff_n = [](int kk) { return (uint32_t)(((kk >> 2) * C::CHUNK_N + (kk & 3) * 32) >> 4); };
        auto moff = [](int kk) { return (uint32_t)((kk * 2048) >> 4) + kMn; };                        // MN-major k-step
        auto issue_s = [&](uint32_t d_col, uint32_t a_lo, uint32_t b_lo, uint32_t bar) {
#pragma unroll
          for (int kk = 0; kk < KS; ++kk)
            mma_ss_w(tmem + d_col, dsc(a_lo + koff_m(kk)), dsc(b_lo + koff_n(kk)), idesc_s, kk > 0);
          tc_commit_w(bar);
        };
        if (warp == kWarpMma) {
          bool ok = mbar_wait_w(bar_q, 0, W_Q_QDO, abort_flag);
          for (int j = 0; j < iters && ok; ++j) {
            const int ks = j % NSK;
            if (j > 0) ok = mbar_wait_w(bar_sread, (j - 1) & 1, W_Q_S, abort_flag);
            if (ok) ok = mbar_wait_w(bar_k_full(ks), (j / NSK) & 1, W_Q_KV_FULL, abort_flag);
            if (!ok) break;
            tc_fence_after();
            issue_s(C::COL_S, oQ, oK + ks * kTile16, bar_s);
          }
        } else {
          auto issue_dp = [&](int i) {
            const int vs = i % NSV;
            const bool k = mbar_wait_w(bar_v_full(vs), (i / NSV) & 1, W_Q_KV_FULL, abort_flag);
            if (k) {
              tc_fence_after();
              issue_s(C::COL_DP, oDO, oV + vs * kTile16, bar_dp);
              tc_commit_w(bar_v_empty(vs));
            }
            return k;
          };
          bool ok = mbar_wait_w(bar_do, 0, W_Q_QDO, abort_flag);
          if (ok) ok = issue_dp(0);
          for (int j = 0; j < iters && ok; ++j) {
            const int ks = j % NSK;
            // dS(j) is in TMEM: dQ += dS K.  Its commit releases the K tile, which S(j) of the other issuer read as well:
            // dS(j) was computed from S(j).
            ok = mbar_wait_w(bar_ds, j & 1, W_Q_DS, abort_flag);
            if (!ok) break;
            tc_fence_after();
#pragma unroll
            for (int kk = 0; kk < KN / 16; ++kk)  // (a warpgroup's dS sits over the first half of its columns of dP)
              mma_ts_w(tmem + C::COL_DQ, tmem + C::COL_DP + kk / (KN / 32) * (KN / 2) + kk % (KN / 32) * 8, dsc(oK + ks * kTile16 + moff(kk)),
                       idesc_dq, (j > 0) || kk > 0);
            tc_commit_w(bar_k_empty(ks));
            if (j + 1 < iters) ok = issue_dp(j + 1);
          }
          if (ok) tc_commit_w(bar_done);
        }
      });
    }
  }

  // ---- teardown
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (*abort_flag) {
    const long long t0 = clock64();
    while (clock64() - t0 < 2000000) {
    }
    __syncthreads();
  }
  if (warp == kWarpTmem) tmem_dealloc(tmem, C::TMEM_COLS);
}


template <typename T, int DH, int KN>
int launch_bwd_dq_tc(const FaBwdArgs& a, cudaStream_t st) {
  using C = QCfg<DH, KN>;
  DqTcParams P;
  P.a = a;
  const bool varlen = a.cu_seqlens_q != nullptr;
  const int64_t q_rows = varlen ? a.total_q : a.seqlen_q, k_rows = varlen ? a.total_k : a.seqlen_k;
  const int64_t nb = varlen ? 1 : a.batch;
  if (make_tmap_4d(&P.tq, a.q, a.dtype, q_rows, a.heads, nb, a.head_dim, kM)) return 1;
  if (make_tmap_4d(&P.tdo, a.dout, a.dtype, q_rows, a.heads, nb, a.head_dim, kM)) return 1;
  if (make_tmap_4d(&P.tk, a.k, a.dtype, k_rows, a.heads_k, nb, a.head_dim, KN)) return 1;
  if (make_tmap_4d(&P.tv, a.v, a.dtype, k_rows, a.heads_k, nb, a.head_dim, KN)) return 1;
  // (CTAs that all start at once need no order)
  const bool uneven = KN <= 64 && (a.window_left >= 0 || a.window_right >= 0 || a.cu_seqlens_q);
  const bool trim = head_trims<DH>(a.head_dim);
  auto kern = trim ? (uneven ? bwd_dq_tc_kernel<T, DH, KN, (KN <= 64), true> : bwd_dq_tc_kernel<T, DH, KN, false, true>)
                   : (uneven ? bwd_dq_tc_kernel<T, DH, KN, (KN <= 64), false> : bwd_dq_tc_kernel<T, DH, KN, false, false>);
  P.status = status_ref(true);
  static fa_host::DeviceOnce once[2][2];
  if (int rc = fa_host::raise_smem_limit(once[trim][uneven], reinterpret_cast<const void*>(kern), C::SMEM_BYTES, "bwd_dq_tc_kernel")) return rc;
  const int rows = a.d_seqlen > a.seqlen_q ? a.d_seqlen : a.seqlen_q;  // the padding rows of D are written too
  dim3 grid((rows + kM - 1) / kM, a.heads, a.batch);
  P.group = fast_div(a.heads / a.heads_k);
  const int head_group = fa_host::cta_head_group(uneven, (int64_t)a.seqlen_k * a.head_dim * 4 / (a.heads / a.heads_k),
                                         (int64_t)a.heads * a.batch);
  P.order = cta_order(head_group, grid);
  kern<<<grid, kThreads, C::SMEM_BYTES, st>>>(P);
  return fa_host::check_launch("bwd_dq_tc_kernel");
}

}  // namespace

template <int KN>
static int dq_dispatch(const FaBwdArgs& a, cudaStream_t st) {
  const bool bf = a.dtype == FA_DTYPE_BF16;
  if (a.head_dim <= 64) return bf ? launch_bwd_dq_tc<__nv_bfloat16, 64, KN>(a, st) : launch_bwd_dq_tc<__half, 64, KN>(a, st);
  return bf ? launch_bwd_dq_tc<__nv_bfloat16, 128, KN>(a, st) : launch_bwd_dq_tc<__half, 128, KN>(a, st);
}

int bwd_dq_tc_main(const FaBwdArgs& a, cudaStream_t st) {
  // 128-key blocks where no two CTAs share an SM: 1 x 1024 tokens, 16 heads of 128 (128 CTAs) 21.5 us with 64 keys, 17.3 with
  // 128; 1 x 2048, 8/2 heads of 128 35.4 and 27.7; 1 x 16384, 1 head of 64 (128 CTAs) 164 and 137.  From 149 CTAs on two share:
  // 8 x 256, 10 heads of 128 (160 CTAs) 13.6 and 16.1; 1 x 2048, 16 heads of 64 (256 CTAs) 39.9 and 42.1.
  const int64_t ctas = (int64_t)((a.seqlen_q + kM - 1) / kM) * a.heads * a.batch;
  return ctas <= fa_host::sm_count() ? dq_dispatch<128>(a, st) : dq_dispatch<64>(a, st);
}

}  // namespace fa
