// Backward attention on tcgen05 tensor cores (head dim <= 128), part 1 of 2: dK and dV.
//
// The backward pass is split in two kernels that each keep their result stationary in tensor memory
// and recompute S and dP: this one (dK, dV; one CTA per 128 keys) and bwd_dq_tc.cu (dQ; one CTA per
// 128 queries).  The single-kernel form of the reference, compute_dq_dk_dv_1colblock
// (csrc/flash_attn/src/flash_bwd_kernel.h:425-1112), adds every block's dQ into an fp32 accumulator
// with atomics; on this GPU an SM sustains only ~26 bytes/clk of fp32 reductions into the L2 (64 KiB
// per block = ~2500 cycles, about the block's whole tensor-core time), and the saturated L2 triples
// the latency of the Q / dO tile loads.  Two more MMAs per block cost less than that, need no
// workspace, and make the gradient deterministic.
//
// One CTA owns 128 keys of one (batch, KV head) and walks every query block (128 rows; 64 mostly at head dim 64) that can see
// them, for every query head of the KV head's group (so grouped-query dK/dV need no expanded
// temporaries or group reduction, cf. flash_api.cpp:744-751, 799-803).  Everything is computed
// TRANSPOSED so that the operands the tensor cores need next are already where tcgen05 wants them:
//   S^T  = K Q^T          (lanes = keys, columns = queries)            SS MMA  -> TMEM tS
//   dP^T = V dO^T                                                       SS MMA  -> TMEM tdP
//   P^T  = exp2(S^T*scale*log2e - LSE*log2e)        one thread per key  -> TMEM (16-bit, over tdP)
//   dS^T = P^T o (dP^T - D)                                             -> TMEM (16-bit, over tdP)
//   dV  += P^T  dO        A = P^T from TMEM, B = dO tile (MN-major)     -> TMEM tdV
//   dK  += dS^T Q         A = dS^T, B = Q tile (MN-major)                -> TMEM tdK
//
// What bounds it: the chain S -> P -> dV | dP -> dS -> dK through the barriers, about 2750 cycles per 128 x 128 block at head
// dim 128 against 2048 of MMA, and per CTA what comes before the first and after the last block.
//   Head dim 128: tensor memory and shared memory are full with one CTA.  16 compute warps instead of 8 were slower (the
//   power cap on long sequences), and so was dS in shared memory (the Q ring shrinks to two slots, S(i+1) waits for Q).
//   Head dim 64: half the tile rows, 256 columns and 113 KiB, so that two CTAs share an SM and one's waits, start and end
//   run under the other's blocks; the exponentials (16 per clock and SM: 1024 cycles per 128 x 128) come next.  Where the
//   grid leaves every CTA an SM of its own, the tiles of head dim 128 (bwd_tc_main).
//   (dS in shared memory, so that dP(i+1) need not wait for dK(i), was slower: 1084 -> 1210 us below.)
//   Start and end: the first loads leave before the CTA has set itself up, and the result leaves in whole rows through
//   shared memory (a row per thread cost 7700 cycles per CTA at head dim 128, it is 4300 now).
// 16 x 2048 tokens: 16 heads of 128 causal 602 -> 535 us, 32 heads of 64 full 1509 -> 1090 us.
//
// Warps: 0-7 compute (warpgroup w handles the half w of a block's query columns; in the epilogue, of the head dim),
// 8 = TMA producer, 9 = MMA issuer, 10 = loader of the per-row LSE / D vectors and TMEM owner, 11 = issuer of S.
#include <cstdlib>

#include "../fa_common.cuh"
#include "ptx.cuh"
#include "tma_host.cuh"

namespace fa {

using namespace ptx;

StatusRef status_ref(bool may_allocate);

namespace {

constexpr int kB = 128;                 // keys per CTA
constexpr int kChunkBytes = kB * 128;   // [128 rows][64 x 16-bit]

enum BwdWait { W_B_KV = 21, W_B_QDO_FULL = 22, W_B_QDO_EMPTY = 23, W_B_STATS_FULL = 24, W_B_STATS_EMPTY = 25,
               W_B_S = 26, W_B_DP = 27, W_B_PDS = 28, W_B_ALIGN = 20 };

// BQ: query rows per block
template <int DH, int BQ>
struct BCfg {
  static constexpr int NCHUNK = DH / 64;
  static constexpr int QCHUNK = BQ * 128;
  static constexpr int TILE_K = NCHUNK * kChunkBytes, TILE_Q = NCHUNK * QCHUNK;  // K / V tile, Q / dO tile
  // 8 compute warps: each takes 32 key rows and half the query columns of a block
  static constexpr int WARPS = 8, CW = BQ / 2;
  static constexpr int THREADS = 32 * WARPS + 128;
  static constexpr int WARP_PRODUCER = WARPS, WARP_MMA = WARPS + 1, WARP_STATS = WARPS + 2, WARP_MMA_S = WARPS + 3;
  static constexpr int CTAS = BQ > 64 ? 1 : 2;  // per SM
  // a thread is launched with 168 (one CTA) or 80 registers (two): setmaxnreg only redistributes those
  static constexpr int REGS = BQ > 64 ? 200 : 88, REGS_OTHER = BQ > 64 ? 104 : 64;
  static_assert(256 * REGS + 128 * REGS_OTHER <= THREADS * (BQ > 64 ? 168 : 80), "the registers of one CTA");
  // Q(i) is needed from S^T(i) (issued a block early) to dK(i), dO(i) from dP^T(i) to dV(i): Q gets the deeper ring
  static constexpr int NSQ = DH > 64 ? 3 : 4, NSO = DH > 64 ? 2 : 4;
  static constexpr int OFF_K = 0;
  static constexpr int OFF_V = TILE_K;
  static constexpr int OFF_Q = 2 * TILE_K;
  static constexpr int OFF_DO = OFF_Q + NSQ * TILE_Q;
  static constexpr int OFF_STATS = OFF_DO + NSO * TILE_Q;  // 2 slots x (BQ -lse2, BQ -dsum) fp32
  static constexpr int OFF_BAR = OFF_STATS + 2 * 2 * BQ * 4;
  static constexpr int NBAR = 2 * NSQ + 2 * NSO + 11;
  static constexpr int SMEM_BYTES = OFF_BAR + NBAR * 8 + 32;
  static constexpr int COL_S = 0, COL_DP = BQ, COL_DV = 2 * BQ, COL_DK = 2 * BQ + DH;
  static constexpr int TMEM_COLS = BQ > 64 ? 512 : 256;
  static_assert(CTAS * (SMEM_BYTES + 1024) <= 228 * 1024 && COL_DK + DH <= TMEM_COLS, "what the CTAs of an SM share");
};

struct BwdTcParams {
  CUtensorMap tq, tk, tv, tdo;
  FaBwdArgs a;
  StatusRef status;
  CtaOrder order;
  FastDiv group;  // query heads per KV head
};

template <typename T>
struct BFmt;
template <>
struct BFmt<__half> {
  static constexpr int kIdesc = 0;
};
template <>
struct BFmt<__nv_bfloat16> {
  static constexpr int kIdesc = 1;
};


// UNEVEN: CTAs in the order of cta_item.  (An instance of its own: with the block and head worked out instead of read from
// blockIdx the even case took 4 % longer at head dim 64.)
template <typename T, int DH, int BQ, bool UNEVEN, bool TRIM>
__global__ void __launch_bounds__(BCfg<DH, BQ>::THREADS, BCfg<DH, BQ>::CTAS) bwd_tc_kernel(const __grid_constant__ BwdTcParams P) {
  using C = BCfg<DH, BQ>;
  const FaBwdArgs& a = P.a;
  extern __shared__ __align__(1024) unsigned char smem[];
  const uint32_t s_base = smem_addr(smem);
  constexpr int NSQ = C::NSQ, NSO = C::NSO, CW = C::CW;
  const uint32_t sK = s_base + C::OFF_K, sV = s_base + C::OFF_V;
  auto sQ = [&](int slot) { return s_base + C::OFF_Q + slot * C::TILE_Q; };
  auto sDO = [&](int slot) { return s_base + C::OFF_DO + slot * C::TILE_Q; };
  float* sStats = reinterpret_cast<float*>(smem + C::OFF_STATS);
  const uint32_t bar0 = s_base + C::OFF_BAR;
  const uint32_t bar_k = bar0;
  auto bar_q_full = [&](int s) { return bar0 + 8 * (1 + s); };
  auto bar_q_empty = [&](int s) { return bar0 + 8 * (1 + NSQ + s); };
  auto bar_do_full = [&](int s) { return bar0 + 8 * (1 + 2 * NSQ + s); };
  auto bar_do_empty = [&](int s) { return bar0 + 8 * (1 + 2 * NSQ + NSO + s); };
  constexpr int kB1 = 1 + 2 * NSQ + 2 * NSO;
  auto bar_st_full = [&](int s) { return bar0 + 8 * (kB1 + s); };
  auto bar_st_empty = [&](int s) { return bar0 + 8 * (kB1 + 2 + s); };
  const uint32_t bar_s = bar0 + 8 * (kB1 + 4), bar_dp = bar0 + 8 * (kB1 + 5), bar_ds = bar0 + 8 * (kB1 + 6),
                 bar_p = bar0 + 8 * (kB1 + 7), bar_sread = bar0 + 8 * (kB1 + 8), bar_v = bar0 + 8 * (kB1 + 9);
  volatile uint32_t* tmem_ptr_smem = reinterpret_cast<volatile uint32_t*>(smem + C::OFF_BAR + C::NBAR * 8);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + C::OFF_BAR + C::NBAR * 8 + 4);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 32) {  // the TMA unit fetches the descriptors while the CTA sets itself up
    prefetch_tensormap(&P.tk);
    prefetch_tensormap(&P.tq);
    prefetch_tensormap(&P.tdo);
    prefetch_tensormap(&P.tv);
  }
  const CtaItem item = UNEVEN ? cta_item(P.order) : CtaItem{(int)blockIdx.x, (int)blockIdx.y, (int)blockIdx.z};
  const int nblk = item.block, hk = item.head, b = item.batch;
  const int group = (int)P.group.d;
  const SeqInfo si = seq_info(a.cu_seqlens_q, a.cu_seqlens_k, nullptr, nullptr, a.seqlen_q, a.seqlen_k,
                              a.use_mask_shift, a.mask_shift, b);
  const int n0 = nblk * kB;
  if (n0 >= si.sk) return;
  int m_lo, m_hi;
  query_block_range(n0, kB, BQ, si.sq, si.shift, a.window_left, a.window_right, m_lo, m_hi);
  const int nmb = m_hi - m_lo;
  const int iters = nmb * group;

  if (threadIdx.x == 64) {  // reads global memory: not in front of the first loads
    abort_init(abort_flag, P.status);
    if (s_base & 1023u) abort_raise(abort_flag, W_B_ALIGN);  // the swizzled tiles need a 1024-byte aligned base
  }
  if (threadIdx.x == 0) {
    mbar_init(bar_k, 1);
    mbar_init(bar_v, 1);
    for (int s = 0; s < NSQ; ++s) {
      mbar_init(bar_q_full(s), 1);
      mbar_init(bar_q_empty(s), 1);
    }
    for (int s = 0; s < NSO; ++s) {
      mbar_init(bar_do_full(s), 1);
      mbar_init(bar_do_empty(s), 1);
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(bar_st_full(s), 1);
      mbar_init(bar_st_empty(s), C::WARPS);
    }
    mbar_init(bar_s, 1);
    mbar_init(bar_dp, 1);
    mbar_init(bar_ds, C::WARPS);
    mbar_init(bar_p, C::WARPS);
    mbar_init(bar_sread, C::WARPS);
    fence_barrier_init();
    fence_proxy_async();
    if (iters > 0) {
      // This thread has made the barriers, so it can start the first block's loads while the CTA still sets itself up:
      // K and Q first, which S^T(0) needs
      auto load = [&](uint32_t dst, const CUtensorMap* tm, uint32_t bar, int chunk, int row, int head, int64_t batch) {
        mbar_expect_tx(bar, C::NCHUNK * chunk);
        for (int c = 0; c < C::NCHUNK; ++c) tma_load_4d(dst + c * chunk, tm, bar, c * 64, row, head, (int)batch);
      };
      const int krow = (int)si.k_row0 + n0, qrow = (int)si.q_row0 + m_lo * BQ;
      load(sK, &P.tk, bar_k, kChunkBytes, krow, hk, si.k_batch);
      load(sQ(0), &P.tq, bar_q_full(0), C::QCHUNK, qrow, hk * group, si.q_batch);
      load(sDO(0), &P.tdo, bar_do_full(0), C::QCHUNK, qrow, hk * group, si.q_batch);
      load(sV, &P.tv, bar_v, kChunkBytes, krow, hk, si.k_batch);
    }
  }
  if (warp == C::WARP_STATS) {
    tmem_alloc(smem_addr(const_cast<uint32_t*>(tmem_ptr_smem)), C::TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_ptr_smem;
  const bool run = (*abort_flag == 0) && iters > 0;

  const float scale_log2 = a.softmax_scale * kLog2e;
  // (query head, query block) of iteration `it`, stepped without divisions: blocks m_lo..m_hi-1 of one head, then the next head
  struct Walk {
    int mb, hq, lo, hi;
    __device__ void next() {
      if (++mb == hi) {
        mb = lo;
        ++hq;
      }
    }
  };
  const Walk walk0{m_lo, hk * group, m_lo, m_hi};

  if (warp < C::WARPS) {
    // ---------------------------------------------------------------- compute warpgroups
    setmaxnreg_inc<C::REGS>();
    const int w = warp >> 2;                       // half of a block's query columns; in the epilogue, of the head dim
    const int kr = (warp & 3) * 32 + lane;         // key row of this thread within the CTA tile
    const int key = n0 + kr;
    const uint32_t lane_off = (uint32_t)((warp & 3) * 32) << 16;
    const uint32_t tS = tmem + lane_off + C::COL_S, tdP = tmem + lane_off + C::COL_DP;
    const uint64_t scale2 = pack2(scale_log2, scale_log2);
    bool ok = (*abort_flag == 0);  // with iters == 0 the loop is skipped and the epilogue writes zeros
    // query rows that see this thread's key: [q_lo, q_hi]
    int q_lo = 0, q_hi = si.sq - 1;
    if (a.window_right >= 0) q_lo = max(q_lo, key - si.shift - a.window_right);
    if (a.window_left >= 0) q_hi = min(q_hi, key - si.shift + a.window_left);
    if (key >= si.sk) q_hi = -1;
    // blocks with a first row in [full_lo, full_hi] are seen whole by all 128 keys
    const int full_lo = n0 + kB > si.sk ? 0x7fffffff : (a.window_right >= 0 ? n0 + kB - 1 - si.shift - a.window_right : 0);
    const int full_hi = min(si.sq, a.window_left >= 0 ? n0 - si.shift + a.window_left + 1 : si.sq) - BQ;
    int m0 = m_lo * BQ;
    for (int it = 0; it < iters && ok; ++it, m0 = m0 + BQ == m_hi * BQ ? m_lo * BQ : m0 + BQ) {
      const int slot = it & 1, par = (it >> 1) & 1;
      // ---- P^T = exp2(S^T * scale - LSE), CW query columns per thread
      ok = mbar_wait(bar_s, it & 1, W_B_S, abort_flag);
      if (!ok) break;
      const ulonglong2* nlse = reinterpret_cast<const ulonglong2*>(sStats + slot * 2 * BQ + w * CW);
      const ulonglong2* ndsum = reinterpret_cast<const ulonglong2*>(sStats + slot * 2 * BQ + BQ + w * CW);
      ok = mbar_wait(bar_st_full(slot), par, W_B_STATS_FULL, abort_flag);
      if (!ok) break;
      tc_fence_after();
      float p[CW];
      {
        uint32_t s[CW / 32][32];
#pragma unroll
        for (int h = 0; h < CW / 32; ++h) tmem_ld32(tS + w * CW + h * 32, s[h]);
        tmem_wait_ld();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(bar_sread);  // S^T(it) is in registers: the next S^T may overwrite it
#pragma unroll
        for (int c = 0; c < CW; c += 4) {
          const ulonglong2 l4 = nlse[c / 4];
          const uint32_t* x = &s[c / 32][c % 32];
          float x0, x1, x2, x3;
          unpack2(fma2(pack2u(x[0], x[1]), scale2, l4.x), x0, x1);
          unpack2(fma2(pack2u(x[2], x[3]), scale2, l4.y), x2, x3);
          p[c] = ex2(x0);
          p[c + 1] = ex2(x1);
          p[c + 2] = ex2(x2);
          p[c + 3] = ex2(x3);
        }
      }
      if (m0 < full_lo || m0 > full_hi) {
        const int c_lo = q_lo - m0 - w * CW, c_hi = q_hi - m0 - w * CW;
#pragma unroll
        for (int c = 0; c < CW; ++c) p[c] = (c >= c_lo && c <= c_hi) ? p[c] : 0.f;
      }
      // ---- dP^T(it) into registers, then P^T (16-bit) over the first half of this warp's own columns of it: the A
      //      operand of dV
      ok = mbar_wait(bar_dp, it & 1, W_B_DP, abort_flag);
      if (!ok) break;
      tc_fence_after();
      uint32_t d[CW / 32][32];
#pragma unroll
      for (int h = 0; h < CW / 32; ++h) tmem_ld32(tdP + w * CW + h * 32, d[h]);
      tmem_wait_ld();
      {
        uint32_t pk[CW / 2];
#pragma unroll
        for (int c = 0; c < CW; c += 2) pk[c >> 1] = Pack<T>::two(p[c], p[c + 1]);
        if constexpr (CW == 64)
          tmem_st32(tdP + w * CW, pk);
        else
          tmem_st16(tdP + w * CW, pk);
      }
      tmem_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar_p);
      // ---- dS^T = P^T o (dP^T - D), 16-bit, over the second half: the A operand of dK
      {
        uint32_t dk[CW / 2];
#pragma unroll
        for (int c = 0; c < CW; c += 4) {
          const ulonglong2 d4 = ndsum[c / 4];
          const uint32_t* x = &d[c / 32][c % 32];
          float x0, x1, x2, x3;
          unpack2(mul2(pack2(p[c], p[c + 1]), add2(pack2u(x[0], x[1]), d4.x)), x0, x1);
          unpack2(mul2(pack2(p[c + 2], p[c + 3]), add2(pack2u(x[2], x[3]), d4.y)), x2, x3);
          dk[c >> 1] = Pack<T>::two(x0, x1);
          dk[(c >> 1) + 1] = Pack<T>::two(x2, x3);
        }
        if constexpr (CW == 64)
          tmem_st32(tdP + w * CW + CW / 2, dk);
        else
          tmem_st16(tdP + w * CW + CW / 2, dk);
      }
      tmem_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) {
        mbar_arrive(bar_st_empty(slot));
        mbar_arrive(bar_ds);
      }
    }
    // every MMA of the CTA has completed once the last block's Q slot has been released
    if (ok && iters > 0) ok = mbar_wait(bar_q_empty((iters - 1) % NSQ), ((iters - 1) / NSQ) & 1, W_B_QDO_EMPTY, abort_flag);
    tc_fence_after();

    // ---- epilogue: dK (scaled) and dV
    ok = __all_sync(0xffffffffu, ok && *abort_flag == 0);  // the TMEM loads below are warp-wide instructions
    const bool accumulate = a.accumulate_dkv != 0;
    if (ok) {
#pragma unroll
      for (int which = 0; which < 2; ++which) {
        const float sc = which ? a.softmax_scale : 1.f;
#pragma unroll
        for (int col0 = 0; col0 < DH / 2; col0 += 32) {
          const int col = w * (DH / 2) + col0;
          uint32_t o[32];
          if (iters > 0) {
            tmem_ld32(tmem + lane_off + (which ? C::COL_DK : C::COL_DV) + col, o);
            tmem_wait_ld();
          } else {
#pragma unroll
            for (int i = 0; i < 32; ++i) o[i] = 0u;
          }
          if (accumulate) {
            float* acc = (which ? a.dk_accum : a.dv_accum) +
                         (((int64_t)si.k_batch * a.seqlen_k + si.k_row0 + key) * a.heads_k + hk) * a.head_dim + col;
#pragma unroll
            for (int i = 0; i < 32; i += 4) {
              if (key < si.sk && col + i < a.head_dim) {
                float4 cur = *reinterpret_cast<float4*>(acc + i);
                cur.x += __uint_as_float(o[i]) * sc;
                cur.y += __uint_as_float(o[i + 1]) * sc;
                cur.z += __uint_as_float(o[i + 2]) * sc;
                cur.w += __uint_as_float(o[i + 3]) * sc;
                *reinterpret_cast<float4*>(acc + i) = cur;
              }
            }
          } else {
            // 16-bit rows over the K and V tiles (every MMA is done), 16-byte pieces swizzled
#pragma unroll
            for (int i = 0; i < 32; i += 8) {
              uint4 v;
              v.x = Pack<T>::two(__uint_as_float(o[i]) * sc, __uint_as_float(o[i + 1]) * sc);
              v.y = Pack<T>::two(__uint_as_float(o[i + 2]) * sc, __uint_as_float(o[i + 3]) * sc);
              v.z = Pack<T>::two(__uint_as_float(o[i + 4]) * sc, __uint_as_float(o[i + 5]) * sc);
              v.w = Pack<T>::two(__uint_as_float(o[i + 6]) * sc, __uint_as_float(o[i + 7]) * sc);
              *reinterpret_cast<uint4*>(smem + which * C::TILE_K + kr * (DH * 2) + ((((col + i) / 8) ^ (kr & 7)) << 4)) = v;
            }
          }
        }
      }
    }
    named_bar_sync(1, 32 * C::WARPS);
    if (ok && !accumulate) {
      // Whole rows by neighbouring threads.  (One row per thread, straight from the registers, put every 16-byte store of
      // a warp in 32 different lines: 7700 cycles per CTA at head dim 128.)
      constexpr int CPR = DH / 8;  // 16-byte pieces per row
#pragma unroll
      for (int which = 0; which < 2; ++which) {
        const FaTensor& tt = which ? a.dk : a.dv;
        T* g = reinterpret_cast<T*>(tt.ptr) + si.k_batch * tt.stride_b + (si.k_row0 + n0) * tt.stride_s + (int64_t)hk * tt.stride_h;
        const int rows = min(kB, si.sk - n0), col = (int)threadIdx.x % CPR;
        if (col * 8 < a.head_dim)
          for (int row = threadIdx.x / CPR; row < rows; row += 32 * C::WARPS / CPR)
            *reinterpret_cast<uint4*>(g + row * tt.stride_s + col * 8) =
                *reinterpret_cast<const uint4*>(smem + which * C::TILE_K + row * (DH * 2) + ((col ^ (row & 7)) << 4));
      }
    }
  } else {
    setmaxnreg_dec<C::REGS_OTHER>();
    if (warp == C::WARP_PRODUCER) {
      // -------------------------------------------------------------- TMA producer
      if (lane == 0 && run) {
        const int qb = (int)si.q_batch;
        bool ok = true;
        Walk wk = walk0;
        wk.next();  // block 0 is on its way
        for (int it = 1; it < iters && ok; ++it, wk.next()) {
          const int qs = it % NSQ, os = it % NSO;
          const int row = (int)si.q_row0 + wk.mb * BQ, hq = wk.hq;
          ok = mbar_wait(bar_q_empty(qs), ((it / NSQ) & 1) ^ 1, W_B_QDO_EMPTY, abort_flag);
          if (!ok) break;
          mbar_expect_tx(bar_q_full(qs), C::TILE_Q);
          for (int c = 0; c < C::NCHUNK; ++c) tma_load_4d(sQ(qs) + c * C::QCHUNK, &P.tq, bar_q_full(qs), c * 64, row, hq, qb);
          ok = mbar_wait(bar_do_empty(os), ((it / NSO) & 1) ^ 1, W_B_QDO_EMPTY, abort_flag);
          if (!ok) break;
          mbar_expect_tx(bar_do_full(os), C::TILE_Q);
          for (int c = 0; c < C::NCHUNK; ++c) tma_load_4d(sDO(os) + c * C::QCHUNK, &P.tdo, bar_do_full(os), c * 64, row, hq, qb);
        }
      }
    } else if (warp == C::WARP_STATS) {
      // -------------------------------------------------------------- LSE / D loader
      // The values of the next block are fetched into registers before the wait for a free slot,
      // so that the global-memory latency is not part of the hand-over.
      bool ok = run;
      constexpr int NL = BQ / 32;
      float l[NL], d[NL];
      Walk wk = walk0;
      auto fetch = [&]() {
        const int m0 = wk.mb * BQ, hq = wk.hq;
        const float* lse_g = a.softmax_lse + ((int64_t)b * a.heads + hq) * a.lse_seqlen;
        const float* d_g = a.softmax_d + ((int64_t)b * a.heads + hq) * a.d_seqlen;
#pragma unroll
        for (int i = 0; i < NL; ++i) {
          const int q = m0 + i * 32 + lane;
          l[i] = q < si.sq ? lse_g[q] : INFINITY;
          d[i] = q < si.sq ? d_g[q] : 0.f;
        }
      };
      if (ok) fetch();
      for (int it = 0; it < iters && ok; ++it) {
        const int slot = it & 1, round = it >> 1;
        ok = mbar_wait(bar_st_empty(slot), (round & 1) ^ 1, W_B_STATS_EMPTY, abort_flag);
        if (!ok) break;
        float* dst = sStats + slot * 2 * BQ;
#pragma unroll
        for (int i = 0; i < NL; ++i) {
          dst[i * 32 + lane] = -l[i] * kLog2e;  // LSE +inf gives exp2(x - inf) = 0 for rows without keys / past the end
          dst[BQ + i * 32 + lane] = -d[i];
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(bar_st_full(slot));
        if (it + 1 < iters) {
          wk.next();
          fetch();
        }
      }
    } else if (warp == C::WARP_MMA || warp == C::WARP_MMA_S) {
      // -------------------------------------------------------------- MMA issuer
      // Two issuing warps.  One issues S^T(i+1) as soon as the compute warps hold S^T(i) in registers.  The other issues
      // the chain dV(i) | dK(i) | dP^T(i+1): dV(i) waits for P^T(i), dK(i) for dS^T(i); both sit over dP^T(i),
      // and the MMAs of one thread execute in order, so dP^T(i+1) overwrites them only after they were read.
      // MMAs of the two threads are not ordered among themselves and need not be.
      if (run) with_head_steps<DH, TRIM>(a.head_dim, [&](auto steps) {  // the whole warp runs the loops (see mma_ss_w); one elected lane issues
        constexpr int F = BFmt<T>::kIdesc;
        constexpr uint32_t idesc_st = make_idesc(kB, BQ, F, 0, 0);   // S^T, dP^T: K-major x K-major, N = BQ queries
        constexpr int KS = decltype(steps)::value;
        constexpr uint32_t idesc_dv = make_idesc(kB, KS * 16, F, 0, 1);  // dV, dK: A K-major (or TMEM), B MN-major, N = head dim
        // One descriptor is built (K tile, K-major); every other operand differs from it only in the
        // low word: the address field (+ byte offset >> 4) and, for MN-major reads, the LBO field.
        const uint64_t d_base = smem_desc_sw128(sK, 16, 1024);
        const uint32_t d_lo = (uint32_t)d_base, d_hi = (uint32_t)(d_base >> 32);
        auto dsc = [&](uint32_t lo_add) { return ((uint64_t)d_hi << 32) | (uint64_t)(d_lo + lo_add); };
        constexpr uint32_t kMn = (uint32_t)((C::QCHUNK - 16) >> 4) << 16;  // K-major -> MN-major (LBO = chunk stride)
        constexpr uint32_t oK = 0, oV = (C::OFF_V - C::OFF_K) >> 4, oQ = (C::OFF_Q - C::OFF_K) >> 4,
                           oDO = (C::OFF_DO - C::OFF_K) >> 4, kTile16 = C::TILE_Q >> 4;
        auto koff = [](int kk) { return (uint32_t)(((kk >> 2) * kChunkBytes + (kk & 3) * 32) >> 4); };  // K-major k-step
        auto koff_q = [](int kk) { return (uint32_t)(((kk >> 2) * C::QCHUNK + (kk & 3) * 32) >> 4); };
        auto moff = [](int kk) { return (uint32_t)((kk * 2048) >> 4) + kMn; };                          // MN-major k-step
        auto pcol = [](int kk) { return kk / (CW / 16) * CW + kk % (CW / 16) * 8; };  // k-step of P in the warps' halves
        auto issue_st = [&](uint32_t d_col, uint32_t a_lo, uint32_t b_lo, uint32_t bar) {
#pragma unroll
          for (int kk = 0; kk < KS; ++kk)
            mma_ss_w(tmem + d_col, dsc(a_lo + koff(kk)), dsc(b_lo + koff_q(kk)), idesc_st, kk > 0);
          tc_commit_w(bar);
        };
        auto issue_dp = [&](int i) {
          const int os = i % NSO;
          bool k = mbar_wait_w(bar_do_full(os), (i / NSO) & 1, W_B_QDO_FULL, abort_flag);
          if (k) {
            tc_fence_after();
            issue_st(C::COL_DP, oV, oDO + os * kTile16, bar_dp);
          }
          return k;
        };
        if (warp == C::WARP_MMA_S) {
          bool ok = mbar_wait_w(bar_k, 0, W_B_KV, abort_flag);
          for (int it = 0; it < iters && ok; ++it) {
            const int qs = it % NSQ;
            if (it > 0) ok = mbar_wait_w(bar_sread, (it - 1) & 1, W_B_S, abort_flag);
            if (ok) ok = mbar_wait_w(bar_q_full(qs), (it / NSQ) & 1, W_B_QDO_FULL, abort_flag);
            if (!ok) break;
            tc_fence_after();
            issue_st(C::COL_S, oK, oQ + qs * kTile16, bar_s);
          }
        } else {
          bool ok = mbar_wait_w(bar_v, 0, W_B_KV, abort_flag);
          if (ok) ok = issue_dp(0);
          for (int it = 0; it < iters && ok; ++it) {
            const int qs = it % NSQ, os = it % NSO;
            // P^T(it) is in TMEM: dV += P^T dO, the last use of this dO tile (dP^T(it) was complete before P^T(it))
            ok = mbar_wait_w(bar_p, it & 1, W_B_PDS, abort_flag);
            if (!ok) break;
            tc_fence_after();
#pragma unroll
            for (int kk = 0; kk < BQ / 16; ++kk)
              mma_ts_w(tmem + C::COL_DV, tmem + C::COL_DP + pcol(kk), dsc(oDO + os * kTile16 + moff(kk)),
                       idesc_dv, (it > 0) || kk > 0);
            tc_commit_w(bar_do_empty(os));
            // dS^T(it) is written: dK += dS^T Q, the last use of this Q tile (S^T(it) of the other issuer read it
            // too: P^T(it) was computed from it)
            ok = mbar_wait_w(bar_ds, it & 1, W_B_PDS, abort_flag);
            if (!ok) break;
            tc_fence_after();
#pragma unroll
            for (int kk = 0; kk < BQ / 16; ++kk)
              mma_ts_w(tmem + C::COL_DK, tmem + C::COL_DP + CW / 2 + pcol(kk), dsc(oQ + qs * kTile16 + moff(kk)),
                       idesc_dv, (it > 0) || kk > 0);
            tc_commit_w(bar_q_empty(qs));
            if (it + 1 < iters) ok = issue_dp(it + 1);
          }
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
  if (warp == C::WARP_STATS) tmem_dealloc(tmem, C::TMEM_COLS);
}


template <typename T, int DH, int BQ>
int launch_bwd_tc(const FaBwdArgs& a, cudaStream_t st) {
  using C = BCfg<DH, BQ>;
  BwdTcParams P;
  P.a = a;
  const bool varlen = a.cu_seqlens_q != nullptr;
  const int64_t q_rows = varlen ? a.total_q : a.seqlen_q, k_rows = varlen ? a.total_k : a.seqlen_k;
  const int64_t nb = varlen ? 1 : a.batch;
  if (make_tmap_4d(&P.tq, a.q, a.dtype, q_rows, a.heads, nb, a.head_dim, BQ)) return 1;
  if (make_tmap_4d(&P.tdo, a.dout, a.dtype, q_rows, a.heads, nb, a.head_dim, BQ)) return 1;
  if (make_tmap_4d(&P.tk, a.k, a.dtype, k_rows, a.heads_k, nb, a.head_dim, kB)) return 1;
  if (make_tmap_4d(&P.tv, a.v, a.dtype, k_rows, a.heads_k, nb, a.head_dim, kB)) return 1;
  constexpr bool kAlone = DH <= 64 && BQ > 64;  // (CTAs that all start at once need no order)
  const bool uneven = !kAlone && (a.window_left >= 0 || a.window_right >= 0 || a.cu_seqlens_q);
  const bool trim = head_trims<DH>(a.head_dim);
  auto kern = trim ? (uneven ? bwd_tc_kernel<T, DH, BQ, !kAlone, true> : bwd_tc_kernel<T, DH, BQ, false, true>)
                   : (uneven ? bwd_tc_kernel<T, DH, BQ, !kAlone, false> : bwd_tc_kernel<T, DH, BQ, false, false>);
  P.status = status_ref(true);
  static fa_host::DeviceOnce once[2][2];
  if (int rc = fa_host::raise_smem_limit(once[trim][uneven], reinterpret_cast<const void*>(kern), C::SMEM_BYTES, "bwd_tc_kernel")) return rc;
  dim3 grid((a.seqlen_k + kB - 1) / kB, a.heads_k, a.batch);
  P.group = fast_div(a.heads / a.heads_k);
  const int head_group = fa_host::cta_head_group(uneven, (int64_t)a.seqlen_q * (a.heads / a.heads_k) * a.head_dim * 4,
                                         (int64_t)a.heads_k * a.batch);
  P.order = cta_order(head_group, grid);
  kern<<<grid, C::THREADS, C::SMEM_BYTES, st>>>(P);
  return fa_host::check_launch("bwd_tc_kernel");
}

}  // namespace

bool bwd_tc_eligible(const FaBwdArgs& a) {
  if (a.head_dim > 256 || a.p_dropout > 0.f) return false;  // head dims 129..256 run in bwd_wide_tc.cu
  if (a.seqlen_k <= 0 || a.seqlen_q <= 0) return false;
  const bool varlen = a.cu_seqlens_q != nullptr;
  const int64_t nb = varlen ? 1 : a.batch, q_rows = varlen ? a.total_q : a.seqlen_q, k_rows = varlen ? a.total_k : a.seqlen_k;
  if (!tma_compatible(a.q, q_rows, a.heads, nb) || !tma_compatible(a.dout, q_rows, a.heads, nb) ||
      !tma_compatible(a.k, k_rows, a.heads_k, nb) || !tma_compatible(a.v, k_rows, a.heads_k, nb))
    return false;
  // the epilogues store 16 bytes at a time
  if (!rows_compatible(a.dq)) return false;
  if (!a.accumulate_dkv && (!rows_compatible(a.dk) || !rows_compatible(a.dv))) return false;
  if (a.head_dim % 8) return false;
  if (a.cu_seqlens_q && (a.total_q <= 0 || a.total_k <= 0)) return false;
  return encode_tiled_fn() != nullptr;
}

int bwd_tc_main(const FaBwdArgs& a, cudaStream_t st) {
  const bool bf = a.dtype == FA_DTYPE_BF16;
  if (a.head_dim <= 64) {
    // 128-row blocks where no two CTAs share an SM: 1 x 2048 tokens, 8/2 heads (32 CTAs) 107.6 us with 64 rows, 81.5 with 128;
    // 1 x 1024, 16 heads (128 CTAs) 19.3 and 16.0.  From 149 CTAs on two share: 8 x 256, 10 heads (160 CTAs) 10.5 and 13.9;
    // 1 x 2048, 16 heads (256 CTAs) 46.1 and 50.2.
    const int64_t ctas = (int64_t)((a.seqlen_k + kB - 1) / kB) * a.heads_k * a.batch;
    if (ctas <= fa_host::sm_count())
      return bf ? launch_bwd_tc<__nv_bfloat16, 64, 128>(a, st) : launch_bwd_tc<__half, 64, 128>(a, st);
    return bf ? launch_bwd_tc<__nv_bfloat16, 64, 64>(a, st) : launch_bwd_tc<__half, 64, 64>(a, st);
  }
  return bf ? launch_bwd_tc<__nv_bfloat16, 128, 128>(a, st) : launch_bwd_tc<__half, 128, 128>(a, st);
}

}  // namespace fa
