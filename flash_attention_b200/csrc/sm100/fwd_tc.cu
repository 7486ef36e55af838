// Forward attention on the 5th-generation tensor cores (tcgen05 + TMEM + TMA), head dim <= 256.
//
// One CTA owns 256 query rows of one (batch, head) [and, with split-KV, one range of key blocks]: two
// 128-row tiles that take turns on the tensor pipe.  Or it owns one tile: two such CTAs share an SM where a tile has few key
// blocks (one_tile), and one has it alone at head dims above 128, where O alone fills 256 TMEM columns.  CTAs are launched heaviest
// first (bottom rows of a causal mask see the most keys).
// Warp roles (384 threads; one tile: 256, without the second four):
//   warps 0-3   softmax of tile 0  (one thread per query row; tcgen05.ld 32x32b gives a thread its row)
//   warps 4-7   softmax of tile 1
//   then        TMA producer: Q tiles once, then K(j), V(j), K(j+1), ... through a ring of slots
//               MMA issuer: the warp stays converged, one elected lane issues every tcgen05.mma
//               owner of the TMEM allocation
//               KV cache: clears the rows of the last V tile that hold no key
// V(j) and K(j+1) arrive on one barrier: a wait of the issuing warp costs 130 to 200 cycles even when there is nothing to wait for
// (16 x 2048 x 16 x 128 causal 328 -> 325 us, 32 x 512 97.0 -> 95.5).
// Registers: 168 (two CTAs per SM: 128) a thread at launch, 4 to 8 bytes spilled.
// With grouped-query heads a tile's 128 rows are (positions x heads of the group), so that both tiles of a CTA end at the same
// key block of a causal mask and a few tokens per sequence fill a tile (prefill of 4096 tokens, 32/8 heads: 179 -> 157 us, and
// 137 with the CTA order of cta_item).  K and V may be a KV cache: lengths on the device, batch index, pages of 64 rows and up.
// What bounds it: the chain S -> softmax -> PV of each tile (about 3100 cycles per pair of 128 x 128 blocks, 2048 of MMA and 2048
// of exponentials at 16 per clock and SM), and per CTA about 5000 cycles before the first and 5000 after the last block (the latter
// worked out from launch times).
// 16 x 2048 x 16 x 128 causal 400 -> 337 us.
// TMEM columns (fp32): S0 [0,128) S1 [128,256) O0 [256,256+D) O1 [256+D,256+2D).  P (16-bit) is
// written over the first 64 columns of its S and fed to the PV MMA as the TMEM A operand.
// MMA order  S0(0) S1(0) | PV0(j) S0(j+1) PV1(j) S1(j+1) | ...  so that while one tile is in its
// softmax the other tile's two MMAs keep the tensor pipe busy; the single in-order issuer is also what
// keeps the two tiles' softmax phases apart (issuers per tile drift into phase and then share the
// exponential unit).  P is handed over in two halves of 64 keys, each followed by its four k-steps
// of PV.
// Softmax works in the exp2 domain with a lazily updated reference maximum: O and the row sum are
// only rescaled when the running maximum has grown by more than 2^8, which keeps the (expensive)
// TMEM round trip of O off the common path; the final O/l and LSE do not depend on that choice.
// Blocks that the mask touches run a second instance of the block code that classifies each 32-column
// chunk for the warp: a chunk that every row sees is left alone, one that no row sees is skipped (no
// exponentials), only the chunks on the mask boundary are tested element by element.  (One instance for
// all blocks, or a masking pre-pass in front of the straight-line code, both measured slower.)
//
// Split-KV (num_splits > 1): the CTA takes one range of key blocks; its normalised partial O and its
// LSE go to the fp32 workspaces and combine.cu merges them (flash_api.cpp:373-389,
// flash_fwd_launch_template.h:70-138).
//
// A persistent form (one CTA per SM drawing items from a counter, the next item's first S behind the
// current item's last PV, a separate epilogue warpgroup or the softmax warps draining O) was built and
// measured: 0.47 ms against 0.40 ms on 16 x 2048 x 16 x 128 causal, 1163 against 1215 TFLOP/s on
// 2 x 8192 full.  The issuing warp pays hundreds of cycles for every barrier test next to warps that
// are busy with exponentials, and the extra item bookkeeping in that warp cost more than the
// overlapped prologue and epilogue gave back.
//
// Same math as compute_attn_1rowblock (csrc/flash_attn/src/flash_fwd_kernel.h:74-580); mask rule of
// csrc/flash_attn/src/softmax.h:142-179; O = 0 and LSE = +inf for rows without a visible key.
#include <cstdlib>
#include <type_traits>

#include "../fa_common.cuh"
#include "ptx.cuh"
#include "tma_host.cuh"

namespace fa {

using namespace ptx;

StatusRef status_ref(bool may_allocate);

namespace {

constexpr int kBM = 128;  // rows per query tile
constexpr int kBN = 128;  // keys per K/V tile
constexpr int kChunkBytes = 128 * 128;  // [128 rows][64 x 16-bit]: one swizzled TMA box
constexpr float kRescaleThreshold = 8.f;

enum WaitCode { W_QFULL = 11, W_KVFULL = 12, W_KVEMPTY = 13, W_SFULL = 14, W_PFULL = 15, W_OFULL = 16, W_VTAIL = 17 };

// NT: query tiles per CTA
template <int DH, int NT>
struct Cfg {
  static constexpr int NCHUNK = DH / 64;
  static constexpr int TILE_BYTES = NCHUNK * kChunkBytes;
  // Head dims up to 128: one 128-row query tile and two CTAs per SM, or two tiles that ping-pong on the tensor pipe and share K
  // and V.  Up to 256: O alone needs 256 TMEM columns and a tile is 64 KiB, so one tile and one CTA per SM, with a 2-slot (K, V) ring.
  static constexpr int CTAS = NT == 1 && DH <= 128 ? 2 : 1;
  static constexpr int WARP_PRODUCER = 4 * NT, WARP_MMA = 4 * NT + 1, WARP_TMEM = 4 * NT + 2, WARP_TAIL = 4 * NT + 3;
  static constexpr int THREADS = 32 * (4 * NT + 4);
  // a thread is launched with 128 (two CTAs), 168 or 255 registers: setmaxnreg only redistributes those
  static constexpr int REGS = CTAS == 2 ? 200 : 216, REGS_OTHER = CTAS == 2 ? 56 : 64, REGS_LAUNCH = CTAS == 2 ? 128 : NT == 2 ? 168 : 255;
  static_assert(128 * NT * REGS + 128 * REGS_OTHER <= THREADS * REGS_LAUNCH, "the registers of one CTA");
  static constexpr int STAGES = DH == 64 ? (CTAS == 2 ? 4 : 8) : DH == 128 ? (CTAS == 2 ? 2 : 4) : 2;
  static constexpr int SMEM_TILES = (NT + STAGES) * TILE_BYTES;
  static constexpr int NBAR = 2 + 2 * STAGES + 10;
  static constexpr int SMEM_BYTES = SMEM_TILES + NBAR * 8 + 32 + 1024;  // + barriers, tmem ptr / abort block, align slack
  static constexpr int TMEM_COLS = CTAS == 2 ? 256 : 512;
  static constexpr int COL_S0 = 0, COL_S1 = 128, COL_O0 = CTAS == 2 ? 128 : 256, COL_O1 = COL_O0 + DH;
  static_assert(CTAS * (SMEM_BYTES + 1024) <= 228 * 1024 && COL_O0 + NT * DH <= TMEM_COLS, "what the CTAs of an SM share");
};

struct FwdTcParams {
  CUtensorMap tq, tk, tv;
  FaFwdArgs a;
  StatusRef status;
  CtaOrder order;
  FastDiv splits, group, page;  // divisors: num_splits, query heads per KV head, rows of a page
  int32_t row_blocks;           // of a sequence's query rows
  int32_t num_splits;  // split-KV: a sequence's key blocks are divided evenly
  // A 128-row query tile holds `tile_pos` positions of `pack` neighbouring heads of one KV head's group, rows ordered
  // (position, head): pack * tile_pos <= 128.  pack = 1: 128 positions of one head.
  int32_t pack, pack_inv, tile_pos;
  int32_t kv_box;  // rows of one K / V load: 128, or 64 where the pages of a paged cache are not a multiple of 128 rows
  int32_t cache;   // K / V are a KV cache: the rows behind a sequence's keys hold anything, NaN patterns included
};

template <typename T>
struct Fmt;
template <>
struct Fmt<__half> {
  static constexpr int kIdesc = 0;
};
template <>
struct Fmt<__nv_bfloat16> {
  static constexpr int kIdesc = 1;
};

// GROUPED: tiles shared by heads and / or keys in a KV cache (the plain instance keeps its geometry as constants: read from
// the parameters it took 436 us instead of 397 on 16 x 2048 x 16 x 128 causal)
template <typename T, int DH, int NT, bool GROUPED, bool TRIM>
__global__ void __launch_bounds__(Cfg<DH, NT>::THREADS, Cfg<DH, NT>::CTAS) fwd_tc_kernel(const __grid_constant__ FwdTcParams P) {
  using C = Cfg<DH, NT>;
  const FaFwdArgs& a = P.a;
  extern __shared__ unsigned char smem_unaligned[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_unaligned) + 1023) & ~uintptr_t(1023));
  const uint32_t s_base = smem_addr(smem);
  const uint32_t sQ = s_base;                          // NT tiles
  const uint32_t sKV = s_base + NT * C::TILE_BYTES;  // STAGES slots
  const uint32_t bar0 = s_base + C::SMEM_TILES;
  auto bar_qfull = [&](int t) { return bar0 + 8 * t; };
  auto bar_full = [&](int s) { return bar0 + 8 * (2 + s); };
  auto bar_empty = [&](int s) { return bar0 + 8 * (2 + C::STAGES + s); };
  auto bar_sfull = [&](int t) { return bar0 + 8 * (2 + 2 * C::STAGES + t); };
  auto bar_pfull = [&](int t) { return bar0 + 8 * (2 + 2 * C::STAGES + 2 + t); };
  auto bar_ofull = [&](int t) { return bar0 + 8 * (2 + 2 * C::STAGES + 4 + t); };
  auto bar_pfull_b = [&](int t) { return bar0 + 8 * (2 + 2 * C::STAGES + 6 + t); };
  const uint32_t bar_vtail = bar0 + 8 * (2 + 2 * C::STAGES + 8), bar_vtail_go = bar0 + 8 * (2 + 2 * C::STAGES + 9);
  volatile uint32_t* tmem_ptr_smem = reinterpret_cast<volatile uint32_t*>(smem + C::SMEM_TILES + C::NBAR * 8);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + C::SMEM_TILES + C::NBAR * 8 + 4);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == C::WARP_PRODUCER * 32) {  // the TMA unit fetches the three descriptors while the CTA sets itself up
    prefetch_tensormap(&P.tq);
    prefetch_tensormap(&P.tk);
    prefetch_tensormap(&P.tv);
  }
  const int pack = GROUPED ? P.pack : 1, tile_pos = GROUPED ? P.tile_pos : kBM, pack_inv = GROUPED ? P.pack_inv : 65536;
  const bool cache = GROUPED && P.cache;
  const CtaItem item = cta_item(P.order);
  const int b = item.batch, h = item.head * pack, hk = (int)P.group.div(h);  // h: first head of the tile rows
  SeqInfo si = seq_info(a.cu_seqlens_q, a.cu_seqlens_k, GROUPED ? a.seqused_k : nullptr, GROUPED ? a.kv_batch_idx : nullptr, a.seqlen_q,
                        a.seqlen_k, a.use_mask_shift, a.mask_shift, b, GROUPED ? a.seqused_k_extra : 0);
  if (cache) si.sk = min(si.sk, a.seqlen_k);
  // heaviest blocks (largest row index under a causal mask) first; with split-KV the splits of a row block are neighbours
  // (Shuffles as in cta_item, but where it was faster to keep the block ranges in ordinary registers: the plain instances of two tiles, whose
  // warps compare every block against them, and of head dim 128.  1 x 2048 x 16384 tokens, 16 heads causal: 128 228.9 us, 240.2 with; 64 209.7,
  // 213.8.  Trimmed, 8192 tokens: no mask, 80 433, 445 in ordinary registers.  One tile: the test of num_splits costs more than a multiplication,
  // 16 x 2048 x 128 85.0, 85.4 with it.)
  constexpr bool kPlainTwo = !GROUPED && NT == 2 && !TRIM;
  const int mrank = kPlainTwo                 ? (P.num_splits > 1 ? (int)P.splits.div(item.block) : item.block)
                    : !GROUPED && DH == 128 ? (int)P.splits.div(item.block)
                    : P.num_splits > 1      ? __shfl_sync(0xffffffffu, (int)P.splits.div(item.block), 0)
                                            : item.block;
  const int split = kPlainTwo && P.num_splits <= 1 ? 0 : item.block - mrank * P.num_splits, mblk = P.row_blocks - 1 - mrank;
  const int m_base = mblk * NT * tile_pos;
  if (m_base >= si.sq) return;  // uniform for the CTA

  // per-tile key block ranges
  auto part_blocks = [&] { return (int)P.splits.div((max(si.sk, 0) + kBN - 1) / kBN + P.num_splits - 1); };
  const int blocks_per_split = kPlainTwo ? part_blocks() : P.num_splits > 1 ? __shfl_sync(0xffffffffu, part_blocks(), 0) : 0;
  if (GROUPED && P.num_splits > 1 && split * blocks_per_split * kBN >= si.sk) {
    // A part behind the last key (most of them where short sequences stand in a large cache) only says so: no barriers, no
    // tensor memory (32 sequences of 124 tokens in caches of 16384, 8/2 heads of 128, 5 parts: 17.9 -> 15.5 us).  Not in the
    // plain instance, whose lengths the host knows: it took 843 us instead of 836 on 16 x 2048, 32 heads of 64.
#pragma unroll 1
    for (int i = threadIdx.x; i < NT * kBM; i += C::THREADS) {
      const int t = i / kBM, r = i % kBM, rp = (r * pack_inv) >> 16, row = m_base + t * tile_pos + rp;
      if (rp < tile_pos && row < si.sq)
        a.lse_accum[((int64_t)split * a.batch * a.heads + (int64_t)b * a.heads + h + r - rp * pack) * a.seqlen_q + row] = -INFINITY;
    }
    return;
  }
  int lo[2], hi[2];
  bool active[2];
#pragma unroll
  for (int t = 0; t < 2; ++t) {
    const int m0 = m_base + t * tile_pos;
    active[t] = t < NT && m0 < si.sq;
    if (active[t]) {
      key_block_range(m0, tile_pos, kBN, si.sk, si.shift, a.window_left, a.window_right, lo[t], hi[t]);
      if (P.num_splits > 1) {
        lo[t] = max(lo[t], split * blocks_per_split);
        hi[t] = min(hi[t], (split + 1) * blocks_per_split);
        if (hi[t] <= lo[t]) lo[t] = hi[t] = 0;
      }
    } else {
      lo[t] = hi[t] = 0;
    }
  }
  int J_lo, J_hi;
  if (hi[0] > lo[0] && hi[1] > lo[1]) {
    J_lo = min(lo[0], lo[1]);
    J_hi = max(hi[0], hi[1]);
  } else if (hi[0] > lo[0]) {
    J_lo = lo[0];
    J_hi = hi[0];
  } else {
    J_lo = lo[1];
    J_hi = hi[1];
  }
  const int nblk = J_hi - J_lo;  // may be 0
  // Cache: block whose V rows past the last key are zeroed in shared memory (their P is 0, but 0 * NaN is not)
  const int j_tail = cache && (si.sk % kBN) && (si.sk - 1) / kBN < J_hi && (si.sk - 1) / kBN >= J_lo ? (si.sk - 1) / kBN : -1;

  const int nchunk = head_chunks<DH, TRIM>(a.head_dim);
  auto load_q = [&](int t) {
    if (!active[t] || hi[t] <= lo[t]) return;
    mbar_expect_tx(bar_qfull(t), nchunk * 128 * pack * tile_pos);
    const int r0 = (int)si.q_row0 + m_base + t * tile_pos;
    for (int c = 0; c < nchunk; ++c)
      tma_load_4d(sQ + t * C::TILE_BYTES + c * kChunkBytes, &P.tq, bar_qfull(t), c * 64, pack > 1 ? h : r0, pack > 1 ? r0 : h, (int)si.q_batch);
  };
  // Paged cache: the page of the block after the current one is looked up a block ahead, so that the producer does not
  // stand in front of a free slot with a global load to wait for.  (With 64-row pages the second half is looked up.)
  int page_key = -1, page_id = 0;
  auto page_at = [&](int key) { return a.block_table[(int64_t)b * a.block_table_stride + P.page.div(key)]; };
  auto page_of = [&](int key) { return key == page_key ? page_id : page_at(key); };
  // ring item idx: K of block J_lo + idx / 2 (idx even) or V (odd)
  // V(j) and K(j + 1), which the MMA warp needs at the same time, arrive on one barrier, that of V's slot.
  auto load_kv = [&](int idx) {
    const int slot = idx % C::STAGES, j = J_lo + (idx >> 1);
    const uint32_t bar = bar_full(idx > 0 && !(idx & 1) ? (idx - 1) % C::STAGES : slot);
    const CUtensorMap* tm = (idx & 1) ? &P.tv : &P.tk;
    const uint32_t dst = sKV + slot * C::TILE_BYTES;
    if (GROUPED && a.block_table) {  // one lookup per load; rows past the last key are not loaded page by page
      const int n_box = min((min(kBN, si.sk - j * kBN) + P.kv_box - 1) / P.kv_box, kBN / P.kv_box);
      mbar_expect_tx(bar, n_box * P.kv_box * nchunk * 128);
      for (int i = 0; i < n_box; ++i) {
        const int key = j * kBN + i * P.kv_box;
        const int page = page_of(key);
        for (int c = 0; c < nchunk; ++c)
          tma_load_4d(dst + c * kChunkBytes + i * P.kv_box * 128, tm, bar, c * 64, key - (int)(P.page.div(key) * P.page.d), hk, page);
      }
    } else {
      mbar_expect_tx(bar, nchunk * kChunkBytes);
      for (int c = 0; c < nchunk; ++c)
        tma_load_4d(dst + c * kChunkBytes, tm, bar, c * 64, (int)si.k_row0 + j * kBN, hk, (int)si.k_batch);
    }
  };

  if (threadIdx.x == 32) abort_init(abort_flag, P.status);  // a read of global memory: not in front of the first loads
  if (threadIdx.x == 0) {
    for (int t = 0; t < 2; ++t) {
      mbar_init(bar_qfull(t), 1);
      mbar_init(bar_sfull(t), 1);
      mbar_init(bar_pfull(t), 4);
      mbar_init(bar_pfull_b(t), 4);
      mbar_init(bar_ofull(t), 1);
    }
    for (int s = 0; s < C::STAGES; ++s) {
      mbar_init(bar_full(s), s & 1 ? 2 : 1);
      mbar_init(bar_empty(s), 1);
    }
    mbar_init(bar_vtail, 1);
    mbar_init(bar_vtail_go, 1);
    fence_barrier_init();
    fence_proxy_async();
    if (nblk > 0) {
      // This thread has made the barriers, so it can start the first block's loads while the CTA still sets itself up:
      // what S of the first tile needs goes first
      load_q(0);
      load_kv(0);
      if (NT > 1) load_q(1);
      load_kv(1);
      if (nblk == 1) mbar_arrive(bar_full(1));  // no K behind the last V
    }
  }
  if (warp == C::WARP_TMEM) {
    tmem_alloc(smem_addr(const_cast<uint32_t*>(tmem_ptr_smem)), C::TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_ptr_smem;

  const float scale_log2 = a.softmax_scale * kLog2e;

  if (warp < 4 * NT) {
    // ------------------------------------------------------------------ softmax warpgroups
    if (C::REGS_LAUNCH < C::REGS) setmaxnreg_inc<C::REGS>();
    const int t = NT > 1 ? warp >> 2 : 0;
    const int lo_t = t ? lo[1] : lo[0], hi_t = t ? hi[1] : hi[0];  // (indexing by t would put the arrays into local memory)
    const bool active_t = t ? active[1] : active[0];
    const int row_in_tile = (warp & 3) * 32 + lane;
    const int m0 = m_base + t * tile_pos;
    const int pos_in_tile = (row_in_tile * pack_inv) >> 16;             // row_in_tile / pack
    const int row = m0 + (GROUPED ? min(pos_in_tile, tile_pos - 1) : pos_in_tile);                  // query position of this thread's row
    const int head = h + row_in_tile - pos_in_tile * pack;
    const bool row_valid = pos_in_tile < tile_pos && row < si.sq;
    const uint32_t lane_off = (uint32_t)((warp & 3) * 32) << 16;
    const uint32_t tS = tmem + lane_off + (t ? C::COL_S1 : C::COL_S0);
    const uint32_t tO = tmem + lane_off + (t ? C::COL_O1 : C::COL_O0);
    float m_used = -INFINITY;
    bool ok = true;
    // first / last visible key of this row (inclusive)
    int col_first = 0, col_last = si.sk - 1;
    if (a.window_right >= 0) col_last = min(col_last, row + si.shift + a.window_right);
    if (a.window_left >= 0) col_first = max(col_first, row + si.shift - a.window_left);

    const uint64_t scale2 = pack2(scale_log2, scale_log2);
    uint64_t l_sum2 = pack2(0.f, 0.f);  // two running partial row sums (even / odd columns)
    for (int j = lo_t; j < hi_t && ok; ++j) {
      const int it = j - lo_t;
      const bool first_block = it == 0;
      ok = mbar_wait(bar_sfull(t), it & 1, W_SFULL, abort_flag);
      if (!ok) break;
      tc_fence_after();
      const int n0 = j * kBN;
      const bool need_mask = (n0 + kBN - 1 >= si.sk) ||
                             (a.window_right >= 0 && n0 + kBN - 1 > m0 + si.shift + a.window_right) ||
                             (a.window_left >= 0 && n0 < m0 + tile_pos - 1 + si.shift - a.window_left);
      // One block of the online softmax.  MASKED = false is the straight-line version for blocks that every row
      // sees entirely; MASKED = true classifies each 32-column chunk for the warp: bit q of `none` = no row of
      // this warp sees chunk q (no maximum, no exponentials, P = 0), bit q of `part` = the mask boundary crosses
      // it (tested element by element), otherwise the chunk is fully visible.
      auto block = [&](auto masked_tag) -> bool {
        constexpr bool MASKED = decltype(masked_tag)::value;
        uint32_t none = 0, part = 0;
        const int c_lo = col_first - n0, c_hi = col_last - n0;
        if (MASKED) {
          // the bounds do not decrease with the row index: lane 0 / lane 31 hold the extremes of the warp
          const int lo_min = __shfl_sync(0xffffffffu, c_lo, 0), lo_max = __shfl_sync(0xffffffffu, c_lo, 31);
          const int hi_min = __shfl_sync(0xffffffffu, c_hi, 0), hi_max = __shfl_sync(0xffffffffu, c_hi, 31);
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const int c0 = 32 * q;
            if (c0 > hi_max || c0 + 31 < lo_min)
              none |= 1u << q;
            else if (!(c0 >= lo_max && c0 + 31 <= hi_min))
              part |= 1u << q;
          }
        }
        // the whole row of S in registers: one round trip to tensor memory
        uint32_t su[4][32];
        tmem_ld32(tS + 0, su[0]);
        tmem_ld32(tS + 32, su[1]);
        tmem_ld32(tS + 64, su[2]);
        tmem_ld32(tS + 96, su[3]);
        tmem_wait_ld();
        if (MASKED) {
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            if (part & (1u << q)) {
#pragma unroll
              for (int i = 0; i < 32; ++i)
                if (!(32 * q + i >= c_lo && 32 * q + i <= c_hi)) su[q][i] = 0xff800000u;  // -inf
            }
          }
        }
        // row maximum: four chains of three-input max
        float mx0 = -INFINITY, mx1 = -INFINITY, mx2 = -INFINITY, mx3 = -INFINITY;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          if (!MASKED || !(none & (1u << q))) {
#pragma unroll
            for (int i = 0; i < 32; i += 8) {
              mx0 = max3(mx0, __uint_as_float(su[q][i]), __uint_as_float(su[q][i + 1]));
              mx1 = max3(mx1, __uint_as_float(su[q][i + 2]), __uint_as_float(su[q][i + 3]));
              mx2 = max3(mx2, __uint_as_float(su[q][i + 4]), __uint_as_float(su[q][i + 5]));
              mx3 = max3(mx3, __uint_as_float(su[q][i + 6]), __uint_as_float(su[q][i + 7]));
            }
          }
        }
        const float m_blk = fmaxf(fmaxf(mx0, mx1), fmaxf(mx2, mx3)) * scale_log2;
        const float m_cand = fmaxf(m_used, m_blk);
        const bool grow = m_cand > m_used + kRescaleThreshold;  // also true when m_used is -inf and m_cand is finite
        if (!first_block && __any_sync(0xffffffffu, grow)) {
          // O and l are relative to m_used: move them to the new reference (PV of the block before must be done)
          if (!mbar_wait(bar_ofull(t), (it - 1) & 1, W_OFULL, abort_flag)) return false;
          tc_fence_after();
          const float f = grow ? fast_exp2(m_used - m_cand) : 1.f;
#pragma unroll
          for (int c0 = 0; c0 < DH; c0 += 16) {
            uint32_t o[16];
            tmem_ld16(tO + c0, o);
            tmem_wait_ld();
#pragma unroll
            for (int i = 0; i < 16; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * f);
            tmem_st16(tO + c0, o);
          }
          l_sum2 = fma2(l_sum2, pack2(f, f), pack2(0.f, 0.f));
        }
        if (grow) m_used = m_cand;
        const float neg_m = m_used == -INFINITY ? 0.f : -m_used;
        const uint64_t neg_m2 = pack2(neg_m, neg_m);
        // P = exp2(S * scale - m), 16-bit, over the first 64 columns of S, handed to the MMA warp in two halves
        // of 64 keys, so that the first four k-steps of PV run while the second half is still being computed
#pragma unroll
        for (int half = 0; half < 2; ++half) {
          uint32_t pu[32];
#pragma unroll
          for (int qq = 0; qq < 2; ++qq) {
            const int q = half * 2 + qq;
            if (MASKED && (none & (1u << q))) {
#pragma unroll
              for (int i = 0; i < 16; ++i) pu[qq * 16 + i] = 0u;
            } else {
#pragma unroll
              for (int i = 0; i < 32; i += 2) {
                const uint64_t x = fma2(pack2u(su[q][i], su[q][i + 1]), scale2, neg_m2);
                float x0, x1;
                unpack2(x, x0, x1);
                const float e0 = ex2(x0), e1 = ex2(x1);
                l_sum2 = add2(l_sum2, pack2(e0, e1));
                pu[qq * 16 + (i >> 1)] = Pack<T>::two(e0, e1);
              }
            }
          }
          tmem_st32(tS + half * 32, pu);
          tmem_wait_st();
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(half ? bar_pfull_b(t) : bar_pfull(t));
        }
        return true;
      };
      ok = need_mask ? block(std::true_type{}) : block(std::false_type{});
    }
    float l_sum;
    {
      float la, lb;
      unpack2(l_sum2, la, lb);
      l_sum = la + lb;
    }

    // ---- epilogue: O / l -> shared (swizzled) -> coalesced global stores; LSE
    if (active_t) {
      const int n_it = hi_t - lo_t;
      bool have_o = n_it > 0 && ok;
      if (have_o) {
        ok = mbar_wait(bar_ofull(t), (n_it - 1) & 1, W_OFULL, abort_flag);
        have_o = ok;
        tc_fence_after();
      }
      float inv = 0.f;
      if (ok) {
        // The sum is 0 without a visible key and NaN where a score is NaN: O and the LSE of a part are NaN then, so that the
        // merge cannot take the part for an empty one.  (In one pass the LSE of both is +inf, as in the reference.)
        const bool empty = l_sum == 0.f;
        inv = empty ? 0.f : 1.f / l_sum;
        const float lse = (m_used + log2f(l_sum)) * kLn2;
        if (row_valid) {
          if (P.num_splits > 1)  // the split workspaces are (split, batch, head, row): not packed, -inf marks an empty part
            a.lse_accum[((int64_t)split * a.batch * a.heads + (int64_t)b * a.heads + head) * a.seqlen_q + row] = empty ? -INFINITY : lse;
          else
            a.softmax_lse[((int64_t)b * a.heads + head) * a.lse_seqlen + row] = l_sum > 0.f ? lse : INFINITY;
        }
      }
      unsigned char* stage = smem + t * C::TILE_BYTES;  // the Q tile of this warpgroup is no longer read
      const int tid = threadIdx.x & 127;
      if (P.num_splits > 1) {
        // normalised fp32 partial, as many columns at a time as fit the Q tile, through shared memory (a row per thread,
        // straight from the registers, put every store of a warp in 32 lines); an empty part is not written: its weight is 0
        constexpr int SC = DH > 64 ? 64 : 32, PPR = SC / 4;  // columns at a time, 16-byte pieces of them per row
        static_assert(kBM * SC * 4 <= C::TILE_BYTES, "the staged part of O");
#pragma unroll 1
        for (int c0 = 0; c0 < DH; c0 += SC) {
          if (have_o) {
#pragma unroll
            for (int half = 0; half < SC; half += 32) {
              uint32_t o[32];
              tmem_ld32(tO + c0 + half, o);
              tmem_wait_ld();
#pragma unroll
              for (int i = 0; i < 32; i += 4)
                *reinterpret_cast<float4*>(stage + row_in_tile * (SC * 4) + (((half + i) / 4 ^ (row_in_tile & 7)) << 4)) =
                    make_float4(__uint_as_float(o[i]) * inv, __uint_as_float(o[i + 1]) * inv, __uint_as_float(o[i + 2]) * inv,
                                __uint_as_float(o[i + 3]) * inv);
            }
          }
          named_bar_sync(1 + t, 128);
          const int piece = tid % PPR, col = c0 + piece * 4;
          if (have_o && col < a.head_dim) {
#pragma unroll 4
            for (int r = tid / PPR; r < kBM; r += 128 / PPR) {
              const int rp = (r * pack_inv) >> 16;  // r / pack
              if (rp < tile_pos && m0 + rp < si.sq)
                *reinterpret_cast<float4*>(a.out_accum + (((int64_t)split * a.batch * a.heads + (int64_t)b * a.heads + h + r - rp * pack) *
                                                              a.seqlen_q + m0 + rp) * a.head_dim + col) =
                    *reinterpret_cast<const float4*>(stage + r * (SC * 4) + ((piece ^ (r & 7)) << 4));
            }
          }
          named_bar_sync(1 + t, 128);
        }
      } else {
        if (ok) {
          constexpr int ROWB = DH * 2;
          // O leaves tensor memory 128 columns per round trip (a trip costs ~250 cycles whatever its size)
          constexpr int OB = DH < 128 ? DH : 128;
          uint32_t ob[OB / 32][32];
#pragma unroll
          for (int c0 = 0; c0 < DH; c0 += 32) {
            if (c0 % OB == 0) {
              if (have_o) {
#pragma unroll
                for (int c = 0; c < OB; c += 32) tmem_ld32(tO + c0 + c, ob[c / 32]);
                tmem_wait_ld();
              } else {
#pragma unroll
                for (int c = 0; c < OB / 32; ++c)
#pragma unroll
                  for (int i = 0; i < 32; ++i) ob[c][i] = 0u;
              }
            }
            const uint32_t(&o)[32] = ob[(c0 % OB) / 32];
#pragma unroll
            for (int q4 = 0; q4 < 4; ++q4) {  // four 16-byte chunks of 8 elements
              uint4 pk;
              pk.x = Pack<T>::two(__uint_as_float(o[q4 * 8 + 0]) * inv, __uint_as_float(o[q4 * 8 + 1]) * inv);
              pk.y = Pack<T>::two(__uint_as_float(o[q4 * 8 + 2]) * inv, __uint_as_float(o[q4 * 8 + 3]) * inv);
              pk.z = Pack<T>::two(__uint_as_float(o[q4 * 8 + 4]) * inv, __uint_as_float(o[q4 * 8 + 5]) * inv);
              pk.w = Pack<T>::two(__uint_as_float(o[q4 * 8 + 6]) * inv, __uint_as_float(o[q4 * 8 + 7]) * inv);
              const int chunk = c0 / 8 + q4;
              const int phys = (chunk & ~7) | ((chunk ^ row_in_tile) & 7);
              *reinterpret_cast<uint4*>(stage + row_in_tile * ROWB + phys * 16) = pk;
            }
          }
        }
        named_bar_sync(1 + t, 128);
        constexpr int CPR = DH / 8;  // 16-byte chunks per row
        const int chunk = tid % CPR;
        if (ok && chunk * 8 < a.head_dim) {
          T* og = reinterpret_cast<T*>(a.out.ptr) + si.q_batch * a.out.stride_b + (si.q_row0 + m0) * a.out.stride_s +
                  (int64_t)h * a.out.stride_h + chunk * 8;
#pragma unroll 4
          for (int r = tid / CPR; r < kBM; r += 128 / CPR) {
            const int rp = (r * pack_inv) >> 16;  // r / pack
            if (rp < tile_pos && m0 + rp < si.sq)
              *reinterpret_cast<uint4*>(og + rp * a.out.stride_s + (r - rp * pack) * a.out.stride_h) =
                  *reinterpret_cast<const uint4*>(stage + r * (DH * 2) + (((chunk & ~7) | ((chunk ^ r) & 7)) << 4));
          }
        }
      }
    }
  } else {
    if (C::REGS_LAUNCH < C::REGS) setmaxnreg_dec<C::REGS_OTHER>();
    if (warp == C::WARP_PRODUCER) {
      // ---------------------------------------------------------------- TMA producer
      if (lane == 0) {
        bool ok = true;
        for (int idx = 2; idx < 2 * nblk && ok; ++idx) {  // K and V of the first block are on their way
          const int slot = idx % C::STAGES, round = idx / C::STAGES;
          if (GROUPED && a.block_table && !(idx & 1)) {
            page_key = (J_lo + (idx >> 1)) * kBN;
            page_id = page_at(page_key);
          }
          ok = mbar_wait(bar_empty(slot), (round & 1) ^ 1, W_KVEMPTY, abort_flag);
          if (ok) load_kv(idx);
          if (idx == 2 * nblk - 1) mbar_arrive(bar_full(slot));  // no K behind the last V
        }
      }
    } else if (warp == C::WARP_MMA) {
      // ---------------------------------------------------------------- MMA issuer
      with_head_steps<DH, TRIM>(a.head_dim, [&](auto steps) {  // the whole warp runs the loop (see mma_ss_w); one elected lane issues
        constexpr uint32_t idesc_s = make_idesc(kBM, kBN, Fmt<T>::kIdesc, 0, 0);
        constexpr int KS = decltype(steps)::value;
        constexpr uint32_t idesc_o = make_idesc(kBM, KS * 16, Fmt<T>::kIdesc, 0, 1);
        bool ok = true;
        int p_iter[2] = {0, 0};  // softmax iterations consumed per tile
        // One descriptor is built (Q tile 0, K-major); every other operand differs from it only in the
        // low word: the address field (+ byte offset >> 4) and, for MN-major reads, the LBO field.
        const uint64_t d_base = smem_desc_sw128(sQ, 16, 1024);
        const uint32_t d_lo = (uint32_t)d_base, d_hi = (uint32_t)(d_base >> 32);
        auto dsc = [&](uint32_t lo_add) { return ((uint64_t)d_hi << 32) | (uint64_t)(d_lo + lo_add); };
        constexpr uint32_t kMn = (uint32_t)((kChunkBytes - 16) >> 4) << 16;  // K-major -> MN-major (LBO = chunk stride)
        constexpr uint32_t kTile16 = C::TILE_BYTES >> 4, oKV = (NT * C::TILE_BYTES) >> 4;
        auto issue_s = [&](int t, int slot) {
          const uint32_t d = tmem + (t ? C::COL_S1 : C::COL_S0);
          const uint32_t a_lo = t ? kTile16 : 0u, b_lo = oKV + slot * kTile16;
#pragma unroll
          for (int kk = 0; kk < KS; ++kk) {
            const uint32_t off = (uint32_t)(((kk >> 2) * kChunkBytes + (kk & 3) * 32) >> 4);
            mma_ss_w(d, dsc(a_lo + off), dsc(b_lo + off), idesc_s, kk > 0);
          }
          tc_commit_w(bar_sfull(t));
        };
        // PV in two halves of four k-steps: the softmax warps hand over P in two pieces (keys 0-63, then 64-127)
        auto issue_pv_half = [&](int t, int slot, bool first, int half) {
          const uint32_t d = tmem + (t ? C::COL_O1 : C::COL_O0);
          const uint32_t pa = tmem + (t ? C::COL_S1 : C::COL_S0);
          const uint32_t b_lo = oKV + slot * kTile16 + kMn;
#pragma unroll
          for (int k4 = 0; k4 < 4; ++k4) {
            const int kk = half * 4 + k4;
            mma_ts_w(d, pa + kk * 8, dsc(b_lo + (uint32_t)((kk * 2048) >> 4)), idesc_o, (!first) || kk > 0);
          }
          if (half) tc_commit_w(bar_ofull(t));
        };
        auto in_range = [&](int t, int j) { return j >= lo[t] && j < hi[t]; };
        auto slot_of = [&](int idx) { return idx % C::STAGES; };
        auto par_of = [&](int idx) { return (uint32_t)((idx / C::STAGES) & 1); };
        // (Testing each barrier one MMA group ahead of its use, so that the answer travels while the group before
        // is being issued, was measured here and lost 3-5 %: the tests themselves take issue slots of this warp.)
        if (nblk > 0) {
          // prologue: S_t(J_lo)
          ok = mbar_wait_w(bar_full(slot_of(0)), par_of(0), W_KVFULL, abort_flag);
          for (int t = 0; t < NT && ok; ++t) {
            if (hi[t] > lo[t]) ok = mbar_wait_w(bar_qfull(t), 0, W_QFULL, abort_flag);
            if (!ok) break;
            tc_fence_after();
            if (in_range(t, J_lo)) issue_s(t, slot_of(0));
          }
          if (ok) tc_commit_w(bar_empty(slot_of(0)));
          for (int j = J_lo; j < J_hi && ok; ++j) {
            const int iv = 2 * (j - J_lo) + 1;  // ring index of V(j)
            const int ik = iv + 1;              // ring index of K(j+1)
            const bool more = j + 1 < J_hi;
            ok = mbar_wait_w(bar_full(slot_of(iv)), par_of(iv), W_KVFULL, abort_flag);  // and K(j+1)
            if (GROUPED && ok && j == j_tail) {  // V has landed: WARP_TAIL clears its rows behind the last key
              if (lane == 0) mbar_arrive(bar_vtail_go);
              ok = mbar_wait_w(bar_vtail, 0, W_VTAIL, abort_flag);
            }
            if (!ok) break;
#pragma unroll
            for (int t = 0; t < NT; ++t) {
              if (!ok) break;
              if (in_range(t, j)) {
                const uint32_t par = (uint32_t)(p_iter[t] & 1);
                ok = mbar_wait_w(bar_pfull(t), par, W_PFULL, abort_flag);
                if (!ok) break;
                tc_fence_after();
                issue_pv_half(t, slot_of(iv), j == lo[t], 0);
                ok = mbar_wait_w(bar_pfull_b(t), par, W_PFULL, abort_flag);
                if (!ok) break;
                tc_fence_after();
                issue_pv_half(t, slot_of(iv), j == lo[t], 1);
                ++p_iter[t];
              }
              if (t == NT - 1) tc_commit_w(bar_empty(slot_of(iv)));
              if (more && in_range(t, j + 1)) issue_s(t, slot_of(ik));
              if (more && t == NT - 1) tc_commit_w(bar_empty(slot_of(ik)));
            }
          }
        }
      });
    } else if (GROUPED && warp == C::WARP_TAIL && j_tail >= 0) {
      // ---------------------------------------------------------------- zeroes the rows of the last V tile that hold no key
      // (The MMA warp says when: a wait of this warp's own on the slot's barrier would have to pass all its earlier phases.)
      const int iv = 2 * (j_tail - J_lo) + 1, slot = iv % C::STAGES;
      if (mbar_wait_w(bar_vtail_go, 0, W_VTAIL, abort_flag)) {
        const int first = si.sk - j_tail * kBN;
        unsigned char* v = smem + (NT + slot) * C::TILE_BYTES + first * 128;
        for (int i = lane; i < (kBN - first) * 8; i += 32)
#pragma unroll
          for (int c = 0; c < C::NCHUNK; ++c) *reinterpret_cast<uint4*>(v + c * kChunkBytes + i * 16) = make_uint4(0, 0, 0, 0);
        fence_proxy_async();
        __syncwarp();
        if (lane == 0) mbar_arrive(bar_vtail);
      }
    }
  }

  // ---- teardown
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (*abort_flag) {
    // give copies that may still be in flight time to land before the shared memory is released
    const long long t0 = clock64();
    while (clock64() - t0 < 2000000) {
    }
    __syncthreads();
  }
  if (warp == C::WARP_TMEM) tmem_dealloc(tmem, C::TMEM_COLS);
}

// Heads of a KV head's group that share a query tile: the largest divisor of the group that leaves at least 120 of the
// 128 rows in use.  With the group's heads in one tile the two tiles of a CTA end at the same key block of a causal mask
// (a block in which only one tile works costs both tiles' time), and a few tokens per sequence fill a tile.
int pack_heads(int group) {
  for (int d = group < kBM ? group : kBM; d > 1; --d)
    if (group % d == 0 && kBM / d * d >= 120) return d;
  return 1;
}

template <typename T, int DH, int NT>
int launch_fwd_tc(const FaFwdArgs& a, int64_t kv_batches, cudaStream_t st) {
  using C = Cfg<DH, NT>;
  FwdTcParams P;
  P.a = a;
  const bool varlen = a.cu_seqlens_q != nullptr;
  const int64_t q_rows = varlen ? a.total_q : a.seqlen_q, k_rows = varlen ? a.total_k : a.seqlen_k;
  const int64_t nb = varlen ? 1 : a.batch;
  P.cache = kv_batches > 0;
  P.pack = pack_heads(a.heads / a.heads_k);
  P.pack_inv = (65536 + P.pack - 1) / P.pack;
  P.tile_pos = kBM / P.pack;
  P.kv_box = a.block_table && a.page_block_size % kBN ? 64 : kBN;
  if (P.pack > 1 ? make_tmap_4d_heads(&P.tq, a.q, a.dtype, q_rows, a.heads, nb, a.head_dim, P.pack, P.tile_pos)
                 : make_tmap_4d(&P.tq, a.q, a.dtype, q_rows, a.heads, nb, a.head_dim, kBM))
    return 1;
  const int64_t kv_rows = a.block_table ? a.page_block_size : k_rows, kv_nb = P.cache ? kv_batches : nb;
  if (make_tmap_4d(&P.tk, a.k, a.dtype, kv_rows, a.heads_k, kv_nb, a.head_dim, P.kv_box)) return 1;
  if (make_tmap_4d(&P.tv, a.v, a.dtype, kv_rows, a.heads_k, kv_nb, a.head_dim, P.kv_box)) return 1;
  P.status = status_ref(true);
  P.num_splits = a.num_splits > 1 ? a.num_splits : 1;
  const bool grouped = P.pack > 1 || P.cache;
  const bool trim = head_trims<DH>(a.head_dim);
  auto kern = trim ? (grouped ? fwd_tc_kernel<T, DH, NT, true, true> : fwd_tc_kernel<T, DH, NT, false, true>)
                   : (grouped ? fwd_tc_kernel<T, DH, NT, true, false> : fwd_tc_kernel<T, DH, NT, false, false>);
  static fa_host::DeviceOnce once[2][2];
  if (int rc = fa_host::raise_smem_limit(once[trim][grouped], reinterpret_cast<const void*>(kern), C::SMEM_BYTES, "fwd_tc_kernel")) return rc;
  const int n_m = (a.seqlen_q + NT * P.tile_pos - 1) / (NT * P.tile_pos);
  dim3 grid(n_m * P.num_splits, a.heads / P.pack, a.batch);
  P.splits = fast_div(P.num_splits);
  P.group = fast_div(a.heads / a.heads_k);
  P.page = fast_div(a.block_table ? a.page_block_size : 1);
  P.row_blocks = n_m;
  const int head_group = fa_host::cta_head_group(a.window_left >= 0 || a.window_right >= 0 || a.cu_seqlens_q, (int64_t)a.seqlen_k * a.head_dim * 4 / (a.heads / P.pack / a.heads_k),
                                         (int64_t)a.heads / P.pack * a.batch);
  P.order = cta_order(head_group, grid);
  kern<<<grid, C::THREADS, C::SMEM_BYTES, st>>>(P);
  return fa_host::check_launch("fwd_tc_kernel");
}

}  // namespace

// kv_batches: 0, or the number of sequence slots (pages) of a KV cache
static bool fwd_tc_takes(const FaFwdArgs& a, int64_t kv_batches) {
  if (a.head_dim > 256 || a.p_dropout > 0.f || a.s_dmask) return false;
  if (a.num_splits > 1 && a.cu_seqlens_q) return false;
  if ((a.seqused_k || a.kv_batch_idx || a.block_table) && kv_batches <= 0) return false;
  if (a.seqlen_k <= 0) return false;
  const bool varlen = a.cu_seqlens_q != nullptr;
  const int64_t nb = varlen ? 1 : a.batch, q_rows = varlen ? a.total_q : a.seqlen_q;
  const int64_t kv_rows = a.block_table ? a.page_block_size : varlen ? a.total_k : a.seqlen_k, kv_nb = kv_batches > 0 ? kv_batches : nb;
  if (!tma_compatible(a.q, q_rows, a.heads, nb) || !tma_compatible(a.k, kv_rows, a.heads_k, kv_nb) ||
      !tma_compatible(a.v, kv_rows, a.heads_k, kv_nb))
    return false;
  if ((reinterpret_cast<uintptr_t>(a.out.ptr) & 15) || a.out.stride_s % 8 || a.out.stride_h % 8 || a.out.stride_b % 8)
    return false;
  if (a.cu_seqlens_q && (a.total_q <= 0 || a.total_k <= 0)) return false;
  return encode_tiled_fn() != nullptr;
}

// One tile per CTA and two CTAs per SM, or two tiles per CTA and one.  What a CTA does outside its key blocks (about 9000 cycles) runs
// under the blocks of the other one, and no tile waits for the longer one beside it; but K and V are loaded for each tile, and nothing
// keeps two CTAs' softmax phases apart: a pair of blocks takes 5 to 9 % longer.  So: few blocks per tile.  Measured, one tile / two
// tiles, us, by key blocks of a tile on average:
// causal, window or packed, tiles of one head: head dim 64 40 / 42 (8 blocks), 166 / 172 (12), 66 / 63 (16), 124 / 119 (16), 982 / 969 (24),
// 1673 / 1619 (32); 128 201 / 212 (6), 312 / 320 (8), 346 / 346 (10), 326 / 324 (12), 541 / 521 (16); 96 505 / 524 (16); window of 512, 16384 tokens
// 122 / 141; packed 65536 tokens of 128 to 4096 845 / 898.  Where the tiles of a CTA end together anyway the line is lower: no mask, head dim 128 67 / 74 (3),
// 92 / 93 (4), 113 / 114 (6), 146 / 139 (8), 64 75 / 81 (4), 94 / 100 (6), 124 / 123 (8), 196 / 189 (12), but where all CTAs
// fit two to an SM, and not one, 128 11.5 / 11.4 (2), 16.4 / 15.0 (4), 64 9.6 / 9.8 (2), 13.9 / 12.8 (4); shared tiles (32/8 heads of 128, causal) 33 / 34
// (3), 105 / 106 (4), 100 / 100 (6), 81 / 79 (8), 160 / 152 (12).
// A packed batch of very unequal lengths goes by the length its work belongs to (work_length): 16384 + 128 x 64 tokens causal, 16 heads of 128 2426
// / 1749, 2 x 8192 + 64 x 128 868 / 702, 16/4 heads 879 / 689; lengths from 128 to 4096, where the tails are uneven, 486 / 520, and 16/4 heads, 8 x 2048
// + 100 x 100 tokens, 322 / 277.
// Rows that are not whole 32-byte sectors (head dims 72, 88, 104, 120) make loads dearer, and one tile loads K and V twice: causal 88 98 / 93 (8),
// 104 77 / 71 (6), 196 / 172 (8), 26.3 / 24.4 (4), 120 67 / 62 (6), with shared tiles 104 36 / 32 (4); no mask 32 / 29 (4), 72 29 / 27 (4); two to an
// SM 104 13.6 / 11.5 (2), 40 11.8 / 10.3 (2); caches 104 -3 to +1 % (4), +1 to +16 % (8), shared tiles +1 to +13 % (4); rows that fill one tile, an SM each,
// 104 +2 to +8 % (4), +8 to +12 % (6).
// KV caches, of which only the capacity is known here, one tile against two, by blocks of a part.  Under 2.5 rounds of one-tile CTAs,
// head dim 128 -15 to +3 % (4), -8 to +2 % (8), -2 to +5 % (12), -3 to +7 % (16), 64 with tiles of one head -12 to -6 % (8), -2 to +6 % (12),
// with shared ones -3 to +5 % (8), +2 to +9 % (12); more rounds 128 -3 to +5 % (12), +1 to +7 % (16), 96 -1 to +5 % (16), 64 -6 to +2 % (16).  An odd
// number of tiles leaves the last two-tile CTA of a sequence with one: 300 rows, 10 blocks, 128 41 / 45, 326 x 4 rows, 13 blocks, 64 53 / 56.
// Rows that fill one tile at most: two CTAs on an SM are 12 to 38 % faster than one after the other.  But a CTA that has its SM alone
// gets nothing from sharing it and wants the longer ring of the two-tile form: head dim 128 -1 to +2 % (8), -2 to +14 % (12), +5 to +17 %
// (16), +10 to +19 % (32), 64 -2 to +3 % (16), -2 to +4 % (32).
static bool one_tile_form(int64_t ctas, int row_tiles, bool cache, bool uneven, bool skewed, int pack, int head_dim, double blocks, int num_sms) {
  const bool small = head_dim <= 64, even = row_tiles % 2 == 0, cut = head_dim % 16 != 0;
  if (row_tiles <= 1) return ctas > num_sms || blocks <= (small ? 16.5 : cut ? 3.5 : 10.5);
  if (!cache && !uneven) return blocks <= (ctas > num_sms && ctas <= 2 * num_sms ? (cut ? 1.5 : 2.5) : cut && !small ? 2.5 : 4.5);
  if (cut && !small) return blocks <= (pack > 1 ? 2.5 : 5.5);
  if (!cache) return blocks <= (pack > 1 ? (skewed ? 2.5 : 4.5) : small || skewed ? 14 : 8.5);
  if (ctas >= 5 * num_sms) return blocks <= (head_dim <= 96 ? 16.5 : 12.5);
  return blocks <= (small ? (!even ? 16.5 : pack == 1 ? 12.5 : 8.5) : head_dim <= 96 ? 16.5 : even ? 8.5 : 12.5);
}
// Length of the sequence that a row's work belongs to, on average over the work of a packed batch, from what the host knows: between the least
// that one sequence of the maximum makes it and that maximum.  (16384 + 128 x 64 tokens: 13390, in truth 10965; 4 x 4096 + 32 x 256: 2189, 2816; evenly
// from 128 to 4096: 3021, 2816.)
static double work_length(double total, double batch, double longest) {
  if (longest > total) longest = total;
  if (batch <= 1 || longest * batch <= total) return total / batch;
  const double rest = total - longest;
  return sqrt((longest * longest + rest * rest / (batch - 1)) / total * longest);
}
static bool one_tile(const FaFwdArgs& a, int64_t kv_batches) {
  const int pack = pack_heads(a.heads / a.heads_k), parts = a.num_splits > 1 ? a.num_splits : 1;
  const bool varlen = a.cu_seqlens_q != nullptr;
  const double sq = varlen ? work_length(a.total_q, a.batch, a.seqlen_q) : a.seqlen_q, sk = varlen ? work_length(a.total_k, a.batch, a.seqlen_k) : a.seqlen_k;
  double keys = sk;  // of a row, on average
  if (a.window_right >= 0) keys = (sq <= sk ? sk - sq / 2 : sk * sk / (2 * sq)) + a.window_right;
  if (a.window_left >= 0 && keys > (double)a.window_left + a.window_right + 1) keys = (double)a.window_left + a.window_right + 1;
  if (keys > sk) keys = sk;
  const int pos = kBM / pack, row_tiles = (int)(((int64_t)a.seqlen_q + pos - 1) / pos);
  return one_tile_form((int64_t)a.batch * (a.heads / pack) * row_tiles * parts, row_tiles, kv_batches > 0,
                       a.window_left >= 0 || a.window_right >= 0 || varlen, varlen && sk * a.batch > 1.2 * a.total_k, pack, a.head_dim,
                       keys / kBN / parts, fa_host::sm_count());
}

static volatile int g_last_tiles = 0;
int fwd_tc_last_tiles() { return g_last_tiles; }

template <typename T>
static int fwd_tc_dispatch(const FaFwdArgs& a, int64_t kv_batches, cudaStream_t st) {
  const bool one = a.head_dim > 128 || one_tile(a, kv_batches);
  g_last_tiles = one ? 1 : 2;
  if (a.head_dim > 128) return launch_fwd_tc<T, 256, 1>(a, kv_batches, st);
  if (a.head_dim > 64) return one ? launch_fwd_tc<T, 128, 1>(a, kv_batches, st) : launch_fwd_tc<T, 128, 2>(a, kv_batches, st);
  return one ? launch_fwd_tc<T, 64, 1>(a, kv_batches, st) : launch_fwd_tc<T, 64, 2>(a, kv_batches, st);
}

static int fwd_tc_run(const FaFwdArgs& a, int64_t kv_batches, cudaStream_t st) {
  return a.dtype == FA_DTYPE_BF16 ? fwd_tc_dispatch<__nv_bfloat16>(a, kv_batches, st) : fwd_tc_dispatch<__half>(a, kv_batches, st);
}

bool fwd_tc_eligible(const FaFwdArgs& a) { return fwd_tc_takes(a, 0); }
int fwd_tc(const FaFwdArgs& a, cudaStream_t st) { return fwd_tc_run(a, 0, st); }

// Parts for several tokens per sequence against a KV cache of which only the capacity is known here: the count with the least
// estimated time, in us.  A CTA takes 6 and 1.65 per key block for two tiles, 1.55 for one tile that has its SM alone, 1.7 for one of
// two on an SM (head dims above 128: 2.25); rounds of CTAs count half whole and half by their share, because the lengths differ and a
// CTA that has fewer keys makes room; the merge takes 4, 0.1 per part and what writing and reading the fp32 rows takes at 3 TB/s.
// 178 calls (55 caches of 1 to 63 sequences and 1024 to 32768 rows, each full, ragged and nearly empty; every count from 1 to 12, then 16,
// 20, 24 and 32): 4.7 % off the best count on average, 67 % at most (nearly empty caches: one part is best there), and 22 % faster on average than two
// rounds of CTAs whatever the lengths (36 % off the best).  Six calls are 2 to 31 % slower than with those: two nearly empty
// caches (31 and 17 %), 11 full sequences that are 1.2 rounds in one part (11 %), three ragged ones (2 to 16 %).  The merge of 16384 rows takes 7 us in 2 parts, less than is
// charged here; charged as 4 to 6 TB/s the count is half a percent further off, because more parts also make ragged lengths less even.
// 4 x 128 tokens, 32/8 heads of 128, full caches of 8192 112 -> 80 us; 512 tokens, one of 32768 292 -> 231.
int fwd_tc_cache_splits(int batch, int heads, int heads_k, int seqlen_q, int capacity, int head_dim, int num_sms) {
  const int group = heads / heads_k, pack = pack_heads(group), tile_pos = kBM / pack, blocks = (capacity + kBN - 1) / kBN;
  const int row_tiles = (int)(((int64_t)seqlen_q + tile_pos - 1) / tile_pos);
  const double rows = (double)batch * heads * seqlen_q;
  int best = 1;
  double best_time = 0;
  for (int s = 1; s <= 128 && s <= (blocks > 1 ? blocks : 1); ++s) {
    const int per = (blocks + s - 1) / s;
    const bool one = head_dim > 128 || one_tile_form((int64_t)batch * heads_k * (group / pack) * row_tiles * s, row_tiles, true, true, false, pack, head_dim,
                                                     (double)blocks / s, num_sms);
    const int64_t pos = (int64_t)tile_pos * (one ? 1 : 2);
    const double ctas = (double)batch * heads_k * (group / pack) * (double)((seqlen_q + pos - 1) / pos) * s;
    const bool pair = one && head_dim <= 128 && ctas > num_sms;
    const double block_us = head_dim > 128 ? 2.25 : !one ? 1.65 : pair ? 1.7 : 1.55;
    const double rounds = ctas / (pair ? 2 * num_sms : num_sms), whole = (double)(int64_t)(rounds + 0.999999);
    const double t = (6 + block_us * per) * (rounds <= 1 ? 1 : 0.5 * rounds + 0.5 * whole) + (s > 1 ? 4 + s * (0.1 + rows * head_dim * 8 / 3e6) : 0);
    if (s == 1 || t < best_time) {
      best_time = t;
      best = s;
    }
  }
  return best;
}

// Several tokens per sequence against a KV cache (4 x 128 tokens, 32/8 heads, pages of 256: 469 us on the any-shape kernel,
// 62 + 13 us merge here).  From 17 rows (tokens x heads of a group) on, where the decode kernel's 16 end: 20 rows, batch 8,
// 8192 keys, 32/8 heads of 128 575 -> 126 us; 17 rows, batch 2, 16384 keys, 8 heads of 64 109 -> 59 us.  With a window
// that cuts keys off, the any-shape kernel's 64-row tiles keep what has 32 rows or fewer, and other head dims' few rows.
// The lengths are on the device and the capacity stands for them.  Short sequences in large caches pay for that (16 x 33 rows,
// 4 heads of 128, capacity 8192, attention and merge here / any-shape: no keys before the call 15 / 10 us, 400 21 / 17,
// 1500 28 / 41, 3900 53 / 137; 64 sequences, 32 heads of 64: 90 / 26 without keys, 151 / 193 with 400, 667 / 1537 with 3900).
bool fwd_tc_cache_eligible(const FaFwdArgs& a, int64_t kv_batches) {
  const int64_t rows = (int64_t)a.seqlen_q * (a.heads / a.heads_k);
  const bool all_keys = a.window_right <= 0 && (a.window_left < 0 || (a.window_right == 0 && a.window_left >= a.seqlen_k));
  return rows > (all_keys ? 16 : 32) && kv_batches > 0 && fwd_tc_takes(a, kv_batches);
}
int fwd_tc_cache(const FaFwdArgs& a, int64_t kv_batches, cudaStream_t st) { return fwd_tc_run(a, kv_batches, st); }

}  // namespace fa
