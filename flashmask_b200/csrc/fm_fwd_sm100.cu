// Forward attention on the 5th-generation tensor cores (tcgen05 / UMMA) for
// head dims up to 128: a 64-column and a 128-column variant; smaller head dims
// (multiples of 8) run in the next variant up, the TMA loads filling the
// columns past the end of a head with zeros.  Two more variants serve d = 192 /
// dv = 128 (same plan, 48 KB K tiles, two ring slots) and short calls at
// d = dv = 256 (below).
//
// One CTA owns 256 query rows of one (batch, q head) as two 128-row sub-tiles
// that share every K/V tile.  Warp roles:
//   warps 0-3   softmax of sub-tile 0 (thread t <-> row t, TMEM lane t)
//   warps 4-7   softmax of sub-tile 1
//   warp  8     TMA producer: Q once, then K and V tiles through a 4-slot ring,
//               plus the column bounds of partial tiles (plain loads -> smem)
//   warp  9     UMMA issuer (one elected thread): S_s = Q_s K^T into TMEM,
//               O_s += P_s V with P_s read from TMEM; owns the TMEM allocation
//   warp 10     builds the list of surviving K tiles with per-sub-tile flags
//   warp 11     idle
// TMEM (512 columns): S0 [0,128) S1 [128,256) O0 [256,256+D) O1 [384,384+D);
// P_s (bf16, 64 columns) overlays the upper half of S_s.
// Online softmax keeps a stale running maximum and only rescales O when the
// maximum grew by more than 2^8 (the rescale is done by the softmax warps
// themselves).  Every mbarrier wait is bounded: on expiry the CTA raises an
// abort flag, all roles unwind, TMEM is freed and a status word is set.
//
// d = dv = 256: the O accumulator of 128 rows alone needs 256 TMEM columns, so a CTA owns 128 query
// rows and its two "sub-tiles" are the two 128-column halves of V / O for the SAME rows: both
// warpgroups run the softmax of the same scores (S is computed once per warpgroup, in its own
// buffer), warpgroup s accumulates O[:, 128 s : 128 s + 128) = P V[:, 128 s : ...).  One 64 KB Q tile
// and a two-slot ring of 64 KB K / V tiles.  The score GEMM runs twice per tile (6 MMA units for the
// 4 the mathematics needs), so the CTA-pair kernel is the faster one wherever its blocks of 256 rows
// are full; where they are not, this variant wastes half as many rows and puts twice as many blocks
// on the chip at a time (fwd_wide_kernels in fm_api.cu has the line and the figures).
#include <algorithm>
#include <type_traits>

#include "fm_attn_params.cuh"
#include "fm_sm100.cuh"

namespace fm {

using namespace sm100;

__device__ int g_fwd_status = 0;

#ifdef FM_TRACE
// Debug build only: clock stamps at the phase boundaries of CTAs (x < 64, y = FM_TRACE_Y, z = 0).
#ifndef FM_TRACE_Y
#define FM_TRACE_Y 0
#endif
__device__ long long g_fprof[64 * 16];
#define FPROF(slot) do { if (blockIdx.y == FM_TRACE_Y && blockIdx.z == 0 && blockIdx.x < 64) g_fprof[blockIdx.x * 16 + (slot)] = clock64(); } while (0)
#define FPROF_VAL(slot, v) do { if (blockIdx.y == FM_TRACE_Y && blockIdx.z == 0 && blockIdx.x < 64) g_fprof[blockIdx.x * 16 + (slot)] = (v); } while (0)
#else
#define FPROF(slot)
#define FPROF_VAL(slot, v)
#endif

// D: width q / k are computed at (64, 128, 192 or 256), DV: width of v / o (64, 128 or 256).
template <int D, int DV = D>
struct FwdSm100Cfg {
  static constexpr bool SPLITV = D == 256;              // sub-tiles are halves of V / O, not of the rows
  static constexpr int ROWS = SPLITV ? 128 : 256;       // query rows per CTA
  static constexpr int DVS = SPLITV ? DV / 2 : DV;      // O columns per warpgroup
  // the 64-column variant doubles the ring depth: its slots are half as large; the 192-column one has room
  // for two slots (one K tile and one V tile in flight) beside its two 48 KB Q sub-tiles
  static constexpr int BM = 128, BN = 128, NSTAGE = (D == 64 ? 8 : (D > 128 ? 2 : 4)), NBND = 2, LIST_MAX = 2048;
  static constexpr int NTHREADS = 384;
  static constexpr int SUB = 128 * 128;                 // bytes of a 128-row x 64-col bf16 sub-tile
  static constexpr int Q_BYTES = BM * D * 2;
  static constexpr int K_BYTES = BN * D * 2, V_BYTES = BN * DV * 2;
  static constexpr int SLOT_BYTES = K_BYTES > V_BYTES ? K_BYTES : V_BYTES;
  static constexpr int BND_BYTES = 128 * 4 * 4;
  static constexpr int OFF_Q = 0;
  static constexpr int OFF_KV = OFF_Q + (SPLITV ? 1 : 2) * Q_BYTES;
  // Causal masks: the K and V tiles of the diagonal (the first tile of the list, right to left) are requested at
  // kernel entry into slots 0 and 1, before the list exists, where the ring is deep enough to keep the list
  // build's staging area (64 KB) clear of those two slots.
  static constexpr bool SPEC = NSTAGE >= 4 && NSTAGE * SLOT_BYTES >= 128 * 1024 && 2 * SLOT_BYTES <= 64 * 1024;
  static constexpr int OFF_STAGE = OFF_KV + (SPEC ? 64 * 1024 : 0);
  static constexpr int OFF_BND = OFF_KV + NSTAGE * SLOT_BYTES;
  static constexpr int OFF_LIST = OFF_BND + NBND * BND_BYTES;
  static constexpr int OFF_BAR = OFF_LIST + LIST_MAX * 4;
  static constexpr int OFF_MISC = OFF_BAR + 32 * 8;
  static constexpr int SMEM = OFF_MISC + 64 + 1024;     // + alignment slack
  // block-score variant only: 16 block maxima per softmax thread behind everything else
  static constexpr int OFF_BS = OFF_MISC + 64;
  static constexpr int SMEM_BS = OFF_BS + 16 * BS_ACC_STRIDE * 4 + 1024;
  static_assert(SMEM_BS <= 227 * 1024, "shared memory of the block-score variant");
  // barrier indices
  static constexpr int B_QFULL = 0, B_KVFULL = 2, B_KVEMPTY = 2 + NSTAGE, B_SFULL = 2 + 2 * NSTAGE,
                       B_PFULL = B_SFULL + 2, B_PPART = B_PFULL + 2, B_ODONE = B_PPART + 2, B_BNDFULL = B_ODONE + 2,
                       B_BNDEMPTY = B_BNDFULL + NBND, B_COUNT = B_BNDEMPTY + NBND;
  static_assert((D == 64 && DV == 64) || (D == 128 && DV == 128) || (D == 192 && DV == 128) ||
                    (D == 256 && DV == 256), "head-dim variants");
  static_assert(SMEM_BS <= 227 * 1024 && SMEM <= 227 * 1024, "shared memory");
  static_assert(B_COUNT <= 32, "barrier storage");
  static_assert(OFF_STAGE + LIST_MAX * 8 * 4 <= OFF_BND, "the ring stages the reductions of the list build");
  static_assert(SMEM > 120 * 1024, "one CTA per SM is assumed by the 512-column TMEM allocation");
};

__device__ __forceinline__ float neg_inf() { return __int_as_float(0xff800000); }

// BLOCK_SCORE: 0, or the block size (32 / 64 / 128) of the block-score side output; BLOCK_BOS: document
// starts are given, so a block may straddle two tiles.
// SPLIT: the variant for calls that leave most of the chip idle otherwise (few query rows against many keys).
// The rows of a CTA are (query, head of the GQA group) pairs, 2^pack_log2 heads per query, so that the heads
// sharing a K / V tile share its loads; the K tiles of a row block are dealt to n_split CTAs, whose partial
// results (fp32 O / l and m + log2 l) fwd_combine_kernel merges.
// p.alternate (SPLIT, all rows of the launch fit one sub-tile): both sub-tiles hold the same rows and take the CTA's
// K tiles in turn, each with its own running maximum, sum and O, merged like two parts.  With the second sub-tile
// idle, scores, softmax and P V of one tile after the other form one dependent chain; two chains overlap.
template <int D, int DV, bool IS_BF16, int BLOCK_SCORE, bool BLOCK_BOS, bool SPLIT>
__global__ void __launch_bounds__(384, 1)
fwd_sm100_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                 const __grid_constant__ CUtensorMap tm_v, const AttnKParams p) {
  using Cfg = FwdSm100Cfg<D, DV>;
  constexpr bool SPLITV = Cfg::SPLITV;
  constexpr int ROWS = Cfg::ROWS, DVS = Cfg::DVS;
  static_assert(!(SPLITV && SPLIT), "split calls have head dims up to 128");
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  const uint32_t sbase = smem_u32(smem);
  const uint32_t sQ = sbase + Cfg::OFF_Q, sKV = sbase + Cfg::OFF_KV;
  uint32_t* list = reinterpret_cast<uint32_t*>(smem + Cfg::OFF_LIST);
  const uint32_t bars = sbase + Cfg::OFF_BAR;
  volatile int* misc = reinterpret_cast<volatile int*>(smem + Cfg::OFF_MISC);
  // misc[0] tmem base, [1] cnt, [4] abort
  auto bar = [&](int i) { return bars + 8u * (uint32_t)i; };

  const int tid = threadIdx.x;
  const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
  const int lane = tid & 31;
  if (tid == 0) FPROF(0);
  // descriptor fetches start before anything else: the first loads wait on them
  if (warp == 8 && lane == 0) { tma_prefetch_desc(&tm_q); tma_prefetch_desc(&tm_k); tma_prefetch_desc(&tm_v); }
  const int lg = SPLIT ? p.pack_log2 : 0;
  const int n_rows = p.Sq << lg;             // row x of the launch: query x >> lg, head hq + (x & (2^lg - 1))
  const int n_tiles = (n_rows + ROWS - 1) / ROWS;
  int t = n_tiles - 1 - (SPLIT ? blockIdx.x / p.n_split : blockIdx.x), hq = blockIdx.y << lg, b = blockIdx.z;
  if (!SPLIT && !SPLITV && p.fwd_order) {
    const OrderedCta c = ordered_cta(p.fwd_order, p.Hq);
    t = c.unit; hq = c.head; b = c.b;
  }
  const int hk = hq / (p.Hq / p.Hkv);
  if (tid == 0) FPROF(8);                    // table entry known
  const MaskDesc& md = p.md;
  const int bh_mask = md.ncols ? ((md.mask_B == 1 ? 0 : b) * md.Hm + hq / (p.Hq / md.Hm)) : 0;
  const int ms = t * ROWS;
  const int off = p.Sk - p.Sq;
  const bool alt = SPLIT && p.alternate;
  const int sub_rows = alt || SPLITV ? 0 : 128;        // first row of sub-tile 1 against that of sub-tile 0
  // queries [q_lo(s), q_hi(s)) of sub-tile s
  auto q_lo = [&](int s) { return (ms + sub_rows * s) >> lg; };
  auto q_hi = [&](int s) { return min(((ms + sub_rows * s + 127) >> lg) + 1, p.Sq); };
  // partial result of sub-tile s: its place among the parts of a row
  const int n_parts = SPLIT ? p.n_split << (alt ? 1 : 0) : 1;
  auto part_of = [&](int s) { return (int)(blockIdx.x % p.n_split) * (alt ? 2 : 1) + (alt ? s : 0); };
  // first K tile right of everything these rows can see, and whether the diagonal tile is loaded ahead of the list
  const int nb = (p.Sk + 127) / 128;
  const int n_hi = md.causal ? max(0, min(nb, (q_hi(1) + off + 127) / 128)) : nb;
  const bool spec = Cfg::SPEC && BLOCK_SCORE == 0 && !SPLIT && md.causal && n_hi > 0;

  if (tid == 0) misc[4] = 0;
  if (warp == 8 && lane == 0) {
    mbar_init(bar(Cfg::B_QFULL + 0), 1); mbar_init(bar(Cfg::B_QFULL + 1), 1);
    for (int i = 0; i < Cfg::NSTAGE; ++i) { mbar_init(bar(Cfg::B_KVFULL + i), 1); mbar_init(bar(Cfg::B_KVEMPTY + i), 1); }
    for (int s = 0; s < 2; ++s) {
      mbar_init(bar(Cfg::B_SFULL + s), 1); mbar_init(bar(Cfg::B_PFULL + s), 4); mbar_init(bar(Cfg::B_PPART + s), 4); mbar_init(bar(Cfg::B_ODONE + s), 1);
    }
    for (int i = 0; i < Cfg::NBND; ++i) { mbar_init(bar(Cfg::B_BNDFULL + i), 32); mbar_init(bar(Cfg::B_BNDEMPTY + i), 256); }
    fence_mbar_init();
    // both Q sub-tiles are requested right away: the loads overlap with the
    // list build (rows past the end of the sequence arrive as zeros)
    for (int s = 0; s < (SPLITV ? 1 : 2); ++s) {
      mbar_arrive_expect_tx(bar(Cfg::B_QFULL + s), Cfg::Q_BYTES);
      for (int dc = 0; dc < D / 64; ++dc)
        tma_load_4d(sQ + s * Cfg::Q_BYTES + dc * Cfg::SUB, &tm_q, bar(Cfg::B_QFULL + s), dc * 64, hq,
                    q_lo(s), b);
    }
    if (spec) {
      const int j0 = (n_hi - 1) * 128;
      mbar_arrive_expect_tx(bar(Cfg::B_KVFULL + 0), Cfg::K_BYTES);
      for (int dc = 0; dc < D / 64; ++dc)
        tma_load_4d(sKV + dc * Cfg::SUB, &tm_k, bar(Cfg::B_KVFULL + 0), dc * 64, hk, j0, b);
      mbar_arrive_expect_tx(bar(Cfg::B_KVFULL + 1), Cfg::V_BYTES);
      for (int dc = 0; dc < DV / 64; ++dc)
        tma_load_4d(sKV + Cfg::SLOT_BYTES + dc * Cfg::SUB, &tm_v, bar(Cfg::B_KVFULL + 1), dc * 64, hk, j0, b);
    }
  }
  if (warp == 9) {
    tmem_alloc(sbase + Cfg::OFF_MISC, 512);
    tmem_relinquish();
    if (lane == 0) FPROF(12);
  }
  if (warp == 10) {
    // surviving K tiles, right to left, with the flags of both sub-tiles
    int cnt = 0;
    // the reductions the classification needs are staged in the (still idle) K/V ring
    const MaskDesc mst = stage_minmax(md, bh_mask, 0, n_hi, reinterpret_cast<int32_t*>(smem + Cfg::OFF_STAGE),
                                      Cfg::LIST_MAX, lane);
    if (lane == 0) FPROF(9);                 // reductions staged
    for (int base = n_hi - 1; base >= 0; base -= 32) {
      const int n = base - lane;
      uint32_t f0 = 0, f1 = 0;
      if (n >= 0) {
        f0 = tile_flags(mst, 0, n, q_lo(0), q_hi(0), 128);
        if (SPLITV) f1 = f0;
        else if (ms + 128 < n_rows) f1 = tile_flags(mst, 0, n, q_lo(1), q_hi(1), 128);
        if (spec && n == n_hi - 1 && (f0 | f1) == 0) {
          // the diagonal tile is already on its way into slots 0 / 1, so it is the first list entry whatever its
          // class: an invisible one is computed with the element mask (every score masked, P = 0)
          f0 = FM_TF_ACTIVE | FM_TF_CAUSAL | FM_TF_RAGGED | (md.ncols ? FM_TF_BOUNDS : 0u);
          if (ms + 128 < n_rows) f1 = f0;
        }
      }
      const bool keep = (f0 | f1) != 0;
      const uint32_t bal = __ballot_sync(0xffffffffu, keep);
      const int pos = cnt + __popc(bal & ((1u << lane) - 1u));
      if (keep && pos < Cfg::LIST_MAX) list[pos] = (uint32_t)n | (f0 << 16) | (f1 << 20);
      cnt += __popc(bal);
    }
    if (lane == 0) { misc[1] = min(cnt, Cfg::LIST_MAX); FPROF(10); }
    fence_proxy_async_smem();   // the staging area is handed back to the TMA loads of the ring
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = (uint32_t)misc[0];
  int cnt = misc[1];
  if constexpr (SPLIT) {
    // this CTA's share of the tiles
    const int part = blockIdx.x % p.n_split, lo = cnt * part / p.n_split;
    cnt = cnt * (part + 1) / p.n_split - lo;
    list += lo;
  }
  if constexpr (SPLIT) { if (n_parts > 1) grid_dep_trigger(); }     // the merge follows
  WaitCtx wc{misc + 4, global_timer_ns() + 2000000000ull};
  if (tid == 0) { FPROF(1); FPROF_VAL(7, (long long)cnt); }
  if (cnt == 0) {
    // nothing visible for these 256 rows: write O = 0 and LSE = -inf (sink
    // present: LSE = sink); the Q loads already in flight are awaited and the
    // tensor memory is returned before leaving
    if (warp == 8 && lane == 0) {
      mbar_wait(bar(Cfg::B_QFULL + 0), 0u, wc);
      if (!SPLITV) mbar_wait(bar(Cfg::B_QFULL + 1), 0u, wc);
    }
    if (warp == 9) tmem_dealloc(tmem, 512);
    if constexpr (SPLIT) {
      if (n_parts > 1) {
        // empty parts: the merge skips them
        for (int s = 0; s <= (alt ? 1 : 0); ++s)
          for (int x = ms + tid; x < min(ms + ROWS, n_rows); x += Cfg::NTHREADS)
            p.part_lse[(((int64_t)b * p.Hq + hq + (x & ((1 << lg) - 1))) * p.Sq + (x >> lg)) * n_parts + part_of(s)] = neg_inf();
        return;
      }
    }
    uint16_t* go = reinterpret_cast<uint16_t*>(p.o) + b * p.o_b + hq * p.o_h;
    for (int x = tid; x < ROWS * (DV / 8); x += Cfg::NTHREADS) {
      const int row = ms + x / (DV / 8), cc = x % (DV / 8);
      if (row < n_rows && cc * 8 < p.dv_dim)
        *reinterpret_cast<uint4*>(go + (int64_t)(row >> lg) * p.o_s + (row & ((1 << lg) - 1)) * p.o_h + cc * 8) = make_uint4(0u, 0u, 0u, 0u);
    }
    for (int row = ms + tid; row < min(ms + ROWS, n_rows); row += Cfg::NTHREADS) {
      const int h = hq + (row & ((1 << lg) - 1));
      p.lse[((int64_t)b * p.Hq + h) * p.Sq + (row >> lg)] = p.sink ? p.sink[h] : neg_inf();
    }
    return;
  }

  if (warp < 8) {
    // =========================== softmax warpgroups ===========================
    setmaxnreg_inc<216>();
    const int s = warp >> 2;
    const int r = tid & 127;                   // row inside the sub-tile == TMEM lane
    const int prow = ms + sub_rows * s + r;    // row of the launch
    const bool no_rows = SPLIT && prow - lane >= n_rows;   // the whole warp: it keeps pace with the barriers only
    const int row = prow >> lg;                // its query
    const int head = hq + (prow & ((1 << lg) - 1));
    const uint32_t lane_field = (uint32_t)((warp & 3) * 32) << 16;
    const uint32_t tS = tmem + lane_field + 128u * s;
    const uint32_t tP = tS + 64u;
    const uint32_t tO = tmem + lane_field + 256u + 128u * s;
    const float scale_log2 = p.scale_log2;
    float m_run = neg_inf(), l_run = 0.f;
    int n_done = 0, nbnd = 0;
    bool ok = true;
    // block-score side output: this thread's row of it, and the first key of the row's document
    // Block scores.  A row whose document starts on a block boundary (always, without block_bos) has
    // every block inside one tile: the maxima are stored straight from registers.  Otherwise a block
    // can straddle two tiles, and the maxima are gathered per thread in shared memory, sixteen
    // consecutive blocks of the row (two groups of eight); a group is merged into global memory once
    // no later tile can touch it: tiles are walked right to left, so its turn comes when a tile lies
    // wholly below it.  The merge (load, fmax, store of 32 contiguous bytes per row) runs BEFORE the
    // thread waits for the scores of the next tile, where its load latency overlaps the tensor pipe.
    float* bs_dst = nullptr;
    float* bs_acc = nullptr;
    int bs_bos = 0, bs_pend_lo = INT_MAX, bs_pend_hi = -1;    // pending groups [lo, hi]; lo > hi: none
    bool bs_vec = false;
    if constexpr (BLOCK_SCORE != 0) {
      // (d = 256: both warpgroups see the same scores; warpgroup 0 writes them)
      if (row < p.Sq && !(SPLITV && s == 1))
        bs_dst = p.block_logit + (((int64_t)b * p.Hq + hq) * p.Sq + row) * p.block_ld;
      if constexpr (BLOCK_BOS) {
        bs_acc = reinterpret_cast<float*>(smem + Cfg::OFF_BS) + tid;
#pragma unroll
        for (int c = 0; c < 16; ++c) bs_acc[c * BS_ACC_STRIDE] = neg_inf();
        if (row < p.Sq) {
          bs_bos = p.block_bos[(int64_t)b * p.Sq + row];
          bs_vec = (reinterpret_cast<uintptr_t>(bs_dst) & 15) == 0;
        }
      }
    }
    auto bs_flush = [&](int g) { block_flush<BS_ACC_STRIDE>(bs_dst, bs_acc, g, bs_vec, p.block_cols); };
    for (int i = 0; i < cnt && ok; ++i) {
      const uint32_t e = list[i];
      uint32_t flags = (e >> (16 + 4 * s)) & 0xFu;
      if constexpr (SPLIT) { if (alt) flags = (i & 1) == s ? (e >> 16) & 0xFu : 0u; }
      const bool any_bounds = (((e >> 16) | (e >> 20)) & FM_TF_BOUNDS) != 0;
      const int bslot = nbnd % Cfg::NBND;
      const uint32_t bpar = (uint32_t)(nbnd / Cfg::NBND) & 1u;
      if (any_bounds) {
        // every softmax thread passes through the full barrier of a bounds slot
        // before releasing it, so a warpgroup that runs ahead (inactive on these
        // tiles) cannot arrive twice within one phase of the empty barrier
        ok = __all_sync(0xffffffffu, mbar_wait(bar(Cfg::B_BNDFULL + bslot), bpar, wc));
        if (!ok) break;
      }
      if (flags) {
        int bs_rel0 = 0;
        if constexpr (BLOCK_SCORE != 0) bs_rel0 = (int)(e & 0xFFFFu) * 128 - bs_bos;
        if constexpr (BLOCK_SCORE != 0 && BLOCK_BOS) {
          constexpr int BS_LOG2 = BLOCK_SCORE == 32 ? 5 : (BLOCK_SCORE == 64 ? 6 : 7);
          if (bs_dst && (bs_rel0 & ((1 << BS_LOG2) - 1)) != 0) {
            // blocks this tile can touch: [base, top]; the groups above them are complete
            const int base = bs_rel0 >> BS_LOG2;
            const int top = base + (128 >> BS_LOG2);
            const int lo_rb = max(base, 0), hi_rb = min(top, p.block_cols - 1);
            if (lo_rb <= hi_rb) {
              const int g_top = hi_rb >> 3, g_bot = lo_rb >> 3;
              for (int g = bs_pend_hi; g >= max(bs_pend_lo, g_top + 1); --g) bs_flush(g);
              bs_pend_hi = min(bs_pend_hi, g_top);
              if (bs_pend_lo > bs_pend_hi) { bs_pend_hi = g_top; bs_pend_lo = g_bot; }
              else bs_pend_lo = min(bs_pend_lo, g_bot);
            }
          }
        }
        ok = __all_sync(0xffffffffu, mbar_wait(bar(Cfg::B_SFULL + s), (uint32_t)n_done & 1u, wc));
        if (!ok) break;
        if (tid == 0 && n_done == 0) FPROF(2);
        if (!no_rows) {
#define FM_N_UNIT n_done
#define FM_N_TOT n_done
#include "fm_fwd_sm100_tile.inc"
#undef FM_N_UNIT
#undef FM_N_TOT
          tc_wait_st();
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(bar(Cfg::B_PFULL + s));   // (an arrival per thread instead of per warp measured the same)
        ++n_done;
      }
      if (any_bounds) {
        mbar_arrive(bar(Cfg::B_BNDEMPTY + bslot));
        ++nbnd;
      }
    }
    if constexpr (BLOCK_SCORE != 0 && BLOCK_BOS) {
      if (ok && bs_dst)
        for (int g = bs_pend_hi; g >= bs_pend_lo; --g) bs_flush(g);
    }
    // ---- epilogue: O / l -> bf16 -> smem staging -> coalesced stores; LSE ----
    if (tid == 0) FPROF(3);
    if (ok && n_done > 0) {
      ok = __all_sync(0xffffffffu, mbar_wait(bar(Cfg::B_ODONE + s), (uint32_t)(n_done - 1) & 1u, wc));
      tc_fence_after();
    }
    if (tid == 0) FPROF(4);
    if (ok) {
      const float m_fin = (m_run == neg_inf()) ? 0.f : m_run;
      float l_tot = l_run;
      if (p.sink && n_parts == 1) l_tot += fast_exp2(p.sink[head] * kLog2e - m_fin);
      const float inv = l_tot > 0.f ? 1.f / l_tot : 0.f;
      if (SPLIT && n_parts > 1) {
        // partial result of this share of the tiles, in fp32: 4 * DV contiguous bytes per row
        const int64_t at = (((int64_t)b * p.Hq + head) * p.Sq + row) * n_parts + part_of(s);
        // (-inf marks a part without a visible key; the sum of a part with a NaN or infinite score is NaN and stays one)
        if (prow < n_rows) p.part_lse[at] = l_tot == 0.f ? neg_inf() : m_fin + log2f(l_tot);
#pragma unroll
        for (int c = 0; c < DV / 32; ++c) {
          uint32_t orr[32];
          if (n_done > 0) {
            tmem_ld32(tO + 32 * c, orr);
            tc_wait_ld();
            if (prow < n_rows) {
#pragma unroll
              for (int j = 0; j < 32; j += 4)
                *reinterpret_cast<float4*>(p.part_o + at * DV + 32 * c + j) =
                    make_float4(__uint_as_float(orr[j]) * inv, __uint_as_float(orr[j + 1]) * inv,
                                __uint_as_float(orr[j + 2]) * inv, __uint_as_float(orr[j + 3]) * inv);
            }
          }
        }
      } else {
        uint8_t* stage = smem + Cfg::OFF_Q + (SPLITV ? 0 : s * Cfg::Q_BYTES);   // Q is no longer needed
        constexpr int CH0 = SPLITV ? DVS / 8 : 0;          // d = 256: warpgroup s stages chunks [16 s, 16 s + 16)
#pragma unroll
        for (int c = 0; c < DVS / 32; ++c) {
          uint32_t orr[32];
          if (n_done > 0) {
            tmem_ld32(tO + 32 * c, orr);
            tc_wait_ld();
          } else {
#pragma unroll
            for (int j = 0; j < 32; ++j) orr[j] = 0u;
          }
#pragma unroll
          for (int q4 = 0; q4 < 4; ++q4) {
            uint4 v;
            v.x = pack2<IS_BF16>(__uint_as_float(orr[8 * q4 + 0]) * inv, __uint_as_float(orr[8 * q4 + 1]) * inv);
            v.y = pack2<IS_BF16>(__uint_as_float(orr[8 * q4 + 2]) * inv, __uint_as_float(orr[8 * q4 + 3]) * inv);
            v.z = pack2<IS_BF16>(__uint_as_float(orr[8 * q4 + 4]) * inv, __uint_as_float(orr[8 * q4 + 5]) * inv);
            v.w = pack2<IS_BF16>(__uint_as_float(orr[8 * q4 + 6]) * inv, __uint_as_float(orr[8 * q4 + 7]) * inv);
            const int chunk = CH0 * s + 4 * c + q4;       // 16-byte chunk inside the row
            *reinterpret_cast<uint4*>(stage + r * (DV * 2) + ((chunk ^ (r & (DV / 8 - 1))) << 4)) = v;
          }
        }
        if (prow < n_rows && !(SPLITV && s == 1))
          p.lse[((int64_t)b * p.Hq + head) * p.Sq + row] = l_tot > 0.f ? (m_fin + log2f(l_tot)) * kLn2 : neg_inf();
        __syncwarp();   // each warp stores the 32 rows it staged itself: no cross-warp dependency
        const int rbase = ms + (SPLITV ? 0 : 128 * s);
        uint16_t* go = reinterpret_cast<uint16_t*>(p.o) + b * p.o_b + hq * p.o_h;
        constexpr int CH = DV / 8, CHW = DVS / 8;          // chunks per row, chunks this warpgroup staged
        const int wrow = (warp & 3) * 32;
#pragma unroll 4
        for (int idx = lane; idx < 32 * CHW; idx += 32) {
          const int rr = wrow + idx / CHW, cc = CH0 * s + idx % CHW;
          const int x = rbase + rr;
          if (x < n_rows && cc * 8 < p.dv_dim) {
            const uint4 v = *reinterpret_cast<const uint4*>(stage + rr * (DV * 2) + ((cc ^ (rr & (CH - 1))) << 4));
            *reinterpret_cast<uint4*>(go + (int64_t)(x >> lg) * p.o_s + (x & ((1 << lg) - 1)) * p.o_h + cc * 8) = v;
          }
        }
      }
    }
    if (tid == 0) FPROF(5);
  } else {
    setmaxnreg_dec<64>();
    if (warp == 8) {
      // =========================== TMA / bounds producer ===========================
      int nbnd = 0;
      bool ok = true;
      for (int i = 0; i < cnt && ok; ++i) {
        const uint32_t e = list[i];
        const int j0 = (int)(e & 0xFFFFu) * 128;
        if (!(spec && i == 0) && elect_one()) {       // (the first tile of a causal mask was requested at entry)
          for (int kv = 0; kv < 2 && ok; ++kv) {
            const int k = 2 * i + kv, slot = k % Cfg::NSTAGE;
            const uint32_t par = ((uint32_t)(k / Cfg::NSTAGE) & 1u) ^ 1u;
            ok = mbar_wait(bar(Cfg::B_KVEMPTY + slot), par, wc);
            if (!ok) break;
            mbar_arrive_expect_tx(bar(Cfg::B_KVFULL + slot), kv == 0 ? Cfg::K_BYTES : Cfg::V_BYTES);
            for (int dc = 0; dc < (kv == 0 ? D : DV) / 64; ++dc)
              tma_load_4d(sKV + slot * Cfg::SLOT_BYTES + dc * Cfg::SUB, kv == 0 ? &tm_k : &tm_v,
                          bar(Cfg::B_KVFULL + slot), dc * 64, hk, j0, b);
          }
        }
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        if ((((e >> 16) | (e >> 20)) & FM_TF_BOUNDS) != 0) {
          const int bslot = nbnd % Cfg::NBND;
          const uint32_t par = ((uint32_t)(nbnd / Cfg::NBND) & 1u) ^ 1u;
          ok = __all_sync(0xffffffffu, mbar_wait(bar(Cfg::B_BNDEMPTY + bslot), par, wc));
          if (!ok) break;
          int* dst = reinterpret_cast<int*>(smem + Cfg::OFF_BND + bslot * Cfg::BND_BYTES);
          const int32_t* src = md.mask + ((size_t)bh_mask * p.Sk + j0) * md.ncols;
          stage_bounds(dst, src, 128, min(128, p.Sk - j0), md.ncols, lane);
          mbar_arrive(bar(Cfg::B_BNDFULL + bslot));
          ++nbnd;
        }
      }
      // a sub-tile without work never consumed its Q load: make sure it has landed
      if (ok && lane == 0) { mbar_wait(bar(Cfg::B_QFULL + 0), 0u, wc); if (!SPLITV) mbar_wait(bar(Cfg::B_QFULL + 1), 0u, wc); }
    } else if (warp == 9) {
      // =========================== UMMA issuer ===========================
      if (elect_one()) {
        constexpr uint32_t idesc_qk = make_idesc(IS_BF16, 128, 128, 0, 0);
        constexpr uint32_t idesc_pv = make_idesc(IS_BF16, 128, DVS, 0, 1);
        // P V starts on the first 96 keys of a tile while the softmax still computes the last 32 (B_PPART): the wait for a
        // tile's P, P V and the next scores is one dependent chain per sub-tile, and this takes up to 384 of its cycles out.
        // Dense 8192 x 2, 32 / 8 heads, d = 64: 1665 -> 1559 us; 32768 share-question, d = 128: 921 -> 907 us.  The split
        // variant, whose sub-tiles mostly take turns, lost 2 % by it and waits for the whole tile.
        constexpr int B_PFIRST = SPLIT ? Cfg::B_PFULL : Cfg::B_PPART;
        int npv[2] = {0, 0};
        bool q_ready[2] = {false, false};
        bool ok = true;
        // descriptors are built once; per MMA only a constant is added to the
        // 14-bit address field (all smem offsets are multiples of 16 bytes)
        const uint64_t dq0 = make_sdesc(sQ, 16, 1024);
        const uint64_t dk0 = make_sdesc(sKV, 16, 1024);
        const uint64_t dv0 = make_sdesc(sKV, Cfg::SUB, 1024);
        auto issue_qk = [&](auto sub, int i) {
            constexpr int s = decltype(sub)::value;   // compile-time: the per-sub-tile counters stay in registers
          const int k = 2 * i, slot = k % Cfg::NSTAGE;
          ok = ok && mbar_wait(bar(Cfg::B_KVFULL + slot), (uint32_t)(k / Cfg::NSTAGE) & 1u, wc);
          if (ok && !q_ready[s]) { ok = mbar_wait(bar(Cfg::B_QFULL + (SPLITV ? 0 : s)), 0u, wc); q_ready[s] = true; }
          if (!ok) return;
          tc_fence_after();
          const uint64_t da = dq0 + (uint64_t)(SPLITV ? 0 : s * (Cfg::Q_BYTES >> 4));
          const uint64_t db = dk0 + (uint64_t)(slot * (Cfg::SLOT_BYTES >> 4));
          const uint32_t dst = tmem + 128u * s;
          if constexpr (D == 128) umma_ss_x8<(Cfg::SUB >> 4), (Cfg::SUB >> 4)>(dst, da, db, idesc_qk, 0u);
          else if constexpr (D == 192) {
            // three 64-column sub-tiles of q / k: eight k-steps, then four more on top
            umma_ss_x8<(Cfg::SUB >> 4), (Cfg::SUB >> 4)>(dst, da, db, idesc_qk, 0u);
            umma_ss_x4(dst, da + (uint64_t)(2 * (Cfg::SUB >> 4)), db + (uint64_t)(2 * (Cfg::SUB >> 4)), idesc_qk, 1u);
          } else if constexpr (D == 256) {
            // four 64-column sub-tiles: eight k-steps over the first two, eight over the last two
            umma_ss_x8<(Cfg::SUB >> 4), (Cfg::SUB >> 4)>(dst, da, db, idesc_qk, 0u);
            umma_ss_x8<(Cfg::SUB >> 4), (Cfg::SUB >> 4)>(dst, da + (uint64_t)(2 * (Cfg::SUB >> 4)),
                                                         db + (uint64_t)(2 * (Cfg::SUB >> 4)), idesc_qk, 1u);
          } else umma_ss_x4(dst, da, db, idesc_qk, 0u);
          tc_commit(bar(Cfg::B_SFULL + s));
        };
        auto issue_pv = [&](auto sub, int i) {
            constexpr int s = decltype(sub)::value;
          const int k = 2 * i + 1, slot = k % Cfg::NSTAGE;
          ok = ok && mbar_wait(bar(Cfg::B_KVFULL + slot), (uint32_t)(k / Cfg::NSTAGE) & 1u, wc);
          ok = ok && mbar_wait(bar(B_PFIRST + s), (uint32_t)npv[s] & 1u, wc);
          if (!ok) return;
          tc_fence_after();
          // (d = 256: warpgroup s owns V columns [128 s, 128 s + 128): sub-tiles 2 s and 2 s + 1 of the V tile)
          const uint64_t db = dv0 + (uint64_t)(slot * (Cfg::SLOT_BYTES >> 4) + (SPLITV ? s * 2 * (Cfg::SUB >> 4) : 0));
          const uint32_t dst = tmem + 256u + 128u * s, src = tmem + 128u * s + 64u;
          const uint32_t acc0 = npv[s] > 0 ? 1u : 0u;
          if constexpr (SPLIT) {
            umma_ts_xn<8>(dst, src, db, idesc_pv, acc0);
          } else {
            umma_ts_xn<4>(dst, src, db, idesc_pv, acc0);
            umma_ts_x2(dst, src + 32u, db + (uint64_t)(4 * 128), idesc_pv);
            ok = mbar_wait(bar(Cfg::B_PFULL + s), (uint32_t)npv[s] & 1u, wc);
            if (!ok) return;
            tc_fence_after();
            umma_ts_x2(dst, src + 48u, db + (uint64_t)(6 * 128), idesc_pv);
          }
          tc_commit(bar(Cfg::B_ODONE + s));
          ++npv[s];
        };
        if (alt) {
          // tile i belongs to sub-tile i & 1; its scores are issued before the P V of the tile ahead of it
          auto pv_then_qk = [&](auto sub, int i) {
            issue_pv(sub, i);
            if (ok) tc_commit(bar(Cfg::B_KVEMPTY + (2 * i + 1) % Cfg::NSTAGE));
            if (ok && i + 2 < cnt) {
              issue_qk(sub, i + 2);
              if (ok) tc_commit(bar(Cfg::B_KVEMPTY + (2 * i + 4) % Cfg::NSTAGE));
            }
          };
          issue_qk(std::integral_constant<int, 0>{}, 0);
          if (ok) tc_commit(bar(Cfg::B_KVEMPTY + 0));
          if (ok && cnt > 1) {
            issue_qk(std::integral_constant<int, 1>{}, 1);
            if (ok) tc_commit(bar(Cfg::B_KVEMPTY + 2 % Cfg::NSTAGE));
          }
          for (int i = 0; i < cnt && ok; i += 2) {
            pv_then_qk(std::integral_constant<int, 0>{}, i);
            if (ok && i + 1 < cnt) pv_then_qk(std::integral_constant<int, 1>{}, i + 1);
          }
        } else if (cnt > 0) {
          const uint32_t e = list[0];
          if ((e >> 16) & 0xFu) issue_qk(std::integral_constant<int, 0>{}, 0);
          if ((e >> 20) & 0xFu) issue_qk(std::integral_constant<int, 1>{}, 0);
          if (ok) tc_commit(bar(Cfg::B_KVEMPTY + 0));
        }
        for (int i = 0; i < cnt && ok && !alt; ++i) {
          const uint32_t e = list[i];
          const uint32_t en = (i + 1 < cnt) ? list[i + 1] : 0u;
          // the sub-tile whose P is ready first goes first (sub-tile 0 when both or neither are)
          bool one_first = false;
          if (((e >> 16) & 0xFu) && ((e >> 20) & 0xFu))
            one_first = !mbar_try_wait(bar(B_PFIRST + 0), (uint32_t)npv[0] & 1u) &&
                        mbar_try_wait(bar(B_PFIRST + 1), (uint32_t)npv[1] & 1u);
          if (one_first) {
            issue_pv(std::integral_constant<int, 1>{}, i);
            if (ok && ((en >> 20) & 0xFu)) issue_qk(std::integral_constant<int, 1>{}, i + 1);
            if (ok) issue_pv(std::integral_constant<int, 0>{}, i);
            if (ok && ((en >> 16) & 0xFu)) issue_qk(std::integral_constant<int, 0>{}, i + 1);
          } else {
            if ((e >> 16) & 0xFu) issue_pv(std::integral_constant<int, 0>{}, i);
            if (ok && ((en >> 16) & 0xFu)) issue_qk(std::integral_constant<int, 0>{}, i + 1);
            if (ok && ((e >> 20) & 0xFu)) issue_pv(std::integral_constant<int, 1>{}, i);
            if (ok && ((en >> 20) & 0xFu)) issue_qk(std::integral_constant<int, 1>{}, i + 1);
          }
          if (!ok) break;
          tc_commit(bar(Cfg::B_KVEMPTY + (2 * i + 1) % Cfg::NSTAGE));
          if (i + 1 < cnt) tc_commit(bar(Cfg::B_KVEMPTY + (2 * i + 2) % Cfg::NSTAGE));
        }
      }
      __syncwarp();
    }
  }

  // =========================== teardown ===========================
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (tid == 0) FPROF(6);
  const bool aborted = misc[4] != 0;
  if (aborted) {
    // give copies and MMAs still in flight a bounded time to land before the
    // shared and tensor memory of this CTA are released
    const uint64_t t_end = global_timer_ns() + 200000ull;
    while (global_timer_ns() < t_end) __nanosleep(1000);
    if (tid == 0) atomicExch(&g_fwd_status, FM_ERR_TIMEOUT);
  }
  if (warp == 9) tmem_dealloc(tmem, 512);
}

// Merges the partial results of every query row: one warp per (batch, head, query), lane l owns columns
// [l DV / 32, (l + 1) DV / 32).  The partials were written a moment ago and are read from the L2.
template <int DV, bool IS_BF16>
__global__ void __launch_bounds__(256) fwd_combine_kernel(const AttnKParams p) {
  constexpr int PER = DV / 32;
  const int lane = threadIdx.x & 31;
  const int64_t row = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);       // (b * Hq + h) * Sq + i
  grid_dep_wait();
  if (row >= (int64_t)p.B * p.Hq * p.Sq) return;
  const int i = (int)(row % p.Sq), h = (int)(row / p.Sq % p.Hq), b = (int)(row / p.Sq / p.Hq);
  const int n_parts = p.n_split << p.alternate;                            // <= 32
  const float* lse = p.part_lse + row * n_parts;
  const float mine = lane < n_parts ? lse[lane] : neg_inf();
  float m = mine;
#pragma unroll
  for (int o = 16; o; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));   // (drops NaN; the weights keep it)
  if (m == neg_inf()) m = 0.f;
  const float w_mine = exp2f(mine - m);
  float l = w_mine;
#pragma unroll
  for (int o = 16; o; o >>= 1) l += __shfl_xor_sync(0xffffffffu, l, o);
  float acc[PER];
#pragma unroll
  for (int c = 0; c < PER; ++c) acc[c] = 0.f;
  const float* src = p.part_o + row * n_parts * DV + lane * PER;
  for (int s = 0; s < n_parts; ++s) {
    const float w = __shfl_sync(0xffffffffu, w_mine, s);
    if (__shfl_sync(0xffffffffu, mine, s) == neg_inf()) continue;         // (an empty part's O is not written)
    if constexpr (PER == 4) {
      const float4 v = *reinterpret_cast<const float4*>(src + s * DV);
      acc[0] += w * v.x; acc[1] += w * v.y; acc[2] += w * v.z; acc[3] += w * v.w;
    } else {
      const float2 v = *reinterpret_cast<const float2*>(src + s * DV);
      acc[0] += w * v.x; acc[1] += w * v.y;
    }
  }
  if (p.sink) l += exp2f(p.sink[h] * kLog2e - m);
  const float inv = l > 0.f ? 1.f / l : 0.f;
  if (lane == 0) p.lse[row] = l > 0.f ? (m + log2f(l)) * kLn2 : neg_inf();
  if (lane * PER < p.dv_dim) {
    uint32_t* out = reinterpret_cast<uint32_t*>(reinterpret_cast<uint16_t*>(p.o) + b * p.o_b + (int64_t)i * p.o_s + h * p.o_h + lane * PER);
#pragma unroll
    for (int c = 0; c < PER; c += 2) out[c / 2] = pack2<IS_BF16>(acc[c] * inv, acc[c + 1] * inv);
  }
}

// ---------------------------------------------------------------------------
// host
// ---------------------------------------------------------------------------
#ifdef FM_TRACE
extern "C" __attribute__((visibility("default"))) int fm_debug_fprof_read(long long* out) {
  return (int)cudaMemcpyFromSymbol(out, g_fprof, sizeof(long long) * 64 * 16);
}
#endif

namespace sm100 {

EncodeTiledFn get_encode_tiled() {
  static EncodeTiledFn fn = nullptr;
  static bool tried = false;
  if (!tried) {
    tried = true;
    void* ptr = nullptr;
    cudaDriverEntryPointQueryResult qres;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &qres) == cudaSuccess &&
        qres == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(ptr);
  }
  return fn;
}

int make_bshd_tmap(CUtensorMap* out, const void* base, int dtype, int B, int S, int H, int D, int64_t sb,
                   int64_t ss, int64_t sh, int box_rows, int box_cols, int box_heads) {
  EncodeTiledFn enc = get_encode_tiled();
  FM_REQUIRE(enc != nullptr, FM_ERR_CUDA, "cuTensorMapEncodeTiled is not available from the driver");
  // a dimension of one element may carry any stride, 0 included: it gets the dense one
  const int64_t th = H > 1 ? sh : D, ts = S > 1 ? ss : th * H, tb = B > 1 ? sb : ts * S;
  FM_REQUIRE(th > 0 && ts > 0 && tb > 0, FM_ERR_INVALID_ARGUMENT,
             "tensor map: strides must be positive (batch %lld, row %lld, head %lld)", (long long)tb, (long long)ts, (long long)th);
  const cuuint64_t dims[4] = {(cuuint64_t)D, (cuuint64_t)H, (cuuint64_t)S, (cuuint64_t)B};
  const cuuint64_t strides[3] = {(cuuint64_t)th * 2, (cuuint64_t)ts * 2, (cuuint64_t)tb * 2};
  const cuuint32_t box[4] = {(cuuint32_t)box_cols, (cuuint32_t)box_heads, (cuuint32_t)box_rows, 1};
  const cuuint32_t estr[4] = {1, 1, 1, 1};
  const CUresult r = enc(out, dtype == FM_DTYPE_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16,
                         4, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                         box_cols == 32 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                         CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  FM_REQUIRE(r == CUDA_SUCCESS, FM_ERR_CUDA, "cuTensorMapEncodeTiled failed with CUresult %d", (int)r);
  return FM_OK;
}

}  // namespace sm100

// One CTA waits on an mbarrier that nothing ever arrives on, with a wall-clock
// budget: exercises the bounded wait and the status word without touching the
// tensor pipe.  The kernel returns normally; the context stays usable.
__global__ void bounded_wait_selftest_kernel(uint64_t budget_ns) {
  __shared__ __align__(8) uint64_t never;
  __shared__ int abort_flag;
  if (threadIdx.x == 0) {
    abort_flag = 0;
    mbar_init(smem_u32(&never), 1);
    fence_mbar_init();
  }
  __syncthreads();
  WaitCtx wc{&abort_flag, global_timer_ns() + budget_ns};
  const bool ok = mbar_wait(smem_u32(&never), 0u, wc);
  __syncthreads();
  if (threadIdx.x == 0 && !ok) atomicExch(&g_fwd_status, FM_ERR_TIMEOUT);
}

int bounded_wait_selftest_launch(uint64_t budget_ns, cudaStream_t s) {
  bounded_wait_selftest_kernel<<<1, 64, 0, s>>>(budget_ns);
  count_launches(1);
  FM_CUDA_TRY(cudaGetLastError());
  return FM_OK;
}

// Split plan of a call (SPLIT above): heads packed per query, parts, bytes of partial results.
//
// The plan is for calls without a mask tensor (the tiles a mask leaves are not known to the host).  Packing the heads
// of a group, dealing K tiles to several CTAs, and (where all rows of a block fit one sub-tile: p.alternate) letting
// both sub-tiles take the tiles of a CTA in turn are each taken where an estimate of the launch says that it pays.
// The estimate, in microseconds, is waves x (entry and exit + tiles per part + fp32 partial results of a part's rows)
// + the merge, fitted to 2000 launches of 1 to 300 rows against 1 to 200 tiles on 1 to 1200 CTAs:
//   alternating, d = 128, 148 CTAs of 64 tiles   1 row 113 -> 98 us, 128 rows 138 -> 117
//                         1200 CTAs of 2 tiles   1 row  69 -> 63 us, 128 rows  85 -> 178: not taken
//                         600 CTAs of 8 tiles   64 rows 98 -> 106 us: not taken
//   keys in two parts, 64 packed CTAs of 128 tiles (512 queries against 16384 keys, 32 / 8 heads, d = 128): 231 -> 153 us
//   packed heads, 3 x 700 queries (16 / 4 heads, 132 CTAs for 144, both one wave): 80 -> 85 us: not taken
struct FwdSplitPlan { int pack_log2, n_split; bool alternate; size_t bytes; };
static FwdSplitPlan fwd_split_plan(const fm_attn_args* a) {
  FwdSplitPlan pl{0, 1, false, 0};
  if (a->ncols != 0 || a->d > 128 || a->dv > 128) return pl;
  const int G = a->Hq / a->Hkv, n_sm = sm_count(), tiles = (a->Sk + 127) / 128;
  const bool small = a->d <= 64 && a->dv <= 64;
  const double entry = small ? 4.9 : 5.7, in_turn = small ? 0.59 : 0.68, partial = small ? 4.5 : 10.0, merge = small ? 3.8 : 2.2;
  auto blocks = [&](int64_t rows) { return (rows + 255) / 256; };
  auto tile = [&](int64_t rows) {                                   // one sub-tile of a CTA's two, or both
    const double one = small ? 1.54 : 1.84, both = small ? 1.95 : 2.0;
    const int64_t nb = blocks(rows);
    return ((nb - 1) * both + (rows - 256 * (nb - 1) <= 128 ? one : both)) / nb;
  };
  if (blocks(a->Sq) * a->Hq * a->B >= 4 * n_sm && blocks(a->Sq) > 1) return pl;
  double best = 1e30;
  auto consider = [&](int pack_log2, double handicap) {
    const int64_t rows = (int64_t)a->Sq << pack_log2, units = blocks(rows) * (a->Hq >> pack_log2) * a->B;
    const double share = std::min<int64_t>(rows, 128) / 128.0;      // of a sub-tile's rows that have a partial result
    for (int s = 1; s <= 32 && s <= tiles && (s == 1 || units < n_sm); ++s) {
      const int n = (tiles + s - 1) / s;                            // tiles of a CTA
      for (int alt = 0; alt <= (rows <= 128 && n >= 2 && s <= 16 ? 1 : 0); ++alt) {
        const bool parts = alt || s > 1;
        const double cost = handicap * (((units * s + n_sm - 1) / n_sm) * (entry + (alt ? in_turn : 1.0) * tile(rows) * n +
                                        (parts ? partial * share : 0.0)) + (parts ? merge : 0.0));
        if (cost < best) { best = cost; pl.pack_log2 = pack_log2; pl.n_split = s; pl.alternate = alt; }
      }
    }
  };
  consider(0, 1.0);
  if (G > 1 && (G & (G - 1)) == 0 && G <= 128 && blocks((int64_t)a->Sq * G) < blocks(a->Sq) * G) {
    int lg = 0;
    while ((1 << lg) < G) ++lg;
    // (few blocks saved: the packed kernel's own pace counts)
    consider(lg, 4 * blocks((int64_t)a->Sq * G) > 3 * blocks(a->Sq) * G ? 1.05 : 1.0);
  }
  const size_t parts = (size_t)pl.n_split << pl.alternate;
  if (parts > 1) pl.bytes = (size_t)a->B * a->Hq * a->Sq * parts * ((small ? 64 : 128) + 1) * sizeof(float);
  return pl;
}

size_t fwd_sm100_workspace_bytes(const fm_attn_args* a) { return fwd_split_plan(a).bytes; }

template <int D, int DV, bool IS_BF16, int BLOCK_SCORE, bool BLOCK_BOS, bool SPLIT = false>
static int launch_fwd_sm100(const AttnKParams& p, const fm_attn_args* a, cudaStream_t s) {
  using Cfg = FwdSm100Cfg<D, DV>;
  FM_REQUIRE((a->Sk + 127) / 128 <= Cfg::LIST_MAX, FM_ERR_UNSUPPORTED,
             "forward: Sk=%d exceeds the %d keys this kernel variant indexes", a->Sk, Cfg::LIST_MAX * 128);
  CUtensorMap tq, tk, tv;
  int rc;
  if ((rc = make_bshd_tmap(&tq, a->q, a->dtype, a->B, a->Sq, a->Hq, a->d, a->q_stride[0], a->q_stride[1], a->q_stride[2], 128 >> p.pack_log2, 64, 1 << p.pack_log2))) return rc;
  if ((rc = make_bshd_tmap(&tk, a->k, a->dtype, a->B, a->Sk, a->Hkv, a->d, a->k_stride[0], a->k_stride[1], a->k_stride[2], 128))) return rc;
  if ((rc = make_bshd_tmap(&tv, a->v, a->dtype, a->B, a->Sk, a->Hkv, a->dv, a->v_stride[0], a->v_stride[1], a->v_stride[2], 128))) return rc;
  auto kern = fwd_sm100_kernel<D, DV, IS_BF16, BLOCK_SCORE, BLOCK_BOS, SPLIT>;
  constexpr int smem_bytes = BLOCK_BOS ? Cfg::SMEM_BS : Cfg::SMEM;
  FM_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_bytes));
  dim3 grid(((p.Sq << p.pack_log2) + Cfg::ROWS - 1) / Cfg::ROWS, p.Hq >> p.pack_log2, p.B);
  if (SPLIT) grid.x *= p.n_split;
  kern<<<grid, Cfg::NTHREADS, smem_bytes, s>>>(tq, tk, tv, p);
  count_launches(1);
  FM_CUDA_TRY(cudaGetLastError());
  if (SPLIT && (p.n_split << p.alternate) > 1) {
    FM_CUDA_TRY(launch_dependent(fwd_combine_kernel<DV, IS_BF16>, dim3((unsigned)(((int64_t)p.B * p.Hq * p.Sq + 7) / 8)), dim3(256), 0, s, p));
    count_launches(1);
  }
  return FM_OK;
}

int fwd_sm100_launch(const AttnKParams& p_in, const fm_attn_args* a, cudaStream_t s) {
  AttnKParams p = p_in;
  const bool bf = a->dtype == FM_DTYPE_BF16;
  const bool small = a->d <= 64 && a->dv <= 64;
  if (!p.block_logit) {
    FwdSplitPlan pl = fwd_split_plan(a);
    if (pl.bytes && (!a->workspace || a->workspace_bytes < pl.bytes || ((uintptr_t)a->workspace & 15))) { pl.n_split = 1; pl.alternate = false; }
    p.pack_log2 = pl.pack_log2;
    p.n_split = pl.n_split;
    p.alternate = pl.alternate;
    const int parts = pl.n_split << pl.alternate;
    if (parts > 1) {
      p.part_o = reinterpret_cast<float*>(a->workspace);
      p.part_lse = p.part_o + (size_t)p.B * p.Hq * p.Sq * parts * (small ? 64 : 128);
    }
    if (parts > 1 || pl.pack_log2) {
      if (small) return bf ? launch_fwd_sm100<64, 64, true, 0, false, true>(p, a, s) : launch_fwd_sm100<64, 64, false, 0, false, true>(p, a, s);
      return bf ? launch_fwd_sm100<128, 128, true, 0, false, true>(p, a, s) : launch_fwd_sm100<128, 128, false, 0, false, true>(p, a, s);
    }
  }
#define FM_FWD_DISPATCH(BSZ, BOS)                                                                         \
  do {                                                                                                    \
    if (a->d == 256)                                                                                      \
      return bf ? launch_fwd_sm100<256, 256, true, BSZ, BOS>(p, a, s) : launch_fwd_sm100<256, 256, false, BSZ, BOS>(p, a, s); \
    if (a->d == 192)                                                                                      \
      return bf ? launch_fwd_sm100<192, 128, true, BSZ, BOS>(p, a, s) : launch_fwd_sm100<192, 128, false, BSZ, BOS>(p, a, s); \
    if (small)                                                                                            \
      return bf ? launch_fwd_sm100<64, 64, true, BSZ, BOS>(p, a, s) : launch_fwd_sm100<64, 64, false, BSZ, BOS>(p, a, s); \
    return bf ? launch_fwd_sm100<128, 128, true, BSZ, BOS>(p, a, s) : launch_fwd_sm100<128, 128, false, BSZ, BOS>(p, a, s); \
  } while (0)
  if (p.block_logit && p.block_bos) {
    if (p.block_log2 == 5) FM_FWD_DISPATCH(32, true);
    if (p.block_log2 == 6) FM_FWD_DISPATCH(64, true);
    FM_FWD_DISPATCH(128, true);
  }
  if (p.block_logit) {
    if (p.block_log2 == 5) FM_FWD_DISPATCH(32, false);
    if (p.block_log2 == 6) FM_FWD_DISPATCH(64, false);
    FM_FWD_DISPATCH(128, false);
  }
  FM_FWD_DISPATCH(0, false);
#undef FM_FWD_DISPATCH
}

int fwd_sm100_status(int* out, bool reset) {
  int v = 0;
  FM_CUDA_TRY(cudaMemcpyFromSymbol(&v, g_fwd_status, sizeof(int)));
  if (reset && v != 0) {
    const int z = 0;
    FM_CUDA_TRY(cudaMemcpyToSymbol(g_fwd_status, &z, sizeof(int)));
  }
  *out = v;
  return FM_OK;
}

}  // namespace fm
