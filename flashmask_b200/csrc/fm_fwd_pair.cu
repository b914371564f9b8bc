// Forward attention for head dims 256/256, 512/512 and 576/512 on CTA pairs (tcgen05, cta_group::2).
//
// Two CTAs of a cluster own 256 query rows of one (batch, q head), 128 each, and one 256-column slice of V / O
// (dv = 512: two slices, two pairs).  Every MMA has M = 256: the pair shares the K / V tile, each CTA loads one
// half of it (64 of a tile's 128 keys for S = Q K^T, 128 of the slice's 256 columns for O += P V).
//
// Why this split.  The accumulators decide: O of 128 rows x 256 columns takes 256 of the 512 tensor-memory
// columns, two score buffers the other 256, so S of tile i+1 is computed while tile i is in the softmax.  At
// dv = 512 a second slice recomputes S (576 of 576 + 256 columns of work per tile): O of 128 rows x 512 columns
// would fill the tensor memory alone.  A single CTA would read 64 B/clk of K / V at d = 256 from the L2, which
// delivers 68 B/clk per SM to all SMs together; the pair reads 32.
//
// Bound: the tensor pipe (2048 cycles per 128 keys and pair at d = 256, 3328 at 576; softmax 1024 exp2 cycles).
// Measured at S = 16384, 16 heads, causal: 256/256 2.67 ms (one CTA, S computed twice) -> 1.47 ms = 1500 TFLOP/s;
// 576/512 29.9 ms (warp MMA) -> 4.56 ms = 1025 TFLOP/s of the mathematics, 1560 executed.
//
// Warp roles of each CTA (384 threads): 0-3 / 4-7 softmax warpgroups 0 / 1: thread r of a warpgroup owns row r
// and 64 of the tile's 128 keys, the pair of threads exchanges the row maximum through shared memory; 8 TMA
// producer (and column bounds of partial tiles); 9 UMMA issuer (the leading CTA's works for both), owns the
// tensor memory; 10 tile list; 11 idle.
// TMEM columns: S / P of even tiles [0,128), of odd tiles [128,256), O [256,512).  P (bf16, 64 columns)
// overlays the first half of its S.  Barriers whose arrivals come from both CTAs live in the leader.
// All waits are bounded.
#include "fm_attn_params.cuh"
#include "fm_sm100_pair.cuh"

namespace fm {

using namespace sm100;

__device__ int g_fwd_pair_status = 0;

// BS: the block-score variants, which keep their accumulators where the others have one more ring slot (512, 576).
template <int D, bool BS = false>
struct FwdPairCfg {
  static constexpr int SLICES = D == 256 ? 1 : 2;       // 256-column slices of V / O
  static constexpr int NTHREADS = 384, LIST_MAX = 2048, NBND = 2;
  static constexpr int SUB128 = 128 * 128, SUB64 = 64 * 128;   // 128- / 64-row x 64-column sub-tiles (bytes)
  static constexpr int Q_BYTES = 128 * D * 2;
  static constexpr int SLOT_BYTES = 2 * SUB64;          // 64 keys x 128 columns of K, or 64 keys x 128 columns of V
  static constexpr int NSTAGE = D == 256 ? 8 : (D == 512 ? 5 : 4) - (BS ? 1 : 0);
  static constexpr int KSLOTS = (D + 127) / 128;        // ring slots of a K tile (the last one half full at D = 576)
  static constexpr int OFF_Q = 0;
  static constexpr int OFF_KV = OFF_Q + Q_BYTES;
  static constexpr int OFF_BND = OFF_KV + NSTAGE * SLOT_BYTES;
  static constexpr int BND_BYTES = 128 * 4 * 4;
  static constexpr int OFF_LIST = OFF_BND + NBND * BND_BYTES;
  static constexpr int OFF_EX = OFF_LIST + LIST_MAX * 4;       // row maxima exchanged between the warpgroups
  static constexpr int OFF_BAR = OFF_EX + 2 * 2 * 128 * 4;
  static constexpr int OFF_MISC = OFF_BAR + 32 * 8;
  static constexpr int SMEM = OFF_MISC + 64 + 1024;
  // block-score variant only: maxima handed over per tile parity, 16 block accumulators per row
  static constexpr int OFF_BSX = OFF_MISC + 64, OFF_BSA = OFF_BSX + 2 * 3 * 128 * 4;
  static constexpr int SMEM_BS = OFF_BSA + 16 * 128 * 4 + 1024;
  static_assert(!BS || SMEM_BS <= 227 * 1024, "shared memory of the block-score variant");
  static constexpr int B_Q = 0, B_KVFULL = 1, B_KVEMPTY = B_KVFULL + NSTAGE, B_SFULL = B_KVEMPTY + NSTAGE,
                       B_PFULL = B_SFULL + 2, B_ODONE = B_PFULL + 2, B_BNDFULL = B_ODONE + 2,
                       B_BNDEMPTY = B_BNDFULL + NBND, B_COUNT = B_BNDEMPTY + NBND;
  static_assert(D == 256 || D == 512 || D == 576, "head-dim variants");
  static_assert(B_COUNT <= 32, "barrier storage");
  static_assert(SMEM > 120 * 1024 && SMEM <= 227 * 1024, "one CTA per SM (512 TMEM columns)");
  static_assert(OFF_KV % 1024 == 0 && 128 * 512 <= Q_BYTES, "aligned tiles; the Q tile stages the output");
  static_assert(LIST_MAX * 8 * 4 <= Q_BYTES, "the Q tile's place stages the reductions of the list build");
};

// Maxima over the blocks (of BS key columns) that 64 masked scores of a row touch: column j of the 64 lies in
// block (rel + j) >> log2(BS), `rel` being the first of them relative to the start of the row's document.
// part[i] belongs to block (rel >> log2(BS)) + i; returns the maximum of all.
template <int BS> struct BlockParts { static constexpr int N = 64 / BS + (BS == 128 ? 2 : 1); };
template <int BS, bool STRADDLE>
__device__ __forceinline__ float half_block_scores(const uint32_t* sr, int rel, float* part) {
  constexpr int N = BlockParts<BS>::N;
  const int t = STRADDLE ? BS - (rel & (BS - 1)) : BS;     // columns of a block at or past t belong to the next one
#pragma unroll
  for (int i = 0; i < N; ++i) part[i] = __int_as_float(0xff800000);
#pragma unroll
  for (int j = 0; j < 64; ++j) {
    const float v = __uint_as_float(sr[j]);
    if (STRADDLE && (j % BS) >= t) part[j / BS + 1] = fmaxf(part[j / BS + 1], v);
    else part[j / BS] = fmaxf(part[j / BS], v);
  }
  float all = part[0];
#pragma unroll
  for (int i = 1; i < N; ++i) all = fmaxf(all, part[i]);
  return all;
}

// BLOCK_SCORE: 0, or the block size of the block-score side output; BLOCK_BOS: document starts are given, so a block
// may straddle two tiles.  The threads of warpgroup 0 (of the first slice's pair) own the output rows; warpgroup 1
// hands them the maxima of its 64 columns through shared memory together with the row maximum.
template <int D, bool IS_BF16, int BLOCK_SCORE = 0, bool BLOCK_BOS = false>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(384, 1)
fwd_pair_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                const __grid_constant__ CUtensorMap tm_v, const AttnKParams p) {
  using Cfg = FwdPairCfg<D, BLOCK_SCORE != 0>;
  extern __shared__ uint8_t smem_raw[];
  // (the dynamic shared memory starts at the same address in both CTAs, so the aligned base is the same too)
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  const uint32_t sbase = smem_u32(smem);
  const uint32_t sQ = sbase + Cfg::OFF_Q, sKV = sbase + Cfg::OFF_KV;
  uint32_t* list = reinterpret_cast<uint32_t*>(smem + Cfg::OFF_LIST);
  const uint32_t bars = sbase + Cfg::OFF_BAR;
  volatile int* misc = reinterpret_cast<volatile int*>(smem + Cfg::OFF_MISC);   // [0] tmem, [1] cnt, [4] abort
  auto bar = [&](int i) { return bars + 8u * (uint32_t)i; };

  const int tid = threadIdx.x;
  const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
  const int lane = tid & 31;
  const int rank = (int)cluster_ctarank();
  if (warp == 8 && lane == 0) { tma_prefetch_desc(&tm_q); tma_prefetch_desc(&tm_k); tma_prefetch_desc(&tm_v); }
  // heaviest row blocks first; the slices of one (row block, head) are neighbours
  const int t = (p.Sq + 255) / 256 - 1 - (int)(blockIdx.x >> 1);
  const int hq = blockIdx.y / Cfg::SLICES, slice = blockIdx.y % Cfg::SLICES, b = blockIdx.z;
  const int hk = hq / (p.Hq / p.Hkv);
  const MaskDesc& md = p.md;
  const int bh_mask = md.ncols ? ((md.mask_B == 1 ? 0 : b) * md.Hm + hq / (p.Hq / md.Hm)) : 0;
  const int ms = t * 256;
  const int off = p.Sk - p.Sq;
  const int nb = (p.Sk + 127) / 128;
  const int n_hi = md.causal ? max(0, min(nb, (min(ms + 256, p.Sq) + off + 127) / 128)) : nb;

  if (tid == 0) misc[4] = 0;
  if (warp == 8 && lane == 0) {
    mbar_init(bar(Cfg::B_Q), 1);
    for (int i = 0; i < Cfg::NSTAGE; ++i) { mbar_init(bar(Cfg::B_KVFULL + i), 1); mbar_init(bar(Cfg::B_KVEMPTY + i), 1); }
    for (int s = 0; s < 2; ++s) { mbar_init(bar(Cfg::B_SFULL + s), 1); mbar_init(bar(Cfg::B_PFULL + s), 16); }
    for (int s = 0; s < 2; ++s) mbar_init(bar(Cfg::B_ODONE + s), 1);
    for (int i = 0; i < Cfg::NBND; ++i) { mbar_init(bar(Cfg::B_BNDFULL + i), 32); mbar_init(bar(Cfg::B_BNDEMPTY + i), 256); }
    fence_mbar_init();
  }
  if (warp == 10) {
    // surviving K tiles, right to left: those that either CTA's rows see, with the flags of both
    int cnt = 0;
    const MaskDesc mst = stage_minmax(md, bh_mask, 0, n_hi, reinterpret_cast<int32_t*>(smem + Cfg::OFF_Q),
                                      Cfg::LIST_MAX, lane);
    for (int base = n_hi - 1; base >= 0; base -= 32) {
      const int n = base - lane;
      uint32_t f0 = 0, f1 = 0;
      if (n >= 0) {
        f0 = tile_flags(mst, 0, n, ms, min(ms + 128, p.Sq), 128);
        if (ms + 128 < p.Sq) f1 = tile_flags(mst, 0, n, ms + 128, min(ms + 256, p.Sq), 128);
      }
      const bool keep = (f0 | f1) != 0;
      const uint32_t bal = __ballot_sync(0xffffffffu, keep);
      const int pos = cnt + __popc(bal & ((1u << lane) - 1u));
      if (keep && pos < Cfg::LIST_MAX) list[pos] = (uint32_t)n | (f0 << 16) | (f1 << 20);
      cnt += __popc(bal);
    }
    if (lane == 0) misc[1] = min(cnt, Cfg::LIST_MAX);
    fence_proxy_async_smem();   // the staging area is handed to the TMA loads of Q
  }
  if (warp == 9) {
    tmem2_alloc(sbase + Cfg::OFF_MISC, 512);
    tmem2_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();            // both CTAs' barriers exist before either is signalled from outside
  tc_fence_after();
  const uint32_t tmem = (uint32_t)misc[0];
  const int cnt = misc[1];
  WaitCtx wc{misc + 4, global_timer_ns() + 2000000000ull};
  if (cnt == 0) {
    // nothing visible for these rows (both CTAs see the same list): O = 0, LSE = -inf or the sink
    uint16_t* go = reinterpret_cast<uint16_t*>(p.o) + b * p.o_b + hq * p.o_h;
    for (int x = tid; x < 128 * 32; x += Cfg::NTHREADS) {
      const int row = ms + 128 * rank + x / 32, col = 256 * slice + (x % 32) * 8;
      if (row < p.Sq) *reinterpret_cast<uint4*>(go + (int64_t)row * p.o_s + col) = make_uint4(0u, 0u, 0u, 0u);
    }
    const float empty_lse = p.sink ? p.sink[hq] : __int_as_float(0xff800000);
    if (slice == 0 && tid < 128 && ms + 128 * rank + tid < p.Sq)
      p.lse[((int64_t)b * p.Hq + hq) * p.Sq + ms + 128 * rank + tid] = empty_lse;
    __syncwarp();
    cluster_sync_all();
    if (warp == 9) tmem2_dealloc(tmem, 512);
    return;
  }

  if (warp < 8) {
    // =========================== softmax warpgroups ===========================
    setmaxnreg_inc<208>();
    const int w = warp >> 2;                   // keys [64 w, 64 w + 64) of every tile
    const int r = tid & 127;                   // row inside the CTA == TMEM lane
    const int row = ms + 128 * rank + r;
    const uint32_t lane_field = (uint32_t)((warp & 3) * 32) << 16;
    const uint32_t tO = tmem + lane_field + 256u + 128u * w;    // the O columns this warpgroup rescales and stores
    float* ex = reinterpret_cast<float*>(smem + Cfg::OFF_EX);   // [tile parity][warpgroup][row]
    const uint32_t pfull0 = map_to_rank(bar(Cfg::B_PFULL), 0);
    const float scale_log2 = p.scale_log2;
    const uint32_t NEG = 0xff800000u;
    const float ninf = __int_as_float(0xff800000);
    // How far (log2) a row's maximum may grow before O and the sum are rescaled to it.  At 512 and 576 / 512 every time it
    // grows: the largest weights then lie just below 1, where 16 bits round least, as in the warp-MMA kernel.  Error of O
    // against 64 bits, 2048 x 2048 causal, 576 / 512, bf16: warp-MMA 2.09e-3, 8 here 2.16e-3, 0 here 2.10e-3; 16384 x
    // 16384 4.46 ms either way (the rescale hides behind the 18 k-steps of the next scores), 512 / 512 3.97 -> 4.20 ms.
    // At 256 the kernels have always rescaled past 2^8.
    constexpr float LAZY = D == 256 ? 8.f : 0.f;
    float m_run = ninf, l_run = 0.f;
    int nbnd = 0;
    bool ok = true;
    // block scores: as in the one-CTA kernel, blocks that lie inside one tile are stored straight from registers,
    // straddling ones gathered in shared memory (two groups of eight consecutive blocks of the row) and merged
    // into the output once no later tile (to the left) can touch their group
    constexpr int BSZ = BLOCK_SCORE ? BLOCK_SCORE : 128, NPART = BlockParts<BSZ>::N;
    constexpr int BS_LOG2 = BSZ == 32 ? 5 : (BSZ == 64 ? 6 : 7);
    float* bs_dst = nullptr;
    float* bs_acc = reinterpret_cast<float*>(smem + Cfg::OFF_BSA) + r;
    int bs_bos = 0, bs_pend_lo = INT_MAX, bs_pend_hi = -1;    // pending groups [lo, hi]; lo > hi: none
    bool bs_vec = false;
    if constexpr (BLOCK_SCORE != 0) {
      if (row < p.Sq) {
        if (w == 0 && slice == 0) bs_dst = p.block_logit + (((int64_t)b * p.Hq + hq) * p.Sq + row) * p.block_ld;
        if constexpr (BLOCK_BOS) bs_bos = p.block_bos[(int64_t)b * p.Sq + row];
      }
      if constexpr (BLOCK_BOS) {
        bs_vec = (reinterpret_cast<uintptr_t>(bs_dst) & 15) == 0;
        if (w == 0) {
#pragma unroll
          for (int c = 0; c < 16; ++c) bs_acc[c * 128] = ninf;
        }
      }
    }
    for (int i = 0; i < cnt; ++i) {
      const uint32_t e = list[i];
      const uint32_t flags = (e >> (16 + 4 * rank)) & 0xFu;
      const bool any_bounds = (((e >> 16) | (e >> 20)) & FM_TF_BOUNDS) != 0;
      const int bslot = nbnd % Cfg::NBND;
      // a wait that gave up does not leave the loop by itself: the warpgroups meet in the barrier of the tile
      if (any_bounds && ok)
        ok = __all_sync(0xffffffffu, mbar_wait(bar(Cfg::B_BNDFULL + bslot), (uint32_t)(nbnd / Cfg::NBND) & 1u, wc));
      if (ok) ok = __all_sync(0xffffffffu, mbar_wait(bar(Cfg::B_SFULL + (i & 1)), (uint32_t)(i >> 1) & 1u, wc));
      tc_fence_after();
      const uint32_t tS = tmem + lane_field + 128u * (uint32_t)(i & 1);
      uint32_t pk[32];
      if (!flags) {
        // only the other CTA's rows see this tile
        ok = group_all(ok, 1, 256);
        if (!ok) break;
#pragma unroll
        for (int j = 0; j < 32; ++j) pk[j] = 0u;
      } else {
        uint32_t sr[64];                   // (after a wait that gave up: whatever the scores hold, unused)
        tmem_ld32(tS + 64u * w, sr); tmem_ld32(tS + 64u * w + 32u, sr + 32);
        tc_wait_ld();
        if (flags & FM_TF_BOUNDS) {
          const int4* bp = reinterpret_cast<const int4*>(smem + Cfg::OFF_BND + bslot * Cfg::BND_BYTES) + 16 * md.ncols * w;
          if (md.ncols == 1) {
#pragma unroll
            for (int j = 0; j < 16; ++j) {
              const int4 v = bp[j];
              if (row >= v.x) sr[4 * j] = NEG;
              if (row >= v.y) sr[4 * j + 1] = NEG;
              if (row >= v.z) sr[4 * j + 2] = NEG;
              if (row >= v.w) sr[4 * j + 3] = NEG;
            }
          } else if (md.ncols == 2 && md.causal) {
#pragma unroll
            for (int j = 0; j < 32; ++j) {
              const int4 v = bp[j];
              if (row >= v.x && row < v.y) sr[2 * j] = NEG;
              if (row >= v.z && row < v.w) sr[2 * j + 1] = NEG;
            }
          } else if (md.ncols == 2) {
#pragma unroll
            for (int j = 0; j < 32; ++j) {
              const int4 v = bp[j];
              if (row >= v.x || row < v.y) sr[2 * j] = NEG;
              if (row >= v.z || row < v.w) sr[2 * j + 1] = NEG;
            }
          } else {
#pragma unroll
            for (int j = 0; j < 64; ++j) {
              const int4 v = bp[j];
              if ((row >= v.x && row < v.y) || (row >= v.z && row < v.w)) sr[j] = NEG;
            }
          }
        }
        if (flags & (FM_TF_CAUSAL | FM_TF_RAGGED)) {
          const int j0 = (int)(e & 0xFFFFu) * 128 + 64 * w;
          int jmax = p.Sk - 1 - j0;                      // last valid key column of this half tile
          if (md.causal) jmax = min(jmax, row + off - j0);
#pragma unroll
          for (int j = 0; j < 64; ++j)
            if (j > jmax) sr[j] = NEG;
        }
        float mx;
        float part[NPART];
        const int bs_rel0 = (int)(e & 0xFFFFu) * 128 - bs_bos;      // first column of the tile inside the document
        float* bsx = reinterpret_cast<float*>(smem + Cfg::OFF_BSX) + (i & 1) * 3 * 128 + r;
        if constexpr (BLOCK_SCORE != 0) {
          mx = half_block_scores<BSZ, BLOCK_BOS>(sr, bs_rel0 + 64 * w, part);
          if (w == 1) {
#pragma unroll
            for (int c = 0; c < NPART; ++c) bsx[c * 128] = part[c];
          }
        } else {
          float mx0 = ninf, mx1 = ninf, mx2 = ninf, mx3 = ninf;
#pragma unroll
          for (int j = 0; j < 64; j += 8) {
            mx0 = fmax3(mx0, __uint_as_float(sr[j]), __uint_as_float(sr[j + 1]));
            mx1 = fmax3(mx1, __uint_as_float(sr[j + 2]), __uint_as_float(sr[j + 3]));
            mx2 = fmax3(mx2, __uint_as_float(sr[j + 4]), __uint_as_float(sr[j + 5]));
            mx3 = fmax3(mx3, __uint_as_float(sr[j + 6]), __uint_as_float(sr[j + 7]));
          }
          mx = fmaxf(fmaxf(mx0, mx1), fmaxf(mx2, mx3));
        }
        float* exi = ex + (i & 1) * 256;
        exi[128 * w + r] = mx;
        // both halves of the row are in registers and their maxima in `ex`
        ok = group_all(ok, 1, 256);
        if (!ok) break;
        mx = fmaxf(mx, exi[128 * (w ^ 1) + r]);
        if constexpr (BLOCK_SCORE != 0) {
          if (bs_dst) {
            if (!BLOCK_BOS || (bs_rel0 & (BSZ - 1)) == 0) {
              // 128 / BSZ whole blocks, this tile's alone
              const int base = bs_rel0 >> BS_LOG2;
#pragma unroll
              for (int c = 0; c < 128 / BSZ; ++c) {
                float v;
                if constexpr (BSZ == 128) v = mx;
                else v = c < 64 / BSZ ? part[c] : bsx[(c - 64 / BSZ) * 128];
                if (base + c >= 0 && base + c < p.block_cols) bs_dst[base + c] = v * p.scale;
              }
            } else {
              const int base = bs_rel0 >> BS_LOG2, top = base + (128 >> BS_LOG2);     // blocks this tile can touch
              const int lo_rb = max(base, 0), hi_rb = min(top, p.block_cols - 1);
              if (lo_rb <= hi_rb) {
                const int g_top = hi_rb >> 3, g_bot = lo_rb >> 3;
                for (int g = bs_pend_hi; g >= max(bs_pend_lo, g_top + 1); --g)
                  block_flush<128>(bs_dst, bs_acc, g, bs_vec, p.block_cols);
                bs_pend_hi = min(bs_pend_hi, g_top);
                if (bs_pend_lo > bs_pend_hi) { bs_pend_hi = g_top; bs_pend_lo = g_bot; }
                else bs_pend_lo = min(bs_pend_lo, g_bot);
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                  const int hb = (bs_rel0 + 64 * h) >> BS_LOG2;
#pragma unroll
                  for (int c = 0; c < NPART; ++c) {
                    const int rb = hb + c;
                    if (rb >= 0 && rb < p.block_cols) {
                      float* a = bs_acc + (rb & 15) * 128;
                      *a = fmaxf(*a, (h ? bsx[c * 128] : part[c]) * p.scale);
                    }
                  }
                }
              }
            }
          }
        }
        const float m_new = fmaxf(m_run, mx * scale_log2);
        const bool need = (m_new - m_run) > LAZY;        // the same decision in both warpgroups
        float alpha = 1.f;
        if (need) {
          alpha = fast_exp2(m_run - m_new);
          m_run = m_new;
          l_run *= alpha;
        }
        if (__any_sync(0xffffffffu, need) && i > 0) {
          ok = __all_sync(0xffffffffu, mbar_wait(bar(Cfg::B_ODONE + ((i - 1) & 1)), (uint32_t)((i - 1) >> 1) & 1u, wc));
          tc_fence_after();
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            uint32_t orr[32];
            tmem_ld32(tO + 32 * c, orr);
            tc_wait_ld();
#pragma unroll
            for (int j = 0; j < 32; ++j) orr[j] = __float_as_uint(__uint_as_float(orr[j]) * alpha);
            tmem_st32(tO + 32 * c, orr);
          }
        }
        const float m_use = (m_run == ninf) ? 0.f : m_run;
        float ls0 = 0.f, ls1 = 0.f;
#pragma unroll
        for (int j = 0; j < 32; ++j) {
          float x0, x1;
          fma2_scalar(x0, x1, __uint_as_float(sr[2 * j]), __uint_as_float(sr[2 * j + 1]), scale_log2, -m_use);
          const float p0 = fast_exp2(x0), p1 = fast_exp2(x1);
          add2(ls0, ls1, p0, p1);
          pk[j] = pack2<IS_BF16>(p0, p1);
        }
        l_run += ls0 + ls1;
      }
      tmem_st32(tS + 32u * w, pk);
      tc_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_remote(pfull0 + 8u * (uint32_t)(i & 1));
      if (any_bounds) {
        mbar_arrive(bar(Cfg::B_BNDEMPTY + bslot));
        ++nbnd;
      }
    }
    if constexpr (BLOCK_SCORE != 0 && BLOCK_BOS) {
      if (ok && bs_dst)
        for (int g = bs_pend_hi; g >= bs_pend_lo; --g) block_flush<128>(bs_dst, bs_acc, g, bs_vec, p.block_cols);
    }
    // ---- epilogue: O / l -> 16 bit -> smem staging -> coalesced stores; LSE ----
    // O of tile i is signalled on the barrier of its parity.  The scores of the last tile prove O of the last tile but
    // two, so the phase before the awaited one is over; and no later phase can pass by a warp that comes late (with one
    // barrier for all tiles, awaited phase by phase, the last one could: the wait then ran out).
    if (ok) {
      ok = __all_sync(0xffffffffu, mbar_wait(bar(Cfg::B_ODONE + ((cnt - 1) & 1)), (uint32_t)((cnt - 1) >> 1) & 1u, wc));
      tc_fence_after();
    }
    // (every warp has read the maxima of the last tile before it handed over P, and O is done only after that)
    ex[128 * w + r] = l_run;
    ok = group_all(ok, 1, 256);
    if (ok) {
      const float m_fin = (m_run == ninf) ? 0.f : m_run;
      float l_tot = ex[r] + ex[128 + r];               // fixed order: the same value in both warpgroups
      if (p.sink) l_tot += fast_exp2(p.sink[hq] * kLog2e - m_fin);
      const float inv = l_tot > 0.f ? 1.f / l_tot : 0.f;
      uint8_t* stage = smem + Cfg::OFF_Q;              // Q is no longer needed; 512-byte rows
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        uint32_t orr[32];
        tmem_ld32(tO + 32 * c, orr);
        tc_wait_ld();
#pragma unroll
        for (int q4 = 0; q4 < 4; ++q4) {
          uint4 v;
          v.x = pack2<IS_BF16>(__uint_as_float(orr[8 * q4 + 0]) * inv, __uint_as_float(orr[8 * q4 + 1]) * inv);
          v.y = pack2<IS_BF16>(__uint_as_float(orr[8 * q4 + 2]) * inv, __uint_as_float(orr[8 * q4 + 3]) * inv);
          v.z = pack2<IS_BF16>(__uint_as_float(orr[8 * q4 + 4]) * inv, __uint_as_float(orr[8 * q4 + 5]) * inv);
          v.w = pack2<IS_BF16>(__uint_as_float(orr[8 * q4 + 6]) * inv, __uint_as_float(orr[8 * q4 + 7]) * inv);
          const int chunk = 16 * w + 4 * c + q4;       // 16-byte chunk inside the row
          *reinterpret_cast<uint4*>(stage + r * 512 + ((chunk ^ (r & 15)) << 4)) = v;
        }
      }
      if (slice == 0 && w == 0 && row < p.Sq)
        p.lse[((int64_t)b * p.Hq + hq) * p.Sq + row] = l_tot > 0.f ? (m_fin + log2f(l_tot)) * kLn2 : ninf;
      __syncwarp();   // each warp stores the 32 rows x 128 columns it staged itself
      uint16_t* go = reinterpret_cast<uint16_t*>(p.o) + b * p.o_b + hq * p.o_h + 256 * slice;
      const int wrow = (warp & 3) * 32;
#pragma unroll 4
      for (int x = lane; x < 32 * 16; x += 32) {
        const int rr = wrow + x / 16, cc = 16 * w + x % 16;
        const int grow = ms + 128 * rank + rr;
        if (grow < p.Sq)
          *reinterpret_cast<uint4*>(go + (int64_t)grow * p.o_s + cc * 8) =
              *reinterpret_cast<const uint4*>(stage + rr * 512 + ((cc ^ (rr & 15)) << 4));
      }
    }
  } else {
    setmaxnreg_dec<64>();
    if (warp == 8) {
      // =========================== TMA / bounds producer ===========================
      const uint32_t q_full = map_to_rank(bar(Cfg::B_Q), 0), kv_full = map_to_rank(bar(Cfg::B_KVFULL), 0);
      bool ok = true;
      int slot = 0, nbnd = 0;                  // ring position: slot and its phase
      uint32_t phase = 1u;
      if (lane == 0) {
        if (rank == 0) mbar_arrive_expect_tx(bar(Cfg::B_Q), 2 * Cfg::Q_BYTES);
        for (int dc = 0; dc < D / 64; ++dc)
          tma2_load_4d(sQ + dc * Cfg::SUB128, &tm_q, q_full, dc * 64, hq, ms + 128 * rank, b);
      }
      // one ring slot: two 64-row x 64-column boxes (one when `cols` is 64)
      auto fill = [&](const CUtensorMap* tm, int col, int row, int cols) {
        if (!ok) return;
        ok = mbar_wait(bar(Cfg::B_KVEMPTY + slot), phase, wc);
        if (!ok) return;
        if (rank == 0) mbar_arrive_expect_tx(bar(Cfg::B_KVFULL + slot), 2 * Cfg::SUB64 * (cols / 64));
        const uint32_t dst = sKV + slot * Cfg::SLOT_BYTES, fb = kv_full + 8u * (uint32_t)slot;
        tma2_load_4d(dst, tm, fb, col, hk, row, b);
        if (cols > 64) tma2_load_4d(dst + Cfg::SUB64, tm, fb, col + 64, hk, row, b);
        if (++slot == Cfg::NSTAGE) { slot = 0; phase ^= 1u; }
      };
      auto fill_k = [&](int i) {
        const int j0 = (int)(list[i] & 0xFFFFu) * 128 + 64 * rank;
        for (int c = 0; c < Cfg::KSLOTS; ++c) fill(&tm_k, 128 * c, j0, min(128, D - 128 * c));
      };
      auto fill_v = [&](int i) {
        const int j0 = (int)(list[i] & 0xFFFFu) * 128;
        for (int h = 0; h < 2; ++h) fill(&tm_v, 256 * slice + 128 * rank, j0 + 64 * h, 128);
      };
      if (lane == 0) fill_k(0);
      for (int i = 0; i < cnt; ++i) {
        const uint32_t e = list[i];
        if ((((e >> 16) | (e >> 20)) & FM_TF_BOUNDS) != 0) {
          const int bslot = nbnd % Cfg::NBND;
          const uint32_t par = ((uint32_t)(nbnd / Cfg::NBND) & 1u) ^ 1u;
          ok = __all_sync(0xffffffffu, ok && mbar_wait(bar(Cfg::B_BNDEMPTY + bslot), par, wc));
          if (!ok) break;
          const int j0 = (int)(e & 0xFFFFu) * 128;
          int* dst = reinterpret_cast<int*>(smem + Cfg::OFF_BND + bslot * Cfg::BND_BYTES);
          stage_bounds(dst, md.mask + ((size_t)bh_mask * p.Sk + j0) * md.ncols, 128, min(128, p.Sk - j0), md.ncols, lane);
          mbar_arrive(bar(Cfg::B_BNDFULL + bslot));
          ++nbnd;
        }
        if (lane == 0) {
          if (i + 1 < cnt) fill_k(i + 1);
          fill_v(i);
        }
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
      }
      // the leader's commits signal this CTA's barriers: none may be on its way when the CTA leaves
      if (ok && lane == 0)
        for (int x = 0; x < Cfg::NSTAGE; ++x) {
          mbar_wait(bar(Cfg::B_KVEMPTY + slot), phase, wc);
          if (++slot == Cfg::NSTAGE) { slot = 0; phase ^= 1u; }
        }
    } else if (warp == 9 && rank == 0) {
      // =========================== UMMA issuer (leading CTA) ===========================
      if (elect_one()) {
        constexpr uint32_t idesc_qk = make_idesc(IS_BF16, 256, 128, 0, 0);
        constexpr uint32_t idesc_pv = make_idesc(IS_BF16, 256, 256, 0, 1);
        const uint64_t dq = make_sdesc(sQ, 16, 1024);
        const uint64_t dk = make_sdesc(sKV, 16, 1024);
        const uint64_t dv = make_sdesc(sKV, Cfg::SUB64, 1024);
        bool ok = mbar_wait_cluster(bar(Cfg::B_Q), 0u, wc);
        int slot = 0;
        uint32_t phase = 0u;
        auto take = [&]() {                      // waits for the next ring slot
          ok = ok && mbar_wait_cluster(bar(Cfg::B_KVFULL + slot), phase, wc);
          if (ok) tc_fence_after();
          return ok;
        };
        auto release = [&]() {
          tc2_commit_both(bar(Cfg::B_KVEMPTY + slot));
          if (++slot == Cfg::NSTAGE) { slot = 0; phase ^= 1u; }
        };
        auto issue_qk = [&](int i) {
          const uint32_t dst = tmem + 128u * (uint32_t)(i & 1);
#pragma unroll
          for (int c = 0; c < Cfg::KSLOTS; ++c) {
            if (!take()) return;
            const uint64_t da = dq + (uint64_t)(2 * c * (Cfg::SUB128 >> 4));
            const uint64_t db = dk + (uint64_t)(slot * (Cfg::SLOT_BYTES >> 4));
#pragma unroll
            for (int u = 0; u < 2; ++u) {
              if (128 * c + 64 * u >= D) break;
#pragma unroll
              for (int ks = 0; ks < 4; ++ks)
                umma2_ss(dst, da + (uint64_t)(u * (Cfg::SUB128 >> 4) + 2 * ks), db + (uint64_t)(u * (Cfg::SUB64 >> 4) + 2 * ks),
                         idesc_qk, (c | u | ks) ? 1u : 0u);
            }
            release();
          }
          tc2_commit_both(bar(Cfg::B_SFULL + (i & 1)));
        };
        issue_qk(0);
        for (int i = 0; i < cnt && ok; ++i) {
          if (i + 1 < cnt) issue_qk(i + 1);
          if (!ok) break;
          ok = mbar_wait_cluster(bar(Cfg::B_PFULL + (i & 1)), (uint32_t)(i >> 1) & 1u, wc);
          if (!ok) break;
          const uint32_t src = tmem + 128u * (uint32_t)(i & 1);
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            if (!take()) break;
            const uint64_t db = dv + (uint64_t)(slot * (Cfg::SLOT_BYTES >> 4));
#pragma unroll
            for (int ks = 0; ks < 4; ++ks)
              umma2_ts(tmem + 256u, src + 32u * h + 8u * ks, db + (uint64_t)(128 * ks), idesc_pv, (i > 0 || h || ks) ? 1u : 0u);
            release();
          }
          if (!ok) break;
          tc2_commit_both(bar(Cfg::B_ODONE + (i & 1)));
        }
      }
      __syncwarp();
    }
  }

  // =========================== teardown ===========================
  tc_fence_before();
  __syncthreads();
  if (misc[4] != 0) {
    // copies and MMAs still in flight get a bounded time to land before the memory of this CTA is released
    const uint64_t t_end = global_timer_ns() + 200000ull;
    while (global_timer_ns() < t_end) __nanosleep(1000);
    if (tid == 0) atomicExch(&g_fwd_pair_status, FM_ERR_TIMEOUT);
  }
  __syncwarp();
  cluster_sync_all();          // the peer's MMAs and arrivals may still use this CTA's memory until here
  tc_fence_after();
  if (warp == 9) tmem2_dealloc(tmem, 512);
}

// ---------------------------------------------------------------------------
// host
// ---------------------------------------------------------------------------
template <int D, bool IS_BF16, int BLOCK_SCORE = 0, bool BLOCK_BOS = false>
static int launch_fwd_pair(const AttnKParams& p, const fm_attn_args* a, cudaStream_t s) {
  using Cfg = FwdPairCfg<D, BLOCK_SCORE != 0>;
  CUtensorMap tq, tk, tv;
  int rc;
  if ((rc = make_bshd_tmap(&tq, a->q, a->dtype, a->B, a->Sq, a->Hq, a->d, a->q_stride[0], a->q_stride[1], a->q_stride[2], 128))) return rc;
  if ((rc = make_bshd_tmap(&tk, a->k, a->dtype, a->B, a->Sk, a->Hkv, a->d, a->k_stride[0], a->k_stride[1], a->k_stride[2], 64))) return rc;
  if ((rc = make_bshd_tmap(&tv, a->v, a->dtype, a->B, a->Sk, a->Hkv, a->dv, a->v_stride[0], a->v_stride[1], a->v_stride[2], 64))) return rc;
  auto kern = fwd_pair_kernel<D, IS_BF16, BLOCK_SCORE, BLOCK_BOS>;
  constexpr int smem_bytes = BLOCK_SCORE ? Cfg::SMEM_BS : Cfg::SMEM;
  FM_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_bytes));
  const dim3 grid(2 * ((p.Sq + 255) / 256), p.Hq * Cfg::SLICES, p.B);
  kern<<<grid, Cfg::NTHREADS, smem_bytes, s>>>(tq, tk, tv, p);
  count_launches(1);
  FM_CUDA_TRY(cudaGetLastError());
  return FM_OK;
}

// d = dv = 256, 512, and 576 / 512, up to 2048 K tiles.
bool fwd_pair_supported(const fm_attn_args* a) {
  return pair_dims(a->d, a->dv) && (a->Sk + 127) / 128 <= FwdPairCfg<256>::LIST_MAX;
}

template <int D, bool IS_BF16>
static int launch_fwd_pair_any(const AttnKParams& p, const fm_attn_args* a, cudaStream_t s) {
  if (!p.block_logit) return launch_fwd_pair<D, IS_BF16>(p, a, s);
  if (p.block_bos) {
    if (p.block_log2 == 5) return launch_fwd_pair<D, IS_BF16, 32, true>(p, a, s);
    if (p.block_log2 == 6) return launch_fwd_pair<D, IS_BF16, 64, true>(p, a, s);
    return launch_fwd_pair<D, IS_BF16, 128, true>(p, a, s);
  }
  if (p.block_log2 == 5) return launch_fwd_pair<D, IS_BF16, 32>(p, a, s);
  if (p.block_log2 == 6) return launch_fwd_pair<D, IS_BF16, 64>(p, a, s);
  return launch_fwd_pair<D, IS_BF16, 128>(p, a, s);
}

int fwd_pair_launch(const AttnKParams& p, const fm_attn_args* a, cudaStream_t s) {
  const bool bf = a->dtype == FM_DTYPE_BF16;
  if (a->d == 256) return bf ? launch_fwd_pair_any<256, true>(p, a, s) : launch_fwd_pair_any<256, false>(p, a, s);
  if (a->d == 512) return bf ? launch_fwd_pair_any<512, true>(p, a, s) : launch_fwd_pair_any<512, false>(p, a, s);
  return bf ? launch_fwd_pair_any<576, true>(p, a, s) : launch_fwd_pair_any<576, false>(p, a, s);
}

int fwd_pair_status(int* out, bool reset) {
  int v = 0;
  FM_CUDA_TRY(cudaMemcpyFromSymbol(&v, g_fwd_pair_status, sizeof(int)));
  if (reset && v != 0) {
    const int z = 0;
    FM_CUDA_TRY(cudaMemcpyToSymbol(g_fwd_pair_status, &z, sizeof(int)));
  }
  *out = v;
  return FM_OK;
}

}  // namespace fm
