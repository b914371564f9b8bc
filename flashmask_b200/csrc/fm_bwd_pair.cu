// Backward attention for head dims 256/256, 512/512 and 576/512 on CTA pairs (tcgen05, cta_group::2), as two
// kernels per chunk of query rows:
//
//   scores   S = Q K^T and dP = dO V^T once per (256 queries, 256 keys), P = exp2(S scale - LSE) and
//            dS = P (dP - rowsum(O dO)) rounded to 16 bits into a workspace;
//   grads    dQ = dS K, dV = P^T dO and dK = dS^T Q as GEMMs whose A operand comes from the workspace.
//
// Why a workspace.  The accumulators of dK and dV for 128 keys take 2 x 256 of the 512 tensor-memory columns at
// d = 256 and 1088 at 576 / 512, so a kernel that keeps them recomputes S and dP for every slice of the outputs:
// 8 GEMM units instead of 5 at 256, 2.6 times the work at 576 / 512.  Per visible pair and head P and dS are 4 bytes
// written and, for each 256-column slice of the gradients, 6 bytes read (dS for dQ and for dK, P for dV): 10 bytes
// against 5 x 512 flops at 256, 16 against 5 x 1100 at 576 / 512.  That HBM time stays below the tensor time at these
// head dims (it would not at 128).  The workspace is bounded (kBudget): a chunk is
// as many kv groups (of all batch entries), or failing that as many query rows of one group, as fit; dK / dV of a group
// that needs several row chunks are summed in fp32 accumulators in chunk order.  Every sum has one owner and a fixed order.
//
// Workspace format.  128 query rows x 64 keys are one 16 KB block [8-key piece][row][8 keys]: a warp (32 rows)
// stores 512 contiguous bytes, the block is at the same time a K-major operand (dQ: M = rows) and an MN-major one
// (dV, dK: M = keys) of 8 x 16-byte core matrices without swizzle, and one contiguous box for the copy engine.
//
// Both kernels are persistent: 74 pairs walk a list of units round-robin, warp 10 builds the next unit's list of
// visible tiles while the current one runs.  Roles of each CTA (384 threads): 0-7 epilogue (thread = row), 8 TMA
// producer, 9 UMMA issuer (leading CTA), 10 list builder, 11 idle.  All waits are bounded.
//
// Bound: HBM.  At 4096 x 4096, 16 heads, d = 256 the score kernel moves 1.57 GB in 315 us (the P / dS stores also
// fill 68 % of the SM's request port to the L2), the gradient kernel 2.1 GB in 361 us; their tensor pipes are 45 and
// 63 % busy.  P and dS therefore pass the L2 as evict-first lines (stores and loads), so that they do not push out
// the Q, K, V and dO tiles that other pairs are about to read: at S = 16384, 16 heads, d = 256, causal, scores
// 2.59 -> 2.49 ms, gradients 2.92 -> 2.83 ms.
#include <algorithm>

#include "fm_attn_params.cuh"
#include "fm_sm100_pair.cuh"

namespace fm {

using namespace sm100;

__device__ int g_bwd_pair_status = 0;

// One chunk: q heads [head0, head0 + heads), counted through all batch entries, query rows
// [row0, row0 + 128 * row_blocks).
struct BwdPairChunk {
  uint4* ws_p; uint4* ws_ds;     // [heads][row_blocks][key_blocks] blocks of 16 KB
  float* acc_dk; float* acc_dv;  // fp32 sums of earlier row chunks, [unit][CTA][column][128 rows]
  int head0, heads, row0, row_blocks, key_blocks;
  int first, last;               // first / last row chunk of its heads
  int n_units, n_seg;            // scores: units; parts a row block's key tiles are dealt into
  int n_dk, n_dv, n_dq;          // grads: units of each kind, in this order
};

// Batch entry and head of a head counted through all entries.
struct BatchHead { int b, h; };
__device__ __forceinline__ BatchHead batch_head(int flat, int heads) { return {flat / heads, flat % heads}; }

constexpr int kPairListMax = 2048;

struct PairInfoBars {            // barrier indices shared by both kernels
  static constexpr int READY = 0, FREE = 2, NEXT = 4;
};

// ---------------------------------------------------------------------------
// scores
// ---------------------------------------------------------------------------
struct PairScoreCfg {
  static constexpr int NTHREADS = 384, NSTAGE = 6;
  static constexpr int SUB128 = 128 * 128;                     // 128 rows x 64 columns (bytes)
  static constexpr int SLOT_BYTES = 2 * SUB128;                // Q (dO) part, K (V) part
  static constexpr int LIST_MAX = kPairListMax / 2;            // 256-key tiles
  static constexpr int OFF_RING = 0;
  static constexpr int OFF_LIST = OFF_RING + NSTAGE * SLOT_BYTES;
  static constexpr int OFF_INFO = OFF_LIST + 2 * LIST_MAX * 4;
  static constexpr int OFF_BAR = OFF_INFO + 64;
  static constexpr int OFF_MISC = OFF_BAR + 32 * 8;
  static constexpr int SMEM = OFF_MISC + 64 + 1024;
  static constexpr int B_FULL = PairInfoBars::NEXT, B_EMPTY = B_FULL + NSTAGE, B_SFULL = B_EMPTY + NSTAGE,
                       B_SREAD = B_SFULL + 1, B_DPFULL = B_SREAD + 1, B_DPREAD = B_DPFULL + 1, B_COUNT = B_DPREAD + 1;
  static_assert(B_COUNT <= 32 && SMEM > 120 * 1024 && SMEM <= 227 * 1024, "one CTA per SM (512 TMEM columns)");
};

// Unit u of the chunk: segment fastest (neighbouring pairs share Q / dO), later row blocks (more keys under a
// causal mask) first.
struct ScoreUnit { int seg, rp, h; };
__device__ __forceinline__ ScoreUnit score_unit(const BwdPairChunk& c, int u) {
  ScoreUnit s;
  s.seg = u % c.n_seg;
  const int v = u / c.n_seg;
  s.h = v % c.heads;
  s.rp = c.row_blocks / 2 - 1 - v / c.heads;
  return s;
}

// Masks the scores of 128 columns whose bounds start at src (`valid` of them exist).
// Every lane reads the same bounds: broadcasts from the L1.  One loop per mask form, so that several columns' bounds
// are in flight (with the form decided inside the loop a partial tile waited for 128 loads in turn: 16 x 1024 rows of
// short documents, 16 heads, d = 256, took 1322 us against 733 us for the causal triangle that contains them).
__device__ __forceinline__ void mask_columns(const MaskDesc& md, const int32_t* src, int valid, int row, uint32_t* sr) {
  const uint32_t NEG = 0xff800000u;
  if (md.ncols == 1) {
    if (valid == 128 && (reinterpret_cast<uintptr_t>(src) & 15) == 0) {
#pragma unroll
      for (int j = 0; j < 32; ++j) {
        const int4 v = __ldg(reinterpret_cast<const int4*>(src) + j);
        if (row >= v.x) sr[4 * j] = NEG;
        if (row >= v.y) sr[4 * j + 1] = NEG;
        if (row >= v.z) sr[4 * j + 2] = NEG;
        if (row >= v.w) sr[4 * j + 3] = NEG;
      }
    } else {
#pragma unroll
      for (int c = 0; c < 128; ++c)
        if (c < valid && row >= __ldg(src + c)) sr[c] = NEG;
    }
  } else if (md.ncols == 2 && md.causal) {
#pragma unroll
    for (int c = 0; c < 128; ++c)
      if (c < valid) {
        const int2 v = __ldg(reinterpret_cast<const int2*>(src) + c);
        if (row >= v.x && row < v.y) sr[c] = NEG;
      }
  } else if (md.ncols == 2) {
#pragma unroll
    for (int c = 0; c < 128; ++c)
      if (c < valid) {
        const int2 v = __ldg(reinterpret_cast<const int2*>(src) + c);
        if (row >= v.x || row < v.y) sr[c] = NEG;
      }
  } else {
#pragma unroll
    for (int c = 0; c < 128; ++c)
      if (c < valid) {
        const int4 v = __ldg(reinterpret_cast<const int4*>(src) + c);
        if ((row >= v.x && row < v.y) || (row >= v.z && row < v.w)) sr[c] = NEG;
      }
  }
}

template <int D, int DV, bool IS_BF16>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(384, 1)
bwd_pair_scores_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_do,
                       const __grid_constant__ CUtensorMap tm_k, const __grid_constant__ CUtensorMap tm_v,
                       const AttnKParams p, const BwdPairChunk ck) {
  using Cfg = PairScoreCfg;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  const uint32_t sbase = smem_u32(smem);
  const uint32_t sRing = sbase + Cfg::OFF_RING;
  uint32_t* lists = reinterpret_cast<uint32_t*>(smem + Cfg::OFF_LIST);
  volatile int* infos = reinterpret_cast<volatile int*>(smem + Cfg::OFF_INFO);     // [2]: tiles of the unit
  const uint32_t bars = sbase + Cfg::OFF_BAR;
  volatile int* misc = reinterpret_cast<volatile int*>(smem + Cfg::OFF_MISC);      // [0] tmem, [4] abort
  auto bar = [&](int i) { return bars + 8u * (uint32_t)i; };
  const int tid = threadIdx.x;
  const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
  const int lane = tid & 31;
  const int rank = (int)cluster_ctarank();
  const int cl = blockIdx.x >> 1, n_cl = gridDim.x >> 1;
  const MaskDesc& md = p.md;
  const int off = p.Sk - p.Sq;

  if (tid == 0) misc[4] = 0;
  if (warp == 8 && lane == 0) {
    tma_prefetch_desc(&tm_q); tma_prefetch_desc(&tm_do); tma_prefetch_desc(&tm_k); tma_prefetch_desc(&tm_v);
    for (int i = 0; i < 2; ++i) { mbar_init(bar(PairInfoBars::READY + i), 1); mbar_init(bar(PairInfoBars::FREE + i), rank == 0 ? 10 : 9); }
    for (int i = 0; i < Cfg::NSTAGE; ++i) { mbar_init(bar(Cfg::B_FULL + i), 1); mbar_init(bar(Cfg::B_EMPTY + i), 1); }
    mbar_init(bar(Cfg::B_SFULL), 1); mbar_init(bar(Cfg::B_DPFULL), 1);
    mbar_init(bar(Cfg::B_SREAD), 16); mbar_init(bar(Cfg::B_DPREAD), 16);
    fence_mbar_init();
  }
  if (warp == 9) {
    tmem2_alloc(sbase + Cfg::OFF_MISC, 512);
    tmem2_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();
  tc_fence_after();
  const uint32_t tmem = (uint32_t)misc[0];
  WaitCtx wc{misc + 4, global_timer_ns() + 2000000000ull};

  if (warp < 8) {
    // =========================== epilogue: P and dS ===========================
    setmaxnreg_inc<208>();
    const int w = warp >> 2;                     // keys [128 w, 128 w + 128) of every 256-key tile
    const int r = tid & 127;
    const uint32_t lane_field = (uint32_t)((warp & 3) * 32) << 16;
    const uint32_t tS = tmem + lane_field + 128u * w, tDP = tS + 256u;
    const uint32_t sread = map_to_rank(bar(Cfg::B_SREAD), 0), dpread = map_to_rank(bar(Cfg::B_DPREAD), 0);
    const uint32_t NEG = 0xff800000u;
    bool ok = true;
    uint32_t it = 0;                             // tiles so far
    int j = 0;
    for (int u = cl; u < ck.n_units && ok; u += n_cl, ++j) {
      ok = __all_sync(0xffffffffu, mbar_wait_idle(bar(PairInfoBars::READY + (j & 1)), (uint32_t)(j >> 1) & 1u, wc));
      if (!ok) break;
      const ScoreUnit un = score_unit(ck, u);
      const int cnt = infos[j & 1];
      const uint32_t* list = lists + (j & 1) * Cfg::LIST_MAX;
      const BatchHead bh = batch_head(ck.head0 + un.h, p.Hq);
      const int rb = 2 * un.rp + rank;
      const int row = ck.row0 + 128 * rb + r;
      const int bh_mask = md.ncols ? ((md.mask_B == 1 ? 0 : bh.b) * md.Hm + bh.h / (p.Hq / md.Hm)) : 0;
      float lse2 = 0.f, dps = 0.f;
      if (row < p.Sq_r) {
        const int64_t at = (int64_t)(ck.head0 + un.h) * p.Sq_r + row;
        lse2 = p.lse_log2[at];
        dps = p.dpsum[at];
      }
      const int64_t blk0 = ((int64_t)un.h * ck.row_blocks + rb) * ck.key_blocks;
      for (int i = 0; i < cnt && ok; ++i, ++it) {
        const uint32_t e = list[i];
        const int n2 = (int)(e & 0xFFFFu);
        const uint32_t flags = (e >> (16 + 8 * rank + 4 * w)) & 0xFu;
        ok = __all_sync(0xffffffffu, mbar_wait(bar(Cfg::B_SFULL), it & 1u, wc));
        if (!ok) break;
        tc_fence_after();
        uint32_t sr[128];
        tmem_ld32(tS, sr); tmem_ld32(tS + 32, sr + 32); tmem_ld32(tS + 64, sr + 64); tmem_ld32(tS + 96, sr + 96);
        tc_wait_ld();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_remote(sread);
        const int j0 = n2 * 256 + 128 * w;
        if (flags & FM_TF_BOUNDS) {
          const int valid = min(128, p.Sk - j0);
          const int32_t* src = md.mask + ((size_t)bh_mask * p.Sk + j0) * md.ncols;
          mask_columns(md, src, valid, row, sr);
        }
        if (flags & (FM_TF_CAUSAL | FM_TF_RAGGED)) {
          int jmax = p.Sk - 1 - j0;
          if (md.causal) jmax = min(jmax, row + off - j0);
#pragma unroll
          for (int c = 0; c < 128; ++c)
            if (c > jmax) sr[c] = NEG;
        }
        if (!flags || row >= p.Sq_r) {
#pragma unroll
          for (int c = 0; c < 128; ++c) sr[c] = NEG;
        }
        const int64_t blk = blk0 + 4 * n2 + 2 * w;
        uint4* gp = ck.ws_p + blk * 1024 + r;              // + 128 * (8-key piece)
        uint4* gd = ck.ws_ds + blk * 1024 + r;
#pragma unroll
        for (int c = 0; c < 128; c += 8) {
          uint32_t pk[4];
#pragma unroll
          for (int x = 0; x < 4; ++x) {
            float x0, x1;
            fma2_scalar(x0, x1, __uint_as_float(sr[c + 2 * x]), __uint_as_float(sr[c + 2 * x + 1]), p.scale_log2, -lse2);
            const float p0 = fast_exp2(x0), p1 = fast_exp2(x1);
            sr[c + 2 * x] = __float_as_uint(p0);
            sr[c + 2 * x + 1] = __float_as_uint(p1);
            pk[x] = pack2<IS_BF16>(p0, p1);
          }
          __stcs(gp + (c >> 3) * 128, make_uint4(pk[0], pk[1], pk[2], pk[3]));
        }
        ok = __all_sync(0xffffffffu, mbar_wait(bar(Cfg::B_DPFULL), it & 1u, wc));
        if (!ok) break;
        tc_fence_after();
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          uint32_t dr[32];
          tmem_ld32(tDP + 32 * q, dr);
          tc_wait_ld();
          if (q == 3) {
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_remote(dpread);
          }
#pragma unroll
          for (int c = 0; c < 32; c += 8) {
            uint32_t pk[4];
#pragma unroll
            for (int x = 0; x < 4; ++x)
              pk[x] = pack2<IS_BF16>(__uint_as_float(sr[32 * q + c + 2 * x]) * (__uint_as_float(dr[c + 2 * x]) - dps),
                                     __uint_as_float(sr[32 * q + c + 2 * x + 1]) * (__uint_as_float(dr[c + 2 * x + 1]) - dps));
            __stcs(gd + (4 * q + (c >> 3)) * 128, make_uint4(pk[0], pk[1], pk[2], pk[3]));
          }
        }
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(bar(PairInfoBars::FREE + (j & 1)));
    }
  } else {
    setmaxnreg_dec<64>();
    if (warp == 10) {
      // =========================== list builder ===========================
      bool ok = true;
      int j = 0;
      for (int u = cl; u < ck.n_units; u += n_cl, ++j) {
        if (j >= 2) ok = __all_sync(0xffffffffu, mbar_wait_idle(bar(PairInfoBars::FREE + (j & 1)), (uint32_t)((j >> 1) - 1) & 1u, wc));
        if (!ok) break;
        const ScoreUnit un = score_unit(ck, u);
        const BatchHead bh = batch_head(ck.head0 + un.h, p.Hq);
        const int bh_mask = md.ncols ? ((md.mask_B == 1 ? 0 : bh.b) * md.Hm + bh.h / (p.Hq / md.Hm)) : 0;
        const int ms = ck.row0 + 256 * un.rp;
        const int nb = (p.Sk + 127) / 128;
        const int n_hi = ms >= p.Sq ? 0 : (md.causal ? max(0, min(nb, (min(ms + 256, p.Sq) + off + 127) / 128)) : nb);
        uint32_t* list = lists + (j & 1) * Cfg::LIST_MAX;
        int cnt = 0;                              // visible 256-key tiles; every n_seg-th of them is this unit's
        for (int base = (n_hi + 1) / 2 - 1; base >= 0; base -= 32) {
          const int n2 = base - lane;
          uint32_t f = 0;
          if (n2 >= 0) {
#pragma unroll
            for (int x = 0; x < 4; ++x) {         // x = 2 * (row half) + key half
              const int m0 = ms + 128 * (x >> 1), n = 2 * n2 + (x & 1);
              if (m0 < p.Sq && n < n_hi) f |= tile_flags(md, bh_mask, n, m0, min(m0 + 128, p.Sq), 128) << (4 * x);
            }
          }
          const uint32_t bal = __ballot_sync(0xffffffffu, f != 0);
          const int pos = cnt + __popc(bal & ((1u << lane) - 1u));
          if (f && pos % ck.n_seg == un.seg) list[pos / ck.n_seg] = (uint32_t)n2 | (f << 16);
          cnt += __popc(bal);
        }
        __syncwarp();
        if (lane == 0) {
          infos[j & 1] = (cnt - un.seg + ck.n_seg - 1) / ck.n_seg;
          mbar_arrive(bar(PairInfoBars::READY + (j & 1)));
        }
      }
    } else if (warp == 8) {
      // =========================== TMA producer ===========================
      const uint32_t full = map_to_rank(bar(Cfg::B_FULL), 0);
      bool ok = true;
      int slot = 0, j = 0;
      uint32_t phase = 1u;
      if (lane == 0) {
        for (int u = cl; u < ck.n_units && ok; u += n_cl, ++j) {
          ok = mbar_wait(bar(PairInfoBars::READY + (j & 1)), (uint32_t)(j >> 1) & 1u, wc);
          if (!ok) break;
          const ScoreUnit un = score_unit(ck, u);
          const int cnt = infos[j & 1];
          const uint32_t* list = lists + (j & 1) * Cfg::LIST_MAX;
          const BatchHead bh = batch_head(ck.head0 + un.h, p.Hq);
          const int hk = bh.h / (p.Hq / p.Hkv);
          const int row = ck.row0 + 128 * (2 * un.rp + rank);
          for (int i = 0; i < cnt && ok; ++i) {
            const int key = (int)(list[i] & 0xFFFFu) * 256 + 128 * rank;
            for (int c = 0; c < (D + DV) / 64; ++c) {
              ok = mbar_wait(bar(Cfg::B_EMPTY + slot), phase, wc);
              if (!ok) break;
              if (rank == 0) mbar_arrive_expect_tx(bar(Cfg::B_FULL + slot), 2 * Cfg::SLOT_BYTES);
              const uint32_t dst = sRing + slot * Cfg::SLOT_BYTES, fb = full + 8u * (uint32_t)slot;
              const bool first = c < D / 64;
              const int col = 64 * (first ? c : c - D / 64);
              tma2_load_4d(dst, first ? &tm_q : &tm_do, fb, col, bh.h, row, bh.b);
              tma2_load_4d(dst + Cfg::SUB128, first ? &tm_k : &tm_v, fb, col, hk, key, bh.b);
              if (++slot == Cfg::NSTAGE) { slot = 0; phase ^= 1u; }
            }
          }
          mbar_arrive(bar(PairInfoBars::FREE + (j & 1)));
        }
        // no commit of the leader may be on its way to this CTA's barriers when it leaves
        for (int x = 0; x < Cfg::NSTAGE && ok; ++x) {
          ok = mbar_wait(bar(Cfg::B_EMPTY + slot), phase, wc);
          if (++slot == Cfg::NSTAGE) { slot = 0; phase ^= 1u; }
        }
      }
      __syncwarp();
    } else if (warp == 9 && rank == 0) {
      // =========================== UMMA issuer ===========================
      if (elect_one()) {
        constexpr uint32_t idesc = make_idesc(IS_BF16, 256, 256, 0, 0);
        const uint64_t da0 = make_sdesc(sRing, 16, 1024), db0 = make_sdesc(sRing + Cfg::SUB128, 16, 1024);
        bool ok = true;
        int slot = 0, j = 0;
        uint32_t phase = 0u, it = 0;
        auto gemm = [&](uint32_t dst, int chunks) {
          for (int c = 0; c < chunks; ++c) {
            ok = mbar_wait_cluster(bar(Cfg::B_FULL + slot), phase, wc);
            if (!ok) return;
            tc_fence_after();
            const uint64_t at = (uint64_t)(slot * (Cfg::SLOT_BYTES >> 4));
#pragma unroll
            for (int ks = 0; ks < 4; ++ks)
              umma2_ss(dst, da0 + at + (uint64_t)(2 * ks), db0 + at + (uint64_t)(2 * ks), idesc, (c | ks) ? 1u : 0u);
            tc2_commit_both(bar(Cfg::B_EMPTY + slot));
            if (++slot == Cfg::NSTAGE) { slot = 0; phase ^= 1u; }
          }
        };
        for (int u = cl; u < ck.n_units && ok; u += n_cl, ++j) {
          ok = mbar_wait(bar(PairInfoBars::READY + (j & 1)), (uint32_t)(j >> 1) & 1u, wc);
          if (!ok) break;
          const int cnt = infos[j & 1];
          mbar_arrive(bar(PairInfoBars::FREE + (j & 1)));
          for (int i = 0; i < cnt && ok; ++i, ++it) {
            if (it > 0) ok = mbar_wait_cluster(bar(Cfg::B_SREAD), (it - 1) & 1u, wc);
            if (!ok) break;
            gemm(tmem, D / 64);
            if (!ok) break;
            tc2_commit_both(bar(Cfg::B_SFULL));
            if (it > 0) ok = mbar_wait_cluster(bar(Cfg::B_DPREAD), (it - 1) & 1u, wc);
            if (!ok) break;
            gemm(tmem + 256u, DV / 64);
            if (!ok) break;
            tc2_commit_both(bar(Cfg::B_DPFULL));
          }
        }
      }
      __syncwarp();
    }
  }

  // =========================== teardown ===========================
  tc_fence_before();
  __syncthreads();
  if (misc[4] != 0) {
    const uint64_t t_end = global_timer_ns() + 200000ull;
    while (global_timer_ns() < t_end) __nanosleep(1000);
    if (tid == 0) atomicExch(&g_bwd_pair_status, FM_ERR_TIMEOUT);
  }
  __syncwarp();
  cluster_sync_all();
  tc_fence_after();
  if (warp == 9) tmem2_dealloc(tmem, 512);
}

// ---------------------------------------------------------------------------
// grads
// ---------------------------------------------------------------------------
// TAIL: d = 576 has a 64-column rest beside its 256-column slices; it rides with the last one (N = 256 + 64).
template <int D, int DV>
struct PairGradCfg {
  static constexpr int NTHREADS = 384, NSTAGE = 3;
  static constexpr bool TAIL = D % 256 != 0;
  static constexpr int NS_D = D / 256, NS_V = DV / 256;        // slices of dQ / dK and of dV
  static constexpr int SUB128 = 128 * 128;
  static constexpr int A_BYTES = 2 * SUB128;                   // 128 x 128 of P or dS (two workspace blocks)
  static constexpr int B_BYTES = 2 * SUB128;                   // 128 rows x 128 columns of K, dO or Q
  static constexpr int T_BYTES = TAIL ? 128 * 64 : 0;          // 128 rows x 32 columns (64-byte swizzle)
  static constexpr int SLOT_BYTES = A_BYTES + B_BYTES + T_BYTES;
  static constexpr int LIST_MAX = kPairListMax;
  static constexpr int OFF_RING = 0;
  static constexpr int OFF_LIST = OFF_RING + NSTAGE * SLOT_BYTES;
  static constexpr int OFF_INFO = OFF_LIST + 2 * LIST_MAX * 2;
  static constexpr int OFF_BAR = OFF_INFO + 64;
  static constexpr int OFF_MISC = OFF_BAR + 32 * 8;
  static constexpr int SMEM = OFF_MISC + 64 + 1024;
  static constexpr int B_FULL = PairInfoBars::NEXT, B_EMPTY = B_FULL + NSTAGE, B_ACC = B_EMPTY + NSTAGE,
                       B_ACCFREE = B_ACC + 1, B_COUNT = B_ACCFREE + 1;
  static_assert(D % 256 == 0 || D % 256 == 64, "whole slices and at most a 64-column rest");
  static_assert(B_COUNT <= 32 && SMEM > 120 * 1024 && SMEM <= 227 * 1024, "one CTA per SM (512 TMEM columns)");
};

enum { GRAD_DK = 0, GRAD_DV = 1, GRAD_DQ = 2 };

// Unit u: dK, then dV (256 keys of a kv head, one column slice), then dQ (256 query rows of a q head, one
// slice).  Slices are neighbours (they read the same P / dS), heads next.
struct GradUnit { int kind, slice, blk, h; };      // h: kv head (dK, dV) or q head (dQ) inside the chunk
template <int D, int DV>
__device__ __forceinline__ GradUnit grad_unit(const BwdPairChunk& c, int u, int groups) {
  using Cfg = PairGradCfg<D, DV>;
  GradUnit g;
  int ns = Cfg::NS_D, heads = groups, v = u;
  if (u < c.n_dk) {
    g.kind = GRAD_DK;
  } else if (u < c.n_dk + c.n_dv) {
    g.kind = GRAD_DV; v = u - c.n_dk; ns = Cfg::NS_V;
  } else {
    g.kind = GRAD_DQ; v = u - c.n_dk - c.n_dv; heads = c.heads;
  }
  g.slice = ns - 1 - v % ns;
  v /= ns;
  g.h = v % heads;
  g.blk = v / heads;
  if (g.kind == GRAD_DQ) g.blk = c.row_blocks / 2 - 1 - g.blk;   // later rows (more keys under a causal mask) first
  return g;
}

template <int D, int DV, bool IS_BF16>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(384, 1)
bwd_pair_grads_kernel(const __grid_constant__ CUtensorMap tm_p, const __grid_constant__ CUtensorMap tm_ds,
                      const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_do,
                      const __grid_constant__ CUtensorMap tm_k, const __grid_constant__ CUtensorMap tm_q_tail,
                      const __grid_constant__ CUtensorMap tm_k_tail, const AttnKParams p, const BwdPairChunk ck) {
  using Cfg = PairGradCfg<D, DV>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  const uint32_t sbase = smem_u32(smem);
  const uint32_t sRing = sbase + Cfg::OFF_RING;
  uint16_t* lists = reinterpret_cast<uint16_t*>(smem + Cfg::OFF_LIST);
  volatile int* infos = reinterpret_cast<volatile int*>(smem + Cfg::OFF_INFO);
  const uint32_t bars = sbase + Cfg::OFF_BAR;
  volatile int* misc = reinterpret_cast<volatile int*>(smem + Cfg::OFF_MISC);
  auto bar = [&](int i) { return bars + 8u * (uint32_t)i; };
  const int tid = threadIdx.x;
  const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
  const int lane = tid & 31;
  const int rank = (int)cluster_ctarank();
  const int cl = blockIdx.x >> 1, n_cl = gridDim.x >> 1;
  const MaskDesc& md = p.md;
  const int G = p.Hq / p.Hkv;
  const int groups = ck.heads / G;
  const int n_units = ck.n_dk + ck.n_dv + ck.n_dq;

  if (tid == 0) misc[4] = 0;
  if (warp == 8 && lane == 0) {
    tma_prefetch_desc(&tm_p); tma_prefetch_desc(&tm_ds); tma_prefetch_desc(&tm_q); tma_prefetch_desc(&tm_do);
    tma_prefetch_desc(&tm_k);
    for (int i = 0; i < 2; ++i) { mbar_init(bar(PairInfoBars::READY + i), 1); mbar_init(bar(PairInfoBars::FREE + i), rank == 0 ? 10 : 9); }
    for (int i = 0; i < Cfg::NSTAGE; ++i) { mbar_init(bar(Cfg::B_FULL + i), 1); mbar_init(bar(Cfg::B_EMPTY + i), 1); }
    mbar_init(bar(Cfg::B_ACC), 1); mbar_init(bar(Cfg::B_ACCFREE), 16);
    fence_mbar_init();
  }
  if (warp == 9) {
    tmem2_alloc(sbase + Cfg::OFF_MISC, 512);
    tmem2_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();
  tc_fence_after();
  const uint32_t tmem = (uint32_t)misc[0];
  WaitCtx wc{misc + 4, global_timer_ns() + 2000000000ull};

  if (warp < 8) {
    // =========================== epilogue ===========================
    setmaxnreg_inc<208>();
    const int w = warp >> 2;
    const int r = tid & 127;
    const uint32_t lane_field = (uint32_t)((warp & 3) * 32) << 16;
    const uint32_t accfree = map_to_rank(bar(Cfg::B_ACCFREE), 0);
    bool ok = true;
    int j = 0, ju = 0;                           // units so far, units with work so far
    for (int u = cl; u < n_units && ok; u += n_cl, ++j) {
      ok = __all_sync(0xffffffffu, mbar_wait_idle(bar(PairInfoBars::READY + (j & 1)), (uint32_t)(j >> 1) & 1u, wc));
      if (!ok) break;
      const int cnt = infos[j & 1];
      __syncwarp();
      if (lane == 0) mbar_arrive(bar(PairInfoBars::FREE + (j & 1)));
      const GradUnit g = grad_unit<D, DV>(ck, u, groups);
      const bool tail = Cfg::TAIL && g.kind != GRAD_DV && g.slice == Cfg::NS_D - 1;
      const int row = (g.kind == GRAD_DQ ? ck.row0 : 0) + 256 * g.blk + 128 * rank + r;
      const int n_rows = g.kind == GRAD_DQ ? p.Sq : p.Sk;
      // where the result goes: the output, or (dK / dV of a group in several row chunks) the fp32 sums
      uint16_t* out;
      const BatchHead bh = g.kind == GRAD_DQ ? batch_head(ck.head0 + g.h, p.Hq) : batch_head(ck.head0 / G + g.h, p.Hkv);
      if (g.kind == GRAD_DQ) out = reinterpret_cast<uint16_t*>(p.dq) + bh.b * p.dq_b + (int64_t)row * p.dq_s + bh.h * p.dq_h;
      else if (g.kind == GRAD_DK) out = reinterpret_cast<uint16_t*>(p.dk) + bh.b * p.dk_b + (int64_t)row * p.dk_s + bh.h * p.dk_h;
      else out = reinterpret_cast<uint16_t*>(p.dv) + bh.b * p.dv_b + (int64_t)row * p.dv_s + bh.h * p.dv_h;
      out += 256 * g.slice;
      const bool sums_in = g.kind != GRAD_DQ && !ck.first, sums_out = g.kind != GRAD_DQ && !ck.last;
      float* acc = nullptr;
      if (sums_in || sums_out) {
        const int width = g.kind == GRAD_DK ? D : DV;
        acc = (g.kind == GRAD_DK ? ck.acc_dk : ck.acc_dv) +
              (((int64_t)(g.h * (ck.key_blocks / 4) + g.blk) * 2 + rank) * width + 256 * g.slice) * 128 + r;
      }
      const float mul = g.kind == GRAD_DV ? 1.f : p.scale;
      if (cnt > 0) {
        ok = __all_sync(0xffffffffu, mbar_wait_idle(bar(Cfg::B_ACC), (uint32_t)ju & 1u, wc));
        if (!ok) break;
        ++ju;
        tc_fence_after();
      }
      if (cnt == 0 && sums_in && sums_out) continue;       // nothing to add to the sums
      // warpgroup w: pieces of 32 columns w, w + 2, ...; the tail is pieces 8 and 9
      const int n_pieces = tail ? 10 : 8;
#pragma unroll 1
      for (int q = w; q < n_pieces; q += 2) {
        uint32_t v[32];
        if (cnt > 0) {
          tmem_ld32(tmem + lane_field + 32u * (uint32_t)q, v);
          tc_wait_ld();
          if (q + 2 >= n_pieces) {
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_remote(accfree);
          }
        } else {
#pragma unroll
          for (int c = 0; c < 32; ++c) v[c] = 0u;
        }
        if (sums_in) {
          float s[32];
#pragma unroll
          for (int c = 0; c < 32; ++c) s[c] = __ldcg(acc + (32 * q + c) * 128);
#pragma unroll
          for (int c = 0; c < 32; ++c) v[c] = __float_as_uint(__uint_as_float(v[c]) + s[c]);
        }
        if (sums_out) {
#pragma unroll
          for (int c = 0; c < 32; ++c) __stcg(acc + (32 * q + c) * 128, __uint_as_float(v[c]));
        } else if (row < n_rows) {
#pragma unroll
          for (int c = 0; c < 32; c += 8) {
            uint4 o;
            o.x = pack2<IS_BF16>(__uint_as_float(v[c]) * mul, __uint_as_float(v[c + 1]) * mul);
            o.y = pack2<IS_BF16>(__uint_as_float(v[c + 2]) * mul, __uint_as_float(v[c + 3]) * mul);
            o.z = pack2<IS_BF16>(__uint_as_float(v[c + 4]) * mul, __uint_as_float(v[c + 5]) * mul);
            o.w = pack2<IS_BF16>(__uint_as_float(v[c + 6]) * mul, __uint_as_float(v[c + 7]) * mul);
            *reinterpret_cast<uint4*>(out + 32 * q + c) = o;
          }
        }
        __syncwarp();
      }
    }
  } else {
    setmaxnreg_dec<64>();
    if (warp == 10) {
      // =========================== list builder ===========================
      bool ok = true;
      int j = 0;
      const int nb = (p.Sk + 127) / 128;
      for (int u = cl; u < n_units; u += n_cl, ++j) {
        if (j >= 2) ok = __all_sync(0xffffffffu, mbar_wait_idle(bar(PairInfoBars::FREE + (j & 1)), (uint32_t)((j >> 1) - 1) & 1u, wc));
        if (!ok) break;
        const GradUnit g = grad_unit<D, DV>(ck, u, groups);
        const BatchHead bh = batch_head(ck.head0 + (g.kind == GRAD_DQ ? g.h : g.h * G), p.Hq);
        const int bh_mask = md.ncols ? ((md.mask_B == 1 ? 0 : bh.b) * md.Hm + bh.h / (p.Hq / md.Hm)) : 0;
        uint16_t* list = lists + (j & 1) * Cfg::LIST_MAX;
        int cnt = 0;
        // dQ: key tiles that either half of the 256 rows sees; dK / dV: 128-row blocks that see either half of the keys
        const int n_all = g.kind == GRAD_DQ ? nb : ck.row_blocks;
        for (int base = 0; base < n_all; base += 32) {
          const int x = base + lane;
          uint32_t f = 0;
          if (x < n_all) {
#pragma unroll
            for (int half = 0; half < 2; ++half) {
              const int n = g.kind == GRAD_DQ ? x : 2 * g.blk + half;
              const int m0 = ck.row0 + (g.kind == GRAD_DQ ? 256 * g.blk + 128 * half : 128 * x);
              if (m0 < p.Sq && n < nb) f |= tile_flags(md, bh_mask, n, m0, min(m0 + 128, p.Sq), 128);
            }
          }
          const uint32_t bal = __ballot_sync(0xffffffffu, f != 0);
          const int pos = cnt + __popc(bal & ((1u << lane) - 1u));
          if (f && pos < Cfg::LIST_MAX) list[pos] = (uint16_t)x;
          cnt += __popc(bal);
        }
        __syncwarp();
        if (lane == 0) {
          infos[j & 1] = cnt;
          mbar_arrive(bar(PairInfoBars::READY + (j & 1)));
        }
      }
    } else if (warp == 8) {
      // =========================== TMA producer ===========================
      const uint32_t full = map_to_rank(bar(Cfg::B_FULL), 0);
      bool ok = true;
      int slot = 0, j = 0;
      uint32_t phase = 1u;
      if (lane == 0) {
        const uint64_t stream_policy = policy_evict_first();
        for (int u = cl; u < n_units && ok; u += n_cl, ++j) {
          ok = mbar_wait(bar(PairInfoBars::READY + (j & 1)), (uint32_t)(j >> 1) & 1u, wc);
          if (!ok) break;
          const GradUnit g = grad_unit<D, DV>(ck, u, groups);
          const int cnt = infos[j & 1];
          const uint16_t* list = lists + (j & 1) * Cfg::LIST_MAX;
          const bool is_dq = g.kind == GRAD_DQ;
          const bool tail = Cfg::TAIL && g.kind != GRAD_DV && g.slice == Cfg::NS_D - 1;
          const CUtensorMap* tA = g.kind == GRAD_DV ? &tm_p : &tm_ds;
          const CUtensorMap* tB = is_dq ? &tm_k : (g.kind == GRAD_DV ? &tm_do : &tm_q);
          const CUtensorMap* tT = is_dq ? &tm_k_tail : &tm_q_tail;
          const int n_heads = is_dq ? 1 : G;
          for (int hh = 0; hh < n_heads && ok; ++hh) {
            const int h = is_dq ? g.h : g.h * G + hh;                  // q head inside the chunk
            const BatchHead bB = is_dq ? batch_head((ck.head0 + g.h) / G, p.Hkv) : batch_head(ck.head0 + h, p.Hq);   // of the B operand
            for (int i = 0; i < cnt && ok; ++i) {
              const int x = list[i];
              const int rb = is_dq ? 2 * g.blk + rank : x;
              const int kb = is_dq ? 2 * x : 4 * g.blk + 2 * rank;
              const int rowB = is_dq ? 128 * x : ck.row0 + 128 * x;
              ok = mbar_wait(bar(Cfg::B_EMPTY + slot), phase, wc);
              if (!ok) break;
              if (rank == 0)
                mbar_arrive_expect_tx(bar(Cfg::B_FULL + slot), 2 * (Cfg::A_BYTES + Cfg::B_BYTES + (tail ? Cfg::T_BYTES : 0)));
              const uint32_t dst = sRing + slot * Cfg::SLOT_BYTES, fb = full + 8u * (uint32_t)slot;
              const int blk = (h * ck.row_blocks + rb) * ck.key_blocks + kb;
              tma2_load_2d(dst, tA, fb, 0, blk * 128, stream_policy);
              tma2_load_2d(dst + Cfg::SUB128, tA, fb, 0, blk * 128 + 128, stream_policy);
              const int col = 256 * g.slice + 128 * rank;
              tma2_load_4d(dst + Cfg::A_BYTES, tB, fb, col, bB.h, rowB, bB.b);
              tma2_load_4d(dst + Cfg::A_BYTES + Cfg::SUB128, tB, fb, col + 64, bB.h, rowB, bB.b);
              if (tail) tma2_load_4d(dst + Cfg::A_BYTES + Cfg::B_BYTES, tT, fb, 256 * Cfg::NS_D + 32 * rank, bB.h, rowB, bB.b);
              if (++slot == Cfg::NSTAGE) { slot = 0; phase ^= 1u; }
            }
          }
          mbar_arrive(bar(PairInfoBars::FREE + (j & 1)));
        }
        for (int x = 0; x < Cfg::NSTAGE && ok; ++x) {
          ok = mbar_wait(bar(Cfg::B_EMPTY + slot), phase, wc);
          if (++slot == Cfg::NSTAGE) { slot = 0; phase ^= 1u; }
        }
      }
      __syncwarp();
    } else if (warp == 9 && rank == 0) {
      // =========================== UMMA issuer ===========================
      if (elect_one()) {
        constexpr uint32_t idesc_k = make_idesc(IS_BF16, 256, 256, 0, 1), idesc_k_tail = make_idesc(IS_BF16, 256, 64, 0, 1);
        constexpr uint32_t idesc_mn = make_idesc(IS_BF16, 256, 256, 1, 1), idesc_mn_tail = make_idesc(IS_BF16, 256, 64, 1, 1);
        const uint64_t dAk = make_sdesc_noswz(sRing, 2048, 128);           // rows x keys, K-major (dQ)
        const uint64_t dAm = make_sdesc_noswz(sRing, 128, 2048);           // the same bytes, M = keys (dV, dK)
        const uint64_t dB = make_sdesc(sRing + Cfg::A_BYTES, Cfg::SUB128, 1024);
        // 32 columns of 64 bytes: 64-byte swizzle, 8-row groups of 512 bytes
        const uint64_t dT = (make_sdesc_noswz(sRing + Cfg::A_BYTES + Cfg::B_BYTES, 16, 512)) | (4ull << 61);
        bool ok = true;
        int slot = 0, j = 0, ju = 0;
        uint32_t phase = 0u;
        for (int u = cl; u < n_units && ok; u += n_cl, ++j) {
          ok = mbar_wait(bar(PairInfoBars::READY + (j & 1)), (uint32_t)(j >> 1) & 1u, wc);
          if (!ok) break;
          const GradUnit g = grad_unit<D, DV>(ck, u, groups);
          const int cnt = infos[j & 1];
          mbar_arrive(bar(PairInfoBars::FREE + (j & 1)));
          if (cnt == 0) continue;
          const bool is_dq = g.kind == GRAD_DQ;
          const bool tail = Cfg::TAIL && g.kind != GRAD_DV && g.slice == Cfg::NS_D - 1;
          const int items = cnt * (is_dq ? 1 : G);
          if (ju > 0) ok = mbar_wait_cluster(bar(Cfg::B_ACCFREE), (uint32_t)(ju - 1) & 1u, wc);
          ++ju;
          const uint64_t dA = is_dq ? dAk : dAm;
          const uint64_t stepA = is_dq ? 256u : 16u;       // 16 of the K extent, in 16-byte units
          const uint32_t idm = is_dq ? idesc_k : idesc_mn, idt = is_dq ? idesc_k_tail : idesc_mn_tail;
          for (int i = 0; i < items && ok; ++i) {
            ok = mbar_wait_cluster(bar(Cfg::B_FULL + slot), phase, wc);
            if (!ok) break;
            tc_fence_after();
            const uint64_t at = (uint64_t)(slot * (Cfg::SLOT_BYTES >> 4));
#pragma unroll
            for (int ks = 0; ks < 8; ++ks)
              umma2_ss(tmem, dA + at + stepA * ks, dB + at + (uint64_t)(128 * ks), idm, (i | ks) ? 1u : 0u);
            if (Cfg::TAIL && tail) {
#pragma unroll
              for (int ks = 0; ks < 8; ++ks)
                umma2_ss(tmem + 256u, dA + at + stepA * ks, dT + at + (uint64_t)(64 * ks), idt, (i | ks) ? 1u : 0u);
            }
            tc2_commit_both(bar(Cfg::B_EMPTY + slot));
            if (++slot == Cfg::NSTAGE) { slot = 0; phase ^= 1u; }
          }
          if (ok) tc2_commit_both(bar(Cfg::B_ACC));
        }
      }
      __syncwarp();
    }
  }

  // =========================== teardown ===========================
  tc_fence_before();
  __syncthreads();
  if (misc[4] != 0) {
    const uint64_t t_end = global_timer_ns() + 200000ull;
    while (global_timer_ns() < t_end) __nanosleep(1000);
    if (tid == 0) atomicExch(&g_bwd_pair_status, FM_ERR_TIMEOUT);
  }
  __syncwarp();
  cluster_sync_all();
  tc_fence_after();
  if (warp == 9) tmem2_dealloc(tmem, 512);
}

// ---------------------------------------------------------------------------
// host
// ---------------------------------------------------------------------------
// Bytes of P and dS a call keeps at a time when the caller gives what it is asked for; with less it works in smaller
// chunks (see bwd_pair_plan).  At S = 16384 that is two heads, or 2048 rows of 16 heads: enough
// tiles for 74 pairs several times over, so a larger budget gains nothing, and each chunk still reads dK / dV
// sums (if any) for 2048 rows of work.
constexpr size_t kBudget = (size_t)2 << 30;

struct BwdPairPlan { int groups, rows, key_blocks; bool sums; size_t block_bytes, acc_dk_bytes, acc_dv_bytes; };
// The plan with up to `budget` bytes of P and dS (at least 256 rows of a group).
static BwdPairPlan bwd_pair_plan_for(const fm_attn_args* a, size_t budget) {
  BwdPairPlan pl;
  const int G = a->Hq / a->Hkv;
  const size_t sq = ((size_t)a->Sq + 255) / 256 * 256, sk = ((size_t)a->Sk + 255) / 256 * 256;
  const size_t row = (size_t)G * sk * 4;              // P and dS of one query row of every head of a group
  pl.key_blocks = (int)(sk / 64);
  pl.groups = (int)std::min<size_t>((size_t)a->B * a->Hkv, std::max<size_t>(1, budget / (row * sq)));
  pl.rows = (int)std::min(sq, std::max<size_t>(256, budget / row / 256 * 256));
  pl.sums = (size_t)pl.rows < sq;
  pl.block_bytes = (size_t)pl.groups * pl.rows * row / 2;
  pl.acc_dk_bytes = pl.sums ? sk * a->d * 4 : 0;
  pl.acc_dv_bytes = pl.sums ? sk * a->dv * 4 : 0;
  return pl;
}
static size_t plan_bytes(const BwdPairPlan& pl) { return 2 * pl.block_bytes + pl.acc_dk_bytes + pl.acc_dv_bytes; }

// The largest plan that fits `bytes` of workspace; false: not even 256 rows of one group do.
static bool bwd_pair_plan(const fm_attn_args* a, size_t bytes, BwdPairPlan* pl) {
  *pl = bwd_pair_plan_for(a, kBudget);
  if (plan_bytes(*pl) <= bytes) return true;
  *pl = bwd_pair_plan_for(a, bytes);                  // whole groups
  if (plan_bytes(*pl) <= bytes) return true;
  const size_t sums = (((size_t)a->Sk + 255) / 256 * 256) * (a->d + a->dv) * 4;
  if (bytes <= sums) return false;
  *pl = bwd_pair_plan_for(a, bytes - sums);           // rows of one group beside its sums
  return plan_bytes(*pl) <= bytes;
}

bool bwd_pair_supported(const fm_attn_args* a) {
  // (a size query comes before the arguments are validated)
  if (!pair_dims(a->d, a->dv) || a->Sq <= 0 || a->Sk <= 0 || a->Hkv <= 0 || a->Hq <= 0 || a->Hq % a->Hkv) return false;
  // Sequences of one 64-row tile: a 256 x 256 tile of the score kernel is mostly padding.  64 x 64 rows with 16 heads,
  // backward: 256 / 256 warp-MMA 162 us against 230, 576 / 512 266 against 322; 64 x 100 rows at 256 351 against 264.
  // With few kv heads the warp-MMA kernels leave the chip idle (8 x 64 rows, 16 / 4 heads: 40 us, pair 36).
  if (a->Sq <= 64 && a->Sk <= 64 && a->B * a->Hkv >= 16 * std::min(a->Hq / a->Hkv, 4)) return false;
  // a chunk is at least 256 rows of every head of one group; past four budgets the warp-MMA kernels, which need no
  // workspace, keep the call
  const size_t least = (size_t)(a->Hq / a->Hkv) * (((size_t)a->Sk + 255) / 256 * 256) * 4 * 256;
  return (a->Sk + 127) / 128 <= kPairListMax && (a->Sq + 127) / 128 <= kPairListMax && least <= 4 * kBudget;
}

size_t bwd_pair_workspace_bytes(const fm_attn_args* a) { return plan_bytes(bwd_pair_plan_for(a, kBudget)); }
bool bwd_pair_fits(const fm_attn_args* a, size_t bytes) { BwdPairPlan pl; return bwd_pair_plan(a, bytes, &pl); }

static int make_block_tmap(CUtensorMap* out, void* base, size_t bytes) {
  EncodeTiledFn enc = get_encode_tiled();
  FM_REQUIRE(enc != nullptr, FM_ERR_CUDA, "cuTensorMapEncodeTiled is not available from the driver");
  const cuuint64_t dims[2] = {64, (cuuint64_t)(bytes / 128)};
  const cuuint64_t strides[1] = {128};
  const cuuint32_t box[2] = {64, 128}, estr[2] = {1, 1};
  const CUresult r = enc(out, CU_TENSOR_MAP_DATA_TYPE_UINT16, 2, base, dims, strides, box, estr,
                         CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                         CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  FM_REQUIRE(r == CUDA_SUCCESS, FM_ERR_CUDA, "cuTensorMapEncodeTiled (P / dS blocks) failed with CUresult %d", (int)r);
  return FM_OK;
}

template <int D, int DV, bool IS_BF16>
static int launch_bwd_pair(const AttnKParams& p, const fm_attn_args* a, uint8_t* ws, const BwdPairPlan& pl, cudaStream_t s) {
  using GC = PairGradCfg<D, DV>;
  const int G = a->Hq / a->Hkv;
  CUtensorMap q, dO, k, v, qt, kt, tp, tds;
  int rc;
#define FM_TMAP(out, ptr, S, H, Dm, st) \
  if ((rc = make_bshd_tmap(&out, ptr, a->dtype, a->B, S, H, Dm, st[0], st[1], st[2], 128))) return rc;
  FM_TMAP(q, a->q, a->Sq, a->Hq, a->d, a->q_stride)
  FM_TMAP(dO, a->d_o, a->Sq, a->Hq, a->dv, a->do_stride)
  FM_TMAP(k, a->k, a->Sk, a->Hkv, a->d, a->k_stride)
  FM_TMAP(v, a->v, a->Sk, a->Hkv, a->dv, a->v_stride)
#undef FM_TMAP
  if ((rc = make_bshd_tmap(&qt, a->q, a->dtype, a->B, a->Sq, a->Hq, a->d, a->q_stride[0], a->q_stride[1], a->q_stride[2], 128, 32))) return rc;
  if ((rc = make_bshd_tmap(&kt, a->k, a->dtype, a->B, a->Sk, a->Hkv, a->d, a->k_stride[0], a->k_stride[1], a->k_stride[2], 128, 32))) return rc;
  if ((rc = make_block_tmap(&tp, ws, pl.block_bytes))) return rc;
  if ((rc = make_block_tmap(&tds, ws + pl.block_bytes, pl.block_bytes))) return rc;
  auto k1 = bwd_pair_scores_kernel<D, DV, IS_BF16>;
  auto k2 = bwd_pair_grads_kernel<D, DV, IS_BF16>;
  FM_CUDA_TRY(cudaFuncSetAttribute(k1, cudaFuncAttributeMaxDynamicSharedMemorySize, PairScoreCfg::SMEM));
  FM_CUDA_TRY(cudaFuncSetAttribute(k2, cudaFuncAttributeMaxDynamicSharedMemorySize, GC::SMEM));
  int dev = 0, n_sm = 0;
  FM_CUDA_TRY(cudaGetDevice(&dev));
  FM_CUDA_TRY(cudaDeviceGetAttribute(&n_sm, cudaDevAttrMultiProcessorCount, dev));
  const int pairs = n_sm / 2;
  const int n_tiles256 = (a->Sk + 255) / 256;
  BwdPairChunk c;
  c.ws_p = reinterpret_cast<uint4*>(ws);
  c.ws_ds = reinterpret_cast<uint4*>(ws + pl.block_bytes);
  c.acc_dk = reinterpret_cast<float*>(ws + 2 * pl.block_bytes);
  c.acc_dv = reinterpret_cast<float*>(ws + 2 * pl.block_bytes + pl.acc_dk_bytes);
  c.key_blocks = pl.key_blocks;
  const int all_groups = a->B * a->Hkv;
  for (int g0 = 0; g0 < all_groups; g0 += pl.groups)
    for (int row0 = 0; row0 < a->Sq; row0 += pl.rows) {
      const int groups = std::min(pl.groups, all_groups - g0);
      const int rows = (std::min(pl.rows, a->Sq - row0) + 255) / 256 * 256;
      c.head0 = g0 * G; c.heads = groups * G; c.row0 = row0; c.row_blocks = rows / 128;
      c.first = row0 == 0; c.last = row0 + pl.rows >= a->Sq;
      // about eight units per pair: the last round of units is then a small part of the launch
      const int blocks = c.heads * c.row_blocks / 2;
      c.n_seg = std::max(1, std::min(n_tiles256, (8 * pairs + blocks / 2) / blocks));
      c.n_units = blocks * c.n_seg;
      c.n_dk = groups * n_tiles256 * GC::NS_D;
      c.n_dv = groups * n_tiles256 * GC::NS_V;
      c.n_dq = blocks * GC::NS_D;
      k1<<<2 * std::min(pairs, c.n_units), 384, PairScoreCfg::SMEM, s>>>(q, dO, k, v, p, c);
      FM_CUDA_TRY(cudaGetLastError());
      k2<<<2 * std::min(pairs, c.n_dk + c.n_dv + c.n_dq), 384, GC::SMEM, s>>>(tp, tds, q, dO, k, qt, kt, p, c);
      FM_CUDA_TRY(cudaGetLastError());
      count_launches(2);
    }
  return FM_OK;
}

int bwd_pair_launch(const AttnKParams& p, const fm_attn_args* a, void* ws, size_t bytes, cudaStream_t s) {
  BwdPairPlan pl;
  FM_REQUIRE(bwd_pair_plan(a, bytes, &pl), FM_ERR_WORKSPACE, "backward: %zu bytes hold no chunk of P and dS", bytes);
  const bool bf = a->dtype == FM_DTYPE_BF16;
  uint8_t* w = reinterpret_cast<uint8_t*>(ws);
  if (a->d == 256) return bf ? launch_bwd_pair<256, 256, true>(p, a, w, pl, s) : launch_bwd_pair<256, 256, false>(p, a, w, pl, s);
  if (a->d == 512) return bf ? launch_bwd_pair<512, 512, true>(p, a, w, pl, s) : launch_bwd_pair<512, 512, false>(p, a, w, pl, s);
  return bf ? launch_bwd_pair<576, 512, true>(p, a, w, pl, s) : launch_bwd_pair<576, 512, false>(p, a, w, pl, s);
}

int bwd_pair_status(int* out, bool reset) {
  int v = 0;
  FM_CUDA_TRY(cudaMemcpyFromSymbol(&v, g_bwd_pair_status, sizeof(int)));
  if (reset && v != 0) {
    const int z = 0;
    FM_CUDA_TRY(cudaMemcpyToSymbol(g_bwd_pair_status, &z, sizeof(int)));
  }
  *out = v;
  return FM_OK;
}

}  // namespace fm
