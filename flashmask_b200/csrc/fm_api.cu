// extern "C" entry points: argument validation, kernel-variant selection,
// workspace carving.  No allocation, no host synchronisation.
#include <algorithm>
#include <atomic>
#include <cstdarg>
#include <cstdlib>
#include <cstring>

#include "fm_attn_params.cuh"

namespace fm {

static thread_local char g_err[512] = "";

void set_error(const char* fmt, ...) {
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(g_err, sizeof(g_err), fmt, ap);
  va_end(ap);
}

int sm_count() {
  static std::atomic<int> cached[64];        // zero-initialised: 0 = not asked yet
  int dev = 0, n = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 148;
  if (dev < 64 && (n = cached[dev].load(std::memory_order_relaxed)) > 0) return n;
  if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) return 148;
  if (dev < 64) cached[dev].store(n, std::memory_order_relaxed);
  return n;
}

static std::atomic<unsigned long long> g_launches{0};
void count_launches(int n) { g_launches.fetch_add((unsigned long long)n, std::memory_order_relaxed); }

int cuda_fail(cudaError_t e, const char* what) {
  set_error("CUDA error %d (%s) at %s", (int)e, cudaGetErrorString(e), what);
  return FM_ERR_CUDA;
}

// implemented in the kernel translation units
int fwd_mma_tile_shape(int d, int dv, int* tile_m, int* tile_n);
int fwd_mma_launch(const AttnKParams& p, int dtype, cudaStream_t s);
int bwd_mma_tile_shape(int d, int dv, int* tile_m, int* tile_n);
int bwd_mma_launch(const AttnKParams& p, int dtype, cudaStream_t s);
int bwd_preprocess_launch(const AttnKParams& p, int dtype, cudaStream_t s);
int bwd_dsink_launch(const AttnKParams& p, cudaStream_t s);
int fwd_sm100_launch(const AttnKParams& p, const fm_attn_args* a, cudaStream_t s);
size_t fwd_sm100_workspace_bytes(const fm_attn_args* a);
int bwd_sm100_launch(const AttnKParams& p, const fm_attn_args* a, cudaStream_t s);
int bwd_sm100_persist_launch(const AttnKParams& p, const fm_attn_args* a, cudaStream_t s);
int bwd_sm100_fused_launch(const AttnKParams& p, const fm_attn_args* a, cudaStream_t s);
int bwd_sm100_fused_status(int* out, bool reset);
size_t bwd_sm100_fused_accum_bytes(const fm_attn_args* a);
int bwd_sm100_persist_status(int* out, bool reset);
size_t bwd_sm100_workspace_bytes(const fm_attn_args* a);

bool fwd_pair_supported(const fm_attn_args* a);
int fwd_pair_launch(const AttnKParams& p, const fm_attn_args* a, cudaStream_t s);
int fwd_pair_status(int* out, bool reset);
bool bwd_pair_supported(const fm_attn_args* a);
size_t bwd_pair_workspace_bytes(const fm_attn_args* a);
bool bwd_pair_fits(const fm_attn_args* a, size_t bytes);
int bwd_pair_launch(const AttnKParams& p, const fm_attn_args* a, void* ws, size_t bytes, cudaStream_t s);
int bwd_pair_status(int* out, bool reset);

int fwd_sm100_status(int* out, bool reset);
int bwd_sm100_status(int* out, bool reset);
int bounded_wait_selftest_launch(uint64_t budget_ns, cudaStream_t s);

static inline int round_up(int x, int m) { return (x + m - 1) / m * m; }

// A/B switches, read from the environment ONCE when the library is loaded (and again only when
// the host asks through fm_reload_options): no entry point touches the environment per call.
//   FLASHMASK_B200_FWD=mma       forward on the warp-MMA kernels for every head dim
//   FLASHMASK_B200_BWD=mma       backward on the warp-MMA kernels for every head dim
//   FLASHMASK_B200_BWD=split     tcgen05 backward as two kernels (dK/dV + dQ) even when the call
//                                did not ask for deterministic gradients
//   FLASHMASK_B200_PERSIST=0     tcgen05 backward: one unit per CTA even with launch tables
//   FLASHMASK_B200_CLASSES=n     work classes of the launch tables (1..8)
struct Options { bool fwd_mma, bwd_mma, bwd_split, bwd_persist; int order_classes; };
static Options read_options() {
  Options o{false, false, false, true, 0};
  if (const char* e = getenv("FLASHMASK_B200_FWD")) o.fwd_mma = strcmp(e, "mma") == 0;
  if (const char* e = getenv("FLASHMASK_B200_BWD")) { o.bwd_mma = strcmp(e, "mma") == 0; o.bwd_split = strcmp(e, "split") == 0; }
  if (const char* e = getenv("FLASHMASK_B200_PERSIST")) o.bwd_persist = !(e[0] == '0' && e[1] == 0);
  if (const char* e = getenv("FLASHMASK_B200_CLASSES")) o.order_classes = atoi(e);
  return o;
}
static Options g_opt = read_options();
int option_order_classes() { return g_opt.order_classes; }

// Kernel variant of the forward for (d, dv): the tcgen05 kernels cover head dims up to 128 (multiples of 8),
// 192 / 128 and, on CTA pairs, 256, 512 and 576 / 512; FLASHMASK_B200_FWD=mma forces the warp-MMA variant (A/B runs).
static bool fwd_uses_sm100(int d, int dv) {
  const bool small = d <= 128 && dv <= 128 && d % 8 == 0 && dv % 8 == 0;
  if (!small && !(d == 192 && dv == 128) && !pair_dims(d, dv)) return false;
  return !g_opt.fwd_mma;
}

static bool stride_ok(const int64_t* s) { return s[0] % 8 == 0 && s[1] % 8 == 0 && s[2] % 8 == 0; }

// What the tcgen05 kernels ask of a call; the warp-MMA kernels serve the others.
// They read q, k, v and d_o through tensor maps, which have no stride 0: a tensor that repeats along a dimension (an
// expanded batch, one key head shown as several) needs computed addresses.  (The torch hosts copy such a tensor
// instead and keep the faster kernels.)
// They mask a score with -inf and take the row maximum before the scale is applied, which needs a positive scale.
static bool mappable(const int64_t* s, int B, int S, int H) {
  return (B == 1 || s[0] > 0) && (S == 1 || s[1] > 0) && (H == 1 || s[2] > 0);
}
static bool fits_tcgen05(const fm_attn_args* a, bool backward) {
  return a->softmax_scale > 0.f && mappable(a->q_stride, a->B, a->Sq, a->Hq) &&
         mappable(a->k_stride, a->B, a->Sk, a->Hkv) && mappable(a->v_stride, a->B, a->Sk, a->Hkv) &&
         (!backward || mappable(a->do_stride, a->B, a->Sq, a->Hq));
}

static int validate_common(const fm_attn_args* a, const char* who) {
  FM_REQUIRE(a != nullptr, FM_ERR_INVALID_ARGUMENT, "%s: args is NULL", who);
  FM_REQUIRE(a->B > 0 && a->Sq > 0 && a->Sk > 0 && a->Hq > 0 && a->Hkv > 0, FM_ERR_INVALID_ARGUMENT,
             "%s: B/Sq/Sk/Hq/Hkv must be positive", who);
  FM_REQUIRE(a->Hq % a->Hkv == 0, FM_ERR_INVALID_ARGUMENT, "%s: Hq (%d) must be a multiple of Hkv (%d)",
             who, a->Hq, a->Hkv);
  FM_REQUIRE(a->d > 0 && a->dv > 0 && a->d % 8 == 0 && a->dv % 8 == 0, FM_ERR_INVALID_ARGUMENT,
             "%s: head dims must be positive multiples of 8 (d=%d, dv=%d)", who, a->d, a->dv);
  FM_REQUIRE(a->dtype == FM_DTYPE_BF16 || a->dtype == FM_DTYPE_FP16, FM_ERR_INVALID_ARGUMENT,
             "%s: dtype must be FM_DTYPE_BF16 or FM_DTYPE_FP16", who);
  FM_REQUIRE(a->q && a->k && a->v && a->o && a->lse, FM_ERR_INVALID_ARGUMENT,
             "%s: q/k/v/o/lse must not be NULL", who);
  FM_REQUIRE(stride_ok(a->q_stride) && stride_ok(a->k_stride) && stride_ok(a->v_stride) &&
                 stride_ok(a->o_stride),
             FM_ERR_INVALID_ARGUMENT, "%s: strides must be multiples of 8 elements (16-byte rows)", who);
  FM_REQUIRE(a->ncols == 0 || a->ncols == 1 || a->ncols == 2 || a->ncols == 4, FM_ERR_INVALID_ARGUMENT,
             "%s: ncols must be 0, 1, 2 or 4", who);
  if (a->ncols) {
    FM_REQUIRE(a->mask && a->minmax, FM_ERR_INVALID_ARGUMENT, "%s: mask given but mask/minmax is NULL", who);
    FM_REQUIRE(((uintptr_t)a->minmax & 15) == 0, FM_ERR_INVALID_ARGUMENT, "%s: minmax must be 16-byte aligned", who);
    FM_REQUIRE(a->Hm == 1 || a->Hm == a->Hkv, FM_ERR_INVALID_ARGUMENT,
               "%s: mask heads (%d) must be 1 or Hkv", who, a->Hm);
    FM_REQUIRE(a->mask_B == a->B || a->mask_B == 1, FM_ERR_INVALID_ARGUMENT,
               "%s: mask batch (%d) must be B or 1", who, a->mask_B);
    FM_REQUIRE(!(a->ncols == 1 && !a->causal) && !(a->ncols == 4 && a->causal), FM_ERR_INVALID_ARGUMENT,
               "%s: ncols=%d is not defined for causal=%d", who, a->ncols, a->causal);
  }
  return FM_OK;
}

int fill_kparams(const fm_attn_args* a, AttnKParams* p, bool backward) {
  memset(p, 0, sizeof(*p));
  p->q = a->q; p->k = a->k; p->v = a->v; p->o = a->o; p->lse = a->lse; p->sink = a->sink;
  p->q_b = a->q_stride[0]; p->q_s = a->q_stride[1]; p->q_h = a->q_stride[2];
  p->k_b = a->k_stride[0]; p->k_s = a->k_stride[1]; p->k_h = a->k_stride[2];
  p->v_b = a->v_stride[0]; p->v_s = a->v_stride[1]; p->v_h = a->v_stride[2];
  p->o_b = a->o_stride[0]; p->o_s = a->o_stride[1]; p->o_h = a->o_stride[2];
  p->B = a->B; p->Sq = a->Sq; p->Sk = a->Sk; p->Hq = a->Hq; p->Hkv = a->Hkv;
  p->d = a->d; p->dv_dim = a->dv;
  p->Sq_r = round_up(a->Sq, 128);
  p->scale = a->softmax_scale;
  p->scale_log2 = a->softmax_scale * kLog2e;
  p->md.mask = a->ncols ? a->mask : nullptr;
  p->md.minmax = a->ncols ? a->minmax : nullptr;
  p->md.ncols = a->ncols; p->md.causal = a->causal; p->md.Hm = a->ncols ? a->Hm : 1;
  p->md.mask_B = a->ncols ? a->mask_B : 1;
  p->md.nblk_pad = fm_mask_nblk_pad(a->Sk, a->tile_n > 0 ? a->tile_n : 64);
  p->md.BHm = p->md.mask_B * p->md.Hm;
  p->md.Sq = a->Sq; p->md.Sk = a->Sk;
  p->mask_tile = a->ncols ? a->tile_n : 0;
  if (a->ncols) { p->fwd_order = a->fwd_order; p->dq_order = a->dq_order; p->dkdv_order = a->dkdv_order; }
  if (backward) {
    p->d_o = a->d_o; p->dq = a->dq; p->dk = a->dk; p->dv = a->dv_out; p->dsink = a->dsink;
    p->do_b = a->do_stride[0]; p->do_s = a->do_stride[1]; p->do_h = a->do_stride[2];
    p->dq_b = a->dq_stride[0]; p->dq_s = a->dq_stride[1]; p->dq_h = a->dq_stride[2];
    p->dk_b = a->dk_stride[0]; p->dk_s = a->dk_stride[1]; p->dk_h = a->dk_stride[2];
    p->dv_b = a->dv_stride[0]; p->dv_s = a->dv_stride[1]; p->dv_h = a->dv_stride[2];
  }
  return FM_OK;
}

}  // namespace fm

using namespace fm;

extern "C" const char* fm_version(void) { return "flashmask_b200 0.1.0 sm_100a"; }
extern "C" const char* fm_last_error(void) { return g_err; }

extern "C" unsigned long long fm_launch_count(void) { return g_launches.load(std::memory_order_relaxed); }

extern "C" int fm_reload_options(void) {
  g_opt = read_options();
  return FM_OK;
}

static bool bwd_uses_sm100(int d, int dv) {
  const bool small = d <= 128 && dv <= 128 && d % 8 == 0 && dv % 8 == 0;
  if (!small && !(d == 192 && dv == 128)) return false;
  return !g_opt.bwd_mma;
}

// Kernel family of a backward call.
// The one-kernel backward (five GEMMs per tile pair, dQ summed into an fp32 accumulator in an order
// that is not fixed) serves the tcgen05 head dims whenever the call does not ask for deterministic
// gradients; the two-kernel variant gives every output element one owner and a fixed order.
// Forward + backward of 8192 to 131072 tokens, masks and full tiles, takes 1.15 to 1.33 times as long with the two kernels at d = dv = 64
// and d = dv = 128 (backward alone 1.20 to 1.55).  Head dims between them run it too where
// one_kernel_pays (the GEMMs stop at the end of a head).
// The CTA-pair backward (256, 512, 576 / 512) keeps P and dS of a chunk of query rows in the caller's workspace;
// without one (fm_bwd_static_scratch) and past its index range the warp-MMA kernels serve these head dims.
enum BwdKernels { BWD_ONE_KERNEL, BWD_TWO_KERNELS, BWD_PAIR, BWD_WARP_MMA };
// Head dims that the one-kernel backward serves whatever the sizes: calls over the same queries may share its accumulator.
static bool bwd_fills_boxes(const fm_attn_args* a) { return a->d == a->dv && (a->d == 64 || a->d == 128); }
// Head dims between 64 and 128.  A unit of the one kernel is a key tile of a kv head with every q head of its group (G), and
// does five GEMMs an item; the two kernels do seven, but spread three of them over the q heads.  So the one kernel needs
// units that fill the chip evenly and rows enough in each to pay for its accumulator (512 bytes a query row, cleared, added
// to and rounded).  The lines were drawn for a form of the one kernel that took 5 to 6 % longer (one buffer of scores), each where it began to
// lose; with the present form most of them lie on the safe side.  Forward + backward in us, two kernels -> one, present form, documents and d = 96
// unless said, (units), inputs changing from pass to pass; after "below" calls that the rule leaves to the two kernels:
//   masks.  A long document is a run of long units in every kv head that shares the mask ("copies"); with few copies and
//   few units the chip waits for them, the more the wider the head:
//     6 copies and more, 2 units an SM: 4800, 32 / 8 heads (304) 416 -> 352, 2432, 16 / 16 (304) 130 -> 114
//     3 to 5, 2.5: 17100, 48 / 3 (402) d = 120 2314 -> 2348; below 12763, 24 / 3 (300) 843 -> 740, 9563, 16 / 4 (300) 452 -> 390, d = 80 442 -> 366,
//       d = 120 495 -> 457, 2 x 3001, 16 / 4 (192) 252 -> 244, 3001, 16 / 4 (96) 189 -> 189
//     2, 3: 28763, 8 / 2 (450) 608 -> 510, 32000, 8 / 2 (500) d = 120 782 -> 728; below 25563, 8 / 2 (400) d = 120 570 -> 525, 19163 (300) 418 -> 374,
//       32 / 2 1592 -> 1511
//     1, 4: 76763, 4 / 1 (600) 1276 -> 1109; below 57563, 4 / 1 (450) 1092 -> 974, 4 x 10000, 4 / 1 (316) 525 -> 530
//   short rows: 5 x 1000, 8 / 8 117 -> 101; below 16 x 640, 16 / 16 262 -> 250, 64 x 256, 16 / 16 303 -> 309, 64 x 200, 16 / 4 252 -> 253
//   and an accumulator past L2: 12 x 520, 32 / 8 (126 MB) 315 -> 291; below 64 x 512, 16 / 4 (268 MB) 596 -> 613
// Without a mask units are even, and the two kernels walk no tables:
//   G >= 4, any length: 64 x 100, 32 / 8 causal 242 -> 224, 40 x 64, 64 / 8 214 -> 181, 4800 full, 32 / 8 1699 -> 1438; below two units an SM
//     2 x 1300 causal, 64 / 8 (176) d = 72 442 -> 397, 2000 causal, 16 / 4 (64) d = 120 202 -> 231
//   G < 4: 8 x 1280 causal, 16 / 16 (1280) 374 -> 331; below 64 x 256 causal, 16 / 16 334 -> 327, 128 x 256 full d = 120 733 -> 744,
//     12000 full, 4 / 2 (188) d = 80 1317 -> 1168
//   G = 1 in less than three waves, where the last is nearly empty: 2432 causal, 16 / 16 (304) 173 -> 157; below 5 x 1000 causal, 8 / 8 (320)
//     112 -> 108, 4 x 1280 full, 8 / 8 (320) d = 120 184 -> 179, 4000 full, 8 / 8 (256) 296 -> 236
static bool one_kernel_pays(const fm_attn_args* a) {
  if (a->Hkv <= 0 || a->Sk <= 0 || a->Hq < a->Hkv) return false;
  const int64_t units = (int64_t)a->Hkv * a->B * ((a->Sk + 127) / 128), sms = sm_count();
  const int64_t G = a->Hq / a->Hkv, rows = G * a->Sq;
  if (a->ncols == 0) return units >= 2 * sms && (G >= 4 || (rows >= 896 && (G >= 2 || a->Sq >= 2048 || units >= 3 * sms)));
  const int64_t copies = (int64_t)(a->Hm > 1 ? 1 : a->Hkv) * (a->mask_B == 1 ? a->B : 1);
  return 2 * units >= (copies >= 6 ? 4 : copies >= 3 ? 5 : copies == 2 ? 6 : 8) * sms && rows >= 896 &&
         (a->Sq >= 896 || bwd_sm100_fused_accum_bytes(a) <= (size_t)126000000);
}
// By geometry and options alone: what the workspace is sized for.
static BwdKernels bwd_kernels_by_geometry(const fm_attn_args* a) {
  if (bwd_uses_sm100(a->d, a->dv)) {
    const bool one = bwd_fills_boxes(a) || (a->d == a->dv && a->d > 64 && one_kernel_pays(a));
    return one && !a->deterministic && !g_opt.bwd_split ? BWD_ONE_KERNEL : BWD_TWO_KERNELS;
  }
  return pair_dims(a->d, a->dv) && !g_opt.bwd_mma && bwd_pair_supported(a) ? BWD_PAIR : BWD_WARP_MMA;
}
static BwdKernels bwd_kernels(const fm_attn_args* a) {
  const BwdKernels k = fits_tcgen05(a, true) ? bwd_kernels_by_geometry(a) : BWD_WARP_MMA;
  // the one-kernel backward divides LSE by the scale: both stay far inside fp32
  return k == BWD_ONE_KERNEL && a->softmax_scale < 0x1p-100f ? BWD_TWO_KERNELS : k;
}

// preprocess -> main kernels of the selected variant -> dsink, on one stream
static int run_bwd_kernels(const fm_attn_args* a, BwdKernels kernels, const AttnKParams& p, cudaStream_t s) {
  FM_REQUIRE((((uintptr_t)a->q | (uintptr_t)a->k | (uintptr_t)a->v | (uintptr_t)a->d_o) & 15) == 0,
             FM_ERR_INVALID_ARGUMENT, "backward: q/k/v/d_o must be 16-byte aligned");
  int rc = bwd_preprocess_launch(p, a->dtype, s);
  if (rc != FM_OK) return rc;
  if (kernels == BWD_ONE_KERNEL || kernels == BWD_TWO_KERNELS) {
    if (p.dq_accum) {
      rc = bwd_sm100_fused_launch(p, a, s);
      if (rc != FM_OK) return rc;
      if (a->sink) rc = bwd_dsink_launch(p, s);
      return rc;
    }
    // With launch tables (a mask tensor) the persistent variant walks them; without, one unit per CTA.
    // Measured on six 8K-32K masks the persistent variant is 3-14 % faster where units are short
    // (documents, windows) and 3-5 % slower where every unit is hundreds of items long (its main loop
    // is slightly slower; the table records in [E+2] which side of that line a mask is on).
    // FLASHMASK_B200_PERSIST=0 keeps the one-unit-per-CTA variant.
    // (Without tables the persistent kernels also work, one unit per CTA, bitwise the same; measured on dense
    // masks they are 5-12 % slower than the one-unit kernels, which is why both exist.)
    const bool persist = p.dq_order && p.dkdv_order && g_opt.bwd_persist && a->d <= 128;   // 192 / 128: one-unit kernels only
    rc = persist ? bwd_sm100_persist_launch(p, a, s) : bwd_sm100_launch(p, a, s);
  } else if (p.pair_ws) {
    rc = bwd_pair_launch(p, a, p.pair_ws, p.pair_ws_bytes, s);
  } else {
    rc = bwd_mma_launch(p, a->dtype, s);
  }
  if (rc != FM_OK) return rc;
  if (a->sink) rc = bwd_dsink_launch(p, s);
  return rc;
}

extern "C" int fm_fwd_tile_shape(int d, int dv, int* tile_m, int* tile_n) {
  FM_REQUIRE(tile_m && tile_n, FM_ERR_INVALID_ARGUMENT, "fm_fwd_tile_shape: NULL output");
  if (fwd_uses_sm100(d, dv)) { *tile_m = 128; *tile_n = 128; return FM_OK; }
  int rc = fwd_mma_tile_shape(d, dv, tile_m, tile_n);
  if (rc != FM_OK) set_error("fm_fwd_tile_shape: unsupported head dims (d=%d, dv=%d)", d, dv);
  return rc;
}

extern "C" int fm_bwd_tile_shape(int d, int dv, int* tile_m, int* tile_n) {
  FM_REQUIRE(tile_m && tile_n, FM_ERR_INVALID_ARGUMENT, "fm_bwd_tile_shape: NULL output");
  if (bwd_uses_sm100(d, dv)) { *tile_m = 64; *tile_n = 128; return FM_OK; }
  if (pair_dims(d, dv) && !g_opt.bwd_mma) { *tile_m = 128; *tile_n = 128; return FM_OK; }
  int rc = bwd_mma_tile_shape(d, dv, tile_m, tile_n);
  if (rc != FM_OK) set_error("fm_bwd_tile_shape: unsupported head dims (d=%d, dv=%d)", d, dv);
  return rc;
}

// Kernel family of a forward at 256, 512 or 576 / 512.
//
// The CTA-pair kernel works on blocks of 256 rows, one block on two SMs: it is the fastest wherever blocks are full,
// and up to four times slower than smaller blocks on batches of short sequences.  There the one-CTA kernel (256, blocks
// of 128 rows) or the warp-MMA kernel (512 and 576, blocks of 64) serves.  The family follows from an estimate of both
// launches in microseconds, the longer of the longest block and waves x the average block, fitted to 976 calls of 1 to
// 64 sequences of 32 to 1024 rows, and of 1 to 128 rows against up to 8192 keys (16 heads, causal and full):
//   64 x 64 rows, 576 / 512 causal    pair 276 us, warp-MMA 105    64 x 128 rows, 256 full    pair 131 us, one CTA 65
//   64 x 128 rows, 576 / 512 full     pair 293 us, warp-MMA 312    32 x 512 rows, 256 full    pair 188 us, one CTA 258
//   8 x 16 rows of 1024 keys, 256, 16 / 4 heads  pair 35, one CTA 27;  8 x 1 row of 8192 keys  pair 173, one CTA 202
// Within 3 %, and past 2048 rows, the pair kernel is kept.
enum FwdWide { FWD_PAIR, FWD_ONE_CTA, FWD_WARP_MMA };
static double fwd_launch_us(const fm_attn_args* a, int rows, int keys, int units, int slots, double fixed, double per_tile) {
  const int n_blocks = (a->Sq + rows - 1) / rows, n_tiles = (a->Sk + keys - 1) / keys;
  int64_t sum = 0;
  int most = 0;
  for (int i = 0; i < n_blocks; ++i) {
    const int last = std::min((i + 1) * rows, a->Sq) + a->Sk - a->Sq;      // keys the block's last row sees
    const int n = a->causal ? std::max(0, std::min(n_tiles, (last + keys - 1) / keys)) : n_tiles;
    sum += n;
    most = std::max(most, n);
  }
  const int64_t waves = ((int64_t)units * n_blocks + slots - 1) / slots;
  return std::max(fixed + per_tile * most, waves * (fixed + per_tile * sum / n_blocks));
}
static FwdWide fwd_wide_kernels(const fm_attn_args* a) {
  if (!fwd_pair_supported(a)) return FWD_WARP_MMA;
  if (a->Sq > 2048) return FWD_PAIR;
  const int n_sm = sm_count(), units = a->B * a->Hq;
  if (a->d == 256) {
    const double pair = fwd_launch_us(a, 256, 128, units, n_sm / 2, a->causal ? 11.8 : 10.5, 0.95);
    return fwd_launch_us(a, 128, 128, units, n_sm, 6.4, 3.2) < 0.97 * pair ? FWD_ONE_CTA : FWD_PAIR;
  }
  const double pair = fwd_launch_us(a, 256, 128, 2 * units, n_sm / 2, a->causal ? 9.2 : 7.8, 2.1);   // (two slices of V)
  return fwd_launch_us(a, 64, 32, units, n_sm, 3.3, 6.2) < 0.97 * pair ? FWD_WARP_MMA : FWD_PAIR;
}

// Side output of the forward (fm_fwd_block_score); block_logit == nullptr: none.
struct BlockScore { float* block_logit; const int32_t* block_bos; int block_size, block_ld; };

static int fwd_impl(const fm_attn_args* a, const BlockScore& bs, void* stream) {
  int rc = validate_common(a, "fm_fwd");
  if (rc != FM_OK) return rc;
  int tm, tn;
  rc = fm_fwd_tile_shape(a->d, a->dv, &tm, &tn);
  if (rc != FM_OK) return rc;
  FM_REQUIRE(a->ncols == 0 || a->tile_n == tn, FM_ERR_INVALID_ARGUMENT,
             "fm_fwd: minmax was prepared for tile_n=%d, this variant needs %d", a->tile_n, tn);
  AttnKParams p;
  fill_kparams(a, &p, false);
  p.md.nblk_pad = fm_mask_nblk_pad(a->Sk, tn);
  if (bs.block_logit) {
    FM_REQUIRE(bs.block_size == 32 || bs.block_size == 64 || bs.block_size == 128, FM_ERR_UNSUPPORTED,
               "fm_fwd_block_score: block_size must be 32, 64 or 128 (got %d)", bs.block_size);
    p.block_cols = (a->Sk + bs.block_size - 1) / bs.block_size;
    FM_REQUIRE(bs.block_ld >= p.block_cols, FM_ERR_INVALID_ARGUMENT,
               "fm_fwd_block_score: block_logit has %d blocks per row, ceil(Sk / block_size) = %d are needed",
               bs.block_ld, p.block_cols);
    p.block_logit = bs.block_logit; p.block_bos = bs.block_bos; p.block_ld = bs.block_ld;
    p.block_log2 = bs.block_size == 32 ? 5 : (bs.block_size == 64 ? 6 : 7);
  }
  cudaStream_t s = (cudaStream_t)stream;
  FM_REQUIRE((((uintptr_t)a->q | (uintptr_t)a->k | (uintptr_t)a->v) & 15) == 0, FM_ERR_INVALID_ARGUMENT,
             "forward: q/k/v must be 16-byte aligned");
  if (!fwd_uses_sm100(a->d, a->dv) || !fits_tcgen05(a, false)) return fwd_mma_launch(p, a->dtype, s);
  if (pair_dims(a->d, a->dv)) {
    const FwdWide kernels = fwd_wide_kernels(a);
    if (kernels == FWD_WARP_MMA) return fwd_mma_launch(p, a->dtype, s);
    if (kernels == FWD_PAIR) return fwd_pair_launch(p, a, s);
  }
  return fwd_sm100_launch(p, a, s);
}

extern "C" size_t fm_fwd_workspace_bytes(const fm_attn_args* a) {
  if (!a || a->B <= 0 || a->Hq <= 0 || a->Hkv <= 0 || a->Hq % a->Hkv || a->Sq <= 0 || a->Sk <= 0) return 0;
  return fwd_uses_sm100(a->d, a->dv) ? fwd_sm100_workspace_bytes(a) : 0;
}

extern "C" int fm_fwd(const fm_attn_args* a, void* stream) { return fwd_impl(a, BlockScore{}, stream); }

extern "C" int fm_fwd_block_score(const fm_attn_args* a, float* block_logit, int block_size, int block_ld,
                                  const int32_t* block_bos, void* stream) {
  FM_REQUIRE(block_logit != nullptr, FM_ERR_INVALID_ARGUMENT, "fm_fwd_block_score: block_logit is NULL");
  return fwd_impl(a, BlockScore{block_logit, block_bos, block_size, block_ld}, stream);
}

// Geometry of a launch order: the ordered axis, rows per unit, the block the work is
// counted in, and how often a unit repeats (heads per mask head, batches per mask batch).
// Only the tcgen05 variants read an order.
struct OrderGeom { int axis, block_rows, n_units, n_other, heads, rep_h, rep_b; int64_t E, n_cta; };
static bool order_geometry_any(const fm_attn_args* a, int which, OrderGeom* g) {
  if (!a || a->ncols == 0 || a->Sq <= 0 || a->Sk <= 0 || a->B <= 0 || a->Hq <= 0 || a->Hkv <= 0) return false;
  if (!(a->Hm == 1 || a->Hm == a->Hkv) || !(a->mask_B == 1 || a->mask_B == a->B) || a->Hq % a->Hkv) return false;
  const int nk = (a->Sk + 127) / 128;
  // (the forward takes no table at 256 and above; the 192-column backward runs the one-unit kernels, which take
  // none either)
  if (which == FM_ORDER_FWD) {
    if (!fwd_uses_sm100(a->d, a->dv) || a->d > 192) return false;
    *g = OrderGeom{0, 256, (a->Sq + 255) / 256, nk, a->Hq};
  } else if (which == FM_ORDER_BWD_DQ) {
    if (!bwd_uses_sm100(a->d, a->dv) || a->d > 128) return false;
    *g = OrderGeom{0, 128, (a->Sq + 127) / 128, nk, a->Hq};
  } else if (which == FM_ORDER_BWD_DKDV) {
    if (!bwd_uses_sm100(a->d, a->dv) || a->d > 128) return false;
    *g = OrderGeom{1, 64, nk, (a->Sq + 63) / 64, a->Hkv};
  } else {
    return false;
  }
  g->rep_h = g->heads / a->Hm;
  g->rep_b = a->B / a->mask_B;
  g->E = (int64_t)a->mask_B * a->Hm * g->n_units;
  g->n_cta = g->E * g->rep_h * g->rep_b;
  return g->E <= FM_ORDER_MAX_UNITS && g->n_cta < (1ll << 30);
}

static bool order_geometry(const fm_attn_args* a, int which, OrderGeom* g) {
  if (!order_geometry_any(a, which, g)) return false;
  // The backward kernels walk their table persistently (the next unit is fetched and its list
  // built while the current one is in its main loop), so a table never costs them a dependent
  // load on the critical path; the forward reads its entry at CTA start and gains wherever CTAs
  // differ in work.  All three are built whenever the geometry allows.
  return true;
}

extern "C" int64_t fm_launch_order_ints(const fm_attn_args* a, int which) {
  OrderGeom g;
  if (!order_geometry(a, which, &g)) return 0;
  return 2 * g.n_cta + 2 * g.E + 4;
}

// An order only matters where CTAs queue: when every CTA of a launch starts at once the table costs its launch
// (9 us, on the critical path of the forward) and changes nothing.  The two backward tables go together, since the
// persistent two-kernel backward walks both.  1024 rows, 2 heads, d = 64, forward + backward: 96 -> 91 us.
extern "C" int fm_launch_order_useful(const fm_attn_args* a, int which) {
  OrderGeom g;
  if (!order_geometry(a, which, &g)) return 0;
  int64_t n = g.n_cta;
  if (which != FM_ORDER_FWD && order_geometry(a, which == FM_ORDER_BWD_DQ ? FM_ORDER_BWD_DKDV : FM_ORDER_BWD_DQ, &g))
    n = std::max(n, g.n_cta);
  return n > sm_count();
}

// A wait of a kernel is given up two seconds after its CTA started.  A CTA of the persistent backward kernels lives as long as
// its launch and one of the others as long as its unit, so they get time for that too: every 64 x 128 item of the call at 20 us, some
// fifteen times what one takes, shared by the SMs, and those of one unit (131072 queries, 262144 keys, 96 / 8 heads, 2.3 s
// of items: 55 s).  The bound lies here and not in the kernels because their waits have no room: with an end for each
// wait from its own first look at the clock (two forms), or a deadline renewed with every unit, forward + backward of 3001 prefix-LM
// tokens, 16 / 4 heads, d = 96, takes 262 -> 272, 262 -> 283, 255 -> 262 us; in this form 264.5 -> 264.7.
static uint64_t bwd_wait_ns(const fm_attn_args* a) {
  const uint64_t halves = ((uint64_t)a->Sq + 63) / 64, tiles = ((uint64_t)a->Sk + 127) / 128;
  const uint64_t of_call = (uint64_t)a->B * a->Hq * halves * tiles, of_key_tile = (uint64_t)(a->Hq / a->Hkv) * halves;
  return 2000000000ull + (of_call / (uint64_t)sm_count() + of_key_tile + 2 * tiles) * 20000ull;
}

// The counters of the persistent kernels live behind the table and the two unit arrays.
static void attach_bwd_tables(const fm_attn_args* a, AttnKParams* p) {
  OrderGeom g;
  p->wait_ns = bwd_wait_ns(a);
  p->dq_sched = p->dkdv_sched = nullptr;
  p->dq_ncta = p->dkdv_ncta = 0;
  if (p->dq_order && order_geometry_any(a, FM_ORDER_BWD_DQ, &g)) {
    p->dq_ncta = (int)g.n_cta;
    p->dq_sched = const_cast<int*>(p->dq_order) + 2 * g.n_cta + 2 * g.E;
  } else {
    p->dq_order = nullptr;
  }
  if (p->dkdv_order && order_geometry_any(a, FM_ORDER_BWD_DKDV, &g)) {
    p->dkdv_ncta = (int)g.n_cta;
    p->dkdv_sched = const_cast<int*>(p->dkdv_order) + 2 * g.n_cta + 2 * g.E;
  } else {
    p->dkdv_order = nullptr;
  }
}

static OrderJob order_job(const fm_attn_args* a, int which, const OrderGeom& g, int32_t* out) {
  // work items per unit of work: two 64-key halves per K tile (dQ), one per q head of the group (dK/dV)
  const int item_mult = which == FM_ORDER_BWD_DQ ? 2 : (which == FM_ORDER_BWD_DKDV ? a->Hq / a->Hkv : 1);
  return OrderJob{g.axis, g.block_rows, g.n_units, g.n_other, g.rep_h, g.rep_b, g.heads, item_mult, out};
}

extern "C" int fm_launch_order(const fm_attn_args* a, int which, int32_t* out, void* stream) {
  int32_t* outs[3] = {nullptr, nullptr, nullptr};
  FM_REQUIRE(which >= 0 && which < 3, FM_ERR_INVALID_ARGUMENT, "fm_launch_order: unknown kernel %d", which);
  FM_REQUIRE(out != nullptr, FM_ERR_INVALID_ARGUMENT, "fm_launch_order: NULL argument");
  outs[which] = out;
  return fm_launch_orders(a, outs[0], outs[1], outs[2], stream);
}

extern "C" int fm_launch_orders(const fm_attn_args* a, int32_t* out_fwd, int32_t* out_dq, int32_t* out_dkdv,
                                void* stream) {
  FM_REQUIRE(a && (out_fwd || out_dq || out_dkdv), FM_ERR_INVALID_ARGUMENT, "fm_launch_orders: NULL argument");
  FM_REQUIRE(a->minmax && a->tile_n == 128, FM_ERR_INVALID_ARGUMENT,
             "fm_launch_orders: minmax must be prepared with tile_n = 128");
  int32_t* outs[3] = {out_fwd, out_dq, out_dkdv};
  OrderJobs jobs;
  int n = 0;
  for (int which = 0; which < 3; ++which) {
    if (!outs[which]) continue;
    OrderGeom g;
    FM_REQUIRE(order_geometry(a, which, &g), FM_ERR_UNSUPPORTED,
               "fm_launch_orders: no order for kernel %d with this variant / mask (fm_launch_order_ints returned 0)",
               which);
    FM_REQUIRE(((uintptr_t)outs[which] & 7) == 0, FM_ERR_INVALID_ARGUMENT, "fm_launch_orders: out must be 8-byte aligned");
    jobs.job[n++] = order_job(a, which, g, outs[which]);
  }
  MaskDesc md{a->mask, a->minmax, a->ncols, a->causal, a->Hm, a->mask_B, fm_mask_nblk_pad(a->Sk, 128),
              a->mask_B * a->Hm, a->Sq, a->Sk};
  return launch_order_build(md, 128, jobs, n, (cudaStream_t)stream);
}

// Workspace layout: rowsum(O dO) and LSE*log2e, one float each per (batch, q head, padded row),
// then (one-kernel backward only) the fp32 dQ accumulator, 256-byte aligned.
static size_t bwd_row_stat_bytes(const fm_attn_args* a) {
  const size_t rows = (size_t)a->B * a->Hq * round_up(a->Sq, 128);
  return (2 * rows * sizeof(float) + 255) & ~(size_t)255;
}

// One-kernel backward: the statistics once more as GEMM operands (bf16 parts), 2 x 16 bytes per row.
static size_t bwd_stat_operand_bytes(const fm_attn_args* a) {
  return (size_t)a->B * a->Hq * round_up(a->Sq, 128) * 32;
}

static size_t bwd_workspace_bytes(const fm_attn_args* a, BwdKernels kernels) {
  size_t n = bwd_row_stat_bytes(a);
  if (kernels == BWD_PAIR) n += bwd_pair_workspace_bytes(a);
  if (kernels == BWD_ONE_KERNEL) n += bwd_sm100_fused_accum_bytes(a) + bwd_stat_operand_bytes(a);
  return n;
}

// What fm_bwd cannot do without: the CTA-pair backward works in smaller chunks when it gets less than it asks for, and
// leaves the call to the warp-MMA kernels, which keep row statistics only, when not even the smallest chunk fits; between the
// head dims 64 and 128 the two-kernel backward takes a call without room for the accumulator.
static size_t bwd_min_workspace_bytes(const fm_attn_args* a, BwdKernels kernels) {
  if (kernels == BWD_ONE_KERNEL && !bwd_fills_boxes(a)) kernels = BWD_TWO_KERNELS;
  return bwd_workspace_bytes(a, kernels == BWD_PAIR ? BWD_WARP_MMA : kernels);
}

// (by geometry: a host may ask before it knows its tensors)
extern "C" size_t fm_bwd_min_workspace_bytes(const fm_attn_args* a) {
  if (!a || a->B <= 0 || a->Hq <= 0 || a->Sq <= 0) return 0;
  return bwd_min_workspace_bytes(a, bwd_kernels_by_geometry(a));
}
extern "C" size_t fm_bwd_workspace_bytes(const fm_attn_args* a) {
  if (!a || a->B <= 0 || a->Hq <= 0 || a->Sq <= 0) return 0;
  return bwd_workspace_bytes(a, bwd_kernels_by_geometry(a));
}

extern "C" int fm_bwd_accumulates(const fm_attn_args* a) {
  return (a && a->d > 0 && a->dv > 0 && bwd_fills_boxes(a) && bwd_kernels(a) == BWD_ONE_KERNEL) ? 1 : 0;
}

extern "C" int fm_bwd(const fm_attn_args* a, void* stream) {
  int rc = validate_common(a, "fm_bwd");
  if (rc != FM_OK) return rc;
  FM_REQUIRE(a->d_o && a->dq && a->dk && a->dv_out, FM_ERR_INVALID_ARGUMENT,
             "fm_bwd: d_o/dq/dk/dv must not be NULL");
  FM_REQUIRE(stride_ok(a->do_stride) && stride_ok(a->dq_stride) && stride_ok(a->dk_stride) &&
                 stride_ok(a->dv_stride),
             FM_ERR_INVALID_ARGUMENT, "fm_bwd: strides must be multiples of 8 elements");
  FM_REQUIRE(!(a->sink && !a->dsink), FM_ERR_INVALID_ARGUMENT, "fm_bwd: sink given but dsink is NULL");
  int tm, tn;
  rc = fm_bwd_tile_shape(a->d, a->dv, &tm, &tn);
  if (rc != FM_OK) return rc;
  FM_REQUIRE(a->ncols == 0 || a->tile_n == tn, FM_ERR_INVALID_ARGUMENT,
             "fm_bwd: minmax was prepared for tile_n=%d, this variant needs %d", a->tile_n, tn);
  BwdKernels kernels = bwd_kernels(a);
  const size_t need = bwd_min_workspace_bytes(a, kernels);
  FM_REQUIRE(a->workspace && a->workspace_bytes >= need, FM_ERR_WORKSPACE,
             "fm_bwd: workspace too small (%zu bytes given, %zu needed)", a->workspace_bytes, need);
  FM_REQUIRE(((uintptr_t)a->workspace & 255) == 0, FM_ERR_WORKSPACE, "fm_bwd: workspace must be 256-byte aligned");
  AttnKParams p;
  fill_kparams(a, &p, true);
  p.md.nblk_pad = fm_mask_nblk_pad(a->Sk, tn);
  const size_t rows = (size_t)a->B * a->Hq * p.Sq_r;
  p.dpsum = reinterpret_cast<float*>(a->workspace);
  p.lse_log2 = p.dpsum + rows;
  if (kernels == BWD_ONE_KERNEL && a->workspace_bytes < bwd_workspace_bytes(a, kernels)) kernels = BWD_TWO_KERNELS;
  if (kernels == BWD_ONE_KERNEL) {
    uint8_t* w = reinterpret_cast<uint8_t*>(a->workspace) + bwd_row_stat_bytes(a);
    p.dq_accum = reinterpret_cast<float*>(w);
    p.stat_s = reinterpret_cast<uint16_t*>(w + bwd_sm100_fused_accum_bytes(a));
    p.stat_dp = p.stat_s + (size_t)a->B * a->Hq * p.Sq_r * 8;
    p.bwd_flags = bwd_fills_boxes(a) ? a->bwd_flags : 0;      // (see fm_bwd_accumulates)
  }
  const size_t beyond_stats = a->workspace_bytes - bwd_row_stat_bytes(a);
  if (kernels == BWD_PAIR && bwd_pair_fits(a, beyond_stats)) {
    p.pair_ws = reinterpret_cast<uint8_t*>(a->workspace) + bwd_row_stat_bytes(a);
    p.pair_ws_bytes = beyond_stats;
  }
  cudaStream_t s = (cudaStream_t)stream;
  attach_bwd_tables(a, &p);
  return run_bwd_kernels(a, kernels, p, s);
}

extern "C" int fm_kernel_status(int* status, int reset) {
  FM_REQUIRE(status != nullptr, FM_ERR_INVALID_ARGUMENT, "fm_kernel_status: NULL output");
  int f = 0, bw = 0;
  int rc = fwd_sm100_status(&f, reset != 0);
  if (rc != FM_OK) return rc;
  rc = bwd_sm100_status(&bw, reset != 0);
  if (rc != FM_OK) return rc;
  int bp = 0, bf = 0, fp = 0, bpair = 0;
  rc = fwd_pair_status(&fp, reset != 0);
  if (rc != FM_OK) return rc;
  rc = bwd_pair_status(&bpair, reset != 0);
  if (rc != FM_OK) return rc;
  rc = bwd_sm100_persist_status(&bp, reset != 0);
  if (rc != FM_OK) return rc;
  rc = bwd_sm100_fused_status(&bf, reset != 0);
  *status = f ? f : (bw ? bw : (bp ? bp : (bf ? bf : (fp ? fp : bpair))));
  return rc;
}

extern "C" int fm_selftest_bounded_wait(int budget_us, void* stream) {
  FM_REQUIRE(budget_us > 0 && budget_us <= 1000000, FM_ERR_INVALID_ARGUMENT,
             "fm_selftest_bounded_wait: budget must be in (0, 1 s]");
  return bounded_wait_selftest_launch((uint64_t)budget_us * 1000ull, (cudaStream_t)stream);
}

// ---------------------------------------------------------------------------
// Backward for callers that must not allocate
// ---------------------------------------------------------------------------
// Row-statistics scratch of the backward (rowsum(O*dO) and LSE*log2(e), one
// float each per (batch, q head, padded query row)) held in the library image
// instead of a caller workspace.  Every GPU that loads the library carries
// these 8 MiB until the process exits.
#define FM_STATIC_SCRATCH_ROWS (1 << 20)
static __device__ __align__(256) float g_bwd_row_scratch[2 * FM_STATIC_SCRATCH_ROWS];

// Device address of the array above, per device ordinal.  In host code the
// array's name is only a handle; the address a kernel can use comes from
// cudaGetSymbolAddress, asked once per device with that device current.
static float* g_bwd_row_scratch_addr[64] = {nullptr};

static int static_scratch_for_current_device(float** out) {
  int dev = -1;
  FM_CUDA_TRY(cudaGetDevice(&dev));
  FM_REQUIRE(dev >= 0 && dev < 64, FM_ERR_UNSUPPORTED, "fm_bwd_static_scratch: device ordinal %d not supported", dev);
  if (g_bwd_row_scratch_addr[dev] == nullptr) {
    void* ptr = nullptr;
    FM_CUDA_TRY(cudaGetSymbolAddress(&ptr, g_bwd_row_scratch));
    FM_REQUIRE(ptr != nullptr, FM_ERR_CUDA, "fm_bwd_static_scratch: cudaGetSymbolAddress returned NULL");
    g_bwd_row_scratch_addr[dev] = static_cast<float*>(ptr);
  }
  *out = g_bwd_row_scratch_addr[dev];
  return FM_OK;
}

extern "C" int fm_bwd_static_scratch(const fm_attn_args* a, void* stream) {
  int rc = validate_common(a, "fm_bwd_static_scratch");
  if (rc != FM_OK) return rc;
  FM_REQUIRE(a->d_o && a->dq && a->dk && a->dv_out, FM_ERR_INVALID_ARGUMENT,
             "fm_bwd_static_scratch: d_o/dq/dk/dv must not be NULL");
  FM_REQUIRE(stride_ok(a->do_stride) && stride_ok(a->dq_stride) && stride_ok(a->dk_stride) &&
                 stride_ok(a->dv_stride),
             FM_ERR_INVALID_ARGUMENT, "fm_bwd_static_scratch: strides must be multiples of 8 elements");
  FM_REQUIRE(!(a->sink && !a->dsink), FM_ERR_INVALID_ARGUMENT,
             "fm_bwd_static_scratch: sink given but dsink is NULL");
  int tm, tn;
  rc = fm_bwd_tile_shape(a->d, a->dv, &tm, &tn);
  if (rc != FM_OK) return rc;
  FM_REQUIRE(a->ncols == 0 || a->tile_n == tn, FM_ERR_INVALID_ARGUMENT,
             "fm_bwd_static_scratch: minmax was prepared for tile_n=%d, this variant needs %d", a->tile_n, tn);
  const size_t rows = (size_t)a->B * a->Hq * round_up(a->Sq, 128);
  FM_REQUIRE(rows <= (size_t)FM_STATIC_SCRATCH_ROWS, FM_ERR_WORKSPACE,
             "fm_bwd_static_scratch: B*Hq*roundup(Sq,128) = %zu rows exceeds the built-in scratch of %d rows; "
             "use fm_bwd with a caller workspace",
             rows, FM_STATIC_SCRATCH_ROWS);
  float* scratch = nullptr;
  rc = static_scratch_for_current_device(&scratch);
  if (rc != FM_OK) return rc;
  AttnKParams p;
  fill_kparams(a, &p, true);
  p.md.nblk_pad = fm_mask_nblk_pad(a->Sk, tn);
  // Both halves are fully rewritten by the preprocess kernel for every row the
  // later kernels read, so nothing left by an earlier call has to be cleared.
  p.dpsum = scratch;
  p.lse_log2 = scratch + rows;
  attach_bwd_tables(a, &p);
  return run_bwd_kernels(a, bwd_kernels(a), p, (cudaStream_t)stream);
}
