// Host path of the public operator in native code: shape checks, allocation of the outputs and workspaces, the
// autograd node, and the calls into the C ABI of libflashmask_b200.so (the only device code involved).
//
// Why native.  At B = 1, H = 2, S = 1024, d = 64 the kernels of a forward + backward take 50 us, and a pass with the
// Python host (argument structs through ctypes, two dozen small calls, a Python autograd node entered from the
// engine's thread) took 269 us, when the kernels took 77; with this one it takes 91.  It makes the calls of ops.py in the same order; results are
// bitwise those of FlashMaskFunc, the same operator over ops.py.
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/extension.h>

#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>

#include "flashmask_b200.h"

namespace {

using at::Tensor;
using torch::autograd::AutogradContext;
using torch::autograd::Variable;
using torch::autograd::variable_list;

void check(int rc, const char* what) {
  if (rc == FM_OK) return;
  TORCH_CHECK_VALUE(rc != FM_ERR_INVALID_ARGUMENT, what, " failed (status ", rc, "): ", fm_last_error());
  TORCH_CHECK_NOT_IMPLEMENTED(rc != FM_ERR_UNSUPPORTED, what, " failed (status ", rc, "): ", fm_last_error());
  TORCH_CHECK(false, what, " failed (status ", rc, "): ", fm_last_error());
}

int dtype_code(const Tensor& t) {
  if (t.scalar_type() == at::kBFloat16) return FM_DTYPE_BF16;
  TORCH_CHECK_TYPE(t.scalar_type() == at::kHalf, "flashmask_attention supports bfloat16 / float16, got ", t.scalar_type());
  return FM_DTYPE_FP16;
}

// Whether t repeats along a dimension (stride 0: an expanded tensor).
bool repeats(const Tensor& t) {
  for (int i = 0; i < 3; ++i)
    if (t.size(i) > 1 && t.stride(i) == 0) return true;
  return false;
}

// t as the kernels' tensor maps can describe it: rows contiguous, nothing repeated.
Tensor rows(const Tensor& t) { return t.stride(-1) == 1 && !repeats(t) ? t : t.contiguous(); }

void strides(int64_t* out, const Tensor& t) { for (int i = 0; i < 3; ++i) out[i] = t.stride(i); }

// Which launch tables FLASHMASK_B200_ORDER leaves on (bit w: FM_ORDER_* w); read per call, as in ops.py.
unsigned wanted_orders() {
  const char* e = std::getenv("FLASHMASK_B200_ORDER");
  if (!e || std::strcmp(e, "1") == 0) return 7u;
  unsigned m = 0;
  static const char* names[3] = {"fwd", "dq", "dkdv"};
  for (const char* p = e; *p;) {
    const char* end = std::strchr(p, ',');
    const size_t n = end ? (size_t)(end - p) : std::strlen(p);
    for (int w = 0; w < 3; ++w)
      if (std::strlen(names[w]) == n && std::strncmp(p, names[w], n) == 0) m |= 1u << w;
    p += n + (end ? 1 : 0);
  }
  return m;
}

// Arguments of a call without the launch tables: inputs, output, LSE, mask.
fm_attn_args base_args(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& out, const Tensor& lse,
                       bool causal, double scale, const Tensor& sink32) {
  fm_attn_args a;
  std::memset(&a, 0, sizeof(a));
  a.B = (int)q.size(0); a.Sq = (int)q.size(1); a.Hq = (int)q.size(2); a.d = (int)q.size(3);
  a.Sk = (int)k.size(1); a.Hkv = (int)k.size(2); a.dv = (int)v.size(3);
  a.causal = causal;
  a.dtype = dtype_code(q);
  a.softmax_scale = (float)scale;
  a.q = q.data_ptr(); a.k = k.data_ptr(); a.v = v.data_ptr(); a.o = out.data_ptr();
  a.lse = lse.data_ptr<float>();
  strides(a.q_stride, q); strides(a.k_stride, k); strides(a.v_stride, v); strides(a.o_stride, out);
  a.ncols = 0; a.Hm = 1; a.mask_B = 1;
  if (sink32.defined()) a.sink = sink32.data_ptr<float>();
  return a;
}

void set_mask(fm_attn_args* a, const Tensor& idx, const Tensor& minmax, int tile_m, int tile_n) {
  if (!idx.defined()) return;
  a->mask_B = (int)idx.size(0); a->Hm = (int)idx.size(1); a->ncols = (int)idx.size(3);
  a->mask = idx.data_ptr<int>();
  a->minmax = minmax.data_ptr<int>();
  a->tile_m = tile_m; a->tile_n = tile_n;
}

Tensor scan_mask(const Tensor& idx, int Sq, bool causal, int tile_m, int tile_n, void* stream) {
  const int B = (int)idx.size(0), Hm = (int)idx.size(1), Sk = (int)idx.size(2);
  Tensor minmax = at::empty({8, (int64_t)B * Hm, fm_mask_nblk_pad(Sk, tile_n)}, idx.options());
  check(fm_mask_prepare(idx.data_ptr<int>(), B, Hm, Sq, Sk, (int)idx.size(3), causal, tile_m, tile_n,
                        minmax.data_ptr<int>(), nullptr, nullptr, stream), "fm_mask_prepare");
  return minmax;
}

Tensor sink_fp32(const Tensor& sink, const Tensor& q) {
  if (!sink.defined()) return sink;
  return sink.detach().reshape({q.size(2)}).to(q.device(), at::kFloat).contiguous();
}

// The launch tables of a geometry in one buffer; empty tensor and zero offsets where a variant takes none.
struct Tables { Tensor buf; int64_t at[3]; };
Tables build_tables(const fm_attn_args& a, const Tensor& like, void* stream) {
  Tables t{Tensor(), {-1, -1, -1}};
  if (a.ncols == 0 || a.tile_n != 128) return t;      // only the kernels with 128-column tiles read tables
  const unsigned want = wanted_orders();
  const bool asked_for = std::getenv("FLASHMASK_B200_ORDER") != nullptr;   // tables for every size (A/B runs)
  int64_t total = 0;
  for (int w = 0; w < 3; ++w) {
    if (!asked_for && !fm_launch_order_useful(&a, w)) continue;
    const int64_t n = (want >> w & 1u) ? fm_launch_order_ints(&a, w) : 0;
    if (n <= 0) continue;
    t.at[w] = total;
    total += (n + 3) & ~(int64_t)3;
  }
  if (!total) return t;
  t.buf = at::empty({total}, like.options().dtype(at::kInt));
  int32_t* p = t.buf.data_ptr<int>();
  check(fm_launch_orders(&a, t.at[0] < 0 ? nullptr : p + t.at[0], t.at[1] < 0 ? nullptr : p + t.at[1],
                         t.at[2] < 0 ? nullptr : p + t.at[2], stream), "fm_launch_orders");
  return t;
}

bool kv_shared(const Tensor& k, const Tensor& v) {
  const int64_t d = k.size(3), dv = v.size(3);
  return dv == 512 && (d == 512 || d == 576) && k.data_ptr() == v.data_ptr() && k.sizes().slice(0, 3) == v.sizes().slice(0, 3) &&
         k.strides() == v.strides();
}

// Key and value as the kernels read them; a value that is a view of the key's storage stays one.
std::pair<Tensor, Tensor> kv_rows(const Tensor& k, const Tensor& v) {
  if (k.stride(-1) == 1 && repeats(k) && kv_shared(k, v)) {
    const Tensor kc = k.contiguous();
    return {kc, kc.slice(3, 0, v.size(3))};
  }
  return {rows(k), rows(v)};
}

// Workspace of a backward call.  When the device has no room for what the call asks for it gets less: by quarters at the
// head dims 256, 512 and 576 (2 GiB and more, used in chunks of any size), else what it cannot do without at once.
Tensor bwd_workspace(fm_attn_args* a, const Tensor& like) {
  const size_t least = fm_bwd_min_workspace_bytes(a);
  for (size_t n = fm_bwd_workspace_bytes(a);; n = a->d >= 256 ? std::max(least, n / 4) : least) {
    try {
      Tensor ws = at::empty({(int64_t)std::max<size_t>(n, 256)}, like.options().dtype(at::kByte));
      a->workspace = ws.data_ptr();
      a->workspace_bytes = n;
      return ws;
    } catch (const c10::OutOfMemoryError&) {
      if (n <= least) throw;
    }
  }
}

class FlashMask : public torch::autograd::Function<FlashMask> {
 public:
  static variable_list forward(AutogradContext* ctx, const Variable& q_in, const Variable& k_in, const Variable& v_in,
                               const std::optional<Tensor>& idx_in, const std::optional<Tensor>& sink_in,
                               double scale, bool causal, int deterministic) {
    const c10::cuda::CUDAGuard guard(q_in.device());
    void* stream = c10::cuda::getCurrentCUDAStream(q_in.get_device()).stream();
    const Tensor q = rows(q_in);
    const auto [k, v] = kv_rows(k_in, v_in);
    const int d = (int)q.size(3), dv = (int)v.size(3);
    int tm = 0, tn = 0;
    check(fm_fwd_tile_shape(d, dv, &tm, &tn), "fm_fwd_tile_shape");
    const Tensor sink = sink_in ? *sink_in : Tensor(), sink32 = sink_fp32(sink, q);
    Tensor idx, minmax;
    if (idx_in) {
      idx = idx_in->contiguous();
      minmax = scan_mask(idx, (int)q.size(1), causal, tm, tn, stream);
    }
    Tensor out = at::empty({q.size(0), q.size(1), q.size(2), dv}, q.options());
    Tensor lse = at::empty({q.size(0), q.size(2), q.size(1)}, q.options().dtype(at::kFloat));
    fm_attn_args a = base_args(q, k, v, out, lse, causal, scale, sink32);
    set_mask(&a, idx, minmax, tm, tn);
    const Tables t = build_tables(a, q, stream);
    if (t.at[0] >= 0) a.fwd_order = t.buf.data_ptr<int>() + t.at[0];
    const size_t nbytes = fm_fwd_workspace_bytes(&a);
    Tensor ws;
    if (nbytes) {
      ws = at::empty({(int64_t)nbytes}, q.options().dtype(at::kByte));
      a.workspace = ws.data_ptr();
      a.workspace_bytes = nbytes;
    }
    check(fm_fwd(&a, stream), "fm_fwd");
    ctx->save_for_backward({q, k, v, out, lse, idx, minmax, t.buf, sink, sink32});
    ctx->saved_data["scale"] = scale;
    ctx->saved_data["causal"] = causal;
    ctx->saved_data["det"] = (int64_t)deterministic;
    ctx->saved_data["tile_n"] = (int64_t)tn;
    ctx->saved_data["dq_at"] = t.at[1];
    ctx->saved_data["dkdv_at"] = t.at[2];
    ctx->mark_non_differentiable({lse});
    ctx->set_materialize_grads(false);
    return {out, lse};
  }

  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    variable_list none(8);
    if (!grads[0].defined()) return none;
    const variable_list s = ctx->get_saved_variables();
    const Tensor &q = s[0], &k = s[1], &v = s[2], &out = s[3], &lse = s[4], &idx = s[5], &sink = s[8], &sink32 = s[9];
    Tensor minmax = s[6], tables = s[7];
    const c10::cuda::CUDAGuard guard(q.device());
    void* stream = c10::cuda::getCurrentCUDAStream(q.get_device()).stream();
    const bool causal = ctx->saved_data["causal"].toBool();
    const int64_t det = ctx->saved_data["det"].toInt();
    const Tensor dout = rows(grads[0]);
    int tm = 0, tn = 0;
    check(fm_bwd_tile_shape((int)q.size(3), (int)v.size(3), &tm, &tn), "fm_bwd_tile_shape");
    int64_t dq_at = ctx->saved_data["dq_at"].toInt(), dkdv_at = ctx->saved_data["dkdv_at"].toInt();
    const bool rescan = idx.defined() && tn != ctx->saved_data["tile_n"].toInt();
    if (rescan) minmax = scan_mask(idx, (int)q.size(1), causal, tm, tn, stream);
    Tensor dq = at::empty_like(q);
    Tensor dk = at::empty({k.size(0), k.size(1), k.size(2), k.size(3)}, k.options());
    Tensor dv = at::empty({v.size(0), v.size(1), v.size(2), v.size(3)}, v.options());
    Tensor dsink32;
    if (sink32.defined()) dsink32 = at::empty({q.size(2)}, sink32.options());
    fm_attn_args a = base_args(q, k, v, out, lse, causal, ctx->saved_data["scale"].toDouble(), sink32);
    set_mask(&a, idx, minmax, tm, tn);
    a.d_o = dout.data_ptr(); a.dq = dq.data_ptr(); a.dk = dk.data_ptr(); a.dv_out = dv.data_ptr();
    strides(a.do_stride, dout); strides(a.dq_stride, dq); strides(a.dk_stride, dk); strides(a.dv_stride, dv);
    a.deterministic = det < 0 ? at::globalContext().deterministicAlgorithms() : det != 0;
    if (dsink32.defined()) a.dsink = dsink32.data_ptr<float>();
    Tables t;
    if (rescan) {
      t = build_tables(a, q, stream);
      tables = t.buf; dq_at = t.at[1]; dkdv_at = t.at[2];
    }
    if (tables.defined() && dq_at >= 0) a.dq_order = tables.data_ptr<int>() + dq_at;
    if (tables.defined() && dkdv_at >= 0) a.dkdv_order = tables.data_ptr<int>() + dkdv_at;
    const Tensor ws = bwd_workspace(&a, q);
    check(fm_bwd(&a, stream), "fm_bwd");
    if (kv_shared(k, v)) {
      // value is a view of key's leading dv columns at these head dims: one gradient for the storage
      dk.slice(3, 0, v.size(3)).add_(dv);
      dv.zero_();
    }
    none[0] = dq; none[1] = dk; none[2] = dv;
    if (dsink32.defined()) none[4] = dsink32.to(sink.scalar_type()).reshape(sink.sizes());
    return none;
  }
};

void require(bool ok, const char* msg) {
  if (ok) return;
  PyErr_SetString(PyExc_AssertionError, msg);
  throw pybind11::error_already_set();
}

// (out, lse) with the gradient attached; `deterministic`: 0 / 1, or -1 for torch's global setting.
std::pair<Tensor, Tensor> attention(const Tensor& q, const Tensor& k, const Tensor& v, const std::optional<Tensor>& idx,
                                    const std::optional<Tensor>& sink, std::optional<double> scale, bool causal,
                                    int deterministic) {
  TORCH_CHECK(q.is_cuda(), "flashmask_b200 runs on CUDA (sm_100a) tensors only; there is no CPU path");
  require(k.device() == q.device() && v.device() == q.device(), "q/k/v must be on one device");
  require(q.dim() == 4 && k.dim() == 4 && v.dim() == 4, "q/k/v must be [B, S, H, D]");
  const int64_t B = q.size(0), Hq = q.size(2), d = q.size(3), Sk = k.size(1), Hkv = k.size(2);
  require(k.size(0) == B && k.size(3) == d && v.size(0) == B && v.size(1) == Sk && v.size(2) == Hkv, "k/v shapes do not match q");
  require(Hkv > 0 && Hq % Hkv == 0, "num q heads must be a multiple of num kv heads");
  require(q.scalar_type() == k.scalar_type() && q.scalar_type() == v.scalar_type(), "q/k/v must share a dtype");
  if (idx) {
    require(idx->device() == q.device(), "startend_row_indices must be on the device of q");
    require(idx->scalar_type() == at::kInt, "startend_row_indices must be int32");
    require(idx->dim() == 4, "startend_row_indices must be [B, Hm, Sk, n]");
    require(idx->size(0) == B || idx->size(0) == 1, "startend_row_indices batch must match q");
    require(idx->size(2) == Sk, "startend_row_indices seqlen must match k");
    require(idx->size(1) == 1 || idx->size(1) == Hkv, "startend_row_indices heads must be 1 or num kv heads");
    const int64_t n = idx->size(3);
    if (causal) require(n == 1 || n == 2, "causal masks carry 1 or 2 bounds per column");
    else require(n == 2 || n == 4, "non-causal masks carry 2 or 4 bounds per column");
  }
  if (sink) require(sink->numel() == Hq, "learnable_sink must have one logit per q head");
  pybind11::gil_scoped_release nogil;
  variable_list r = FlashMask::apply(q, k, v, idx, sink, scale ? *scale : 1.0 / std::sqrt((double)d), causal, deterministic);
  return {r[0], r[1]};
}

}  // namespace

PYBIND11_MODULE(_host, m) { m.def("attention", &attention); }
