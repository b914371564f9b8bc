"""CPU-side checks: the shared library exports what the header declares, the
host helpers behave, the workload generators have the promised shapes."""
import ctypes
import os
import re

import numpy as np
import pytest
import torch

import flashmask_b200 as fm
from flashmask_b200 import _lib, workloads as W

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _declared():
    text = ""
    inc = os.path.join(ROOT, "include")
    for f in sorted(os.listdir(inc)):
        if f.endswith(".h"):
            text += open(os.path.join(inc, f)).read()
    return sorted(set(re.findall(r"FM_API\s+[\w\s\*]+?\b(fm_\w+)\s*\(", text)))


def test_library_exports_every_declared_symbol():
    names = _declared()
    assert len(names) >= 10
    lib = ctypes.CDLL(_lib.LIB_PATH)
    for n in names:
        assert hasattr(lib, n), f"{n} declared in include/*.h but not exported"
    assert sorted(_lib.SIGNATURES) == names, "ctypes binding and header disagree"


def test_version_and_pad_without_gpu():
    lib = _lib.load()
    assert b"sm_100a" in lib.fm_version()
    for sk, tn in [(1, 64), (8192, 128), (8193, 128), (333, 32)]:
        assert lib.fm_mask_nblk_pad(sk, tn) == ((sk + tn - 1) // tn + 3) & ~3


def test_argument_errors_need_no_gpu():
    lib = _lib.load()
    rc = lib.fm_mask_prepare(None, 1, 1, 8, 8, 3, 1, 64, 64, None, None, None, None)
    assert rc == 1 and b"ncols" in lib.fm_last_error()
    a = _lib.AttnArgs()
    assert lib.fm_fwd(ctypes.byref(a), None) == 1
    assert lib.fm_fwd_block_score(ctypes.byref(a), None, 64, 1, None, None) == 1
    assert b"block_logit is NULL" in lib.fm_last_error()
    with pytest.raises(NotImplementedError):
        fm.fwd_tile_shape(100, 300)
    with pytest.raises(RuntimeError):
        q = torch.zeros(1, 8, 1, 64, dtype=torch.bfloat16)
        fm.flashmask_attention(q, q, q)


def test_kernel_variant_routing_needs_no_gpu():
    """Tile shapes and launch tables by head dim: the tcgen05 variants (128-column K tiles; 64-query items in the
    backward up to 192) serve every head dim up to 128, 192 / 128, 256 / 256, 512 / 512 and 576 / 512 in both directions;
    a launch table exists only where the variant walks one (not at 256 and above, not for the 192 backward)."""
    for d, dv in [(8, 8), (64, 64), (96, 80), (128, 128), (192, 128), (256, 256)]:
        assert fm.fwd_tile_shape(d, dv) == (128, 128), (d, dv)
    for d, dv in [(64, 64), (128, 64), (128, 128), (192, 128)]:
        assert fm.bwd_tile_shape(d, dv) == (64, 128), (d, dv)
    assert fm.bwd_tile_shape(256, 256) != (64, 128) and fm.bwd_tile_shape(576, 512) != (64, 128)
    lib = _lib.load()
    a = _lib.AttnArgs()
    a.B, a.Sq, a.Sk, a.Hq, a.Hkv, a.Hm, a.mask_B, a.ncols = 2, 4096, 4096, 8, 2, 1, 2, 2
    want = {(128, 128): (True, True, True), (64, 64): (True, True, True), (192, 128): (True, False, False),
            (256, 256): (False, False, False), (576, 512): (False, False, False)}
    for (d, dv), has in want.items():
        a.d, a.dv = d, dv
        got = tuple(lib.fm_launch_order_ints(ctypes.byref(a), w) > 0 for w in
                    (_lib.FM_ORDER_FWD, _lib.FM_ORDER_BWD_DQ, _lib.FM_ORDER_BWD_DKDV))
        assert got == has, (d, dv, got)


def test_partial_results_of_the_forward_are_asked_for_where_they_pay():
    """The forward's workspace query says which calls are split: few rows against many keys, not a chip full of
    short calls, where the fp32 partial results would cost several times the output."""
    lib = _lib.load()

    def nbytes(B, Sq, Sk, Hq, Hkv, d, ncols=0):
        a = _lib.AttnArgs()
        a.B, a.Sq, a.Sk, a.Hq, a.Hkv, a.Hm, a.mask_B, a.d, a.dv, a.causal = B, Sq, Sk, Hq, Hkv, 1, 1, d, d, 1
        a.ncols = ncols
        return lib.fm_fwd_workspace_bytes(ctypes.byref(a))
    for d in (64, 128):
        assert nbytes(8, 1, 8192, 32, 8, d) > 0 and nbytes(1, 1, 32768, 32, 8, d) > 0
        assert nbytes(1, 512, 16384, 32, 8, d) > 0
        assert nbytes(512, 128, 256, 16, 16, d) == 0 and nbytes(48, 128, 1024, 16, 16, d) == 0
        assert nbytes(16, 128, 384, 16, 16, d) == 0 and nbytes(1, 4096, 4096, 32, 8, d) == 0
        assert nbytes(8, 1, 8192, 32, 8, d, ncols=1) == 0        # (a mask's tiles are not known to the host)
        # never more than 32 parts of a row
        for args in ((1, 1, 262144, 1, 1, d), (1, 7, 100000, 4, 1, d), (3, 200, 65536, 2, 2, d)):
            assert nbytes(*args) <= 32 * args[0] * args[1] * args[3] * (d + 1) * 4


def test_repeated_operands_take_no_tensor_map():
    """A dimension of several elements with stride 0 cannot be described to the kernels' tensor maps: the hosts copy
    such a tensor (and keep a value that is a view of the key), and the C ABI routes the call to the kernels that
    compute addresses."""
    from flashmask_b200.ops import _kernel_operand, _key_value_operands
    k = torch.randn(1, 6, 1, 576)
    for t in (k.expand(3, 6, 1, 576), k.expand(1, 6, 4, 576), k[:, :1].expand(1, 6, 1, 576)):
        got = _kernel_operand(t)
        assert got.is_contiguous() and torch.equal(got, t)
    one = torch.empty_strided((1, 6, 1, 8), (0, 8, 0, 1))        # one element: any stride will do
    assert _kernel_operand(one) is one and _kernel_operand(k) is k
    ke = k.expand(3, 6, 1, 576)
    kc, vc = _key_value_operands(ke, ke[..., :512])
    assert kc.data_ptr() == vc.data_ptr() and kc.stride() == vc.stride() and vc.shape[-1] == 512
    assert min(kc.stride()) > 0 and torch.equal(kc, ke)
    lib = _lib.load()
    a = _lib.AttnArgs()
    a.B, a.Sq, a.Sk, a.Hq, a.Hkv, a.Hm, a.mask_B, a.d, a.dv, a.softmax_scale = 2, 64, 64, 4, 2, 1, 1, 128, 128, 0.1

    def accumulates(**strides):
        for name, H in (("q", 4), ("k", 2), ("v", 2), ("do", 4)):
            setattr(a, name + "_stride", _lib.I64x3(*strides.get(name, (64 * H * 128, H * 128, 128))))
        return lib.fm_bwd_accumulates(ctypes.byref(a))
    assert accumulates() == 1
    for name, H in (("q", 4), ("k", 2), ("v", 2), ("do", 4)):
        for s in ((0, H * 128, 128), (64 * H * 128, 0, 128), (64 * H * 128, H * 128, 0)):
            assert accumulates(**{name: s}) == 0, (name, s)
    a.B = a.mask_B = 1
    assert accumulates(k=(0, 256, 128)) == 1
    for scale in (0.0, -0.1, float("nan")):
        a.softmax_scale = scale
        assert accumulates() == 0, scale


@pytest.mark.parametrize("d,dv", [(64, 64), (256, 256), (576, 512)])
def test_size_queries_survive_arguments_that_a_call_would_refuse(d, dv):
    """Hosts ask for sizes before anything is validated: heads that do not divide or are missing, lengths of 0."""
    lib = _lib.load()
    for Sq, Sk, Hq, Hkv in ((512, 512, 4, 8), (512, 512, 6, 4), (512, 512, 4, 0), (512, 512, 0, 4), (512, 0, 4, 4),
                            (0, 512, 4, 4), (512, 512, 4, -1), (-1, -1, -1, -1)):
        a = _lib.AttnArgs()
        a.B, a.Sq, a.Sk, a.Hq, a.Hkv, a.Hm, a.mask_B, a.d, a.dv = 1, Sq, Sk, Hq, Hkv, 1, 1, d, dv
        # without a usable geometry no variant with a large workspace is meant
        assert lib.fm_bwd_workspace_bytes(ctypes.byref(a)) <= 4 << 20, (Sq, Sk, Hq, Hkv)
        assert lib.fm_bwd_accumulates(ctypes.byref(a)) == 0
        assert lib.fm_fwd_workspace_bytes(ctypes.byref(a)) == 0 or Hq % max(Hkv, 1) == 0
        assert [lib.fm_launch_order_ints(ctypes.byref(a), w) for w in range(3)] == [0, 0, 0]


def test_pair_backward_workspace_is_bounded():
    """The CTA-pair backward keeps P and dS of at least 256 rows of a kv group: up to 8 GiB, and none at all (the
    kernels without a workspace serve the call) where that would not do."""
    lib = _lib.load()
    sizes = {}
    for Hq, Sk in ((16, 16384), (128, 65536), (128, 131072), (16, 262144), (64, 262144)):
        a = _lib.AttnArgs()
        a.B, a.Sq, a.Sk, a.Hq, a.Hkv, a.Hm, a.mask_B, a.d, a.dv = 1, 4096, Sk, Hq, 1, 1, 1, 576, 512
        stats = 2 * 4 * Hq * 4096
        n = lib.fm_bwd_workspace_bytes(ctypes.byref(a)) - stats
        sizes[Hq, Sk] = n
        assert n == 0 or n <= (8 << 30) + Sk * (576 + 512) * 4
        assert (n == 0) == (Hq * Sk * 4 * 256 > 8 << 30), (Hq, Sk, n)
    assert sizes[128, 131072] == 0 and sizes[128, 65536] > 8 << 30


def test_least_workspace_of_the_backward():
    """What fm_bwd cannot do without: everything it asks for, but at the head dims of the CTA-pair backward the row
    statistics alone."""
    lib = _lib.load()
    for d, dv in ((64, 64), (128, 128), (192, 128), (256, 256), (512, 512), (576, 512)):
        a = _lib.AttnArgs()
        a.B, a.Sq, a.Sk, a.Hq, a.Hkv, a.Hm, a.mask_B, a.d, a.dv = 2, 4096, 4096, 8, 2, 1, 1, d, dv
        n, least = lib.fm_bwd_workspace_bytes(ctypes.byref(a)), lib.fm_bwd_min_workspace_bytes(ctypes.byref(a))
        assert least == (n if d < 256 else 2 * 4 * 2 * 8 * 4096)
        assert n - least == (0 if d < 256 else 4 << 28)         # (P and dS of four groups, 256 MiB each)


@pytest.mark.parametrize("one,B,S,Hq,Hkv,ncols", [
    # (without a GPU the library counts 148 multiprocessors)
    (1, 2, 8192, 32, 8, 1), (1, 1, 4800, 32, 8, 1), (1, 8, 517, 16, 8, 2), (0, 1, 4600, 32, 8, 1),   # two units each
    (0, 1, 19163, 32, 2, 1), (1, 1, 28763, 32, 2, 2), (0, 1, 12763, 12, 3, 1), (1, 1, 19163, 6, 3, 1),    # few copies
    (0, 1, 57563, 4, 1, 4), (1, 1, 76763, 4, 1, 1), (0, 1, 9563, 16, 4, 1), (1, 1, 11900, 16, 4, 1),
    (0, 4, 10000, 4, 1, 1), (0, 4, 5000, 8, 2, 2),
    (0, 16, 640, 16, 16, 1), (1, 8, 900, 8, 8, 1), (0, 64, 200, 16, 4, 1),                              # short units
    (0, 64, 512, 16, 4, 1), (1, 12, 520, 32, 8, 1), (1, 20, 900, 16, 16, 1),                            # accumulator in L2
    (1, 64, 100, 32, 8, 0), (0, 64, 256, 16, 16, 0), (1, 1, 19000, 32, 2, 0), (0, 1, 18800, 32, 2, 0),  # no mask
    (0, 5, 1000, 8, 8, 0), (1, 8, 1280, 16, 16, 0), (1, 1, 2432, 16, 16, 0), (1, 8, 517, 16, 8, 0)])
@pytest.mark.parametrize("d", [72, 96, 120])
def test_which_backward_serves_head_dims_between_64_and_128(d, one, B, S, Hq, Hkv, ncols):
    """Either side of every line of the rule: only the one-kernel backward asks for an accumulator."""
    lib = _lib.load()
    a = _lib.AttnArgs()
    a.B, a.Sq, a.Sk, a.Hq, a.Hkv, a.Hm, a.mask_B, a.ncols, a.d, a.dv = B, S, S, Hq, Hkv, 1, B, ncols, d, d
    rows = B * Hq * -(-S // 128) * 128
    sizes = lambda: (lib.fm_bwd_workspace_bytes(ctypes.byref(a)), lib.fm_bwd_min_workspace_bytes(ctypes.byref(a)))
    assert sizes() == (rows * (552 if one else 8), rows * 8)
    assert lib.fm_bwd_accumulates(ctypes.byref(a)) == 0
    a.deterministic = 1
    assert sizes() == (rows * 8, rows * 8)
    a.deterministic, a.dv = 0, d - 8                              # unequal head dims: two kernels
    assert sizes() == (rows * 8, rows * 8)


def test_heads_and_batch_entries_that_share_a_mask_are_copies():
    lib = _lib.load()
    for one, Hm, mask_B in ((0, 1, 4), (1, 1, 1), (0, 2, 4), (0, 2, 1)):      # copies: 2, 8, 1, 4
        a = _lib.AttnArgs()
        a.B, a.Sq, a.Sk, a.Hq, a.Hkv, a.d, a.dv, a.ncols = 4, 5000, 5000, 8, 2, 96, 96, 2
        a.Hm, a.mask_B = Hm, mask_B
        n, least = lib.fm_bwd_workspace_bytes(ctypes.byref(a)), lib.fm_bwd_min_workspace_bytes(ctypes.byref(a))
        assert (n > least) == bool(one), (Hm, mask_B)


@pytest.mark.parametrize("d", [96, 128])
def test_size_queries_of_impossible_heads(d):
    for Hq, Hkv, Sk in ((4, 0, 512), (0, 4, 512), (4, -1, 512), (4, 4, 0)):
        a = _lib.AttnArgs()
        a.B, a.Sq, a.Sk, a.Hq, a.Hkv, a.Hm, a.mask_B, a.d, a.dv = 1, 4096, Sk, Hq, Hkv, 1, 1, d, d
        assert _lib.load().fm_bwd_workspace_bytes(ctypes.byref(a)) <= (8 + 32 + 512) * 4 * 4096


@pytest.mark.parametrize("d,B,S,Hq,Hkv,ncols,want", [
    # (without a GPU the library counts 148 multiprocessors; CTAs of the forward, dQ and dK / dV launch behind each call)
    (64, 1, 1024, 2, 2, 1, (0, 0, 0)),       # 8, 16, 16
    (128, 1, 1024, 37, 1, 1, (0, 1, 1)),     # 148, 296, 8
    (128, 1, 1025, 37, 1, 2, (1, 1, 1)),     # 185
    (96, 2, 1100, 8, 8, 1, (0, 0, 0)),       # 80, 144, 144
    (96, 3, 1100, 8, 8, 1, (0, 1, 1)),       # 120, 216, 216
    (128, 4, 8192, 32, 8, 0, (0, 0, 0)),     # no mask, no table
    (192, 1, 8192, 32, 8, 1, (1, 0, 0)),     # the backward takes none
    (256, 1, 8192, 32, 8, 1, (0, 0, 0))])
def test_launch_tables_are_useful_where_ctas_queue(d, B, S, Hq, Hkv, ncols, want):
    lib = _lib.load()
    a = _lib.AttnArgs()
    a.B, a.Sq, a.Sk, a.Hq, a.Hkv, a.Hm, a.mask_B, a.ncols, a.d, a.dv = B, S, S, Hq, Hkv, 1, B, ncols, d, min(d, 128 if d < 256 else d)
    assert tuple(lib.fm_launch_order_useful(ctypes.byref(a), w) for w in range(3)) == want
    assert lib.fm_launch_order_useful(None, 0) == 0


def test_struct_layout_matches_header():
    # 18 int32/float + 15 pointers/size_t + 24 int64
    assert ctypes.sizeof(_lib.AttnArgs) == 18 * 4 + 15 * 8 + 24 * 8 + 3 * 8


def test_workload_shapes():
    w = W.make_workload("causal_doc_8k_gqa")
    assert w.idx.shape == (2, 1, 8192, 1) and w.idx.dtype == np.int32 and w.causal
    assert (w.idx[..., 0] > np.arange(8192)).all() and w.idx.max() == 8192
    fwd, bwd = w.flops()
    assert fwd * 5 == bwd * 2
    w5 = W.make_workload("cp_causal_doc_128k", S=8192)
    assert w5.idx.shape == (1, 1, 8192, 2) and not w5.causal
    # the non-causal 2-column form masks exactly what the causal 1-column form does
    lens = np.diff(np.concatenate([[0], np.unique(w5.idx[0, 0, :, 0])]))
    a = W.dense_visible(w5.idx[:, :, :512], 512, False)
    idx1 = np.minimum(w5.idx[:, :, :512, :1], 512)
    b = W.dense_visible(idx1, 512, True)
    assert np.array_equal(a[..., :512, :], b)
    for name in W.WORKLOADS:
        s = 2048 if "128k" in name or "32k" in name or "16k" in name else None
        wl = W.make_workload(name, S=s)
        assert 0.0 <= wl.sparsity() < 1.0


def test_operands_on_several_devices_are_refused():
    from flashmask_b200.ops import _check_shapes
    x = torch.zeros(1, 8, 1, 64, dtype=torch.bfloat16)
    idx = torch.zeros(1, 1, 8, 1, dtype=torch.int32)
    _check_shapes(x, x, x, idx, True)
    m = x.to("meta")
    for args in ((x, m, x, None), (x, x, m, None), (m, x, x, None), (m, m, m, idx)):
        with pytest.raises(AssertionError, match="device"):
            _check_shapes(*args, True)


def test_sliding_window_kwarg_bounds():
    idx = fm.sliding_window_indices(16, 16, 4, True, 2, "cpu")
    ref, _ = W.sliding_window(2, 16, 16, 4)
    assert np.array_equal(idx.numpy(), ref)
    idx2 = fm.sliding_window_indices(16, 16, (3, 2), False, 1, "cpu")
    vis = W.dense_visible(idx2.numpy(), 16, False)[0, 0]
    i, j = np.indices((16, 16))
    assert np.array_equal(vis, (j - i <= 2) & (i - j <= 3))


def test_every_included_file_is_a_dependency_of_the_objects():
    """An object is compiled again when anything that a source includes has changed, textually included sources too."""
    from flashmask_b200 import build as b
    known = {os.path.basename(h) for h in b.headers()}
    csrc = os.path.join(ROOT, "flashmask_b200", "csrc")
    own = set(os.listdir(csrc)) | set(os.listdir(os.path.join(ROOT, "include")))
    seen = set()
    for f in sorted(os.listdir(csrc)):
        if f.endswith((".cu", ".cuh", ".cpp", ".inc")):
            seen |= {os.path.basename(n) for n in re.findall(r'#include "([^"]+)"', open(os.path.join(csrc, f)).read())}
    assert len(seen & own) >= 5 and (seen & own) <= known, sorted((seen & own) - known)
