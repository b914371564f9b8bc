"""GPU parity of forward / backward against the CPU oracle, through the public
operator (which calls the C ABI).  Tolerance: the reference's own rule."""
import glob
import math
import os

import numpy as np
import pytest
import torch

from flashmask_b200 import workloads as W
import flashmask_b200 as fm
import oracle
from flashmask_b200 import _lib
from _util import (assert_lse, assert_parity, make_inputs, naive_lowp, run_c_abi, run_oracle, run_product)

pytestmark = pytest.mark.gpu


@pytest.fixture(params=["sm100", "split", "mma"])
def fwd_variant(request):
    """Head dims up to 128 have two kernel families, the tcgen05 ones (default) and the warp-MMA
    ones, and the tcgen05 backward has a one-kernel variant (default when the call does not ask for
    deterministic gradients) and a two-kernel one ("split"); FLASHMASK_B200_FWD / FLASHMASK_B200_BWD
    select them."""
    names = ("FLASHMASK_B200_FWD", "FLASHMASK_B200_BWD")
    old = {n: os.environ.get(n) for n in names}
    os.environ["FLASHMASK_B200_FWD"] = "mma" if request.param == "mma" else "sm100"
    os.environ["FLASHMASK_B200_BWD"] = request.param
    _lib.reload_options()
    yield request.param
    for n in names:
        if old[n] is None:
            os.environ.pop(n, None)
        else:
            os.environ[n] = old[n]
    _lib.reload_options()


def _kernel_status():
    import ctypes as C
    from flashmask_b200 import _lib
    v = C.c_int(0)
    _lib.check(_lib.load().fm_kernel_status(C.byref(v), 1), "fm_kernel_status")
    return v.value

GOLDEN = sorted(glob.glob(os.path.join(os.path.dirname(__file__), "golden", "attention_*.npz")))


def _docs(rng, S, n):
    return W.uniform_doc_lengths(rng, S, n)


def _mask(kind, B, Sq, Sk, seed):
    rng = np.random.default_rng(seed)
    if kind == "none_causal":
        return None, True
    if kind == "none_full":
        return None, False
    if kind == "causal_doc":
        m = [W.causal_document(1, Sq, Sk, _docs(rng, Sk, 5))[0] for _ in range(B)]
        return np.concatenate(m), True
    if kind == "bidir_doc":
        m = [W.bidirectional_document(1, Sq, Sk, _docs(rng, Sk, 4))[0] for _ in range(B)]
        return np.concatenate(m), False
    if kind == "sliding_window":
        return W.sliding_window(B, Sq, Sk, max(3, Sk // 7))
    if kind == "share_question":
        return W.share_question(B, Sq, Sk, Sk // 6, Sk // 12, 3)
    if kind == "random_eviction":
        return W.random_eviction(B, Sq, Sk, rng)
    if kind == "four_column":
        return W.four_column_bands(B, Sq, Sk, rng)
    if kind == "prefix_lm":
        third = Sk // 3
        return W.prefix_lm_document(B, Sq, Sk, [(third // 2, third), (third // 4, third), (5, Sk - 2 * third)])
    if kind == "cp_form":
        return W.causal_document_noncausal_form(B, Sq, Sk, _docs(rng, Sk, 6))
    if kind == "empty":
        return W.empty_mask(B, Sq, Sk)
    raise KeyError(kind)


MASKS = ["none_causal", "none_full", "causal_doc", "bidir_doc", "sliding_window", "share_question",
         "random_eviction", "four_column", "prefix_lm", "cp_form", "empty"]


def _run(kind, B, Sq, Sk, Hq, Hkv, d, dv, sink=False, seed=0, dtype=torch.bfloat16, hm=1):
    idx_np, causal = _mask(kind, B, Sq, Sk, seed)
    if idx_np is not None and hm > 1:
        rng = np.random.default_rng(seed + 99)
        per = [_mask(kind, B, Sq, Sk, seed + 1 + h)[0] for h in range(hm)]
        idx_np = np.ascontiguousarray(np.concatenate(per, axis=1))
    q, k, v, do, s = make_inputs(B, Sq, Sk, Hq, Hkv, d, dv, seed, dtype=dtype, sink=sink)
    idx = None if idx_np is None else torch.from_numpy(np.ascontiguousarray(idx_np).copy()).cuda()
    qc, kc, vc, doc = q.cuda(), k.cuda(), v.cuda(), do.cuda()
    got = run_product(qc, kc, vc, doc, idx, causal, s)
    ref = run_oracle(q, k, v, do, idx, causal, s)
    lowp = naive_lowp(qc, kc, vc, doc, idx, causal, s)
    assert_parity(got, ref, lowp, label=f"{kind}: ")
    assert_lse(got, ref)
    if sink:
        scale = ref["dsink"].abs().max().item() + 1.0
        # the kernel against its own definition, evaluated on the tensors it read (the bf16 O and the LSE of this
        # forward): dsink[h] = -sum_{b,i} exp(sink[h] - lse[b,h,i]) * rowsum(O * dO)[b,i,h]
        dps = (got["out"].float() * doc.float()).sum(-1).permute(0, 2, 1)
        own = -(torch.exp(s.cuda()[None, :, None] - got["lse"].float()) * dps).sum((0, 2))
        err_own = (got["dsink"].float() - own).abs().max().item()
        assert err_own <= 1e-3 + 2 ** -10 * scale, f"dsink vs its definition: {err_own}"
        # and against the fp32 oracle: what is left is the rounding of O to 16 bits before rowsum(O * dO), which
        # the reference's preprocess kernel has too and which grows with the width of the row
        # (noise model: every element of O carries a relative rounding error of up to 2^-9, independent
        # between elements; four standard deviations of the resulting sum, per head)
        w2 = torch.exp(s[None, :, None] - ref["lse"].float()) ** 2
        var = (w2 * ((ref["out"].float() * do.float()) ** 2).sum(-1).permute(0, 2, 1)).sum((0, 2))
        tol = 1e-2 + 4 * 2 ** -9 * var.sqrt()
        err = (got["dsink"].float().cpu() - ref["dsink"]).abs()
        assert (err <= tol).all(), f"dsink err {err.tolist()} > {tol.tolist()}"
    return got, ref


@pytest.mark.parametrize("kind", MASKS)
def test_masks_d128_gqa(kind, fwd_variant):
    _run(kind, 2, 384, 384, 4, 2, 128, 128, seed=11)
    _run(kind, 1, 1024, 1024, 2, 1, 128, 128, seed=12)
    assert _kernel_status() == 0


@pytest.mark.parametrize("kind", ["causal_doc", "bidir_doc", "four_column", "none_causal"])
def test_ragged_shapes(kind, fwd_variant):
    # sequence lengths that are not multiples of any tile, Sq != Sk
    _run(kind, 1, 300, 300, 2, 2, 128, 128, seed=3)
    if kind in ("causal_doc", "none_causal"):
        _run(kind, 1, 203, 333, 2, 1, 64, 64, seed=4)
        _run(kind, 1, 203, 333, 2, 1, 128, 128, seed=4)
        _run(kind, 2, 333, 203, 2, 2, 128, 128, seed=4)
    assert _kernel_status() == 0


@pytest.mark.parametrize("d,dv,Hq,Hkv", [(64, 64, 2, 2), (80, 80, 2, 1), (128, 128, 4, 1),
                                         (192, 128, 4, 2), (256, 256, 2, 2), (576, 512, 2, 1),
                                         (512, 512, 2, 1)])
@pytest.mark.parametrize("kind", ["causal_doc", "bidir_doc"])
def test_head_dims(kind, d, dv, Hq, Hkv):
    _run(kind, 1, 320, 320, Hq, Hkv, d, dv, sink=True, seed=5)


@pytest.mark.parametrize("kind", MASKS)
def test_masks_d192(kind):
    """Every mask family through the 192 / 128 variants of the tcgen05 kernels (forward: two-slot K/V ring,
    twelve k-steps per score GEMM; backward: three-slot ring, single dP buffer, operands written over the
    score buffer): GQA, ragged sizes, rows long enough to wrap the rings many times."""
    _run(kind, 2, 384, 384, 4, 2, 192, 128, seed=31)
    _run(kind, 1, 1411, 1411, 2, 1, 192, 128, sink=True, seed=32)
    assert _kernel_status() == 0


@pytest.mark.parametrize("d,dv", [(192, 128), (256, 256)])
@pytest.mark.parametrize("kind", ["causal_doc", "none_causal", "bidir_doc"])
def test_ragged_shapes_big_head_dims(kind, d, dv):
    """Sq != Sk and lengths that are no multiple of any tile through the 192 / 128 and 256 / 256 variants."""
    _run(kind, 1, 300, 300, 2, 2, d, dv, seed=61)
    if kind != "bidir_doc":
        _run(kind, 1, 203, 333, 2, 1, d, dv, sink=True, seed=62)
        _run(kind, 2, 333, 203, 4, 2, d, dv, seed=63)
    assert _kernel_status() == 0


@pytest.mark.parametrize("kind", MASKS)
def test_masks_d256_short_sequences(kind):
    """Batches of short sequences at 256 / 256: the forward of blocks of 128 rows (one CTA, its two warpgroups own the
    two halves of V / O).  One partial block, a full and a nearly empty one, three blocks with several key tiles."""
    for S in (40, 129, 300):
        _run(kind, 10, S, S, 8, 4, 256, 256, sink=True, seed=53)
    assert _kernel_status() == 0


@pytest.mark.parametrize("kind", ["causal_doc", "none_full", "sliding_window"])
@pytest.mark.parametrize("B,S,Hq,Hkv,d,dv", [(3, 300, 4, 2, 256, 256), (5, 130, 2, 1, 576, 512), (4, 64, 4, 4, 256, 256),
                                             (4, 65, 4, 4, 256, 256), (2, 257, 3, 3, 512, 512)])
def test_batches_through_the_pair_backward(kind, B, S, Hq, Hkv, d, dv):
    """Heads of several batch entries in one pair of launches, masks of their own, either side of the line to the
    warp-MMA kernels."""
    _run(kind, B, S, S, Hq, Hkv, d, dv, sink=True, seed=55)
    _run(kind, B, S, S, Hq, Hkv, d, dv, seed=56, hm=Hkv if Hkv > 1 else 1)
    assert _kernel_status() == 0


@pytest.mark.parametrize("kind", ["causal_doc", "random_eviction", "bidir_doc", "four_column"])
@pytest.mark.parametrize("S", [512, 513, 515])
def test_bounds_of_partial_tiles_in_the_pair_backward(kind, S):
    """The mask forms of partial tiles (one, two and four bounds per column), whole and ragged tiles, and bounds whose
    rows start on and off a 16-byte boundary (a second mask head after an odd number of columns)."""
    _run(kind, 1, S, S, 2, 2, 256, 256, seed=59, hm=2)
    assert _kernel_status() == 0


def _pair_row_bytes(Sk, G):
    return G * -(-Sk // 256) * 256 * 4          # P and dS of one query row of every head of a group


@pytest.mark.parametrize("kind", ["causal_doc", "none_causal", "four_column"])
@pytest.mark.parametrize("d,dv", [(256, 256), (512, 512), (576, 512)])
def test_pair_backward_in_smaller_workspaces(d, dv, kind):
    """The chunks of the CTA-pair backward: whole groups, one group, row chunks whose dK / dV are summed in fp32 (the
    last one short, some without visible work for a key block), and none at all (the warp-MMA kernels, on mask
    reductions over wider tiles than their own)."""
    B, S, Hq, Hkv = 2, 700, 8, 1
    G = Hq // Hkv
    idx_np, causal = _mask(kind, B, S, S, 57)
    idx = None if idx_np is None else torch.from_numpy(np.ascontiguousarray(idx_np).copy()).cuda()
    q, k, v, do, s = make_inputs(B, S, S, Hq, Hkv, d, dv, 57, sink=True)
    dev = [t.cuda() for t in (q, k, v, do)]
    ref = run_oracle(q, k, v, do, idx, causal, s)
    lowp = naive_lowp(*dev, idx, causal, s)
    stats = 2 * 4 * B * Hq * 768
    row, sums = _pair_row_bytes(S, G), 768 * (d + dv) * 4
    # (workspace, launches of the score and gradient kernels: two per chunk)
    sizes = [(stats + 2 * 768 * row, 2), (stats + 768 * row, 4), (stats + 768 * row - 1, 8),
             (stats + 512 * row + sums, 8), (stats + 256 * row + sums, 12), (stats + 256 * row + sums - 1, 2), (stats, 2)]
    full = None
    for nbytes, launches in sizes:
        got = run_c_abi(*dev, idx, causal, s, workspace=nbytes, count=(before := []))
        assert before[0] == launches + 2, (nbytes, before)          # + row statistics and sink gradient
        assert_parity(got, ref, lowp, label=f"{nbytes}: ")
        again = run_c_abi(*dev, idx, causal, s, workspace=nbytes)
        for n in ("dq", "dk", "dv", "dsink"):
            assert torch.equal(got[n], again[n]), n
        full = full or got
        if nbytes >= stats + 256 * row + sums:
            assert torch.equal(got["dq"], full["dq"])               # only dK and dV are summed in another order
    with pytest.raises(RuntimeError, match="workspace too small"):
        run_c_abi(*dev, idx, causal, s, workspace=stats - 1)
    # without a workspace: the warp-MMA kernels
    got = run_c_abi(*dev, idx, causal, s, static_scratch=True)
    least = run_c_abi(*dev, idx, causal, s, workspace=stats)
    for n in ("dq", "dk", "dv", "dsink"):
        assert torch.equal(got[n], least[n]), n
    assert _kernel_status() == 0


def test_backward_when_memory_is_short():
    """A backward that gets no room for the workspace it asks for works in smaller chunks (an allocator limit of this
    process stands in for a full device)."""
    B, S, H, d = 1, 4096, 8, 256                                    # asks for 512 MiB
    q, k, v, do, _ = (t if t is None else t.cuda() for t in make_inputs(B, S, S, H, H, d, d, 58))
    x = [t.requires_grad_(True) for t in (q, k, v)]
    grads = lambda: torch.autograd.grad(fm.flashmask_attention(*x, causal=True), x, do)
    py = lambda: fm._flash_attn_bwd(q.detach(), k.detach(), v.detach(), *fwd, lse=lse, causal=True)[:3]
    with torch.no_grad():
        out, lse = fm._flash_attn_fwd(q, k, v, causal=True)
    fwd = (out, do)
    want = [t.clone() for t in grads()]
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    total = torch.cuda.get_device_properties(0).total_memory
    torch.cuda.set_per_process_memory_fraction((torch.cuda.memory_reserved() + (256 << 20)) / total)
    try:
        with pytest.raises(torch.OutOfMemoryError):
            torch.empty(512 << 20, dtype=torch.uint8, device="cuda")
        for call in (grads, py):
            for g_, w_ in zip(call(), want):
                # the sums of dK and dV are rounded to bf16 once, from another order of fp32 additions
                assert (g_.float() - w_.float()).norm() <= 2 ** -8 * w_.float().norm()
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)
    assert _kernel_status() == 0


def test_backward_without_room_for_its_accumulator():
    """Between the head dims 64 and 128 a backward that gets no room for the accumulator runs the two kernels, and holds
    no more memory than they use."""
    B, S, Hq, Hkv, d = 2, 8192, 16, 8, 96
    q, k, v, do, _ = (t if t is None else t.cuda() for t in make_inputs(B, S, S, Hq, Hkv, d, d, 58))
    x = [t.requires_grad_(True) for t in (q, k, v)]
    want = torch.autograd.grad(fm.flashmask_attention(*x, causal=True, deterministic=True), x, do)
    out, lse = fm.flashmask_attention(*x, causal=True, return_lse=True, deterministic=False)
    native = lambda: torch.autograd.grad(out, x, do, retain_graph=True)
    py = lambda: fm._flash_attn_bwd(q.detach(), k.detach(), v.detach(), out.detach(), do, lse, causal=True)[:3]
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    rows, results = B * Hq * S, sum(t.numel() * 2 for t in x)
    assert rows * 552 > 128 << 20
    total = torch.cuda.get_device_properties(0).total_memory
    torch.cuda.set_per_process_memory_fraction((torch.cuda.memory_reserved() + results + (100 << 20)) / total)
    try:
        for call in (native, py):
            torch.cuda.reset_peak_memory_stats()
            before = torch.cuda.memory_allocated()
            got = call()
            assert torch.cuda.max_memory_allocated() - before <= results + 8 * rows + (1 << 20)
            assert all(torch.equal(g_, w_) for g_, w_ in zip(got, want))
            del got
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)
    assert _kernel_status() == 0


@pytest.mark.parametrize("d,dv", [(512, 512), (576, 512)])
@pytest.mark.parametrize("kind", ["causal_doc", "none_full", "four_column"])
def test_short_sequences_of_the_widest_heads(kind, d, dv):
    """Batches of short sequences at 512 and 576 / 512: the warp-MMA forward, here with mask reductions over tiles
    wider than its own."""
    for S in (33, 64, 100):
        _run(kind, 16, S, S, 8, 1, d, dv, sink=True, seed=54)
    assert _kernel_status() == 0


@pytest.mark.parametrize("kind", MASKS)
def test_masks_d256(kind):
    """Every mask family through the CTA-pair kernels at 256 / 256, forward and backward."""
    _run(kind, 2, 384, 384, 4, 2, 256, 256, seed=51)
    _run(kind, 1, 1411, 1411, 2, 1, 256, 256, sink=True, seed=52)
    assert _kernel_status() == 0


@pytest.mark.parametrize("d,dv", [(576, 512), (512, 512)])
@pytest.mark.parametrize("kind", MASKS)
def test_masks_pair_kernels_two_slices(kind, d, dv):
    """Every mask family through the CTA-pair kernels at the head dims whose V / O have two 256-column slices (and,
    at 576, whose dQ / dK have a 64-column rest): lengths off every tile, Sq != Sk, one CTA of a pair without rows,
    rows and keys long enough to wrap every ring, sink, GQA and MQA."""
    _run(kind, 1, 129, 129, 2, 1, d, dv, sink=True, seed=81)
    _run(kind, 2, 300, 300, 4, 2, d, dv, seed=82)
    _run(kind, 1, 1411, 1411, 2, 1, d, dv, sink=True, seed=83)
    if kind in ("causal_doc", "none_causal"):
        _run(kind, 1, 203, 333, 2, 1, d, dv, seed=84)
        _run(kind, 1, 333, 203, 2, 2, d, dv, seed=85)
    assert _kernel_status() == 0


@pytest.mark.parametrize("kind", ["none_causal", "none_full"])
@pytest.mark.parametrize("B,Sq,Sk,Hq,Hkv,d,dv,sink", [
    (1, 1, 2048, 8, 1, 128, 128, True),       # one query, every head of the group in one row block
    (2, 1, 2304, 4, 2, 64, 64, False),
    (1, 33, 4097, 8, 1, 128, 128, False),     # packed rows end inside the second sub-tile, one key in the last tile
    (1, 129, 2050, 6, 2, 96, 80, True),       # three heads per group: split, not packed; padded head dims
    (1, 300, 700, 4, 1, 128, 128, False),     # packed, too few keys to split
    (1, 4, 5000, 128, 1, 64, 64, False)])     # 128 heads per query: one query per sub-tile
def test_few_queries_many_keys(kind, B, Sq, Sk, Hq, Hkv, d, dv, sink):
    """The forward that packs the heads of a group into the rows of a CTA and deals the K tiles of a row block to
    several CTAs (calls without a mask tensor that would leave most of the chip idle)."""
    _run(kind, B, Sq, Sk, Hq, Hkv, d, dv, sink=sink, seed=91)
    _run(kind, B, Sq, Sk, Hq, Hkv, d, dv, sink=sink, seed=92, dtype=torch.float16)
    assert _kernel_status() == 0


@pytest.mark.parametrize("B,Sq,Sk,Hq,Hkv,d,dv", [
    (1, 1, 129, 4, 1, 128, 128),      # two tiles: one per sub-tile
    (2, 1, 300, 4, 4, 64, 64),        # an odd number of tiles, one row
    (1, 32, 641, 4, 1, 128, 128),     # 128 packed rows: a full sub-tile
    (1, 33, 641, 4, 1, 128, 128),     # 132: past it, so one tile serves both sub-tiles again
    (1, 128, 1500, 3, 1, 64, 48),     # 128 rows unpacked, several diagonal tiles
    (3, 2, 9000, 16, 2, 96, 96)])     # several CTAs per row block, some of them with an odd share
def test_rows_of_one_sub_tile(B, Sq, Sk, Hq, Hkv, d, dv):
    """Calls whose rows fit one sub-tile of a CTA: the two sub-tiles take the K tiles in turn and are merged."""
    for kind in ("none_causal", "none_full"):
        _run(kind, B, Sq, Sk, Hq, Hkv, d, dv, sink=True, seed=93)
    assert _kernel_status() == 0


@pytest.mark.parametrize("B,Sq,Sk,Hq,Hkv,d,dv,parts", [
    (160, 1, 200, 4, 4, 128, 128, 2),     # two tiles: one per sub-tile
    (150, 2, 330, 4, 4, 64, 64, 2),       # three
    (8, 32, 3000, 16, 4, 128, 128, 8),    # 128 packed rows, a full sub-tile; four CTAs of six tiles
    (3, 2, 9000, 16, 2, 96, 96, 24),      # a dozen CTAs, some of them with an odd share
    (1, 33, 641, 4, 1, 128, 128, 6),      # 132 packed rows: one tile serves both sub-tiles
    (300, 64, 140, 2, 2, 64, 64, 0)])     # a chip full of short calls: none
def test_partial_results(B, Sq, Sk, Hq, Hkv, d, dv, parts):
    """Either side of the rule that deals K tiles to several CTAs and to the two sub-tiles of a CTA."""
    import ctypes as C
    a = _lib.AttnArgs()
    a.B, a.Sq, a.Sk, a.Hq, a.Hkv, a.Hm, a.mask_B, a.d, a.dv, a.causal = B, Sq, Sk, Hq, Hkv, 1, 1, d, dv, 1
    assert _lib.load().fm_fwd_workspace_bytes(C.byref(a)) == B * Hq * Sq * parts * ((64 if d <= 64 else 128) + 1) * 4
    for kind in ("none_causal", "none_full"):
        _run(kind, B, Sq, Sk, Hq, Hkv, d, dv, sink=True, seed=94)
    assert _kernel_status() == 0


@pytest.mark.parametrize("what", ["k nan", "k inf", "q nan", "v nan", "v inf"])
@pytest.mark.parametrize("B,Sq,Sk,Hq,Hkv,d", [(1, 1, 8192, 4, 1, 128),       # split and alternating
                                              (160, 1, 200, 4, 4, 128),      # alternating only
                                              (1, 256, 8192, 2, 2, 128)])    # split only
def test_non_finite_inputs_of_a_split_forward(B, Sq, Sk, Hq, Hkv, d, what):
    """A NaN or an infinity that a query sees reaches its output whatever share of the keys holds it: the elements
    that are NaN or infinite are those of the dense softmax, the others are finite and right."""
    q, k, v, _, _ = (t if t is None else t.cuda() for t in make_inputs(B, Sq, Sk, Hq, Hkv, d, d, 95))
    q[0, 0, 0, 5] = q[0, 0, 0, 5].abs() + 1          # (the first query's score of an infinite key is +inf)
    dict(q=q, k=k, v=v)[what[0]][0, 0, 0, 5] = float(what[2:])
    with torch.no_grad():
        out, lse = fm.flashmask_attention(q, k, v, causal=True, return_lse=True)
    rep = lambda t: t.double().repeat_interleave(Hq // Hkv, dim=2).permute(0, 2, 1, 3)
    s = rep(q) if Hq == Hkv else q.double().permute(0, 2, 1, 3)
    s = s @ rep(k).transpose(-1, -2) / math.sqrt(d)
    hidden = torch.arange(Sk, device="cuda")[None] > torch.arange(Sq, device="cuda")[:, None] + Sk - Sq
    att = torch.softmax(s.masked_fill(hidden, -math.inf), -1)
    want = (att @ rep(v)).permute(0, 2, 1, 3)
    if what == "v inf":      # the weight of the infinite element is positive in both
        assert torch.isinf(want).any()
    else:
        assert torch.isnan(want).any()
    assert torch.equal(torch.isnan(out), torch.isnan(want)) and torch.equal(torch.isinf(out), torch.isinf(want))
    fin = torch.isfinite(want)
    # P and the result are rounded to 8 bits of mantissa each (half a unit: 2^-9 relative)
    bound = 2 ** -8 * (att @ rep(v).abs()).permute(0, 2, 1, 3)
    assert ((out.double() - want)[fin].abs() <= bound[fin]).all()
    bad = torch.isnan(want).all(-1)                  # rows whose softmax sum is NaN: LSE -inf, as in an unsplit call
    assert torch.equal(torch.isneginf(lse), bad.permute(0, 2, 1))
    assert _kernel_status() == 0


@pytest.mark.parametrize("kind", MASKS)
def test_masks_d64(kind, fwd_variant):
    """Every mask family through the 64-column variants: GQA, rows long enough to wrap the K/V ring."""
    _run(kind, 2, 384, 384, 4, 2, 64, 64, seed=21)
    _run(kind, 1, 1280, 1280, 2, 1, 64, 64, seed=22)
    assert _kernel_status() == 0


@pytest.mark.parametrize("d,dv", [(32, 32), (64, 32), (96, 96), (64, 128), (128, 64), (8, 8)])
def test_padded_head_dims(d, dv, fwd_variant):
    """Head dims below a variant's width: the columns past the end of a head must read as zeros and stay unwritten."""
    _run("causal_doc", 1, 333, 333, 2, 1, d, dv, sink=True, seed=23)
    _run("bidir_doc", 2, 256, 256, 2, 2, d, dv, seed=24)
    assert _kernel_status() == 0


@pytest.mark.parametrize("kind", ["causal_doc", "bidir_doc", "none_full"])
@pytest.mark.parametrize("d", [72, 80, 96, 104, 120])
def test_one_kernel_backward_between_64_and_128(d, kind):
    """320 key tiles fill the chip twice, so the one-kernel backward serves head dims that do not fill their second 64-column
    box: GEMMs that stop at 5, 6, 7 and 8 k-steps, ragged last tiles, and nothing past the end of a head.  With room for the
    row statistics only the two-kernel backward takes the call."""
    B, S, Hq, Hkv = 8, 517, 16, 8
    idx_np, causal = _mask(kind, B, S, S, 61)
    idx = None if idx_np is None else torch.from_numpy(np.ascontiguousarray(idx_np).copy()).cuda()
    q, k, v, do, s = make_inputs(B, S, S, Hq, Hkv, d, d, 61, sink=True)
    dev = [t.cuda() for t in (q, k, v, do)]
    stats = 2 * 4 * B * Hq * 640
    got = run_c_abi(*dev, idx, causal, s, deterministic=False)
    assert_parity(got, run_oracle(q, k, v, do, idx, causal, s), naive_lowp(*dev, idx, causal, s))
    least = run_c_abi(*dev, idx, causal, s, deterministic=False, workspace=stats)
    fixed = run_c_abi(*dev, idx, causal, s, deterministic=True)
    for n in ("dq", "dk", "dv", "dsink"):
        assert torch.equal(least[n], fixed[n]), n
    assert not torch.equal(got["dq"], fixed["dq"])              # sums over the key tiles in another order
    assert _kernel_status() == 0


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("Sq,Sk,Hq,Hkv", [(517, 517, 16, 8), (330, 645, 32, 8)])
@pytest.mark.parametrize("d", [72, 88, 96, 112, 120])
def test_one_kernel_backward_between_64_and_128_walks_units(d, Sq, Sk, Hq, Hkv, dtype, monkeypatch):
    """The same with launch tables, as masked calls of both hosts run it: a CTA takes several of 320 or 384 units, some of
    them empty, over accumulators as wide as the head.  dK and dV are bitwise those of one unit per CTA; nothing of the
    workspace reaches a result that the call has not written."""
    B = 8
    idx_np, causal = _mask("causal_doc", B, Sq, Sk, 63)
    idx_np = idx_np.copy()
    idx_np[1::2, :, 128:256, 0] = np.clip(np.arange(128, 256) - (Sk - Sq), 0, Sq)    # a key tile that no query sees
    idx = torch.from_numpy(np.ascontiguousarray(idx_np)).cuda()
    q, k, v, do, s = make_inputs(B, Sq, Sk, Hq, Hkv, d, d, 63, dtype=dtype, sink=True)
    dev = [t.cuda() for t in (q, k, v, do)]
    sizes, plain = [], fm.ops._bwd_workspace

    def workspace_of_nans(a, device):
        ws = plain(a, device).fill_(255)
        sizes.append(ws.numel())
        return ws
    got = run_product(*dev, idx, causal, s, deterministic=False)
    assert_parity(got, run_oracle(q, k, v, do, idx, causal, s), naive_lowp(*dev, idx, causal, s))
    monkeypatch.setattr(fm.ops, "_bwd_workspace", workspace_of_nans)
    info = fm.prepare_mask(idx, Sq, causal, 128, 128)
    py = fm._flash_attn_bwd(*dev[:3], got["out"], dev[3], got["lse"], idx, causal=causal, learnable_sink=s, mask_info=info)
    assert sizes == [B * Hq * -(-Sq // 128) * 128 * 552]               # with the accumulator: the one kernel
    assert any(t is not None for key, t in info.orders.items() if key[0] == _lib.FM_ORDER_BWD_DKDV)
    alone = run_c_abi(*dev, idx, causal, s, deterministic=False)
    for n, t in zip(("dq", "dk", "dv", "dsink"), py):
        assert torch.isfinite(t).all()
        if n != "dq":
            assert torch.equal(t, got[n]) and torch.equal(t, alone[n]), n
    # dQ: fp32 sums over six key tiles in any order, rounded to 16 bits once
    u = 2 ** -8 if dtype == torch.bfloat16 else 2 ** -11
    assert ((py[0].double() - got["dq"].double()).norm() <= u * got["dq"].double().norm())
    assert _kernel_status() == 0


def _assert_gradients_as_in_64_bits(d, B, Sq, Sk, Hq, Hkv, idx_np, causal, dtype):
    G, scale, dv = Hq // Hkv, 1 / math.sqrt(d), min(d, 128)
    idx = None if idx_np is None else torch.from_numpy(np.ascontiguousarray(idx_np).copy()).cuda()
    q, k, v, do, _ = (t if t is None else t.cuda().to(dtype) for t in make_inputs(B, Sq, Sk, Hq, Hkv, d, dv, 72))
    x = [t.detach().requires_grad_(True) for t in (q, k, v)]
    out, lse = fm.flashmask_attention(*x, idx, causal=causal, return_lse=True)
    got = torch.autograd.grad(out, x, do)
    i, j = torch.arange(Sq, device="cuda")[:, None], torch.arange(Sk, device="cuda")
    visible = (j <= i + Sk - Sq if causal else torch.ones(Sq, Sk, device="cuda", dtype=torch.bool))[None, None]
    if idx_np is not None:
        visible = torch.from_numpy(oracle.dense_bias(idx_np, Sq, Sk, causal)).cuda() == 0
    heads = lambda t: t.double().permute(0, 2, 1, 3)
    by_key = lambda t: t.reshape(B, Hkv, G, Sk, -1).sum(2)
    u, tiny = (2 ** -8, 0.0) if dtype == torch.bfloat16 else (2 ** -11, 2 ** -25)
    q64, do64, k64, v64 = heads(q), heads(do), *(heads(t).repeat_interleave(G, dim=1) for t in (k, v))
    lse = torch.nan_to_num(lse.detach().double(), neginf=0.0)[..., None]
    p = torch.exp((q64 @ k64.transpose(-1, -2) * scale - lse).masked_fill(~visible, -math.inf))
    ds = p * (do64 @ v64.transpose(-1, -2) - (heads(out.detach()) * do64).sum(-1, keepdim=True))
    ref = [scale * ds @ k64, by_key(scale * ds.transpose(-1, -2) @ q64), by_key(p.transpose(-1, -2) @ do64)]
    # P and dS are rounded to the 16-bit type (and S, dP and the sums to fp32: some 2^-16 of the largest terms), the results once more
    d_p, d_ds = p * (u + 2 ** -14) + tiny, ds.abs() * (u + 2 ** -14) + p * 2 ** -14 + tiny
    bound = [scale * d_ds @ k64.abs(), by_key(scale * d_ds.transpose(-1, -2) @ q64.abs()), by_key(d_p.transpose(-1, -2) @ do64.abs())]
    for g_, r, b, n in zip(got, ref, bound, ("dq", "dk", "dv")):
        assert torch.isfinite(g_).all(), n
        assert ((heads(g_) - r).abs() <= b + u * r.abs() + 2 * tiny + 1e-6).all(), n
    assert _kernel_status() == 0


@pytest.mark.parametrize("d,B,Sq,Sk,Hq,Hkv,kind", [
    (64, 1, 1, 130, 2, 1, "none_causal"),             # one query: items, row groups and boxes of one row
    (64, 1, 65, 65, 3, 1, "causal_doc"),              # odd numbers of items, a second item of one query
    (64, 2, 200, 129, 4, 2, "bidir_doc"),             # more queries than keys, a key tile of one key
    (64, 1, 449, 449, 2, 2, "sliding_window"),
    (64, 24, 517, 517, 16, 8, "causal_doc"),          # CTAs walk several units; one in ten is empty, at the end of the table
    (128, 1, 15, 257, 2, 1, "none_causal"),
    (128, 2, 63, 64, 1, 1, "none_full"),
    (128, 1, 333, 200, 6, 2, "bidir_doc"),
    (128, 24, 517, 517, 16, 8, "causal_doc"),
    (192, 1, 1, 65, 2, 1, "none_causal"),             # (two kernels, both warpgroups on an item)
    (192, 2, 333, 200, 6, 2, "bidir_doc"),
    (192, 1, 700, 700, 3, 1, "causal_doc")])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_backward_at_the_edges_of_items_units_and_accumulator(d, B, Sq, Sk, Hq, Hkv, kind, dtype):
    """dQ, dK and dV against 64 bits where items, units and the blocks of the dQ accumulator are not whole."""
    idx_np, causal = _mask(kind, B, Sq, Sk, 71)
    if kind == "causal_doc" and B > 1:
        idx_np = idx_np.copy()
        idx_np[::2, :, 128:256] = 0                   # nobody sees the second key tile of every other sequence
    _assert_gradients_as_in_64_bits(d, B, Sq, Sk, Hq, Hkv, idx_np, causal, dtype)


@pytest.mark.parametrize("what", ["runs of empty units", "empty and light units"])
@pytest.mark.parametrize("d,dtype", [(64, torch.bfloat16), (64, torch.float16), (40, torch.bfloat16), (128, torch.bfloat16)])
def test_backward_walks_units_that_nobody_sees(d, dtype, what):
    """Key tiles without a query among the units that a CTA of the one-kernel backward walks: runs of four and more of them
    behind two others, and, where one document is much longer than the rest, in turn with tiles of one or two items."""
    if what == "runs of empty units":
        B, S, H = 37, 300, 8                          # 888 units, two of three empty
        idx_np, causal = _mask("causal_doc", B, S, S, 73)
        idx_np = idx_np.copy()
        for b in range(B):
            for n in range(3):
                if n != b % 3:
                    idx_np[b, :, 128 * n:128 * n + 128] = 0
    else:
        B, S, H = 6, 2100, 8                          # 816 units; the long document's reach 33 items
        short = [[61] * (S // 61) + [S % 61] for _ in range(B - 1)]
        idx_np = np.concatenate([W.causal_document(1, S, S, np.array(lens))[0] for lens in [[S]] + short])
        causal = True
        for b in range(1, B):
            for n in range(17):
                if (n * n + b) % 3 == 0:
                    idx_np[b, :, 128 * n:128 * n + 128] = 0
                elif (n + b) % 2:
                    idx_np[b, :, 128 * n + 50:128 * n + 128] = 0     # fewer items still
    _assert_gradients_as_in_64_bits(d, B, S, S, H, H, idx_np, causal, dtype)


@pytest.mark.parametrize("what", ["row sums", "scores", "small scale"])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("d", [64, 96, 128])
def test_row_statistics_beyond_16_bits(d, dtype, what):
    """rowsum(O dO) of a million, LSE of thousands, LSE / scale of a hundred thousand: the backward subtracts both with the
    range and precision of fp32, whatever the type of the call and whichever kernels serve it (320 key tiles: the
    one-kernel backward, with launch tables).  Against 64 bits, on the O and LSE that the backward reads."""
    B, S, Hq, Hkv = 8, 517, 16, 8
    G, scale = Hq // Hkv, 5e-5 if what == "small scale" else 1 / math.sqrt(d)
    idx_np, causal = _mask("causal_doc", B, S, S, 61)
    idx = torch.from_numpy(np.ascontiguousarray(idx_np).copy()).cuda()
    q, k, v, do, _ = (t if t is None else t.cuda().float() for t in make_inputs(B, S, S, Hq, Hkv, d, d, 62))
    if what == "row sums":
        v, do = v + 128, do + 100
    elif what == "scores":
        q, k, do = 20 + q / 8, 20 + k / 8, do.abs()
    q, k, v, do = (t.to(dtype) for t in (q, k, v, do))
    visible = torch.from_numpy(oracle.dense_bias(idx_np, S, S, causal)).cuda() == 0
    heads = lambda t: t.double().permute(0, 2, 1, 3)
    q64, do64 = heads(q), heads(do)
    k64, v64 = (heads(t).repeat_interleave(G, dim=1) for t in (k, v))
    by_key = lambda t: t.reshape(B, Hkv, G, S, -1).sum(2)              # the q heads of a group share dK and dV
    u, tiny = (2 ** -8, 0.0) if dtype == torch.bfloat16 else (2 ** -11, 2 ** -25)
    for deterministic in (False, True):
        x = [t.detach().requires_grad_(True) for t in (q, k, v)]
        out, lse = fm.flashmask_attention(*x, idx, causal=causal, softmax_scale=scale, return_lse=True,
                                          deterministic=deterministic)
        got = torch.autograd.grad(out, x, do)
        dsum = (heads(out.detach()) * do64).sum(-1, keepdim=True)
        lse = lse.detach().double()[..., None]
        if what == "row sums":
            assert dsum.abs().min() > 65504
        else:
            assert (lse / scale).abs().median() > 2e4
        # exponent and dP - rowsum(O dO): fp32 sums of head-dim products, a few units of 2^-24 of their largest terms;
        # the exponent is then a relative error of P (and exp2 itself has one of 2^-22)
        p = torch.exp(q64 @ k64.transpose(-1, -2) * scale - lse) * visible
        e_p = 2 ** -21 * (scale * q64.norm(dim=-1, keepdim=True) * k64.norm(dim=-1)[:, :, None] + lse.abs() + 1)
        dp = do64 @ v64.transpose(-1, -2) - dsum
        e_dp = 2 ** -21 * (do64.norm(dim=-1, keepdim=True) * v64.norm(dim=-1)[:, :, None] + dsum.abs())
        ds = p * dp
        # P and dS are rounded to the 16-bit type, the results once more; the sums are fp32
        d_p = p * (e_p + u + 2 ** -18) + tiny
        d_ds = ds.abs() * (e_p + u + 2 ** -18) + p * e_dp + tiny
        ref = [(scale * ds) @ k64, by_key((scale * ds).transpose(-1, -2) @ q64), by_key(p.transpose(-1, -2) @ do64)]
        bound = [scale * (d_ds @ k64.abs()), by_key(scale * (d_ds.transpose(-1, -2) @ q64.abs())),
                 by_key(d_p.transpose(-1, -2) @ do64.abs())]
        for g_, r, b, n in zip(got, ref, bound, ("dq", "dk", "dv")):
            err = (heads(g_) - r).abs()
            assert (err <= b + u * (r.abs() + b) + tiny).all(), (n, deterministic, (err - b).max().item())
    assert _kernel_status() == 0


@pytest.mark.parametrize("kind", ["none_causal", "causal_doc", "random_eviction"])
def test_sink(kind, fwd_variant):
    _run(kind, 2, 256, 256, 4, 2, 128, 128, sink=True, seed=7)


def test_mask_heads_per_kv_head(fwd_variant):
    _run("causal_doc", 2, 256, 256, 4, 2, 128, 128, seed=8, hm=2)


def test_fp16(fwd_variant):
    _run("causal_doc", 1, 256, 256, 2, 2, 128, 128, seed=9, dtype=torch.float16)
    _run("bidir_doc", 1, 384, 384, 4, 2, 64, 64, seed=10, dtype=torch.float16)


def test_long_rows_many_tiles(fwd_variant):
    """Enough K tiles per Q tile to wrap the K/V ring and the bounds slots many times."""
    _run("random_eviction", 1, 2048, 2048, 2, 1, 128, 128, seed=13)
    _run("sliding_window", 1, 2048, 2048, 1, 1, 128, 128, seed=14)
    assert _kernel_status() == 0


def test_cpu_config_shape():
    """The CPU-runnable configuration: B=1, H=2, S=1024, d=64, 4 documents."""
    w = W.make_workload("cpu_causal_doc_1k")
    q, k, v, do, _ = make_inputs(w.B, w.Sq, w.Sk, w.Hq, w.Hkv, w.d, w.dv, w.seed)
    idx = torch.from_numpy(w.idx).cuda()
    got = run_product(q.cuda(), k.cuda(), v.cuda(), do.cuda(), idx, w.causal, None)
    ref = run_oracle(q, k, v, do, idx, w.causal, None)
    lowp = naive_lowp(q.cuda(), k.cuda(), v.cuda(), do.cuda(), idx, w.causal, None)
    assert_parity(got, ref, lowp)
    assert_lse(got, ref)


@pytest.mark.parametrize("path", GOLDEN, ids=lambda p: os.path.basename(p)[10:-4])
def test_against_reference_golden(path):
    """Vectors produced by the reference's own dense-mask attention (fp32).
    Head dim 16 is padded to the 64 bucket by the kernels."""
    z = np.load(path)
    c = {k_: z[k_] for k_ in z.files}
    causal = bool(c["causal"])
    dt = torch.bfloat16
    q, k, v, do = (torch.from_numpy(c[n]).to(dt) for n in ("q", "k", "v", "do"))
    sink = torch.from_numpy(c["sink"]) if "sink" in c else None
    idx = torch.from_numpy(c["idx"]).cuda() if "idx" in c else None
    got = run_product(q.cuda(), k.cuda(), v.cuda(), do.cuda(), idx, causal, sink)
    ref = run_oracle(q, k, v, do, idx, causal, sink)       # oracle on the bf16-rounded inputs
    lowp = naive_lowp(q.cuda(), k.cuda(), v.cuda(), do.cuda(), idx, causal, sink)
    assert_parity(got, ref, lowp)
    # and against the stored reference outputs themselves (fp32 inputs there, bf16 here)
    for n in ("out", "dq", "dk", "dv"):
        err = (got[n].float().cpu() - torch.from_numpy(c[n])).abs().max().item()
        assert err < 0.15, (n, err)


def test_deterministic_bitwise(fwd_variant):
    idx_np, causal = _mask("causal_doc", 2, 512, 512, 21)
    q, k, v, do, s = make_inputs(2, 512, 512, 8, 2, 128, 128, 21, sink=True)
    idx = torch.from_numpy(np.ascontiguousarray(idx_np).copy()).cuda()
    a = run_product(q.cuda(), k.cuda(), v.cuda(), do.cuda(), idx, causal, s, deterministic=True)
    for _ in range(3):
        b = run_product(q.cuda(), k.cuda(), v.cuda(), do.cuda(), idx, causal, s, deterministic=True)
        for n in ("out", "lse", "dq", "dk", "dv", "dsink"):
            assert torch.equal(a[n], b[n]), n


def test_d192_deterministic_bitwise_and_fp16():
    """The 192 / 128 backward is the two-kernel variant whatever `deterministic` says: repeated runs are
    bitwise equal (sink gradient included); fp16 inputs run the same kernels."""
    idx_np, causal = _mask("share_question", 2, 640, 640, 41)
    q, k, v, do, s = make_inputs(2, 640, 640, 8, 2, 192, 128, 41, sink=True)
    idx = torch.from_numpy(np.ascontiguousarray(idx_np).copy()).cuda()
    a = run_product(q.cuda(), k.cuda(), v.cuda(), do.cuda(), idx, causal, s, deterministic=True)
    for det in (True, False, True):
        b = run_product(q.cuda(), k.cuda(), v.cuda(), do.cuda(), idx, causal, s, deterministic=det)
        for n in ("out", "lse", "dq", "dk", "dv", "dsink"):
            assert torch.equal(a[n], b[n]), (n, det)
    _run("causal_doc", 1, 448, 448, 4, 2, 192, 128, seed=42, dtype=torch.float16)
    assert _kernel_status() == 0


@pytest.mark.parametrize("persist", ["0", "1"])
@pytest.mark.parametrize("kind,mask_b,hm", [("causal_doc", 2, 1), ("four_column", 1, 2), ("share_question", 2, 2),
                                            ("bidir_doc", 1, 1)])
def test_launch_order_changes_no_bit(kind, mask_b, hm, persist, monkeypatch):
    """The longest-work-first launch order only permutes which CTA runs which tile, and the
    persistent backward variant only changes which CTA runs which unit: results are bitwise
    those of the index order, for every mask batch / head broadcast and both backward variants."""
    monkeypatch.setenv("FLASHMASK_B200_PERSIST", persist)
    _lib.reload_options()
    B, S, Hq, Hkv = 2, 1024, 8, 2
    idx_np, causal = _mask(kind, B, S, S, 33)
    idx_np = np.ascontiguousarray(idx_np[:mask_b]).copy()
    if hm > 1:   # distinct masks per mask head
        other = np.clip(idx_np + np.array(S // 7, dtype=np.int32), 0, S).astype(np.int32)
        idx_np = np.concatenate([idx_np, other], axis=1)
    q, k, v, do, s = make_inputs(B, S, S, Hq, Hkv, 128, 128, 33, sink=True)
    idx = torch.from_numpy(idx_np).cuda()
    monkeypatch.setenv("FLASHMASK_B200_ORDER", "0")
    a = run_product(q.cuda(), k.cuda(), v.cuda(), do.cuda(), idx, causal, s, deterministic=True)
    monkeypatch.setenv("FLASHMASK_B200_ORDER", "1")
    b = run_product(q.cuda(), k.cuda(), v.cuda(), do.cuda(), idx, causal, s, deterministic=True)
    for n in ("out", "lse", "dq", "dk", "dv", "dsink"):
        assert torch.equal(a[n], b[n]), n


def test_launch_tables_are_reusable():
    """One FlashMaskInfo (one set of launch tables, whose unit counters the persistent backward
    advances and rewinds) serves many launches: every repeat gives the first result."""
    B, S, Hq, Hkv = 1, 2048, 4, 2
    idx_np, causal = _mask("causal_doc", B, S, S, 9)
    q, k, v, do, _ = make_inputs(B, S, S, Hq, Hkv, 128, 128, 9)
    q, k, v, do = q.cuda(), k.cuda(), v.cuda(), do.cuda()
    idx = torch.from_numpy(np.ascontiguousarray(idx_np).copy()).cuda()
    info = fm.prepare_mask(idx, S, causal, 128, 128)
    out, lse = fm._flash_attn_fwd(q, k, v, idx, causal=causal, mask_info=info)
    first = fm._flash_attn_bwd(q, k, v, out, do, lse, idx, causal=causal, mask_info=info)
    assert any(t is not None for t in info.orders.values())
    for _ in range(4):
        out2, lse2 = fm._flash_attn_fwd(q, k, v, idx, causal=causal, mask_info=info)
        again = fm._flash_attn_bwd(q, k, v, out, do, lse, idx, causal=causal, mask_info=info)
        assert torch.equal(out, out2) and torch.equal(lse, lse2)
        for a, b in zip(first[:3], again[:3]):
            assert torch.equal(a, b)
    # the counters behind the backward tables are back at zero
    torch.cuda.synchronize()
    for key, t in info.orders.items():
        if t is not None and key[0] != 0:
            assert t[-4:-2].tolist() == [0, 0], key


def test_layout_invariance(fwd_variant):
    """Contiguous vs permuted storage of q/k/v give bitwise equal results
    (reference: tests/torch/test_flashmask.py:354-396)."""
    idx_np, causal = _mask("causal_doc", 1, 256, 256, 5)
    q, k, v, do, _ = make_inputs(1, 256, 256, 4, 2, 128, 128, 5)
    idx = torch.from_numpy(np.ascontiguousarray(idx_np).copy()).cuda()
    a = run_product(q.cuda(), k.cuda(), v.cuda(), do.cuda(), idx, causal, None, deterministic=True)

    def bhsd(t):  # same values, [B,H,S,D] storage viewed as [B,S,H,D]
        return t.cuda().permute(0, 2, 1, 3).contiguous().permute(0, 2, 1, 3)
    b = run_product(bhsd(q), bhsd(k), bhsd(v), bhsd(do), idx, causal, None, deterministic=True)
    for n in ("out", "dq", "dk", "dv"):
        assert torch.equal(a[n], b[n]), n


@pytest.mark.parametrize("what", ["kv batch", "kv heads", "q batch", "do batch", "k rows"])
@pytest.mark.parametrize("d,dv", [(64, 64), (128, 128), (192, 128), (256, 256), (512, 512), (576, 512)])
def test_expanded_tensors(d, dv, what):
    """Tensors that repeat along a dimension (stride 0).  Through the operator they are copied: bitwise the call on
    dense copies.  Through the C ABI the warp-MMA kernels take them as they are, with mask reductions over the wider
    tiles of the kernels that would have run."""
    B, S, Hq, Hkv = 2, 200, 4, 2
    idx_np, causal = _mask("causal_doc", B, S, S, 71)
    idx = torch.from_numpy(np.ascontiguousarray(idx_np).copy()).cuda()
    q, k, v, do, s = make_inputs(B, S, S, Hq, Hkv, d, dv, 71, sink=True)
    q, k, v, do = q.cuda(), k.cuda(), v.cuda(), do.cuda()
    if what == "kv batch":
        k, v = k[:1].expand_as(k), v[:1].expand_as(v)
    elif what == "kv heads":
        k, v = k[:, :, :1].expand_as(k), v[:, :, :1].expand_as(v)
    elif what == "q batch":
        q = q[:1].expand_as(q)
    elif what == "do batch":
        do = do[:1].expand_as(do)
    else:
        k = k[:, :1].expand_as(k)
    dense = [t.contiguous() for t in (q, k, v, do)]
    assert any(0 in t.stride() for t in (q, k, v, do)) and not any(0 in t.stride() for t in dense)
    leaves = [t.detach().requires_grad_(True) for t in (q, k, v)]
    out, lse = fm.flashmask_attention(*leaves, idx, causal=causal, sink=s.cuda(), return_lse=True, deterministic=True)
    got = [out.detach(), lse, *torch.autograd.grad(out, leaves, do)]
    ref = run_product(*dense, idx, causal, s, deterministic=True)
    for g_, n in zip(got, ("out", "lse", "dq", "dk", "dv")):
        assert torch.equal(g_, ref[n]), n
    raw = run_c_abi(q, k, v, do, idx, causal, s)
    cpu = [t.cpu() for t in dense]
    oracle_ = run_oracle(*cpu, idx, causal, s)
    assert_parity(raw, oracle_, naive_lowp(*dense, idx, causal, s))
    assert_lse(raw, oracle_)
    assert _kernel_status() == 0


@pytest.mark.parametrize("scale", [0.0, -0.07])
@pytest.mark.parametrize("d,dv", [(64, 64), (128, 128), (192, 128), (256, 256), (512, 512), (576, 512)])
def test_scale_that_is_not_positive(d, dv, scale):
    """A masked score stays masked whatever the sign of the scale (0: every visible key has the same weight)."""
    S = 200
    idx_np, causal = _mask("causal_doc", 1, S, S, 73)
    idx = torch.from_numpy(np.ascontiguousarray(idx_np).copy()).cuda()
    q, k, v, do, _ = (t if t is None else t.cuda() for t in make_inputs(1, S, S, 2, 2, d, dv, 73))
    x = [t.clone().requires_grad_(True) for t in (q, k, v)]
    out, lse = fm.flashmask_attention(*x, idx, causal=causal, softmax_scale=scale, return_lse=True)
    got = [out.detach(), *torch.autograd.grad(out, x, do)]
    y = [t.double().requires_grad_(True) for t in (q, k, v)]
    s = torch.einsum("bihd,bjhd->bhij", y[0], y[1]) * scale + torch.from_numpy(oracle.dense_bias(idx_np, S, S, causal)).cuda()
    ref = torch.einsum("bhij,bjhd->bihd", torch.softmax(s, -1), y[2])
    assert (lse.double() - torch.logsumexp(s, -1)).abs().max() < 1e-4
    for g_, r, n in zip(got, [ref.detach(), *torch.autograd.grad(ref, y, do.double())], ("out", "dq", "dk", "dv")):
        # P, dS and the results are rounded to 16 bits: a few units of 2^-9 in the 2-norm
        assert (g_.double() - r).norm() <= 1e-2 * r.norm(), n
    assert _kernel_status() == 0


def test_expanded_shared_key_value():
    """One latent shown to every batch entry, the value a view of it: gradients as on a dense copy (dV folded into
    dK, the value's own gradient zero)."""
    B, S, d, dv = 2, 160, 576, 512
    q, k, _, do, _ = make_inputs(B, S, S, 2, 1, d, dv, 72)
    q, do, lat = q.cuda(), do.cuda(), k[:1].cuda()
    res = []
    for kk in (lat.expand(B, S, 1, d), lat.expand(B, S, 1, d).contiguous()):
        kk = kk.detach().requires_grad_(True)
        vv = kk[..., :dv].detach().requires_grad_(True)
        out = fm.flashmask_attention(q, kk, vv, causal=True, deterministic=True)
        res.append([out.detach(), *torch.autograd.grad(out, [kk, vv], do)])
    assert float(res[0][2].abs().max()) == 0.0 and float(res[0][1].abs().max()) > 0.0
    for a, b in zip(*res):
        assert torch.equal(a, b)


@pytest.mark.parametrize("kind,d,dv,B,Hq,Hkv,hm,dtype,sink", [
    ("causal_doc", 64, 64, 2, 4, 2, 1, torch.bfloat16, torch.float32),      # launch tables
    ("four_column", 128, 128, 1, 4, 2, 2, torch.float16, torch.bfloat16),   # a mask per kv head
    ("bidir_doc", 96, 80, 2, 3, 3, 1, torch.bfloat16, None),                # padded head dims
    ("none_causal", 128, 128, 3, 4, 1, 1, torch.bfloat16, torch.float32),
    ("sliding_window", 192, 128, 1, 4, 2, 1, torch.bfloat16, torch.float32),  # two tile shapes
    ("share_question", 256, 256, 2, 2, 2, 1, torch.float16, torch.float32),
    ("causal_doc", 576, 512, 1, 4, 1, 1, torch.bfloat16, torch.bfloat16)])
@pytest.mark.parametrize("layout", ["dense", "transposed", "shared kv"])
def test_native_host_and_python_autograd_function_agree(kind, d, dv, B, Hq, Hkv, hm, dtype, sink, layout):
    """flashmask_attention (native checks, allocations, autograd node) against FlashMaskFunc (the same over ops.py):
    output, LSE and every gradient bitwise."""
    S = 330
    idx_np, causal = _mask(kind, B, S, S, 101)
    if hm > 1:
        idx_np = np.concatenate([_mask(kind, B, S, S, 101 + h)[0] for h in range(hm)], axis=1)
    idx = None if idx_np is None else torch.from_numpy(np.ascontiguousarray(idx_np).copy()).cuda()
    q, k, v, do, s = make_inputs(B, S, S, Hq, Hkv, d, dv, 101, dtype=dtype, sink=True)
    q, k, v, do = q.cuda(), k.cuda(), v.cuda(), do.cuda()
    if layout == "transposed":
        q, k, v, do = (t.transpose(1, 2).contiguous().transpose(1, 2) for t in (q, k, v, do))
    elif layout == "shared kv":
        v = k[..., :dv]
    s = None if sink is None else s.cuda().to(sink).reshape(1, Hq, 1, 1)
    res = []
    for call in (lambda *a: fm.flashmask_attention(*a[:4], causal=causal, sink=a[4], softmax_scale=0.11, return_lse=True,
                                                   deterministic=True),
                 lambda *a: fm.FlashMaskFunc.apply(*a[:4], 0.11, causal, a[4], True)):
        leaves = [t.detach().requires_grad_(True) for t in (q, k, v)]
        sk = None if s is None else s.detach().requires_grad_(True)
        out, lse = call(*leaves, idx, sk)
        assert out.requires_grad and not lse.requires_grad
        res.append([out.detach(), lse, *torch.autograd.grad(out, leaves + ([] if sk is None else [sk]), do)])
    assert len(res[0]) == (5 if sink is None else 6)
    for a, b in zip(*res):
        assert a.dtype == b.dtype and a.shape == b.shape and torch.equal(a, b)
    assert _kernel_status() == 0


@pytest.mark.parametrize("kind,d,dv,B,S,Hq,Hkv,hm,tables", [
    ("causal_doc", 64, 64, 2, 330, 4, 2, 1, 0),           # every CTA of every launch starts at once
    ("causal_doc", 128, 128, 3, 1025, 8, 8, 1, 1),        # the backward's two tables
    ("four_column", 96, 80, 2, 1100, 16, 2, 2, 1),        # all three, the launch of dK / dV is the short one
    ("bidir_doc", 192, 128, 2, 1300, 16, 4, 1, 1)])       # the forward's
def test_launch_tables_of_the_native_host(kind, d, dv, B, S, Hq, Hkv, hm, tables, monkeypatch):
    """The tables that the native host builds on its own (FLASHMASK_B200_ORDER unset), either side of its rule: bitwise
    the Python host, which always builds them."""
    monkeypatch.delenv("FLASHMASK_B200_ORDER", raising=False)
    idx_np, causal = _mask(kind, B, S, S, 102)
    if hm > 1:
        idx_np = np.concatenate([_mask(kind, B, S, S, 102 + h)[0] for h in range(hm)], axis=1)
    idx = torch.from_numpy(np.ascontiguousarray(idx_np).copy()).cuda()
    q, k, v, do, s = make_inputs(B, S, S, Hq, Hkv, d, dv, 102, sink=True)
    dev = [t.cuda() for t in (q, k, v, do)]
    lib = _lib.load()
    with torch.no_grad():
        before = lib.fm_launch_count()
        fm.flashmask_attention(*dev[:3], idx, causal=causal)
        assert lib.fm_launch_count() - before == 2 + tables      # scan of the mask, tables, forward
    got = run_product(*dev, idx, causal, s, deterministic=True)
    x = [t.detach().requires_grad_(True) for t in dev[:3]]
    sk = s.cuda().requires_grad_(True)
    out, lse = fm.FlashMaskFunc.apply(*x, idx, 1 / math.sqrt(d), causal, sk, True)
    for t, n in zip((out, lse, *torch.autograd.grad(out, [*x, sk], dev[3])), ("out", "lse", "dq", "dk", "dv", "dsink")):
        assert torch.equal(t.detach(), got[n]), n
    assert _kernel_status() == 0


def test_window_size_kwarg():
    q, k, v, do, _ = make_inputs(1, 256, 256, 2, 2, 64, 64, 1)
    out = fm.flashmask_attention(q.cuda(), k.cuda(), v.cuda(), causal=True, window_size=32)
    idx, causal = W.sliding_window(1, 256, 256, 32)
    ref = fm.flashmask_attention(q.cuda(), k.cuda(), v.cuda(), torch.from_numpy(idx).cuda(), causal=True)
    assert torch.equal(out, ref)


def test_errors():
    q, k, v, do, _ = make_inputs(1, 64, 64, 2, 2, 64, 64, 1)
    with pytest.raises(RuntimeError):
        fm.flashmask_attention(q, k, v)  # CPU tensors: no fallback
    with pytest.raises(AssertionError):
        fm.flashmask_attention(q.cuda(), k.cuda(), v.cuda(),
                               torch.zeros(1, 1, 64, 4, dtype=torch.int32).cuda(), causal=True)
    with pytest.raises(NotImplementedError):
        fm.flashmask_attention(q.cuda()[..., :40].contiguous().repeat(1, 1, 1, 8),
                               k.cuda()[..., :40].contiguous().repeat(1, 1, 1, 8),
                               v.cuda()[..., :40].contiguous().repeat(1, 1, 1, 8))


def test_operands_elsewhere_are_refused_before_any_launch():
    """A key, value or mask that is not on the query's device never reaches a kernel as a raw pointer."""
    q, k, v, do, _ = make_inputs(1, 64, 64, 2, 2, 64, 64, 1)
    c = [t.cuda() for t in (q, k, v)]
    idx = torch.full((1, 1, 64, 1), 64, dtype=torch.int32)
    before = _lib.load().fm_launch_count()
    for args in ((c[0], k, c[2], None), (c[0], c[1], v, None), (*c, idx)):
        with pytest.raises(AssertionError, match="device"):
            fm.flashmask_attention(*args, causal=True)
        with pytest.raises(AssertionError, match="device"):
            fm._flash_attn_fwd(*args, causal=True)
    assert _lib.load().fm_launch_count() == before


def test_bounded_wait_reports_timeout_without_fault():
    """A wait on a barrier nothing arrives on gives up after its budget, the kernel
    returns, the status word says FM_ERR_TIMEOUT and the context keeps working."""
    from flashmask_b200 import _lib
    assert _kernel_status() == 0
    _lib.check(_lib.load().fm_selftest_bounded_wait(2000, torch.cuda.current_stream().cuda_stream),
               "fm_selftest_bounded_wait")
    torch.cuda.synchronize()
    assert _kernel_status() == 5          # FM_ERR_TIMEOUT, and the read cleared it
    assert _kernel_status() == 0
    x = torch.ones(8, device="cuda")
    assert float(x.sum()) == 8.0          # the context is still usable
    _run("causal_doc", 1, 256, 256, 2, 2, 128, 128, seed=2)


def test_one_kernel_backward_runs_longer_than_a_wait_is_given():
    """A launch of more than the two seconds that a wait has (131072 queries, 262144 keys, 96 / 8 heads, nothing masked): no wait
    is given up, and dK and dV of a kv head are those of a call of its own, an eighth as long."""
    Sq, Sk, Hq, Hkv, d = 131072, 262144, 96, 8, 64
    g = torch.Generator(device="cuda").manual_seed(5)
    q, out, do = (torch.randn(1, Sq, Hq, d, generator=g, device="cuda", dtype=torch.bfloat16) for _ in range(3))
    k, v = (torch.randn(1, Sk, Hkv, d, generator=g, device="cuda", dtype=torch.bfloat16) for _ in range(2))
    lse = torch.full((1, Hq, Sq), 13.0, device="cuda")               # log(262144) = 12.5, + 0.5 for the scores' variance
    idx = torch.zeros(1, 1, Sk, 2, dtype=torch.int32, device="cuda")
    idx[..., 0] = Sq
    start, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    info = fm.prepare_mask(idx, Sq, False, 128, 128)
    start.record()
    _, dk, dv, _ = fm._flash_attn_bwd(q, k, v, out, do, lse, idx, mask_info=info)
    end.record()
    torch.cuda.synchronize()
    assert _kernel_status() == 0
    assert start.elapsed_time(end) > 2000, "larger sizes are needed to outlast a wait's budget"
    for h in (0, Hkv - 1):
        r = slice(h * 12, h * 12 + 12)
        _, dk1, dv1, _ = fm._flash_attn_bwd(q[:, :, r].contiguous(), k[:, :, h:h + 1].contiguous(), v[:, :, h:h + 1].contiguous(),
                                            out[:, :, r].contiguous(), do[:, :, r].contiguous(), lse[:, r].contiguous(), idx)
        assert torch.equal(dk[:, :, h:h + 1], dk1) and torch.equal(dv[:, :, h:h + 1], dv1)
    assert torch.isfinite(dk).all() and torch.isfinite(dv).all() and _kernel_status() == 0


def test_shared_kv_convention():
    """value = key[..., :dv] on the same storage (576/512): dv comes back zero and dk
    carries dK + dV (reference: flashmask/cute/ops/_common.py:52-88)."""
    B, S, Hq, Hkv, d, dv = 1, 256, 2, 1, 576, 512
    g = torch.Generator().manual_seed(3)
    q = torch.randn(B, S, Hq, d, generator=g).bfloat16().cuda()
    kv = torch.randn(B, S, Hkv, d, generator=g).bfloat16().cuda()
    do = torch.randn(B, S, Hq, dv, generator=g).bfloat16().cuda()
    k, v = kv, kv[..., :dv]
    out, lse = fm._flash_attn_fwd(q, k, v, None, causal=True)
    dq, dk, dvv, _ = fm._flash_attn_bwd(q, k, v, out, do, lse, None, causal=True)
    assert float(dvv.abs().max()) == 0.0
    v2 = v.contiguous()                    # separate storage: plain gradients
    dq2, dk2, dv2, _ = fm._flash_attn_bwd(q, k, v2, out, do, lse, None, causal=True)
    want = dk2.float()
    want[..., :dv] += dv2.float()
    assert torch.equal(dq, dq2)
    assert (dk.float() - want).abs().max().item() <= 2 ** -6 * max(1.0, want.abs().max().item())


@pytest.mark.parametrize("deterministic", [True, False])
def test_four_column_mask_long_lists_both_backward_variants(deterministic):
    """A 4-column mask whose units carry far more than 64 work items (S = 8192: up to 128 half
    tiles per unit and q head), through the two-kernel and the one-kernel backward: the case on
    which an MMA issue order that let the second score GEMM of item k+2 overwrite the P^T / dS^T
    of item k once gave wrong gradients."""
    B, S, Hq, Hkv, d = 1, 8192, 2, 1, 128
    rng = np.random.default_rng(77)
    idx_np, causal = W.four_column_bands(B, S, S, rng)
    q, k, v, do, _ = make_inputs(B, S, S, Hq, Hkv, d, d, 77)
    idx = torch.from_numpy(np.ascontiguousarray(idx_np).copy()).cuda()
    got = run_product(q.cuda(), k.cuda(), v.cuda(), do.cuda(), idx, causal, None, deterministic=deterministic)
    import oracle
    from _util import assert_close_rule, lowp_rows
    bd = idx_np[0, 0]
    dk_ref = torch.zeros(S, d); dv_ref = torch.zeros(S, d); dk_lp = torch.zeros(S, d); dv_lp = torch.zeros(S, d)
    for h in range(Hq):
        ref = oracle.attention_rows(q[0, :, h], k[0, :, 0], v[0, :, 0], do[0, :, h], bd, causal)
        lp = lowp_rows(q[0, :, h].cuda(), k[0, :, 0].cuda(), v[0, :, 0].cuda(), do[0, :, h].cuda(), bd, causal, None)
        assert_close_rule(got["dq"][0, :, h], ref["dq"], lp["dq"], f"dq h{h}")
        assert_close_rule(got["out"][0, :, h], ref["out"], lp["out"], f"out h{h}")
        dk_ref += ref["dk"]; dv_ref += ref["dv"]
        dk_lp += lp["dk"].float().cpu(); dv_lp += lp["dv"].float().cpu()
    assert_close_rule(got["dk"][0, :, 0], dk_ref, dk_lp, "dk")
    assert_close_rule(got["dv"][0, :, 0], dv_ref, dv_lp, "dv")
    assert _kernel_status() == 0


def test_aliased_value_keeps_its_own_gradient_below_the_shared_head_dims():
    """The merge of dV into dK is the reference's convention for (512, 512) and (576, 512) only
    (flashmask/cute/ops/bwd.py:136-139); at d = 128 a value that aliases the key still gets its dV."""
    B, S, H, d = 1, 256, 2, 128
    g = torch.Generator().manual_seed(4)
    q = torch.randn(B, S, H, d, generator=g).bfloat16().cuda()
    kv = torch.randn(B, S, H, d, generator=g).bfloat16().cuda()
    do = torch.randn(B, S, H, d, generator=g).bfloat16().cuda()
    out, lse = fm._flash_attn_fwd(q, kv, kv, None, causal=True)
    dq, dk, dv, _ = fm._flash_attn_bwd(q, kv, kv, out, do, lse, None, causal=True)
    dq2, dk2, dv2, _ = fm._flash_attn_bwd(q, kv, kv.clone(), out, do, lse, None, causal=True)
    assert float(dv.abs().max()) > 0.0
    assert torch.equal(dk, dk2) and torch.equal(dv, dv2) and torch.equal(dq, dq2)


@pytest.mark.parametrize("d", [64, 128])
def test_forward_and_backward_replay_from_a_cuda_graph(d):
    """fm_fwd / fm_bwd synchronise nothing and allocate nothing: with the mask prepared and the launch
    tables built beforehand, forward + backward capture into one CUDA graph, and a replay on new input
    values gives the bits of an eager run (the persistent kernels rewind their own table counters)."""
    B, S, Hq, Hkv = 2, 1024, 4, 2
    idx_np, causal = _mask("causal_doc", B, S, S, 41)
    idx = torch.from_numpy(np.ascontiguousarray(idx_np).copy()).cuda()
    a = [t.cuda() for t in make_inputs(B, S, S, Hq, Hkv, d, d, 42)[:4]]
    b = [t.cuda() for t in make_inputs(B, S, S, Hq, Hkv, d, d, 43)[:4]]
    info = fm.prepare_mask(idx, S, causal, *fm.fwd_tile_shape(d, d))

    def step(q, k, v, do):
        out, lse = fm._flash_attn_fwd(q, k, v, idx, causal=causal, mask_info=info)
        dq, dk, dv, _ = fm._flash_attn_bwd(q, k, v, out, do, lse, idx, causal=causal, mask_info=info)
        return out, lse, dq, dk, dv

    want = [t.clone() for t in step(*b)]            # eager; also builds the launch tables
    static = [t.clone() for t in a]
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        step(*static)
    torch.cuda.current_stream().wait_stream(side)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = step(*static)
    for s_, n_ in zip(static, b):
        s_.copy_(n_)
    graph.replay()
    graph.replay()                                   # a second replay: the table counters were rewound
    torch.cuda.synchronize()
    for g_, w_ in zip(got, want):
        assert torch.equal(g_, w_)
    assert _kernel_status() == 0


@pytest.mark.parametrize("Sq,Sk,kind", [(700, 700, "causal_doc"), (512, 512, "none_causal"), (4, 3000, "none_causal")])
def test_overlapping_kernels_of_a_call_replay_from_a_cuda_graph(Sq, Sk, kind):
    """The programmatic launches inside a call (split forward + merge; dK / dV + dQ kernel of the deterministic
    backward) under capture: replays on new inputs are bitwise eager calls."""
    from flashmask_b200.ops import _flash_attn_bwd, _flash_attn_fwd
    causal, idx = True, None
    if kind == "causal_doc":
        idx = torch.full((1, 1, Sk, 1), Sk, dtype=torch.int32, device="cuda")
        idx[:, :, :300] = 300
    g = torch.Generator(device="cuda").manual_seed(5)
    new = lambda *shape: torch.randn(*shape, generator=g, device="cuda", dtype=torch.bfloat16)
    ins = [new(1, Sq, 4, 128), new(1, Sk, 2, 128), new(1, Sk, 2, 128), new(1, Sq, 4, 128)]

    def call(q, k, v, do):
        out, lse = _flash_attn_fwd(q, k, v, idx, causal=causal)
        return [out, lse, *_flash_attn_bwd(q, k, v, out, do, lse, idx, causal=causal, deterministic=True)[:3]]

    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        call(*ins)
    torch.cuda.current_stream().wait_stream(side)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = call(*ins)
    for _ in range(3):
        for t in ins:
            t.copy_(new(*t.shape))
        graph.replay()
        for a, b in zip(got, call(*ins)):
            assert torch.equal(a, b)
    assert _kernel_status() == 0
