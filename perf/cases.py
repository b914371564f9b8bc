"""The work that users of flashmask_b200 have it do, as cases that can be timed and compared.

A case is a dict of plain values.  ``use`` says which call it is:

* ``train``        ``flashmask_attention`` and the gradients of every input that takes one, as an
                   attention layer of a training step does it;
* ``forward``      ``flashmask_attention`` without gradients: evaluation, a chunk of a prompt against the
                   keys before it, one more token against a cache (``Sq < Sk``, bottom-right causal);
* ``block_score``  ``_flash_attn_fwd`` with the block-score side output (key-block selection).

Document layouts are lognormal, as in the benchmark's workloads.  A case fixes the document LENGTHS through
``layout``; their order in the packed sequence comes from the seed, so every seed is another mask with exactly
the same number of visible pairs.
"""
import math

import numpy as np
import torch

from flashmask_b200 import flashmask_attention
from flashmask_b200 import workloads as W
from flashmask_b200.ops import _flash_attn_fwd

DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16}


def _case(use, B, Sq, Sk, Hq, Hkv, d, dv, mask, dtype="bf16", sink=False, deterministic=False, layout=1, block=0,
          name=None):
    c = {"use": use, "B": B, "Sq": Sq, "Sk": Sk, "Hq": Hq, "Hkv": Hkv, "d": d, "dv": dv, "mask": mask,
         "dtype": dtype, "sink": sink, "deterministic": deterministic, "layout": layout, "block": block}
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the smallest training call of the configurations: launches and host work count, not the kernels
        _case("train", 1, 1024, 1024, 2, 2, 64, 64, "causal_doc", name="train_1k_d64"),
        # packed fine-tuning at 8K tokens with grouped heads: the benchmark's headline
        _case("train", 2, 8192, 8192, 32, 8, 128, 128, "causal_doc", name="train_8k_gqa"),
        # the same mask for models with 64-wide heads, in the other 16-bit type
        _case("train", 2, 8192, 8192, 32, 8, 64, 64, "causal_doc", dtype="fp16", name="train_8k_gqa_d64_fp16"),
        # prefix-LM batches are rarely a round length, and 96-wide heads fill no tile exactly
        _case("train", 2, 3001, 3001, 16, 4, 96, 96, "prefix_lm", layout=2, name="train_3001_d96_prefix_lm"),
        # preference tuning: one shared question, several answers, at 32K
        _case("train", 1, 32768, 32768, 16, 16, 128, 128, "share_question", name="train_32k_share_question"),
        # large head dims, reproducible gradients and a sink logit per head
        _case("train", 1, 16384, 16384, 32, 8, 192, 128, "causal", sink=True, deterministic=True,
              name="train_16k_192_128"),
        _case("train", 1, 16384, 16384, 16, 16, 256, 256, "causal", sink=True, deterministic=True,
              name="train_16k_256_256"),
        # one latent key/value head shared by all query heads
        _case("train", 1, 16384, 16384, 16, 1, 576, 512, "causal", sink=True, deterministic=True,
              name="train_16k_576_512_mqa"),
        # the longest context: packed documents of up to 32K in 128K tokens, the bidirectional form of the bounds
        _case("train", 1, 131072, 131072, 32, 8, 128, 128, "long_doc", layout=4, name="train_128k_doc"),
        # a chunk of a long prompt against everything before it
        _case("forward", 1, 512, 16384, 32, 8, 128, 128, "causal", name="prefill_512_of_16k"),
        # one more token for each of eight sequences
        _case("forward", 8, 1, 8192, 32, 8, 128, 128, "causal", name="decode_8x8k"),
        # the forward that also scores blocks of 64 keys for a sparse layer behind it
        _case("block_score", 2, 8192, 8192, 32, 8, 128, 128, "causal_doc", layout=3, block=64,
              name="block_score_8k_gqa"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the ranges above."""
    use = rng.choice(["train", "train", "train", "big", "big", "forward", "forward", "block_score"])
    dtype = rng.choice(["bf16", "bf16", "fp16"])
    layout = rng.randrange(1, 1 << 20)
    if use == "train":
        S = _log_int(rng, 512, 32768)
        if rng.random() < 0.5:
            S = max(512, S // 128 * 128)
        hkv = rng.choice([2, 4, 8, 16])
        hq = min(32, hkv * rng.choice([1, 2, 4]))
        d = rng.choice([64, 64, 80, 96, 128, 128, 128, 128])
        mask = rng.choice(["causal_doc", "causal_doc", "bidir_doc", "sliding_window", "share_question", "prefix_lm",
                           "random_eviction", "causal", "full"])
        return _case("train", rng.randint(1, max(1, min(4, 32768 // S))), S, S, hq, hkv, d, d, mask, dtype,
                     deterministic=rng.random() < 0.2, layout=layout)
    if use == "big":
        S = _log_int(rng, 1024, 16384)
        if rng.random() < 0.5:
            S = S // 128 * 128
        hq, hkv, d, dv = rng.choice([(32, 8, 192, 128), (16, 16, 192, 128), (16, 16, 256, 256), (16, 4, 256, 256),
                                     (16, 1, 576, 512), (8, 1, 576, 512)])
        mask = rng.choice(["causal", "causal_doc", "bidir_doc"])
        return _case("train", 1, S, S, hq, hkv, d, dv, mask, dtype, sink=rng.random() < 0.7,
                     deterministic=rng.random() < 0.7, layout=layout)
    if use == "forward":
        Sk = _log_int(rng, 2048, 32768)
        Sq = 1 if rng.random() < 0.35 else _log_int(rng, 2, 2048)
        B = rng.randint(1, max(1, min(16, 65536 // Sk, 8192 // Sq)))
        hkv = rng.choice([4, 8])
        hq = hkv * rng.choice([1, 4, 8])
        d = rng.choice([64, 128, 128])
        return _case("forward", B, Sq, Sk, hq, hkv, d, d, "causal", dtype, layout=layout)
    S = _log_int(rng, 2048, 16384)
    hkv = rng.choice([4, 8])
    hq = hkv * rng.choice([1, 4])
    return _case("block_score", rng.randint(1, max(1, 16384 // S)), S, S, hq, hkv, 128, 128,
                 rng.choice(["causal_doc", "causal"]), dtype, layout=layout, block=rng.choice([64, 128]))


def _doc_lengths(case, b):
    """Document lengths of batch entry b: a function of the case alone."""
    rng = np.random.default_rng([case["layout"], b])
    S = case["Sk"]
    if case["mask"] == "long_doc":
        return W.lognormal_doc_lengths(rng, S, math.log(4096), 1.5, 512, 32768)
    return W.lognormal_doc_lengths(rng, S, math.log(1024), 1.0, 64, 8192)


def _mask(case, seed):
    """(startend_row_indices as numpy or None, causal)."""
    kind, B, Sq, Sk = case["mask"], case["B"], case["Sq"], case["Sk"]
    if kind == "causal":
        return None, True
    if kind == "full":
        return None, False
    if kind == "sliding_window":
        return W.sliding_window(B, Sq, Sk, 1024)
    if kind == "share_question":
        return W.share_question(B, Sq, Sk, 4096, 2048, 4)
    if kind == "random_eviction":
        return W.random_eviction(B, Sq, Sk, np.random.default_rng([case["layout"], seed]))
    parts, causal = [], None
    for b in range(B):
        lens = np.random.default_rng([seed, b]).permutation(_doc_lengths(case, b))
        if kind == "causal_doc":
            idx, causal = W.causal_document(1, Sq, Sk, lens)
        elif kind == "bidir_doc":
            idx, causal = W.bidirectional_document(1, Sq, Sk, lens)
        elif kind == "prefix_lm":
            idx, causal = W.prefix_lm_document(1, Sq, Sk, [(int(n) // 3, int(n)) for n in lens])
        elif kind == "long_doc":
            idx, causal = W.causal_document_noncausal_form(1, Sq, Sk, lens)
        else:
            raise KeyError(kind)
        parts.append(idx)
    return np.ascontiguousarray(np.concatenate(parts, axis=0)), causal


def prepare(case, seed):
    dev = torch.device("cuda")
    g = torch.Generator(device=dev).manual_seed(seed)
    dt = DTYPES[case["dtype"]]
    B, Sq, Sk, Hq, Hkv, d, dv = (case[k] for k in ("B", "Sq", "Sk", "Hq", "Hkv", "d", "dv"))

    def normal(*shape):
        return torch.randn(*shape, generator=g, device=dev, dtype=dt)

    idx, causal = _mask(case, seed)
    s = {"use": case["use"], "causal": causal, "deterministic": case["deterministic"], "block": case["block"],
         "q": normal(B, Sq, Hq, d), "k": normal(B, Sk, Hkv, d), "v": normal(B, Sk, Hkv, dv),
         "idx": None if idx is None else torch.from_numpy(idx).to(dev), "sink": None}
    if case["sink"]:
        s["sink"] = torch.randn(Hq, generator=g, device=dev, dtype=torch.float32)
    if case["use"] == "train":
        s["do"] = normal(B, Sq, Hq, dv)
        s["wrt"] = [t.requires_grad_(True) for t in (s["q"], s["k"], s["v"], s["sink"]) if t is not None]
    elif case["use"] == "block_score":
        s["scores"] = torch.empty(B, Hq, Sq, -(-Sk // case["block"]), device=dev, dtype=torch.float32)
    return s


def run(s):
    if s["use"] == "train":
        out = flashmask_attention(s["q"], s["k"], s["v"], s["idx"], causal=s["causal"], learnable_sink=s["sink"],
                                  deterministic=s["deterministic"])
        return [out.detach(), *torch.autograd.grad(out, s["wrt"], s["do"])]
    with torch.no_grad():
        if s["use"] == "forward":
            return flashmask_attention(s["q"], s["k"], s["v"], s["idx"], causal=s["causal"], return_lse=True)
        s["scores"].fill_(-math.inf)     # blocks of tiles that are never visited stay as the caller left them
        out, lse = _flash_attn_fwd(s["q"], s["k"], s["v"], s["idx"], causal=s["causal"], block_logit=s["scores"],
                                   block_size=s["block"])
        return out, lse, s["scores"]


def work(case):
    B, Sq, Sk, Hq, Hkv, d, dv = (case[k] for k in ("B", "Sq", "Sk", "Hq", "Hkv", "d", "dv"))
    idx, causal = _mask(case, 1)
    pairs = int(W.count_visible(idx, B, Sq, Sk, causal).sum()) * Hq
    q, k, v, o, lse = B * Sq * Hq * d * 2, B * Sk * Hkv * d * 2, B * Sk * Hkv * dv * 2, B * Sq * Hq * dv * 2, B * Sq * Hq * 4
    bounds = 0 if idx is None else idx.nbytes
    nbytes, flops = q + k + v + bounds + o, 2 * pairs * (d + dv)
    if case["use"] == "train":
        nbytes += o + q + k + v                    # dO in; dQ, dK, dV out
        flops += 2 * pairs * (3 * d + 2 * dv)
    else:
        nbytes += lse
        if case["use"] == "block_score":
            nbytes += B * Hq * Sq * -(-Sk // case["block"]) * 4
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    # P and dS are rounded to the 16-bit type before the second GEMMs, the results once more: a few units of
    # 2^-9 (bf16) or 2^-12 (fp16) in the 2-norm
    return {"rel": 1e-2} if case["dtype"] == "bf16" else {"rel": 2e-3}
