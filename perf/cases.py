"""The work users of the attention operators have them do, as cases that can be timed and compared.

A case is a dict of plain values.  `path` says which public entry points a pass goes through:

  fwd      torch.ops.mha_manual.fmha_fwd on [B,H,S,D] tensors (inference, or the forward half of a training step)
  fwd_bwd  fmha_fwd, then fmha_bwd (a training step that calls the two operators itself)
  autograd torch.ops.mha_manual.fmha under autograd, and its gradients
  qkv      torch.ops.mha_manual.fmha_qkvpacked under autograd: one [B,S,3,H,D] projection in, one gradient out
  varlen   torch.ops.mha_manual.fmha_varlen_qkvpacked under autograd: the same, padding removed
  keep, train, train_save
           the dense-mask operators fmha_nvfuser, fmha_train_nvfuser and fmha_train_saveim_nvfuser on [B*H,S,D]

`mask` is how a batch says where its padding is: "none", "lens" (int32 valid lengths) or "key" (a float [B,S_k] row
that is added to the scores).  Valid lengths are spread evenly over [min_len, S_k], in an order drawn from the seed,
so that the amount of work of a case does not depend on the seed.
"""
import math
import random

import torch

import mha_manual  # noqa: F401  registers torch.ops.mha_manual.*

DTYPES = {"fp16": torch.float16, "bf16": torch.bfloat16}
TRAINING = ("fwd_bwd", "autograd", "qkv", "varlen")
DENSE = ("keep", "train", "train_save")


def _case(path, B, H, S_q, S_k, D, dtype, mask, min_len, p_drop):
    return {"path": path, "B": B, "H": H, "S_q": S_q, "S_k": S_k, "D": D, "dtype": dtype, "mask": mask,
            "min_len": min_len, "p_drop": p_drop}


def listed():
    cases = [
        # one request of an encoder being served: 12 heads, 128 tokens, nothing to pad; all launch and latency
        ("one_request", _case("fwd", 1, 12, 128, 128, 64, "fp16", "none", 128, 0.0)),
        # the smallest named configuration (B=2, H=4, S=128, D=64) as a training step: launches and host work
        ("small_train", _case("autograd", 2, 4, 128, 128, 64, "fp16", "lens", 64, 0.1)),
        # the inference operator at the shape of the project this one replaces: 512 heads, dense keep mask
        ("dense_keep", _case("keep", 32, 16, 128, 128, 64, "fp16", "dense", 64, 0.0)),
        # its training operator that also writes the softmax and the dropped-out softmax, same shape
        ("dense_train_save", _case("train_save", 32, 16, 128, 128, 64, "fp16", "dense", 64, 0.5)),
        # BERT-base forward in training mode: the named configuration
        ("bert_base_fwd", _case("fwd", 32, 12, 512, 512, 64, "fp16", "lens", 256, 0.1)),
        # BERT-large batch scoring: the named sizes, no dropout, padding as the additive row most callers hold
        ("bert_large_infer", _case("fwd", 64, 16, 384, 384, 64, "bf16", "key", 128, 0.0)),
        # BERT-large training step: the named configuration and the repository's benchmark
        ("bert_large_train", _case("fwd_bwd", 32, 16, 512, 512, 64, "fp16", "lens", 256, 0.1)),
        # the same batch with its padding removed, on the layout of a fused QKV projection
        ("unpadded_train", _case("varlen", 32, 16, 512, 512, 64, "bf16", "lens", 256, 0.1)),
        # image patches plus a class token: an odd length that is no multiple of a tile, an odd batch, no mask
        ("patches_train", _case("qkv", 13, 12, 197, 197, 64, "bf16", "none", 197, 0.0)),
        # long documents, head dimension 128: batch scoring ("prefill")
        ("long_infer", _case("fwd", 4, 16, 2048, 2048, 128, "bf16", "lens", 1024, 0.0)),
        # the long-sequence training configuration, one GPU's share of it (32 of 256 sequences): the largest
        ("long_train", _case("fwd_bwd", 32, 16, 2048, 2048, 128, "bf16", "lens", 1024, 0.0)),
        # one new query row per sequence against keys and values computed before ("decode", cross-attention)
        ("few_queries", _case("fwd", 2, 16, 1, 4096, 128, "bf16", "lens", 2048, 0.0)),
    ]
    return [dict(c, name=name) for name, c in cases]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    """One more case: a use drawn evenly, its sizes spread over the logarithm of that use's range."""
    use = rng.choice(("serve", "step", "step", "unpadded", "dense", "long", "few_queries"))
    dtype = rng.choice(("fp16", "bf16"))
    H = rng.choice((4, 8, 12, 16))
    mask = rng.choice(("none", "lens", "key"))
    while True:
        if use == "serve":        # encoder inference, from one short request to a large batch
            c = _case("fwd", _log_int(rng, 1, 64), H, 0, _log_int(rng, 16, 1024), rng.choice((64, 64, 128)), dtype, mask, 0, 0.0)
        elif use == "step":       # encoder training steps, from a toy model to BERT-large
            c = _case(rng.choice(("fwd", "fwd_bwd", "autograd", "qkv")), _log_int(rng, 1, 48), H, 0, _log_int(rng, 32, 1024),
                      rng.choice((64, 64, 128)), dtype, mask, 0, rng.choice((0.0, 0.1)))
        elif use == "unpadded":   # the same without padding
            c = _case("varlen", _log_int(rng, 2, 48), H, 0, _log_int(rng, 64, 1024), rng.choice((64, 64, 128)), dtype, "lens", 0,
                      rng.choice((0.0, 0.1)))
        elif use == "dense":      # the dense-mask operators: up to four times the shape they were written for
            S = _log_int(rng, 32, 384)
            S = S if rng.random() < 0.2 else (S + 7) // 8 * 8   # mostly rows of whole 16-byte pieces
            path = rng.choice(DENSE)
            c = _case(path, _log_int(rng, 1, 64), H, 0, S, 64, dtype, "dense", 0, 0.0 if path == "keep" else 0.5)
        elif use == "long":       # long sequences, with and without gradients
            c = _case(rng.choice(("fwd", "fwd_bwd")), _log_int(rng, 1, 16), H, 0, _log_int(rng, 1024, 6144), rng.choice((64, 128, 128)),
                      dtype, rng.choice(("none", "lens")), 0, 0.0)
        else:                     # a few new rows against long keys
            c = _case("fwd", _log_int(rng, 1, 16), H, _log_int(rng, 1, 64), _log_int(rng, 256, 12288), rng.choice((64, 128)), dtype,
                      rng.choice(("none", "lens")), 0, 0.0)
        c["S_q"] = c["S_q"] or c["S_k"]
        c["min_len"] = c["S_k"] if c["mask"] == "none" else max(1, int(c["S_k"] * rng.uniform(0.3, 0.6)))
        if work(c)["flops"] <= 0.5 * work(listed()[10])["flops"] and work(c)["bytes"] <= 0.5 * work(listed()[10])["bytes"]:
            return c


def _lengths(case):
    """Valid lengths of the batch, before they are put in an order."""
    B, lo, hi = case["B"], case["min_len"], case["S_k"]
    return [hi] if B == 1 else [lo + (hi - lo) * i // (B - 1) for i in range(B)]


def prepare(case, seed):
    B, H, S_q, S_k, D = (case[n] for n in ("B", "H", "S_q", "S_k", "D"))
    path, dtype = case["path"], DTYPES[case["dtype"]]
    g = torch.Generator(device="cuda").manual_seed(seed)

    def normal(*shape):   # scores of N(0,1) rows, scaled by 1/sqrt(D), are N(0,1) themselves
        return torch.randn(*shape, device="cuda", dtype=dtype, generator=g)

    lens = _lengths(case)
    random.Random(seed).shuffle(lens)
    s = {"case": dict(case), "philox": (0x5EED0000 + seed, seed % 1000)}
    lens_dev = torch.tensor(lens, dtype=torch.int32, device="cuda")
    if path in DENSE:
        s["q"], s["k"], s["v"] = normal(B * H, S_q, D), normal(B * H, S_k, D), normal(B * H, S_k, D)
        keep = (torch.arange(S_k, device="cuda")[None, :] < lens_dev[:, None]).to(dtype)           # [B,S_k], 1 = key exists
        keep = keep if path == "keep" else (1 - keep) * -10000.0
        s["mask"] = keep[:, None, None, :].expand(B, H, S_q, S_k).reshape(B * H, S_q, S_k).contiguous()
        if path != "keep":
            s["drop"] = (torch.rand(B * H, S_q, S_k, device="cuda", generator=g) >= case["p_drop"]).to(dtype)
        return s
    s["lens"] = s["mask"] = None
    if case["mask"] == "lens":
        s["lens"] = lens_dev
    elif case["mask"] == "key":
        pad = torch.arange(S_k, device="cuda")[None, :] >= lens_dev[:, None]
        s["mask"] = pad.to(torch.float32) * -10000.0
    if path == "varlen":
        cu = [0]
        for n in lens:
            cu.append(cu[-1] + n)
        s["cu"] = torch.tensor(cu, dtype=torch.int32, device="cuda")
        s["qkv"], s["d_o"] = normal(cu[-1], 3, H, D).requires_grad_(), normal(cu[-1], H, D)
    elif path == "qkv":
        s["qkv"], s["d_o"] = normal(B, S_k, 3, H, D).requires_grad_(), normal(B, S_k, H, D)
    else:
        s["q"], s["k"], s["v"] = normal(B, H, S_q, D), normal(B, H, S_k, D), normal(B, H, S_k, D)
        if path in TRAINING:
            s["d_o"] = normal(B, H, S_q, D)
        if path == "autograd":
            for n in "qkv":
                s[n].requires_grad_()
    return s


def run(s):
    ops, c = torch.ops.mha_manual, s["case"]
    path, p = c["path"], c["p_drop"]
    if path == "keep":
        return ops.fmha_nvfuser(s["q"], s["k"], s["v"], s["mask"])
    if path == "train":
        return ops.fmha_train_nvfuser(s["q"], s["k"], s["v"], s["mask"], s["drop"])
    if path == "train_save":
        return ops.fmha_train_saveim_nvfuser(s["q"], s["k"], s["v"], s["mask"], s["drop"])
    seed, offset = s["philox"]
    if path == "varlen":
        o = ops.fmha_varlen_qkvpacked(s["qkv"], s["cu"], c["S_k"], p, seed, offset)
        return (o, *torch.autograd.grad(o, s["qkv"], s["d_o"]))
    if path == "qkv":
        o = ops.fmha_qkvpacked(s["qkv"], s["mask"], s["lens"], p, seed, offset)
        return (o, *torch.autograd.grad(o, s["qkv"], s["d_o"]))
    q, k, v = s["q"], s["k"], s["v"]
    if path == "autograd":
        o = ops.fmha(q, k, v, s["mask"], s["lens"], p, seed, offset)
        return (o, *torch.autograd.grad(o, (q, k, v), s["d_o"]))
    o, lse = ops.fmha_fwd(q, k, v, s["mask"], s["lens"], p, seed, offset)
    if path == "fwd":
        return o, lse
    return (o, lse, *ops.fmha_bwd(s["d_o"], q, k, v, o, lse, s["mask"], s["lens"], p, seed, offset))


def work(case):
    """Each input read once, each output written once; keys and values past a valid length need not be read, and
    scores of such keys need not be formed.  4*D flops per score forward, 10*D backward."""
    B, H, S_q, S_k, D, path = (case[n] for n in ("B", "H", "S_q", "S_k", "D", "path"))
    lens = _lengths(case)
    if path == "varlen":
        q_rows = k_rows = H * sum(lens)
        scores = H * sum(n * n for n in lens)
    else:
        q_rows, k_rows, scores = B * H * S_q, H * sum(lens), H * S_q * sum(lens)
    elems = 2 * q_rows * D + 2 * k_rows * D                     # q, o and k, v
    flops = 4 * D * scores
    if path in TRAINING:
        k_out = k_rows if path == "varlen" else B * H * S_k     # dk, dv of padded keys are zeros, but are written
        elems += 2 * q_rows * D + 2 * k_out * D                 # d_o, dq and dk, dv
        flops += 10 * D * scores
    if path in DENSE:                                           # masks read, saved tensors written, whole
        elems += B * H * S_q * S_k * {"keep": 1, "train": 2, "train_save": 4}[path]
    lse = 4 * q_rows if path in ("fwd", "fwd_bwd") else 0
    return {"bytes": 2 * elems + lse, "flops": flops}


def tolerance(case):
    """Probabilities and results are rounded to 16 bits: two correct implementations differ by a few units in the last
    place of their type (2^-11 for fp16, 2^-8 for bf16), a single value by more where its sum cancels."""
    return {"rel": 2e-3, "max": 0.03} if case["dtype"] == "fp16" else {"rel": 1e-2, "max": 0.15}
