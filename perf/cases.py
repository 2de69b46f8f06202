"""Performance cases of the attention operators: what is timed, over which ranges, and what a pass costs at the least.

Five ways in which programs call the package, all through its public entry points:

  fwd           gqa_forward: inference / prefill, or the forward of a hand-written training loop
  bwd           gqa_backward on saved O and LSE with a workspace the program keeps, as the headline benchmark calls it
  train         gqa_attention under autograd, forward and backward: one attention layer of a training step
  train_varlen  gqa_attention_varlen under autograd: a packed batch of sequences of different lengths
  bwd_varlen    gqa_backward_varlen with a kept workspace

Sequence lengths run from 64 to 32 768 tokens, batches from 1 to 16, the head counts are the ones of the benchmark
configurations and tests, head dimensions 64 and 128 (native) and other multiples of 8; causal or not, both tensor
layouts, bit-reproducible dQ and the head split where they are used.  Inputs are N(0, 1) in bf16, like activations
behind a normalisation and as in the benchmark's own workloads.
"""
import math
import random

import torch

from hopper_jeni_b200 import ops
from hopper_jeni_b200.autograd import gqa_attention, gqa_attention_varlen

HEADS = [(4, 2), (6, 2), (8, 1), (8, 8), (12, 4), (16, 2), (16, 4), (24, 8), (32, 8), (64, 8)]


def _case(op, B, Hq, Hkv, S, D, causal, layout="bhsd", deterministic=False, split_heads=False, name=None):
    c = {"op": op, "B": B, "Hq": Hq, "Hkv": Hkv, "S": S, "D": D, "causal": causal, "layout": layout,
         "deterministic": deterministic, "split_heads": split_heads}
    return dict(c, name=name) if name else c


def _packed(op, n_seqs, min_len, max_len, lens_seed, Hq, Hkv, D, causal, name=None):
    c = {"op": op, "n_seqs": n_seqs, "min_len": min_len, "max_len": max_len, "lens_seed": lens_seed, "Hq": Hq,
         "Hkv": Hkv, "D": D, "causal": causal}
    return dict(c, name=name) if name else c


def listed():
    return [
        # a short prompt through one small layer: nothing but latency
        _case("fwd", 1, 4, 2, 128, 64, True, name="fwd_short_prompt"),
        # one layer's training step on a short sequence (the smoke test's size): host path and launches
        _case("train", 1, 6, 2, 256, 64, True, name="train_short"),
        # prefill of two prompts padded to a length that is no multiple of any tile
        _case("fwd", 2, 12, 4, 1000, 128, True, name="fwd_ragged_prefill"),
        # training step of a mid-size layer at an odd length, sequence-major tensors as projections produce them
        _case("train", 2, 32, 8, 1537, 128, True, layout="bshd", name="train_ragged_bshd"),
        # fine-tuning with a head dimension that is not native (runs on the next kernel size up)
        _case("train", 2, 16, 4, 1024, 80, True, name="train_head_dim_80"),
        # bidirectional encoder inference, a point of the forward sweep
        _case("fwd", 16, 16, 2, 2048, 64, False, name="fwd_encoder_d64"),
        # long-document prefill, the sweep's largest causal point
        _case("fwd", 16, 16, 2, 16384, 128, True, name="fwd_long_prefill"),
        # the headline benchmark: backward alone, non-causal
        _case("bwd", 8, 12, 4, 4096, 64, False, name="bwd_headline"),
        # reproducible training: bit-identical dQ at a size of the reference's sweep
        _case("bwd", 2, 24, 8, 4096, 128, True, deterministic=True, name="bwd_deterministic"),
        # pretraining step of a large layer
        _case("train", 4, 32, 8, 8192, 128, True, name="train_pretrain_8k"),
        # pretraining on packed documents of very different lengths
        _packed("train_varlen", 28, 128, 8192, 7, 32, 8, 128, True, name="train_packed_documents"),
        # long-context training step, one sequence of 32k tokens
        _case("train", 1, 64, 8, 32768, 128, True, name="train_long_context_32k"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _length(rng, lo=64, hi=32768):
    """A sequence length: half are multiples of 64 (padded batches), half are whatever the text gave."""
    n = _log_int(rng, lo, hi)
    return max(lo, n // 64 * 64) if rng.random() < 0.5 else n


_MOST_FLOPS = 1.2e13  # of a drawn case: a quarter of the largest listed one


def draw(rng):
    op = rng.choice(["fwd"] * 3 + ["train"] * 3 + ["bwd"] * 2 + ["train_varlen", "bwd_varlen"])
    Hq, Hkv = rng.choice(HEADS)
    D = rng.choice([64, 128])
    causal = rng.random() < 0.65
    if op.endswith("varlen"):
        while True:
            max_len = _log_int(rng, 256, 8192)
            c = _packed(op, _log_int(rng, 2, 48), rng.choice([1, 64, 128]), max_len, rng.randrange(1 << 20), Hq, Hkv, D,
                        causal)
            if work(c)["flops"] <= _MOST_FLOPS:
                return c
    layout = "bshd" if rng.random() < 0.3 else "bhsd"
    if layout == "bhsd" and rng.random() < 0.15:
        D = rng.choice([32, 40, 72, 80, 96, 112])
    deterministic = op != "fwd" and rng.random() < 0.15
    split_heads = op == "bwd" and not deterministic and layout == "bhsd" and rng.random() < 0.2
    while True:
        c = _case(op, _log_int(rng, 1, 16), Hq, Hkv, _length(rng), D, causal, layout, deterministic, split_heads)
        if work(c)["flops"] <= _MOST_FLOPS:
            return c


def _lens(case):
    """Lengths of a packed batch: spread over their logarithm, the longest one present."""
    r = random.Random(case["lens_seed"])
    lens = [_log_int(r, case["min_len"], case["max_len"]) for _ in range(case["n_seqs"] - 1)] + [case["max_len"]]
    r.shuffle(lens)
    return lens


def prepare(case, seed):
    g = torch.Generator(device="cuda").manual_seed(int(seed))

    def rand(*shape, grad=False):
        return torch.randn(*shape, generator=g, device="cuda", dtype=torch.bfloat16).requires_grad_(grad)

    Hq, Hkv, D, op = case["Hq"], case["Hkv"], case["D"], case["op"]
    grad = op.startswith("train")
    st = {"case": case}
    if op.endswith("varlen"):
        lens = _lens(case)
        T = sum(lens)
        starts = [0]
        for n in lens:
            starts.append(starts[-1] + n)
        st.update(q=rand(T, Hq, D, grad=grad), k=rand(T, Hkv, D, grad=grad), v=rand(T, Hkv, D, grad=grad),
                  do=rand(T, Hq, D), cu=torch.tensor(starts, dtype=torch.int32, device="cuda"), max_len=max(lens))
        if op == "bwd_varlen":
            st["o"], st["lse"] = ops.gqa_forward_varlen(st["q"], st["k"], st["v"], st["cu"], st["max_len"],
                                                        causal=case["causal"])
            st["ws"] = torch.empty(ops.bwd_varlen_workspace_bytes(T, Hq, Hkv, D), dtype=torch.uint8, device="cuda")
        return st
    B, S = case["B"], case["S"]

    def shape(h):
        return (B, S, h, D) if case["layout"] == "bshd" else (B, h, S, D)

    st.update(q=rand(*shape(Hq), grad=grad), k=rand(*shape(Hkv), grad=grad), v=rand(*shape(Hkv), grad=grad))
    if op != "fwd":
        st["do"] = rand(*shape(Hq))
    if op == "bwd":
        st["o"], st["lse"] = ops.gqa_forward(st["q"], st["k"], st["v"], causal=case["causal"], layout=case["layout"])
        st["ws"] = torch.empty(ops.bwd_workspace_bytes(B, Hq, Hkv, S, D, case["causal"], case["split_heads"]),
                               dtype=torch.uint8, device="cuda")
    return st


def run(st):
    c = st["case"]
    op, causal = c["op"], c["causal"]
    if op == "fwd":
        return ops.gqa_forward(st["q"], st["k"], st["v"], causal=causal, layout=c["layout"])
    if op == "bwd":
        return ops.gqa_backward(st["q"], st["k"], st["v"], st["o"], st["do"], st["lse"], causal=causal,
                                workspace=st["ws"], deterministic=c["deterministic"], layout=c["layout"],
                                split_heads=c["split_heads"])
    if op == "bwd_varlen":
        return ops.gqa_backward_varlen(st["q"], st["k"], st["v"], st["o"], st["do"], st["lse"], st["cu"],
                                       st["max_len"], causal=causal, workspace=st["ws"])
    qkv = (st["q"], st["k"], st["v"])
    if op == "train":
        o = gqa_attention(*qkv, causal=causal, layout=c["layout"], deterministic=c["deterministic"])
    else:
        o = gqa_attention_varlen(*qkv, st["cu"], st["max_len"], causal=causal)
    return (o.detach(), *torch.autograd.grad(o, qkv, st["do"]))


def work(case):
    """Bytes: every input read and every output written once (bf16; LSE fp32).  Operations: two products per visible
    (query, key) pair in the forward and five in the backward, which recomputes the scores."""
    Hq, Hkv, D, op = case["Hq"], case["Hkv"], case["D"], case["op"]
    if op.endswith("varlen"):
        lens = _lens(case)
        tokens = sum(lens)
        pairs = sum(n * (n + 1) // 2 if case["causal"] else n * n for n in lens)
    else:
        n = case["S"]
        tokens = case["B"] * n
        pairs = case["B"] * (n * (n + 1) // 2 if case["causal"] else n * n)
    q_bytes, kv_bytes, lse_bytes = tokens * Hq * D * 2, tokens * Hkv * D * 2, tokens * Hq * 4
    fwd_bytes = 2 * q_bytes + 2 * kv_bytes + lse_bytes      # Q, K, V -> O, LSE
    bwd_bytes = 4 * q_bytes + 4 * kv_bytes + lse_bytes      # Q, O, dO, K, V, LSE -> dQ, dK, dV
    fwd_flops, bwd_flops = 4 * pairs * Hq * D, 10 * pairs * Hq * D
    bytes_, flops = 0, 0
    if op.startswith(("fwd", "train")):
        bytes_, flops = bytes_ + fwd_bytes, flops + fwd_flops
    if op.startswith(("bwd", "train")):
        bytes_, flops = bytes_ + bwd_bytes, flops + bwd_flops
    return {"bytes": bytes_, "flops": flops}


def tolerance(case):
    # bf16 operands and results with fp32 accumulation; P and dS are rounded to bf16 on the way (2^-9 each).  Largest
    # difference: a row that sees few keys has gradients of order 1 with roundings of about 1e-2 in them, while the root
    # mean square over a long causal sequence is 0.03.
    return {"rel": 1e-2, "max": 0.5}
