"""Autograd over the C ABI: the forward keeps O and LSE for the backward, so the backward does not recompute the
forward (the hand-off the reference does through files, src/attention/GQA_bwd_baseline.cu:641-643).  The nodes are
native (csrc/torch_binding.cpp)."""
from __future__ import annotations

from . import capi


def gqa_attention(q, k, v, causal: bool = False, scale: float | None = None, layout: str = "bhsd",
                  deterministic: bool = False):
    """Differentiable GQA attention on bf16 CUDA tensors ``[B,Hq,S,D]`` / ``[B,Hkv,S,D]``; same semantics as
    ``F.scaled_dot_product_attention(q, k, v, scale=scale, is_causal=causal, enable_gqa=True)``.
    ``layout="bshd"`` takes and returns ``[B,S,H,D]`` tensors; ``deterministic`` makes the gradient of q
    bit-reproducible (the other two always are)."""
    return capi.load_torch_binding().attention(q, k, v, causal, scale, layout, deterministic)


def gqa_attention_varlen(q, k, v, cu_seqlens, max_seqlen: int, causal: bool = False, scale: float | None = None):
    """Differentiable GQA attention over a packed variable-length batch: q ``[T,Hq,D]``, k and v ``[T,Hkv,D]`` bf16,
    ``cu_seqlens`` int32 ``[n_seqs+1]`` on the same device; every sequence attends only to itself."""
    return capi.load_torch_binding().attention_varlen(q, k, v, cu_seqlens, int(max_seqlen), causal, scale)
