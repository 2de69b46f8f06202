"""GPU tests of the forward's work items: a thread block works through its own item and then takes over blocks that have
not started (several per SM here), with rings and barrier phases running on; items of one key block, pairs whose second
tile is missing or holds one row, the line between one and two query tiles per item, packed batches with items to pass
over.  Parity per (sequence, KV head) against fp32 attention; tolerances are the common ones of the forward (bf16 P and
O)."""
import pytest
import torch

import util
from hopper_jeni_b200 import ops
from oracle import sdpa_ref

pytestmark = pytest.mark.gpu


def _check(o, lse, q, k, v, scale, causal):  # [G, S, D], [G, S]; k, v [S, D]
    torch.backends.cuda.matmul.allow_tf32 = False
    z = torch.matmul(q.float(), k.float().t()) * scale
    if causal:
        z.masked_fill_(torch.ones_like(z[0], dtype=torch.bool).triu_(1), float("-inf"))
    lse_ref, o_ref = torch.logsumexp(z, -1), torch.matmul(torch.softmax(z, -1), v.float())
    m = sdpa_ref.metrics(o, o_ref)
    assert m["finite"] and m["gate_ok"] and m["rel_rms"] <= util.REL_RMS_FWD, m
    torch.testing.assert_close(lse, lse_ref, rtol=1e-3, atol=2e-3)


BATCHED = [
    # B, Hq, Hkv, S, D
    (8, 24, 8, 300, 64),     # 384 items of three tiles (two + one) on 148 SMs
    (8, 24, 8, 385, 128),    # the fourth tile holds one row
    (16, 32, 4, 70, 64),     # 512 items of one key block
    (16, 32, 4, 130, 128),   # one key block and two keys
    (1, 4, 2, 4731, 64),     # 148 tiles: one tile per item
    (1, 4, 2, 4737, 128),    # 152 tiles: two per item, the last one of a head holds one row
    (5, 6, 2, 640, 40),      # 150 tiles, head dimension below the kernel's
    (1, 16, 4, 1280, 64),    # 160 tiles in 80 pairs
    (1, 16, 4, 1537, 128),   # 208 tiles; the last tile of a head holds one row
    (4, 32, 8, 256, 64),     # 256 tiles of one and two key blocks
    (2, 24, 8, 129, 128),    # 96 tiles, the second key block holds one key
    (1, 16, 4, 2560, 64),    # 160 pairs: more items than SMs by a few
]


@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("shape", BATCHED)
def test_items_batched(gqa_lib, shape, causal):
    B, Hq, Hkv, S, D = shape
    G = Hq // Hkv
    gen = torch.Generator(device="cuda").manual_seed(7)
    q, k, v = (torch.randn(B, h, S, D, generator=gen, device="cuda").bfloat16() for h in (Hq, Hkv, Hkv))
    o, lse = torch.full_like(q, float("nan")), torch.full((B, Hq, S), float("nan"), device="cuda")
    scale = util.default_scale(D)
    ops.gqa_forward(q, k, v, causal=causal, scale=scale, out=o, lse=lse)
    ops.check_status()
    for b in range(B):
        for g in range(Hkv):
            h = slice(g * G, (g + 1) * G)
            _check(o[b, h], lse[b, h], q[b, h], k[b, g], v[b, g], scale, causal)


@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("Hq,Hkv,S,D", [
    (4, 2, 640, 64),
    (12, 4, 1000, 128),
    (6, 2, 256, 64),
    (16, 4, 1024, 80),
    (2, 2, 3000, 128),
])
def test_bits_do_not_depend_on_the_launch(gqa_lib, Hq, Hkv, S, D, causal):
    """O and LSE of a sequence are the same bits alone (one tile per item), among a few and in a large batch (pairs, several
    items per SM), and of a head's shard alone: a row's arithmetic depends on its own tile and nothing else."""
    B = 24
    gen = torch.Generator(device="cuda").manual_seed(9)
    q, k, v = (torch.randn(B, h, S, D, generator=gen, device="cuda").bfloat16() for h in (Hq, Hkv, Hkv))
    o, lse = ops.gqa_forward(q, k, v, causal=causal)
    for n in (1, 2, 5):
        o_n, lse_n = ops.gqa_forward(q[:n], k[:n], v[:n], causal=causal)
        assert torch.equal(o_n, o[:n]) and torch.equal(lse_n, lse[:n]), n
    G = Hq // Hkv
    o_1, lse_1 = ops.gqa_forward(q[:1, :G].contiguous(), k[:1, :1].contiguous(), v[:1, :1].contiguous(), causal=causal)
    assert torch.equal(o_1, o[:1, :G]) and torch.equal(lse_1, lse[:1, :G])
    ops.check_status()


@pytest.mark.parametrize("Hq,Hkv,S,D", [
    (24, 8, 1000, 128),   # 192 single tiles: the longest item bounds the launch
    (28, 4, 1024, 64),    # 224
    (36, 6, 1024, 64),    # 288 tiles in pairs: one head more than the line allows
    (24, 8, 900, 80),     # the last tile holds four rows
    (64, 8, 600, 128),    # an odd number of tiles, the last one partial
    (5, 1, 5000, 128),    # 200 single tiles, 40 key blocks in the longest
])
def test_single_tiles_and_pairs_are_the_same_bits(gqa_lib, Hq, Hkv, S, D):
    """Causal launches of more tiles than SMs on both sides of the line between one and two query tiles per item."""
    gen = torch.Generator(device="cuda").manual_seed(12)
    q, k, v = (torch.randn(1, h, S, D, generator=gen, device="cuda").bfloat16() for h in (Hq, Hkv, Hkv))
    o, lse = ops.gqa_forward(q, k, v, causal=True)
    G = Hq // Hkv
    for h in range(Hkv):  # a head's shard: every tile gets an SM of its own
        r = slice(h * G, (h + 1) * G)
        o_h, lse_h = ops.gqa_forward(q[:, r].contiguous(), k[:, h:h + 1].contiguous(), v[:, h:h + 1].contiguous(), causal=True)
        assert torch.equal(o_h, o[:, r]) and torch.equal(lse_h, lse[:, r]), h
    ops.check_status()


@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("D", [64, 128])
def test_items_packed(gqa_lib, D, causal):
    Hq, Hkv = 8, 2
    G = Hq // Hkv
    lens = [1, 0, 700, 128, 129, 0, 256, 33, 1500, 64, 257, 2, 511, 0, 90, 384] * 2
    T = sum(lens)
    gen = torch.Generator(device="cuda").manual_seed(8)
    q, k, v = (torch.randn(T, h, D, generator=gen, device="cuda").bfloat16() for h in (Hq, Hkv, Hkv))
    cu = torch.tensor([sum(lens[:i]) for i in range(len(lens) + 1)], dtype=torch.int32, device="cuda")
    o, lse = torch.full_like(q, float("nan")), torch.full((Hq, T), float("nan"), device="cuda")
    scale = util.default_scale(D)
    ops.gqa_forward_varlen(q, k, v, cu, 2048, causal=causal, scale=scale, out=o, lse=lse)
    ops.check_status()
    start = 0
    for n in lens:
        r = slice(start, start + n)
        start += n
        for g in range(Hkv if n else 0):
            h = slice(g * G, (g + 1) * G)
            _check(o[r, h].transpose(0, 1), lse[h, r], q[r, h].transpose(0, 1), k[r, g], v[r, g], scale, causal)


@pytest.mark.parametrize("causal", [False, True])
def test_long_run_of_empty_items(gqa_lib, causal):
    """65 534 empty sequences in front of one of 32 768 tokens: 7.3 million empty items per SM in a row, about two
    seconds, and the bounded wait of the other roles lasts one (2e9 cycles), so they must be woken in between."""
    S, Hq, Hkv, D, n_seqs = 32768, 128, 8, 64, 65535
    gen = torch.Generator(device="cuda").manual_seed(10)
    q, k, v = (torch.randn(S, h, D, generator=gen, device="cuda").bfloat16() for h in (Hq, Hkv, Hkv))
    cu = torch.zeros(n_seqs + 1, dtype=torch.int32, device="cuda")
    cu[-1] = S
    o, lse = ops.gqa_forward_varlen(q, k, v, cu, S, causal=causal)
    ops.check_status()
    o_ref, lse_ref = ops.gqa_forward(q[None], k[None], v[None], causal=causal, layout="bshd")
    assert torch.equal(o, o_ref[0]) and torch.equal(lse, lse_ref[0])
