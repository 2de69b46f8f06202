"""GPU tests of the forward's work items: a thread block works through its own item and then takes over blocks that have
not started (several per SM here), with rings and barrier phases running on; items of one key block, pairs whose second
tile is missing or holds one row, the line between one and two query tiles per item, packed batches with items to pass
over.  Parity per (sequence, KV head) against fp32 attention; tolerances are the common ones of the forward (bf16 P and
O)."""
import statistics

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


@pytest.mark.parametrize("B,Hq,Hkv,S,D", [
    (2, 12, 4, 1000, 128),  # the last 4 of a head's 8 tiles are items of their own, the others pairs; one item per SM at the most
    (1, 28, 4, 1024, 64),   # 2 of 8
    (1, 32, 8, 1024, 128),  # 2 of 8: as many heads as the line allows; 160 items
    (1, 33, 11, 1024, 128), # pairs: one head more
    (4, 10, 2, 700, 80),    # 2 of 6; the last tile is partial; padded head dimension
    (1, 17, 1, 1600, 128),  # 5 of 13: an odd number of tiles
    (1, 23, 23, 1300, 40),  # 3 of 11; the last tile holds 20 rows
    (2, 32, 8, 600, 128),   # pairs, an odd number of tiles: the last one alone
    (1, 5, 1, 5000, 128),   # 12 of 40
])
def test_single_tiles_and_pairs_are_the_same_bits(gqa_lib, B, Hq, Hkv, S, D):
    """Causal launches of more tiles than SMs on both sides of the line between pairs of query tiles and the longest ones alone,
    against one head at a time, where every tile gets an SM of its own."""
    gen = torch.Generator(device="cuda").manual_seed(12)
    q, k, v = (torch.randn(B, h, S, D, generator=gen, device="cuda").bfloat16() for h in (Hq, Hkv, Hkv))
    o, lse = torch.full_like(q, float("nan")), torch.full((B, Hq, S), float("nan"), device="cuda")
    ops.gqa_forward(q, k, v, causal=True, out=o, lse=lse)
    for b in range(B):
        for h in range(Hq):
            g = h // (Hq // Hkv)
            o_h, lse_h = ops.gqa_forward(q[b:b + 1, h:h + 1].contiguous(), k[b:b + 1, g:g + 1].contiguous(),
                                         v[b:b + 1, g:g + 1].contiguous(), causal=True)
            assert torch.equal(o_h[0, 0], o[b, h]) and torch.equal(lse_h[0, 0], lse[b, h]), (b, h)
    if D in (64, 128):
        o_t, lse_t = ops.gqa_forward(*(t.transpose(1, 2).contiguous() for t in (q, k, v)), causal=True, layout="bshd")
        assert torch.equal(o_t.transpose(1, 2), o) and torch.equal(lse_t, lse)
    ops.check_status()


def test_single_tiles_cost_four_streams_little(gqa_lib):
    """Causal forwards of 32 heads end sooner alone with the longest tiles as items of their own; of 33 heads they are pairs.  Four
    streams that fill the chip pay for the SMs' time: 1.19 times as much with the longest two of eight tiles alone, 1.41 times
    with all eight alone.  The bound lies between."""
    calls, S, D = 8, 1024, 128
    streams = [torch.cuda.Stream() for _ in range(4)]

    def captured(heads):
        problems = []
        for _ in streams:
            q, k, v = (torch.randn(1, h, S, D, device="cuda").bfloat16() for h in (heads, 1, 1))
            problems.append((q, k, v, torch.empty_like(q), torch.empty(1, heads, S, device="cuda")))
        ops.gqa_forward(*problems[0][:3], causal=True)  # first use of the kernel, outside the capture
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            cur = torch.cuda.current_stream()
            for s, (q, k, v, o, lse) in zip(streams, problems):
                s.wait_stream(cur)
                with torch.cuda.stream(s):
                    for _ in range(calls):
                        ops.gqa_forward(q, k, v, causal=True, out=o, lse=lse)
            for s in streams:
                cur.wait_stream(s)
        return graph, problems

    def ms(graph):
        times = []
        for _ in range(9):
            a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            a.record()
            graph.replay()
            b.record()
            torch.cuda.synchronize()
            times.append(a.elapsed_time(b))
        return statistics.median(times)

    alone, pairs = captured(32), captured(33)
    ms(pairs[0])
    ratio = 33 / 32 * ms(alone[0]) / ms(pairs[0])
    assert ratio <= 1.30, ratio


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
