"""GPU tests of the alternative dQ path (GQA_BWD_DQ_SEPARATE): dQ from a separate query-parallel pass, the layout of
the reference's first generations (a dQ kernel per query tile beside a dK/dV kernel per key tile,
src/attention/GQA_bwd.cu:29, :415, :1416), instead of fp32 reductions into an accumulator
(src/attention/GQA_bwd_baseline.cu:360-365).  All three gradients must match the oracle, dQ must be bit-identical
from run to run (its summation order is fixed), and dK / dV must be the bits the default path produces (the main
kernel computes them the same way with or without its dQ part)."""
import pytest
import torch

import util
from hopper_jeni_b200 import ops

pytestmark = pytest.mark.gpu

CASES = [
    # B, Hq, Hkv, S, D, causal
    (1, 2, 1, 128, 64, False),      # one tile
    (2, 6, 2, 512, 64, True),       # G = 3, diagonal blocks
    (1, 4, 4, 640, 64, False),      # MHA; five key blocks wrap the four-stage ring
    (1, 4, 2, 384, 128, True),      # D = 128 (two-stage ring)
    (1, 8, 1, 200, 96, True),       # padded head dimension, partial tile, MQA
    (1, 4, 2, 450, 64, False),      # ragged
]


@pytest.mark.parametrize("case", CASES)
def test_separate_dq_matches_oracle_and_is_bit_reproducible(gqa_lib, oracle, case):
    B, Hq, Hkv, S, D, causal = case
    q, k, v, do = util.make_inputs(B, Hq, Hkv, S, D, seed=23)
    sc = util.default_scale(D)
    tq, tk, tv, tdo = (util.to_dev_bf16(x) for x in (q, k, v, do))
    o_ref, lse_ref = oracle.forward(q, k, v, causal, sc)
    to = util.to_dev_bf16(util.bf16_round(o_ref))
    tlse = torch.from_numpy(lse_ref).cuda()
    ws = torch.empty(ops.bwd_workspace_bytes(B, Hq, Hkv, S, D, causal), dtype=torch.uint8, device="cuda")
    runs = []
    for _ in range(3):
        dq, dk, dv = (torch.full_like(t, float("nan")) for t in (tq, tk, tv))
        ops.gqa_backward(tq, tk, tv, to, tdo, tlse, causal=causal, scale=sc, workspace=ws, dq=dq, dk=dk, dv=dv,
                         dq_separate=True)
        ops.check_status(ws)
        runs.append((dq, dk, dv))
    dq_ref, dk_ref, dv_ref = oracle.backward(q, k, v, do, causal, sc)
    util.assert_close_bf16(util.to_np(runs[0][0]), dq_ref, "dQ", util.REL_RMS_BWD)
    util.assert_close_bf16(util.to_np(runs[0][1]), dk_ref, "dK", util.REL_RMS_BWD)
    util.assert_close_bf16(util.to_np(runs[0][2]), dv_ref, "dV", util.REL_RMS_BWD)
    for dq, dk, dv in runs[1:]:
        assert torch.equal(dq, runs[0][0]) and torch.equal(dk, runs[0][1]) and torch.equal(dv, runs[0][2])
    dq0, dk0, dv0 = ops.gqa_backward(tq, tk, tv, to, tdo, tlse, causal=causal, scale=sc, workspace=ws)
    assert torch.equal(dk0, runs[0][1]) and torch.equal(dv0, runs[0][2])
    assert util.metrics(util.to_np(runs[0][0]), util.to_np(dq0))["rel_rms"] < 5e-3


def test_separate_dq_at_the_headline_shape(gqa_lib):
    """B8 Hq12 Hkv4 S4096 D64: the two dQ paths agree (relative RMS; both are rounded to bf16 once)."""
    B, Hq, Hkv, S, D = 8, 12, 4, 4096, 64
    g = torch.Generator(device="cuda").manual_seed(5)
    q = torch.randn(B, Hq, S, D, generator=g, device="cuda").bfloat16()
    k = torch.randn(B, Hkv, S, D, generator=g, device="cuda").bfloat16()
    v = torch.randn(B, Hkv, S, D, generator=g, device="cuda").bfloat16()
    do = torch.randn(B, Hq, S, D, generator=g, device="cuda").bfloat16()
    o, lse = ops.gqa_forward(q, k, v)
    ws = torch.empty(ops.bwd_workspace_bytes(B, Hq, Hkv, S, D), dtype=torch.uint8, device="cuda")
    dq_a, dk_a, dv_a = ops.gqa_backward(q, k, v, o, do, lse, workspace=ws)
    dq_b, dk_b, dv_b = ops.gqa_backward(q, k, v, o, do, lse, workspace=ws, dq_separate=True)
    ops.check_status(ws)
    assert torch.equal(dk_a, dk_b) and torch.equal(dv_a, dv_b)
    m = util.metrics(util.to_np(dq_b[:2]), util.to_np(dq_a[:2]))
    assert m["rel_rms"] < 3e-3 and m["gate_ok"], m


@pytest.mark.parametrize("S", [65, 127, 129, 257, 385, 513])
@pytest.mark.parametrize("D,causal,layout", [(64, True, "bhsd"), (128, False, "bhsd"), (80, True, "bhsd"), (32, False, "bhsd"),
                                             (128, True, "bshd")])
def test_separate_dq_at_tile_edges(gqa_lib, oracle, S, D, causal, layout):
    """One to five key blocks: the two S buffers, the key ring of three blocks and the value ring of two wrap, the last block and
    the last tile are partial; padded head dimensions.  dQ written over dO is the same bits (the pass then waits for the main
    kernel instead of running beside it)."""
    B, Hq, Hkv = 2, 4, 2
    q, k, v, do = util.make_inputs(B, Hq, Hkv, S, D, seed=31)
    sc = util.default_scale(D)
    o_ref, lse_ref = oracle.forward(q, k, v, causal, sc)
    order = (lambda t: t.transpose(1, 2).contiguous()) if layout == "bshd" else (lambda t: t)
    tq, tk, tv, tdo, to = (order(util.to_dev_bf16(x)) for x in (q, k, v, do, util.bf16_round(o_ref)))
    tlse = torch.from_numpy(lse_ref).cuda()
    ws = torch.empty(ops.bwd_workspace_bytes(B, Hq, Hkv, S, D, causal), dtype=torch.uint8, device="cuda")
    kw = dict(causal=causal, scale=sc, workspace=ws, layout=layout)
    dq, dk, dv = ops.gqa_backward(tq, tk, tv, to, tdo, tlse, dq=torch.full_like(tq, float("nan")), dq_separate=True, **kw)
    ops.check_status(ws)
    dq0, dk0, dv0 = ops.gqa_backward(tq, tk, tv, to, tdo, tlse, **kw)
    assert torch.equal(dk, dk0) and torch.equal(dv, dv0)
    dq_ref, _, _ = oracle.backward(q, k, v, do, causal, sc)
    util.assert_close_bf16(util.to_np(order(dq)), dq_ref, "dQ", util.REL_RMS_BWD)
    over = tdo.clone()
    dq1, dk1, dv1 = ops.gqa_backward(tq, tk, tv, to, over, tlse, dq=over, dq_separate=True, **kw)
    ops.check_status(ws)
    assert torch.equal(dq1, dq) and torch.equal(dk1, dk) and torch.equal(dv1, dv)


# Shapes whose main kernel takes much longer than the pass beside it: one KV head, so few KV tiles with all query heads each,
# while the pass has a thread block per query tile.
OUTLASTING = [(1, 8, 1, 1024, 64, True), (1, 8, 1, 1024, 128, False), (2, 6, 1, 700, 80, True)]


def _problems(n, B, Hq, Hkv, S, D, causal):
    """n problems as (inputs, expected gradients); the expected ones from calls with the host waiting before and after each."""
    gen = torch.Generator(device="cuda").manual_seed(41)
    out = []
    for _ in range(n):
        q, k, v, do = (torch.randn(B, h, S, D, generator=gen, device="cuda").bfloat16() for h in (Hq, Hkv, Hkv, Hq))
        o, lse = ops.gqa_forward(q, k, v, causal=causal)
        ws = torch.empty(ops.bwd_workspace_bytes(B, Hq, Hkv, S, D, causal), dtype=torch.uint8, device="cuda")
        torch.cuda.synchronize()
        want = ops.gqa_backward(q, k, v, o, do, lse, causal=causal, workspace=ws, dq_separate=True)
        torch.cuda.synchronize()
        ops.check_status(ws)
        out.append(((q, k, v, o, do, lse), want))
    return out


def _call_and_consume(inputs, ws, grads, results, causal):
    """The backward; directly behind it a reader of all it writes and a writer of all it reads (copies that later calls do not
    use): kernels that come too early if the call's last kernel does not wait for the main kernel."""
    q, k, v, o, do, lse = inputs
    ops.gqa_backward(q, k, v, o, do, lse, causal=causal, workspace=ws, dq_separate=True, dq=grads[0], dk=grads[1], dv=grads[2])
    for r, g in zip(results, grads):
        r.copy_(g)
    for g in grads:
        g.zero_()
    for t in (q, k, v, do):
        t.fill_(float("nan"))


@pytest.mark.parametrize("case", OUTLASTING)
def test_separate_dq_keeps_the_order_of_the_stream(gqa_lib, case):
    """Calls one behind the other on one workspace and one set of gradients, with no wait on the host: eagerly, from a captured graph
    and on two streams at once with a workspace each."""
    B, Hq, Hkv, S, D, causal = case
    n = 6
    problems = _problems(n, *case)
    results = [[torch.empty_like(g) for g in want] for _, want in problems]
    n_ws = ops.bwd_workspace_bytes(B, Hq, Hkv, S, D, causal)
    lanes = [(torch.cuda.Stream(), torch.empty(n_ws, dtype=torch.uint8, device="cuda"), [torch.empty_like(g) for g in problems[0][1]])
             for _ in range(2)]  # stream, workspace, gradients
    work = [[t.clone() for t in inputs] for inputs, _ in problems]

    def refill():
        for w, (inputs, _) in zip(work, problems):
            for dst, src in zip(w, inputs):
                dst.copy_(src)
        for r in results:
            for t in r:
                t.fill_(float("nan"))

    def check(what):
        torch.cuda.synchronize()
        for _, ws, _ in lanes:
            ops.check_status(ws)
        for i, (r, (_, want)) in enumerate(zip(results, problems)):
            for name, a, b in zip(("dQ", "dK", "dV"), r, want):
                assert torch.equal(a, b), (what, i, name)

    def run(streams):
        for i in range(n):
            st, ws, grads = lanes[i % len(streams)]
            with torch.cuda.stream(streams[i % len(streams)]):
                _call_and_consume(work[i], ws, grads, results[i], causal)

    lanes[0][1].fill_(255)
    lanes[1][1].zero_()  # not used by the first runs: its status word reads as no report
    for trial in range(3):
        refill()
        torch.cuda.synchronize()
        run([lanes[0][0]])
        check(("one stream", trial))
    for trial in range(3):
        refill()
        torch.cuda.synchronize()
        run([lanes[0][0], lanes[1][0]])
        check(("two streams", trial))
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=lanes[0][0]):
        run([lanes[0][0]])
    for trial in range(3):
        refill()
        graph.replay()
        check(("graph", trial))


@pytest.mark.parametrize("D,causal", [(64, True), (128, False), (80, True)])
def test_separate_dq_with_a_head_split(gqa_lib, D, causal):
    """A split that takes effect puts the sum of the parts between the two kernels: dK and dV are the bits of the split alone, dQ
    the bits of the separate pass alone."""
    B, Hq, Hkv, S = 1, 8, 1, 1000
    n_ws = ops.bwd_workspace_bytes(B, Hq, Hkv, S, D, causal, split_heads=True)
    assert n_ws > ops.bwd_workspace_bytes(B, Hq, Hkv, S, D, causal)
    ((q, k, v, o, do, lse), want), = _problems(1, B, Hq, Hkv, S, D, causal)
    ws = torch.full((n_ws,), 255, dtype=torch.uint8, device="cuda")
    _, dk0, dv0 = ops.gqa_backward(q, k, v, o, do, lse, causal=causal, workspace=ws, split_heads=True)
    for _ in range(3):
        dq, dk, dv = ops.gqa_backward(q, k, v, o, do, lse, causal=causal, workspace=ws, split_heads=True, dq_separate=True)
        got = [t.clone() for t in (dq, dk, dv)]  # directly behind the call
        ops.check_status(ws)
        assert torch.equal(got[0], want[0]) and torch.equal(got[1], dk0) and torch.equal(got[2], dv0)


@pytest.mark.parametrize("S,over", [(128, "q"), (128, "k"), (128, "v"), (100, "k"), (500, "q"), (1024, "do")])
@pytest.mark.parametrize("D", [64, 128])
def test_separate_dq_in_place_of_an_input(gqa_lib, S, over, D):
    """dQ written over an input of its own size is the same bits: over Q and dO, whose rows only their own thread block reads, at any
    length; over K and V where one query tile sees one key block."""
    B, H = 3, 4
    ((q, k, v, o, do, lse), want), = _problems(1, B, H, H, S, D, False)
    ws = torch.full((ops.bwd_workspace_bytes(B, H, H, S, D),), 255, dtype=torch.uint8, device="cuda")
    t = {"q": q, "k": k, "v": v, "do": do}
    t[over] = t[over].clone()
    dq, dk, dv = ops.gqa_backward(t["q"], t["k"], t["v"], o, t["do"], lse, workspace=ws, dq=t[over], dq_separate=True)
    got = [x.clone() for x in (dq, dk, dv)]
    ops.check_status(ws)
    for name, a, b in zip(("dQ", "dK", "dV"), got, want):
        assert torch.equal(a, b), name
