"""GPU tests of the deterministic backward (gqa_bwd_ex with GQA_BWD_DETERMINISTIC): dQ is bit-identical from
run to run (what the reference's vj1d_determinism_probe.cu measures for its own kernel), agrees with the CPU
oracle, and equals the default mode up to the order of the fp32 additions."""
import ctypes

import pytest
import torch

import util
from hopper_jeni_b200 import capi, ops

pytestmark = pytest.mark.gpu


def _inputs(B, Hq, Hkv, S, D, causal, seed):
    q, k, v, do = util.make_inputs(B, Hq, Hkv, S, D, seed=seed)
    tq, tk, tv, tdo = (util.to_dev_bf16(x) for x in (q, k, v, do))
    o, lse = ops.gqa_forward(tq, tk, tv, causal=causal)
    return (q, k, v, do), (tq, tk, tv, tdo, o, lse)


@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("shape", [(2, 6, 2, 256, 64), (1, 4, 2, 384, 128)])
def test_deterministic_backward_matches_oracle(gqa_lib, oracle, shape, causal):
    B, Hq, Hkv, S, D = shape
    (q, k, v, do), (tq, tk, tv, tdo, o, lse) = _inputs(B, Hq, Hkv, S, D, causal, seed=71)
    sc = util.default_scale(D)
    dq_ref, dk_ref, dv_ref = oracle.backward(q, k, v, do, causal, sc)
    ws = torch.empty(ops.bwd_workspace_bytes(B, Hq, Hkv, S, D, causal), dtype=torch.uint8, device="cuda")
    dq, dk, dv = ops.gqa_backward(tq, tk, tv, o, tdo, lse, causal=causal, scale=sc, workspace=ws, deterministic=True)
    ops.check_status(ws)
    util.assert_close_bf16(util.to_np(dq), dq_ref, "dQ", util.REL_RMS_BWD)
    util.assert_close_bf16(util.to_np(dk), dk_ref, "dK", util.REL_RMS_BWD)
    util.assert_close_bf16(util.to_np(dv), dv_ref, "dV", util.REL_RMS_BWD)


@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("shape", [
    (1, 4, 2, 100, 64),     # one tile: a single turn
    (2, 4, 2, 333, 40),
    (1, 6, 2, 333, 80),     # the padded form
    (1, 8, 1, 129, 128),    # the second tile holds one row
    (1, 2, 1, 1100, 64),    # nine tiles: four of them in descending order when causal, five more behind
])
def test_ordered_form_matches_oracle_at_odd_sizes(gqa_lib, oracle, shape, causal):
    B, Hq, Hkv, S, D = shape
    (q, k, v, do), (tq, tk, tv, tdo, o, lse) = _inputs(B, Hq, Hkv, S, D, causal, seed=73)
    refs = oracle.backward(q, k, v, do, causal, util.default_scale(D))
    ws = torch.full((ops.bwd_workspace_bytes(B, Hq, Hkv, S, D, causal),), 255, dtype=torch.uint8, device="cuda")
    runs = [ops.gqa_backward(tq, tk, tv, o, tdo, lse, causal=causal, workspace=ws, deterministic=True) for _ in range(2)]
    ops.check_status(ws)
    for name, a, b, ref in zip(("dQ", "dK", "dV"), *runs, refs):
        assert torch.equal(a, b), name
        util.assert_close_bf16(util.to_np(a), ref, name, util.REL_RMS_BWD)


@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("shape", [(2, 12, 4, 2048, 64), (2, 8, 2, 2048, 128), (8, 12, 4, 4096, 64)])
def test_deterministic_backward_is_bit_reproducible(gqa_lib, shape, causal):
    """More thread blocks than SMs, several per (batch, KV head) group: every dQ tile gets up to S/128 ordered
    reductions.  Four runs, all three gradients bit-identical; the default mode agrees up to the order of its fp32
    sums."""
    B, Hq, Hkv, S, D = shape
    gen = torch.Generator(device="cuda").manual_seed(5)
    q = torch.randn(B, Hq, S, D, generator=gen, device="cuda").bfloat16()
    k = torch.randn(B, Hkv, S, D, generator=gen, device="cuda").bfloat16()
    v = torch.randn(B, Hkv, S, D, generator=gen, device="cuda").bfloat16()
    do = torch.randn(B, Hq, S, D, generator=gen, device="cuda").bfloat16()
    o, lse = ops.gqa_forward(q, k, v, causal=causal)
    ws = torch.empty(ops.bwd_workspace_bytes(B, Hq, Hkv, S, D, causal), dtype=torch.uint8, device="cuda")
    runs = []
    for _ in range(4):
        runs.append(ops.gqa_backward(q, k, v, o, do, lse, causal=causal, workspace=ws, deterministic=True))
        ops.check_status(ws)
    for dq, dk, dv in runs[1:]:
        assert torch.equal(dq, runs[0][0]), "dQ differs between deterministic runs"
        assert torch.equal(dk, runs[0][1]) and torch.equal(dv, runs[0][2])
    dq0, dk0, dv0 = ops.gqa_backward(q, k, v, o, do, lse, causal=causal, workspace=ws)
    ops.check_status(ws)
    if causal:
        assert torch.equal(dk0, runs[0][1]) and torch.equal(dv0, runs[0][2])
    else:
        # without a mask the default mode starts each KV tile's loop over the query tiles at a different tile (the
        # ordered mode does not): the same fp32 sums in another order
        for got, want in ((dk0, runs[0][1]), (dv0, runs[0][2])):
            m = util.metrics(util.to_np(got), util.to_np(want))
            assert m["rel_rms"] < 2e-3, m
    m = util.metrics(util.to_np(dq0), util.to_np(runs[0][0]))
    assert m["rel_rms"] < 2e-3, m


@pytest.mark.parametrize("shape", [
    (1, 2, 1, 1664, 64),     # one group of 13 KV tiles
    (2, 40, 20, 1024, 128),  # 40 groups of eight
    (1, 74, 74, 700, 64),    # 74 groups of six, a partial last tile
    (10, 16, 16, 300, 64),   # more groups than SMs, two of three tiles in descending order
    (1, 4, 2, 520, 72),      # three of five; a head dimension that is not native
])
def test_causal_order_of_the_reductions(gqa_lib, shape):
    """The causal list starts with half of the KV tiles of a group, four at most, in descending order, and the turns follow it.  Three
    runs bit-identical, dK and dV the default mode's bits, dQ its sums in another order (as above)."""
    B, Hq, Hkv, S, D = shape
    gen = torch.Generator(device="cuda").manual_seed(6)
    q, do = (torch.randn(B, Hq, S, D, generator=gen, device="cuda").bfloat16() for _ in range(2))
    k, v = (torch.randn(B, Hkv, S, D, generator=gen, device="cuda").bfloat16() for _ in range(2))
    o, lse = ops.gqa_forward(q, k, v, causal=True)
    ws = torch.empty(ops.bwd_workspace_bytes(B, Hq, Hkv, S, D, True), dtype=torch.uint8, device="cuda")
    want = ops.gqa_backward(q, k, v, o, do, lse, causal=True, workspace=ws)
    runs = []
    for _ in range(3):
        ws.fill_(0xA5)
        runs.append(ops.gqa_backward(q, k, v, o, do, lse, causal=True, workspace=ws, deterministic=True))
        ops.check_status(ws)
    for got in runs:
        assert all(torch.equal(a, b) for a, b in zip(got, runs[0]))
    assert torch.equal(runs[0][1], want[1]) and torch.equal(runs[0][2], want[2])
    m = util.metrics(util.to_np(runs[0][0]), util.to_np(want[0]))
    assert m["rel_rms"] < 2e-3, m


@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("Hq,Hkv,S,D", [(4, 2, 640, 64), (4, 4, 300, 64), (6, 2, 1100, 128), (4, 2, 2048, 80)])
def test_ordered_gradients_do_not_depend_on_the_launch(gqa_lib, Hq, Hkv, S, D, causal):
    """The order of the fp32 sums depends on S and the mask alone: the gradients of a sequence are the same bits alone, in
    batches of every size and on a shard that holds one KV head."""
    B, G = 40, Hq // Hkv
    gen = torch.Generator(device="cuda").manual_seed(12)
    q, do = (torch.randn(B, Hq, S, D, generator=gen, device="cuda").bfloat16() for _ in range(2))
    k, v = (torch.randn(B, Hkv, S, D, generator=gen, device="cuda").bfloat16() for _ in range(2))
    o, lse = ops.gqa_forward(q, k, v, causal=causal)

    def grads(n, hq=Hq, hkv=Hkv):
        args = [t[:n, :h].contiguous() for t, h in ((q, hq), (k, hkv), (v, hkv), (o, hq), (do, hq), (lse, hq))]
        return ops.gqa_backward(*args, causal=causal, deterministic=True)

    whole = grads(B)
    for n, hq, hkv in ((1, Hq, Hkv), (7, Hq, Hkv), (1, G, 1)):
        for got, want, h in zip(grads(n, hq, hkv), whole, (hq, hkv, hkv)):
            assert torch.equal(got, want[:n, :h]), (n, hq)


def test_unknown_flag_bits_are_refused(gqa_lib):
    lib = capi.load_library()
    q = torch.zeros(1, 2, 128, 64, dtype=torch.bfloat16, device="cuda")
    lse = torch.zeros(1, 2, 128, dtype=torch.float32, device="cuda")
    ws = torch.empty(ops.bwd_workspace_bytes(1, 2, 2, 128, 64), dtype=torch.uint8, device="cuda")
    p = q.data_ptr()
    rc = lib.gqa_bwd_ex(p, p, p, p, p, lse.data_ptr(), p, p, p, 1, 2, 2, 128, 64, 0, 0.125, ws.data_ptr(), ws.numel(),
                        None, ctypes.c_uint(0x10))
    assert rc == -1
