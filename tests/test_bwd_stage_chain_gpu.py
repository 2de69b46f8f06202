"""GPU test of the backward's launch chain: the preprocess kernel zeroes the status word, the work counter and the ordered
mode's turn counters itself, and each later stage may start while the one before it still runs.  Calls back to back on one
workspace, poisoned in front of each, give the same bits (dK, dV; dQ too in the ordered mode) as a call on a fresh one, and
dQ of the default mode differs by the order of its fp32 sums alone (rounded to bf16: 2^-8 relative, 4e-3 in 2-norm)."""
import ctypes

import pytest
import torch

import util
from hopper_jeni_b200 import ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("deterministic", [False, True])
@pytest.mark.parametrize("shape", [(1, 2, 1, 1, 64), (1, 6, 2, 257, 64), (2, 8, 2, 700, 128), (4, 24, 8, 1024, 64)])
def test_poisoned_workspace_back_to_back(gqa_lib, shape, deterministic):
    B, Hq, Hkv, S, D = shape
    gen = torch.Generator(device="cuda").manual_seed(9)
    q, k, v, do = (torch.randn(B, h, S, D, generator=gen, device="cuda").bfloat16() for h in (Hq, Hkv, Hkv, Hq))
    scale = util.default_scale(D)
    o, lse = ops.gqa_forward(q, k, v, causal=True, scale=scale)
    n = ops.bwd_workspace_bytes(B, Hq, Hkv, S, D, True)

    def run(ws):
        return ops.gqa_backward(q, k, v, o, do, lse, causal=True, scale=scale, workspace=ws, deterministic=deterministic)

    ref = run(torch.zeros(n, dtype=torch.uint8, device="cuda"))
    ws = torch.empty(n, dtype=torch.uint8, device="cuda")
    outs = []
    for _ in range(6):
        ws.fill_(0xFF)
        outs.append(run(ws))
    outs += [run(ws) for _ in range(6)]  # no kernel of another kind in between
    ops.check_status(ws)
    for dq, dk, dv in outs:
        assert torch.equal(dk, ref[1]) and torch.equal(dv, ref[2])
        if deterministic:
            assert torch.equal(dq, ref[0])
        else:
            assert (dq.float() - ref[0].float()).norm() <= 4e-3 * ref[0].float().norm() + 1e-12


def test_refused_launch_leaves_no_error_behind(selftest_lib):
    """The launch helper of the dependent stages, given a launch that the runtime refuses on the host (an empty grid): an
    error left on the thread would be reported by the check behind the next launch, though that one is good."""
    left = ctypes.c_int(-1)
    assert selftest_lib.gqa_selftest_refused_launch(ctypes.byref(left)) == -4  # GQA_ERR_CUDA
    assert left.value == 0
