"""GPU test: backward calls that leave SMs idle run side by side on several streams.  A kernel of a call that waits for the
one in front of it must not hold the idle SMs meanwhile."""
import statistics

import pytest
import torch

from hopper_jeni_b200 import ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("deterministic", [False, True])
@pytest.mark.parametrize("D", [64, 128])
def test_small_backwards_of_four_streams_overlap(gqa_lib, D, deterministic):
    """32 of 148 SMs per call, so four calls have room side by side: 1.1 times one call's time, and two times where they keep
    one another off the SMs.  The bound lies halfway."""
    B, Hq, Hkv, S, calls = 1, 8, 2, 2048, 8
    gen = torch.Generator(device="cuda").manual_seed(23)

    def problem():
        q, k, v, do = (torch.randn(B, h, S, D, generator=gen, device="cuda").bfloat16() for h in (Hq, Hkv, Hkv, Hq))
        o, lse = ops.gqa_forward(q, k, v)
        ws = torch.empty(ops.bwd_workspace_bytes(B, Hq, Hkv, S, D), dtype=torch.uint8, device="cuda")
        out = dict(dq=torch.empty_like(q), dk=torch.empty_like(k), dv=torch.empty_like(v))
        return lambda: ops.gqa_backward(q, k, v, o, do, lse, workspace=ws, deterministic=deterministic, **out)

    problems, streams = [problem() for _ in range(4)], [torch.cuda.Stream() for _ in range(4)]

    def captured(n):
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            cur = torch.cuda.current_stream()
            for s in streams[:n]:
                s.wait_stream(cur)
            for s, call in zip(streams[:n], problems):
                with torch.cuda.stream(s):
                    for _ in range(calls):
                        call()
            for s in streams[:n]:
                cur.wait_stream(s)
        return graph

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

    problems[0]()  # first use of the kernels, outside the capture
    torch.cuda.synchronize()
    one, four = captured(1), captured(4)
    alone = ms(one)
    together = ms(four)
    assert together <= 1.55 * alone, (alone, together)
