"""GPU tests of a call on a stream that is not torch's current one: what it allocates (workspace, outputs) is neither
handed out again while its kernels are queued there, nor memory that the current stream still uses, and what it returns
outlives the caller's own use of it."""
import pytest
import torch

from hopper_jeni_b200 import ops

pytestmark = pytest.mark.gpu

SLEEP = 20_000_000  # cycles: about ten milliseconds, against one for everything else here


def _problem(packed):
    Hq, Hkv, S, D = 8, 2, 512, 64
    gen = torch.Generator(device="cuda").manual_seed(17)
    shape = (lambda h: (S, h, D)) if packed else (lambda h: (1, h, S, D))
    q, k, v, do = (torch.randn(*shape(h), generator=gen, device="cuda").bfloat16() for h in (Hq, Hkv, Hkv, Hq))
    cu = torch.tensor([0, 200, S], dtype=torch.int32, device="cuda")
    args = (cu, 312) if packed else ()
    fwd, bwd = (ops.gqa_forward_varlen, ops.gqa_backward_varlen) if packed else (ops.gqa_forward, ops.gqa_backward)
    o, lse = fwd(q, k, v, *args, causal=True)
    return {"forward": lambda **s: fwd(q, k, v, *args, causal=True, **s),
            "backward": lambda **s: bwd(q, k, v, o, do, lse, *args, causal=True, **s)}


def _same(got, ref, name):
    for i, (g, r) in enumerate(zip(got, ref)):
        if name == "backward" and i == 0:  # dQ: same sums, order of the fp32 reductions varies (rounded to bf16: 2^-8)
            assert (g.float() - r.float()).norm() <= 4e-3 * r.float().norm()
        else:
            assert torch.equal(g, r), i


@pytest.mark.parametrize("packed", [False, True])
@pytest.mark.parametrize("name", ["forward", "backward"])
def test_call_on_another_stream(gqa_lib, name, packed):
    call = _problem(packed)[name]
    ref = [t.clone() for t in call()]
    sizes = sorted({t.numel() * t.element_size() for t in ref} | {1 << n for n in range(12, 23)})
    side, cur = torch.cuda.Stream(), torch.cuda.current_stream()
    torch.cuda.synchronize()
    torch.cuda.empty_cache()

    # blocks that the current stream still reads when the call allocates its outputs
    held = [torch.full((n,), 7, dtype=torch.uint8, device="cuda") for n in sizes]
    kept = [torch.empty_like(t) for t in held]
    side.wait_stream(cur)
    torch.cuda._sleep(SLEEP)
    for a, b in zip(held, kept):
        b.copy_(a)
    del held, a
    with torch.cuda.stream(side):
        torch.cuda._sleep(SLEEP)          # the call's kernels are queued behind this ...
    got = call(stream=side)
    fill = [torch.full((n,), 255, dtype=torch.uint8, device="cuda") for n in sizes for _ in range(2)]  # ... while this runs
    torch.cuda.synchronize()
    for t in kept:
        assert bool((t == 7).all())
    _same(got, ref, name)
    del fill, kept

    # results released while the current stream still reads them
    got = call(stream=side)
    cur.wait_stream(side)
    torch.cuda._sleep(SLEEP)
    copies = [t.clone() for t in got]
    shapes = [t.shape for t in got]
    dtypes = [t.dtype for t in got]
    del got
    with torch.cuda.stream(side):
        over = [torch.full(s, float("nan"), dtype=d, device="cuda") for s, d in zip(shapes, dtypes) for _ in range(2)]
    torch.cuda.synchronize()
    _same(copies, ref, name)
    del over
    ops.check_status()


def test_given_stream_is_the_one_that_runs(gqa_lib):
    """With every tensor given, nothing is allocated and the work is ordered on the given stream alone."""
    call = _problem(False)["forward"]
    ref = [t.clone() for t in call()]
    out, lse = (torch.full_like(t, float("nan")) for t in ref)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        torch.cuda._sleep(5 * SLEEP)
    got = call(stream=side, out=out, lse=lse)
    assert got[0] is out and got[1] is lse
    assert not side.query()
    torch.cuda.current_stream().wait_stream(side)
    assert torch.equal(out, ref[0]) and torch.equal(lse, ref[1])
