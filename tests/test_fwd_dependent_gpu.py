"""GPU tests of the forward behind work that is not this library's: it is launched so that its blocks may come up under the end
of whatever stands in front of it in the stream, and waits there before it touches memory.  In front here: copies, memset and
kernels of torch, an event of another stream, cuBLAS products, and forwards that write what the next one reads or read
what it writes; eagerly and as nodes of a graph.  Expected values are the same calls with a synchronisation on both sides
(the forward's bits do not vary)."""
import pytest
import torch

from hopper_jeni_b200 import ops

pytestmark = pytest.mark.gpu

SHAPES = [  # B, Hq, Hkv, S, D, causal
    (1, 4, 2, 128, 64, True),     # one short launch
    (2, 12, 4, 1000, 128, True),  # fewer items than SMs
    (4, 16, 4, 1500, 64, False),  # more
]


def _fresh(shape, gen):
    B, Hq, Hkv, S, D, _ = shape
    return [torch.randn(B, h, S, D, generator=gen, device="cuda").bfloat16() for h in (Hq, Hkv, Hkv)]


def _settled(q, k, v, causal):
    torch.cuda.synchronize()
    out = ops.gqa_forward(q, k, v, causal=causal)
    torch.cuda.synchronize()
    return out


@pytest.mark.parametrize("shape", SHAPES)
def test_behind_copies_memset_and_another_stream_in_a_graph(gqa_lib, shape):
    causal = shape[-1]
    gen = torch.Generator(device="cuda").manual_seed(41)
    src = _fresh(shape, gen)
    q, k, v = (torch.empty_like(t) for t in src)
    o, o2 = torch.empty_like(q), torch.empty_like(q)
    lse = torch.empty(q.shape[:3], dtype=torch.float32, device="cuda")
    side = torch.cuda.Stream()

    def step():
        main = torch.cuda.current_stream()
        side.wait_stream(main)
        with torch.cuda.stream(side):
            k.copy_(src[1])
            v.copy_(src[2])
        o.zero_()                    # memset node
        main.wait_stream(side)       # two nodes in front of the next one
        q.copy_(src[0])              # copy node, directly in front of the forward
        ops.gqa_forward(q, k, v, causal=causal, out=o, lse=lse)
        ops.gqa_forward(o, k, v, causal=causal, out=o2, lse=lse)  # reads what the one before it writes
        q.fill_(float("nan"))        # overwrites what the first one reads

    step()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        step()
    for trial in range(4):
        for t, x in zip(src, _fresh(shape, gen)):
            t.copy_(x)
        for t in (q, k, v, o, o2):
            t.fill_(float("nan"))
        torch.cuda.synchronize()
        graph.replay()
        graph.replay()               # and behind itself
        torch.cuda.synchronize()
        ops.check_status()
        want, _ = _settled(*src, causal)
        want2, want_lse = _settled(want, src[1], src[2], causal)
        assert torch.equal(o, want) and torch.equal(o2, want2) and torch.equal(lse, want_lse), trial


@pytest.mark.parametrize("shape", SHAPES)
def test_behind_products_and_forwards_of_its_own_stream(gqa_lib, shape):
    B, Hq, Hkv, S, D, causal = shape
    gen = torch.Generator(device="cuda").manual_seed(42)
    w = (torch.randn(D, D, generator=gen, device="cuda") / D ** 0.5).bfloat16()
    n = 12
    sets = [_fresh(shape, gen) for _ in range(n)]
    torch.cuda.synchronize()
    got, buf = [], torch.empty_like(sets[0][0])
    for q, k, v in sets:
        torch.matmul(q, w, out=buf)                  # a cuBLAS kernel writes Q ...
        a = ops.gqa_forward(buf, k, v, causal=causal)
        b = ops.gqa_forward(a[0], k, v, causal=causal, out=buf)  # ... and the second forward overwrites it
        got.append((*a, buf.clone(), b[1]))
    torch.cuda.synchronize()
    ops.check_status()
    for (q, k, v), g in zip(sets, got):
        a = _settled(torch.matmul(q, w), k, v, causal)
        b = _settled(a[0], k, v, causal)
        assert all(torch.equal(x, y) for x, y in zip(g, (*a, *b)))


@pytest.mark.parametrize("shape", SHAPES)
def test_behind_an_event_of_another_stream(gqa_lib, shape):
    causal = shape[-1]
    gen = torch.Generator(device="cuda").manual_seed(43)
    n = 12
    sets = [_fresh(shape, gen) for _ in range(n)]
    late = [[torch.empty_like(t) for t in s] for s in sets]
    busy = torch.randn(4096, 4096, device="cuda")
    torch.cuda.synchronize()
    side, got = torch.cuda.Stream(), []
    for s, d in zip(sets, late):
        with torch.cuda.stream(side):
            torch.mm(busy, busy)     # the inputs arrive late, while the forward before still runs or has long ended
            for x, y in zip(s, d):
                y.copy_(x)
            arrived = side.record_event()
        torch.cuda.current_stream().wait_event(arrived)
        got.append(ops.gqa_forward(*d, causal=causal))
    torch.cuda.synchronize()
    ops.check_status()
    for s, g in zip(sets, got):
        want = _settled(*s, causal)
        assert torch.equal(g[0], want[0]) and torch.equal(g[1], want[1])
