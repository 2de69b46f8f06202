"""GPU tests of what the native host path owes its callers besides numbers: the classes of its outputs, the forms in which
it takes its arguments, errors raised in the autograd engine's thread, calls from several threads."""
import fractions
import threading

import numpy as np
import pytest
import torch

from hopper_jeni_b200 import capi, ops
from hopper_jeni_b200.autograd import gqa_attention, gqa_attention_varlen

pytestmark = pytest.mark.gpu

B, HQ, HKV, S, D = 1, 4, 2, 200, 64


class Tagged(torch.Tensor):
    """A subclass that hears which functions are called on it."""

    heard = []

    @classmethod
    def __torch_function__(cls, func, types, args=(), kwargs=None):
        cls.heard.append(getattr(func, "__name__", str(func)))
        return super().__torch_function__(func, types, args, kwargs or {})


class WrongShape(torch.Tensor):
    """A subclass whose empty_like does not do what it says."""

    @classmethod
    def __torch_function__(cls, func, types, args=(), kwargs=None):
        r = super().__torch_function__(func, types, args, kwargs or {})
        return r[..., :8].contiguous() if func is torch.empty_like else r


def _inputs(packed, seed=41):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    shape = (lambda h: (S, h, D)) if packed else (lambda h: (B, h, S, D))
    return [torch.randn(*shape(h), generator=gen, device="cuda").bfloat16() for h in (HQ, HKV, HKV, HQ)]


def _entry_points(packed):
    extra = (torch.tensor([0, 50, S], dtype=torch.int32, device="cuda"), 150) if packed else ()
    fwd, bwd, att = ((ops.gqa_forward_varlen, ops.gqa_backward_varlen, gqa_attention_varlen) if packed else
                     (ops.gqa_forward, ops.gqa_backward, gqa_attention))
    return (lambda q, k, v: fwd(q, k, v, *extra, causal=True),
            lambda q, k, v, o, do, lse: bwd(q, k, v, o, do, lse, *extra, causal=True),
            lambda q, k, v: att(q, k, v, *extra, causal=True))


@pytest.mark.parametrize("packed", [False, True])
def test_outputs_are_of_the_inputs_subclass(gqa_lib, packed):
    q, k, v, do = _inputs(packed)
    fwd, bwd, att = _entry_points(packed)
    o_ref, lse_ref = fwd(q, k, v)
    _, dk_ref, dv_ref = bwd(q, k, v, o_ref, do, lse_ref)
    tq, tk, tv = (t.as_subclass(Tagged) for t in (q, k, v))
    Tagged.heard.clear()
    o, lse = fwd(tq, tk, v)
    assert type(o) is Tagged and type(lse) is torch.Tensor and "empty_like" in Tagged.heard
    grads = bwd(q, tk, tv, o_ref, do, lse_ref)
    assert [type(g) for g in grads] == [torch.Tensor, Tagged, Tagged]
    plain = lambda t: t.as_subclass(torch.Tensor)
    assert torch.equal(plain(o), o_ref) and torch.equal(plain(grads[1]), dk_ref)
    # autograd, Q not contiguous
    sq = tq.transpose(0, 1).contiguous().transpose(0, 1).detach().requires_grad_(True)
    sk, sv = (t.detach().requires_grad_(True) for t in (tk, tv))
    out = att(sq, sk, sv)
    assert type(out) is Tagged
    dq, dk, dv = torch.autograd.grad(out, (sq, sk, sv), do)
    assert type(dk) is Tagged and type(dv) is Tagged
    assert torch.equal(plain(out), o_ref)
    assert torch.equal(plain(dk), dk_ref) and torch.equal(plain(dv), dv_ref)


def test_parameters_are_plain_tensors(gqa_lib):
    q, k, v, _ = _inputs(False)
    o, _ = ops.gqa_forward(*(torch.nn.Parameter(t) for t in (q, k, v)))
    assert type(o) is torch.Tensor and not o.requires_grad


def test_output_of_an_override_is_checked(gqa_lib):
    q, k, v, _ = (t.as_subclass(WrongShape) for t in _inputs(False))
    with pytest.raises(ValueError, match="O has shape"):
        ops.gqa_forward(q, k, v)


@pytest.mark.parametrize("scale", [np.float32(0.125), fractions.Fraction(1, 8), "0.125", torch.tensor(0.125)])
def test_scale_is_whatever_float_takes(gqa_lib, scale):
    q, k, v, do = _inputs(False)
    o, lse = ops.gqa_forward(q, k, v, scale=0.125)
    assert torch.equal(ops.gqa_forward(q, k, v, scale=scale)[0], o)
    assert torch.equal(gqa_attention(q, k, v, scale=scale), o)
    assert torch.equal(ops.gqa_backward(q, k, v, o, do, lse, scale=scale)[1],
                       ops.gqa_backward(q, k, v, o, do, lse, scale=0.125)[1])


def _misaligned(t):
    """The same values two bytes off a 16-byte boundary: contiguous, and refused by the library on the host."""
    return torch.cat([t.new_zeros(1), t.flatten()])[1:].view(t.shape)


@pytest.mark.parametrize("packed", [False, True])
@pytest.mark.parametrize("unpack,error,words", [
    (lambda t: t[..., :8], ValueError, "must be contiguous"),                            # refused by the binding
    (_misaligned, capi.GqaError, "gqa_bwd.* failed with GQA_ERR_BAD_ARGUMENT"),          # refused by the library
])
def test_error_in_the_backward_node(gqa_lib, packed, unpack, error, words):
    """The node runs in the engine's thread; its error reaches the caller, and the next call is good."""
    q, k, v, do = _inputs(packed)
    _, _, att = _entry_points(packed)
    leaves = [t.requires_grad_(True) for t in (q, k, v)]
    with torch.autograd.graph.saved_tensors_hooks(lambda t: t, lambda t: unpack(t) if t.dtype == torch.bfloat16 else t):
        out = att(*leaves)
    with pytest.raises(error, match=words):
        torch.autograd.grad(out, leaves, do)
    ref = torch.autograd.grad(att(*leaves), leaves, do)
    assert all(torch.isfinite(g.float()).all() for g in ref)


@pytest.mark.parametrize("packed", [False, True])
def test_threads_with_streams_of_their_own(gqa_lib, packed):
    """Four threads, each with its own inputs and stream: every call runs on the calling thread's current stream, in the
    backward on the forward's, and gives the bits of a call made alone."""
    fwd, _, att = _entry_points(packed)
    data = [_inputs(packed, seed=50 + i) for i in range(4)]

    def step(i):
        leaves = [t.clone().requires_grad_(True) for t in data[i][:3]]
        out = att(*leaves)
        return [out.detach(), *torch.autograd.grad(out, leaves, data[i][3])[1:], fwd(*data[i][:3])[1]]

    ref = [step(i) for i in range(4)]
    torch.cuda.synchronize()
    bad = []

    def work(i):
        try:
            stream = torch.cuda.Stream()
            with torch.cuda.stream(stream):
                for _ in range(25):
                    got = step(i)
                    stream.synchronize()
                    if not all(torch.equal(a, b) for a, b in zip(got, ref[i])):
                        bad.append((i, "differs"))
        except Exception as e:  # noqa: BLE001 (reported below)
            bad.append((i, e))

    threads = [threading.Thread(target=work, args=(i,)) for i in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join(timeout=60)
    assert not bad and not any(t.is_alive() for t in threads), bad
    ops.check_status()
