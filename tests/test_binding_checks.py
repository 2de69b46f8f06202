"""CPU tests of the argument checks in the native tensor-level host path.  The inputs are fake tensors (sizes, strides,
types and CUDA devices without memory behind them), so a check that lets a wrong call through cannot launch anything:
the call would fail with another error than the ValueError asked for."""
import pytest
import torch
from torch._subclasses.fake_tensor import FakeTensorMode

from hopper_jeni_b200 import ops
from hopper_jeni_b200.autograd import gqa_attention, gqa_attention_varlen

B, HQ, HKV, S, D, T = 2, 4, 2, 96, 64, 160


def _fake(*shape, device="cuda:0", dtype=torch.bfloat16):
    with FakeTensorMode():
        return torch.empty(*shape, dtype=dtype, device=device)


def _calls(kv=None, packed_kv=None):
    """Every entry point as (name, call); the arguments given replace K and V."""
    f32 = torch.float32
    q = _fake(B, HQ, S, D)
    k, v = kv or (_fake(B, HKV, S, D), _fake(B, HKV, S, D))
    o, lse = _fake(B, HQ, S, D), _fake(B, HQ, S, dtype=f32)
    pq = _fake(T, HQ, D)
    pk, pv = packed_kv or (_fake(T, HKV, D), _fake(T, HKV, D))
    po, plse, cu = _fake(T, HQ, D), _fake(HQ, T, dtype=f32), _fake(3, dtype=torch.int32)
    return [
        ("forward", lambda **a: ops.gqa_forward(q, k, v, **a)),
        ("backward", lambda **a: ops.gqa_backward(q, k, v, o, o, lse, **a)),
        ("attention", lambda: gqa_attention(q, k, v)),
        ("forward_varlen", lambda **a: ops.gqa_forward_varlen(pq, pk, pv, cu, S, **a)),
        ("backward_varlen", lambda **a: ops.gqa_backward_varlen(pq, pk, pv, po, po, plse, cu, S, **a)),
        ("attention_varlen", lambda: gqa_attention_varlen(pq, pk, pv, cu, S)),
    ]


ENTRY_POINTS = [n for n, _ in _calls()]


@pytest.mark.parametrize("entry", ENTRY_POINTS)
def test_k_and_v_on_another_device_are_refused(gqa_lib, entry):
    """The kernels run on Q's device: K and V of another one would be read, and dK and dV written, across devices."""
    kv = [_fake(B, HKV, S, D, device="cuda:1") for _ in range(2)]
    packed = [_fake(T, HKV, D, device="cuda:1") for _ in range(2)]
    with pytest.raises(ValueError, match="K is on cuda:1, expected cuda:0"):
        dict(_calls(kv=kv, packed_kv=packed))[entry]()


def _wrong(kind, shape, dtype):
    """A tensor that differs from what is wanted in one point, and the words of the refusal."""
    if kind == "shape":
        return _fake(*shape[:-1], shape[-1] - 1, dtype=dtype), "has shape"
    if kind == "dtype":
        return _fake(*shape, dtype=torch.float16), "must be"
    if kind == "device":
        return _fake(*shape, dtype=dtype, device="cuda:1"), "is on cuda:1"
    if kind == "cpu":
        return _fake(*shape, dtype=dtype, device="cpu"), "must be a CUDA tensor"
    return _fake(*reversed(shape), dtype=dtype).permute(*reversed(range(len(shape)))), "must be contiguous"


BF16, F32 = torch.bfloat16, torch.float32
GIVEN = {  # the tensors that a call writes into: name of the argument -> (name in the error, shape, type)
    "forward": {"out": ("O", (B, HQ, S, D), BF16), "lse": ("LSE", (B, HQ, S), F32)},
    "backward": {"dq": ("dQ", (B, HQ, S, D), BF16), "dk": ("dK", (B, HKV, S, D), BF16), "dv": ("dV", (B, HKV, S, D), BF16)},
    "forward_varlen": {"out": ("O", (T, HQ, D), BF16), "lse": ("LSE", (HQ, T), F32)},
    "backward_varlen": {"dq": ("dQ", (T, HQ, D), BF16), "dk": ("dK", (T, HKV, D), BF16), "dv": ("dV", (T, HKV, D), BF16)},
}


@pytest.mark.parametrize("kind", ["shape", "dtype", "device", "cpu", "stride"])
@pytest.mark.parametrize("entry", GIVEN)
def test_given_outputs_are_checked(gqa_lib, entry, kind):
    """The library gets raw pointers: these checks keep its stores inside the tensors."""
    call = dict(_calls())[entry]
    for arg, (name, shape, dtype) in GIVEN[entry].items():
        t, words = _wrong(kind, shape, dtype)
        with pytest.raises(ValueError, match=f"^{name} {words}"):
            call(**{arg: t})


@pytest.mark.parametrize("entry", ["backward", "backward_varlen"])
def test_given_workspace_is_checked(gqa_lib, entry):
    u8 = torch.uint8
    for ws in (_fake(1 << 20, dtype=u8, device="cpu"), _fake(1 << 20, dtype=u8, device="cuda:1"),
               _fake(1 << 10, 1 << 10, dtype=u8).t()):
        with pytest.raises(ValueError, match="workspace must be contiguous memory on cuda:0"):
            dict(_calls())[entry](workspace=ws)
    with pytest.raises(TypeError, match="workspace must be a torch.Tensor"):
        dict(_calls())[entry](workspace=4096)
