"""Activation epilogues over the whole range of their argument, on every GEMM kernel: w is the identity, so the accumulator is exactly
the 16-bit input and the result is act(x) rounded once."""
import pytest
import torch

pytestmark = pytest.mark.gpu

_ACTS = {
    "silu": lambda x: x * torch.sigmoid(x),
    "relu": lambda x: x.clamp(min=0),
    "gelu_tanh": lambda x: x * torch.sigmoid(2 * 0.7978845608 * (x + 0.044715 * x**3)),
    "sigmoid": torch.sigmoid,
    "tanh": torch.tanh,
}


@pytest.mark.parametrize("schedule", ["single", "pair", "split"])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("act", list(_ACTS))
def test_tails(built_lib, act, dtype, schedule):
    from heddle_b200 import ops

    mag = torch.logspace(-4, 4.4, 200 * 72, dtype=torch.float64)
    x = torch.where(torch.arange(mag.numel()) % 2 == 0, mag, -mag)
    x[:2] = 0.0
    x = x.reshape(200, 72).to(dtype)
    prev = ops.set_gemm_schedule(schedule)
    try:
        out = ops.gemm_epilogue(x.cuda(), torch.eye(72, dtype=dtype).cuda(), act)
    finally:
        ops.set_gemm_schedule(prev)
    ref = _ACTS[act](x.double())
    # one rounding of the 16-bit type (half an ulp); the fp32 value in front of it is off by the argument's rounding,
    # |2u| 2^-24 <= 3e-6 relative where the result is a normal number, far below another half ulp
    ulp = 2.0**-7 if dtype == torch.bfloat16 else 2.0**-10
    tiny = torch.finfo(dtype).tiny
    err = (out.cpu().double() - ref).abs()
    worst = (err / (ref.abs() + tiny)).argmax()
    assert bool((err <= ulp * ref.abs() + tiny).all()), [t.flatten()[worst].item() for t in (x, out.cpu(), ref)]
