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


_PROBE = r"""
#include "heddle_b200/csrc/gemm_sm100.cuh"
using namespace hb;
template <int ACT>
__global__ void probe(const float* x, float* y, float* division, int n) {
  const int i = (blockIdx.x * 256 + threadIdx.x) * 8;
  if (i + 8 > n) return;
  float v[8];
  for (int e = 0; e < 8; ++e) v[e] = x[i + e];
  for (int e = 0; e < 8; ++e) division[i + e] = (ACT == kActSilu ? v[e] : 1.0f) * (1.0f / (1.0f + __expf(-v[e])));
  apply_act8<ACT>(v);
  for (int e = 0; e < 8; ++e) y[i + e] = v[e];
}
extern "C" int run(int act, const float* x, float* y, float* division, int n) {
  if (act == kActSilu) probe<kActSilu><<<(n / 8 + 255) / 256, 256>>>(x, y, division, n);
  else probe<kActSigmoid><<<(n / 8 + 255) / 256, 256>>>(x, y, division, n);
  return static_cast<int>(cudaDeviceSynchronize());
}
"""


def test_reciprocal_is_as_good_as_a_division(built_lib, tmp_path):
    """SiLU and sigmoid in fp32, in front of the rounding to 16 bits: no further from 64 bits than with an IEEE division."""
    import ctypes
    import subprocess
    from pathlib import Path

    from heddle_b200 import _build

    (tmp_path / "probe.cu").write_text(_PROBE)
    subprocess.run([_build._nvcc(), *_build.NVCC_FLAGS, "-shared", "-I", str(Path(__file__).resolve().parent.parent), str(tmp_path / "probe.cu"),
                    "-o", str(tmp_path / "probe.so")], check=True)
    run = ctypes.CDLL(str(tmp_path / "probe.so")).run
    run.argtypes = [ctypes.c_int, *[ctypes.c_void_p] * 3, ctypes.c_int]
    for lo, hi in ((-20.0, -4.0), (-4.0, -1.0), (-1.0, 1.0), (1.0, 4.0), (4.0, 20.0)):
        x = torch.linspace(lo, hi, 1 << 20, device="cuda") * 0.99997
        y, division = torch.full_like(x, float("nan")), torch.full_like(x, float("nan"))
        for act, ref in ((1, x.double() * torch.sigmoid(x.double())), (4, torch.sigmoid(x.double()))):
            assert run(act, x.data_ptr(), y.data_ptr(), division.data_ptr(), x.numel()) == 0
            rms = [(((t.double() - ref) / ref) ** 2).mean().sqrt().item() for t in (y, division)]
            # both round the exponential, the sum, the quotient and the product; a part in a hundred for where the samples lie
            assert rms[0] <= 1.01 * rms[1], (act, lo, hi, rms)
