"""Compiled row reductions that keep a row's inputs in registers between the passes: every loop length (1 to 8 iterations and
the uncached form), widths just over and under them, one to three inputs, an input that only the last pass reads."""
import pytest
import torch

from oracle.program_oracle import run_program

pytestmark = pytest.mark.gpu

NORM = (("load", "input", 0, 0.0), ("reduce_mean", None, 0, 0.0), ("sub", "reduced", 0, 0.0), ("store_tmp", None, 0, 0.0),
        ("mul", "tmp", 0, 0.0), ("reduce_mean", None, 1, 0.0), ("load", "reduced", 1, 0.0), ("add", "imm", 0, 1e-5),
        ("rsqrt", None, 0, 0.0), ("mul", "tmp", 0, 0.0), ("store_out", None, 0, 0.0))
# (x + y) scaled by its row maximum, times z in the last pass only
SCALED = (("load", "input", 0, 0.0), ("add", "input", 1, 0.0), ("store_tmp", None, 0, 0.0), ("reduce_max", None, 0, 0.0),
          ("load", "tmp", 0, 0.0), ("div", "reduced", 0, 0.0), ("mul", "input", 2, 0.0), ("store_out", None, 0, 0.0))


@pytest.mark.parametrize("cols", [8, 248, 512, 520, 1024, 1032, 2048, 2056, 4096, 4104, 8192, 8200, 16384])
@pytest.mark.parametrize("program,n_in", [(NORM, 1), (SCALED, 3)], ids=["norm", "scaled"])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_against_the_oracle(built_lib, cols, program, n_in, dtype):
    from heddle_b200 import ops

    if not built_lib.hb_rowwise_compiler_available():
        pytest.skip("libnvrtc cannot be loaded in this process")
    g = torch.Generator().manual_seed(cols)
    xs = [(torch.randn(5, cols, generator=g) + 0.25).to(dtype) for _ in range(n_in)]
    out = ops.rowwise_program(program, [x.cuda() for x in xs], mode="compiled")
    ref = run_program(program, xs).float()
    # the oracle's result is rounded to 16 bits as well, so a value next to a tie may differ by one unit in the last place: at
    # most 2^-7 (bf16) or 2^-10 (fp16) of it; the fp32 reductions themselves are within 1e-5
    tol = (2.0**-7 if dtype == torch.bfloat16 else 2.0**-10) * ref.abs() + 1e-5
    assert ((out.float().cpu() - ref).abs() <= tol).all()


def test_a_width_met_first_inside_a_capture(built_lib):
    """Each power of two of the width has a kernel of its own, so a program that has run may still compile inside a capture."""
    from heddle_b200 import ops

    if not built_lib.hb_rowwise_compiler_available():
        pytest.skip("libnvrtc cannot be loaded in this process")
    program = (("load", "input", 0, 0.0), ("mul", "imm", 0, 1.37), *NORM[1:])  # no other test's program
    x = {cols: torch.randn(6, cols, generator=torch.Generator().manual_seed(cols)).to(torch.bfloat16).cuda() for cols in (2048, 16384)}
    ops.rowwise_program(program, [x[2048]], mode="compiled")
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = ops.rowwise_program(program, [x[16384]], mode="compiled")
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(out, ops.rowwise_program(program, [x[16384]], mode="compiled"))
