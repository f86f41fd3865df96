"""A single row may carry any row stride: a slice of a wider buffer keeps the buffer's, the transpose of a column has 1, and
``contiguous()`` returns both unchanged because a size of one does not count.  No second row is ever read."""
import pytest
import torch

pytestmark = pytest.mark.gpu

COLS = 4096


def _slice_of_a_wider_buffer(row):
    buf = torch.empty(3, COLS + 4, dtype=row.dtype, device="cuda")
    buf[0, :COLS] = row
    return buf[0:1, :COLS]


def _transposed_column(row):
    return row.reshape(COLS, 1).clone().t()


CALLS = {
    "gemm_epilogue": lambda ops, x: ops.gemm_epilogue(x, torch.linspace(-1, 1, 64 * COLS, device="cuda").reshape(64, COLS).to(x.dtype)),
    "row_softmax": lambda ops, x: ops.row_softmax(x, 0.5),
    "rowwise_program": lambda ops, x: ops.rowwise_program((("load", "input", 0, 0.0), ("silu", None, 0, 0.0), ("store_out", None, 0, 0.0)), [x]),
}


@pytest.mark.parametrize("view", [_slice_of_a_wider_buffer, _transposed_column])
@pytest.mark.parametrize("call", CALLS)
def test_any_row_stride_of_one_row_is_taken(built_lib, call, view):
    from heddle_b200 import ops

    row = torch.randn(COLS, generator=torch.Generator().manual_seed(3)).to(torch.bfloat16).cuda()
    x = view(row)
    assert x.shape == (1, COLS) and x.stride() != (COLS, 1)
    assert torch.equal(CALLS[call](ops, x), CALLS[call](ops, row[None].clone()))
