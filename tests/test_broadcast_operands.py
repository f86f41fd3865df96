"""Operands whose rows or batches are one broadcast row or batch (a stride of 0).  What the wrappers hand to the library must stay
inside the tensor's storage; on the GPU the results equal those of a dense copy."""
import pytest
import torch

BF16 = torch.bfloat16


@pytest.fixture()
def handed_over(monkeypatch):
    """The arguments that the wrappers pass to the library, with CPU tensors in the place of CUDA ones."""
    from heddle_b200 import ops

    calls = []
    monkeypatch.setattr(ops, "_require_cuda", lambda *t: None)
    monkeypatch.setattr(ops, "_stream_ptr", lambda device: 0)
    monkeypatch.setattr(ops, "_call", lambda device, fn, *args: calls.append(args))
    return ops, calls


def test_row_softmax_reads_inside_a_broadcast_row(built_lib, handed_over):
    ops, calls = handed_over
    row = torch.randn(4096).to(BF16)
    ops.row_softmax(row.expand(16, 4096))
    x, _, rows, cols, ld = calls[0][:5]
    assert (rows, cols) == (16, 4096)
    assert ld == 4096 and x != row.data_ptr()  # a dense copy: 16 rows of 4096 do not fit behind the row itself


@pytest.mark.parametrize("which", ["a", "b"])
def test_bmm_reads_inside_a_broadcast_batch(built_lib, handed_over, which):
    ops, calls = handed_over
    a, b = torch.randn(1, 24, 64).to(BF16), torch.randn(1, 64, 40).to(BF16)
    wide = {"a": (a.expand(8, 24, 64), b.repeat(8, 1, 1)), "b": (a.repeat(8, 1, 1), b.expand(8, 64, 40))}[which]
    ops.bmm(*wide)
    g = calls[0][0]._obj
    assert g.batch == 8 and g.a_batch_stride == 24 * 64 and g.w_batch_stride == 64 * 40
    assert (g.a != a.data_ptr()) if which == "a" else (g.w != b.data_ptr())  # 0 would select densely packed batches


@pytest.mark.gpu
def test_results_equal_those_of_a_dense_copy(built_lib):
    from heddle_b200 import ops

    g = torch.Generator().manual_seed(4)
    x = torch.randn(4096, generator=g).to(BF16).cuda().expand(16, 4096)
    assert torch.equal(ops.row_softmax(x), ops.row_softmax(x.contiguous()))
    a, b = torch.randn(1, 24, 64, generator=g).to(BF16).cuda(), torch.randn(1, 64, 40, generator=g).to(BF16).cuda()
    for wide in ((a.expand(8, 24, 64), b.repeat(8, 1, 1)), (a.repeat(8, 1, 1), b.expand(8, 64, 40)),
                 (a.repeat(8, 1, 1), b.transpose(1, 2).contiguous().expand(8, 40, 64).transpose(1, 2))):
        assert torch.equal(ops.bmm(*wide), ops.bmm(*(t.contiguous() for t in wide)))
