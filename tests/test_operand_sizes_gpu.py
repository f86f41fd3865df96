"""Operands smaller than the kernels read are refused on the host, by the native and by the general path: the kernels take pointers and read
as many rows as the product has."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _t(*shape, dtype=torch.bfloat16):
    return torch.zeros(*shape, dtype=dtype, device="cuda")


CALLS = {
    "residual": lambda ops: ops.gemm_epilogue(_t(40, 64), _t(72, 64), residual=_t(1, 72)),
    "strided residual": lambda ops: ops.gemm_epilogue(_t(40, 64), _t(72, 64), residual=_t(39, 80)[:, :72]),
    "out": lambda ops: ops.gemm_epilogue(_t(40, 64), _t(72, 64), out=_t(39, 72)),
    "cos": lambda ops: ops.gemm_epilogue(_t(40, 64), _t(128, 64), "rope", rope=(_t(40, 16), _t(40, 32), 64, 128)),
    "sin": lambda ops: ops.gemm_epilogue(_t(40, 64), _t(128, 64), "rope", rope=(_t(40, 32, dtype=torch.float32), _t(39, 32, dtype=torch.float32), 64, 128)),
    "norm residual": lambda ops: ops.rms_rowstat(_t(40, 64), _t(39, 64)),
    "gamma": lambda ops: ops.prepare_weight([_t(8, 64)], _t(63)),
}


@pytest.mark.parametrize("native", [True, False])
@pytest.mark.parametrize("call", list(CALLS))
def test_too_small_is_refused(built_lib, monkeypatch, call, native):
    from heddle_b200 import _lib, ops

    if not native:
        monkeypatch.setattr(_lib, "native", None)
    with pytest.raises(ValueError):
        CALLS[call](ops)
    torch.cuda.synchronize()
    assert ops.status_word() == 0
