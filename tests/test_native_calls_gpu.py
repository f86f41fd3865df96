"""The native host path of the tensor-level calls against the general path of ops.py, over the forms that either takes: the same values,
shapes and strides, the same refusals; and that it stands back where a mode, a subclass or a transform is in force."""
import pytest
import torch
from torch.utils._python_dispatch import TorchDispatchMode

pytestmark = pytest.mark.gpu

BF, HF, F32 = torch.bfloat16, torch.float16, torch.float32
NORM = (("load", "input", 0, 0.0), ("reduce_mean", None, 0, 0.0), ("sub", "reduced", 0, 0.0), ("mul", "imm", 0, 0.5), ("store_out", None, 0, 0.0))
AFFINE = [("load", "input", 0, 0.0), ("mul", "rowvec", 0, 0.0), ("add", "rowscalar", 0, 0.0), ("store_out", None, 0, 0.0),
          ("add", "input", 1, 0.0), ("store_out", None, 1, 0.0)]


def R(*shape, dtype=BF, seed=0):
    return torch.randn(*shape, generator=torch.Generator().manual_seed(seed + sum(shape))).to(dtype).cuda()


def _heads(layout, B, H, S, D, dtype=BF, seed=0):
    return R(B, H, S, D, dtype=dtype, seed=seed) if layout == "bhsd" else R(B, S, H, D, dtype=dtype, seed=seed)


def _fa(layout, B, Hq, Hkv, Sq, Skv, D, dtype=BF, view=None, **kw):
    def call(ops):
        q, k, v = _heads(layout, B, Hq, Sq, D, dtype), _heads(layout, B, Hkv, Skv, D, dtype, 1), _heads(layout, B, Hkv, Skv, D, dtype, 2)
        if view is not None:
            q, k, v = view(q), view(k), view(v)
        return ops.fa_fwd(q, k, v, layout=layout, **kw)
    return call


def _fa8(**kw):
    def call(ops):
        q, k, v = (R(1, 2, 200, 128, dtype=F32, seed=i).to(torch.float8_e4m3fn) for i in range(3))
        return ops.fa_fwd(q, k, v, scales=(1.0, 0.5, 2.0), **kw)
    return call


def _fa_out(ops):
    q = R(2, 4, 150, 64)
    out = torch.empty(2, 150, 4, 64, dtype=BF, device="cuda").transpose(1, 2)
    r = ops.fa_fwd(q, q, q, causal=True, out=out)
    assert r is out
    return r


def _bwd(layout, Hq, Hkv, S, D, lse_dtype=F32, **kw):
    def call(ops):
        q, k, v, g = _heads(layout, 2, Hq, S, D), _heads(layout, 2, Hkv, S, D, seed=1), _heads(layout, 2, Hkv, S, D, seed=2), _heads(layout, 2, Hq, S, D, seed=3)
        o, lse = ops.fa_fwd(q, k, v, layout=layout, return_lse=True, **kw)
        return ops.fa_bwd(q, k, v, o, g, lse.to(lse_dtype), layout=layout, **kw)
    return call


def _h2o(ops):
    q, k = R(1, 4, 77, 64), R(1, 2, 77, 64, seed=1)
    _, lse = ops.fa_fwd(q, k, k, causal=True, return_lse=True)
    return ops.h2o_score(q, k, lse, softmax_scale=0.125)


def _rope(dtype):
    def call(ops):
        cos, sin = R(30, 64, dtype=dtype), R(30, 64, dtype=dtype, seed=1)
        return ops.gemm_epilogue(R(2, 30, 72), R(384, 72), "rope", rope=(cos, sin, 128, 256))
    return call


FORMS = {
    "fa bhsd": _fa("bhsd", 2, 4, 2, 300, 300, 128, causal=True),
    "fa bshd lse scale": _fa("bshd", 1, 3, 3, 129, 200, 64, HF, causal=True, return_lse=True, softmax_scale=0.2),
    "fa few rows": _fa("bhsd", 3, 8, 2, 1, 777, 128, causal=True),
    "fa inner stride": _fa("bhsd", 1, 2, 2, 140, 140, 64, view=lambda t: t.transpose(2, 3).contiguous().transpose(2, 3)),
    "fa prefix": _fa("bhsd", 2, 2, 2, 160, 160, 64, view=lambda t: torch.cat([t, t], 2)[:, :, :160]),
    "fa fp8": _fa8(causal=True, return_lse=True),
    "fa out": _fa_out,
    "fa empty": _fa("bhsd", 0, 2, 2, 140, 140, 64),
    "fa bad heads": _fa("bhsd", 1, 3, 2, 140, 140, 64),
    "fa bad layout": lambda ops: ops.fa_fwd(R(1, 1, 8, 64), R(1, 1, 8, 64), R(1, 1, 8, 64), layout="sbhd"),
    "fa bad dims": lambda ops: ops.fa_fwd(R(1, 8, 64), R(1, 8, 64), R(1, 8, 64)),
    "fa mixed types": lambda ops: ops.fa_fwd(R(1, 1, 8, 64), R(1, 1, 8, 64, dtype=HF), R(1, 1, 8, 64)),
    "fa misaligned": lambda ops: ops.fa_fwd(R(1 * 150 * 64 + 1)[1:].view(1, 1, 150, 64), R(1, 1, 150, 64), R(1, 1, 150, 64)),
    "bwd": _bwd("bhsd", 2, 2, 130, 64, causal=True),
    "bwd grouped bshd": _bwd("bshd", 4, 1, 200, 128, softmax_scale=0.1),
    "bwd lse 64 bits": _bwd("bhsd", 2, 2, 130, 64, torch.float64),
    "h2o": _h2o,
    "gemm": lambda ops: ops.gemm_epilogue(R(3, 5, 64), R(40, 64), "silu", bias=R(40), row_scale=R(3, 5, dtype=F32), residual=R(3, 5, 40)),
    "gemm swiglu": lambda ops: ops.gemm_epilogue(R(70, 64), R(48, 64), "swiglu", row_scale=R(70, dtype=F32)),
    "gemm 1-d": lambda ops: ops.gemm_epilogue(R(64), R(40, 64)),
    "gemm one row any stride": lambda ops: ops.gemm_epilogue(R(3, 72)[1:2, :64], R(40, 64)),
    "gemm column slice": lambda ops: ops.gemm_epilogue(R(9, 80)[:, 8:72], R(40, 64)),
    "gemm transposed": lambda ops: ops.gemm_epilogue(R(64, 9).t(), R(64, 40).t()),
    "gemm 16-bit row scale": lambda ops: ops.gemm_epilogue(R(9, 64), R(40, 64), row_scale=R(9)),
    "gemm fp32 bias": lambda ops: ops.gemm_epilogue(R(9, 64), R(40, 64), bias=R(40, dtype=F32)),
    "gemm out": lambda ops: ops.gemm_epilogue(R(9, 64), R(40, 64), out=torch.empty(9, 40, dtype=BF, device="cuda")),
    "gemm no rows": lambda ops: ops.gemm_epilogue(R(0, 64), R(40, 64)),
    "gemm K % 8": lambda ops: ops.gemm_epilogue(R(9, 60), R(40, 60)),
    "gemm odd swiglu": lambda ops: ops.gemm_epilogue(R(9, 64), R(41, 64), "swiglu"),
    "gemm wrong K": lambda ops: ops.gemm_epilogue(R(9, 64), R(40, 72)),
    "gemm bad bias": lambda ops: ops.gemm_epilogue(R(9, 64), R(40, 64), bias=R(48)),
    "gemm unknown": lambda ops: ops.gemm_epilogue(R(9, 64), R(40, 64), "softsign"),
    "rope 16-bit tables": _rope(BF),
    "rope fp32 tables": _rope(F32),
    "rope 64-bit tables": _rope(torch.float64),
    "bmm kn": lambda ops: ops.bmm(R(3, 20, 64), R(3, 64, 40)),
    "bmm nk": lambda ops: ops.bmm(R(3, 20, 64), R(3, 40, 64).transpose(1, 2), "relu"),
    "bmm broadcast": lambda ops: ops.bmm(R(1, 20, 64).expand(3, -1, -1), R(1, 64, 40).expand(3, -1, -1)),
    "bmm odd stride": lambda ops: ops.bmm(R(3, 20, 65)[:, :, :64], R(3, 64, 41)[:, :, :40]),
    "bmm bias": lambda ops: ops.bmm(R(3, 20, 64), R(3, 64, 40), bias=R(40)),
    "bmm no rows": lambda ops: ops.bmm(R(3, 0, 64), R(3, 64, 40)),
    "bmm N % 8": lambda ops: ops.bmm(R(3, 20, 64), R(3, 64, 41)),
    "rowstat": lambda ops: ops.rms_rowstat(R(2, 9, 72)),
    "rowstat strided": lambda ops: ops.rms_rowstat(R(9, 80)[:, :72]),
    "rowstat residual": lambda ops: ops.rms_rowstat(R(9, 72), R(9, 72, seed=1)),
    "rowstat odd": lambda ops: ops.rms_rowstat(R(9, 70)),
    "softmax": lambda ops: ops.row_softmax(R(4, 9, 72), 0.3),
    "softmax rows apart": lambda ops: ops.row_softmax(R(9, 80)[:, :72]),
    "softmax broadcast": lambda ops: ops.row_softmax(R(1, 72).expand(9, -1)),
    "softmax fp32": lambda ops: ops.row_softmax(R(9, 72, dtype=F32)),
    "softmax odd": lambda ops: ops.row_softmax(R(9, 70)),
    "rowwise": lambda ops: ops.rowwise_program(NORM, [R(2, 9, 72)]),
    "rowwise operands": lambda ops: ops.rowwise_program(AFFINE, (R(9, 72), R(9, 72, seed=1)), [R(72)], [R(9, 1, dtype=F32)], 2),
    "rowwise converted": lambda ops: ops.rowwise_program(AFFINE, (R(9, 72), R(9, 72, seed=1)), [R(72, dtype=F32)], [R(9, 1)], 2, "interpret"),
    "rowwise strided": lambda ops: ops.rowwise_program(NORM, [R(9, 73)[:, :72]]),
    "rowwise no inputs": lambda ops: ops.rowwise_program(NORM, []),
    "rowwise unknown op": lambda ops: ops.rowwise_program((("load", "input", 0, 0.0), ("cosh", None, 0, 0.0), ("store_out", None, 0, 0.0)), [R(9, 72)]),
    "rowwise unlike shapes": lambda ops: ops.rowwise_program(AFFINE[:1], (R(9, 72), R(8, 72))),
}
# forms whose last call the general path has to take (it converts, copies or refuses before the library is asked)
GENERAL = {"fa inner stride", "fa empty", "fa bad layout", "fa bad dims", "fa mixed types", "bwd lse 64 bits", "gemm transposed",
           "gemm 16-bit row scale", "gemm fp32 bias", "gemm out", "gemm no rows", "gemm wrong K", "gemm bad bias", "gemm unknown",
           "rope 64-bit tables", "bmm broadcast", "bmm odd stride", "bmm bias", "bmm no rows", "bmm N % 8", "rowstat strided", "rowstat residual",
           "softmax broadcast", "softmax fp32", "softmax odd", "rowwise converted", "rowwise strided", "rowwise no inputs", "rowwise unknown op", "rowwise unlike shapes"}


class _Spy:
    """The native module, noting whether the last call was taken."""

    def __init__(self, native):
        self._native, self.taken = native, None

    def __getattr__(self, name):
        fn = getattr(self._native, name)

        def call(*args):
            self.taken = False
            r = fn(*args)  # a refusal of the library's own leaves `taken` as it is
            self.taken = r is not NotImplemented
            return r
        return call


def _outcome(call, ops):
    try:
        r = call(ops)
    except Exception as e:  # noqa: BLE001  (a refusal is an outcome)
        return type(e), str(e)
    torch.cuda.synchronize()
    return r if isinstance(r, tuple) else (r,)


@pytest.mark.parametrize("form", list(FORMS))
def test_same_as_the_general_path(built_lib, monkeypatch, form):
    from heddle_b200 import _lib, ops

    spy = _Spy(_lib.native)
    monkeypatch.setattr(_lib, "native", spy)
    got = _outcome(FORMS[form], ops)
    refused = isinstance(got[0], type)
    if not refused:
        assert bool(spy.taken) == (form not in GENERAL)
    monkeypatch.setattr(_lib, "native", None)
    ref = _outcome(FORMS[form], ops)
    assert len(got) == len(ref)
    for a, b in zip(got, ref):
        if isinstance(b, torch.Tensor):
            assert a.dtype == b.dtype and a.shape == b.shape and a.stride() == b.stride() and a.device == b.device
            assert torch.equal(a.float(), b.float())
        else:
            assert a == b
    assert ops.status_word() == 0


def test_stands_back(built_lib):
    from heddle_b200 import _lib

    class Sub(torch.Tensor):
        pass

    class Mode(TorchDispatchMode):
        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            return func(*args, **(kwargs or {}))

    x = R(8, 64)
    native = _lib.native
    assert isinstance(native.row_softmax(x, 1.0), torch.Tensor)
    assert native.row_softmax(x.as_subclass(Sub), 1.0) is NotImplemented
    with Mode():
        assert native.row_softmax(x, 1.0) is NotImplemented
    seen = []

    def inner(t):
        seen.append(native.row_softmax(t, 1.0))
        return t

    torch.func.vmap(inner)(x)
    torch.func.grad(lambda t: inner(t).float().sum())(x)
    torch.func.functionalize(inner)(x)
    assert all(r is NotImplemented for r in seen) and len(seen) == 3


def test_tensors_state(built_lib):
    from heddle_b200 import _lib

    state = _lib.native.tensors_state
    t, u = torch.zeros(4, 6), torch.zeros(4, 6)
    a = state((t, u))
    assert a == state((t, u)) and a != state((u, t)) and a != state((t,))
    assert state((t.t(),)) != state((t,)) and state((t.view(6, 4),)) != state((t,)) and state((t.view(torch.int32),)) != state((t,))
    t.add_(1)
    assert state((t, u)) != a
    with torch.inference_mode():
        assert isinstance(state((torch.zeros(3),)), bytes)


def test_rowwise_reads_no_list_that_an_operand_may_change(built_lib):
    """An immediate's __float__ is other people's code: it is left to the general path, which holds what it reads."""
    from heddle_b200 import _lib, ops

    x = R(8, 64)
    program = [("load", "input", 0, 0.0), ("mul", "imm", 0, 0.5), ("store_out", None, 0, 0.0)]
    ref = ops.rowwise_program(program, [x])

    class Half:
        asked = 0

        def __float__(self):
            Half.asked += 1
            return 0.5

    odd = [program[0], ("mul", "imm", 0, Half()), program[2]]
    assert _lib.native.rowwise_program(odd, [x], (), (), 1, _lib.ROWWISE_AUTO) is NotImplemented and Half.asked == 0
    assert torch.equal(ops.rowwise_program(odd, [x]), ref)
