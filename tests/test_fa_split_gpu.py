"""Attention with few query rows (the split-key kernel): row packing, segments that start or end inside an item, the merge of
partial results and the tails of the key tiles, against the oracle."""
import ctypes as C
import math

import pytest
import torch

from oracle import attention_oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops(built_lib):
    from heddle_b200 import ops as _ops

    return _ops


# (B, Hq, Hkv, Sq, Skv, D, causal, dtype): one key; tile edges; runs longer and shorter than an item; a packed tile that is
# exactly full (16 x 8), just over (17 x 8: two row tiles, the second not full), one head per tile (65 x 2), 65 rows;
# more items than pipelines; one item over every SM
CASES = [
    (1, 1, 1, 1, 1, 128, True, torch.bfloat16),
    (2, 8, 1, 1, 128, 64, False, torch.float16),
    (3, 4, 2, 1, 129, 128, False, torch.bfloat16),
    (16, 16, 2, 1, 2001, 128, True, torch.bfloat16),
    (2, 16, 2, 4, 1000, 64, True, torch.float16),
    (1, 8, 1, 16, 777, 128, True, torch.float16),
    (2, 8, 1, 17, 900, 128, True, torch.bfloat16),
    (1, 4, 2, 65, 333, 64, False, torch.bfloat16),
    (2, 3, 3, 128, 128, 128, True, torch.bfloat16),
    (1, 6, 2, 127, 640, 64, True, torch.float16),
    (40, 32, 32, 1, 300, 128, False, torch.bfloat16),
    (1, 8, 1, 1, 40000, 128, False, torch.bfloat16),
]


@pytest.mark.parametrize("case", CASES, ids=lambda c: "x".join(str(x) for x in c[:6]))
@pytest.mark.parametrize("layout", ["bhsd", "bshd"])
def test_against_the_oracle(ops, case, layout):
    B, Hq, Hkv, Sq, Skv, D, causal, dt = case
    q, k, v = O.make_qkv(B, Hq, Hkv, Sq, Skv, D, seed=Skv + Sq, dtype=dt)
    k = (k.float() * torch.linspace(0.3, 2.0, Skv)[:, None]).to(dt)  # row maxima that grow: rescales inside a segment
    ref, ref_lse = O.attention_eager(q, k, v, causal=causal)
    # the cache is a prefix of a longer buffer of NaN: nothing past Skv may be read into the result
    kc, vc = (torch.full((B, Hkv, Skv + 70, D), float("nan"), dtype=dt, device="cuda") for _ in range(2))
    kc[:, :, :Skv], vc[:, :, :Skv] = k.cuda(), v.cuda()
    qc, kc, vc = q.cuda(), kc[:, :, :Skv], vc[:, :, :Skv]
    if layout == "bshd":
        qc, kc, vc = (t.transpose(1, 2) for t in (qc.transpose(1, 2).contiguous().transpose(1, 2), kc, vc))
    out, lse = ops.fa_fwd(qc, kc, vc, causal=causal, layout=layout, return_lse=True)
    torch.cuda.synchronize()
    assert ops.status_word() == 0
    out = out.transpose(1, 2) if layout == "bshd" else out
    # P and O are rounded to 16 bits once each: 2 * 2^-9 (bf16) / 2^-12 (fp16) of values up to max |v|
    tol = (2e-2 if dt == torch.bfloat16 else 4e-3)
    assert (out.float().cpu() - ref.float()).abs().max().item() <= tol
    assert (lse.cpu() - ref_lse).abs().max().item() <= 2e-3


def test_workspace_is_asked_for_and_checked(ops, built_lib):
    from heddle_b200 import _lib

    q = torch.randn(1, 8, 1, 128, device="cuda").to(torch.bfloat16)
    k = torch.randn(1, 1, 4096, 128, device="cuda").to(torch.bfloat16)
    out = torch.empty_like(q)
    a = _lib.FaArgs()
    a.q, a.k, a.v, a.o = q.data_ptr(), k.data_ptr(), k.data_ptr(), out.data_ptr()
    a.B, a.Hq, a.Hkv, a.Sq, a.Skv, a.D = 1, 8, 1, 1, 4096, 128
    for name, t in (("q", q), ("k", k), ("v", k), ("o", out)):
        for ax, s in zip("bhs", t.stride()):
            setattr(a, f"{name}_stride_{ax}", s)
    a.softmax_scale, a.dtype = 1.0 / math.sqrt(128), _lib.HB_BF16
    a.stream = torch.cuda.current_stream().cuda_stream
    need = C.c_uint64(0)
    assert built_lib.hb_fa_fwd_workspace(C.byref(a), C.byref(need)) == _lib.HB_OK and need.value > 0
    assert built_lib.hb_fa_fwd_ws(C.byref(a), None, 0) == _lib.HB_ERR_BAD_ARG
    ws = torch.empty(need.value, dtype=torch.uint8, device="cuda")
    assert built_lib.hb_fa_fwd_ws(C.byref(a), ws.data_ptr(), need.value - 4) == _lib.HB_ERR_BAD_ARG
    assert built_lib.hb_fa_fwd_ws(C.byref(a), ws.data_ptr(), need.value) == _lib.HB_OK
    assert torch.equal(out, ops.fa_fwd(q, k, k))
