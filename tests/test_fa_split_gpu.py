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


# (B, Hq, Hkv, Sq, Skv, D, causal, dtype, runs on 148 SMs: 0 where items stay whole): one key; tile edges; runs longer and shorter
# than an item; a packed tile that is exactly full (16 x 8), just over (17 x 8: two row tiles, the second not full), one head per
# tile (65 x 2), 65 rows; more items than pipelines; one item over every SM; items cut into equal runs; runs that cross items (their
# second segment is a part too), with fewer items than runs and with more (whole items in the middle of a run), with up to 64 rows
# a tile and with more
CASES = [
    (1, 1, 1, 1, 1, 128, True, torch.bfloat16, 0),
    (2, 8, 1, 1, 128, 64, False, torch.float16, 0),
    (3, 4, 2, 1, 129, 128, False, torch.bfloat16, 0),
    (16, 16, 2, 1, 2001, 128, True, torch.bfloat16, 288),
    (2, 16, 2, 4, 1000, 64, True, torch.float16, 32),
    (1, 8, 1, 16, 777, 128, True, torch.float16, 0),
    (2, 8, 1, 17, 900, 128, True, torch.bfloat16, 0),
    (1, 4, 2, 65, 333, 64, False, torch.bfloat16, 0),
    (2, 3, 3, 128, 128, 128, True, torch.bfloat16, 0),
    (1, 6, 2, 127, 640, 64, True, torch.float16, 0),
    (40, 32, 32, 1, 300, 128, False, torch.bfloat16, 0),
    (1, 8, 1, 1, 40000, 128, False, torch.bfloat16, 296),
    (1, 17, 1, 4, 1265, 128, True, torch.bfloat16, 10),
    (1, 8, 1, 17, 1181, 64, False, torch.float16, 20),
    (19, 4, 4, 1, 777, 128, True, torch.bfloat16, 296),
    (5, 16, 16, 1, 777, 64, False, torch.float16, 296),
    (19, 16, 16, 1, 583, 128, False, torch.bfloat16, 296),
    (40, 8, 8, 2, 600, 64, True, torch.float16, 296),
    (19, 4, 1, 65, 2393, 128, True, torch.bfloat16, 296),
    (9, 34, 2, 65, 1326, 64, False, torch.float16, 296),
]


def _fa_args(q, k, v, out, layout="bhsd", causal=False):
    from heddle_b200 import _lib

    h, s = (1, 2) if layout == "bhsd" else (2, 1)
    a = _lib.FaArgs()
    a.q, a.k, a.v, a.o = q.data_ptr(), k.data_ptr(), v.data_ptr(), out.data_ptr()
    a.B, a.Hq, a.Hkv, a.Sq, a.Skv, a.D = q.shape[0], q.shape[h], k.shape[h], q.shape[s], k.shape[s], q.shape[3]
    for name, t in (("q", q), ("k", k), ("v", v), ("o", out)):
        for ax, d in zip("bhs", (0, h, s)):
            setattr(a, f"{name}_stride_{ax}", t.stride(d))
    a.causal, a.softmax_scale, a.dtype = int(causal), 1.0 / math.sqrt(q.shape[3]), _lib.HB_BF16 if q.dtype == torch.bfloat16 else _lib.HB_FP16
    a.stream = torch.cuda.current_stream().cuda_stream
    return a


@pytest.mark.parametrize("case", CASES, ids=lambda c: "x".join(str(x) for x in c[:6]))
@pytest.mark.parametrize("layout", ["bhsd", "bshd"])
def test_against_the_oracle(ops, built_lib, case, layout):
    B, Hq, Hkv, Sq, Skv, D, causal, dt, runs = case
    q, k, v = O.make_qkv(B, Hq, Hkv, Sq, Skv, D, seed=Skv + Sq, dtype=dt)
    k = (k.float() * torch.linspace(0.3, 2.0, Skv)[:, None]).to(dt)  # row maxima that grow: rescales inside a segment
    # every key tile has a column of its own in V (two or three share one where there are more tiles than columns): a part that is
    # lost, read twice or wrongly weighted shows there, however many parts there are
    v = (0.1 * v.float() + 4.0 * torch.nn.functional.one_hot(torch.arange(Skv) // 128 % D, D)).to(dt)
    ref, ref_lse = O.attention_eager(q, k, v, causal=causal)
    mass, _ = O.attention_eager(q, k, v.abs(), causal=causal)
    # the cache is a prefix of a longer buffer of NaN: nothing past Skv may be read into the result
    kc, vc = (torch.full((B, Hkv, Skv + 70, D), float("nan"), dtype=dt, device="cuda") for _ in range(2))
    kc[:, :, :Skv], vc[:, :, :Skv] = k.cuda(), v.cuda()
    qc, kc, vc = q.cuda(), kc[:, :, :Skv], vc[:, :, :Skv]
    if layout == "bshd":
        qc, kc, vc = (t.transpose(1, 2) for t in (qc.transpose(1, 2).contiguous().transpose(1, 2), kc, vc))
    out, lse = ops.fa_fwd(qc, kc, vc, causal=causal, layout=layout, return_lse=True)
    torch.cuda.synchronize()
    assert ops.status_word() == 0
    if torch.cuda.get_device_properties(0).multi_processor_count == 148:
        # two slots a run, each a tile's rows of O and LSE
        need, a = C.c_uint64(0), _fa_args(qc, kc, vc, out, layout, causal)
        assert built_lib.hb_fa_fwd_workspace(C.byref(a), C.byref(need)) == 0
        per_tile = max(1, 128 // Sq)
        tiles = -(-(Hq // Hkv) // per_tile)
        assert need.value == 2 * runs * -(-(Hq // Hkv) // tiles) * Sq * (D + 1) * 4
    out = out.transpose(1, 2) if layout == "bshd" else out
    # P and O are rounded to 16 bits once each, P against the weight of |v|; fp16 P below 2^-14 loses up to 2^-25 a key; fp32
    # scores, exponentials and sums are within 1e-4 of the weight
    unit = 2.0**-8 if dt == torch.bfloat16 else 2.0**-11
    tol = unit * (mass + ref.abs()) + 1e-4 * mass + (Skv * 2.0**-25 * 4.5 if dt == torch.float16 else 0.0)
    worst = ((out.float().cpu() - ref).abs() / tol).max().item()
    assert worst <= 1.0, worst
    assert (lse.cpu() - ref_lse).abs().max().item() <= 2e-3


def test_workspace_is_asked_for_and_checked(ops, built_lib):
    from heddle_b200 import _lib

    q = torch.randn(1, 8, 1, 128, device="cuda").to(torch.bfloat16)
    k = torch.randn(1, 1, 4096, 128, device="cuda").to(torch.bfloat16)
    out = torch.empty_like(q)
    a = _fa_args(q, k, k, out)
    need = C.c_uint64(0)
    assert built_lib.hb_fa_fwd_workspace(C.byref(a), C.byref(need)) == _lib.HB_OK and need.value > 0
    assert built_lib.hb_fa_fwd_ws(C.byref(a), None, 0) == _lib.HB_ERR_BAD_ARG
    ws = torch.empty(need.value, dtype=torch.uint8, device="cuda")
    assert built_lib.hb_fa_fwd_ws(C.byref(a), ws.data_ptr(), need.value - 4) == _lib.HB_ERR_BAD_ARG
    assert built_lib.hb_fa_fwd_ws(C.byref(a), ws.data_ptr(), need.value) == _lib.HB_OK
    assert torch.equal(out, ops.fa_fwd(q, k, k))


@pytest.mark.parametrize("group,Sq", [(1, 1), (7, 1), (2, 4), (9, 1), (3, 5), (8, 2), (17, 1)])
@pytest.mark.parametrize("Skv", [5, 130, 1100])
@pytest.mark.parametrize("D,dt", [(64, torch.float16), (128, torch.bfloat16)])
def test_few_rows(ops, group, Sq, Skv, D, dt):
    """Up to 8, up to 16 and more rows a tile, which three softmax forms turn over: masks inside a tile for every row, maxima that grow along the
    keys and rows whose maxima differ, partial segments and whole ones (two heads of keys on two pipelines, and twelve)."""
    for B, Hkv in ((1, 2), (6, 2)):
        q, k, v = O.make_qkv(B, group * Hkv, Hkv, Sq, Skv, D, seed=Skv + group, dtype=dt)
        q = (q.float() * torch.linspace(0.2, 3.0, group * Hkv)[:, None, None]).to(dt)
        k = (k.float() * torch.linspace(0.3, 2.0, Skv)[:, None]).to(dt)
        ref, ref_lse = O.attention_eager(q, k, v, causal=True)
        mass, _ = O.attention_eager(q, k, v.abs(), causal=True)
        out, lse = ops.fa_fwd(q.cuda(), k.cuda(), v.cuda(), causal=True, return_lse=True)
        torch.cuda.synchronize()
        assert ops.status_word() == 0
        # as in test_against_the_oracle
        unit = 2.0**-8 if dt == torch.bfloat16 else 2.0**-11
        tol = unit * (mass + ref.abs()) + 1e-4 * mass + (Skv * 2.0**-25 * 4.5 if dt == torch.float16 else 0.0)
        assert ((out.float().cpu() - ref).abs() / tol).max().item() <= 1.0
        assert (lse.cpu() - ref_lse).abs().max().item() <= 2e-3
