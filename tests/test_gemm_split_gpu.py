"""The split-K GEMM (clusters that share one tile's K range) against the oracle: single rows, tile tails in every dimension,
K ranges that do not divide evenly over a cluster, all epilogue classes, both weight layouts, batches."""
import pytest
import torch

from oracle import attention_oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops(built_lib):
    from heddle_b200 import ops as _ops

    prev = _ops.set_gemm_schedule("split")
    yield _ops
    _ops.set_gemm_schedule(prev)


def _check(ops, out, ref, dtype):
    torch.cuda.synchronize()
    assert ops.status_word() == 0
    # fp32 sums of K products rounded once to 16 bits: half an ulp of the largest value, plus the fp32 sum's own error
    scale = max(1.0, ref.float().abs().max().item())
    assert (out.float().cpu() - ref.float()).abs().max().item() <= (1e-2 if dtype == torch.bfloat16 else 2e-3) * scale


def _mk(M, N, K, dtype):
    g = torch.Generator().manual_seed(M + N + K)
    return torch.randn(M, K, generator=g).to(dtype), (torch.randn(N, K, generator=g) * 0.05).to(dtype), g


@pytest.mark.parametrize("M,N,K", [(1, 8, 8), (1, 4096, 4096), (7, 264, 72), (24, 512, 4096), (33, 200, 1000), (120, 1024, 2048),
                                   (128, 256, 512), (129, 776, 520), (300, 520, 4104), (64, 5000, 64)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_plain(ops, M, N, K, dtype):
    a, w, g = _mk(M, N, K, dtype)
    _check(ops, ops.gemm_epilogue(a.cuda(), w.cuda()), O.gemm_epilogue(a, w, "none"), dtype)
    bias, res, rs = torch.randn(N, generator=g).to(dtype), torch.randn(M, N, generator=g).to(dtype), torch.rand(M, generator=g) + 0.5
    out = ops.gemm_epilogue(a.cuda(), w.cuda(), "silu", bias=bias.cuda(), row_scale=rs.cuda(), residual=res.cuda())
    ref = O.epilogue_fp32(a.float() @ w.float().T * rs[:, None] + bias.float(), "silu") + res.float()
    _check(ops, out, ref, dtype)


@pytest.mark.parametrize("M,N_out,K", [(1, 8, 64), (24, 11008, 512), (100, 360, 4096), (130, 1000, 256)])
def test_swiglu(ops, M, N_out, K):
    dt = torch.bfloat16
    a, w, g = _mk(M, 2 * N_out, K, dt)
    bias, rs = torch.randn(2 * N_out, generator=g).to(dt), torch.rand(M, generator=g) + 0.5
    out = ops.gemm_epilogue(a.cuda(), w.cuda(), "swiglu", bias=bias.cuda(), row_scale=rs.cuda())
    y = a.float() @ w.float().T * rs[:, None] + bias.float()
    _check(ops, out, torch.nn.functional.silu(y[:, :N_out]) * y[:, N_out:], dt)


@pytest.mark.parametrize("hd,heads,rot,M,S", [(64, 6, 4, 50, 17), (128, 5, 3, 120, 120), (256, 2, 1, 9, 9), (128, 32, 32, 140, 70)])
def test_rope(ops, hd, heads, rot, M, S):
    dt, N, K = torch.float16, hd * heads, 1032
    a, w, g = _mk(M, N, K, dt)
    ang = torch.rand(S, hd // 2, generator=g) * 6
    out = ops.gemm_epilogue(a.cuda(), w.cuda(), "rope", rope=(ang.cos().cuda(), ang.sin().cuda(), hd, rot * hd))
    y = (a.float() @ w.float().T).reshape(M, heads, hd)
    c, s = (t[torch.arange(M) % S][:, None] for t in (ang.cos(), ang.sin()))
    x1, x2 = y[..., :hd // 2], y[..., hd // 2:]
    r = torch.cat([x1 * c - x2 * s, x2 * c + x1 * s], -1)
    r[:, rot:] = y[:, rot:]
    _check(ops, out, r.reshape(M, N), dt)


@pytest.mark.parametrize("B,M,N,K", [(3, 17, 200, 520), (2, 130, 72, 64), (5, 1, 64, 2048)])
@pytest.mark.parametrize("nk", [False, True])
def test_batched(ops, B, M, N, K, nk):
    dt = torch.bfloat16
    g = torch.Generator().manual_seed(B + M)
    a = torch.randn(B, M, K, generator=g).to(dt)
    b = (torch.randn(B, N, K, generator=g) * 0.05).to(dt).transpose(1, 2) if nk else (torch.randn(B, K, N, generator=g) * 0.05).to(dt)
    bc = b.transpose(1, 2).cuda().transpose(1, 2) if nk else b.cuda()
    _check(ops, ops.bmm(a.cuda(), bc), torch.matmul(a.float(), b.float()), dt)


def test_the_sum_over_the_cluster_has_one_order(ops):
    a, w, _ = _mk(48, 1024, 8192, torch.bfloat16)
    a, w = a.cuda(), w.cuda()
    first = ops.gemm_epilogue(a, w)
    for _ in range(5):
        assert torch.equal(ops.gemm_epilogue(a, w), first)


@pytest.mark.parametrize("schedule", ["single", "pair", "split"])
@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float16])
def test_16_bit_rope_tables_are_read_as_they_are(ops, schedule, dt):
    a, w, g = _mk(100, 512, 256, dt)
    a, w, ang = a.cuda(), w.cuda(), torch.rand(40, 64, generator=g) * 6
    cos, sin = ang.cos().to(dt).cuda(), ang.sin().to(dt).cuda()
    prev = ops.set_gemm_schedule(schedule)
    try:
        out = ops.gemm_epilogue(a, w, "rope", rope=(cos, sin, 128, 384))
        assert torch.equal(out, ops.gemm_epilogue(a, w, "rope", rope=(cos.float(), sin.float(), 128, 384)))
        # a table that is not 16-byte aligned is converted first
        off = torch.cat([cos.reshape(-1)[:1], cos.reshape(-1)])[1:].reshape(40, 64)
        assert torch.equal(out, ops.gemm_epilogue(a, w, "rope", rope=(off, sin, 128, 384)))
    finally:
        ops.set_gemm_schedule(prev)


@pytest.mark.parametrize("K", [72, 136, 184, 248, 264, 320, 520, 1000, 2040])
@pytest.mark.parametrize("w_layout", ["nk", "kn"])
def test_tail_of_k(ops, K, w_layout):
    """A K that is not a multiple of 64 is whole slabs, several to a stage, and a tail of its own.  What lies behind K in either operand
    is NaN: nothing of it may be read into a product."""
    dt, B, M, N = torch.bfloat16, 3, 40, 144
    g = torch.Generator().manual_seed(K)
    a = torch.full((B, M, K + 64), float("nan"), dtype=dt)
    a[:, :, :K] = torch.randn(B, M, K, generator=g).to(dt)
    w = torch.full((B, N, K + 64), float("nan"), dtype=dt)
    w[:, :, :K] = (torch.randn(B, N, K, generator=g) * 0.05).to(dt)
    ref = a[:, :, :K].float() @ w[:, :, :K].float().transpose(1, 2)
    if w_layout == "nk":
        b = w.cuda()[:, :, :K].transpose(1, 2)
    else:
        b = w.transpose(1, 2).contiguous().cuda()[:, :K]
    _check(ops, ops.bmm(a.cuda()[:, :, :K], b), ref, dt)
    if w_layout == "nk":
        one = ops.gemm_epilogue(a[0].cuda()[:, :K], w[0].cuda()[:, :K], "swiglu")
        _check(ops, one, torch.nn.functional.silu(ref[0][:, : N // 2]) * ref[0][:, N // 2:], dt)
