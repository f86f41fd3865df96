"""Kernels start while their predecessors still run and wait for them themselves (programmatic dependent launch).  Chains of
dependent calls over reused buffers must give the bits that the same calls give one at a time: eagerly, from a graph whose inputs
change between replays, and on two streams at once."""
import pytest
import torch

pytestmark = pytest.mark.gpu

H, HKV, S, D, CACHE = 8, 2, 48, 128, 4000
HIDDEN = H * D
NORM = (("load", "input", 0, 0.0), ("mul", "input", 0, 0.0), ("reduce_mean", None, 0, 0.0), ("load", "reduced", 0, 0.0),
        ("add", "imm", 0, 1e-5), ("rsqrt", None, 0, 0.0), ("mul", "input", 0, 0.0), ("store_out", None, 0, 0.0))
ADD_SILU = (("load", "input", 0, 0.0), ("silu", None, 0, 0.0), ("add", "input", 1, 0.0), ("store_out", None, 0, 0.0))


@pytest.fixture(scope="module")
def ops(built_lib):
    from heddle_b200 import ops as _ops

    return _ops


class Chain:
    """Every kind of launch in one chain: statistic, row softmax, compiled rowwise programs (both forms), split-K and persistent
    GEMMs, attention on split keys (with its merge), the general kernel, H2O score, the backward kernels (with
    the merge of grouped heads).  ``x``, ``y`` and ``a`` are written again while the call before may still read them."""

    def __init__(self, ops, seed):
        g = torch.Generator().manual_seed(seed)

        def mk(*shape, scale=1.0):
            return (torch.randn(*shape, generator=g) * scale).to(torch.bfloat16).cuda()

        self.ops, self.x0 = ops, mk(S, HIDDEN)
        self.w1, self.w2, self.wide = mk(HIDDEN, HIDDEN, scale=0.03), mk(HIDDEN, HIDDEN, scale=0.03), mk(6144, HIDDEN, scale=0.03)
        self.k, self.v = mk(1, HKV, CACHE, D), mk(1, HKV, CACHE, D)
        self.qkv = mk(1, H + 2 * HKV, 400, D)
        self.big = mk(2000, HIDDEN)
        self.x, self.y, self.a = (torch.empty(S, HIDDEN, dtype=torch.bfloat16, device="cuda") for _ in range(3))

    def steps(self):
        o, out = self.ops, []
        self.x.copy_(self.x0)
        for _ in range(2):
            def stat():
                self.rstd = o.rms_rowstat(self.x)[1]

            def project():
                o.gemm_epilogue(self.x, self.w1, "none", row_scale=self.rstd, out=self.y)

            def norm():
                self.n = o.rowwise_program(NORM, [self.y])

            def attend():
                q = self.n.view(1, S, H, D).transpose(1, 2)
                o.fa_fwd(q, self.k, self.v, causal=True, out=self.a.view(1, S, H, D).transpose(1, 2))

            def project_back():
                o.gemm_epilogue(self.a, self.w2, "none", residual=self.x, out=self.y)

            def mix():
                self.x.copy_(o.rowwise_program(ADD_SILU, [self.y, self.x]))

            def soften():
                self.p = o.row_softmax(self.x)

            def widen():
                self.u = o.gemm_epilogue(self.big + self.p[:1], self.wide)

            def train():
                q, k, v = self.qkv[:, :H], self.qkv[:, H:H + HKV], self.qkv[:, H + HKV:]
                self.f, lse = o.fa_fwd(q, k, v, causal=True, return_lse=True)
                self.score = o.h2o_score(q, k, lse)
                self.grads = o.fa_bwd(q, k, v, self.f, self.f, lse, causal=True)

            yield from (stat, project, norm, attend, project_back, mix, soften, widen, train)
            yield lambda: out.extend(t.clone() for t in (self.x, self.y, self.a, self.p, self.u, self.f, self.score, *self.grads))
        self.out = out

    def run(self, each=lambda: None):
        for step in self.steps():
            step()
            each()
        return self.out


def _same(got, want):
    return all(torch.equal(a, b) for a, b in zip(got, want, strict=True))


def _checked(chain):
    want = chain.run(torch.cuda.synchronize)
    torch.cuda.synchronize()
    assert all(torch.isfinite(t).all() for t in want)
    return want


def test_a_chain_gives_the_bits_of_single_calls(ops):
    chain = Chain(ops, 1)
    want = _checked(chain)
    for _ in range(20):
        got = chain.run()
        torch.cuda.synchronize()
        assert _same(got, want)
    assert ops.status_word() == 0


def test_a_captured_chain_follows_its_inputs(ops):
    chain = Chain(ops, 2)
    _checked(chain)
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        chain.run()
    torch.cuda.current_stream().wait_stream(stream)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = chain.run()
    for seed in (3, 4):
        other = Chain(ops, seed)
        for name in ("x0", "k", "v", "qkv", "big"):
            getattr(chain, name).copy_(getattr(other, name))
        for _ in range(3):  # back to back: a replay's first kernel follows the last one of the replay before
            graph.replay()
        torch.cuda.synchronize()
        kept = [t.clone() for t in got]
        assert _same(kept, _checked(chain))
    assert ops.status_word() == 0


def test_two_chains_on_two_streams(ops):
    chains = [Chain(ops, 5), Chain(ops, 6)]
    want = [_checked(c) for c in chains]
    streams = [torch.cuda.Stream() for _ in chains]
    torch.cuda.synchronize()
    for _ in range(5):
        got = []
        for chain, stream in zip(chains, streams):
            with torch.cuda.stream(stream):
                got.append(chain.run())
        torch.cuda.synchronize()
        assert all(_same(g, w) for g, w in zip(got, want))
    assert ops.status_word() == 0


def test_the_h2o_score_is_cleared_behind_its_last_reader(ops):
    """With the same storage in every call, the kernel of one call must stay between the reader of the call before and its own reader."""
    g = torch.Generator().manual_seed(7)
    qs, ks = ([torch.randn(1, 4, 300, 64, generator=g).to(torch.float16).cuda() for _ in range(4)] for _ in range(2))
    lse = [ops.fa_fwd(q, k, k, causal=True, return_lse=True)[1] for q, k in zip(qs, ks)]
    want = []
    for i in range(4):
        want.append(ops.h2o_score(qs[i], ks[i], lse[i]))
        torch.cuda.synchronize()
    where, got = set(), []
    for i in range(24):
        score = ops.h2o_score(qs[i % 4], ks[i % 4], lse[i % 4])
        where.add(score.data_ptr())
        got.append(score * 1.0)
        del score  # its storage goes to the next call
    torch.cuda.synchronize()
    assert len(where) < 24 and ops.status_word() == 0
    assert all(torch.equal(t, want[i % 4]) for i, t in enumerate(got))
