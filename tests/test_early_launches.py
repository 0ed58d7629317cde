"""Launches that are set up while the kernel before them finishes keep the order of a stream: passes that reuse and rewrite the
same buffers, one behind the other without a host synchronisation, against the same passes with one after every launch."""
import pytest
import torch

from ultraattn_b200.ops import attention as A
from ultraattn_b200.ops import elementwise as E

pytestmark = pytest.mark.gpu

# (batch, queries, keys, query heads, kv heads): few items, several items per CTA, split keys (with a merging launch behind)
SHAPES = [(1, 512, 512, 8, 8), (2, 1500, 1500, 16, 4), (2, 1, 5000, 8, 2), (1, 200, 4000, 8, 2)]
N = 12


class _Pass:
    """One forward and backward in buffers that stay; `load` rewrites the inputs with those of pass i."""

    def __init__(self, B, Sq, Skv, H, Hk, sync=False):
        if not torch.cuda.is_available():
            pytest.skip("needs a CUDA GPU")
        g = torch.Generator(device="cuda").manual_seed(Sq + Skv)
        mk = lambda s, h: torch.randn(N, B, s, h, 128, device="cuda", dtype=torch.bfloat16, generator=g)
        self.given = (mk(Sq, H), mk(Skv, Hk), mk(Skv, Hk), mk(Sq, H))
        self.q, self.k, self.v, self.d_o = (torch.zeros_like(t[0]) for t in self.given)
        self.o, self.dq = torch.zeros_like(self.q), torch.zeros_like(self.q)
        self.dk, self.dv = torch.zeros_like(self.k), torch.zeros_like(self.v)
        self.lse = torch.zeros(B, H, Sq, device="cuda")
        self.sync = torch.cuda.synchronize if sync else (lambda: None)
        A.status_buffer(self.q.device)

    def load(self, i):
        for dst, src in zip((self.q, self.k, self.v, self.d_o), self.given):
            dst.copy_(src[i])
            self.sync()

    def run(self, between=None):
        A.attn_fwd_dense(self.q, self.k, self.v, (self.o, self.lse), True)
        self.sync()
        if between is not None:
            between(self)
            self.sync()
        self.d = A.attn_bwd_local(self.q, self.k, self.v, self.o, self.lse, self.d_o, self.dq, self.dk, self.dv, None, 2)
        self.sync()

    def results(self):
        return [t.clone() for t in (self.o, self.lse, self.d, self.dk, self.dv, self.dq)]


def _same(got, want):
    for i, (a, b) in enumerate(zip(got, want)):
        *exact, (dq, dq0) = zip(a, b)
        assert all(torch.equal(x, y) for x, y in exact), i
        assert (dq.float() - dq0.float()).norm() <= 2 ** -8 * dq0.float().norm(), i          # (summed in arrival order, then rounded)


def _passes(shape, sync, between=None):
    p = _Pass(*shape, sync=sync)
    out = []
    for i in range(N):
        p.load(i)
        p.run(between)
        out.append(p.results())
    A.check_status()
    return out


@pytest.mark.parametrize("shape", SHAPES)
def test_buffers_rewritten_by_the_next_pass(shape):
    _same(_passes(shape, False), _passes(shape, True))


@pytest.mark.parametrize("shape", SHAPES)
def test_other_kernels_between_the_launches(shape):
    """A plain kernel of the library and one of PyTorch read what the forward wrote and change what the backward reads."""
    def between(p):
        E.lse_merge([(p.o[0], p.lse[0]), (p.q[0], torch.zeros_like(p.lse[0]))], (p.o[0], p.lse[0]))
        p.d_o.mul_(0.5)

    _same(_passes(shape, False, between), _passes(shape, True, between))


@pytest.mark.parametrize("shape", SHAPES)
def test_captured_passes_replayed_back_to_back(shape):
    """Two passes in one graph (the second one rewrites the first one's results), replayed with other inputs each time."""
    p = _Pass(*shape)
    p.load(0)
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        p.run()
    torch.cuda.current_stream().wait_stream(stream)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        p.run()
        p.run()
    got = []
    for i in range(N):
        p.load(i)
        graph.replay()
        got.append(p.results())
    A.check_status()
    del graph
    _same(got, _passes(shape, True))
