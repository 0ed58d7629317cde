"""Two-sided segments (upper bound ``diag``, lower bound ``lo``): the band plans against the mask they
stand for, on the CPU; the kernels against dense masked attention, on the GPU."""
import math

import pytest
import torch

from ultraattn_b200.ops import attention as A
from ultraattn_b200.ops import window as W

# (queries, keys, left, right, position of the first query, sinks): tile edges (127 ... 257), bands narrower
# than a tile, bounds that never bind, rows in front of / behind the point where the lower bound starts
CASES = [(1, 1, 0, 0, 0, 0), (700, 700, 290, 45, 0, 0), (513, 513, 0, 0, 0, 0), (640, 640, 127, 0, 0, 0),
         (640, 640, 128, 0, 0, 0), (900, 900, 900, 64, 0, 0), (900, 900, 257, 900, 0, 0), (300, 1000, 400, 0, 700, 0),
         (256, 600, 50, 400, 0, 0), (100, 700, 255, 33, 300, 0), (1, 900, 300, 0, 899, 0), (1000, 1000, 300, 0, 0, 4),
         (700, 700, 255, 0, 0, 256), (520, 520, 40, 0, 0, 41), (900, 900, 128, 30, 0, 16), (2500, 2500, 90, 0, 0, 5),
         (256, 256, 100, 0, 0, 3), (1300, 1300, 511, 0, 0, 1)]


def _mask(Sq, Skv, left, right, off, sink):
    r, c = torch.arange(Sq)[:, None] + off, torch.arange(Skv)[None, :]
    return ((c >= r - left) | (c < sink)) & (c <= r + right)


def _count(work, Sq, Skv):
    n = torch.zeros(Sq, Skv, dtype=torch.int32)
    for (q0, ql, k0, kl, sg) in work:
        m = A._visible(ql, kl, sg, "cpu")
        n[q0:q0 + ql, k0:k0 + kl] += 1 if m is None else m.int()
    return n


@pytest.mark.parametrize("Sq,Skv,left,right,off,sink", CASES)
def test_every_visible_pair_is_covered_once_and_tiles_are_visited(Sq, Skv, left, right, off, sink):
    rows, cols = W.band_rows_cols(Sq, Skv, left, right, off, sink=sink)
    want = _mask(Sq, Skv, left, right, off, sink).int()
    assert torch.equal(_count([(r.q_start, r.q_len, s.start, s.length, s) for r in rows for s in r.segs], Sq, Skv), want)
    assert torch.equal(_count([(s.start, s.length, c.kv_start, c.kv_len, s) for c in cols for s in c.segs], Sq, Skv), want)
    assert sorted(t for r in rows for t in range(r.q_start, r.q_start + r.q_len)) == list(range(Sq))
    writers = sorted(t for c in cols if c.g_slot == 0 for t in range(c.kv_start, c.kv_start + c.kv_len))
    assert writers == list(range(sink, Skv))          # one producer per gradient row; the sinks' share is added up
    # the tile range a row / key tile walks holds every visible pair (what lies outside is never computed)
    for r in rows:
        for s in r.segs:
            m = A._visible(r.q_len, s.length, s, "cpu")
            m = torch.ones(r.q_len, s.length, dtype=torch.bool) if m is None else m
            for r0 in range(0, r.q_len, 256):
                rows_here = min(256, r.q_len - r0)
                end = -(-s.length // 128)
                if s.causal:
                    last = r0 + rows_here - 1 + s.diag
                    end = 0 if last < 0 else min(end, last // 128 + 1)
                first = 0 if s.lo is None else min(end, max(0, r0 + s.lo) // 128)
                assert A._seg_tiles(s, r0, rows_here) == end - first
                seen = m[r0:r0 + rows_here].any(0).nonzero()
                if len(seen):
                    assert first * 128 <= int(seen[0]) and int(seen[-1]) < end * 128


def test_reference_of_two_sided_segments():
    """The fp32 restatement of both launches under the band plans is dense masked attention."""
    torch.manual_seed(0)
    Sq, Skv, left, right, off = 150, 400, 90, 20, 200
    q, k, v = torch.randn(1, Sq, 4, 16), torch.randn(1, Skv, 2, 16), torch.randn(1, Skv, 2, 16)
    rows, cols = W.band_rows_cols(Sq, Skv, left, right, off)
    o, lse = torch.empty_like(q), torch.empty(1, 4, Sq)
    A.attn_fwd([q], [k], [v], [(o, lse)], A.FwdPlan(rows))
    qg, kg, vg = (t.clone().requires_grad_() for t in (q, k, v))
    s = torch.einsum("bqhd,bkhd->bhqk", qg, kg.repeat_interleave(2, 2)) / 4
    s = s.masked_fill(~_mask(Sq, Skv, left, right, off, 0), float("-inf"))
    ref = torch.einsum("bhqk,bkhd->bqhd", torch.softmax(s, -1), vg.repeat_interleave(2, 2))
    g = torch.randn_like(ref)
    ref.backward(g)
    assert (o - ref).abs().max() < 2e-5
    dq, kv = torch.zeros_like(q), A.BwdKvOut(torch.zeros_like(k), torch.zeros_like(v))
    A.attn_bwd([A.BwdQSide(q, g, lse, (o * g).sum(-1).transpose(1, 2).contiguous(), dq)], [k], [v], [kv], A.BwdPlan(cols))
    for got, want in ((dq, qg.grad), (kv.dk, kg.grad), (kv.dv, vg.grad)):
        assert (got - want).abs().max() < 5e-5


@pytest.mark.gpu
@pytest.mark.parametrize("Sq,Skv,left,right,off,sink", CASES)
def test_band_on_the_kernels(Sq, Skv, left, right, off, sink, monkeypatch):
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA GPU")
    monkeypatch.setenv("UA_DEBUG_BOUNDS", "1")
    g = torch.Generator(device="cuda").manual_seed(Sq + left)
    mk = lambda s, h: torch.randn(2, s, h, 128, device="cuda", dtype=torch.bfloat16, generator=g)
    q, k, v, d_o = mk(Sq, 4), mk(Skv, 2), mk(Skv, 2), mk(Sq, 4)
    kw = dict(sink_tokens=sink) if sink else dict(q_offset=off)
    o, lse = W.window_forward(q, k, v, (left, right), False, **kw)
    got = W.window_backward(d_o, q, k, v, o, lse, (left, right), False, **kw)
    A.check_status()
    qd, kd, vd = (t.double().requires_grad_() for t in (q, k, v))
    s = torch.einsum("bqhd,bkhd->bhqk", qd, kd.repeat_interleave(2, 2)) / math.sqrt(128)
    s = s.masked_fill(~_mask(Sq, Skv, left, right, off, sink).cuda(), float("-inf"))
    ref = torch.einsum("bhqk,bkhd->bqhd", torch.softmax(s, -1), vd.repeat_interleave(2, 2))
    ref.backward(d_o.double())
    assert (lse - torch.logsumexp(s, -1)).abs().max() < 1e-3
    # bf16 keeps 8 bits: O, P and dS are rounded to 2^-9 each, independent errors; 8 of them is far outside
    for a, b in ((o, ref), (got[0], qd.grad), (got[1], kd.grad), (got[2], vd.grad)):
        assert (a.double() - b).norm() <= 8 * 2 ** -9 * b.norm() + 1e-3 * math.sqrt(b.numel()) * (b.norm() < 1e-2)
