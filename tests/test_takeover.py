"""Launches with several work items per CTA (a CTA that is done takes over one that has not started) against
float64 attention: barrier phases, item slots and buffers have to carry over from item to item."""
import math

import pytest
import torch

from ultraattn_b200.ops import attention as A

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _needs_gpu():
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA GPU")


def _rand(seed, *shapes):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return [torch.randn(*s, 128, device="cuda", dtype=torch.bfloat16, generator=g) for s in shapes]


def _attend(q, k, v, seen):
    """(o, lse) in the type of the inputs; rows that see nothing: zeros and -inf."""
    s = torch.einsum("bqhd,bkhd->bhqk", q, k.repeat_interleave(q.shape[2] // k.shape[2], 2)) / math.sqrt(128)
    some = seen.any(-1)
    lse = torch.logsumexp(s.detach().masked_fill(~seen, float("-inf")), -1)
    p = torch.softmax(s.masked_fill(~seen, -1e30), -1) * some[:, None]
    return torch.einsum("bhqk,bkhd->bqhd", p, v.repeat_interleave(q.shape[2] // v.shape[2], 2)), lse


def _close(got, want, parts=4):
    # O: P and O are rounded to bf16 (2^-9 each); gradients: P, dS and the result. 4 resp. 8 of them is far outside
    return (got.double() - want).norm() <= parts * 2 ** -9 * want.norm()


# (batch, queries, keys, query heads, kv heads, key splits): few rows, five key tiles. As many splits as
# tiles: one tile per item, the second half of the warps never has one; 4: items of one and two tiles in turn
@pytest.mark.parametrize("B,Sq,Skv,H,Hk,n_split", [(64, 1, 520, 8, 8, 5), (64, 1, 520, 16, 8, 4), (48, 40, 640, 8, 8, 5),
                                                   (48, 33, 640, 16, 8, 3), (64, 2, 520, 16, 8, 0), (96, 1, 600, 32, 8, 1)])
def test_few_rows_many_items(B, Sq, Skv, H, Hk, n_split):
    q, k, v = _rand(Skv + B, (B, Sq, H), (B, Skv, Hk), (B, Skv, Hk))
    for _ in range(3):
        o, lse = torch.full_like(q, 7.0), torch.full((B, H, Sq), 7.0, device="cuda")
        A.attn_fwd_dense(q, k, v, (o, lse), True, None, n_split)
    A.check_status()
    r, c = torch.arange(Sq, device="cuda")[:, None], torch.arange(Skv, device="cuda")[None]
    ref, ref_lse = _attend(q.double(), k.double(), v.double(), c <= r + Skv - Sq)
    assert (lse - ref_lse).abs().max() < 1e-3
    assert _close(o, ref)


def _check(o, lse, grads, q, k, v, d_o, seen):
    A.check_status()
    ref = [t.detach().double().requires_grad_() for t in (q, k, v)]
    want, want_lse = _attend(*ref, seen)
    want.backward(d_o.double())
    some = torch.isfinite(want_lse)
    if lse is not None:
        assert torch.equal(torch.isfinite(lse), some) and (lse[some] - want_lse[some]).abs().max() < 1e-3
    assert _close(o.detach(), want.detach()) and (o.transpose(1, 2)[~some] == 0).all()
    # queries that see nothing and keys that nothing sees: exactly zero
    for got, t, used in zip(grads, ref, (seen.any(1), seen.any(0), seen.any(0))):
        assert _close(got, t.grad, 8) and (got[:, ~used] == 0).all()


def _index(S):
    return torch.arange(S, device="cuda")[:, None], torch.arange(S, device="cuda")[None]


@pytest.mark.parametrize("H,Hk", [(16, 16), (32, 8)])
def test_documents(H, Hk):
    from ultraattn_b200.api import varlen_attention
    cu = [0, 700, 701, 1500, 1503, 2500]
    q, k, v, d_o = _rand(1, (1, 2500, H), (1, 2500, Hk), (1, 2500, Hk), (1, 2500, H))
    q, k, v = (t.requires_grad_() for t in (q, k, v))
    o = varlen_attention(q, k, v, cu)
    grads = torch.autograd.grad(o, (q, k, v), d_o)
    r, c = _index(2500)
    doc = torch.bucketize(torch.arange(2500, device="cuda"), torch.tensor(cu[1:], device="cuda"), right=True)
    _check(o, None, grads, q, k, v, d_o, (c <= r) & (doc[:, None] == doc[None]))


@pytest.mark.parametrize("left,sink", [(300, 0), (100, 4)])
def test_windows(left, sink):
    from ultraattn_b200.ops.window import window_backward, window_forward
    S, H, Hk = 2600, 32, 16
    q, k, v, d_o = _rand(2, (1, S, H), (1, S, Hk), (1, S, Hk), (1, S, H))
    o, lse = window_forward(q, k, v, (left, 0), True, sink_tokens=sink)
    grads = window_backward(d_o, q, k, v, o, lse, (left, 0), True, sink_tokens=sink)
    r, c = _index(S)
    _check(o, lse, grads, q, k, v, d_o, (c <= r) & ((c >= r - left) | (c < sink)))


def test_block_tables_with_empty_rows_and_columns():
    import numpy as np
    from ultraattn_b200.api import local_backward
    B, S, H, blk = 2, 2048, 16, 256
    table = np.random.default_rng(0).integers(0, 3, (8, 8))
    table[[2, 7]] = 0
    table[:, [0, 5]] = 0
    q, k, v, d_o = _rand(3, (B, S, H), (B, S, H), (B, S, H), (B, S, H))
    o, lse = torch.full_like(q, 7.0), torch.full((B, H, S), 7.0, device="cuda")
    A.attn_fwd([q], [k], [v], [(o, lse)], A.FwdPlan(A.rows_from_block_table(table, blk), "cuda"))
    grads = local_backward(q, k, v, o, lse, d_o, A.BwdPlan(A.cols_from_block_table(table, blk), "cuda"))
    r, c = _index(S)
    kind = torch.from_numpy(table).cuda()[r // blk, c // blk]
    _check(o, lse, grads, q, k, v, d_o, (kind == 1) | ((kind == 2) & (c % blk <= r % blk)))


@pytest.mark.parametrize("B,Sq,Skv,H,Hk,causal", [(1, 2500, 2500, 16, 16, True), (8, 700, 300, 16, 16, True), (2, 1100, 1100, 32, 8, False)])
def test_dense(B, Sq, Skv, H, Hk, causal):
    """(700 queries, 300 keys: the first row tile sees nothing)"""
    from ultraattn_b200.api import local_backward
    q, k, v, d_o = _rand(4, (B, Sq, H), (B, Skv, Hk), (B, Skv, Hk), (B, Sq, H))
    o, lse = torch.full_like(q, 7.0), torch.full((B, H, Sq), 7.0, device="cuda")
    A.attn_fwd_dense(q, k, v, (o, lse), causal)
    grads = local_backward(q, k, v, o, lse, d_o, None, None, 2 if causal else 1)
    r, c = torch.arange(Sq, device="cuda")[:, None], torch.arange(Skv, device="cuda")[None]
    _check(o, lse, grads, q, k, v, d_o, (c <= r + Skv - Sq) if causal else torch.ones(Sq, Skv, dtype=torch.bool, device="cuda"))


def test_backward_with_a_limited_number_of_interleaved_heads():
    """12288 tokens, groups of four: five of the six heads end the launch together, one runs in front. Every
    head's dK and dV as in a launch of its own, bit for bit; dQ is summed in arrival order."""
    from ultraattn_b200.api import local_backward
    S, H, Hk = 12288, 24, 6
    q, k, v, d_o = _rand(5, (1, S, H), (1, S, Hk), (1, S, Hk), (1, S, H))
    o, lse = torch.empty_like(q), torch.empty(1, H, S, device="cuda")
    A.attn_fwd_dense(q, k, v, (o, lse), True)
    dq, dk, dv = local_backward(q, k, v, o, lse, d_o, None, None, 2)
    for h in range(Hk):
        qs, ks = slice(4 * h, 4 * h + 4), slice(h, h + 1)
        part = local_backward(q[:, :, qs], k[:, :, ks], v[:, :, ks], o[:, :, qs], lse[:, qs].contiguous(), d_o[:, :, qs], None, None, 2)
        assert torch.equal(dk[:, :, ks], part[1]) and torch.equal(dv[:, :, ks], part[2])
        assert (dq[:, :, qs].float() - part[0].float()).norm() <= 2 ** -8 * part[0].float().norm()
    A.check_status()
