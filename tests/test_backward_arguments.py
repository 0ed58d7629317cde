"""What the one-call backward accepts and refuses before anything is launched (CPU, the library replaced by a
recorder), and packed batches with tokens outside every sequence (GPU, against float64)."""
import math

import pytest
import torch

from ultraattn_b200 import _lib
from ultraattn_b200.ops import attention as A
from ultraattn_b200.ops import flash_compat as F


@pytest.fixture
def calls(monkeypatch):
    """Calls of the one-call backward as (fields of the argument block, scale); nothing is launched."""
    got = []

    class Library:
        def ua_attn_bwd_local(self, block, scale, status, stream):
            got.append((A._LOCAL_BWD.unpack(block), scale))
            return 0

    monkeypatch.setattr(_lib, "load", lambda: Library())
    monkeypatch.setattr(_lib, "stream_of", lambda t: 0)
    monkeypatch.setattr(A, "status_buffer", lambda device: torch.zeros(4, dtype=torch.int32))
    return got


def _bf16(*shape):
    return torch.zeros(*shape, dtype=torch.bfloat16)


def _local(B=1, S=64, H=4, Hk=2, **other):
    t = dict(q=_bf16(B, S, H, 128), k=_bf16(B, S, Hk, 128), v=_bf16(B, S, Hk, 128), o=_bf16(B, S, H, 128),
             lse=torch.zeros(B, H, S), d_o=_bf16(B, S, H, 128), dq=_bf16(B, S, H, 128), dk=_bf16(B, S, Hk, 128),
             dv=_bf16(B, S, Hk, 128))
    t.update(other)
    return A.attn_bwd_local(plan=None, dense=2, **t)


def test_one_call_backward_refuses_other_shapes(calls):
    _local()
    assert len(calls) == 1
    for bad in (dict(lse=torch.zeros(1, 4, 63)), dict(lse=torch.zeros(1, 4, 65)), dict(lse=torch.zeros(1, 64, 4)),
                dict(lse=torch.zeros(1, 1, 64)), dict(dk=_bf16(1, 63, 2, 128)), dict(dv=_bf16(1, 64, 1, 128))):
        with pytest.raises(AssertionError):
            _local(**bad)
    assert len(calls) == 1


def test_one_call_backward_refuses_plans_that_write_behind_the_gradients(calls, monkeypatch):
    """A block pattern over more queries than keys; documents that end behind the buffer, also where the numbers of
    tokens agree."""
    from ultraattn_b200 import api, patterns as P
    monkeypatch.setattr(A, "_native", lambda *t: True)
    monkeypatch.setattr(_lib, "host", lambda: pytest.fail("the native route was taken"), raising=False)
    shapes = dict(k=_bf16(1, 32, 2, 128), v=_bf16(1, 32, 2, 128), dk=_bf16(1, 32, 2, 128), dv=_bf16(1, 32, 2, 128))
    t = dict(q=_bf16(1, 64, 4, 128), o=_bf16(1, 64, 4, 128), lse=torch.zeros(1, 4, 64), d_o=_bf16(1, 64, 4, 128))
    for plan in (api.local_plans(P.causal(2), 64, "cpu")[1], api.varlen_plans([32, 64], True, "cpu")[1]):
        with pytest.raises(AssertionError, match="behind the end"):
            A.attn_bwd_local(plan=plan, dq=_bf16(1, 64, 4, 128), **t, **shapes)
        assert A.local_backward(t["q"], shapes["k"], shapes["v"], t["o"], t["lse"], t["d_o"], plan) is None
    fits = api.varlen_plans([0, 32], True, "cpu")[1]
    state = {n: x for n, x in vars(fits).items() if n != "kv_end"}
    fits = A.BwdPlan.__new__(A.BwdPlan)
    fits.__dict__.update(state)                                    # (as a plan comes out of a file written before)
    A.attn_bwd_local(plan=fits, dq=_bf16(1, 64, 4, 128), **t, **shapes)
    assert len(calls) == 1


def test_returned_row_products_do_not_keep_the_workspace(calls):
    d = _local()
    assert d.shape == (1, 4, 64) and d.untyped_storage().nbytes() == 4 * d.numel()


def _one_head(S, pad=0):
    """[2, S, 1, 128] whose head axis has the stride of all tokens."""
    t = _bf16(2, 1, S + pad, 128)[:, :, :S].transpose(1, 2)
    assert t.stride(2) == (S + pad) * 128
    return t


def test_one_call_backward_takes_any_stride_of_an_axis_of_one(calls):
    S = 64
    t = {n: _one_head(S) for n in ("o", "d_o", "dk", "dv")}
    _local(B=2, S=S, H=1, Hk=1, **t)
    _local(B=2, S=S, H=1, Hk=1, dk=_one_head(S), dv=_bf16(2, S, 1, 128))             # the same addresses
    # one token: its stride means nothing either
    one = _bf16(2, 4, 1, 128).transpose(1, 2)
    _local(B=2, S=1, H=4, Hk=4, o=one, d_o=one, dk=one, dv=_bf16(2, 1, 4, 128))
    assert len(calls) == 3
    f = calls[0][0]
    assert f[21:28] == (t["d_o"].data_ptr(), S, 1, 2, 128, S * 128, S * 128)         # q, k, v: seven fields each
    assert f[28:31] == (t["o"].data_ptr(), 128, S * 128)
    assert f[35:39] == (t["dk"].data_ptr(), t["dv"].data_ptr(), 128, S * 128)
    heads_apart = _bf16(2, 4, S, 128).transpose(1, 2)                                # more than one: they must lie side by side
    for bad in (dict(o=heads_apart), dict(d_o=heads_apart), dict(H=2, Hk=1, dk=_one_head(S), dv=_one_head(S, 3))):
        with pytest.raises(AssertionError):
            _local(**{"B": 2, "S": S, **bad})
    assert len(calls) == 3


@pytest.mark.parametrize("full", [True, False])
def test_window_gradients_of_one_head_are_laid_out_for_the_kernel(monkeypatch, full):
    from ultraattn_b200.ops import window as W
    outs = []
    monkeypatch.setattr(A, "attn_bwd", lambda sides, k, v, kv, plan, scale: outs.extend(kv))
    S, k, v = 64, _one_head(64), _one_head(64)
    q = _bf16(2, S, 4, 128)
    z = torch.zeros(2, 4, S)
    dq, dk, dv = W._cuda_backward(q, q, k, v, z, z, torch.zeros(2, S, 4, 128), None, None, full, 1.0)
    assert dk.shape == k.shape and dv.shape == v.shape
    for t in (outs[0].dk, outs[0].dv):
        assert t.stride() == (S * 128, 128, 128, 1)


def test_packed_lse_covers_the_whole_buffer():
    cu, H, total = [0, 5, 5, 12], 3, 16
    lse = torch.randn(H, total)
    packed = F._packed_lse(F._pad_lse(lse, cu, 7), cu, total)
    assert packed.shape == (H, total) and packed.is_contiguous()
    assert torch.equal(packed[:, :12], lse[:, :12]) and (packed[:, 12:] == -math.inf).all()


def _documents(q, k, v, cu, causal):
    """float64 attention of the documents ``cu``; zeros elsewhere. ``[tokens, heads, 128]``."""
    o = torch.zeros_like(q)
    for a, b in zip(cu[:-1], cu[1:]):
        G = q.shape[1] // k.shape[1]
        s = torch.einsum("qhd,khd->hqk", q[a:b], k[a:b].repeat_interleave(G, 1)) / math.sqrt(128)
        if causal:
            s = s.masked_fill(torch.ones(b - a, b - a, dtype=torch.bool, device=q.device).triu(1), float("-inf"))
        o[a:b] = torch.einsum("hqk,khd->qhd", torch.softmax(s, -1), v[a:b].repeat_interleave(G, 1))
    return o


def _close(got, want):
    # P, dS and every result are rounded to bf16 (2^-9 each, independent errors); 8 of them is far outside
    return (got.double() - want).norm() <= 8 * 2 ** -9 * want.norm()


@pytest.mark.gpu
@pytest.mark.parametrize("window", [(-1, -1), (60, 0)])
def test_packed_batch_with_a_tail_outside_the_sequences(window):
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA GPU")
    T, H, Hk, cu = 512, 4, 2, [0, 100, 421]
    g = torch.Generator(device="cuda").manual_seed(0)
    mk = lambda h: torch.randn(T, h, 128, device="cuda", dtype=torch.bfloat16, generator=g)
    q, k, v, d_o = mk(H), mk(Hk), mk(Hk), mk(H)
    d_o[cu[-1]:] = 0
    args = (cu, cu, 321, 321, 0.0, None, True, window)
    o, *_, lse, _, _ = F._flash_attn_varlen_forward(q, k, v, *args)
    dq, dk, dv = (torch.full_like(t, float("nan")) for t in (q, k, v))
    F._flash_attn_varlen_backward(d_o, q, k, v, o, lse, dq, dk, dv, *args)
    A.check_status()
    qd, kd, vd = (t.double().requires_grad_() for t in (q, k, v))
    if window == (-1, -1):
        ref = _documents(qd, kd, vd, cu, True)
    else:
        s = torch.einsum("qhd,khd->hqk", qd, kd.repeat_interleave(2, 1)) / math.sqrt(128)
        r, c = torch.arange(T, device="cuda")[:, None], torch.arange(T, device="cuda")[None]
        doc = torch.bucketize(torch.arange(T, device="cuda"), torch.tensor(cu, device="cuda"), right=True)
        seen = (c <= r) & (c >= r - window[0]) & (doc[:, None] == doc[None]) & (r < cu[-1])
        p = torch.softmax(s.masked_fill(~seen, -1e30), -1) * seen
        ref = torch.einsum("hqk,khd->qhd", p, vd.repeat_interleave(2, 1))
    ref.backward(d_o.double())
    assert _close(o, ref.detach())
    for got, want in ((dq, qd.grad), (dk, kd.grad), (dv, vd.grad)):
        assert _close(got, want) and (got[cu[-1]:] == 0).all()


def _attend(kind, q, k, v):
    from ultraattn_b200 import api, attention, patterns as P
    if kind == "dense":
        return attention(q, k, v, P.causal(1))
    if kind == "blocks":
        return attention(q, k, v, P.causal(2))
    if kind == "flash":
        return F.flash_attn_func(q, k, v, causal=True)
    if kind == "varlen":
        return api.varlen_attention(q, k, v, [0, q.shape[1]])
    from ultraattn_b200.ops.window import sliding_window_attention
    return sliding_window_attention(q, k, v, (k.shape[1] - 1 if kind == "wide window" else 70, 0), causal=True)


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["dense", "blocks", "flash", "varlen", "window", "wide window"])
def test_one_head_through_transposes(kind):
    """The output's gradient, and a single key / value head, come in as views of [B, 1, S, 128]."""
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA GPU")
    B, S = (1 if kind == "varlen" else 2), 300
    g = torch.Generator(device="cuda").manual_seed(1)
    mk = lambda *s: torch.randn(*s, 128, device="cuda", dtype=torch.bfloat16, generator=g)
    for H in (1, 4):
        q, d_o, k, v = mk(B, S, H), mk(B, H, S), mk(B, 1, S).transpose(1, 2), mk(B, 1, S).transpose(1, 2)
        q, k, v = (t.requires_grad_() for t in (q, k, v))
        o = _attend(kind, q, k, v)
        got = torch.autograd.grad(o.transpose(1, 2), (q, k, v), d_o)
        A.check_status()
        qd, kd, vd = (t.detach().double().requires_grad_() for t in (q, k, v))
        s = torch.einsum("bqhd,bkd->bhqk", qd, kd[:, :, 0]) / math.sqrt(128)
        r, c = torch.arange(S, device="cuda")[:, None], torch.arange(S, device="cuda")[None]
        s = s.masked_fill((c > r) | ((c < r - 70) & (kind == "window")), float("-inf"))
        ref = torch.einsum("bhqk,bkd->bhqd", torch.softmax(s, -1), vd[:, :, 0])
        want = torch.autograd.grad(ref, (qd, kd, vd), d_o.double())
        assert _close(o.transpose(1, 2).detach(), ref.detach())
        assert all(_close(a, b) for a, b in zip(got, want))


@pytest.mark.gpu
@pytest.mark.parametrize("packed", [False, True])
def test_fp32_key_gradients_are_added_into(packed):
    """dK / dV in fp32: the same gradients with and without D given, on top of what the buffers hold (the packed
    form clears them first)."""
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA GPU")
    B, S, H, Hk = 1, 300, 4, 2
    g = torch.Generator(device="cuda").manual_seed(2)
    mk = lambda h: torch.randn(B, S, h, 128, device="cuda", dtype=torch.bfloat16, generator=g)
    q, k, v, d_o = mk(H), mk(Hk), mk(Hk), mk(H)
    cu = [0, 120, 300]
    if packed:
        q, k, v, d_o = (t[0] for t in (q, k, v, d_o))
        o, *_, lse, _, _ = F._flash_attn_varlen_forward(q, k, v, cu, cu, 180, 180, 0.0, None, True)
        back = lambda dq, dk, dv, d: F._flash_attn_varlen_backward(d_o, q, k, v, o, lse, dq, dk, dv, cu, cu, 180, 180, 0.0, None,
                                                                   True, softmax_d=d)[3]
    else:
        o, *_, lse, _, _ = F._flash_attn_forward(q, k, v, 0.0, None, True)
        back = lambda dq, dk, dv, d: F._flash_attn_backward(d_o, q, k, v, o, lse, dq, dk, dv, 0.0, None, True, softmax_d=d)[3]
    dq, dk, dv = (torch.empty_like(t) for t in (q, k, v))
    d = back(dq, dk, dv, None)                                     # bf16: written
    start = 0.0 if packed else 3.0
    for given in (None, d):
        dq2, dk2, dv2 = torch.empty_like(q), torch.full_like(k, 3.0, dtype=torch.float32), torch.full_like(v, 3.0, dtype=torch.float32)
        d2 = back(dq2, dk2, dv2, given)
        A.check_status()
        assert torch.equal(d2, d)
        assert (dq2.float() - dq.float()).norm() <= 2 ** -8 * dq.float().norm()      # (summed in arrival order, then rounded)
        for a, b in ((dk2, dk), (dv2, dv)):
            assert (a - start - b.float()).norm() <= 2 ** -8 * b.float().norm()


def test_preparation_refuses_misaligned_tensors_before_the_launch():
    """Argument checks at the C entry: no launch happens (and no GPU is needed)."""
    lib = _lib.load()
    n = 4 * 2 * 128
    ok = dict(o=1 << 20, d_o=2 << 20, dvec=3 << 20, dq=4 << 20, o_b=n, o_t=256, d_b=n, d_t=256, batch=2, tokens=4, heads=2)
    for bad in (dict(o=(1 << 20) + 2), dict(d_o=(2 << 20) + 8), dict(dq=(4 << 20) + 4), dict(o_t=257), dict(d_t=260),
                dict(o_b=n + 1), dict(d_b=n + 4)):
        a = {**ok, **bad}
        assert lib.ua_bwd_prepare(*a.values(), None) != 0
        assert b"16 bytes" in lib.ua_last_error()


@pytest.mark.gpu
def test_preparation_reads_heads_that_lie_apart():
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA GPU")
    from ultraattn_b200.ops import elementwise as E
    B, S, H = 2, 70, 3
    g = torch.Generator(device="cuda").manual_seed(3)
    mk = lambda *s: torch.randn(*s, 128, device="cuda", dtype=torch.bfloat16, generator=g)
    plain, apart, one = mk(B, S, H), mk(B, H, S).transpose(1, 2), mk(B, 1, S).transpose(1, 2)
    for o, d_o in ((plain, apart), (apart, plain), (one, one * 2)):
        d, zero = E.bwd_prepare(o, d_o)
        assert (zero == 0).all()
        assert (d - (o.double() * d_o.double()).sum(-1).transpose(1, 2)).abs().max() < 1e-3


def test_plans_know_how_many_gradient_rows_they_write():
    from ultraattn_b200 import api, patterns as P
    tokens = lambda plans: plans[1].kv_tokens
    assert tokens(api.varlen_plans([0, 5, 5, 12], True, "cpu")) == 12
    assert tokens(api.prefix_lm_plans(16, 3, "cpu", [0, 2, 9])) == 9
    for pattern in (P.causal(4), P.star(4, 1), P.streaming(4, 1, 2)):       # (empty blocks are columns too: zeros)
        assert tokens(api.local_plans(pattern, 64, "cpu")) == 64


@pytest.mark.gpu
@pytest.mark.parametrize("prefix", [None, 30])
def test_gradients_of_tokens_outside_every_sequence_are_zero(prefix):
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA GPU")
    from ultraattn_b200 import api
    T, H, Hk, cu = 512, 4, 2, [0, 100, 421]
    g = torch.Generator(device="cuda").manual_seed(4)
    mk = lambda h: torch.randn(T, h, 128, device="cuda", dtype=torch.bfloat16, generator=g)
    q, k, v, d_o = mk(H).requires_grad_(), mk(Hk).requires_grad_(), mk(Hk).requires_grad_(), mk(H)
    o = (api.varlen_attention(q, k, v, cu) if prefix is None else
         api.prefix_lm_attention(q, k, v, prefix, cu_seqlens=cu))
    junk = [torch.full_like(t, float("nan")) for t in (q, k, v, k, v)]      # what the allocator hands out next holds NaN
    del junk
    got = torch.autograd.grad(o, (q, k, v), d_o)
    A.check_status()
    assert (o[cu[-1]:] == 0).all() and all((t[cu[-1]:] == 0).all() for t in got)
    if prefix is None:
        ref = [t.detach().double().requires_grad_() for t in (q, k, v)]
        _documents(*ref, cu, True).backward(d_o.double())
        assert all(_close(a, b.grad) for a, b in zip(got, ref))


def test_plans_know_whether_a_few_tiles_hold_most_of_the_work():
    from ultraattn_b200 import api, patterns as P
    skewed = lambda pattern: api.local_plans(pattern, 4096, "cpu")[1].skewed
    assert not any(skewed(p) for p in (P.causal(1), P.full(1), P.strided(32, 4, 2)))
    assert all(skewed(p) for p in (P.global_local(32, 1, 2), P.star(32, 1), P.streaming(32, 1, 2)))
    assert not A.BwdPlan([]).skewed


@pytest.mark.gpu
@pytest.mark.parametrize("S", [256, 300])
@pytest.mark.parametrize("causal,scale", [(True, -0.05), (False, -0.05), (True, 0.05)])
def test_backward_with_a_negative_scale(S, causal, scale):
    """Masked scores, and rows behind the last one (300), are hidden after they are scaled, whatever the sign."""
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA GPU")
    B, H, Hk = 1, 4, 2
    g = torch.Generator(device="cuda").manual_seed(5)
    mk = lambda h: torch.randn(B, S, h, 128, device="cuda", dtype=torch.bfloat16, generator=g)
    q, k, v, d_o = mk(H), mk(Hk), mk(Hk), mk(H)
    qd, kd, vd = (t.double().requires_grad_() for t in (q, k, v))
    s = torch.einsum("bqhd,bkhd->bhqk", qd, kd.repeat_interleave(2, 2)) * scale
    if causal:
        s = s.masked_fill(torch.ones(S, S, dtype=torch.bool, device="cuda").triu(1), float("-inf"))
    o = torch.einsum("bhqk,bkhd->bqhd", torch.softmax(s, -1), vd.repeat_interleave(2, 2))
    want = torch.autograd.grad(o, (qd, kd, vd), d_o.double())
    dq, dk, dv = (torch.empty_like(t) for t in (q, k, v))
    lse = torch.logsumexp(s, -1).detach().float().contiguous()
    F._flash_attn_backward(d_o, q, k, v, o.detach().bfloat16().contiguous(), lse, dq, dk, dv, 0.0, scale, causal)
    A.check_status()
    assert all(_close(a, b) for a, b in zip((dq, dk, dv), want))
