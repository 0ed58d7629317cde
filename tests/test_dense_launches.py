"""Dense launches (no tables; packed query heads, keys split over CTAs) against float64 attention; the dense
backward against the table launch."""
import math

import pytest
import torch

from ultraattn_b200.ops import attention as A

pytestmark = pytest.mark.gpu

# (batch, queries, keys, query heads, kv heads, causal, key splits): one query and a full / overfull 128-row tile
# of packed rows, ungrouped heads, a group that is no power of two, fewer keys than one tile, more splits than
# key tiles, rows that see no key (more queries than keys under a causal mask), ragged everything
CASES = [(2, 1, 1000, 8, 2, True, 0), (1, 1, 513, 4, 4, True, 3), (3, 1, 4096, 16, 2, False, 7), (1, 1, 100, 8, 8, True, 0),
         (1, 32, 900, 8, 2, True, 0), (1, 33, 900, 8, 2, True, 5), (1, 128, 640, 2, 2, True, 2), (1, 129, 640, 2, 2, True, 2),
         (2, 17, 700, 6, 2, True, 0), (1, 40, 700, 12, 2, False, 4), (1, 300, 1111, 8, 1, True, 0), (1, 257, 257, 4, 2, True, 3),
         (1, 1000, 1000, 8, 2, True, 0), (1, 1000, 1000, 8, 2, True, 1), (1, 700, 300, 4, 2, True, 2), (1, 5, 1, 2, 1, False, 9),
         (1, 512, 4100, 4, 1, True, 0), (2, 260, 260, 2, 2, False, 1), (1, 64, 60, 2, 1, True, 1), (1, 1, 70000, 2, 1, True, 0)]


@pytest.mark.parametrize("B,Sq,Skv,H,Hk,causal,n_split", CASES)
def test_dense_forward_matches_float64(B, Sq, Skv, H, Hk, causal, n_split):
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA GPU")
    g = torch.Generator(device="cuda").manual_seed(Sq * 7 + Skv)
    mk = lambda s, h: torch.randn(B, s, h, 128, device="cuda", dtype=torch.bfloat16, generator=g)
    q, k, v = mk(Sq, H), mk(Skv, Hk), mk(Skv, Hk)
    o = torch.full_like(q, 7.0)
    lse = torch.full((B, H, Sq), 7.0, device="cuda")
    A.attn_fwd_dense(q, k, v, (o, lse), causal, None, n_split)
    A.check_status()
    s = torch.einsum("bqhd,bkhd->bhqk", q.double(), k.double().repeat_interleave(H // Hk, 2)) / math.sqrt(128)
    if causal:
        r, c = torch.arange(Sq, device="cuda")[:, None], torch.arange(Skv, device="cuda")[None, :]
        s = s.masked_fill(c > r + Skv - Sq, float("-inf"))
    ref_lse = torch.logsumexp(s, -1)
    p = torch.exp(s - ref_lse.masked_fill(ref_lse == float("-inf"), 0.0)[..., None])
    ref = torch.einsum("bhqk,bkhd->bqhd", p, v.double().repeat_interleave(H // Hk, 2))
    seen = torch.isfinite(ref_lse)
    assert torch.equal(torch.isfinite(lse), seen)
    assert (lse[seen] - ref_lse[seen]).abs().max() < 1e-3
    # P and O are rounded to bf16 (2^-9 each), rows without keys are exactly zero
    assert (o.double() - ref).norm() <= 4 * 2 ** -9 * ref.norm()
    assert (o.transpose(1, 2)[~seen] == 0).all()


def test_dense_forward_writes_into_strided_outputs_and_reads_strided_inputs():
    """K / V as views of a packed projection, O as a slice of a larger buffer."""
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA GPU")
    torch.manual_seed(0)
    kv = torch.randn(1, 900, 2, 2, 128, device="cuda", dtype=torch.bfloat16)
    q = torch.randn(1, 9, 8, 128, device="cuda", dtype=torch.bfloat16)
    big = torch.zeros(1, 9, 12, 128, device="cuda", dtype=torch.bfloat16)
    lse = torch.empty(1, 8, 9, device="cuda")
    A.attn_fwd_dense(q, kv[:, :, 0], kv[:, :, 1], (big[:, :, 2:10], lse), True)
    o2, lse2 = torch.empty_like(q), torch.empty_like(lse)
    A.attn_fwd_dense(q, kv[:, :, 0].contiguous(), kv[:, :, 1].contiguous(), (o2, lse2), True)
    assert torch.equal(big[:, :, 2:10], o2) and torch.equal(lse, lse2)
    assert (big[:, :, :2] == 0).all() and (big[:, :, 10:] == 0).all()


@pytest.mark.parametrize("B,Sq,Skv,H,Hk,causal", [(2, 300, 300, 4, 2, True), (1, 129, 700, 4, 1, True), (3, 200, 77, 2, 2, True),
                                                  (2, 128, 129, 4, 4, False), (1, 1, 130, 2, 1, True), (1, 1000, 1000, 8, 2, False)])
def test_dense_backward_equals_the_table_launch(B, Sq, Skv, H, Hk, causal):
    """Same kernel, same order of work: dK and dV bit for bit; dQ is summed in arrival order (fp32)."""
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA GPU")
    from ultraattn_b200.ops import elementwise as E
    g = torch.Generator(device="cuda").manual_seed(Sq + Skv)
    mk = lambda s, h: torch.randn(B, s, h, 128, device="cuda", dtype=torch.bfloat16, generator=g)
    q, k, v, d_o = mk(Sq, H), mk(Skv, Hk), mk(Skv, Hk), mk(Sq, H)
    o, lse = torch.empty_like(q), torch.empty(B, H, Sq, device="cuda")
    A.attn_fwd_dense(q, k, v, (o, lse), causal)
    dvec, zero = E.bwd_prepare(o, d_o)
    assert (zero == 0).all()
    assert (dvec - (o.double() * d_o.double()).sum(-1).transpose(1, 2)).abs().max() < 1e-3
    res = []
    for dense in (True, False):
        dq, out = torch.zeros_like(zero), A.BwdKvOut(torch.empty_like(k), torch.empty_like(v))
        side = A.BwdQSide(q, d_o, lse, dvec, dq)
        if dense:
            A.attn_bwd_dense(side, k, v, out, causal)
        else:
            A.attn_bwd([side], [k], [v], [out], A.BwdPlan([A.Col(0, 0, Skv, (A.Seg(0, 0, Sq, causal, Skv - Sq),))], "cuda"))
        res.append((out.dk, out.dv, dq))
    A.check_status()
    assert torch.equal(res[0][0], res[1][0]) and torch.equal(res[0][1], res[1][1])
    assert (res[0][2] - res[1][2]).norm() <= 1e-6 * res[1][2].norm()


@pytest.mark.parametrize("B,S,H,Hk,kind", [(1, 130, 2, 1, "causal"), (2, 257, 4, 2, "full"), (3, 64, 2, 2, "causal"), (1, 256, 4, 4, "blocks")])
def test_backward_in_one_call_equals_its_parts(B, S, H, Hk, kind):
    """attn_bwd_local against rowdot / fill, table launch and cast made one by one; K / V as views of one buffer."""
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA GPU")
    from ultraattn_b200 import api, patterns as P
    from ultraattn_b200.ops import elementwise as E
    g = torch.Generator(device="cuda").manual_seed(S)
    mk = lambda s, h: torch.randn(B, s, h, 128, device="cuda", dtype=torch.bfloat16, generator=g)
    q, d_o, kv = mk(S, H), mk(S, H), mk(S, 2 * Hk)
    k, v = kv[:, :, :Hk], kv[:, :, Hk:]
    pat = {"causal": P.causal(1), "full": P.full(1), "blocks": P.causal(2)}[kind]
    fplan, bplan = api.local_plans(pat, S, q.device)
    o, lse = torch.empty_like(q), torch.empty(B, H, S, device="cuda")
    A.attn_fwd([q], [k], [v], [(o, lse)], fplan)
    dense = {"causal": 2, "full": 1, "blocks": 0}[kind]
    got = api.local_backward(q, k, v, o, lse, d_o, bplan, None, dense)
    dvec, dq32 = E.bwd_prepare(o, d_o)
    out = A.BwdKvOut(torch.empty_like(k.contiguous()), torch.empty_like(v.contiguous()))
    A.attn_bwd([A.BwdQSide(q, d_o, lse, dvec, dq32)], [k], [v], [out], bplan)
    A.check_status()
    assert torch.equal(got[1], out.dk) and torch.equal(got[2], out.dv)
    assert (got[0].float() - dq32).norm() <= 2 ** -8 * dq32.norm()


@pytest.mark.parametrize("Sq", [1, 300])
@pytest.mark.parametrize("n_split", [1, 4])
def test_values_that_are_not_finite_do_not_depend_on_the_split(Sq, n_split):
    """A NaN or infinite score: the row has O = 0 and lse = -inf. A NaN in V: NaN in that column of O."""
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA GPU")
    Skv, H = 1400, 2
    g = torch.Generator(device="cuda").manual_seed(5)
    mk = lambda s: torch.randn(1, s, H, 128, device="cuda", dtype=torch.bfloat16, generator=g)
    q, k, v = mk(Sq), mk(Skv), mk(Skv)
    for value in (float("nan"), float("inf")):
        k2 = k.clone()
        k2[0, 700, 0, 5] = value
        q2 = q.clone()
        q2[:, :, 0, 5] = 1.0
        o, lse = torch.full_like(q, 7.0), torch.full((1, H, Sq), 7.0, device="cuda")
        A.attn_fwd_dense(q2, k2, v, (o, lse), False, None, n_split)
        assert (o[:, :, 0] == 0).all() and (lse[:, 0] == -math.inf).all()
        assert torch.isfinite(lse[:, 1]).all() and (o[:, :, 1] != 0).any(-1).all()
    v2 = v.clone()
    v2[0, 900, 1, 3] = float("nan")
    k2 = k * 30                                     # parts whose weight is exactly zero, too
    o, lse = torch.full_like(q, 7.0), torch.full((1, H, Sq), 7.0, device="cuda")
    A.attn_fwd_dense(q, k2, v2, (o, lse), False, None, n_split)
    A.check_status()
    bad = torch.isnan(o[0])
    assert bad[:, 1, 3].all() and bad.sum() == Sq and torch.isfinite(lse).all()
