"""Score tiles of the forward kernel that a warp's 32 rows see all of, part of or nothing of, in every position of an
item (first, last, all of them), against float64 attention."""
import math

import pytest
import torch

from ultraattn_b200.ops import attention as A

pytestmark = pytest.mark.gpu

# (queries, [(first key, keys, causal, diag, lo)]): a band that is narrower than a warp's rows, one that starts inside a
# tile, edges at multiples of 32 and of 128 and one beside them, a first segment that no row or only the last rows see, a
# last one of the same kind, one that ends before it begins (lo > diag), a segment of one key, 1 to 300 rows
BANDS = [(256, [(0, 256, True, 0, -20)]), (300, [(0, 300, True, 0, -127)]), (300, [(0, 300, True, 0, -128)]),
         (300, [(0, 300, True, 0, -129)]), (256, [(0, 640, True, 384, 352)]), (256, [(0, 640, True, 383, 353)]),
         (257, [(0, 400, True, -200, None), (400, 100, False, 0, None)]),
         (257, [(400, 100, False, 0, None), (0, 400, True, -200, None)]),
         (200, [(0, 128, True, -300, None), (128, 130, True, 0, None)]), (200, [(0, 300, True, 10, 20)]),
         (64, [(0, 700, False, 0, 600)]), (130, [(0, 4, True, -60, None), (4, 500, True, 100, -60)]),
         (1, [(0, 1, True, 0, None)]), (33, [(7, 1, False, 0, None), (8, 260, True, 3, -1)])]


@pytest.mark.parametrize("n_q,segs", BANDS)
@pytest.mark.parametrize("heads,kv_heads", [(2, 2), (4, 1)])
def test_tiles_in_every_position(n_q, segs, heads, kv_heads):
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA GPU")
    n_k = max(s + n for s, n, *_ in segs)
    g = torch.Generator(device="cuda").manual_seed(n_q + n_k)
    mk = lambda s, h: torch.randn(2, s, h, 128, device="cuda", dtype=torch.bfloat16, generator=g)
    q, k, v = mk(n_q, heads), mk(n_k, kv_heads), mk(n_k, kv_heads)
    o, lse = torch.full_like(q, 7.0), torch.full((2, heads, n_q), 7.0, device="cuda")
    row = A.Row(0, 0, n_q, tuple(A.Seg(0, s, n, c, d, lo=lo) for s, n, c, d, lo in segs), 0, 0, False)
    A.attn_fwd_cuda([q], [k], [v], [(o, lse)], A.FwdPlan([row], q.device))
    A.check_status()
    r = torch.arange(n_q, device="cuda")[:, None]
    parts, vals = [], []
    for s, n, causal, diag, lo in segs:
        c = torch.arange(n, device="cuda")[None]
        see = torch.ones(n_q, n, dtype=torch.bool, device="cuda")
        if causal:
            see &= c <= r + diag
        if lo is not None:
            see &= c >= r + lo
        sc = torch.einsum("bqhd,bkhd->bhqk", q.double(), k[:, s:s + n].double().repeat_interleave(heads // kv_heads, 2))
        parts.append((sc / math.sqrt(128)).masked_fill(~see, float("-inf")))
        vals.append(v[:, s:s + n].double().repeat_interleave(heads // kv_heads, 2))
    sc = torch.cat(parts, -1)
    ref_lse = torch.logsumexp(sc, -1)
    p = torch.exp(sc - ref_lse.masked_fill(ref_lse == float("-inf"), 0.0)[..., None])
    ref = torch.einsum("bhqk,bkhd->bqhd", p, torch.cat(vals, 1))
    seen = torch.isfinite(ref_lse)
    assert torch.equal(torch.isfinite(lse), seen)
    assert not seen.any() or (lse[seen] - ref_lse[seen]).abs().max() < 1e-3
    # P and O are rounded to bf16 (2^-9 each); rows without keys are exactly zero
    assert (o.double() - ref).norm() <= 4 * 2 ** -9 * ref.norm()
    assert (o.transpose(1, 2)[~seen] == 0).all()


@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
@pytest.mark.parametrize("tile", [0, 3])
def test_a_row_with_a_bad_score_is_empty_and_alone(bad, tile):
    """A query that makes one score NaN or infinite comes out as O = 0 and lse = -inf; its neighbours are untouched."""
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA GPU")
    torch.manual_seed(tile)
    q, k, v = (torch.randn(1, 512, 1, 128, device="cuda", dtype=torch.bfloat16) for _ in range(3))
    plan = A.FwdPlan([A.Row(0, 0, 512, (A.Seg(0, 0, 512, False, 0),), 0, 0, False)], q.device)
    run = lambda: (torch.empty_like(q), torch.empty(1, 1, 512, device="cuda"))
    o0, l0 = run()
    A.attn_fwd_cuda([q], [k], [v], [(o0, l0)], plan)
    q2, k2 = q.clone(), k.clone()
    k2[0, tile * 128 + 5, 0] = 0
    q2[:, :, :, 7] = 0
    o1, l1 = run()
    A.attn_fwd_cuda([q2], [k2], [v], [(o1, l1)], plan)
    k2[0, tile * 128 + 5, 0, 7] = 3.0              # only the one query with a non-zero component there sees it
    q3 = q2.clone()
    q3[0, 200, 0, 7] = bad
    o2, l2 = run()
    A.attn_fwd_cuda([q3], [k2], [v], [(o2, l2)], plan)
    A.check_status()
    assert (o2[0, 200] == 0).all() and l2[0, 0, 200] == float("-inf")
    rest = torch.arange(512, device="cuda") != 200
    assert torch.equal(o2[0, rest], o1[0, rest]) and torch.equal(l2[0, 0, rest], l1[0, 0, rest])
