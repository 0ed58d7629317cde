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


def _scores(q, k, seen):
    s = torch.einsum("bqhd,bkhd->bhqk", q, k.repeat_interleave(q.shape[2] // k.shape[2], 2)) / math.sqrt(128)
    return s if seen is None else s.masked_fill(~seen, float("-inf"))


def _attend(q, k, v, seen):
    """(o, lse) in the type of the inputs; rows that see nothing: zeros and -inf."""
    s = _scores(q, k, seen)
    lse = torch.logsumexp(s, -1)
    p = torch.exp(s - lse.masked_fill(lse == float("-inf"), 0.0)[..., None])
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
