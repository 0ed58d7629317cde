"""Dense launches of a few items: the two sub-tiles of a CTA share 128 rows and take the key tiles in turn, against
float64 attention."""
import math

import pytest
import torch

from ultraattn_b200.ops import attention as A

pytestmark = pytest.mark.gpu

# (batch, queries, keys, query heads, kv heads, causal): four key tiles (the fewest) and five, one more query than a tile,
# rows of the first tile that see one key tile (the second sub-tile sees none), more queries than keys (rows, and whole tiles, that
# see no key), groups of 1, 2 and 8 and one that is no power of two, the last query tile ragged, many keys for few rows
SHAPES = [(1, 500, 500, 4, 4, True), (2, 513, 513, 2, 1, True), (1, 129, 400, 2, 2, False), (1, 1500, 520, 2, 2, True),
          (1, 385, 1000, 8, 1, True), (1, 200, 640, 12, 4, False), (3, 333, 1030, 4, 4, True), (1, 1000, 1000, 8, 8, False)]


@pytest.mark.parametrize("B,Sq,Skv,H,Hk,causal", SHAPES)
@pytest.mark.parametrize("offset", [0, 4])
def test_row_tiles_whose_sub_tiles_share_the_keys(B, Sq, Skv, H, Hk, causal, offset):
    """offset 4: rows of O that begin 8 bytes past a multiple of 16, where the stores are of 8 bytes."""
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA GPU")
    g = torch.Generator(device="cuda").manual_seed(Sq + Skv)
    mk = lambda s, h: torch.randn(B, s, h, 128, device="cuda", dtype=torch.bfloat16, generator=g)
    q, k, v = mk(Sq, H), mk(Skv, Hk), mk(Skv, Hk)
    k[0, -60, 0, 5], q[:, :, 0, 5] = float("nan"), 1.0     # rows of the first group that see this key: no result
    flat = torch.full((B * Sq * H * 128 + 128,), 7.0, device="cuda", dtype=torch.bfloat16)
    o, lse = flat[offset:offset + B * Sq * H * 128].view(B, Sq, H, 128), torch.full((B, H, Sq), 7.0, device="cuda")
    A.attn_fwd_dense(q, k, v, (o, lse), causal)
    A.check_status()
    s = torch.einsum("bqhd,bkhd->bhqk", q.double(), k.double().repeat_interleave(H // Hk, 2)) / math.sqrt(128)
    if causal:
        r, c = torch.arange(Sq, device="cuda")[:, None], torch.arange(Skv, device="cuda")[None, :]
        s = s.masked_fill(c > r + Skv - Sq, float("-inf"))
    s = s.masked_fill(torch.isnan(s).any(-1, keepdim=True), float("-inf"))
    ref_lse = torch.logsumexp(s, -1)
    p = torch.exp(s - ref_lse.masked_fill(ref_lse == float("-inf"), 0.0)[..., None])
    ref = torch.einsum("bhqk,bkhd->bqhd", p, v.double().repeat_interleave(H // Hk, 2))
    seen = torch.isfinite(ref_lse)
    assert torch.equal(torch.isfinite(lse), seen)
    assert (lse[seen] - ref_lse[seen]).abs().max() < 1e-3
    # P and O are rounded to bf16 (2^-9 each), rows without keys are exactly zero
    assert (o.double() - ref).norm() <= 4 * 2 ** -9 * ref.norm()
    assert (o.transpose(1, 2)[~seen] == 0).all()
    assert (flat[:offset] == 7).all() and (flat[offset + B * Sq * H * 128:] == 7).all()
