"""Keys and values that do not fit the queries are refused by the library before anything is launched (no GPU needed: the
pointers are never followed)."""
import re

import pytest

from ultraattn_b200 import _lib
from ultraattn_b200.ops import attention as A

GOOD = dict(q=(2, 300, 4), k=(2, 300, 2), v=(2, 300, 2))
# one sequence of keys for two of queries (their gradients would be written behind the end of dK and dV), fewer values
# than keys, heads that do not divide or are not there
BAD = [dict(k=(1, 300, 2), v=(1, 300, 2)), dict(k=(1, 300, 2)), dict(v=(1, 300, 2)), dict(v=(2, 300, 1)), dict(v=(2, 299, 2)),
       dict(k=(2, 300, 3), v=(2, 300, 3)), dict(k=(2, 300, 8), v=(2, 300, 8)), dict(k=(2, 300, 0), v=(2, 300, 0))]
# ... and gradients of sequences that no query reads, which nothing would write
BAD_BACKWARD = [dict(k=(3, 300, 2), v=(3, 300, 2)), dict(v=(3, 300, 2))]


def _src(shape, at):
    """(pointer, tokens, heads, batch, strides of token, head and batch) of [batch, tokens, heads, 128]"""
    B, S, H = shape
    return at << 24, S, H, B, H * 128, 128, S * H * 128


def _refusal(rc):
    assert rc != 0
    return _lib.load().ua_last_error().decode()


def _names_the_shapes(msg):
    return re.match(r"ua_attn_\w+: .*(sequences|heads of keys|do not divide|values for)", msg) is not None


@pytest.mark.parametrize("other", BAD)
def test_dense_forward_refuses(other):
    s = {**GOOD, **other}
    B, S, H = s["q"]
    block = A._DENSE_FWD.pack(*_src(s["q"], 1), *_src(s["k"], 2), *_src(s["v"], 3), 4 << 24, 5 << 24, H * 128, S * H * 128, S, H * S)
    assert _names_the_shapes(_refusal(_lib.load().ua_attn_fwd_dense(block, 1, 0.1, 1, None, None, None)))


@pytest.mark.parametrize("other", BAD + BAD_BACKWARD)
def test_one_call_backward_refuses(other):
    s = {**GOOD, **other}
    B, S, H = s["q"]
    block = A._LOCAL_BWD.pack(*_src(s["q"], 1), *_src(s["k"], 2), *_src(s["v"], 3), *_src(s["q"], 4), 5 << 24, H * 128, S * H * 128,
                              6 << 24, 7 << 24, 8 << 24, 9 << 24, 10 << 24, 11 << 24, s["k"][2] * 128, S * s["k"][2] * 128, 0, 0, 0, 0, 2, 0)
    assert _names_the_shapes(_refusal(_lib.load().ua_attn_bwd_local(block, 0.1, None, None)))


@pytest.mark.parametrize("other", [o for o in BAD if o != dict(v=(2, 299, 2))])       # (a table may read a part of the values)
@pytest.mark.parametrize("backward", [False, True])
def test_table_launches_refuse(other, backward):
    s = {n: (_lib.UaTensorSrc * 1)(_lib.UaTensorSrc(*_src(x, i + 1))) for i, (n, x) in enumerate({**GOOD, **other}.items())}
    heads, kv_heads = s["q"][0].heads, s["k"][0].heads
    lib, stage = _lib.load(), (None, 0, 0, None, 1, None)
    if backward:
        side = (_lib.UaBwdQSide * 1)(_lib.UaBwdQSide(4 << 24, 5 << 24, 300, 1200, 6 << 24, 512, 153600))
        out = (_lib.UaBwdKvOut * 1)(_lib.UaBwdKvOut(7 << 24, 8 << 24, 256, 76800, 0, 0))
        rc = lib.ua_attn_bwd(s["q"], s["q"], side, 1, s["k"], s["v"], 1, out, 1, None, None, None, 3, 0, 0, heads, kv_heads, 2, 0.1, None,
                             *stage, None)
    else:
        out = (_lib.UaOutDst * 1)(_lib.UaOutDst(4 << 24, 5 << 24, 512, 153600, 300, 1200))
        rc = lib.ua_attn_fwd(s["q"], 1, s["k"], s["v"], 1, out, 1, None, None, None, 3, heads, kv_heads, 2, 0.1, None, *stage, None)
    assert _names_the_shapes(_refusal(rc))


def test_more_sequences_of_keys_than_of_queries_are_read_as_before():
    """A cache with room for more sequences. (The address of q is one that no tensor map takes: nothing is launched.)"""
    q, k = (1, 300, 4), (2, 300, 2)
    block = A._DENSE_FWD.pack(3, *_src(q, 1)[1:], *_src(k, 2), *_src(k, 3), 4 << 24, 5 << 24, 512, 300 * 512, 300, 1200)
    assert not _names_the_shapes(_refusal(_lib.load().ua_attn_fwd_dense(block, 1, 0.1, 1, None, None, None)))


def test_a_given_split_stays_where_the_shares_of_the_keys_are_exact():
    """(more parts than 2^16 for 2^18 key tiles: the products of the remainder and a part's number left 32 bits)"""
    parts = _lib.load().ua_attn_fwd_dense_parts
    keys = 128 << 18
    assert parts(1, 1, keys, 1, 1, 0, 1000) == 1000 and parts(1, 1, 700, 1, 1, 0, 1000) == 6
    for n_split in (65535, 65536, 70000, 200000):
        z = parts(1, 1, keys, 1, 1, 0, n_split)
        assert z == min(n_split, 65536)
        for n in (1 << 18, (1 << 18) - 1, 3 * z - 1):               # r is largest, z - 1, where n + 1 is a multiple of z
            q, r = divmod(n, z)
            for split in (0, 1, z // 2, z - 1):
                for at in (split, split + 1):
                    assert r * at < 1 << 32 and q * at + r * at // z == n * at // z
