"""The native host part of dense and planned calls against the same calls made from Python: same outputs for every layout
that either takes, the same refusals, and autograd's own machinery around it."""
import threading

import pytest
import torch

import ultraattn_b200 as ua
from ultraattn_b200 import _lib
from ultraattn_b200 import patterns as P
from ultraattn_b200.api import local_backward
from ultraattn_b200.ops import attention as A
from ultraattn_b200.ops.flash_compat import flash_attn_func

pytestmark = pytest.mark.gpu


def _rand(*shape, seed=0):
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA GPU")
    g = torch.Generator(device="cuda").manual_seed(seed + sum(shape))
    return torch.randn(*shape, generator=g, device="cuda", dtype=torch.bfloat16)


# the layouts of [batch, tokens, heads, 128] that are refused, and by which pass (by both routes: O, dK and dV are laid out like
# q, k and v, and a token's heads have to lie side by side there); all others are taken by the native part
REFUSED = {"heads before tokens": "forward", "one head through a transpose": "forward", "k and v laid out differently": "backward"}


class _Recorder:
    """The native part, and whether it took the calls."""

    def __init__(self, host):
        self.host, self.taken = host, []

    def __getattr__(self, name):
        def call(*args):
            r = getattr(self.host, name)(*args)
            self.taken.append((name, r is not None))
            return r
        return call


@pytest.fixture
def native(monkeypatch):
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA GPU")
    assert _lib.host() is not None, "the native host part has not been built"
    rec = _Recorder(_lib.host())
    monkeypatch.setattr(_lib, "_host", [rec])
    return rec


def _layouts():
    """name -> (q, k, v) of [batch, tokens, heads, 128]"""
    packed = _rand(2, 300, 3, 4, 128)
    return {
        "contiguous": (_rand(2, 300, 8, 128), _rand(2, 300, 2, 128, seed=1), _rand(2, 300, 2, 128, seed=2)),
        "packed projection": (packed[:, :, 0], packed[:, :, 1], packed[:, :, 2]),
        "heads before tokens": tuple(_rand(1, 4, 257, 128, seed=i).transpose(1, 2) for i in range(3)),
        "one head through a transpose": (_rand(1, 1, 130, 128).transpose(1, 2), _rand(1, 1, 130, 128, seed=1).transpose(1, 2),
                                         _rand(1, 1, 130, 128, seed=2).transpose(1, 2)),
        "k and v laid out differently": (_rand(1, 200, 2, 128), _rand(1, 200, 2, 128, seed=1), _rand(1, 2, 200, 128, seed=2).transpose(1, 2)),
        "one token": (_rand(3, 1, 2, 128), _rand(3, 1, 2, 128, seed=1), _rand(3, 1, 2, 128, seed=2)),
    }


def _both(monkeypatch, f):
    out = []
    for native in (True, False):
        if not native:
            monkeypatch.setattr(A, "_native", lambda *t: False)
        try:
            out.append(f())
        except Exception as e:          # (what was refused stays refused, in the same words)
            out.append((type(e), str(e)))
    A.check_status()
    return out


@pytest.mark.parametrize("name", ["contiguous", "packed projection", "heads before tokens", "one head through a transpose",
                                  "k and v laid out differently", "one token"])
@pytest.mark.parametrize("pattern", ["causal", "full", "blocks"])
def test_native_calls_equal_python_calls(name, pattern, monkeypatch, native):
    q, k, v = (t.detach().requires_grad_() for t in _layouts()[name])
    n = q.shape[1]
    pat = P.causal(1) if pattern == "causal" else P.full(1) if pattern == "full" else P.causal(n if n < 4 else 1 if n % 2 else 2)
    dense = pat.block_table_int.shape == (1, 1)          # (forwards under a plan have no native part)
    d_o = _rand(*q.shape, seed=9)

    def f():
        o = ua.attention(q, k, v, pat)
        return (o.detach(), *torch.autograd.grad(o, (q, k, v), d_o))

    a, b = _both(monkeypatch, f)
    refused = REFUSED.get(name)
    assert native.taken == ([("dense_forward", refused != "forward")] if dense else []) + (
        [] if refused == "forward" else [("local_backward", refused is None)])
    if refused is not None:
        assert a == b and a[0] is AssertionError
        return
    for i, (x, y) in enumerate(zip(a, b)):
        assert x.shape == y.shape and x.dtype == y.dtype and x.stride() == y.stride()
        if i == 1:          # dQ is summed in arrival order (fp32), then rounded to bf16
            assert (x.float() - y.float()).norm() <= 2 ** -8 * y.float().norm()
        else:
            assert torch.equal(x, y)


@pytest.mark.parametrize("sq,skv", [(1, 700), (40, 40), (300, 100)])
def test_flash_calls(sq, skv, monkeypatch, native):
    q, k, v = _rand(2, sq, 4, 128), _rand(2, skv, 2, 128, seed=1), _rand(2, skv, 2, 128, seed=2)
    a, b = _both(monkeypatch, lambda: flash_attn_func(q, k, v, causal=True, return_attn_probs=True)[:2])
    assert native.taken == [("dense_forward", True)]
    assert all(torch.equal(x, y) for x, y in zip(a, b))


def test_the_same_tensors_are_refused(monkeypatch):
    bf = _rand(1, 64, 2, 128)
    for q, k, v in ((bf.half(), bf.half(), bf.half()), (bf[..., ::2], bf[..., ::2], bf[..., ::2]), (bf, bf[:, :, :1].repeat(1, 1, 3, 1), bf),
                    (bf, bf.float(), bf)):
        a, b = _both(monkeypatch, lambda: flash_attn_func(q, k, v))
        assert a == b and isinstance(a[0], type)


@pytest.mark.parametrize("B,Bk,Bv", [(2, 1, 1), (2, 2, 1), (2, 1, 2)])
def test_missing_sequences_are_refused(B, Bk, Bv, monkeypatch):
    """(on the host: without keys of a sequence its output would be zeros, and its gradients would be written behind dK and dV)"""
    q, k, v = _rand(B, 300, 4, 128), _rand(Bk, 300, 2, 128, seed=1), _rand(Bv, 300, 2, 128, seed=2)
    for f in (lambda: flash_attn_func(q, k, v), lambda: ua.attention(q, k, v, P.causal(1)), lambda: ua.attention(q, k, v, P.causal(2))):
        a, b = _both(monkeypatch, f)
        monkeypatch.undo()
        assert a == b and a[0] is RuntimeError and "sequences" in a[1]
    o, lse = torch.zeros_like(q), torch.zeros(B, 4, 300, device="cuda")
    with pytest.raises((RuntimeError, AssertionError), match="sequences|no room for every key"):
        local_backward(q, k, v, o, lse, q, None, dense=1)


def test_without_the_extension_calls_go_through_python(monkeypatch):
    q, k, v = (_rand(1, 200, 2, 128, seed=i).requires_grad_() for i in range(3))
    d_o = _rand(1, 200, 2, 128, seed=5)
    out = []
    for missing in (False, True):
        if missing:
            monkeypatch.setattr(_lib, "_host", [None])
        o = flash_attn_func(q, k, v, causal=True)
        out.append((o, *torch.autograd.grad(o, (q, k, v), d_o)))
    A.check_status()
    assert all(torch.equal(x, y) for i, (x, y) in enumerate(zip(*out)) if i != 1)          # (dQ is summed in arrival order)


class _Sub(torch.Tensor):
    pass


def test_subclasses_hooks_threads_and_streams():
    q, k, v = (_rand(1, 200, 2, 128, seed=i).requires_grad_() for i in range(3))
    d_o, pat = _rand(1, 200, 2, 128, seed=5), P.causal(1)
    ref = ua.attention(q, k, v, pat)
    want = torch.autograd.grad(ref, (q, k, v), d_o)
    sub = ua.attention(q.as_subclass(_Sub), k, v, pat)
    assert type(sub) is _Sub and torch.equal(sub.as_subclass(torch.Tensor), ref)
    with torch.autograd.graph.saved_tensors_hooks(lambda t: t.cpu(), lambda t: t.cuda()):
        o = ua.attention(q, k, v, pat)
    got = torch.autograd.grad(o, (q, k, v), d_o)
    assert torch.equal(got[1], want[1]) and torch.equal(got[2], want[2])
    bad = []

    def work(i):
        st = torch.cuda.Stream()
        st.wait_stream(torch.cuda.default_stream())
        with torch.cuda.stream(st):
            for _ in range(5):
                a = [t.detach().clone().requires_grad_() for t in (q, k, v)]
                o = ua.attention(*a, pat)
                g = torch.autograd.grad(o, a, d_o)
                if not (torch.equal(o, ref) and torch.equal(g[1], want[1]) and torch.equal(g[2], want[2])):
                    bad.append(i)
            st.synchronize()

    torch.cuda.synchronize()
    threads = [threading.Thread(target=work, args=(i,)) for i in range(4)]
    [t.start() for t in threads]
    [t.join() for t in threads]
    A.check_status()
    assert not bad
