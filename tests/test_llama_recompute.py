"""What a training step of the model no longer computes twice: the last product of a recomputed layer and
the last chunk's logits; and the embedding's gradient kernel."""
import pytest
import torch

from ultraattn_b200 import patterns as P
from ultraattn_b200.models.llama import LlamaConfig, LlamaModel, _LinearBackwardOnly
from ultraattn_b200.ops import elementwise as E


def _model():
    return LlamaModel(LlamaConfig(n_layers=2, hidden=32, n_heads=2, head_dim=16, ffn=48, vocab=40), pattern=P.causal(2), seed=1)


def test_backward_twice_through_a_kept_graph_doubles_the_gradients():
    """The kept logits are overwritten by their gradient: a second backward computes them again."""
    m = _model()
    ids = torch.randint(0, 40, (48,), generator=torch.Generator().manual_seed(0))
    loss = m.loss(ids, ids.roll(-1), chunk=20)
    loss.backward(retain_graph=True)
    once = m.flat_grad.clone()
    loss.backward()
    assert (m.flat_grad - 2 * once).abs().max() < 1e-6 and once.abs().max() > 0


def test_stand_in_for_a_product_has_its_gradients():
    x, w = torch.randn(6, 8, requires_grad=True), torch.randn(5, 8, requires_grad=True)
    y = _LinearBackwardOnly.apply(x, w)
    assert y.shape == (6, 5)
    g = torch.randn(6, 5)
    dx, dw = torch.autograd.grad(y, (x, w), g)
    assert torch.allclose(dx, g @ w, atol=1e-6) and torch.allclose(dw, g.t() @ x, atol=1e-6)


@pytest.mark.gpu
@pytest.mark.parametrize("T,H,V,kind", [(1, 8, 3, "any"), (257, 2056, 50, "any"), (300, 4096, 1000, "any"), (513, 64, 7, "same"),
                                        (100, 128, 5, "int32")])
def test_embedding_gradient_on_the_kernel(T, H, V, kind):
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA GPU")
    g = torch.Generator(device="cuda").manual_seed(T)
    ids = torch.full((T,), V - 1, device="cuda") if kind == "same" else torch.randint(0, V, (T,), device="cuda", generator=g)
    dy = torch.randn(T, H, device="cuda", dtype=torch.bfloat16, generator=g)
    got = E.embedding_bwd(ids.int() if kind == "int32" else ids, dy, V)
    ref = torch.zeros(V, H, device="cuda", dtype=torch.float64).index_add_(0, ids, dy.double())
    # one rounding to bf16 of an fp32 sum
    assert ((got.double() - ref).abs() <= 2 ** -8 * ref.abs() + 1e-5).all()


@pytest.mark.gpu
@pytest.mark.parametrize("T,H,kind", [(33, 8, "runs"), (2000, 64, "runs"), (3001, 2056, "runs"), (6000, 128, "one id"),
                                      (6000, 128, "a third"), (20000, 256, "runs")])
def test_embedding_gradient_of_frequent_ids(T, H, kind):
    """Runs around the length from which on an id's rows are summed in pieces, at every place in a piece."""
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA GPU")
    V, c = 400, E._embedding_chunk(T)
    g = torch.Generator().manual_seed(T)
    if kind == "runs":
        lengths = torch.tensor([c, c + 1, 1, c - 1, 2 * c + 1, 3, 2 * c, 5 * c + 2, c + 1]).repeat(T)
        ids = torch.repeat_interleave(torch.arange(len(lengths)) * 2 % V, lengths)[:T].sort().values     # (odd ids do not occur)
    else:
        ids = torch.randint(0, V, (T,), generator=g)
        ids[torch.rand(T, generator=g) < (1.0 if kind == "one id" else 0.3)] = V - 1
    ids = ids[torch.randperm(T, generator=g)].cuda()
    dy = torch.randn(T, H, generator=g).to("cuda", torch.bfloat16)
    got = E.embedding_bwd(ids, dy, V)
    zero = torch.zeros(V, H, device="cuda", dtype=torch.float64)
    ref, size = zero.index_add(0, ids, dy.double()), zero.index_add(0, ids, dy.double().abs())
    # additions in a row: along a piece, then along the pieces; each rounds to 2^-24 of what has been summed; bf16 once
    assert ((got.double() - ref).abs() <= 2 ** -8 * ref.abs() + (c + T // c + 2) * 2 ** -24 * size).all()
    assert torch.equal(got, E.embedding_bwd(ids, dy, V))
