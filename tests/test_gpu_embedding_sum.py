"""Summed embedding vectors and the table's gradient against fp64 (sums of fp32 values: relative 2-norm error of a sum of n
terms below n^0.5 * 2^-24 of their norm; cancellation aside, 1e-5 covers the longest segment here)."""
import pytest
import torch
from torch import nn

pytestmark = pytest.mark.gpu

TOL = 1e-5


def _rel(got, ref):
    return float((got.detach().double() - ref.detach()).norm() / ref.detach().norm().clamp_min(1e-30))


@pytest.mark.parametrize("padding", [None, 0, 5])
@pytest.mark.parametrize("n,hidden,shape", [(7, 64, (1, 1)), (7, 64, (3, 1, 5)), (7000, 64, (4, 5000, 5)), (64, 32, (2, 900, 3)),
                                            (100000, 128, (1, 300, 9)), (6, 64, (60000, 2))])
def test_sum_and_table_gradient(n, hidden, shape, padding):
    from torchgt_b200.linear import embedding_sum
    torch.manual_seed(n + hidden)
    table = nn.Embedding(n, hidden, padding_idx=padding).cuda()
    gen = torch.Generator().manual_seed(1)
    ids = torch.randint(0, n, shape, generator=gen)
    ids[ids % 3 == 0] = 0                       # a hub
    ids = ids.cuda()
    y = embedding_sum(table, ids)
    assert "EmbeddingSum" in y.grad_fn.name()
    ref = nn.Embedding(n, hidden, padding_idx=padding).cuda().double()
    ref.load_state_dict({k: v.double() for k, v in table.state_dict().items()})
    y64 = ref(ids).sum(dim=-2)
    assert y.shape == y64.shape and (_rel(y, y64) < TOL or not y64.any())
    dy = torch.randn(y.shape, device="cuda")
    g, = torch.autograd.grad(y, table.weight, dy, retain_graph=True)
    again, = torch.autograd.grad(y, table.weight, dy)
    g64, = torch.autograd.grad(y64, ref.weight, dy.double())
    assert torch.equal(g, again) and (_rel(g, g64) < TOL or not g64.any())
    assert torch.equal(g.abs().sum(1) == 0, g64.abs().sum(1) == 0)
    with torch.no_grad():
        assert torch.equal(embedding_sum(table, ids), y)


def test_calls_that_go_through_the_module():
    from torchgt_b200.linear import embedding_sum
    ids = torch.randint(0, 9, (5, 3), device="cuda")
    for table in (nn.Embedding(9, 48), nn.Embedding(9, 64, max_norm=1.0), nn.Embedding(9, 64, scale_grad_by_freq=True),
                  nn.Embedding(9, 64).double()):
        table = table.cuda()
        y = embedding_sum(table, ids)
        assert torch.equal(y, table(ids).sum(dim=-2))
        y.sum().backward()
    table = nn.Embedding(9, 64).cuda()
    assert torch.equal(embedding_sum(table, ids.int()), table(ids).sum(dim=-2))
    assert embedding_sum(table, ids[:0]).shape == (0, 64) and embedding_sum(table, ids[:, :0]).shape == (5, 64)
    flipped = ids.t().contiguous().t()           # not contiguous
    assert _rel(embedding_sum(table, flipped), table(ids).double().sum(dim=-2)) < TOL
    y = embedding_sum(table, ids)
    dy = torch.randn(5, 64, device="cuda", requires_grad=True)
    g, = torch.autograd.grad(y, table.weight, dy, create_graph=True)
    back, = torch.autograd.grad(g.sum(), dy)
    assert torch.allclose(back, torch.full_like(back, 3.0))


def test_many_gradients_at_once():
    from torchgt_b200.linear import embedding_sum
    torch.manual_seed(8)
    emb = torch.nn.Embedding(50, 64, padding_idx=0).cuda()
    ids = torch.randint(0, 50, (7, 3), device="cuda")
    dy = torch.randn(4, 7, 64, device="cuda")
    got, = torch.autograd.grad(embedding_sum(emb, ids), emb.weight, dy, is_grads_batched=True)
    y = emb(ids).sum(-2)
    for g, d in zip(got, dy):
        ref, = torch.autograd.grad(y, emb.weight, d, retain_graph=True)
        assert (g - ref).abs().max() <= 1e-5 * ref.abs().max()
