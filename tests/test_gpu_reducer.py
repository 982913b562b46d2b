"""The flat-gradient averager when a model runs its branches on several CUDA streams."""
import pytest
import torch
from torch import nn

pytestmark = pytest.mark.gpu

DELAY = 100_000_000   # clock cycles, about 50 ms: far longer than the host takes to enqueue a step


class _LateGradient(torch.autograd.Function):
    """Identity whose gradient is handed on after a long wait on the stream it arrives on."""

    @staticmethod
    def forward(ctx, x):
        return x.clone()

    @staticmethod
    def backward(ctx, grad):
        torch.cuda._sleep(DELAY)
        return grad * 1


class _Branches(nn.Module):
    def __init__(self):
        super().__init__()
        self.main, self.side = nn.Linear(64, 32), nn.Linear(64, 32)
        self.stream = torch.cuda.Stream()

    def forward(self, x):
        y = self.main(x)
        self.stream.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(self.stream):          # built last, so its backward is enqueued first
            z = _LateGradient.apply(self.side(x))
        torch.cuda.current_stream().wait_stream(self.stream)
        return y + z


class _Work:
    def wait(self):
        pass


@pytest.mark.parametrize("world", [1, 2])
def test_gradients_of_another_stream_are_complete_when_they_are_read(world, monkeypatch):
    """With two ranks the all-reduce is replaced by a copy of what it would send, on the stream it is called on."""
    from torchgt_b200.gt_sp import reducer as module
    sent = []
    monkeypatch.setattr(module.dist, "all_reduce", lambda t, **_: (sent.append(t.clone()), _Work())[1])
    torch.manual_seed(0)
    model = _Branches().cuda()
    reducer = module.Reducer(world_size=world).init(model)
    for step in range(4):                             # step 0 learns which parameters get gradients
        x = torch.randn(1000, 64, device="cuda")
        reducer.prepare()
        model(x).square().sum().backward()
        reducer.synchronize()
        got = [p.grad.clone() for p in model.parameters()]
        flat = sent[-1] if world > 1 else reducer.flat_gradients
        views = [flat[v.storage_offset():v.storage_offset() + v.numel()].view_as(v) for v in reducer._views]
        for p in model.parameters():
            p.grad = None
        model(x).square().sum().backward()
        for p, g, v in zip(model.parameters(), got, views):
            assert torch.equal(g, v)
            assert torch.allclose(g * world, p.grad, rtol=1e-5, atol=1e-5 * float(p.grad.abs().max())), step
        torch.cuda.synchronize()
