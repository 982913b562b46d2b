"""The projections of one input as one node and the feed-forward block as one node against the modules in fp64, and the
calls that have to go through the modules."""
import pytest
import torch
from torch import nn

pytestmark = pytest.mark.gpu

# 2-norm, relative: chains of two products, each below 1e-6 (test_gpu_linear_tensor_cores.py; the library's sums of up to 512
# terms, rounded to nearest, below 512^0.5 * 2^-24).  A product without the third piece of an operand is 2.6e-6 off.
TOL = 2e-6


@pytest.fixture(autouse=True)
def full_fp32():
    before = torch.backends.cuda.matmul.allow_tf32
    torch.backends.cuda.matmul.allow_tf32 = False
    yield
    torch.backends.cuda.matmul.allow_tf32 = before


def _rel(got, ref):
    return float((got.detach().double() - ref.detach()).norm() / ref.detach().norm().clamp_min(1e-30))


def _layers(n, inp, out, bias=True):
    from torchgt_b200.linear import Linear
    return [Linear(inp, out, bias=bias).cuda() for _ in range(n)]


def _double(module):
    ref = nn.Linear(module.in_features, module.out_features, bias=module.bias is not None).cuda().double()
    ref.load_state_dict({k: v.double() for k, v in module.state_dict().items()})
    return ref


def _compare(outs, refs, x, x64, modules, modules64, extra=(), extra64=()):
    gen = torch.Generator(device="cuda").manual_seed(1)
    dy = [torch.randn(o.shape, generator=gen, device="cuda") for o in outs]
    leaves = [x, *extra, *(p for m in modules for p in m.parameters())]
    leaves64 = [x64, *extra64, *(p for m in modules64 for p in m.parameters())]
    for got, ref in zip(outs, refs):
        assert got.shape == ref.shape and _rel(got, ref) < TOL
    got = torch.autograd.grad(outs, leaves, dy)
    ref = torch.autograd.grad(refs, leaves64, [d.double() for d in dy])
    for g, r in zip(got, ref):
        assert g.shape == r.shape and _rel(g, r) < TOL


@pytest.mark.parametrize("bias", [True, False])
@pytest.mark.parametrize("shape,out", [((1023, 64), 64), ((1024, 64), 64), ((3, 700, 64), 64), ((1, 2689, 64), 64), ((30001, 128), 64), ((10300, 64), 100)])
def test_three_projections(shape, out, bias):
    from torchgt_b200.linear import linear3
    torch.manual_seed(shape[-2])
    layers = _layers(3, shape[-1], out, bias)
    x = torch.randn(shape, device="cuda").requires_grad_()
    y = linear3(x, *layers)
    if x.numel() // shape[-1] >= 1024:
        assert "NarrowLinear3" in y[0].grad_fn.name() and y[0].grad_fn is y[2].grad_fn
    x64, layers64 = x.detach().double().requires_grad_(), [_double(m) for m in layers]
    _compare(y, [m(x64) for m in layers64], x, x64, layers, layers64)
    with torch.no_grad():
        assert all(torch.equal(a, b.detach()) for a, b in zip(linear3(x, *layers), y))


@pytest.mark.parametrize("act", ["relu", "gelu"])
@pytest.mark.parametrize("residual", [True, False])
@pytest.mark.parametrize("shape,mid", [((1023, 64), 64), ((1024, 64), 64), ((1, 2000, 64), 128), ((20001, 64), 128), ((10300, 128), 64)])
def test_feed_forward(shape, mid, residual, act):
    from torchgt_b200.linear import feed_forward
    torch.manual_seed(shape[-2] + mid)
    layers = _layers(1, shape[-1], mid) + _layers(1, mid, shape[-1])
    x = torch.randn(shape, device="cuda").requires_grad_()
    r = torch.randn(shape, device="cuda").requires_grad_() if residual else None
    y = feed_forward(x, *layers, act, r)
    if x.numel() // shape[-1] >= 1024:
        assert "FeedForward" in y.grad_fn.name()
    x64, layers64 = x.detach().double().requires_grad_(), [_double(m) for m in layers]
    r64 = r.detach().double().requires_grad_() if residual else None
    fn = torch.relu if act == "relu" else nn.functional.gelu
    ref = layers64[1](fn(layers64[0](x64)))
    _compare([y], [ref + r64 if residual else ref], x, x64, layers, layers64, [r] if residual else [], [r64] if residual else [])
    with torch.no_grad():
        assert torch.equal(feed_forward(x, *layers, act, r), y.detach())


@pytest.mark.parametrize("tf32,width", [(False, 512), (True, 512), (True, 256)])
def test_wide_and_tf32_products_of_the_blocks_are_the_librarys(tf32, width):
    """Where the library is ahead: the same bits, forward and input gradient."""
    from torchgt_b200.linear import feed_forward, linear3
    torch.backends.cuda.matmul.allow_tf32 = tf32
    torch.manual_seed(width)
    layers = _layers(3, width, width)
    x, dy = torch.randn(2048, width, device="cuda").requires_grad_(), torch.randn(2048, width, device="cuda")
    y, z = linear3(x, *layers), feed_forward(x, layers[0], layers[1], "gelu", x)
    with torch.no_grad():
        refs = [nn.functional.linear(x, m.weight, m.bias) for m in layers]
        ref = x + nn.functional.linear(nn.functional.gelu(refs[0]), layers[1].weight, layers[1].bias)
        dx = dy @ layers[2].weight
    assert torch.equal(z, ref) and (not tf32 or all(torch.equal(a, b) for a, b in zip(y, refs)))
    assert torch.equal(torch.autograd.grad(y[2], x, dy)[0], dx)


@pytest.mark.parametrize("rows,inp,out,bias", [(1023, 64, 64, True), (12287, 64, 64, False), (12288, 64, 64, False),
                                               (10112, 256, 64, True), (10113, 256, 64, True), (5000, 384, 128, True),
                                               (5000, 448, 128, True), (16257, 64, 28, True), (8129, 128, 320, False), (8065, 512, 448, True)])
@pytest.mark.parametrize("tf32", [False, True])
def test_both_sides_of_the_lines_between_the_kernels(rows, inp, out, bias, tf32):
    from torchgt_b200.linear import linear3
    torch.manual_seed(rows + out)
    layers = _layers(3, inp, out, bias)
    x, dy = torch.randn(rows, inp, device="cuda").requires_grad_(), torch.randn(rows, out, device="cuda")
    x64, layers64 = x.detach().double().requires_grad_(), [_double(m) for m in layers]
    torch.backends.cuda.matmul.allow_tf32 = tf32
    for ys, refs, ms in ((linear3(x, *layers), [m(x64) for m in layers64], range(3)), ([layers[0](x)], [layers64[0](x64)], [0])):
        got = [*ys, *torch.autograd.grad(ys, [x, *(p for i in ms for p in layers[i].parameters())], [dy] * len(ys))]
        torch.backends.cuda.matmul.allow_tf32 = False
        want = [*refs, *torch.autograd.grad(refs, [x64, *(p for i in ms for p in layers64[i].parameters())],
                                            [dy.double()] * len(ys))]
        torch.backends.cuda.matmul.allow_tf32 = tf32
        for i, (a, b) in enumerate(zip(got, want)):      # TF32 rounds operands to 11 bits; parameter gradients stay fp32
            assert _rel(a, b) < (1e-3 if tf32 and i <= len(ys) else TOL)


def test_a_missing_gradient_and_gradients_nobody_wants():
    from torchgt_b200.linear import feed_forward, linear3
    torch.manual_seed(0)
    layers = _layers(3, 64, 64)
    x = torch.randn(1500, 64, device="cuda").requires_grad_()
    q, k, v = linear3(x, *layers)
    (q.sum() + 2 * v.sum()).backward()
    assert layers[1].weight.grad is None or not layers[1].weight.grad.any()
    ref = (layers[0].weight.detach().double().sum(0) + 2 * layers[2].weight.detach().double().sum(0)).expand(1500, 64)
    assert _rel(x.grad, ref) < TOL
    layers[0].weight.requires_grad_(False)
    layers[0].bias.requires_grad_(False)
    y = feed_forward(x.detach(), layers[0], layers[1], "relu")
    layers[1].weight.grad = None
    y.sum().backward()
    assert layers[1].weight.grad is not None


def test_second_order_gradients():
    from torchgt_b200.linear import feed_forward, linear3
    torch.manual_seed(1)
    layers = _layers(3, 64, 64)
    layers64 = [_double(m) for m in layers]
    x = torch.randn(1100, 64, device="cuda").requires_grad_()
    x64 = x.detach().double().requires_grad_()
    for act, fn in (("relu", torch.relu), ("gelu", nn.functional.gelu)):
        y, ref = feed_forward(x, layers[0], layers[1], act, x), x64 + layers64[1](fn(layers64[0](x64)))
        got, want = [], []
        for out, leaf, w, into in ((y, x, layers[0].weight, got), (ref, x64, layers64[0].weight, want)):
            g, = torch.autograd.grad((out * out).sum(), leaf, create_graph=True)
            into.extend(torch.autograd.grad((g * g).sum(), [leaf, w]))
        assert all(_rel(a, b) < 1e-5 for a, b in zip(got, want))
    g, = torch.autograd.grad(sum(t.sum() for t in linear3(x, *layers)), x, create_graph=True)
    dw, = torch.autograd.grad((g * g).sum(), layers[1].weight)
    total = sum(m.weight.detach().double().sum(0) for m in layers)
    assert _rel(dw, (2 * 1100 * total).expand(64, 64)) < 1e-5


@pytest.mark.parametrize("bias", [True, False])
@pytest.mark.parametrize("block", ["linear", "linear3"])
def test_second_order_gradients_through_the_parameters_gradients(block, bias):
    """What is built on dW and db reaches the input, the weights and the gradient that came in; dW has the same bits as without
    create_graph."""
    from torchgt_b200.linear import linear3
    torch.manual_seed(6)
    layers = _layers(3, 64, 64, bias)
    x = (0.3 * torch.randn(1100, 64, device="cuda")).requires_grad_()
    x64, layers64 = x.detach().double().requires_grad_(), [_double(m) for m in layers]
    got, want = [], []
    for leaf, mods, into in ((x, layers, got), (x64, layers64, want)):
        if block == "linear":
            loss = (mods[0](leaf) ** 2).sum()
            mods = mods[:1]
        else:
            q, k, v = linear3(leaf, *mods) if leaf is x else [m(leaf) for m in mods]
            loss = (q * k).sum() + (v * v * v).sum()
        params = [p for m in mods for p in m.parameters()]
        first = torch.autograd.grad(loss, params, create_graph=True)
        assert all(g.requires_grad for g in first)
        if leaf is x:
            assert all(torch.equal(a, b) for a, b in zip(first, torch.autograd.grad(loss, params, retain_graph=True)))
        into.extend(torch.autograd.grad(sum((g * g).sum() for g in first), [leaf, *params]))
    # chains of four products of at most 1,100 terms of mixed sign
    assert all(_rel(a, b) < 2e-5 for a, b in zip(got, want))


def test_infinities_and_nan_pass_as_through_the_modules():
    from torchgt_b200.linear import feed_forward, linear3
    torch.manual_seed(2)
    layers = _layers(3, 64, 64)
    for rows in (1300, 10300):
        x = torch.randn(rows, 64, device="cuda")
        x[3, 7], x[11, 0] = float("inf"), float("nan")
        with torch.no_grad():
            refs = [nn.functional.linear(x, m.weight, m.bias) for m in layers]
            outs = linear3(x, *layers)
            for act, fn in (("relu", torch.relu), ("gelu", nn.functional.gelu)):
                outs = [*outs, feed_forward(x, layers[0], layers[1], act)]
                refs.append(nn.functional.linear(fn(refs[0]), layers[1].weight, layers[1].bias))
        for y, ref in zip(outs, refs):
            assert torch.equal(y.isnan(), ref.isnan()) and torch.equal(y.isinf(), ref.isinf())


def test_layers_that_differ_and_observed_modules_are_called_one_by_one():
    from torchgt_b200.linear import Linear, feed_forward, linear3, passes_through
    torch.manual_seed(3)
    a, b = _layers(2, 64, 64)
    c = Linear(64, 128).cuda()
    x = torch.randn(10, 64, device="cuda")
    outs = linear3(x, a, b, c)
    assert [tuple(o.shape) for o in outs] == [(10, 64), (10, 64), (10, 128)]
    seen = []
    handle = a.register_forward_hook(lambda m, i, o: seen.append(m))
    linear3(x, a, b, b)
    assert seen == [a] and feed_forward(x, a, b, "relu") is None
    handle.remove()
    assert feed_forward(x, a, b, "relu") is not None
    assert feed_forward(x, Linear(64, 64, bias=False).cuda(), b, "relu") is None
    y = feed_forward(x, Linear(64, 44).cuda(), Linear(44, 64).cuda(), "gelu", x)       # no kernel: 44 wide in between
    assert y.shape == x.shape
    with pytest.raises(RuntimeError):
        feed_forward(x, a, b, "tanh")
    with torch.autocast("cuda", dtype=torch.bfloat16):
        assert feed_forward(x, a, b, "relu") is None and linear3(x, a, b, b)[0].dtype == torch.bfloat16
    z = torch.func.vmap(lambda t: linear3(t, a, b, b)[1])(torch.randn(3, 5, 64, device="cuda"))
    assert z.shape == (3, 5, 64)
    drop = nn.Dropout(0.1).train()
    assert not passes_through(drop) and passes_through(drop.eval()) and passes_through(nn.Dropout(0.0).train())
