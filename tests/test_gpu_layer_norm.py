"""The short-row LayerNorm kernels (forward, backward) against torch.nn.functional.layer_norm in fp64."""
import pytest
import torch

pytestmark = pytest.mark.gpu

TOL = 1e-5   # relative to the largest reference value, fp32


def _reference(x, w, b, dy, eps):
    xd, wd, bd = (t.detach().double().cpu().requires_grad_() for t in (x, w, b))
    y = torch.nn.functional.layer_norm(xd, (xd.shape[-1],), wd, bd, eps)
    y.backward(dy.double().cpu())
    return y.detach(), xd.grad, wd.grad, bd.grad


def _close(got, ref, tol=TOL):
    scale = float(ref.abs().max()) if ref.numel() else 0.0
    err = float((got.double().cpu() - ref).abs().max()) if ref.numel() else 0.0
    return err <= tol * max(scale, 1e-30), (err, scale)


@pytest.mark.parametrize("hidden", [4, 8, 24, 32, 64, 80, 128, 256, 512])
@pytest.mark.parametrize("rows", [1, 5, 257, 4099])
def test_layer_norm_forward_and_backward_match_torch(rows, hidden):
    from torchgt_b200.layer_norm import LayerNorm
    gen = torch.Generator().manual_seed(rows * 1000 + hidden)
    x = (torch.randn(rows, hidden, generator=gen) * 2 + 0.5).cuda().requires_grad_()
    dy = torch.randn(rows, hidden, generator=gen).cuda()
    mod = LayerNorm(hidden).cuda()
    with torch.no_grad():
        mod.weight.copy_(torch.randn(hidden, generator=gen).cuda())
        mod.bias.copy_(torch.randn(hidden, generator=gen).cuda())
    y = mod(x)
    y.backward(dy)
    ref_y, ref_dx, ref_dw, ref_db = _reference(x, mod.weight, mod.bias, dy, mod.eps)
    for got, ref in ((y, ref_y), (x.grad, ref_dx), (mod.weight.grad, ref_dw), (mod.bias.grad, ref_db)):
        ok, info = _close(got, ref)
        assert ok, info


def test_layer_norm_benchmark_shape_three_dimensional_input_and_reproducibility():
    """[1, 64001, 64] as the encoder layers see it; two runs give the same bits (no atomics)."""
    from torchgt_b200.layer_norm import LayerNorm
    gen = torch.Generator().manual_seed(11)
    x0 = torch.randn(1, 64001, 64, generator=gen).cuda()
    dy = torch.randn(1, 64001, 64, generator=gen).cuda()
    mod = LayerNorm(64).cuda()
    with torch.no_grad():
        mod.weight.copy_(torch.rand(64, generator=gen).cuda() + 0.5)
        mod.bias.copy_(torch.randn(64, generator=gen).cuda())
    runs = []
    for _ in range(2):
        x = x0.clone().requires_grad_()
        mod.zero_grad()
        y = mod(x)
        y.backward(dy)
        runs.append((y.detach().clone(), x.grad.clone(), mod.weight.grad.clone(), mod.bias.grad.clone()))
    for a, b in zip(*runs):
        assert torch.equal(a, b)
    ref = _reference(x0, mod.weight, mod.bias, dy, mod.eps)
    for got, want in zip(runs[0], ref):
        ok, info = _close(got, want.view_as(got.cpu()))
        assert ok, info


def test_layer_norm_falls_back_to_torch_for_what_the_kernels_do_not_cover():
    from torchgt_b200.layer_norm import LayerNorm
    for mod, x in ((LayerNorm(6).cuda(), torch.randn(3, 6).cuda()),                       # not a multiple of 4
                   (LayerNorm(64).cuda().double(), torch.randn(3, 64).cuda().double()),   # fp64
                   (LayerNorm(64, elementwise_affine=False).cuda(), torch.randn(3, 64).cuda()),
                   (LayerNorm((2, 32)).cuda(), torch.randn(3, 2, 32).cuda())):
        ref = torch.nn.functional.layer_norm(x, mod.normalized_shape, mod.weight, mod.bias, mod.eps)
        assert torch.equal(mod(x), ref)


def test_layer_norm_argument_errors_come_back_as_codes():
    import ctypes
    from torchgt_b200 import _cabi
    lib = _cabi.load()
    x = torch.randn(4, 64).cuda()
    nb = ctypes.c_size_t()
    assert lib.tgt_layer_norm_bwd_scratch_bytes(4, 6, ctypes.byref(nb)) == 3
    assert lib.tgt_layer_norm_fwd(x.data_ptr(), None, None, 1e-5, 4, 64, x.data_ptr(), None, None) == 1
    assert lib.tgt_layer_norm_fwd(x.data_ptr(), x.data_ptr(), x.data_ptr(), 1e-5, 4, 1024, x.data_ptr(), None,
                                  None) == 3
    assert lib.tgt_layer_norm_bwd(x.data_ptr(), x.data_ptr(), x.data_ptr(), x.data_ptr(), 4, 64, x.data_ptr(),
                                  x.data_ptr(), x.data_ptr(), None, 0, None) == 4


def test_layer_norm_and_linear_accept_views_that_start_off_a_16_byte_boundary():
    """A contiguous view four bytes into its storage cannot be read 16 bytes at a time: the modules copy it."""
    from torchgt_b200.layer_norm import LayerNorm
    from torchgt_b200.linear import Linear
    torch.manual_seed(9)
    rows = 300
    flat = torch.randn(rows * 64 + 1, device="cuda")
    x = flat[1:].view(rows, 64)
    assert x.data_ptr() % 16 != 0 and x.is_contiguous()
    ln, lin = LayerNorm(64).cuda(), Linear(64, 64).cuda()
    xa = x.detach().requires_grad_()
    y = lin(ln(xa))
    gflat = torch.randn(rows * 64 + 1, device="cuda")
    y.backward(gflat[1:].view(rows, 64))
    xd = x.detach().double().requires_grad_()
    ref = torch.nn.functional.linear(
        torch.nn.functional.layer_norm(xd, (64,), ln.weight.double(), ln.bias.double(), ln.eps),
        lin.weight.double(), lin.bias.double())
    ref.backward(gflat[1:].view(rows, 64).double())
    tol = 2e-3 if torch.backends.cuda.matmul.allow_tf32 else 1e-5
    assert _close(y, ref.detach().cpu(), tol)[0]
    assert _close(xa.grad, xd.grad.cpu(), tol)[0]


@pytest.mark.parametrize("hidden", [4, 24, 64, 512])
@pytest.mark.parametrize("rows", [1, 257, 4099])
@pytest.mark.parametrize("use", ["both", "norm", "sum"])
def test_residual_addition_inside_the_norm_gives_the_bits_of_the_two_operations(rows, hidden, use):
    from torchgt_b200.layer_norm import LayerNorm, add_layer_norm
    gen = torch.Generator().manual_seed(rows + hidden)
    x, r, dy, ds = (torch.randn(rows, hidden, generator=gen).cuda() for _ in range(4))
    norm = LayerNorm(hidden).cuda()
    with torch.no_grad():
        norm.weight.copy_(torch.randn(hidden, generator=gen).cuda())

    def run(fused):
        norm.zero_grad()
        a, b = x.clone().requires_grad_(), r.clone().requires_grad_()
        y, s = add_layer_norm(a, b, norm) if fused else (norm(a + b), None)
        if not fused:
            s = a + b
        outs = {"both": ((y, dy), (s, ds)), "norm": ((y, dy),), "sum": ((s, ds),)}[use]
        torch.autograd.backward([o for o, _ in outs], [g for _, g in outs])
        return [y, s, a.grad, b.grad, norm.weight.grad, norm.bias.grad]

    for got, want in zip(run(True), run(False)):
        assert (got is None and want is None) or torch.equal(got, want)
    with torch.no_grad():
        y, s = add_layer_norm(x, r, norm, want_sum=False)
        assert s is None and torch.equal(y, norm(x + r))


def test_residual_addition_leaves_hooked_and_uncovered_norms_to_their_own_call():
    from torchgt_b200.layer_norm import LayerNorm, add_layer_norm
    norm = LayerNorm(64).cuda()
    x, r = torch.randn(9, 64, device="cuda"), torch.randn(9, 64, device="cuda")
    seen = []
    handle = norm.register_forward_hook(lambda m, args, out: seen.append(args[0]))
    y, s = add_layer_norm(x, r, norm)
    assert len(seen) == 1 and torch.equal(seen[0], x + r) and torch.equal(s, x + r)
    handle.remove()
    assert torch.equal(add_layer_norm(x, r, norm)[0], y)
    wide = LayerNorm(64).cuda().double()
    assert torch.equal(add_layer_norm(x.double(), r.double(), wide)[0], wide(x.double() + r.double()))


@pytest.mark.parametrize("with_residual", [False, True])
def test_saved_tensor_hooks_see_everything_the_backward_keeps(with_residual):
    """Offloading what is saved to the host leaves the gradients' bits as they are."""
    from torchgt_b200.layer_norm import LayerNorm, add_layer_norm
    norm = LayerNorm(64).cuda()
    x, r = (torch.randn(37, 64, device="cuda", requires_grad=True) for _ in range(2))
    inputs = [x, norm.weight, norm.bias] + ([r] if with_residual else [])
    call = lambda: add_layer_norm(x, r, norm)[0] if with_residual else norm(x)
    want = torch.autograd.grad(call().square().sum(), inputs)
    shapes = []

    def pack(t):
        shapes.append(tuple(t.shape))
        return t.detach().cpu()

    with torch.autograd.graph.saved_tensors_hooks(pack, lambda t: t.cuda()):
        y = call()
    assert sorted(shapes) == sorted([(37, 64), (64,), (37, 2)])      # the norm's input, its weight, mean and deviation
    for a, b in zip(torch.autograd.grad(y.square().sum(), inputs), want):
        assert torch.equal(a, b)


@pytest.mark.parametrize("shape", [(3, 64), (2, 17, 96)])
@pytest.mark.parametrize("outputs", ["norm", "sum", "both", "alone"])
def test_second_order_gradients(shape, outputs):
    """A gradient penalty against torch's norm in 64 bits, through the norm and through the residual stream.  Tolerance:
    about ten roundings of 6e-8 per value, sums over up to 96 columns and three nested means: 1e-5 of the largest value."""
    from torchgt_b200.layer_norm import LayerNorm, add_layer_norm
    gen = torch.Generator().manual_seed(shape[-1])
    x, r, a, b = (torch.randn(shape, generator=gen, dtype=torch.float64) for _ in range(4))
    w, c = torch.rand(shape[-1], generator=gen, dtype=torch.float64) + 0.5, torch.randn(shape[-1], generator=gen, dtype=torch.float64)

    def penalty(call, x, r, a, b, norm):
        y, s = call(x, r, norm)
        terms = {"norm": [y * a], "sum": [s.square() * b], "both": [y.sin() * a, s.square() * b], "alone": [y.sin() * a]}[outputs]
        first = torch.autograd.grad(sum(t.sum() for t in terms), (x, r, norm.weight), create_graph=True, allow_unused=True)
        kept = [g for g in first if g is not None]
        wrt = (x, r, norm.weight)
        second = torch.autograd.grad(sum(g.square().sum() for g in kept) + kept[0].sin().sum(), wrt, allow_unused=True)
        return [*first, *second]

    def torch_call(x, r, norm):
        s = x if outputs == "alone" else x + r
        return norm(s), s

    def own_call(x, r, norm):
        return (norm(x), x) if outputs == "alone" else add_layer_norm(x, r, norm)

    results = []
    for call, norm, device, dtype in ((torch_call, torch.nn.LayerNorm(shape[-1]), "cpu", torch.float64),
                                      (own_call, LayerNorm(shape[-1]), "cuda", torch.float32)):
        norm = norm.to(device, dtype)
        with torch.no_grad():
            norm.weight.copy_(w)
            norm.bias.copy_(c)
        xs = [t.to(device, dtype) for t in (x, r, a, b)]
        results.append(penalty(call, xs[0].requires_grad_(), xs[1].requires_grad_(), xs[2], xs[3], norm))
    for got, want in zip(results[1], results[0]):
        assert (got is None) == (want is None)
        if want is not None:
            assert float((got.double().cpu() - want).abs().max()) <= 1e-5 * float(want.abs().max()) + 1e-12
