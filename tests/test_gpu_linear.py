"""The weight/bias-gradient kernel of the narrow linear layers against fp64 products."""
import pytest
import torch

pytestmark = pytest.mark.gpu

TOL = 1e-5   # relative to the largest reference value; fp32 FMA sums over the rows


def _err(got, ref):
    ref = ref.double().cpu()
    return float((got.double().cpu() - ref).abs().max() / ref.abs().max().clamp_min(1e-30))


@pytest.mark.parametrize("in_features,out_features", [(64, 64), (128, 64), (64, 128), (192, 64), (64, 40), (128, 4),
                                                      (64, 100)])
@pytest.mark.parametrize("rows", [1, 31, 33, 4099, 64001])
def test_weight_and_bias_gradients_match_fp64(rows, in_features, out_features):
    from torchgt_b200.linear import wgrad
    gen = torch.Generator().manual_seed(rows + in_features * 7 + out_features)
    dy = torch.randn(rows, out_features, generator=gen).cuda()
    x = torch.randn(rows, in_features, generator=gen).cuda()
    dw, db = wgrad(dy, x)
    dw2, db2 = wgrad(dy, x)
    assert torch.equal(dw, dw2) and torch.equal(db, db2)          # fixed summation order
    assert _err(dw, dy.double().t() @ x.double()) < TOL
    assert _err(db, dy.double().sum(0)) < TOL
    dw3, none = wgrad(dy, x, with_bias=False)
    assert none is None and torch.equal(dw3, dw)


def test_linear_module_matches_nn_linear_and_keeps_its_state_dict():
    from torchgt_b200.linear import Linear
    torch.manual_seed(3)
    ours, ref = Linear(64, 128).cuda(), torch.nn.Linear(64, 128).cuda().double()
    assert set(ours.state_dict()) == set(ref.state_dict())
    ref.load_state_dict({k: v.double() for k, v in ours.state_dict().items()})
    x = torch.randn(1, 5000, 64, device="cuda")
    dy = torch.randn(1, 5000, 128, device="cuda")
    xa, xb = x.clone().requires_grad_(), x.double().requires_grad_()
    ya, yb = ours(xa), ref(xb)
    ya.backward(dy)
    yb.backward(dy.double())
    tf32 = torch.backends.cuda.matmul.allow_tf32
    tol = 2e-3 if tf32 else 1e-5        # the forward product and the input gradient are library GEMMs
    assert _err(ya, yb) < tol and _err(xa.grad, xb.grad) < tol
    assert _err(ours.weight.grad, ref.weight.grad) < TOL and _err(ours.bias.grad, ref.bias.grad) < TOL


def test_linear_falls_back_to_torch_for_what_the_kernel_does_not_cover():
    from torchgt_b200.linear import Linear
    torch.manual_seed(4)
    for mod, x in ((Linear(64, 42).cuda(), torch.randn(9, 64).cuda()),               # 42 outputs
                   (Linear(24, 64).cuda(), torch.randn(9, 24).cuda()),               # 24 inputs
                   (Linear(64, 64).cuda().double(), torch.randn(9, 64).cuda().double()),
                   (Linear(64, 64, bias=False).cuda(), torch.randn(9, 64).cuda())):
        x = x.requires_grad_()
        y = mod(x)
        y.sum().backward()
        ref = torch.nn.functional.linear(x, mod.weight, mod.bias)
        assert torch.equal(y, ref)
        assert mod.weight.grad is not None and x.grad is not None


def test_linear_wgrad_argument_errors_come_back_as_codes():
    import ctypes
    from torchgt_b200 import _cabi
    lib = _cabi.load()
    t = torch.randn(8, 64).cuda()
    nb = ctypes.c_size_t()
    assert lib.tgt_linear_wgrad_scratch_bytes(8, 40, 64, ctypes.byref(nb)) == 3       # TGT_ERR_UNSUPPORTED
    assert lib.tgt_linear_wgrad_scratch_bytes(8, 64, 42, ctypes.byref(nb)) == 3
    assert lib.tgt_linear_wgrad(t.data_ptr(), t.data_ptr(), 8, 64, 64, None, None, None, 0, None) == 1   # INVALID
    assert lib.tgt_linear_wgrad(t.data_ptr(), t.data_ptr(), 8, 64, 64, t.data_ptr(), None, None, 0, None) == 4   # WORKSPACE


@pytest.fixture(params=[False, True], ids=["fp32", "tf32"])
def tf32(request):
    before = torch.backends.cuda.matmul.allow_tf32
    torch.backends.cuda.matmul.allow_tf32 = request.param
    yield request.param
    torch.backends.cuda.matmul.allow_tf32 = before


@pytest.mark.parametrize("in_features,out_features", [(64, 64), (64, 128), (128, 64), (64, 40), (192, 4), (64, 100)])
@pytest.mark.parametrize("rows", [1, 1025, 4097, 40000])
def test_forward_and_input_gradient_match_fp64(rows, in_features, out_features, tf32):
    """Both tile heights, partial tiles of rows and columns, one and several reduction chunks."""
    from torchgt_b200.linear import linear
    gen = torch.Generator().manual_seed(rows + in_features + 3 * out_features)
    x = torch.randn(rows, in_features, generator=gen).cuda().requires_grad_()
    w = torch.randn(out_features, in_features, generator=gen).cuda().requires_grad_()
    b = torch.randn(out_features, generator=gen).cuda().requires_grad_()
    dy = torch.randn(rows, out_features, generator=gen).cuda()
    y = linear(x, w, b)
    grads = torch.autograd.grad(y, (x, w, b), dy)
    x64, w64, b64 = (t.detach().double().requires_grad_() for t in (x, w, b))
    y64 = torch.nn.functional.linear(x64, w64, b64)
    refs = (y64, *torch.autograd.grad(y64, (x64, w64, b64), dy.double()))
    # fp32: at most 192 products per sum, each sum's error below 192 * 2^-24 of its largest partial sum; tf32 operands
    # are rounded to 11 bits (2^-11 each)
    for got, ref, library in zip((y, *grads), refs, (tf32, tf32, False, False)):
        assert got.shape == ref.shape and _err(got.detach(), ref.detach()) < (2e-3 if library else TOL)
    with torch.no_grad():
        assert _err(linear(x, w, b), y64.detach()) < (2e-3 if tf32 else TOL)
        assert _err(linear(x, w, None), torch.nn.functional.linear(x64, w64).detach()) < (2e-3 if tf32 else TOL)


@pytest.mark.parametrize("rows,reduce,cols", [(1, 4, 4), (33, 100, 44), (31, 1024, 68), (50001, 68, 200)])
def test_row_kernel_at_the_edges_of_its_tiles(rows, reduce, cols):
    """Reductions and columns that end inside a chunk, with and without a bias, through the C entry."""
    from torchgt_b200 import _cabi
    gen = torch.Generator().manual_seed(rows + reduce)
    x, w, b = (torch.randn(*s, generator=gen).cuda() for s in ((rows, reduce), (cols, reduce), (cols,)))
    for bias in (b, None):
        y = torch.full((rows, cols), float("nan"), device="cuda")
        _cabi.check(_cabi.load().tgt_linear_rows(x.data_ptr(), w.data_ptr(), None if bias is None else b.data_ptr(), rows,
                                                 reduce, cols, y.data_ptr(), torch.cuda.current_stream().cuda_stream))
        ref = torch.nn.functional.linear(x.double(), w.double(), None if bias is None else b.double())
        assert _err(y, ref) < TOL


def test_linear_takes_every_call_that_f_linear_takes():
    """Views off a 16-byte boundary, transposed inputs and weights, leading dimensions, no rows, other widths,
    infinities, torch.func and second-order gradients."""
    from torchgt_b200.linear import linear
    F = torch.nn.functional
    torch.manual_seed(5)
    w, b = torch.randn(64, 64, device="cuda"), torch.randn(64, device="cuda")
    base = torch.randn(2000 * 64 + 1, device="cuda")
    calls = [(base[1:].view(2000, 64), w, b), (torch.randn(64, 2000, device="cuda").t(), w.t(), b),
             (torch.randn(2, 30, 50, 64, device="cuda"), w, b), (torch.randn(64, device="cuda"), w, b),
             (torch.empty(0, 64, device="cuda"), w, b), (torch.randn(9, 100, device="cuda"), torch.randn(47, 100, device="cuda"), None)]
    for args in calls:
        x = args[0].detach().requires_grad_()
        y, ref = linear(x, *args[1:]), F.linear(args[0].double(), *(None if t is None else t.double() for t in args[1:]))
        assert y.shape == ref.shape and (ref.numel() == 0 or _err(y.detach(), ref) < TOL)
        dx, = torch.autograd.grad(y.sum(), x)
        assert dx.shape == x.shape
    x = torch.randn(4000, 64, device="cuda")
    x[3, 7], x[11, 0] = float("inf"), float("nan")
    y, ref = linear(x, w, b), F.linear(x, w, b)
    assert torch.equal(y.isnan(), ref.isnan()) and torch.equal(y.isinf(), ref.isinf())
    z = torch.randn(6, 5, 64, device="cuda")
    assert _err(torch.func.vmap(lambda t: linear(t, w, b))(z), F.linear(z.double(), w.double(), b.double())) < 2e-3
    x = torch.randn(8, 64, device="cuda", requires_grad=True)
    w2 = w.clone().requires_grad_()
    g, = torch.autograd.grad(linear(x, w2, b).sum(), x, create_graph=True)
    dw, = torch.autograd.grad((g * g).sum(), w2)
    assert _err(dw, (2 * 8 * w.double().sum(0)).expand(64, 64)) < 2e-3


# either side of every line of the rule: rows, reduction, columns, bias
@pytest.mark.parametrize("rows,reduce,cols,bias,own", [
    (1023, 64, 64, True, False), (1024, 64, 64, True, True), (32768, 64, 28, True, False), (32767, 64, 28, True, True),
    (32768, 64, 32, True, True), (8191, 128, 64, True, True), (8192, 128, 64, True, False), (32768, 128, 64, True, True),
    (4097, 192, 64, True, False), (4097, 512, 512, True, False), (65535, 64, 64, False, False), (65536, 64, 64, False, True),
    (65536, 128, 64, False, False), (65536, 64, 28, False, False)])
def test_full_fp32_products_take_the_kernel_that_is_ahead(rows, reduce, cols, bias, own):
    """Bit for bit the library's product, or the row kernel's; both within the bound of a fp32 sum of 64-bit values."""
    from torchgt_b200 import _cabi
    from torchgt_b200.linear import linear
    gen = torch.Generator().manual_seed(rows + reduce + cols)
    x, w, b = (torch.randn(*s, generator=gen).cuda() for s in ((rows, reduce), (cols, reduce), (cols,)))
    b = b if bias else None
    before = torch.backends.cuda.matmul.allow_tf32
    torch.backends.cuda.matmul.allow_tf32 = False
    try:
        with torch.no_grad():
            y, library = linear(x, w, b), torch.nn.functional.linear(x, w, b)
    finally:
        torch.backends.cuda.matmul.allow_tf32 = before
    kernel = torch.empty_like(y)
    _cabi.check(_cabi.load().tgt_linear_rows(x.data_ptr(), w.data_ptr(), b.data_ptr() if bias else None, rows, reduce, cols,
                                             kernel.data_ptr(), torch.cuda.current_stream().cuda_stream))
    assert torch.equal(y, kernel if own else library)
    assert _err(y, torch.nn.functional.linear(x.double(), w.double(), b.double() if bias else None)) < TOL
