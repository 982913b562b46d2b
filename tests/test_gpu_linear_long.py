"""Lists long enough that the products' kernels bring rows into the L2 ahead of their loads (64 MB of them and more): around the
line, with last tiles that are not whole and tiles that would lie behind the end."""
import pytest
import torch

pytestmark = pytest.mark.gpu

LINE = 64 << 20
# 2-norm over 2-norm against 64 bits; measured 7e-8 to 1.5e-7 (products), 1.5e-7 (parameter gradients over 320,000 rows)
TOL = 6e-7


def _far(got, want):
    return float((got.double() - want).norm() / want.norm())


@pytest.mark.parametrize("width", [64, 128])
@pytest.mark.parametrize("extra", [-1, 0, 1, 127, 128 * 300 + 5])
def test_products_and_gradients_around_the_line(width, extra):
    import ctypes
    from torchgt_b200 import _cabi
    from torchgt_b200.linear import wgrad
    lib = _cabi.load()
    rows = LINE // (4 * width) + extra
    gen = torch.Generator(device="cuda").manual_seed(width + extra)
    x = torch.randn(rows, width, generator=gen, device="cuda")
    w = torch.randn(64, width, generator=gen, device="cuda")
    b = torch.randn(64, generator=gen, device="cuda")
    y = torch.full((rows, 64), float("nan"), device="cuda")
    stream = torch.cuda.current_stream().cuda_stream
    _cabi.check(lib.tgt_linear_rows(x.data_ptr(), w.data_ptr(), b.data_ptr(), rows, width, 64, y.data_ptr(), stream))
    assert _far(y, x.double() @ w.double().t() + b.double()) < TOL
    dw, db = wgrad(y, x)
    assert _far(dw, y.double().t() @ x.double()) < TOL and _far(db, y.double().sum(0)) < TOL
    third = rows // 3 + 2                      # three sources of which the sum is longer than the line
    dys = [torch.randn(third, width, generator=gen, device="cuda") for _ in range(3)]
    ws = [torch.randn(width, 64, generator=gen, device="cuda") for _ in range(3)]
    dx = torch.full((third, 64), float("nan"), device="cuda")
    arr = lambda ts: (ctypes.c_void_p * 3)(*[t.data_ptr() for t in ts])   # noqa: E731
    _cabi.check(lib.tgt_linear_input_grad_multi(arr(dys), arr(ws), 3, third, width, 64, 0, None, dx.data_ptr(), stream))
    assert _far(dx, sum(d.double() @ v.double() for d, v in zip(dys, ws))) < TOL
