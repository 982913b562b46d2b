"""Products and parameter gradients of the narrow linear layers on the tensor cores, at the edges of their tiles, against
fp64.  Three bf16 pieces carry 24 bits of an operand and the dropped piece products stay below 2^-23 of a product.  A running
sum takes at most 128 products in 8 steps of a rounding of at most 2^-23 each: below 8 * 2^-23 < 1e-6 of the result in the
2-norm where the signs are mixed.  (Without the third piece of one operand the error is 2.6e-6: tests/test_host_logic.py.)"""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu

TOL = 1e-6


def _lib():
    from torchgt_b200 import _cabi
    return _cabi


def _stream():
    return torch.cuda.current_stream().cuda_stream


def _rand(seed, *shapes):
    gen = torch.Generator().manual_seed(seed)
    return [torch.randn(*s, generator=gen).cuda() for s in shapes]


def _rel(got, ref):
    return float((got.double() - ref).norm() / ref.norm().clamp_min(1e-30))


def _array(tensors):
    return (ctypes.c_void_p * len(tensors))(*[None if t is None else t.data_ptr() for t in tensors])


def _act(name, t):
    return {"none": lambda v: v, "relu": torch.relu, "gelu": torch.nn.functional.gelu}[name](t)


ACTS = {"none": 0, "relu": 1, "gelu": 2}


@pytest.mark.parametrize("count", [1, 3])
@pytest.mark.parametrize("rows,reduce,cols", [
    (1, 64, 64), (4064, 64, 64), (10112, 64, 64), (10113, 64, 64), (10240, 64, 64), (20001, 64, 64), (38017, 64, 40),
    (10300, 128, 64), (10300, 64, 128), (10300, 68, 100), (10300, 4, 4), (2049, 64, 1024), (10300, 384, 64), (10300, 448, 64),
    (10300, 832, 64), (10300, 1024, 8)])
def test_products_and_input_gradients(rows, reduce, cols, count):
    c = _lib()
    x, = _rand(rows + reduce, (rows, reduce))
    w, b = _rand(cols, (count, cols, reduce), (count, cols))
    w, b = list(w.contiguous().unbind(0)), list(b.contiguous().unbind(0))
    y = [torch.full((rows, cols), float("nan"), device="cuda") for _ in range(count)]
    c.check(c.load().tgt_linear_rows_multi(x.data_ptr(), _array(w), _array(b), count, rows, reduce, cols, 0, None, None,
                                           _array(y), _stream()))
    for i in range(count):
        assert _rel(y[i], x.double() @ w[i].double().t() + b[i].double()) < TOL
    dx = torch.full((rows, reduce), float("nan"), device="cuda")
    c.check(c.load().tgt_linear_input_grad_multi(_array(y), _array(w), count, rows, cols, reduce, 0, None, dx.data_ptr(),
                                                 _stream()))
    assert _rel(dx, sum(y[i].double() @ w[i].double() for i in range(count))) < TOL
    again = torch.empty_like(dx)
    c.check(c.load().tgt_linear_input_grad_multi(_array(y), _array(w), count, rows, cols, reduce, 0, None, again.data_ptr(),
                                                 _stream()))
    assert torch.equal(dx, again)


@pytest.mark.parametrize("signs", ["mixed", "one"])
@pytest.mark.parametrize("reduce,count", [(64, 3), (128, 1), (192, 1), (132, 2), (128, 3), (448, 1), (448, 3), (1024, 1), (1024, 3)])
def test_long_reductions_are_no_further_off_than_sums_rounded_to_nearest(reduce, count, signs):
    """Tensor cores round a running sum towards zero at each of its steps of 16: where all products have one sign that adds up.
    With at most 128 products per running sum the loss is below 8 steps of 2^-23 of the sum, and 24 such sums are added with
    rounding to nearest: below 1e-6 + 24^0.5 * 2^-24 in all.  With mixed signs it averages out and has to stay below the error
    of the library's fp32 product."""
    c = _lib()
    rows, cols = 10300, 64
    x, = _rand(reduce, (rows, reduce))
    dy = list(_rand(count, (count, rows, reduce))[0].unbind(0))
    w = list(_rand(reduce + count, (count, reduce, cols))[0].unbind(0))
    if signs == "one":
        x, dy, w = x.abs(), [t.abs() for t in dy], [t.abs() for t in w]
    y, dx = torch.empty(rows, cols, device="cuda"), torch.empty(rows, cols, device="cuda")
    wt = w[0].t().contiguous()
    c.check(c.load().tgt_linear_rows(x.data_ptr(), wt.data_ptr(), None, rows, reduce, cols, y.data_ptr(), _stream()))
    c.check(c.load().tgt_linear_input_grad_multi(_array(dy), _array(w), count, rows, reduce, cols, 0, None, dx.data_ptr(),
                                                 _stream()))
    before = torch.backends.cuda.matmul.allow_tf32
    torch.backends.cuda.matmul.allow_tf32 = False
    library = x @ w[0], sum(d @ v for d, v in zip(dy, w))
    torch.backends.cuda.matmul.allow_tf32 = before
    refs = x.double() @ w[0].double(), sum(d.double() @ v.double() for d, v in zip(dy, w))
    for got, near, ref in zip((y, dx), library, refs):
        assert _rel(got, ref) < (_rel(near, ref) if signs == "mixed" else 1.3e-6)


@pytest.mark.parametrize("act", ["relu", "gelu"])
@pytest.mark.parametrize("rows", [33, 10113])
def test_activation_residual_and_gate(rows, act):
    _follow_a_sum(rows, act, 64)


@pytest.mark.parametrize("act", ["relu", "gelu"])
@pytest.mark.parametrize("reduce", [388, 832])      # two and three launches
def test_activation_residual_and_gate_after_a_sum_in_parts(reduce, act):
    _follow_a_sum(10113, act, reduce)


def _follow_a_sum(rows, act, reduce):
    c = _lib()
    x, w, b, add, dy = _rand(rows, (rows, reduce), (128, reduce), (128,), (rows, 128), (rows, reduce))
    pre, y = torch.empty(rows, 128, device="cuda"), torch.empty(rows, 128, device="cuda")
    c.check(c.load().tgt_linear_rows_multi(x.data_ptr(), _array([w]), _array([b]), 1, rows, reduce, 128, ACTS[act],
                                           pre.data_ptr(), add.data_ptr(), _array([y]), _stream()))
    z = x.double() @ w.double().t() + b.double()
    assert _rel(pre, z) < TOL and _rel(y, _act(act, z) + add.double()) < TOL
    gate = torch.relu(pre) if act == "relu" else pre
    w2, = _rand(1, (reduce, 128))
    dx = torch.empty(rows, 128, device="cuda")
    c.check(c.load().tgt_linear_input_grad_multi(_array([dy]), _array([w2]), 1, rows, reduce, 128, ACTS[act], gate.data_ptr(),
                                                 dx.data_ptr(), _stream()))
    leaf = pre.double().requires_grad_()
    ref, = torch.autograd.grad(_act(act, leaf), leaf, dy.double() @ w2.double())
    assert _rel(dx, ref) < TOL


@pytest.mark.parametrize("count", [1, 2, 3])
@pytest.mark.parametrize("rows,inp,out", [(1, 64, 64), (63, 64, 64), (64, 64, 64), (65, 64, 4), (9473, 64, 64),
                                          (20001, 128, 64), (20001, 64, 100), (150001, 64, 64)])
def test_parameter_gradients(rows, inp, out, count):
    c = _lib()
    x, = _rand(rows + inp, (rows, inp))
    dy = list(_rand(out, (count, rows, out))[0].unbind(0))
    dw = [torch.full((out, inp), float("nan"), device="cuda") for _ in range(count)]
    db = [torch.full((out,), float("nan"), device="cuda") for _ in range(count - 1)] + [None]
    need = ctypes.c_size_t()
    c.check(c.load().tgt_linear_wgrad_multi_scratch_bytes(count, rows, inp, out, ctypes.byref(need)))
    scratch = torch.full((need.value + 512,), 171, dtype=torch.uint8, device="cuda")
    c.check(c.load().tgt_linear_wgrad_multi(_array(dy), x.data_ptr(), count, rows, inp, out, _array(dw), _array(db),
                                            scratch.data_ptr(), need.value, _stream()))
    assert (scratch[need.value:] == 171).all()
    for i in range(count):
        assert _rel(dw[i], dy[i].double().t() @ x.double()) < TOL
        assert db[i] is None or _rel(db[i], dy[i].double().sum(0)) < TOL


def test_values_that_are_not_finite_and_sums_past_the_range():
    """They come out as fp32 FMAs give them: infinities and NaN where those belong, and nowhere else."""
    c = _lib()
    rows = 10300
    x, w = _rand(3, (rows, 64), (64, 64))
    x[5, 3], x[700, 1], x[10299] = float("inf"), float("nan"), 3e38
    w[9, 2] = float("-inf")
    y = torch.empty(rows, 64, device="cuda")
    c.check(c.load().tgt_linear_rows(x.data_ptr(), w.data_ptr(), None, rows, 64, 64, y.data_ptr(), _stream()))
    before = torch.backends.cuda.matmul.allow_tf32
    torch.backends.cuda.matmul.allow_tf32 = False
    ref = x @ w.t()
    torch.backends.cuda.matmul.allow_tf32 = before
    assert torch.equal(y.isnan()[:10299], ref.isnan()[:10299]) and torch.equal(y.isinf()[:10299], ref.isinf()[:10299])
    assert not y[10299].isfinite().all()
    fine = ref.isfinite() & y.isfinite()
    fine[10299] = False
    assert _rel(y[fine], (x.double() @ w.double().t())[fine]) < TOL
    dy, = _rand(4, (rows, 64))
    x[10299] = 0
    need = ctypes.c_size_t()
    c.check(c.load().tgt_linear_wgrad_scratch_bytes(rows, 64, 64, ctypes.byref(need)))
    scratch, dw = torch.empty(need.value, dtype=torch.uint8, device="cuda"), torch.empty(64, 64, device="cuda")
    c.check(c.load().tgt_linear_wgrad(dy.data_ptr(), x.data_ptr(), rows, 64, 64, dw.data_ptr(), None, scratch.data_ptr(),
                                      need.value, _stream()))
    assert dw[:, 3].isinf().all() and dw[:, 1].isnan().all()
    rest = [i for i in range(64) if i not in (1, 3)]
    assert _rel(dw[:, rest], (dy.double().t() @ x.double())[:, rest]) < TOL


@pytest.mark.parametrize("act", ["none", "relu"])
@pytest.mark.parametrize("count,reduce,cols", [(1, 64, 64), (3, 64, 64), (1, 68, 100), (3, 132, 36)])
def test_input_gradients_that_are_not_finite(count, reduce, cols, act):
    """Transposed weights, several sources, the last chunk and column tile in part, with a gate and without."""
    c = _lib()
    rows = 10300
    dy, w = list(_rand(8, (count, rows, reduce))[0].unbind(0)), list(_rand(9, (count, reduce, cols))[0].unbind(0))
    dy[-1][5, 3], dy[0][700, reduce - 1], dy[0][701, 0], dy[-1][10299] = float("inf"), float("nan"), float("-inf"), 1e38
    w[-1][2, 9], w[0][reduce - 1, cols - 1] = float("-inf"), float("nan")
    gate = torch.relu(_rand(10, (rows, cols))[0]) if act == "relu" else None
    dx = torch.empty(rows, cols, device="cuda")
    c.check(c.load().tgt_linear_input_grad_multi(_array(dy), _array(w), count, rows, reduce, cols, ACTS[act],
                                                 None if gate is None else gate.data_ptr(), dx.data_ptr(), _stream()))
    before = torch.backends.cuda.matmul.allow_tf32
    torch.backends.cuda.matmul.allow_tf32 = False
    ref, exact = sum(d @ v for d, v in zip(dy, w)), sum(d.double() @ v.double() for d, v in zip(dy, w))
    torch.backends.cuda.matmul.allow_tf32 = before
    if gate is not None:
        ref, exact = torch.where(gate <= 0, 0.0, ref), torch.where(gate <= 0, 0.0, exact)
    # in the last row, whose sums pass the range of fp32, the order of the additions may decide
    assert torch.equal(dx.isnan()[:10299], ref.isnan()[:10299]) and torch.equal(dx.isinf()[:10299], ref.isinf()[:10299])
    fine = ref.isfinite()
    fine[10299] = False
    assert fine.sum() > rows * cols // 3 and _rel(dx[fine], exact[fine]) < TOL

def test_one_nan_costs_a_small_multiple():
    """The elements it reaches are summed again by whole blocks; one thread per element took 130 times as long."""
    c = _lib()
    rows = 200000
    dy, x, w = _rand(5, (rows, 64), (rows, 64), (64, 64))
    need = ctypes.c_size_t()
    c.check(c.load().tgt_linear_wgrad_scratch_bytes(rows, 64, 64, ctypes.byref(need)))
    scratch, dw = torch.empty(need.value, dtype=torch.uint8, device="cuda"), torch.empty(64, 64, device="cuda")
    y, events = torch.empty(rows, 64, device="cuda"), [torch.cuda.Event(enable_timing=True) for _ in range(3)]

    def times():
        best = [1e9, 1e9]
        for _ in range(5):
            events[0].record()
            c.check(c.load().tgt_linear_wgrad(dy.data_ptr(), x.data_ptr(), rows, 64, 64, dw.data_ptr(), None,
                                              scratch.data_ptr(), need.value, _stream()))
            events[1].record()
            c.check(c.load().tgt_linear_rows(x.data_ptr(), w.data_ptr(), None, rows, 64, 64, y.data_ptr(), _stream()))
            events[2].record()
            torch.cuda.synchronize()
            best = [min(b, events[i].elapsed_time(events[i + 1])) for i, b in enumerate(best)]
        return best
    fine = times()
    x[777, 5] = dy[1234, 7] = float("nan")
    assert all(slow < 20 * fast for slow, fast in zip(times(), fine))


def test_arguments_the_calls_refuse():
    c = _lib()
    lib = c.load()
    t = torch.randn(8, 64, device="cuda")
    one = _array([t])
    assert lib.tgt_linear_rows_multi(t.data_ptr(), one, one, 4, 8, 64, 64, 0, None, None, one, None) == 1
    assert lib.tgt_linear_rows_multi(t.data_ptr(), one, one, 1, 8, 62, 64, 0, None, None, one, None) == 3
    assert lib.tgt_linear_rows_multi(t.data_ptr(), one, one, 1, 8, 64, 64, 7, None, None, one, None) == 1
    assert lib.tgt_linear_input_grad_multi(one, one, 1, 8, 64, 64, 1, None, t.data_ptr(), None) == 1     # a gate is missing
    assert lib.tgt_linear_input_grad(t.data_ptr() + 4, t.data_ptr(), 8, 64, 64, t.data_ptr(), None) == 1
    n = ctypes.c_size_t()
    assert lib.tgt_linear_wgrad_multi_scratch_bytes(4, 8, 64, 64, ctypes.byref(n)) == 1


def test_a_wait_that_runs_out_is_reported_once():
    from torchgt_b200.linear import linear
    c = _lib()
    lib = c.load()
    x, w, y = torch.randn(64, 64, device="cuda"), torch.randn(64, 64, device="cuda"), torch.empty(64, 64, device="cuda")
    wide = torch.randn(20000, 64, device="cuda")

    def product():
        return lib.tgt_linear_rows(x.data_ptr(), w.data_ptr(), None, 64, 64, 64, y.data_ptr(), _stream())
    assert product() == 0 and lib.tgt_products_status() == 0
    c.check(lib.tgt_debug_expire_wait(_stream()))
    torch.cuda.synchronize()
    assert product() == 2 and b"tensor cores" in lib.tgt_last_error()
    assert product() == 0 and lib.tgt_products_status() == 0
    c.check(lib.tgt_debug_expire_wait(_stream()))
    torch.cuda.synchronize()
    with pytest.raises(c.TgtError):
        linear(wide, w, w[0])
    assert _rel(linear(wide, w, w[0]), wide.double() @ w.double().t() + w[0].double()) < 1e-3
