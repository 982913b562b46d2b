"""Rows that cross tiles, and the two routes of the bias gradient.

A row's tiles leave partial sums that a second kernel adds up: up to eight further tiles by one lane group, more by a
whole CTA.  dbias is written by the pass over the sources when both passes run in one call, by the pass over the
destinations when the caller runs them one by one."""
import numpy as np
import pytest
import torch

from helpers import TOL_BF16, TOL_F32, rel_err
from oracle import sparse_attn_oracle as sao

pytestmark = pytest.mark.gpu

GROUP_TILES = 8


@pytest.fixture(autouse=True)
def _own_tiles():
    from torchgt_b200 import _cabi
    yield
    _cabi.check(_cabi.load().tgt_debug_set_tile_edges(0))


def _graph_with_rows_of(lengths, extra, seed):
    """Edges in which row i is the destination of exactly lengths[i] edges and the source of as many; their other ends are
    `extra` rows behind those."""
    rng = np.random.default_rng(seed)
    rows = np.concatenate([np.full(m, i) for i, m in enumerate(lengths)])
    ends = rng.integers(len(lengths), len(lengths) + extra, (2, rows.size))
    ei = np.concatenate([np.stack([ends[0], rows]), np.stack([rows, ends[1]])], axis=1)
    for side in ei:
        assert np.array_equal(np.bincount(side, minlength=len(lengths))[:len(lengths)], lengths)
    return torch.from_numpy(ei[:, rng.permutation(ei.shape[1])])


def _lengths(tile, slots):
    """Edges per row: one less than, as many as and one more than fill 1 or 2 tiles, those on both sides of the line between
    the finishing kernel's routes, and more than one round of its CTA's slots; each of these rows starts with a tile, the row
    behind it fills its last one up.  Then rows that start anywhere in a tile."""
    lengths, further = [], []
    for m in (1, 2, GROUP_TILES, GROUP_TILES + 1, GROUP_TILES + 2, slots + 2):
        for n in (m * tile - 1, m * tile, m * tile + 1):
            lengths += [n, -n % tile]
            further.append((n - 1) // tile)
    assert set(further) >= {0, 1, GROUP_TILES, GROUP_TILES + 1, slots + 1, slots + 2}
    return lengths + [3, 0, (GROUP_TILES - 1) * tile - 1, 1, 0, 0, 3 * tile + 1, 2]


@pytest.mark.parametrize("heads,head_dim,dtype", [(8, 8, torch.float32), (1, 8, torch.float32), (2, 8, torch.float32),
                                                  (8, 16, torch.float32), (3, 8, torch.float32), (8, 8, torch.bfloat16)])
@pytest.mark.parametrize("bias", ["none", "edge", "head"])
def test_rows_over_one_to_many_tiles_match_the_oracle(heads, head_dim, dtype, bias):
    from torchgt_b200 import SparseGraph, _cabi, sparse_graph_attention
    _cabi.check(_cabi.load().tgt_debug_set_tile_edges(4))
    # lanes of a group; a tile is 128 / lanes groups of 4 edges, the finishing CTA has 128 or 512 / lanes slots
    lanes = {(8, 8): 8 if dtype == torch.bfloat16 else 16, (1, 8): 2, (2, 8): 4, (8, 16): 32, (3, 8): 2}[heads, head_dim]
    lengths = _lengths(4 * 128 // lanes, (128 if lanes <= 4 else 512) // lanes)
    n = len(lengths) + 40
    ei = _graph_with_rows_of(lengths, 40, 5)
    gen = torch.Generator().manual_seed(6)
    q, k, v, dout = (torch.randn(n, heads, head_dim, generator=gen).to(dtype) for _ in range(4))
    b = None if bias == "none" else torch.randn((ei.shape[1],) + ((heads,) if bias == "head" else ()), generator=gen) * 0.1
    if bias == "edge" and heads == 3:
        pytest.skip("a shared bias of three heads is expanded per head")
    qc, kc, vc = (t.cuda().requires_grad_() for t in (q, k, v))
    bc = None if b is None else b.cuda().requires_grad_()
    out = sparse_graph_attention(qc, kc, vc, SparseGraph(ei.cuda(), n), bc)
    out.backward(dout.cuda())
    ref, _ = sao.forward_closed_form(q.float(), k.float(), v.float(), ei, b)
    dq, dk, dv, dt = sao.backward_closed_form(q.float(), k.float(), v.float(), ei, dout.float(), b)
    tol = TOL_F32 if dtype == torch.float32 else TOL_BF16
    assert rel_err(out.detach().float(), ref) < tol
    for got, want in ((qc.grad, dq), (kc.grad, dk), (vc.grad, dv)):
        assert rel_err(got.float(), want) < tol
    if b is not None:
        assert rel_err(bc.grad, dt if bias == "head" else dt.sum(axis=1)) < tol


@pytest.mark.parametrize("columns", [1, 8])
def test_passes_one_by_one_and_in_one_call_agree(columns):
    import ctypes
    from torchgt_b200 import SparseGraph, _cabi
    lib = _cabi.load()
    n, heads, dim = 700, 8, 8
    rng = np.random.default_rng(3)
    ei = torch.from_numpy(np.concatenate([rng.integers(0, n, (2, 5000)), np.stack([np.zeros(900, int), rng.integers(0, n, 900)])],
                                         axis=1)).cuda()
    graph = SparseGraph(ei, n)
    gen = torch.Generator(device="cuda").manual_seed(4)
    q, k, v, dout = (torch.randn(n, heads, dim, generator=gen, device="cuda") for _ in range(4))
    bias = torch.randn(ei.shape[1] * columns, generator=gen, device="cuda") * 0.1
    stream = torch.cuda.current_stream().cuda_stream
    size = ctypes.c_size_t()
    _cabi.check(lib.tgt_sparse_attn_scratch_bytes(graph.by_dst.byref(), graph.by_src.byref(), heads, dim, 0, 1, ctypes.byref(size)))
    out, z = torch.empty_like(q), torch.empty(n, heads, device="cuda")
    scratch = torch.empty(max(size.value, 1 << 20), dtype=torch.uint8, device="cuda")
    _cabi.check(lib.tgt_sparse_attn_fwd(q.data_ptr(), k.data_ptr(), v.data_ptr(), bias.data_ptr(), columns, graph.by_dst.byref(),
                                        out.data_ptr(), z.data_ptr(), heads, dim, 0, scratch.data_ptr(), scratch.numel(), stream))
    results = []
    for sequence in ((7,), (0,), (1, 2, 4), (3, 4), (1, 6)):
        got = [torch.full_like(t, float("nan")) for t in (q, k, v, bias)]
        scratch.fill_(255)
        for passes in sequence:
            entry = lib.tgt_sparse_attn_bwd_passes if passes else lib.tgt_sparse_attn_bwd
            _cabi.check(entry(dout.data_ptr(), q.data_ptr(), k.data_ptr(), v.data_ptr(), bias.data_ptr(), columns, out.data_ptr(),
                              z.data_ptr(), graph.by_dst.byref(), graph.by_src.byref(), *(t.data_ptr() for t in got), heads, dim,
                              0, scratch.data_ptr(), scratch.numel(), stream, *([passes] if passes else [])))
        torch.cuda.synchronize()
        results.append(got)
    for got in results[1:]:
        for a, b in zip(got, results[0]):
            assert torch.isfinite(a).all()
            assert float((a - b).abs().max()) <= TOL_F32 * float(b.abs().max())


@pytest.mark.parametrize("heads,head_dim", [(8, 8), (4, 16), (8, 16)])
@pytest.mark.parametrize("degree", [30, 200])
def test_dq_of_a_learnt_bias_subtracts_delta_edge_by_edge(heads, head_dim, degree):
    """Values with a mean of three standard deviations: subtracting delta from every edge's gradient keeps the cancellation in
    front of the rounding of the sums.  Against 64 bits dQ is then 0.7 to 0.8 times as far off as that of the same call with the
    bias as a plain input, which has no statistics of the output and subtracts the rounded sums; the same route would give 1."""
    from torchgt_b200 import SparseGraph, sparse_graph_attention
    n = 600
    gen = torch.Generator().manual_seed(degree)
    ei = torch.randint(0, n, (2, n * degree), generator=gen)
    q, k, v, dout = (torch.randn(n, heads, head_dim, generator=gen) for _ in range(4))
    v, b = v + 3, 0.1 * torch.randn(n * degree, generator=gen)
    want = sao.backward_closed_form(q, k, v, ei, dout, b)[0]
    graph, off = SparseGraph(ei.cuda(), n), []
    for learnt in (True, False):
        leaf = q.cuda().requires_grad_()
        sparse_graph_attention(leaf, k.cuda(), v.cuda(), graph, b.cuda().requires_grad_(learnt)).backward(dout.cuda())
        off.append(float(np.linalg.norm(leaf.grad.cpu().double().numpy() - want)))
    assert off[0] < 0.9 * off[1], off
