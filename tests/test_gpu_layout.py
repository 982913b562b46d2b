"""Edge layouts built on the GPU against the CPU oracle: bit-exact integer arrays."""
import numpy as np
import pytest
import torch

from helpers import random_graph
from oracle import edge_layout_oracle as elo

pytestmark = pytest.mark.gpu


def _check(ei_cpu: torch.Tensor, n_rows: int):
    from torchgt_b200.graph import SparseGraph
    graph = SparseGraph(ei_cpu.cuda(), n_rows)
    for group_by, lay in ((1, graph.by_dst), (0, graph.by_src)):
        ptr, other, perm = elo.segment_layout(ei_cpu.numpy(), n_rows, group_by)
        key = ei_cpu.numpy()[1 if group_by == 1 else 0]
        assert np.array_equal(lay.ptr.cpu().numpy().astype(np.int64), ptr)
        assert np.array_equal(lay.other.cpu().numpy().astype(np.int64), other)
        assert np.array_equal(lay.perm.cpu().numpy().astype(np.int64), perm)
        assert np.array_equal(lay.seg.cpu().numpy().astype(np.int64), key[perm])
    return graph


@pytest.mark.parametrize("n,deg", [(1, 0.0), (2, 1.0), (97, 4.0), (1000, 8.0), (5000, 3.0), (4097, 9.0)])
def test_random_graphs(n, deg):
    _check(random_graph(11 + n, n, deg), n)


def test_no_edges_and_single_edge():
    _check(torch.zeros((2, 0), dtype=torch.long), 5)
    _check(torch.tensor([[3], [1]]), 5)


def test_sorted_by_source_with_duplicates():
    ei = random_graph(5, 300, 6.0, duplicates=True)
    ei = ei[:, torch.argsort(ei[0])]            # the order reformat_graph leaves (gt_sp/utils.py:354-356)
    ei = torch.cat([ei, ei[:, :50]], dim=1)     # exact duplicates
    _check(ei, 300)


def test_benchmark_sized_graph():
    from torchgt_b200.synthetic import benchmark_64k
    ei, n_rows = benchmark_64k()
    assert ei.shape[1] == 526450 and n_rows == 64001
    _check(ei, n_rows)


def test_out_of_range_index_is_reported():
    from torchgt_b200._cabi import TgtError
    from torchgt_b200.graph import SparseGraph
    ei = torch.tensor([[0, 1, 9], [1, 2, 0]]).cuda()
    with pytest.raises(TgtError, match="INDEX_RANGE"):
        SparseGraph(ei, 5, defer_check=False)
    ei = torch.tensor([[0, 1, 2], [1, -1, 0]]).cuda()
    with pytest.raises(TgtError, match="INDEX_RANGE"):
        SparseGraph(ei, 5, defer_check=False)
    # the context is still usable afterwards
    SparseGraph(torch.tensor([[0, 1], [1, 2]]).cuda(), 5)


def test_deferred_range_check_does_not_raise_at_build_time_but_on_check():
    from torchgt_b200._cabi import TgtError
    from torchgt_b200.graph import SparseGraph
    good = SparseGraph(random_graph(2, 50, 3.0).cuda(), 50)     # the default build does not synchronise
    good.by_src
    good.check()
    bad = SparseGraph(torch.tensor([[0, 1, 9], [1, 2, 0]]).cuda(), 5)   # id 9 >= 5
    with pytest.raises(TgtError, match="INDEX_RANGE"):
        bad.check()
    with pytest.raises(TgtError, match="INDEX_RANGE"):
        bad.poll()                                                       # stays reported
    # the layout itself is in bounds (the bad id was replaced by 0), so using it cannot fault
    assert int(bad.by_dst.other.max()) < 5 and int(bad.by_dst.seg.max()) < 5


def test_graph_cache_hits_on_identity_and_on_content():
    from torchgt_b200.graph import clear_graph_cache, graph_for
    clear_graph_cache()
    ei = random_graph(3, 200, 4.0).cuda()
    g1 = graph_for(ei, 200)
    assert graph_for(ei, 200) is g1                 # same tensor object
    assert graph_for(ei.clone(), 200) is g1         # fresh upload of the same edges
    other = ei.clone()
    other[0, 0] = (other[0, 0] + 1) % 200
    assert graph_for(other, 200) is not g1
    ei[0, 0] = (ei[0, 0] + 1) % 200                 # in-place edit invalidates the identity entry
    assert graph_for(ei, 200) is not g1


def test_bad_graph_is_reported_by_the_first_use_that_finds_the_build_finished():
    from torchgt_b200 import sparse_graph_attention
    from torchgt_b200._cabi import TgtError
    from torchgt_b200.graph import SparseGraph
    bad = SparseGraph(torch.tensor([[0, 1, 9], [1, 2, 0]]).cuda(), 5)
    torch.cuda.synchronize()                     # the build has finished; nobody has looked at its result yet
    q = torch.randn(5, 2, 8, device="cuda")
    with pytest.raises(TgtError, match="INDEX_RANGE"):
        sparse_graph_attention(q, q, q, bad)


def test_graph_cache_compares_edge_lists_exactly():
    """Lists that differ only by the order of two columns, or by transposition, are different graphs
    (their perm differs, so per-edge biases would be applied to the wrong edges)."""
    from torchgt_b200.graph import clear_graph_cache, graph_for
    clear_graph_cache()
    n, e = 300, 2 * 4099
    gen = torch.Generator().manual_seed(9)
    ei = torch.randint(0, n, (2, e), generator=gen).cuda()
    g1 = graph_for(ei, n)
    swapped = ei.clone()
    swapped[:, [5, 5 + 4099]] = ei[:, [5 + 4099, 5]]
    assert not torch.equal(swapped, ei)
    g2 = graph_for(swapped, n)
    assert g2 is not g1
    g3 = graph_for(ei.flip(0).contiguous(), n)               # transposed graph
    assert g3 is not g1 and g3 is not g2
    assert graph_for(ei.clone(), n) is g1                    # all three stay cached side by side
    assert graph_for(swapped.clone(), n) is g2
    perm1, perm2 = g1.by_dst.perm.cpu(), g2.by_dst.perm.cpu()
    assert torch.equal(ei[1].cpu()[perm1.long()], g1.by_dst.seg.cpu().long())
    assert torch.equal(swapped[1].cpu()[perm2.long()], g2.by_dst.seg.cpu().long())


def test_int32_edge_lists_build_the_same_layouts():
    from torchgt_b200.graph import SparseGraph
    ei = random_graph(21, 700, 5.0)
    a, b = SparseGraph(ei.cuda(), 700), SparseGraph(ei.to(torch.int32).cuda(), 700)
    for la, lb in ((a.by_dst, b.by_dst), (a.by_src, b.by_src)):
        for name in ("ptr", "other", "perm", "seg"):
            assert torch.equal(getattr(la, name), getattr(lb, name)), name
    b.check()


@pytest.mark.parametrize("world", [1, 2, 4])
def test_device_side_batch_edges_equal_the_reference_helpers(world):
    """fix -> adjust -> flatten in one kernel against the CPU restatement of the three helpers
    (itself pinned to the reference's outputs in tests/golden/edges.npz)."""
    from torchgt_b200 import prepare_edges
    gen = torch.Generator().manual_seed(40 + world)
    nodes = [37, 64, 5, 120]
    raws = [torch.randint(0, n, (2, 3 * n + 1), generator=gen) for n in nodes]
    sub = -(-max(nodes) // world)                             # per-rank rows of the padded batch
    rows_per_graph = (sub + 1) * world
    fixed = [elo.fix_edge_index(r.numpy(), n) for r, n in zip(raws, nodes)]
    ref = elo.flatten_edge_index_nopad([elo.adjust_edge_index_nomerge(f, sub) for f in fixed], rows_per_graph)
    got = prepare_edges(torch.cat(raws, dim=1).cuda(), nodes, [r.shape[1] for r in raws], True, sub, rows_per_graph)
    assert got.dtype == torch.int32 and np.array_equal(got.cpu().numpy().astype(np.int64), ref)
    # single graph, no global token, no adjust: a plain narrowing copy
    plain = prepare_edges(raws[1].cuda(), nodes[1], None, False, 0, 0)
    assert np.array_equal(plain.cpu().numpy().astype(np.int64), raws[1].numpy())


def test_device_side_batch_edges_on_the_reference_golden_ring():
    from helpers import load_golden
    from torchgt_b200 import prepare_edges
    g = load_golden("edges.npz")
    got = prepare_edges(torch.from_numpy(g["ring"]).cuda(), 4, None, True, 2, 0)
    assert np.array_equal(got.cpu().numpy().astype(np.int64), g["ring_adjusted_L2"])
    for i in range(4):
        n, sub = int(g[f"rand{i}_n"]), int(g[f"rand{i}_sub"])
        got = prepare_edges(torch.from_numpy(g[f"rand{i}_in"]).cuda(), n, None, True, sub, 0)
        assert np.array_equal(got.cpu().numpy().astype(np.int64), g[f"rand{i}_adjusted"]), i


def test_a_graph_is_asked_by_one_thread_while_the_first_backward_builds_its_source_layout():
    """The backward runs on autograd's own thread and builds the layout there; other threads poll, check and ask for the
    layouts of the same graph meanwhile."""
    import threading
    from torchgt_b200 import SparseGraph, sparse_graph_attention
    ei = random_graph(8, 300, 5.0)
    bad = ei.clone()
    bad[0, 3] = 300
    q = torch.randn(300, 8, 8, device="cuda", requires_grad=True)
    for edges, wrong in ((ei.cuda(), False), (bad.cuda(), True)):
        for _ in range(20):
            graph, stop, failures, reported = SparseGraph(edges, 300), threading.Event(), [], []

            def ask():
                from torchgt_b200 import _cabi
                while not stop.is_set():
                    try:
                        graph.poll()
                        graph.check()
                        graph.native.has_by_src()
                        graph.by_dst.verified
                    except _cabi.TgtError:
                        reported.append(True)
                    except Exception as e:
                        failures.append(e)

            threads = [threading.Thread(target=ask) for _ in range(3)]
            for t in threads:
                t.start()
            try:
                out = sparse_graph_attention(q, q, q, graph)
                out.sum().backward()
            except Exception as e:
                if not wrong:
                    failures.append(e)
            finally:
                stop.set()
                for t in threads:
                    t.join()
            assert not failures, failures
            assert bool(reported) <= wrong
            if not wrong:
                graph.check()
                assert graph.by_dst.verified and graph.by_src.verified
                for lay, group_by in ((graph.by_dst, 1), (graph.by_src, 0)):
                    ptr, other, perm = elo.segment_layout(ei.numpy(), 300, group_by)
                    assert np.array_equal(lay.ptr.cpu().numpy(), ptr) and np.array_equal(lay.perm.cpu().numpy(), perm)
            else:
                with pytest.raises(Exception, match="outside"):
                    graph.check()


def test_other_threads_run_while_a_layout_check_waits_for_the_gpu():
    import threading
    import time
    from torchgt_b200 import SparseGraph
    ei = random_graph(8, 300, 5.0).cuda()
    SparseGraph(ei, 300).check()                      # everything is loaded
    stop, ticks = threading.Event(), []

    def tick():
        while not stop.is_set():
            ticks.append(time.perf_counter())
            time.sleep(0.001)

    thread = threading.Thread(target=tick)
    thread.start()
    try:
        torch.cuda._sleep(400_000_000)                # about 0.2 s of the GPU
        graph = SparseGraph(ei, 300)
        before = time.perf_counter()
        graph.check()
        after = time.perf_counter()
    finally:
        stop.set()
        thread.join()
    assert after - before > 0.05
    assert sum(before < t < after for t in ticks) >= 10


@pytest.mark.parametrize("n_edges", [1, 64, 65, 5000])
def test_an_int32_list_needs_no_workspace_for_a_narrow_copy(n_edges):
    """Its build fits the smaller size, to the byte, and gives the arrays of the int64 list."""
    import ctypes
    from torchgt_b200 import _cabi
    lib, n_rows = _cabi.load(), 300
    wide, narrow = ctypes.c_size_t(), ctypes.c_size_t()
    _cabi.check(lib.tgt_edge_layout_sizes(n_rows, n_edges, ctypes.byref(wide)))
    _cabi.check(lib.tgt_edge_layout_sizes_i32(n_rows, n_edges, ctypes.byref(narrow)))
    assert wide.value - narrow.value == (4 * n_edges + 255) // 256 * 256
    edges = torch.randint(0, n_rows, (2, n_edges), generator=torch.Generator().manual_seed(n_edges))
    i32 = edges.int().cuda()
    workspace = torch.full((narrow.value + 4096,), 171, dtype=torch.uint8, device="cuda")
    ptr = torch.empty(n_rows + 1, dtype=torch.int32, device="cuda")
    other, perm, seg = (torch.empty(n_edges, dtype=torch.int32, device="cuda") for _ in range(3))
    for group_by in (0, 1):
        args = (i32.data_ptr(), n_edges, n_rows, group_by, ptr.data_ptr(), other.data_ptr(), perm.data_ptr(), seg.data_ptr(),
                workspace.data_ptr())
        assert lib.tgt_edge_layout_build_i32(*args, narrow.value - 1, None, None) == 4     # TGT_ERR_WORKSPACE
        torch.cuda.synchronize()
        _cabi.check(lib.tgt_edge_layout_build_i32(*args, narrow.value, None, torch.cuda.current_stream().cuda_stream))
        assert (workspace[narrow.value:] == 171).all()
        want = elo.segment_layout(edges.numpy(), n_rows, group_by)
        for got, ref in zip((ptr, other, perm), want):
            assert np.array_equal(got.cpu().numpy().astype(np.int64), ref)


def test_a_graph_from_an_int32_list_allocates_no_narrow_copy():
    import ctypes
    from torchgt_b200 import _cabi
    from torchgt_b200.graph import SparseGraph
    n_rows, n_edges = 1000, 4_000_000
    edges = torch.randint(0, n_rows, (2, n_edges), dtype=torch.int32, device="cuda")
    need = ctypes.c_size_t()
    _cabi.check(_cabi.load().tgt_edge_layout_sizes_i32(n_rows, n_edges, ctypes.byref(need)))
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    torch.cuda.reset_peak_memory_stats()
    before = torch.cuda.memory_allocated()
    graph = SparseGraph(edges, n_rows)
    graph.check()
    # other, perm, seg and the workspace; a megabyte of rounding per allocation is below the 16 MB of a copy
    assert torch.cuda.max_memory_allocated() - before < 3 * 4 * n_edges + need.value + (6 << 20)


@pytest.mark.parametrize("n_rows,n_edges", [(1, 1), (3, 2), (40, 65), (70000, 200003), (5000, (1 << 20) - 1), (5000, 1 << 20),
                                            (70000, (1 << 20) + 63), (900, (1 << 20) + 64), (70000, (1 << 20) + 65)])
def test_second_orientation_from_what_the_first_kept(n_rows, n_edges):
    """The sources' layout from the endpoints the first build kept (same stream), from the list itself (another stream, as
    before), and the CPU's stable sort; rows without edges in runs of every length up to thousands."""
    from torchgt_b200 import SparseGraph
    gen = torch.Generator().manual_seed(n_edges)
    used = torch.randperm(n_rows, generator=gen)[:max(1, n_rows // 50)]
    ei = used[torch.randint(0, used.numel(), (2, n_edges), generator=gen)]
    here, there = SparseGraph(ei.cuda(), n_rows), SparseGraph(ei.cuda(), n_rows)
    kept = here.by_src
    torch.cuda.synchronize()
    with torch.cuda.stream(torch.cuda.Stream()):
        other = there.by_src
        torch.cuda.synchronize()
    perm = torch.sort(ei[0], stable=True).indices
    ptr = torch.cat([torch.zeros(1, dtype=torch.long), torch.bincount(ei[0], minlength=n_rows).cumsum(0)])
    for layout in (kept, other):
        assert torch.equal(layout.perm.cpu().long(), perm)
        assert torch.equal(layout.seg.cpu().long(), ei[0][perm])
        assert torch.equal(layout.other.cpu().long(), ei[1][perm])
        assert torch.equal(layout.ptr.cpu().long(), ptr)
    here.check()
    bad = ei.clone()
    bad[0, 0] = n_rows
    with pytest.raises(Exception, match="outside"):
        SparseGraph(bad.cuda(), n_rows).by_src.verify()


def test_what_is_kept_for_the_second_orientation_is_bounded():
    """A graph built where no gradients are recorded holds its one orientation and nothing else; elsewhere 8 bytes per edge
    more until the second is built, in the place of two of the workspace's arrays and not on top of them."""
    import ctypes
    from torchgt_b200 import SparseGraph, _cabi
    n_rows, n_edges = 4000, 1 << 21
    layout, slack = 4 * (3 * n_edges + n_rows), 6 << 20
    edges = torch.randint(0, n_rows, (2, n_edges), device="cuda")
    need, second = ctypes.c_size_t(), ctypes.c_size_t()
    _cabi.check(_cabi.load().tgt_edge_layout_sizes(n_rows, n_edges, ctypes.byref(need)))
    _cabi.check(_cabi.load().tgt_edge_layout_sizes_kept(n_rows, n_edges, ctypes.byref(second)))
    assert need.value - second.value == 8 * n_edges

    def build():
        torch.cuda.synchronize()
        before = torch.cuda.memory_allocated()
        torch.cuda.reset_peak_memory_stats()
        graph = SparseGraph(edges, n_rows)
        graph.check()
        return graph, before, torch.cuda.max_memory_allocated() - before, torch.cuda.memory_allocated() - before

    with torch.no_grad():
        graph, before, peak, held = build()
    assert peak < layout + need.value + slack
    assert held < layout + slack
    with torch.no_grad():
        by_src = graph.by_src                       # from the list itself
    assert torch.equal(by_src.seg.long(), edges[0].sort().values)
    del graph, by_src
    graph, before, peak, held = build()
    assert peak < layout + need.value + slack
    assert held < layout + 8 * n_edges + slack
    torch.cuda.reset_peak_memory_stats()
    graph.by_src.verify()
    assert torch.cuda.max_memory_allocated() - before < 2 * layout + 8 * n_edges + second.value + slack
    assert torch.cuda.memory_allocated() - before < 2 * layout + slack
