"""Batch construction on the GPU (csrc/batching.cu) against the PyTorch / numpy formulation on the CPU, which the
reference's own vectors pin (test_batching_gloo.py).  Integer work: every array bit for bit."""
import types

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _no_group():
    import torchgt_b200.gt_sp.initialize as init
    init.destroy_sequence_parallel()
    yield
    init.destroy_sequence_parallel()


def _graph(seed, n, m):
    gen = torch.Generator().manual_seed(seed)
    return torch.randint(0, n, (2, m), generator=gen), torch.randperm(n, generator=gen)


# sizes around the marking pass's chunk of 2048 candidates and its 256 threads, self loops and duplicates among them
@pytest.mark.parametrize("n,m,b", [(1, 0, 1), (5, 40, 5), (100, 1948, 60), (100, 1949, 99), (255, 5000, 1), (3000, 20000, 1500),
                                   (40000, 300001, 20000)])
def test_induced_subgraph(n, m, b):
    from torchgt_b200.gt_sp.utils import gen_sub_edge_index
    edges, perm = _graph(n + m, n, m)
    idx = perm[:b]
    want = gen_sub_edge_index(edges, idx, n)
    assert torch.equal(gen_sub_edge_index(edges.cuda(), idx.cuda(), n).cpu(), want)
    assert torch.equal(gen_sub_edge_index(edges.cuda(), (idx - n).cuda(), n).cpu(), want)   # counted from the end
    if m:
        edges[1, m // 2] = n
        with pytest.raises(IndexError):
            gen_sub_edge_index(edges.cuda(), idx.cuda(), n)


# unequal partitions (different bounds for rows and columns), one block per side (no random number drawn), more than
# 624 coordinates for a pair, partitions smaller than a block
@pytest.mark.parametrize("n,m,k,block", [(64, 500, 1, 4), (97, 400, 3, 4), (50, 300, 8, 5), (33, 200, 4, 16), (2000, 60000, 3, 4),
                                         (5000, 30000, 8, 16), (700, 3000, 70, 2)])
def test_block_generator(n, m, k, block):
    from torchgt_b200.gt_sp.batching import contiguous_partition, generate_new_edges_optimized, reformat_graph
    edges, perm = _graph(n * k + block, n, m)
    for part in (contiguous_partition(edges, n, k), (perm.double() / n).pow(1.5).mul(k).long()):
        mapping = np.argsort(np.argsort(part.numpy(), kind="stable"), kind="stable")
        for p in (1, 0.02):
            want = generate_new_edges_optimized(edges, k, part, p, block, mapping)
            assert torch.equal(generate_new_edges_optimized(edges.cuda(), k, part, p, block, mapping).cpu(), want)
        for ids in (part, None):
            want, order = reformat_graph(edges, k, block, partition_ids=ids)
            got, got_order = reformat_graph(edges.cuda(), k, block, partition_ids=ids)
            assert torch.equal(got.cpu(), want) and torch.equal(got_order.cpu(), order)


@pytest.mark.parametrize("model", ["graphormer", "gt"])
@pytest.mark.parametrize("reorder", [False, True])
@pytest.mark.parametrize("features,dtype", [(64, torch.float32), (3, torch.float32), (5, torch.bfloat16)])
def test_training_batch(model, reorder, features, dtype):
    from torchgt_b200.gt_sp.batching import get_batch_reorder_blockize, set_partitioner
    from torchgt_b200.gt_sp.initialize import get_last_batch_flag
    n, seq_len = 3001, 1000
    edges, perm = _graph(9, n, 25000)
    gen = torch.Generator().manual_seed(1)
    x, y = torch.randn(n, features, generator=gen).to(dtype), torch.randint(0, 40, (n,), generator=gen)
    args = types.SimpleNamespace(seq_len=seq_len, model=model, reorder=reorder)
    scatter = lambda e, nodes, k: ((torch.arange(nodes) * 13) % nodes) * k // nodes
    for idx, rest in ((perm[:seq_len], None), (perm[:777], [777]), (perm[:777], [800])):
        for partitioner in (None, scatter):
            set_partitioner(partitioner)
            try:
                want = get_batch_reorder_blockize(args, x, y, idx, rest, "cpu", edges, n, 4, 8)
                flag = get_last_batch_flag()
                got = get_batch_reorder_blockize(args, x.cuda(), y.cuda(), idx.cuda(), rest, "cuda", edges.cuda(), n, 4, 8)
            finally:
                set_partitioner(None)
            assert got[3] is None and get_last_batch_flag() == flag
            for a, b in zip(got[:3], want[:3]):
                assert a.dtype == b.dtype and torch.equal(a.cpu(), b)


@pytest.mark.parametrize("model", ["graphormer", "gt"])
@pytest.mark.parametrize("nodes,rest", [(1000, None), (777, [300, 300, 177, 0]), (250, [250, 0, 0, 0])])
def test_every_rank_takes_its_slice(model, nodes, rest, monkeypatch):
    """Slices that start inside the batch, end with it, or are empty, as four ranks take them (no collective is part of it)."""
    from torchgt_b200.gt_sp import batching
    n = 3001
    edges, perm = _graph(21, n, 25000)
    x, y, idx = torch.randn(n, 6), torch.arange(n), perm[:nodes]
    args = types.SimpleNamespace(seq_len=1000, model=model, reorder=False)
    monkeypatch.setattr(batching, "sequence_parallel_is_initialized", lambda: True)
    monkeypatch.setattr(batching, "get_sequence_parallel_world_size", lambda: 4)
    taken = []
    device_batch = batching._device_batch
    monkeypatch.setattr(batching, "_device_batch", lambda *a: (taken.append(a[-3:-1]), device_batch(*a))[1])
    for rank in range(4):
        monkeypatch.setattr(batching, "get_sequence_parallel_rank", lambda: rank)
        want = batching.get_batch_reorder_blockize(args, x, y, idx, rest, "cpu", edges, n, 4, 8)
        got = batching.get_batch_reorder_blockize(args, x.cuda(), y.cuda(), idx.cuda(), rest, "cuda", edges.cuda(), n, 4, 8)
        assert len(taken) == rank + 1
        for a, b in zip(got[:3], want[:3]):
            assert a.dtype == b.dtype and torch.equal(a.cpu(), b)
    if rest is not None:
        assert taken[-1] == (nodes, nodes)


def test_lists_the_kernels_cannot_number_take_the_pytorch_formulation(monkeypatch):
    from torchgt_b200.gt_sp import batching
    edges, perm = _graph(5, 300, 2000)
    want = batching.gen_sub_edge_index(edges, perm[:200], 300)
    monkeypatch.setattr(batching, "_MAX_CANDIDATES", 2300)
    no_kernels = types.SimpleNamespace(plain=lambda tensors: True)
    monkeypatch.setattr(batching._cabi, "native", lambda: no_kernels)
    assert torch.equal(batching.gen_sub_edge_index(edges.cuda(), perm[:200].cuda(), 300).cpu(), want)
    args = types.SimpleNamespace(seq_len=200, model="graphormer", reorder=False)
    x, y = torch.randn(300, 4), torch.arange(300)
    want = batching.get_batch_reorder_blockize(args, x, y, perm[:200], None, "cpu", edges, 300, 4, 8)
    got = batching.get_batch_reorder_blockize(args, x.cuda(), y.cuda(), perm[:200].cuda(), None, "cuda", edges.cuda(), 300, 4, 8)
    assert all(torch.equal(a.cpu(), b) for a, b in zip(got[:3], want[:3]))


def test_a_traced_sub_graph_runs_again_on_other_batches():
    from torchgt_b200.gt_sp.batching import gen_sub_edge_index
    edges, perm = _graph(5, 300, 2000)
    edges, perm = edges.cuda(), perm.cuda()
    traced = torch.jit.trace(lambda e, i: gen_sub_edge_index(e, i, 300), (edges, perm[:200]), check_trace=False)
    for idx in (perm[100:], perm[:50]):
        assert torch.equal(traced(edges, idx), gen_sub_edge_index(edges, idx, 300))


def test_features_with_a_pending_conjugation():
    from torchgt_b200.gt_sp.batching import get_batch_reorder_blockize
    edges, perm = _graph(5, 300, 2000)
    x, y = torch.randn(300, 4, dtype=torch.complex64), torch.arange(300)
    args = types.SimpleNamespace(seq_len=200, model="graphormer", reorder=False)
    got = get_batch_reorder_blockize(args, x.cuda().conj(), y.cuda(), perm[:200].cuda(), None, "cuda", edges.cuda(), 300, 4, 8)
    assert torch.equal(got[0].cpu(), x[perm[:200]].conj())


def test_block_generator_with_ids_outside_the_nodes_and_the_partitions():
    """What numpy's indexing makes of them: negative ids count from the end, a partition that no edge mentions may lie
    beyond k, an id beyond the nodes is an error."""
    from torchgt_b200.gt_sp.batching import contiguous_partition, generate_new_edges_optimized
    edges, _ = _graph(11, 200, 900)
    part = contiguous_partition(edges, 200, 4)
    mapping = np.arange(200)
    negative, alone, beyond = edges.clone(), part.clone(), edges.clone()
    negative[0, :50] -= 200
    edges_without_7 = edges[:, (edges != 7).all(0)]
    alone[7] = 4
    for e, p in ((negative, part), (edges_without_7, alone)):
        want = generate_new_edges_optimized(e, 4, p, 1, 8, mapping)
        assert torch.equal(generate_new_edges_optimized(e.cuda(), 4, p, 1, 8, mapping).cpu(), want)
    beyond[1, 5] = 200
    for e in (beyond, beyond.cuda()):
        with pytest.raises(IndexError):
            generate_new_edges_optimized(e, 4, part, 1, 8, mapping)


def test_threads_that_build_batches_leave_no_pinned_memory_behind():
    import threading
    from torchgt_b200.gt_sp.batching import gen_sub_edge_index
    edges, perm = _graph(5, 300, 2000)
    edges, idx, results = edges.cuda(), perm[:200].cuda(), []
    results.append(gen_sub_edge_index(edges, idx, 300))
    before = torch.cuda.host_memory_stats()
    for _ in range(100):
        thread = threading.Thread(target=lambda: results.append(gen_sub_edge_index(edges, idx, 300)))
        thread.start()
        thread.join()
    after = torch.cuda.host_memory_stats()
    assert all(torch.equal(r, results[0]) for r in results) and len(results) == 101
    assert after["active_requests.allocated"] >= before["active_requests.allocated"] + 100    # each call asked the pool,
    assert after["num_host_alloc"] == before["num_host_alloc"]                                  # which had what it needs
