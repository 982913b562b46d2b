"""The encoder layer as one call into the host module against its modules one by one: the same operations, the same bits."""
import pytest
import torch
from torch import nn

pytestmark = pytest.mark.gpu


def _step(layer, x, graph, dy):
    layer.zero_grad(set_to_none=True)
    leaf = x.clone().requires_grad_()
    y = layer(leaf, None, graph, "sparse")
    y.backward(dy)
    return [y.detach(), leaf.grad] + [p.grad for p in layer.parameters()]


def _layer(hidden, heads, ffn, nodes):
    from torchgt_b200 import SparseGraph
    from torchgt_b200.graphormer import EncoderLayer
    torch.manual_seed(nodes)
    layer = EncoderLayer(hidden, ffn, 0.0, 0.0, heads).cuda()
    edges = torch.randint(0, nodes, (2, 6 * nodes), device="cuda")
    x, dy = (torch.randn(1, nodes, hidden, device="cuda") for _ in range(2))
    return layer, SparseGraph(edges, nodes), x, dy


@pytest.mark.parametrize("tf32", [False, True])
@pytest.mark.parametrize("hidden,heads,ffn,nodes", [(64, 8, 64, 300), (64, 8, 64, 1500), (64, 4, 128, 5000), (32, 4, 64, 2000),
                                                    (128, 8, 64, 20000)])
def test_one_call_gives_the_bits_of_the_modules(hidden, heads, ffn, nodes, tf32):
    before = torch.backends.cuda.matmul.allow_tf32
    torch.backends.cuda.matmul.allow_tf32 = tf32
    try:
        layer, graph, x, dy = _layer(hidden, heads, ffn, nodes)
        assert layer._native_layer(x, None, graph, "sparse") is not None
        together = _step(layer, x, graph, dy)
        with torch.no_grad():
            assert torch.equal(layer(x, None, graph, "sparse"), together[0])
        layer._native_layer = lambda *args: None            # the same layer through its modules
        for a, b in zip(together, _step(layer, x, graph, dy)):
            assert torch.equal(a, b)
    finally:
        torch.backends.cuda.matmul.allow_tf32 = before


def test_what_can_be_noticed_goes_through_the_modules():
    layer, graph, x, _ = _layer(64, 8, 64, 1200)
    call = lambda: layer._native_layer(x, None, graph, "sparse")   # noqa: E731
    assert call() is not None
    for module in (layer.self_attention, layer.self_attention.linear_v, layer.ffn_norm, layer.ffn, layer.ffn.layer2,
                   layer.self_attention.dist_attn.local_attn):
        handle = module.register_forward_hook(lambda *args: None)
        assert call() is None
        handle.remove()
    handle = nn.modules.module.register_module_forward_hook(lambda *args: None)
    assert call() is None
    handle.remove()
    layer.ffn_dropout.p = 0.5
    assert call() is None
    layer.eval()
    assert call() is not None
    layer.ffn.gelu = nn.GELU(approximate="tanh")
    assert call() is None
    layer.ffn.gelu = nn.GELU()
    assert layer._native_layer(x, torch.zeros(1, device="cuda"), graph, "sparse") is None
    assert layer._native_layer(x, None, graph, None) is None
    assert layer._native_layer(x.double(), None, graph, "sparse") is None
    with torch.autocast("cuda", dtype=torch.bfloat16):
        assert call() is None
    with pytest.raises(ValueError, match="rows"):
        layer._native_layer(x[:, 1:], None, graph, "sparse")


@pytest.mark.parametrize("nodes", [300, 1500])
@pytest.mark.parametrize("name", ["linear_q", "linear_k", "linear_v"])
@pytest.mark.parametrize("width", [32, 128])
def test_projections_of_unequal_widths_are_refused(name, width, nodes):
    """The kernels read and write rows of heads * head_dim values: a layer with a pruned or replaced projection goes through
    its modules, which refuse it."""
    from torchgt_b200.linear import Linear
    layer, graph, x, _ = _layer(64, 8, 64, nodes)
    mha = layer.self_attention
    setattr(mha, name, Linear(64, width).cuda())
    assert layer._native_layer(x, None, graph, "sparse") is None
    with pytest.raises(ValueError):
        layer(x, None, graph, "sparse")


@pytest.mark.parametrize("wrong", ["rows", "heads", "dtype"])
def test_the_attention_itself_refuses_rows_that_are_not_the_graphs(wrong):
    from torchgt_b200 import _cabi
    _, graph, _, _ = _layer(64, 8, 64, 300)
    native = _cabi.native()
    good = torch.randn(300, 8, 8, device="cuda")
    other = {"rows": good[:299], "heads": good[:, :4], "dtype": good.bfloat16()}[wrong]
    calls = [(other, good, good), (good, other, good), (good, good, other)] + ([(other,) * 3] if wrong == "rows" else [])
    for q, k, v in calls:
        for run in (lambda: native.attention(q, k, v, None, graph.native), lambda: native.attention_forward(q, k, v, None, graph.native)):
            with pytest.raises(TypeError if wrong == "dtype" else ValueError):
                run()


def test_the_attention_itself_refuses_a_bias_of_other_edges():
    """A traced call checks its arguments when it is traced; it runs again on whatever it is given."""
    from torchgt_b200 import _cabi, sparse_graph_attention
    _, graph, _, _ = _layer(64, 8, 64, 300)
    rows = [torch.randn(300, 8, 8, device="cuda") for _ in range(3)]
    bias = torch.zeros(graph.n_edges, device="cuda")
    traced = torch.jit.trace(lambda q, k, v, b: sparse_graph_attention(q, k, v, graph, b), (*rows, bias), check_trace=False)
    assert torch.equal(traced(*rows, bias), sparse_graph_attention(*rows, graph, bias))
    with pytest.raises(Exception, match="bias must be"):
        traced(*rows, bias[:-1].contiguous())
    for wrong in (bias[:-1], bias.double(), bias.view(-1, 1).expand(-1, 4)):
        with pytest.raises(ValueError, match="bias must be"):
            _cabi.native().attention(*rows, wrong, graph.native)
    with pytest.raises(Exception, match="share the shape"):
        traced(*(t[:299] for t in rows), bias)
