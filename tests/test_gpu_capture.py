"""State that the host extension keeps between calls, across the boundary of a CUDA graph: workspaces,
remembered quantisations and de-quantised weights.

A pass through a graph must not depend on which other graph, or which eager call, came before it."""
import pytest
import torch

from test_gpu_moe import _MoE
from test_gpu_stream import _bf16_default, _weight  # noqa: F401

pytestmark = pytest.mark.gpu


def _polluted_pool(stream):
    """A graph pool whose free blocks hold non-zero bytes; the graph that keeps it alive."""
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        blocks = [torch.full((24 << 20,), 7, dtype=torch.uint8, device="cuda") for _ in range(8)]
    graph.replay()
    torch.cuda.synchronize()
    del blocks
    return graph


def _split_linear():
    """A Linear whose K is split with tickets."""
    import dsv3_b200
    import kernel
    g = torch.Generator(device="cuda").manual_seed(5)
    a, a_s = kernel.act_quant(torch.randn(8, 4096, generator=g, device="cuda", dtype=torch.float32).bfloat16())
    w = _weight(1024, 4096, g)
    dsv3_b200.set_gemm_policy(dsv3_b200.KERNEL_TC_WEIGHT_MAJOR, 4)
    return lambda: kernel.fp8_gemm(a, a_s, w, w.scale)


def _cut_experts():
    """An expert layer with few tiles of many K chunks, which are cut."""
    import dsv3_b200
    moe = _MoE(4096, 256, 8, 2, 0, 8, seed=11)
    x = torch.randn(2, 4096, generator=torch.Generator(device="cuda").manual_seed(6), device="cuda", dtype=torch.float32).bfloat16()
    return lambda: dsv3_b200.grouped_moe_forward(moe, x)


@pytest.mark.parametrize("make", [_split_linear, _cut_experts])
@pytest.mark.parametrize("order", ["second graph first", "eager call first"])
def test_ticket_header_of_a_workspace_that_a_capture_made(order, make):
    """Two graphs captured on one stream, the first of them replayed last (or after an eager call)."""
    call = make()
    want = call()
    stream = torch.cuda.Stream()
    keep = _polluted_pool(stream)
    graphs, outs = [], []
    for _ in range(2):
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, pool=keep.pool(), stream=stream):
            outs.append(call())
        graphs.append(graph)
    torch.cuda.synchronize()
    if order == "eager call first":
        with torch.cuda.stream(stream):
            got = call()
        stream.synchronize()
        assert torch.equal(got, want)
    for i in (1, 0, 1):
        outs[i].fill_(float("nan"))
        graphs[i].replay()
        torch.cuda.synchronize()
        assert torch.equal(outs[i], want)


def _inputs():
    g = torch.Generator(device="cuda").manual_seed(8)
    x = torch.randn(2, 40, 1024, generator=g, device="cuda", dtype=torch.float32).bfloat16()
    return x[0].clone(), x[1].clone(), _weight(256, 1024, g), _weight(384, 1024, g)


def test_a_graph_does_not_use_the_quantisation_of_an_eager_call():
    """The usual order of a host: a warm pass and the capture on one stream, then replays with new contents."""
    from dsv3_b200 import linear_seam as L
    x, new, w, w3 = _inputs()
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        L.linear(x, w)
    stream.synchronize()
    L.stats.update(act_quant_calls=0, act_quant_reused=0)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        y, y3 = L.linear(x, w), L.linear(x, w3)
    assert (L.stats["act_quant_calls"], L.stats["act_quant_reused"]) == (1, 1), "shared inside the capture"
    want, want3 = L.linear(new, w), L.linear(new, w3)
    x.copy_(new)
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(y, want) and torch.equal(y3, want3)


def test_an_eager_call_does_not_use_the_quantisation_of_a_graph():
    """A quantisation recorded in a capture has not been computed; another capture does not own it either."""
    from dsv3_b200 import linear_seam as L
    x, _, w, w3 = _inputs()
    want, want3 = L.linear(x.clone(), w), L.linear(x.clone(), w3)
    stream = torch.cuda.Stream()
    keep = _polluted_pool(stream)
    graphs, outs = [], []
    for _ in range(2):
        graphs.append(torch.cuda.CUDAGraph())
        with torch.cuda.graph(graphs[-1], pool=keep.pool(), stream=stream):
            outs.append(L.linear(x, w3))
    with torch.cuda.stream(stream):
        got = L.linear(x, w)
    stream.synchronize()
    assert torch.equal(got, want)
    for i in (1, 0):
        graphs[i].replay()
        torch.cuda.synchronize()
        assert torch.equal(outs[i], want3)


def test_a_de_quantised_weight_of_a_graph_is_not_remembered():
    """weight_dequant's cache: what a capture recorded is computed at its replays, an eager call before them computes its own."""
    import dsv3_b200
    import kernel
    w = _weight(512, 512, torch.Generator(device="cuda").manual_seed(2))
    want = kernel.weight_dequant(w, w.scale)
    stream = torch.cuda.Stream()
    keep = _polluted_pool(stream)
    graph = torch.cuda.CUDAGraph()
    dsv3_b200.enable_weight_dequant_cache()
    try:
        with torch.cuda.graph(graph, pool=keep.pool(), stream=stream):
            y = kernel.weight_dequant(w, w.scale)
        got = kernel.weight_dequant(w, w.scale)
        assert torch.equal(got, want)
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(y, want) and kernel.weight_dequant(w, w.scale) is got
    finally:
        dsv3_b200.disable_weight_dequant_cache()
