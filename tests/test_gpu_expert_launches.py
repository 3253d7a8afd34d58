"""The launches of the expert layer, read from a captured graph: how many, and how many CTAs its GEMMs have."""
import pytest
import torch

from test_gpu_moe import _MoE, _bf16_default  # noqa: F401

pytestmark = pytest.mark.gpu

GEMM_THREADS = 384


def _kernels(call):
    """(CTAs, threads of a CTA) of every kernel that the call launches."""
    driver = pytest.importorskip("cuda.bindings.driver")
    call()
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph):
        y = call()
    raw = driver.CUgraph(graph.raw_cuda_graph())
    err, _, count = driver.cuGraphGetNodes(raw)
    assert int(err) == 0
    err, nodes, _ = driver.cuGraphGetNodes(raw, count)
    assert int(err) == 0
    found = []
    for node in nodes:
        err, kind = driver.cuGraphNodeGetType(node)
        if int(err) == 0 and kind == driver.CUgraphNodeType.CU_GRAPH_NODE_TYPE_KERNEL:
            err, k = driver.cuGraphKernelNodeGetParams(node)
            assert int(err) == 0
            found.append((k.gridDimX * k.gridDimY * k.gridDimZ, k.blockDimX))
    del y
    return found


def _layer(tokens):
    import dsv3_b200
    moe = _MoE(512, 512, 4, 2, 0, 4, seed=23)
    x = torch.randn(tokens, 512, generator=torch.Generator(device="cuda").manual_seed(tokens), device="cuda", dtype=torch.float32).bfloat16()
    routing = moe.gate(x)
    moe.gate, moe.shared_experts = lambda x: routing, lambda x: x
    return lambda: dsv3_b200.grouped_moe_forward(moe, x)


@pytest.mark.parametrize("tokens", [4, 40, 200])
def test_the_gemms_keep_to_an_sm_budget(tokens):
    """Two of them, each with no more CTAs than SMs it may occupy (all of a launch's can be resident at once)."""
    import dsv3_b200
    call = _layer(tokens)
    dsv3_b200.set_num_sms(8)
    try:
        gemms = [ctas for ctas, threads in _kernels(call) if threads == GEMM_THREADS]
    finally:
        dsv3_b200.set_num_sms(0)
    assert len(gemms) == 2 and max(gemms) <= 8


@pytest.mark.parametrize("tokens", [40, 200])
def test_four_launches_whatever_the_tiles(tokens):
    """Groups that are divided between two kinds of tiles are worked on in one launch: all of its CTAs wait for what came before."""
    assert len(_kernels(_layer(tokens))) == 4
