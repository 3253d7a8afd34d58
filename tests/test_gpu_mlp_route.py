"""An MLP that only the host's launches are a reason to run in three launches: so from Python, in five in a graph."""
import pytest
import torch

from test_gpu_expert_launches import _kernels
from test_gpu_mlp_launches import _host, _i64, _rows
from test_gpu_stream import _bf16_default  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,dim,inter", [(6, 2048, 1408), (24, 7168, 2304), (2, 2048, 1408)])
def test_a_graph_takes_what_is_faster_on_the_device(M, dim, inter):
    from dsv3_b200 import _lib
    from dsv3_b200._lib import host
    assert not _lib.lib.dsv3_swiglu_linear_pays(_i64(M), _i64(inter), _i64(dim))
    mlp, model = _host(dim, inter)
    x = _rows(M, dim)
    args = (mlp.w1.weight, mlp.w3.weight, mlp.w2.weight, None, None, False)
    want = mlp(x)
    assert torch.equal(host.mlp(x, *args), want), "three launches"
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        assert host.mlp(x, *args) is None
        got = mlp(x)
    graph.replay()
    err, rms = (got.float() - want.float()).abs(), want.float().pow(2).mean().sqrt()
    assert bool((err <= 2e-2 * (want.float().abs() + rms)).all())         # the bound of test_gpu_moe.py: sums in another order
    # w1 and w3 with their activations quantised inside (one or two rows), or after a launch of its own
    assert len(_kernels(lambda: mlp(x.view(x.shape)))) == (4 if M <= 2 else 5)


def test_a_pinned_gemm_is_honoured():
    import dsv3_b200
    mlp, model = _host(2048, 1408)
    x = _rows(64, 2048)
    dsv3_b200.set_gemm_policy(dsv3_b200.KERNEL_CUDA_CORE, 0)
    assert len(_kernels(lambda: mlp(x.view(x.shape)))) == 5
    dsv3_b200.set_gemm_policy(dsv3_b200.KERNEL_TC_TOKEN_PAIR, 0)
    with pytest.raises(dsv3_b200.Dsv3Error):                               # more than 128 rows only
        mlp(x.view(x.shape))
