"""The expert layer for a handful of tokens as its callers use it: what it takes and refuses, and when the weights are read."""
import pytest
import torch

from test_gpu_moe import _MoE, _bf16_default  # noqa: F401

pytestmark = pytest.mark.gpu


def _layer(topk=2, tokens=2, n_routed=64, local=4, dim=512, inter=256):
    moe = _MoE(dim, inter, n_routed, topk, 0, local, seed=17)
    x = torch.randn(tokens, dim, generator=torch.Generator(device="cuda").manual_seed(5), device="cuda", dtype=torch.float32).bfloat16()
    return moe, x


def test_more_experts_per_token_than_the_dispatch_takes_are_refused():
    """At most 32, as with more tokens."""
    import dsv3_b200
    moe, x = _layer(tokens=1, local=2)
    for topk in (32, 33):
        indices = torch.arange(topk, device="cuda").view(1, topk)
        moe.gate = lambda x: (torch.ones(1, topk, device="cuda"), indices)
        if topk == 32:
            assert dsv3_b200.grouped_moe_forward(moe, x).shape == x.shape
        else:
            with pytest.raises(dsv3_b200.Dsv3Error) as e:
                dsv3_b200.grouped_moe_forward(moe, x)
            assert e.value.status == -2


@pytest.mark.parametrize("world_size", [1, 2])
def test_weights_are_read_before_the_shared_experts_are_called(world_size, monkeypatch):
    """A host may give the routed experts' weights other contents (the next layer's, say) from there on."""
    import dsv3_b200
    monkeypatch.setattr(torch.distributed, "all_reduce", lambda y: y.mul_(2))
    moe, x = _layer()
    moe.gate = lambda x: (torch.ones(2, 2, device="cuda"), torch.tensor([[0, 1], [3, 60]], device="cuda"))
    z = torch.randn(2, 512, device="cuda")
    moe.shared_experts = lambda x: z
    want = dsv3_b200.grouped_moe_forward(moe, x, world_size=world_size)

    def overwrite(x):
        for e in moe.experts[:4]:
            e.w2.weight.view(torch.uint8).zero_()
        return z

    moe.shared_experts = overwrite
    assert torch.equal(dsv3_b200.grouped_moe_forward(moe, x, world_size=world_size), want)
    assert not torch.equal(want, z)


def _close(got, want):
    err, rms = (got.float() - want.float()).abs(), want.float().pow(2).mean().sqrt()
    return bool((err <= 2e-2 * (want.float().abs() + rms)).all())               # the bound of test_gpu_moe.py


ROUTINGS = [[[0, 1], [2, 3]], [[3, 3], [3, 3]], [[9, 60], [17, 2]], [[10, 11], [12, 13]]]      # all, one, one pair, none of them local


def test_replays_of_a_graph_follow_the_routing():
    import dsv3_b200
    from test_gpu_few_experts import _pairs_one_by_one
    moe, x = _layer()
    weights, indices = torch.ones(2, 2, device="cuda"), torch.tensor(ROUTINGS[0], device="cuda")
    moe.gate, moe.shared_experts = lambda x: (weights, indices), lambda x: torch.zeros_like(x)
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        dsv3_b200.grouped_moe_forward(moe, x)
    stream.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        y = dsv3_b200.grouped_moe_forward(moe, x)
    for step, routing in enumerate(ROUTINGS[1:] + ROUTINGS):
        indices.copy_(torch.tensor(routing))
        weights.uniform_(0.2, 1.0)
        x.normal_()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(y, dsv3_b200.grouped_moe_forward(moe, x)), step
        assert _close(y, _pairs_one_by_one(moe, x, weights, indices)), step
    dsv3_b200.check_device_status()


@pytest.mark.parametrize("world_size", [1, 2])
def test_shared_experts_beside_the_two_launches(world_size, monkeypatch):
    """In the same launches, and behind them where there are several ranks."""
    import dsv3_b200
    from test_gpu_few_experts import _pairs_one_by_one
    from test_gpu_moe_calls import _host
    monkeypatch.setattr(torch.distributed, "all_reduce", lambda y: y.mul_(2))
    moe, x = _host()
    x = x[:1]
    weights, indices = torch.tensor([[0.3, 0.7]], device="cuda"), torch.tensor([[3, 1]], device="cuda")
    moe.gate = lambda x: (weights, indices)
    want = _pairs_one_by_one(moe, x, weights, indices) * world_size + moe.shared_experts(x)
    for _ in range(2):
        assert _close(dsv3_b200.grouped_moe_forward(moe, x, world_size=world_size), want)


def test_two_threads():
    """Layers of different sizes, each thread on a stream of its own."""
    import threading
    import dsv3_b200
    calls, wrong = [], []
    for tokens, dim, inter in ((2, 512, 256), (1, 2048, 384)):
        moe, x = _layer(tokens=tokens, dim=dim, inter=inter)
        moe.shared_experts = lambda x: torch.zeros_like(x)
        routing = torch.rand(tokens, 2, device="cuda"), torch.tensor(ROUTINGS[0][:tokens], device="cuda")
        moe.gate = lambda x, routing=routing: routing
        calls.append((moe, x, dsv3_b200.grouped_moe_forward(moe, x)))
    torch.cuda.synchronize()

    def repeat(moe, x, want):
        torch.set_default_dtype(torch.bfloat16)
        with torch.cuda.stream(torch.cuda.Stream()):
            wrong.append(torch.stack([(dsv3_b200.grouped_moe_forward(moe, x) != want).any() for _ in range(200)]).any())
            torch.cuda.current_stream().synchronize()

    threads = [threading.Thread(target=repeat, args=c) for c in calls]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert len(wrong) == 2 and not any(bool(w) for w in wrong)
