"""The calls that an inference host makes into this library, as cases that can be timed.

A case is a dict of plain values.  `prepare` builds what the host holds before the call (weights in the checkpoint's
block-scaled FP8 format, activations, routing results, a captured graph where the host replays one), `run` makes one
pass through the public entry points, `work` says what the pass cannot do without, `tolerance` how far two correct
implementations of it may be apart.  Dimensions are those of the configurations that bench.py and the tests use
(hidden sizes 7168, 5120 and 2048 with their MLA, MLP and expert widths), whole or as one rank's tensor-parallel shard.
"""
import os
import statistics
import sys
import types

import torch

_PACKAGE = os.path.join(os.getcwd(), "deepseek-v3_b200")
if _PACKAGE not in sys.path:
    sys.path.insert(0, _PACKAGE)

import dsv3_b200  # noqa: E402
import kernel  # noqa: E402

torch.set_default_dtype(torch.bfloat16)  # as every entry point of such a host does before it builds the model


# ---------------------------------------------------------------------------------------------------------------------
# The host: the few classes of a model that the seams attach to, with the dispatch of the model they stand for
# ---------------------------------------------------------------------------------------------------------------------
class Linear:
    """An FP8 Linear: weight [out, in] with its scales as an attribute, called through the model's `linear`."""

    def __init__(self, weight, scale, scale_fmt=None):
        self.weight, self.bias, self.scale_fmt = weight, None, scale_fmt
        self.weight.scale = scale

    def __call__(self, x):
        return model.linear(x, self.weight, self.bias, self.scale_fmt)


class MLP:
    def __init__(self, w1, w2, w3):
        self.w1, self.w2, self.w3 = w1, w2, w3

    def forward(self, x):
        return self.w2(torch.nn.functional.silu(self.w1(x)) * self.w3(x))

    def __call__(self, x):
        return self.forward(x)


class Expert(MLP):
    def forward(self, x):
        return self.w2(torch.nn.functional.silu(self.w1(x)) * self.w3(x))


class MoE:
    """The router belongs to the host and is not part of the library: `gate` hands over its result."""

    def __init__(self, dim, n_routed, start, experts, shared):
        self.dim, self.n_routed_experts, self.n_local_experts = dim, n_routed, len(experts)
        self.experts_start_idx, self.experts_end_idx = start, start + len(experts)
        self.experts = [None] * start + list(experts) + [None] * (n_routed - start - len(experts))
        self.shared_experts = shared
        self.routing = None

    def gate(self, x):
        return self.routing

    def forward(self, x):
        raise NotImplementedError("replaced by install_moe")

    def __call__(self, x):
        return self.forward(x)


model = types.SimpleNamespace(gemm_impl="fp8", block_size=128, world_size=1, dist=None, MLP=MLP, Expert=Expert, MoE=MoE)
dsv3_b200.install_linear(model)
dsv3_b200.install_mlp(model)
dsv3_b200.install_moe(model)


# ---------------------------------------------------------------------------------------------------------------------
# Cases
# ---------------------------------------------------------------------------------------------------------------------
def listed():
    return [
        # absorbed attention de-quantises one rank's wkv_b in every layer of every decode step
        {"name": "dequant_wkv_b_shard", "kind": "weight_dequant", "rows": 4096, "cols": 512},
        # conversion of an FP8 checkpoint to bf16, its largest matrices
        {"name": "dequant_checkpoint", "kind": "weight_dequant", "rows": 18432, "cols": 7168},
        # quantisation of a prefill's hidden states
        {"name": "quant_prefill", "kind": "act_quant", "rows": 16384, "cols": 7168, "fmt": "fp32"},
        # the drop-in operators in the unchanged model: one token ...
        {"name": "linear_decode_1", "kind": "linear", "rows": 1, "k": 7168, "n": 1536, "fmt": "fp32"},
        # ... a batch of decoding sequences on the attention output projection ...
        {"name": "linear_decode_32", "kind": "linear", "rows": 32, "k": 16384, "n": 7168, "fmt": "fp32"},
        # ... an uneven prompt on the narrow latent projection, power-of-two scales ...
        {"name": "linear_prompt_ragged", "kind": "linear", "rows": 1003, "k": 7168, "n": 576, "fmt": "ue8m0"},
        # ... and a full prefill batch
        {"name": "linear_prefill_4096", "kind": "linear", "rows": 4096, "k": 16384, "n": 7168, "fmt": "fp32"},
        # dense MLP of a long prefill through the seams
        {"name": "mlp_prefill_8192", "kind": "mlp", "rows": 8192, "dim": 7168, "inter": 18432, "fmt": "fp32"},
        # expert layer of a prefill, all experts on the device
        {"name": "moe_prefill_2048", "kind": "moe", "rows": 2048, "dim": 7168, "inter": 2048, "experts": 256, "local": 256,
         "topk": 8, "shared": 1, "fmt": "fp32"},
        # expert layer of the small configuration, an uneven prompt
        {"name": "moe_small_ragged", "kind": "moe", "rows": 333, "dim": 2048, "inter": 1408, "experts": 64, "local": 64,
         "topk": 6, "shared": 2, "fmt": "fp32"},
        # one layer of a decode step of a single sequence, one rank's shards of eight, launched from Python
        {"name": "layer_decode_1", "kind": "layer", "rows": 1, "layers": 1, "ranks": 8, "graph": False},
        # two layers of a decode step of sixteen sequences, replayed as a CUDA graph
        {"name": "layer_decode_16_graph", "kind": "layer", "rows": 16, "layers": 2, "ranks": 8, "graph": True},
    ]


#: (in, out) of the Linears of the configurations, whole and as shards over eight ranks
_SHAPES = [(7168, 1536), (7168, 576), (16384, 7168), (7168, 18432), (7168, 2048), (2048, 7168), (1536, 24576), (1536, 3072),
           (512, 32768), (512, 4096), (7168, 2304), (2304, 7168), (256, 7168), (7168, 256), (5120, 1536),
           (5120, 12288), (12288, 5120), (2048, 10944), (2048, 1408), (1408, 2048), (2048, 3072), (2048, 576)]
#: (hidden, expert width, experts, experts per token, shared experts)
_EXPERT_LAYERS = [(7168, 2048, 256, 8, 1), (5120, 1536, 160, 6, 2), (2048, 1408, 64, 6, 2)]


def _log(rng, lo, hi):
    """A whole number between lo and hi, spread over its logarithm."""
    return max(lo, min(hi, int(round(lo * (hi / lo) ** rng.random()))))


def draw(rng):
    kind = rng.choice(["weight_dequant", "act_quant", "linear", "linear", "linear", "linear", "mlp", "moe", "moe", "layer"])
    fmt = rng.choice(["fp32", "fp32", "ue8m0"])
    if kind == "weight_dequant":
        rows, cols = _log(rng, 500, 24576), 32 * _log(rng, 16, 512)
        while rows * cols > 18432 * 7168:
            rows = max(1, rows // 2)
        return {"kind": kind, "rows": rows, "cols": cols}
    if kind == "act_quant":
        rows, cols = _log(rng, 1, 32768), 128 * _log(rng, 4, 144)
        while rows * cols > 16384 * 7168:
            rows = max(1, rows // 2)
        return {"kind": kind, "rows": rows, "cols": cols, "fmt": fmt}
    if kind == "linear":
        rows = _log(rng, 1, 16384)
        k, n = rng.choice(_SHAPES) if rng.random() < 0.6 else (128 * _log(rng, 4, 128), 16 * _log(rng, 16, 1152))
        while 2.0 * rows * k * n > 2e12:
            rows = max(1, rows * 2 // 3)
        return {"kind": kind, "rows": rows, "k": k, "n": n, "fmt": fmt}
    if kind == "mlp":
        dim, inter = rng.choice([(7168, 18432), (7168, 2304), (7168, 2048), (5120, 12288), (2048, 2816), (2048, 1408)])
        return {"kind": kind, "rows": _log(rng, 1, 8192), "dim": dim, "inter": inter, "fmt": fmt}
    if kind == "moe":
        dim, inter, experts, topk, shared = rng.choice(_EXPERT_LAYERS)
        return {"kind": kind, "rows": _log(rng, 1, 4096), "dim": dim, "inter": inter, "experts": experts,
                "local": experts // rng.choice([1, 2, 4, 8]), "topk": topk, "shared": shared, "fmt": fmt}
    return {"kind": kind, "rows": _log(rng, 1, 96), "layers": rng.choice([1, 2]), "ranks": rng.choice([8, 16]),
            "graph": rng.random() < 0.5}


# ---------------------------------------------------------------------------------------------------------------------
# What the host holds before the call
# ---------------------------------------------------------------------------------------------------------------------
class _Source:
    """Seeded inputs, made on the device: N(0, 1) activations, N(0, 0.02) weights quantised per 128 x 128 block."""

    def __init__(self, seed):
        self.g = torch.Generator(device="cuda").manual_seed(int(seed))

    def rows(self, *shape):
        return torch.randn(*shape, device="cuda", dtype=torch.bfloat16, generator=self.g)

    def weight(self, n, k):
        w = self.rows(n, k)
        w *= 0.02
        return dsv3_b200.weight_quant(w)

    def linear(self, n, k, fmt=None):
        return Linear(*self.weight(n, k), fmt)

    def mlp(self, dim, inter, fmt=None, cls=MLP):
        return cls(self.linear(inter, dim, fmt), self.linear(dim, inter, fmt), self.linear(inter, dim, fmt))

    def experts(self, count, dim, inter, fmt=None):
        """The widths are multiples of 128, so the experts of one projection are quantised together."""
        made = []
        for n, k in ((inter, dim), (dim, inter), (inter, dim)):
            w, s = self.weight(count * n, k)
            made.append([Linear(a, b, fmt) for a, b in zip(w.view(count, n, k).unbind(0), s.view(count, n // 128, k // 128).unbind(0))])
        return [Expert(w1, w2, w3) for w1, w2, w3 in zip(*made)]

    def routing(self, rows, experts, topk):
        """What a router hands over: unlike experts (some are asked for more often), normalised weights."""
        scores = torch.randn(rows, experts, device="cuda", dtype=torch.float32, generator=self.g)
        scores += 0.5 * torch.randn(experts, device="cuda", dtype=torch.float32, generator=self.g)
        top, index = scores.sigmoid().topk(topk, dim=-1)
        return (top / top.sum(dim=-1, keepdim=True) * 2.5).to(torch.bfloat16), index

    def moe(self, rows, dim, inter, experts, local, topk, shared_width, fmt=None):
        start = (experts - local) // 2 // 8 * 8
        m = MoE(dim, experts, start, self.experts(local, dim, inter, fmt), self.mlp(dim, shared_width, fmt))
        m.routing = self.routing(rows, experts, topk)
        return m


class _Layer:
    """One rank's shards of a layer of the large configuration: MLA projections and the expert layer.  Attention,
    norms and the held bf16 copy of wkv_b are the host's own."""

    def __init__(self, src, rows, ranks):
        heads = 128 // ranks
        self.wq_a, self.wq_b = src.linear(1536, 7168), src.linear(heads * 192, 1536)
        self.wkv_a, self.wo = src.linear(576, 7168), src.linear(7168, heads * 128)
        self.moe = src.moe(rows, 7168, 2048, 256, 256 // ranks, 8, 2048 // ranks)
        self.hidden, self.attended, self.normed = src.rows(rows, 7168), src.rows(rows, heads * 128), src.rows(rows, 7168)

    def __call__(self):
        # a view is a tensor of its own, as a new step's hidden state is
        x = self.hidden.view(self.hidden.shape)
        return self.wq_b(self.wq_a(x)), self.wkv_a(x), self.wo(self.attended.view(self.attended.shape)), self.moe(self.normed)


def _fmt(case):
    return "ue8m0" if case.get("fmt") == "ue8m0" else None


_side_stream = None


def _captured(layers):
    """The host's decode step as a CUDA graph: one warm pass, then the capture, both on a stream of their own."""
    global _side_stream
    _side_stream = _side_stream or torch.cuda.Stream()
    _side_stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(_side_stream):
        for layer in layers:
            layer()
    _side_stream.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=_side_stream):
        out = [layer() for layer in layers]
    return graph, out


def prepare(case, seed):
    src, kind = _Source(seed), case["kind"]
    if kind == "weight_dequant":
        return {"kind": kind, "w": src.weight(case["rows"], case["cols"])}
    if kind == "act_quant":
        return {"kind": kind, "x": src.rows(case["rows"], case["cols"]), "fmt": _fmt(case)}
    if kind == "linear":
        return {"kind": kind, "x": src.rows(case["rows"], case["k"]), "w": src.weight(case["n"], case["k"]), "fmt": _fmt(case)}
    if kind == "mlp":
        return {"kind": kind, "x": src.rows(case["rows"], case["dim"]), "mlp": src.mlp(case["dim"], case["inter"], _fmt(case))}
    if kind == "moe":
        m = src.moe(case["rows"], case["dim"], case["inter"], case["experts"], case["local"], case["topk"],
                    case["shared"] * case["inter"], _fmt(case))
        return {"kind": kind, "x": src.rows(case["rows"], case["dim"]), "moe": m}
    layers = [_Layer(src, case["rows"], case["ranks"]) for _ in range(case["layers"])]
    if not case["graph"]:
        return {"kind": kind, "layers": layers}
    graph, out = _captured(layers)
    return {"kind": "graph", "layers": layers, "graph": graph, "out": out}


# ---------------------------------------------------------------------------------------------------------------------
# One pass
# ---------------------------------------------------------------------------------------------------------------------
def run(state):
    kind = state["kind"]
    if kind == "weight_dequant":
        return kernel.weight_dequant(*state["w"])
    if kind == "act_quant":
        return kernel.act_quant(state["x"], 128, state["fmt"])
    if kind == "linear":
        xq, xs = kernel.act_quant(state["x"], 128, state["fmt"])
        return kernel.fp8_gemm(xq, xs, *state["w"])
    if kind == "mlp":
        return state["mlp"](state["x"].view(state["x"].shape))
    if kind == "moe":
        return state["moe"](state["x"])
    if kind == "layer":
        return [layer() for layer in state["layers"]]
    state["graph"].replay()
    return state["out"]


# ---------------------------------------------------------------------------------------------------------------------
# What a pass cannot do without, and how exact it is
# ---------------------------------------------------------------------------------------------------------------------
def _linear_work(m, k, n):
    """bf16 in, FP8 weight and its scales, bf16 out."""
    return 2 * m * k + n * k + 4 * -(-n // 128) * -(-k // 128) + 2 * m * n, 2.0 * m * k * n


def _mlp_work(m, dim, inter):
    return 2 * m * dim + 3 * inter * dim + 12 * -(-inter // 128) * -(-dim // 128) + 2 * m * dim, 6.0 * m * dim * inter


def _touched(m, experts, topk):
    """Expected share of the experts that m tokens ask for, under the scores of _Source.routing: noise N(0, 1) plus an
    expert's own N(0, 0.5), the highest topk / experts of them chosen."""
    normal = statistics.NormalDist()
    bar = 1.25 ** 0.5 * normal.inv_cdf(1.0 - topk / experts)
    likings = [0.5 * normal.inv_cdf((i + 0.5) / 200) for i in range(200)]
    return sum(1.0 - normal.cdf(bar - z) ** m for z in likings) / len(likings)


def _moe_work(m, dim, inter, experts, local, topk, shared_width):
    """Weights of the local experts that the router is expected to touch, the hidden states once in and once out;
    arithmetic of the local share of the pairs and of the shared expert."""
    touched = local * _touched(m, experts, topk)
    by, fl = _mlp_work(m, dim, shared_width)
    return by + touched * (3 * inter * dim + 12 * (inter // 128) * (dim // 128)) + 12 * m * topk, fl + 6.0 * m * topk * local / experts * dim * inter


def work(case):
    kind = case["kind"]
    if kind == "weight_dequant":
        r, c = case["rows"], case["cols"]
        return {"bytes": 3 * r * c + 4 * -(-r // 128) * -(-c // 128), "flops": r * c}
    if kind == "act_quant":
        n = case["rows"] * case["cols"]
        return {"bytes": 3 * n + n // 32, "flops": 2 * n}
    if kind == "linear":
        by, fl = _linear_work(case["rows"], case["k"], case["n"])
    elif kind == "mlp":
        by, fl = _mlp_work(case["rows"], case["dim"], case["inter"])
    elif kind == "moe":
        by, fl = _moe_work(case["rows"], case["dim"], case["inter"], case["experts"], case["local"], case["topk"],
                           case["shared"] * case["inter"])
    else:
        m, ranks = case["rows"], case["ranks"]
        parts = [_linear_work(m, 7168, 1536), _linear_work(m, 1536, 24576 // ranks), _linear_work(m, 7168, 576),
                 _linear_work(m, 16384 // ranks, 7168), _moe_work(m, 7168, 2048, 256, 256 // ranks, 8, 2048 // ranks)]
        by, fl = (case["layers"] * sum(p[i] for p in parts) for i in (0, 1))
    return {"bytes": by, "flops": fl}


def tolerance(case):
    """Quantising and de-quantising round every value in one given way.  A Linear accumulates in fp32 in any order and
    rounds to bf16; behind a second quantisation such a difference can move single FP8 codes."""
    if case["kind"] in ("weight_dequant", "act_quant"):
        return "exact"
    if case["kind"] == "linear":
        return {"rel": 1e-2, "max": 2e-2}
    return {"rel": 1e-2, "max": 5e-2}
