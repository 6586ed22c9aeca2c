"""The work that users of this framework have it do, as cases that can be timed.

Two kinds of pass, both through the public entry points and both over a few layers with weights of
their own, as a model runs them (one layer's experts are 428 MB, so a pass finds its weights in HBM
and not in L2; with one token it reads 27 MB a layer, so eight layers are needed for that):

  moe  per layer: router (projection and top-8 in one call, in bf16 or from E4M3 rows, or top-8 of
       logits that the caller projected), then Nvfp4ExpertRunner.launch_batch: what a host that has
       its own attention and dense parts calls
  ffn  FeedForwardLayer.forward of a stack: pre-norms, router, experts (unreduced), the dense FP8
       GeGLU MLP on a second stream, fused finalize; each layer's output is the next one's input

A case with "graph" replays the pass as one CUDA graph, the way a decode loop runs; without it the
calls are made one by one from Python.  Token counts run from one (a single decoding stream) over
decode batches, speculative-verification and chunked-prefill sizes to 16384-token prefills.
"""
import functools

import numpy as np
import torch

import gevva_b200
from gevva_b200.feedforward import pack_fp8
from gevva_b200.runtime import EXPERTS, HIDDEN, TOP_K, Nvfp4ExpertRunner
from gevva_b200.synthetic import SyntheticLayer, SyntheticStack

DEVICE = "cuda:0"
CAPACITY = 4096                    # tokens a runner is made for, unless the batch is larger
EXPERT_BYTES = 3345408             # codes and block scales of one expert's three matrices
DENSE_BYTES = 2112 * 2816 * 3      # E4M3 gate, up and down of the dense MLP
EXPERT_FLOPS_PER_TOKEN = TOP_K * 3 * 2 * 704 * HIDDEN
DENSE_FLOPS_PER_TOKEN = 3 * 2 * 2112 * HIDDEN
ROUTER_FLOPS_PER_TOKEN = 2 * EXPERTS * HIDDEN


def _case(kind, tokens, layers, router="bf16", skew="none", graph=False, name=None):
    case = {"kind": kind, "tokens": tokens, "layers": layers, "router": router, "skew": skew, "graph": graph}
    return dict(case, name=name) if name else case


def listed():
    return [
        # one user's chat reply, token by token: latency of a chain of short kernels
        _case("moe", 1, 8, graph=True, name="decode_1_graph"),
        # a handful of parallel replies from a Python loop without graphs: launches and host work
        _case("moe", 5, 8, name="decode_5_eager"),
        # a busy decode batch behind the FP8 sidecar's router
        _case("moe", 37, 8, router="fp8", graph=True, name="decode_37_fp8_router_graph"),
        # the full decode batch: the experts' weights stream once
        _case("moe", 64, 8, graph=True, name="decode_64_graph"),
        # drafts of several sequences verified together, or a small prefill chunk: all weights, few rows each
        _case("moe", 200, 4, name="verify_200_eager"),
        # one short prompt of odd length whose host projects the router logits itself
        _case("moe", 613, 2, router="logits", name="prompt_613_logits_eager"),
        # a prefill batch of about ten prompts, experts unevenly loaded
        _case("moe", 4096, 1, skew="normal", name="prefill_4096_eager"),
        # the largest prefill, with a few experts that take much of it
        _case("moe", 16384, 1, skew="zipf", name="prefill_16384_zipf_eager"),
        # decoding through whole feed-forward layers, captured as the serving loop captures them
        _case("ffn", 40, 4, graph=True, name="ffn_decode_40_graph"),
        # the same for one stream, called from Python
        _case("ffn", 1, 4, name="ffn_decode_1_eager"),
        # a short prompt through whole layers
        _case("ffn", 301, 3, name="ffn_prompt_301_eager"),
        # the prefill of the feed-forward stack
        _case("ffn", 2048, 2, name="ffn_prefill_2048_eager"),
    ]


def _log_size(rng, low, high):
    return min(high, max(low, int(round(low * (high / low) ** rng.random()))))


def draw(rng):
    """One more case: sizes over their whole range by logarithm, options as they occur at that size."""
    kind = rng.choice(("moe", "moe", "ffn"))
    if kind == "ffn":
        tokens = _log_size(rng, 1, 4096)
        layers = 4 if tokens <= 128 else 3 if tokens <= 512 else 2 if tokens <= 2048 else 1
        return _case("ffn", tokens, layers, graph=rng.random() < (0.6 if tokens <= 256 else 0.2))
    tokens = _log_size(rng, 1, 16384)
    layers = 8 if tokens <= 64 else 6 if tokens <= 128 else 4 if tokens <= 512 else 2 if tokens <= 2048 else 1
    return _case("moe", tokens, layers, router=rng.choice(("bf16", "bf16", "fp8", "logits")),
                 skew=rng.choice(("none", "normal", "zipf")), graph=rng.random() < (0.6 if tokens <= 256 else 0.2))


def _router_operands(layer, x, router):
    """What the router call of one layer takes, by the kind of router."""
    if router == "logits":
        return {"logits": layer.logits(x)}
    if router == "fp8":
        # per-row dynamic scales and a per-tensor weight scale, as the FP8 sidecar has them
        scale = x.float().abs().amax(dim=1) / 448.0
        rows = (x.float() / scale[:, None]).to(torch.float8_e4m3fn).view(torch.uint8)
        weight, weight_scale = pack_fp8(layer.router_w.float())
        return {"x": rows, "w": weight, "activation_scales": scale,
                "weight_scale": torch.tensor([weight_scale], device=x.device)}
    return {"x": x, "w": layer.router_w}


def _captured(state):
    """The pass as one CUDA graph; its outputs stay where the capture put them."""
    _pass(state)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = _pass(state)
    state.update(graph=graph, out=out)
    return state


def prepare(case, seed):
    tokens, layers = case["tokens"], case["layers"]
    generator = torch.Generator(device=DEVICE)
    generator.manual_seed(seed)
    if case["kind"] == "ffn":
        stack = SyntheticStack(layers, max(tokens, CAPACITY), DEVICE, seed=1000 * seed)
        hidden = torch.randn((tokens, HIDDEN), generator=generator, device=DEVICE).to(torch.bfloat16)
        state = {"kind": "ffn", "stack": stack, "hidden": hidden}
        return _captured(state) if case["graph"] else state
    steps, first = [], None
    for index in range(layers):
        layer = SyntheticLayer(1000 * seed + index, max(tokens, CAPACITY), DEVICE, zipf=case["skew"] == "zipf",
                               bias_std=0.5 if case["skew"] == "normal" else 0.0,
                               shared_scratch=first)
        if first is None:
            scales = layer.calibrate(layer.inputs(256, seed))
            first = layer.runner
        else:
            layer.set_scales(*scales)
        x = torch.randn((tokens, HIDDEN), generator=generator, device=DEVICE).to(torch.bfloat16)
        steps.append({"layer": layer, "runner": layer.runner, "input": x, "router": case["router"],
                      "operands": _router_operands(layer, x, case["router"]),
                      "weights": torch.empty((tokens, TOP_K), dtype=torch.float32, device=DEVICE),
                      "ids": torch.empty((tokens, TOP_K), dtype=torch.int32, device=DEVICE),
                      "output": torch.empty_like(x)})
    state = {"kind": "moe", "steps": steps, "tokens": tokens}
    return _captured(state) if case["graph"] else state


def _route(step):
    layer, operands = step["layer"], step["operands"]
    if step["router"] == "logits":
        gevva_b200.route_128_top8(operands["logits"], layer.expert_scale, weights=step["weights"], ids=step["ids"])
    elif step["router"] == "fp8":
        gevva_b200.route_project(operands["x"], operands["w"], layer.expert_scale, status_of=step["runner"],
                                 activation_scales=operands["activation_scales"],
                                 weight_scale=operands["weight_scale"], weights=step["weights"], ids=step["ids"])
    else:
        gevva_b200.route_project(operands["x"], operands["w"], layer.expert_scale, bias=layer.bias,
                                 status_of=step["runner"], weights=step["weights"], ids=step["ids"])


def _pass(state):
    if state["kind"] == "ffn":
        return [state["stack"].forward(state["hidden"])]
    for step in state["steps"]:
        _route(step)
        step["runner"].launch_batch(step["input"], step["ids"], step["weights"], step["output"], state["tokens"])
    return [[step["output"], step["ids"], step["weights"]] for step in state["steps"]]


def run(state):
    if "graph" in state:
        state["graph"].replay()
        return state["out"]
    return _pass(state)


@functools.lru_cache(maxsize=None)
def _inclusion(skew):
    """How often a token's eight experts include each expert, for the router that prepare() makes."""
    rng = np.random.RandomState(0)
    bias = np.zeros(EXPERTS)
    if skew == "normal":
        bias = rng.randn(EXPERTS) * 0.5
    elif skew == "zipf":
        bias = -1.1 * np.log(np.arange(1, EXPERTS + 1))
    logits = rng.randn(8192, EXPERTS) * (0.02 * HIDDEN ** 0.5) + bias
    return np.bincount(np.argsort(-logits, axis=1)[:, :TOP_K].ravel(), minlength=EXPERTS) / 8192.0


def work(case):
    """Weights of the experts that the batch is expected to reach, the other weights, and the batch
    in and out, each once; the operations of the projections."""
    tokens, layers = case["tokens"], case["layers"]
    experts = float((1.0 - (1.0 - _inclusion(case["skew"])) ** tokens).sum())
    row = 2 * HIDDEN
    flops = tokens * EXPERT_FLOPS_PER_TOKEN
    if case["kind"] == "ffn":
        # hidden state in and out; the steps between are the layer's own affair
        moved = experts * EXPERT_BYTES + DENSE_BYTES + EXPERTS * row + tokens * 2 * row
        return {"bytes": layers * moved, "flops": layers * (flops + tokens * (DENSE_FLOPS_PER_TOKEN + ROUTER_FLOPS_PER_TOKEN))}
    moved = experts * EXPERT_BYTES + tokens * (2 * row + TOP_K * 8)
    if case["router"] == "logits":
        moved += tokens * EXPERTS * 2
    else:
        flops += tokens * ROUTER_FLOPS_PER_TOKEN
        moved += EXPERTS * row if case["router"] == "bf16" else EXPERTS * HIDDEN + tokens * (HIDDEN + 4)
    return {"bytes": layers * moved, "flops": layers * flops}


def tolerance(case):
    """Outputs are bf16 (2^-9 each) behind FP4 codes that are decided exactly.  Router logits are fp32
    sums rounded to bf16: in another order of summation about one in a hundred moves by one step, and
    where the eighth and the ninth logit are that close the last expert of that token changes (a few of
    ten thousand ids), which moves its row by the weight of one expert, up to the size of a value."""
    return {"rel": 1e-2, "max": 0.9, "differ": 0.002}
