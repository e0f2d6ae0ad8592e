"""The work that a user of this backend has it do: calls of the MegaMoE layer, as a serving engine makes them, and the
preparation of its weights.

A layer case is one pass of a layer on one GPU: the hidden states and the routing of ``tokens`` tokens are staged into the
workspace (with the router's top-k in front where the engine leaves that to the backend), then the layer call writes
``y`` and adds to the per-expert receive counts.  ``experts`` is the number of experts resident on the GPU: 384 is the
target model on one GPU, 192 / 96 / 48 its share at 2 / 4 / 8 GPUs with every routed token that such a GPU receives, 128
and 16 the draft model whole and at 8 GPUs.  A load case turns expert weights from checkpoint order into the two-slice
form that the kernels read, which happens at start-up and at each reload.
"""

import math

import torch

from vllm_plugin_b200 import api, testing
from vllm_plugin_b200.backend.weights import sf_to_required_layout
from vllm_plugin_b200.backend.workspace import SingleRankGroup

HIDDEN, INTER = 5120, 2304      # both models
MAX_TOKENS = 3840               # most tokens of one call: a capacity of 2 x 1920
CLAMP = 10.0                    # both models' SwiGLU clamp


def _layer(name, tokens, experts, topk=6, **other):
    case = {
        "name": name, "kind": "layer", "tokens": tokens, "experts": experts, "topk": topk,
        "graph": False,         # replayed from a CUDA graph, as engines run decode; else called eagerly
        "router": False,        # the backend chooses the experts from the gate logits
        "skewed": False,        # Zipf(1.2) popularity, two hot experts, 5 % of the routes masked; else Gaussian gates
        "two_slice": True,      # routed weights as the engine's layer keeps them; else one plain tensor per matrix
        "residual": False,      # the residual stream is added in the call
        "fast_math": True,
    }
    case.update(other)
    return case


def listed():
    return [
        # one sequence being generated, the smallest call there is: latency
        _layer("decode-1-graph", 1, 384, graph=True),
        # the draft model proposing for a batch of sequences
        _layer("draft-decode-32-graph", 32, 128, topk=3, graph=True),
        # an engine run without graphs, a few sequences: host work and launches count
        _layer("decode-7-eager", 7, 384),
        # a decode batch: over 60 % of all experts are read, for one or two tokens each
        _layer("decode-64-graph", 64, 384, graph=True),
        # the benchmark's plumbing configuration, plain weight tensors
        _layer("config0-128", 128, 32, two_slice=False),
        # a large decode batch through the router, residual added in the call
        _layer("batch-256-router", 256, 384, router=True, residual=True),
        # a mixed prefill and decode step of no round size, with skewed routing
        _layer("mixed-1021-skewed", 1021, 384, skewed=True),
        # full prefill steps: the whole model on one GPU, and the shares of a GPU at 4 and 8 GPUs
        _layer("prefill-3840", 3840, 384),
        _layer("prefill-3001-share4-skewed", 3001, 96, skewed=True),
        _layer("prefill-3840-share8", 3840, 48),
        # the draft model's prefill share at 8 GPUs, most batched tokens
        _layer("draft-prefill-2560", 2560, 16, topk=3),
        # loading, and reloading after a rebalance, the experts of one of 8 GPUs
        {"name": "load-48", "kind": "load", "experts": 48},
    ]


def draw(rng):
    if rng.random() < 0.08:
        return {"kind": "load", "experts": rng.randint(8, 60)}
    draft = rng.random() < 0.25
    experts = rng.choice((16, 32, 64, 128, 132)) if draft else rng.choice((32, 48, 49, 96, 97, 192, 384, 392))
    tokens = min(MAX_TOKENS, int(math.exp(rng.uniform(0.0, math.log(MAX_TOKENS + 1)))))
    case = _layer("", tokens, experts, topk=3 if draft else 6, graph=tokens <= 256 and rng.random() < 0.5,
                  router=rng.random() < 0.2, two_slice=rng.random() < 0.8, residual=rng.random() < 0.25,
                  fast_math=rng.random() < 0.9)
    case["skewed"] = not case["router"] and rng.random() < 0.35
    del case["name"]
    return case


def _routing(case, seed, device):
    skew = {"zipf_s": 1.2, "mask_frac": 0.05, "hot": 2} if case["skewed"] else {}
    return testing.make_routing(case["tokens"], case["experts"], case["topk"], seed, device, **skew)


def _checkpoint_weights(experts, gen, seed, device):
    """``experts`` routed experts in checkpoint order: every row is one of the quantised N(0, 0.02) rows of four experts,
    drawn for each place anew (quantising 384 experts one by one takes minutes, and the kernels do not care)."""
    pool = [testing.routed_expert_raw(HIDDEN, INTER, seed, index, device) for index in range(4)]
    mats = [torch.cat([p[i] for p in pool]) for i in range(4)]
    out = []
    for w, sf in ((mats[0], mats[1]), (mats[2], mats[3])):
        rows = w.shape[0] // 4
        pick = torch.randint(w.shape[0], (experts * rows,), generator=gen, device=device)
        for m in (w, sf):
            wide = m.contiguous().view(torch.int64).index_select(0, pick)
            out.append(wide.view(m.dtype).view(experts, rows, m.shape[1]))
    w13, s13, w2, s2 = out
    return ((w13, sf_to_required_layout(s13, 2 * INTER, HIDDEN, experts)),
            (w2, sf_to_required_layout(s2, HIDDEN, INTER, experts)))


def prepare(case, seed):
    device = torch.device("cuda", torch.cuda.current_device())
    gen = torch.Generator(device=device).manual_seed(seed)
    l1, l2 = _checkpoint_weights(case["experts"], gen, seed, device)
    if case["kind"] == "load":
        return {"kind": "load", "l1": l1, "l2": l2}
    l1, l2 = api.transform_weights_for_mega_moe(l1, l2)
    if case["two_slice"]:
        l1, l2 = api.localize_mega_moe_weights(l1, l2)
    q13, e13, q2, e2 = testing.shared_expert_raw(HIDDEN, INTER, seed, device)
    shared_l1, shared_l2 = api.transform_weights_for_mega_moe(
        (q13, sf_to_required_layout(e13, 2 * INTER, HIDDEN)), (q2, sf_to_required_layout(e2, HIDDEN, INTER)))

    tokens, experts, topk = case["tokens"], case["experts"], case["topk"]
    buf = api.get_symm_buffer_for_mega_moe(SingleRankGroup(), experts, MAX_TOKENS, topk, HIDDEN, INTER, 1)
    api.precompile_mega_moe_variants(1, experts, MAX_TOKENS, topk, HIDDEN, INTER, 1, activation_clamp=CLAMP)

    def gaussian(*shape, dtype=torch.bfloat16):
        return torch.randn(shape, generator=gen, device=device).to(dtype)

    state = {
        "kind": "layer", "buf": buf, "l1": l1, "l2": l2, "shared_l1": shared_l1, "shared_l2": shared_l2,
        "fast_math": case["fast_math"], "hidden": gaussian(tokens, HIDDEN),
        "logits": gaussian(tokens, experts, dtype=torch.float32) if case["router"] else None,
        "residual": gaussian(tokens, HIDDEN) if case["residual"] else None,
        "y": torch.empty((tokens, HIDDEN), dtype=torch.bfloat16, device=device),
        "stats": torch.zeros(experts, dtype=torch.int32, device=device), "graph": None,
    }
    if not case["router"]:
        state["ids"], state["weights"] = _routing(case, seed, device)
    if case["graph"]:
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            _call(state)
        torch.cuda.current_stream().wait_stream(side)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            _call(state)
        state["graph"] = graph
        state["stats"].zero_()
    return state


def _call(state):
    if state["logits"] is not None:
        api.route_and_stage_inputs_for_mega_moe(state["buf"], state["hidden"], state["logits"])
    else:
        api.stage_inputs_for_mega_moe(state["buf"], state["hidden"], state["ids"], state["weights"])
    api.fp8_fp4_mega_moe(state["y"], state["l1"], state["l2"], state["buf"], state["shared_l1"], state["shared_l2"],
                         cumulative_local_expert_recv_stats=state["stats"], activation_clamp=CLAMP,
                         fast_math=state["fast_math"], residual=state["residual"])


def run(state):
    if state["kind"] == "load":
        l1, l2 = api.transform_weights_for_mega_moe(state["l1"], state["l2"])
        return api.localize_mega_moe_weights(l1, l2)
    if state["graph"] is not None:
        state["graph"].replay()
    else:
        _call(state)
    return {"y": state["y"], "stats": state["stats"]}


def work(case):
    if case["kind"] == "load":
        # every weight and scale byte in once and out once
        return {"bytes": 2 * case["experts"] * (3 * HIDDEN * INTER // 2 + 3 * HIDDEN * INTER // 32), "flops": 0}
    ids, _ = _routing(case, 0, "cpu")
    hit = ids[ids >= 0]
    flops, nbytes = testing.layer_work(hit.numel(), case["tokens"], hit.unique().numel(), HIDDEN, INTER, True)
    nbytes += case["tokens"] * (case["experts"] * 4 if case["router"] else case["topk"] * 12)
    nbytes += case["tokens"] * HIDDEN * 2 if case["residual"] else 0
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    """Weights move bit for bit and receive counts are whole numbers.  ``y`` is BF16, summed in FP32 in whatever order, with
    activations rounded to E4M3 halfway, where another order of summation turns single roundings: 1e-3 over all of ``y``,
    and a BF16 step or a turned rounding at a single value."""
    if case["kind"] == "load":
        return "exact"
    return {"rel": 1e-3, "max": 0.05}
