"""Performance cases of the FP8 block-scale mixture-of-experts operator and layer.

A case names one of the public entry points and the batch it gets:

* ``run``    -- ``op.run``: one 32-expert shard, token tensors on the GPU (a serving engine's call);
* ``host``   -- ``op.run_host``: the same with token tensors and result in pinned host memory;
* ``layer``  -- ``ExpertParallelMoE.forward``: the 256-expert layer, all eight shards on this GPU;
* ``layer_bf16`` -- ``ExpertParallelMoE.forward_bf16``: the layer for activations that are still bf16.

``routing`` says which tokens a batch holds: ``plain`` (logits ~ N(0, 1); half of the tokens have no expert on the
shard), ``dispatched`` (only tokens that selected the shard, what an expert-parallel dispatch hands to its owner) or
``skewed`` (bias + 4.0 on sixteen experts of the shard: every token sends all eight of its rows there).
"""
import torch

from __graft_entry__ import load_package

H, I, E_LOCAL, E_GLOBAL, BLOCK, N_SHARDS = 7168, 2048, 32, 256, 128, 8
RSF = 2.5                                                    # routed scaling factor
EXPERT_BYTES = 3 * I * H + 4 * 3 * (I // BLOCK) * (H // BLOCK)   # both weight matrices of an expert and their scales
ROW_FLOPS = 2 * 3 * I * H                                    # both GEMMs for one (token, expert) pair
LARGEST_T, LARGEST_SKEWED_T, LARGEST_HOST_T, LARGEST_LAYER_T = 14107, 1024, 256, 16384


def _case(name, entry, T, routing="plain", offset=0):
    return {"name": name, "entry": entry, "T": T, "routing": routing, "offset": offset}


def listed():
    return [
        # one sequence decoding: the latency floor of the operator (two or so experts' weights are read)
        _case("decode_t1", "run", 1, "dispatched"),
        # the same through host buffers, copies and the wait included: a caller without device-resident activations
        _case("host_t3", "host", 3, "dispatched"),
        # a handful of concurrent sequences
        _case("decode_t8", "run", 8),
        # the largest batch of the decode regime, every token with work on this shard, not the first shard
        _case("decode_t16", "run", 16, "dispatched", 224),
        # an odd batch just above it
        _case("ragged_t37", "run", 37, "plain", 64),
        # load imbalance: all rows of the batch on sixteen experts
        _case("skew_t64", "run", 64, "skewed"),
        # a large decode batch / a short prompt
        _case("mid_t512", "run", 512),
        # an odd size near the end of the middle regime
        _case("ragged_t901", "run", 901, "plain", 128),
        # a prefill chunk
        _case("prefill_t4096", "run", 4096),
        # a long odd prompt, the largest batch the operator's trace set has
        _case("prefill_t14107", "run", LARGEST_T, "plain", 32),
        # the whole layer for a decode batch, activations quantised on the way
        _case("layer_bf16_t256", "layer_bf16", 256),
        # the whole layer for a prefill batch of many sequences
        _case("layer_t16384", "layer", LARGEST_LAYER_T),
    ]


def _log_uniform(rng, lo, hi):
    return max(lo, min(hi, int(round(lo * (hi / lo) ** rng.random()))))


def draw(rng):
    kind = rng.choices(("plain", "dispatched", "skewed", "host", "layer", "layer_bf16"), (6, 4, 3, 2, 1, 1))[0]
    offset = E_LOCAL * rng.randrange(N_SHARDS)
    if kind == "host":
        case = _case("", "host", _log_uniform(rng, 1, LARGEST_HOST_T), "dispatched", offset)
    elif kind in ("layer", "layer_bf16"):
        case = _case("", kind, _log_uniform(rng, 16, LARGEST_LAYER_T))
    else:
        hi = {"plain": LARGEST_T, "dispatched": LARGEST_T // 2, "skewed": LARGEST_SKEWED_T}[kind]
        case = _case("", "run", _log_uniform(rng, 1, hi), kind, offset)
    del case["name"]
    return case


def _weights(gen, g, device):
    """One shard's weights, N(0, 0.02) quantised per 128 x 128 block."""
    w13 = torch.empty((E_LOCAL, 2 * I, H), dtype=torch.float8_e4m3fn, device=device)
    s13 = torch.empty((E_LOCAL, 2 * I // BLOCK, H // BLOCK), dtype=torch.float32, device=device)
    w2 = torch.empty((E_LOCAL, H, I), dtype=torch.float8_e4m3fn, device=device)
    s2 = torch.empty((E_LOCAL, H // BLOCK, I // BLOCK), dtype=torch.float32, device=device)
    for e in range(E_LOCAL):
        for w, s in ((w13, s13), (w2, s2)):
            w[e], s[e] = gen.quant_128x128(torch.randn(w.shape[1:], generator=g, device=device) * 0.02)
    return gen.ShardWeights(w13, s13, w2, s2)


def _experts(logits, bias):
    """The eight experts of every token: the best of the four routing groups with the largest sum of two best scores."""
    score = torch.sigmoid(logits) + bias.float()
    groups = score.view(-1, N_SHARDS, E_LOCAL)
    kept = groups.topk(2, dim=2).values.sum(2).topk(4, dim=1).indices
    open_ = torch.zeros(groups.shape[:2], dtype=torch.bool, device=logits.device).scatter_(1, kept, True)
    return groups.masked_fill(~open_.unsqueeze(2), -1.0).flatten(1).topk(8, dim=1).indices


def _router_inputs(case, g, device):
    """(logits, bias) of a batch."""
    T, first = case["T"], case["offset"]
    bias = torch.randn(E_GLOBAL, generator=g, device=device) * 0.1
    if case["routing"] == "skewed":
        bias[first:first + 16] += 4.0
    bias = bias.to(torch.bfloat16)
    logits = torch.randn((T, E_GLOBAL), generator=g, device=device)
    if case["routing"] == "dispatched":
        kept = logits[:0]
        while kept.shape[0] < T:
            kept = torch.cat([kept, logits[(_experts(logits, bias) // E_LOCAL == first // E_LOCAL).any(1)]])
            logits = torch.randn((T + 64, E_GLOBAL), generator=g, device=device)
        logits = kept[:T].contiguous()
    return logits, bias


def _tokens(gen, case, g, device):
    """(logits, bias, bf16 activations, e4m3 activations, their [56, T] scales)."""
    logits, bias = _router_inputs(case, g, device)
    hidden = torch.randn((case["T"], H), generator=g, device=device).to(torch.bfloat16)
    q, scale = gen.quant_1x128(hidden.float())
    return logits, bias, hidden, q, scale.t().contiguous()


def prepare(case, seed):
    pkg = load_package()
    device = torch.device("cuda", torch.cuda.current_device())
    g = torch.Generator(device=device)
    g.manual_seed(seed)
    entry = case["entry"]
    logits, bias, hidden, q, scale = _tokens(pkg.gen, case, g, device)
    if entry.startswith("layer"):
        weights = [_weights(pkg.gen, g, device) for _ in range(N_SHARDS)]
        layer = pkg.ep.ExpertParallelMoE(weights, transport="p2p")
        if entry == "layer_bf16":
            return {"call": layer.forward_bf16, "args": (logits, bias, hidden, RSF)}
        return {"call": layer.forward, "args": (logits, bias, q, scale, RSF)}
    w = _weights(pkg.gen, g, device)
    tokens = [logits, bias, q, scale]
    out = torch.empty((case["T"], H), dtype=torch.bfloat16, device=device)
    if entry == "host":
        # pinned memory of PyTorch's own caching host allocator; the operator gets it as plain addresses
        tokens = [t.cpu().pin_memory() for t in tokens]
        out = torch.empty((case["T"], H), dtype=torch.bfloat16, pin_memory=True)
    return {"call": pkg.op.run_host if entry == "host" else pkg.op.run,
            "args": (*tokens, w.gemm1_weights, w.gemm1_weights_scale, w.gemm2_weights, w.gemm2_weights_scale,
                     case["offset"], RSF, out)}


def run(state):
    return state["call"](*state["args"])


def work(case):
    """Weights of the experts that get a row, the token tensors and the result once.  How many experts, rows and tokens
    with work there are follows from the seed; these are the means over eight batches."""
    T, layer = case["T"], case["entry"].startswith("layer")
    active = rows = readers = 0.0
    for k in range(8):
        g = torch.Generator()
        g.manual_seed(k)
        e = _experts(*_router_inputs(case, g, "cpu"))
        here = torch.ones_like(e, dtype=torch.bool) if layer else e // E_LOCAL == case["offset"] // E_LOCAL
        active += e[here].unique().numel() / 8
        rows += int(here.sum()) / 8
        readers += int(here.any(1).sum()) / 8
    row_in = 2 * H if case["entry"] == "layer_bf16" else H + 4 * (H // BLOCK)
    return {"bytes": active * EXPERT_BYTES + T * (4 * E_GLOBAL + 2 * H) + readers * row_in, "flops": rows * ROW_FLOPS}


def tolerance(case):
    """bf16 results of fp32 sums.  The order of the sums moves some elements by one bf16 step (2^-8 to 2^-7 of the
    element), which is 1e-3 in the 2-norm even if every fourth element moves; a row of the layer is the rounded sum of
    up to eight rounded rows."""
    return {"rel": 2e-3, "max": 2e-2}
