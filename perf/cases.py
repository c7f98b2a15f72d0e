"""The work that a user of this package has it do, as cases that can be timed: one FP8 MoE layer pass per case,
through the public entry points (``MonoKernel.prefill`` / ``prefill_out`` and the allocation-free C entry).

A case names a compiled geometry (``variant``), the tokens of the batch, where the router linear runs
(``router``: the caller's logits, or ``inside`` the launch), whether the shared expert is computed in the same
launch, how uneven the routing is (``skew``: standard deviation of a per-expert logit offset) and the entry that
is called. An engine offers every batch up to 30720 tokens to the layer: single tokens and the short prompts of
a quiet server, the ragged chunks of chunked prefill, and full prefill batches of 8192 and 16384 tokens.
Values and distributions are those of ``unimonomoe_b200.synth``: weights N(0, 0.02) in block FP8, hidden states
N(0, 1) in bf16.
"""
import ctypes
import math

import torch

from unimonomoe_b200 import MonoKernel, synth, variant_path
from unimonomoe_b200.loader import prepare_router_weight, prepare_shared_expert

# variant -> (layer, columns of the intermediate held by this rank, experts held by this rank)
GEOMETRY = {
    "qwen_w1": (synth.QWEN, 512, 256),       # the whole Qwen-like layer on one GPU
    "qwen_sig_w1": (synth.QWEN, 512, 256),   # the same with the plain sigmoid + bias router
    "qwen_tp2": (synth.QWEN, 256, 256),      # one rank of a tensor-parallel group
    "qwen_tp4": (synth.QWEN, 128, 256),
    "qwen_ep2": (synth.QWEN, 512, 128),      # one rank of an expert-parallel group
    "qwen_ep4": (synth.QWEN, 512, 64),
    "qwen_ep8": (synth.QWEN, 512, 32),
    "ds_tp8": (synth.DEEPSEEK, 256, 256),    # one rank of the DeepSeek-V3-like layer
    "ds_tp4": (synth.DEEPSEEK, 512, 256),
    "ds_ep8": (synth.DEEPSEEK, 2048, 32),
}
ROUTER_MODE = {"qwen_sig_w1": 1}             # others: the layer's own
NOALLOC_TOKENS = 256                         # cap of the allocation-free entry at these widths (H = 2048)
MAX_TOKENS = 30720


def listed():
    return [
        # one sequence waiting for its next token: launches and latency are all there is
        case("one token", "qwen_w1", 1),
        # a short prompt on an engine that leaves the router linear to the launch
        case("short prompt, router inside", "qwen_w1", 61, router="inside"),
        # a batch of an engine whose KV pool already owns the GPU's memory
        case("no-alloc batch", "qwen_w1", 200, entry="noalloc"),
        # a ragged chunk of chunked prefill, with the uneven expert loads of real text
        case("ragged chunk, skewed", "qwen_w1", 1000, skew=1.0),
        # an ordinary prefill batch of the model as shipped: gated shared expert in the same launch
        case("prefill 4096, shared expert", "qwen_w1", 4096, shared=True),
        # the two batch sizes of the benchmark, logits handed over and router inside
        case("prefill 16384", "qwen_w1", 16384, entry="out"),
        case("prefill 8192, router inside", "qwen_w1", 8192, router="inside"),
        # ranks of multi-GPU groups: tensor parallel (narrow experts), expert parallel (ragged ownership)
        case("TP4 rank 8192", "qwen_tp4", 8192, entry="out"),
        case("EP4 rank 8192, skewed", "qwen_ep4", 8192, skew=0.5),
        # the DeepSeek-V3-like layer: a short ragged batch and a full one of a TP=8 rank, and an EP=8 rank that
        # takes its share of the (ungated) shared expert and scales the routed half
        case("DeepSeek TP8 rank 777", "ds_tp8", 777),
        case("DeepSeek TP8 rank 16384", "ds_tp8", 16384),
        case("DeepSeek EP8 rank 2048, shared", "ds_ep8", 2048, shared=True),
    ]


def case(name, variant, tokens, router="logits", shared=False, skew=0.0, entry="prefill"):
    c = {"variant": variant, "tokens": tokens, "router": router, "shared": shared, "skew": skew, "entry": entry}
    return dict(c, name=name) if name else c


def draw(rng):
    """Any geometry above, 1 to 30720 tokens, spread over the logarithm; never more work than the largest listed case."""
    variant = rng.choice(["qwen_w1"] * 4 + ["qwen_sig_w1", "qwen_tp2", "qwen_tp4", "qwen_ep2", "qwen_ep4", "qwen_ep8"]
                         + ["ds_tp8"] * 2 + ["ds_tp4", "ds_ep8"])
    most = MAX_TOKENS
    while flops_of(variant, most) > flops_of("ds_tp8", 16384) or most * GEOMETRY[variant][0].hidden > 16384 * 7168:
        most //= 2
    # an expert-parallel rank is given the tokens of every rank: at least two each
    least = 2 * (256 // GEOMETRY[variant][2]) if GEOMETRY[variant][2] < 256 else 1
    tokens = min(most, int(round(math.exp(rng.uniform(math.log(least), math.log(most))))))
    option = rng.choice(["plain", "plain", "router", "shared"])
    skew = rng.choice([0.0, 0.0, 0.5, 1.0])
    entry = rng.choice(["prefill", "prefill", "out"])
    if option == "plain" and variant.startswith("qwen") and tokens <= NOALLOC_TOKENS and rng.random() < 0.3:
        entry = "noalloc"
    return case(None, variant, tokens, router="inside" if option == "router" else "logits", shared=option == "shared",
                skew=0.0 if option == "router" else skew, entry=entry)


_loaded = {}


def kernel(variant):
    """One loaded binary per process, as a serving process keeps it for all of its layers."""
    if variant not in _loaded:
        _loaded[variant] = MonoKernel(variant_path(variant))
    return _loaded[variant]


def prepare(case, seed):
    spec, width, local = GEOMETRY[case["variant"]]
    T, dev = case["tokens"], torch.device("cuda", torch.cuda.current_device())
    mode = ROUTER_MODE.get(case["variant"], spec.router_mode)
    ranks = spec.experts // local
    rank = seed % ranks
    layer = synth.make_layer(spec, seed=seed % 100003, device=dev, inter_slice=(0, width) if width != spec.inter else None,
                             expert_slice=(rank * local, (rank + 1) * local) if ranks > 1 else None, with_shared=case["shared"])
    batch = synth.make_batch(spec, layer, T, seed=seed % 100003, device=dev, skew=case["skew"])
    mk = kernel(case["variant"])
    s = {"mk": mk, "entry": case["entry"], "layer": layer, "hs": batch["hs"], "logits": batch["logits"],
         "bias": layer["bias"] if mode == spec.router_mode else torch.zeros(spec.experts, device=dev),
         "emap": synth.expert_map(spec, rank, ranks, device=dev) if ranks > 1 else None,
         "rw": None, "shared": None, "part": (0, 1), "scale": 1.0, "out": None}
    if case["router"] == "inside":
        # the gate weight as checkpoints store it
        s["rw"], s["logits"] = prepare_router_weight(layer["router_w"].to(torch.bfloat16)), None
    if case["shared"]:
        sh = layer["shared"]
        a, b = slice(0, width), slice(0, width // 128)
        n, nb = spec.shared_inter, spec.shared_inter // 128
        s["shared"] = prepare_shared_expert(
            torch.cat([sh["w13"].view(torch.uint8)[:n][a], sh["w13"].view(torch.uint8)[n:][a]]),
            torch.cat([sh["w13_scale"][:nb][b], sh["w13_scale"][nb:][b]]),
            sh["w2"].view(torch.uint8)[:, a], sh["w2_scale"][:, b], sh["gate"])
        s["part"], s["scale"] = (rank, ranks), spec.routed_scaling
    if case["entry"] != "prefill":
        s["out"] = torch.empty(T, spec.hidden, dtype=torch.bfloat16, device=dev)
    if case["entry"] == "noalloc":
        mk.lib.launch_prefill_moe_noalloc.restype = ctypes.c_int
    return s


def run(s):
    mk, w = s["mk"], s["layer"]
    weights = (w["w13"], w["w13_scale"], w["w2"], w["w2_scale"])
    if s["entry"] == "noalloc":
        ptr = lambda t: ctypes.c_void_p(0 if t is None else t.data_ptr())  # noqa: E731
        rc = mk.lib.launch_prefill_moe_noalloc(
            ptr(s["logits"]), ctypes.c_int(s["hs"].size(0)), ptr(s["hs"]), *map(ptr, weights), ptr(s["out"]), ptr(s["bias"]),
            ptr(s["emap"]), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
        if rc != 0:
            raise RuntimeError(f"launch_prefill_moe_noalloc: {rc}")
        return s["out"]
    if s["entry"] == "out":
        mk.prefill_out(s["hs"], s["logits"], *weights, s["out"], 8, True, s["bias"], expert_map=s["emap"],
                       router_weight=s["rw"], shared=s["shared"], shared_part=s["part"], tp_out_scale=s["scale"])
        return s["out"]
    return mk.prefill(s["hs"], s["logits"], *weights, 8, True, s["bias"], expert_map=s["emap"], router_weight=s["rw"],
                      shared=s["shared"], shared_part=s["part"], out_scale=s["scale"])


def flops_of(variant, tokens):
    spec, width, local = GEOMETRY[variant]
    return 6.0 * spec.hidden * width * tokens * spec.top_k * local / spec.experts


def work(case):
    """Weights of the experts that the batch is expected to reach, each once; activations, logits (or the gate
    weight) and scales in, output out. Operations: the routed rows' products, the router linear and the shared
    expert where the launch computes them."""
    spec, width, local = GEOMETRY[case["variant"]]
    T, H, E = case["tokens"], spec.hidden, spec.experts
    per_expert = 3 * H * width * (1 + 4 / 128 / 128)
    reached = local * (1.0 - (1.0 - spec.top_k / E) ** T)
    nbytes = reached * per_expert + 2 * T * H * 2
    flops = flops_of(case["variant"], T)
    if case["router"] == "inside":
        nbytes += 2 * E * H
        flops += 2.0 * T * H * E
    else:
        nbytes += 4 * T * E
    if case["shared"]:
        nbytes += per_expert
        flops += 6.0 * H * width * T * local / E
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    """bf16 outputs of an FP8 path: a partial row and the sum are each rounded to bf16 (2^-9 relative), and an e4m3
    code of the intermediate that sits on a rounding boundary may fall either way. With the router linear inside,
    fp32 logits summed in another order may also exchange two experts of nearly equal score in a few tokens,
    whose rows then differ by the share of one expert of eight."""
    if case["router"] == "inside":
        return {"rel": 5e-3, "max": 0.9}
    return {"rel": 4e-3, "max": 4e-2}


EXACT_FLOPS = 2.2e11                         # beyond this the 64-bit computation takes too long


def exact(case, seed):
    """The layer in 64 bits with the quantisation points that the FP8 path has by definition (activations and
    intermediate to e4m3 per 128 columns); nothing else is rounded."""
    if work(case)["flops"] > EXACT_FLOPS:
        return None
    spec, width, local = GEOMETRY[case["variant"]]
    s = prepare(case, seed)
    mode = ROUTER_MODE.get(case["variant"], spec.router_mode)
    hs, layer = s["hs"].double(), s["layer"]
    logits = s["logits"].double() if s["rw"] is None else hs @ s["rw"].double().t()
    ids, weights = _route(logits, mode, s["bias"], spec)
    x = _through_e4m3(hs)
    owner = s["emap"].long() if s["emap"] is not None else torch.arange(spec.experts, device=hs.device)
    ids = owner[ids]
    out = torch.zeros_like(hs)
    for e in torch.unique(ids).tolist():
        if e >= 0:
            tok, slot = (ids == e).nonzero(as_tuple=True)
            y = _expert(x[tok], layer["w13"][e], layer["w13_scale"][e], layer["w2"][e], layer["w2_scale"][e])
            out.index_add_(0, tok, y * weights[tok, slot, None])
    out *= s["scale"] if s["shared"] is not None else 1.0
    if s["shared"] is not None:
        sh, (part, parts) = s["shared"], s["part"]
        tok = (torch.arange(len(hs), device=hs.device) // 128 % parts == part).nonzero(as_tuple=True)[0]
        y = _expert(x[tok], sh["w13"], sh["w13_scale"], sh["w2"], sh["w2_scale"])
        if sh.get("gate") is not None:
            y *= torch.sigmoid(hs[tok] @ sh["gate"].double())[:, None]
        out.index_add_(0, tok, y)
    return out


def _route(logits, mode, bias, spec):
    if mode == 0:
        score = sel = torch.softmax(logits, dim=-1)
    else:
        score = torch.sigmoid(logits)
        sel = score + bias.double()
    if mode == 2:
        groups = sel.unflatten(1, (spec.n_group, -1))
        best = groups.topk(2, dim=-1).values.sum(-1).topk(spec.topk_group, dim=-1).indices
        keep = torch.zeros(groups.shape[:2], dtype=torch.bool, device=sel.device).scatter_(1, best, True)
        sel = groups.masked_fill(~keep[..., None], -math.inf).flatten(1)
    ids = sel.topk(spec.top_k, dim=-1).indices
    w = score.gather(1, ids)
    return ids, w / w.sum(-1, keepdim=True)


def _through_e4m3(x):
    g = x.unflatten(-1, (-1, 128))
    amax = g.abs().amax(-1, keepdim=True)
    amax = torch.where(amax > 0, amax, 1.0)
    return ((g * (448.0 / amax)).float().to(torch.float8_e4m3fn).double() * (amax / 448.0)).flatten(-2)


def _weight(w, scale):
    w = w.view(torch.float8_e4m3fn).double().unflatten(0, (-1, 128)).unflatten(2, (-1, 128))
    return (w * scale.double()[:, None, :, None]).flatten(2).flatten(0, 1)


def _expert(x, w13, s13, w2, s2):
    gate, up = (x @ _weight(w13, s13).t()).chunk(2, dim=-1)
    return _through_e4m3(torch.nn.functional.silu(gate) * up) @ _weight(w2, s2).t()
