"""The work a user of the layer has it do, as measurable cases: what each holds in hand before the call, one pass through
the public entry points, the work the pass cannot do without, and how far two correct results may lie apart.

Four ways into the library are taken, each as a serving program takes it:

  graph    ``FusedMoEMxfp4.capture`` once, then one graph replay per decode step (router, alignment, experts)
  forward  ``FusedMoEMxfp4.forward`` called eagerly, from activations or from given router logits
  apply    ``B200FusedExperts.apply`` - a serving engine's experts object; the engine has routed already
  op       ``torch_ops.fused_moe_mxfp4`` - the plain function, routing given

Shapes are those of the benchmark configurations (``vkernels_b200.synthetic.CONFIGS``), of the routing shape with
sixteen experts a token, and, in ``draw``, generic multiples of 64 between them. Every case has expert weights of its own,
larger than the L2 together with the other states a measurement rotates through.
"""
import math

import torch

from vkernels_b200 import synthetic as syn
from vkernels_b200 import torch_ops as ops
from vkernels_b200.experts import layer_from_config
from vkernels_b200.vllm_experts import B200FusedExperts, convert_weights_for_b200

DEVICE = "cuda:0"

# Model shapes: hidden, ispp, experts, top_k, routing, shared experts, clamp of the activation's inputs.
SHAPES = {
    "e32": dict(hidden=2880, ispp=2880, experts=32, top_k=4, routing="softmax", shared=0, limit=7.0),
    "e128": dict(hidden=2880, ispp=2880, experts=128, top_k=4, routing="softmax", shared=0, limit=0.0),
    "e256s": dict(hidden=7168, ispp=2048, experts=256, top_k=8, routing="sigmoid_group", shared=1, limit=0.0),
    "e256k16": dict(hidden=7168, ispp=512, experts=256, top_k=16, routing="softmax", shared=0, limit=0.0),
}
OPTIONS = dict(prepack=False, bias=False, situ=False, zipf=0.0)


def _case(entry, tokens, shape, **options):
    return dict(entry=entry, tokens=tokens, **SHAPES[shape], **dict(OPTIONS, **options))


def listed():
    named = {
        # one user's decode step: a handful of routed slots, latency and launches are what counts
        "step_1": _case("graph", 1, "e32"),
        # small decode batches from weights that the server rewrote at load time
        "step_8_packed": _case("graph", 8, "e32", prepack=True),
        "step_64_packed": _case("graph", 64, "e32", prepack=True),
        # the same model served from the checkpoint's own layout (no second copy of the weights)
        "step_128": _case("graph", 128, "e32"),
        # decode of a wide model: group-limited sigmoid router, always-on shared expert, most experts touched
        "step_32_wide": _case("graph", 32, "e256s", prepack=True),
        # eager decode with an odd number of running sequences: the host path counts too
        "eager_37": _case("forward", 37, "e32"),
        # a serving engine's experts call, sixteen experts a token, the other activation
        "apply_48": _case("apply", 48, "e256k16", situ=True),
        # decode tokens and a prompt's tail in one batch: ten tokens an expert
        "mixed_333": _case("forward", 333, "e128"),
        # one chunk of a chunked prefill through the plain function, with the model's biases
        "op_2047": _case("op", 2047, "e128", bias=True),
        # the headline prefill batch
        "prefill_8192": _case("forward", 8192, "e128"),
        # skewed routing: some experts hold a large part of the batch, many a handful of tokens
        "zipf_4096": _case("forward", 4096, "e128", zipf=1.2),
        # the largest batch: long prompts of the wide model
        "prefill_16384_wide": _case("forward", 16384, "e256s"),
    }
    return [dict(case, name=name) for name, case in named.items()]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """Decode batches of 1..256 tokens (replayed or eager, either weight form), batches of up to 16384 (eager), on the listed
    shapes or on a generic one; the biases, the activation and the skew as a model may have them."""
    if rng.random() < 0.5:
        shape = dict(SHAPES[rng.choice(sorted(SHAPES))])
    else:   # generic: any multiple of 64 in either dimension, power-of-two expert counts
        hidden, ispp = 64 * _log_int(rng, 8, 112), 64 * _log_int(rng, 4, 45)
        experts = 2 ** rng.randint(3, 8)
        while experts * hidden * ispp > 256 * 7168 * 2048:   # no more weight bytes than the widest listed model
            experts //= 2
        shape = dict(hidden=hidden, ispp=ispp, experts=experts, top_k=rng.choice([2, 4, 6, 8]), routing="softmax", shared=0,
                     limit=rng.choice([0.0, 7.0]))
    if rng.random() < 0.5:
        entry, tokens = rng.choice(["graph", "graph", "forward", "apply"]), _log_int(rng, 1, 256)
    else:
        entry, tokens = rng.choice(["forward", "op", "apply"]), _log_int(rng, 257, 16384)
    options = dict(OPTIONS)
    routed_inside = entry in ("graph", "forward")
    if routed_inside and tokens <= 256:
        options["prepack"] = rng.random() < 0.5
    if not routed_inside:
        shape.update(routing="softmax", shared=0)
        options["bias"], options["situ"] = rng.random() < 0.5, rng.random() < 0.25
    if entry == "forward" and shape["routing"] == "softmax" and rng.random() < 0.25:
        options["zipf"] = 1.2
    return dict(entry=entry, tokens=tokens, **shape, **options)


def _config(case):
    return syn.MoEConfig("case", 0, H=case["hidden"], I=case["ispp"], E=case["experts"], top_k=case["top_k"], T=(case["tokens"],),
                         routing=case["routing"], scaling=2.5 if case["routing"] == "sigmoid_group" else 1.0,
                         n_group=8 if case["routing"] == "sigmoid_group" else 1,
                         topk_group=4 if case["routing"] == "sigmoid_group" else 1, swiglu_limit=case["limit"],
                         shared_experts=case["shared"], zipf_alpha=case["zipf"] or None)


def prepare(case, seed):
    cfg, T = _config(case), case["tokens"]
    seed &= 0x3FFFFFFF
    w = syn.make_expert_weights(cfg, seed=seed, backend="torch", device=DEVICE)
    x = syn.make_activations(cfg, T, seed=seed, backend="torch", device=DEVICE)
    g = torch.Generator(device=DEVICE)
    g.manual_seed(seed * 7919 + 3)
    state = {"entry": case["entry"], "x": x}
    if case["entry"] in ("graph", "forward"):
        wr = 0.02 * torch.randn((cfg.E, cfg.H), generator=g, device=DEVICE)
        bias = 0.01 * torch.randn(cfg.E, generator=g, device=DEVICE) if cfg.routing == "sigmoid_group" else None
        layer = layer_from_config(cfg, w, {"wr": wr, "bias": bias}, max_tokens=T, prepack=case["prepack"])
        state["layer"] = layer
        state["logits"] = syn.make_zipf_logits(cfg, T, seed=seed, device=DEVICE) if cfg.zipf_alpha else None
        if case["entry"] == "graph":
            state["graph"], state["y"] = layer.capture(x)
        return state
    # routing given: softmax over random logits, the largest top_k renormalised
    score, ids = torch.softmax(1.07 * torch.randn((T, cfg.E), generator=g, device=DEVICE), dim=1).topk(cfg.top_k, dim=1)
    state["ids"], state["weights"] = ids.to(torch.int32), (score / score.sum(1, keepdim=True)).float()
    b13 = b2 = None
    if case["bias"]:
        b13 = 0.1 * torch.randn((cfg.E, 2 * cfg.I), generator=g, device=DEVICE)
        b2 = 0.1 * torch.randn((cfg.E, cfg.H), generator=g, device=DEVICE)
    w13, w2, s13, s2, b13, b2 = convert_weights_for_b200(w["w13"], w["w2"], w["w13_scale"], w["w2_scale"], w13_bias=b13, w2_bias=b2)
    state.update(w13=w13, w2=w2, s13=s13, s2=s2, b13=b13, b2=b2, limit=cfg.swiglu_limit, situ=case["situ"])
    if case["entry"] == "apply":
        experts = B200FusedExperts(w13_scale=s13, w2_scale=s2, w13_bias=b13, w2_bias=b2, swiglu_limit=cfg.swiglu_limit, max_num_tokens=T)
        shape13, _, shape_y = experts.workspace_shapes(T, 2 * cfg.I, cfg.H, cfg.top_k, cfg.E, cfg.E)
        state.update(experts=experts, workspace13=torch.empty(shape13, dtype=torch.bfloat16, device=DEVICE),
                     y=torch.empty(shape_y, dtype=torch.bfloat16, device=DEVICE))
    return state


def run(s):
    if s["entry"] == "graph":
        s["graph"].replay()
        return s["y"]
    if s["entry"] == "forward":
        return s["layer"].forward(s["x"], logits=s["logits"])
    if s["entry"] == "apply":
        s["experts"].apply(s["y"], s["x"], s["w13"], s["w2"], s["weights"], s["ids"], activation="situ" if s["situ"] else "silu",
                           workspace13=s["workspace13"])
        return s["y"]
    return ops.fused_moe_mxfp4(s["x"], s["w13"], s["s13"], s["w2"], s["s2"], s["ids"], s["weights"], swiglu_limit=s["limit"],
                               activation=ops.moe_fused_mxfp4.SITU if s["situ"] else ops.moe_fused_mxfp4.SWIGLU, b13=s["b13"],
                               b2=s["b2"])


def _dense(codes, scale):
    """[rows, K / 2] packed codes and [rows, K / 32] exponent bytes -> [rows, K] in 64 bits, by the layer's own table."""
    table = torch.tensor([0.0, 0.25, 1.0, 1.5, 2.0, 3.0, math.inf, math.nan], dtype=torch.float64, device=codes.device)
    table = torch.cat([table, -table])
    v = table[torch.stack([codes & 15, codes >> 4], dim=-1).flatten(-2).long()]
    return v * torch.exp2(scale.double() - 127.0).repeat_interleave(32, dim=1)


def exact(case, seed):
    """The layer in 64 bits from end to end, nothing rounded in between."""
    s, T = prepare(case, seed), case["tokens"]
    x = s["x"].double()
    layer = s.get("layer")
    if layer is not None:
        w13, s13, w2, s2, b13, b2 = layer.w13, layer.w13_scale, layer.w2, layer.w2_scale, None, None
        logits = x @ layer.router_weight.double().T if s["logits"] is None else s["logits"].double()
        E, k = logits.shape[1], case["top_k"]
        if case["routing"] == "softmax":
            score = torch.softmax(logits, dim=1)
            weights, ids = score.topk(k, dim=1)
            weights = weights / weights.sum(1, keepdim=True)
        else:   # the best four of eight groups by the sum of a group's two largest choices; weights without the bias
            score = torch.sigmoid(logits)
            choice = score + layer.router_bias.double()
            groups = choice.view(T, 8, E // 8)
            kept = groups.topk(2, dim=2)[0].sum(2).topk(4, dim=1)[1]
            open_ = torch.zeros(T, 8, dtype=torch.bool, device=x.device).scatter_(1, kept, True)
            ids = groups.masked_fill(~open_[:, :, None], -math.inf).flatten(1).topk(k, dim=1)[1]
            weights = score.gather(1, ids)
            weights = 2.5 * weights / weights.sum(1, keepdim=True)
        if case["shared"]:
            ids = torch.cat([ids, torch.full((T, 1), E, device=x.device)], dim=1)
            weights = torch.cat([weights, torch.ones((T, 1), dtype=torch.float64, device=x.device)], dim=1)
    else:
        w13, s13, w2, s2, b13, b2 = (s[n] for n in ("w13", "s13", "w2", "s2", "b13", "b2"))
        ids, weights = s["ids"].long(), s["weights"].double()
    out = torch.zeros((T, case["hidden"]), dtype=torch.float64, device=x.device)
    for e in range(w13.shape[0]):
        rows, slot = (ids == e).nonzero(as_tuple=True)
        if rows.numel() == 0:
            continue
        h = x[rows] @ _dense(w13[e], s13[e]).T
        if b13 is not None:
            h = h + b13[e].double()
        g, u = h.chunk(2, dim=1)
        if case["situ"]:
            a = 4.0 * torch.tanh(g / 4.0) * torch.sigmoid(g) * (25.0 * torch.tanh(u / 25.0))
        else:
            if case["limit"] > 0:
                g, u = g.clamp(max=case["limit"]), u.clamp(-case["limit"], case["limit"])
            a = g * torch.sigmoid(g) * u
        y = a @ _dense(w2[e], s2[e]).T
        if b2 is not None:
            y = y + b2[e].double()
        out.index_add_(0, rows, y * weights[rows, slot][:, None])
    return out


def work(case):
    """Weights and scales of the experts the batch is expected to touch, activations in, bf16 result out, and the router
    weight or the given routing; three multiply-add GEMMs per routed slot."""
    cfg, T = _config(case), case["tokens"]
    if cfg.zipf_alpha:
        p = [(1.0 + e) ** -cfg.zipf_alpha for e in range(cfg.E)]
        touched = sum(1.0 - (1.0 - min(1.0, cfg.top_k * q / sum(p))) ** T for q in p)
    else:
        touched = cfg.E * (1.0 - (1.0 - cfg.top_k / cfg.E) ** T)
    routing = cfg.E * cfg.H * 4 if case["entry"] in ("graph", "forward") and not cfg.zipf_alpha else \
        (T * cfg.E * 4 if cfg.zipf_alpha else T * cfg.top_k * 8)
    return {"bytes": (touched + cfg.shared_experts) * cfg.expert_weight_bytes() + 2 * T * cfg.H * 2 + routing,
            "flops": cfg.flops(T)}


def tolerance(case):
    """The result is bf16 and the activation between the GEMMs is rounded to bf16 once. Measured against the same path in 64
    bits with the same two roundings (all listed cases and eight drawn ones, 48 tokens each): 2-norm 1.4e-4 to 4.1e-4, largest
    difference 0.008 to 0.032 of the root mean square (one bf16 step of a large value). About four times that is stated.

    Batches routed from their activations also carry the router's ties: fp32 logits summed in another order differ by about
    1e-6, and in a batch of thousands of tokens one may have its last pick change places with the runner-up. Such a token is off
    by about half its size, which is 0.5 / sqrt(tokens) of the whole batch's 2-norm: at 8192 tokens 0.0055."""
    if case["entry"] in ("graph", "forward") and not case["zipf"] and case["tokens"] > 512:
        return {"rel": 6e-3}
    return {"rel": 1.6e-3, "max": 0.12}
