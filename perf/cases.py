"""Workloads of the Pairformer hot path, as the programs that embed this package run it.

``kind`` says which public module is called:

  trunk      ``PairFormerStack`` on a pair and a single tensor (the model's trunk, the confidence head's four blocks)
  pair       ``PairStack`` on a pair tensor alone (the MSA module's pair stacks, large complexes)
  template   ``PairStack`` at the template embedder's widths: two blocks, c = 64, 4 heads x 16, transition n = 2, 5-D input
             [1, templates, N, N, 64]
  diffusion  ``DiffusionTransformer`` on the noisy token activations of some samples that share one pair tensor

The other keys: ``n`` tokens, ``blocks`` of the stack, ``dtype`` bf16 or f32 (the validation mode), ``pad`` the share of
tokens that are padding and ``where`` they lie ("tail", or "random" for unresolved tokens), ``lead`` the templates or the
diffusion samples, ``kept`` whether the diffusion stack keeps its pair-bias projections while the pair tensor stays the
same (its default, a rollout) or computes them in the call, ``graph`` whether the call is replayed by ``GraphedModule``.

The trunk has 48 blocks; its cases take a few of them, since the blocks are alike and the time of a pass grows with their
number, while the rounding differences between two correct bf16 programs grow with depth.
"""

from __future__ import annotations

import math

import torch

from __graft_entry__ import load_package

pkg = load_package()

PAIR = dict(c_z=128, c_hidden_mul=128, c_hidden_pair_att=32, no_heads_pair=4, transition_n=4)
TEMPLATE = dict(c_z=64, c_hidden_mul=64, c_hidden_pair_att=16, no_heads_pair=4, transition_n=2)
SINGLE = dict(c_s=384, c_hidden_pair_bias=24, no_heads_pair_bias=16)
DIFFUSION = dict(c_a=768, c_s=384, c_z=128, c_hidden=48, no_heads=16, n_transition=2)
COMMON = dict(transition_type="swiglu", pair_dropout=0.25, fuse_projection_weights=False, inf=1e9)

# n from .. to, and the most flop one pass may take (that of the largest listed case)
RANGES = {"trunk": (24, 1100), "pair": (24, 2048), "template": (32, 384), "diffusion": (24, 1024), "f32": (16, 256)}
MOST_FLOPS = 3.58e13


def _case(kind, n, blocks, dtype="bf16", pad=0.0, where="tail", lead=1, kept=False, graph=False):
    return dict(kind=kind, n=n, blocks=blocks, dtype=dtype, pad=pad, where=where, lead=lead, kept=kept, graph=graph)


def listed():
    return [
        # a peptide: every kernel is a few blocks wide, launches and host work are what a pass costs
        dict(_case("trunk", 37, 4), name="trunk_n37"),
        # a single protein chain padded to a bucket, the confidence head's depth
        dict(_case("trunk", 256, 4, pad=0.1), name="trunk_n256_pad"),
        # the size at which the trunk is quoted
        dict(_case("trunk", 768, 4), name="trunk_n768"),
        # a complex of no round size with unresolved tokens
        dict(_case("trunk", 1003, 2, pad=0.05, where="random"), name="trunk_n1003_ragged"),
        # the pair stack alone, the last 32 of 384 tokens padded
        dict(_case("pair", 384, 4, pad=32 / 384), name="pair_n384_pad"),
        # the pair stack of a large complex on one GPU
        dict(_case("pair", 2048, 2, pad=0.05, where="random"), name="pair_n2048"),
        # the template embedder over four templates
        dict(_case("template", 300, 2, pad=0.08, lead=4), name="template_n300_t4"),
        # one denoising step of five samples that projects its pair bias in the call, as one graph
        dict(_case("diffusion", 768, 24, lead=5, graph=True), name="diffusion_n768_s5_graph"),
        # a step in the middle of a rollout over five samples, called directly
        dict(_case("diffusion", 500, 24, pad=0.06, lead=5, kept=True), name="diffusion_n500_s5_rollout"),
        # a rollout step of one small sample, called directly: host and launch time
        dict(_case("diffusion", 111, 24, lead=1, kept=True), name="diffusion_n111_s1_rollout"),
        # the validation mode
        dict(_case("trunk", 128, 1, dtype="f32", pad=0.1), name="trunk_f32_n128"),
    ]


def draw(rng):
    while True:
        kind = rng.choice(["trunk", "trunk", "pair", "template", "diffusion", "diffusion", "f32"])
        lo, hi = RANGES[kind]
        n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
        pad = rng.choice([0.0, round(rng.uniform(0.02, 0.15), 3)])
        where = rng.choice(["tail", "random"])
        if kind == "f32":
            c = _case("trunk", n, 1, "f32", pad, where)
        elif kind == "template":
            c = _case(kind, n, 2, pad=pad, where=where, lead=rng.randint(1, 4))
        elif kind == "diffusion":
            c = _case(kind, n, 24, pad=pad, where=where, lead=rng.randint(1, 5), kept=rng.random() < 0.5,
                      graph=rng.random() < 0.4)
        else:
            c = _case(kind, n, rng.randint(1, 4), pad=pad, where=where)
        if work(c)["flops"] <= MOST_FLOPS:
            return c


def _dtype(case):
    return torch.float32 if case["dtype"] == "f32" else torch.bfloat16


def _build(case):
    """The module with its own initialisation, made on the GPU."""
    blocks = case["blocks"]
    with torch.device("cuda"):
        if case["kind"] == "trunk":
            return pkg.PairFormerStack(**PAIR, **SINGLE, **COMMON, no_blocks=blocks, blocks_per_ckpt=None)
        if case["kind"] == "pair":
            return pkg.PairStack(no_blocks=blocks, **PAIR, **COMMON)
        if case["kind"] == "template":
            return pkg.PairStack(no_blocks=blocks, **TEMPLATE, **COMMON)
        return pkg.DiffusionTransformer(**DIFFUSION, no_blocks=blocks, use_ada_layer_norm=True, n_query=None, n_key=None,
                                        inf=1e9)


def _draw_weights(model, g):
    """Values with the spreads of a trained stack: LayerNorm weights around 1, fan-in scaled projections, and small ones
    where the initialisation puts zeros (the gates and most output projections)."""
    with torch.no_grad():
        for name, p in model.named_parameters():
            r = torch.randn(p.shape, generator=g, device="cuda")
            if "layer_norm" in name and p.dim() == 1 and "linear" not in name:
                p.copy_(0.1 * r + (1.0 if name.endswith("weight") else 0.0))
            elif p.dim() == 1:
                p.copy_(0.1 * r + (-2.0 if bool((p == -2.0).all()) else 0.0))
            elif bool((p == 0).all()):
                p.copy_(0.02 * r)
            else:
                p.copy_(r * (1.0 / math.sqrt(p.shape[1])))


def _token_mask(case, g):
    n = case["n"]
    m = torch.ones(n, device="cuda")
    gone = int(round(case["pad"] * n))
    if gone:
        if case["where"] == "tail":
            m[n - gone:] = 0
        else:
            m[torch.randperm(n, generator=g, device="cuda")[:gone]] = 0
    return m


def prepare(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    dt, n, kind, lead = _dtype(case), case["n"], case["kind"], case["lead"]
    model = _build(case)
    _draw_weights(model, g)
    model = model.to(dt).eval().requires_grad_(False)
    normal = lambda *shape: torch.randn(shape, generator=g, device="cuda", dtype=dt)  # noqa: E731
    tm = _token_mask(case, g)
    pm = (tm[:, None] * tm[None, :]).to(dt)
    tm = tm.to(dt)
    if kind == "trunk":
        args = (normal(1, n, SINGLE["c_s"]), normal(1, n, n, PAIR["c_z"]), tm[None], pm[None])
        call = model
    elif kind == "pair":
        args = (normal(1, n, n, PAIR["c_z"]), pm[None])
        call = model
    elif kind == "template":
        args = (normal(1, lead, n, n, TEMPLATE["c_z"]), pm.expand(1, lead, n, n))
        call = model
    else:
        model.hoist_pair_bias = case["kept"]
        args = (normal(1, lead, n, DIFFUSION["c_a"]), normal(1, lead, n, DIFFUSION["c_s"]),
                normal(1, 1, n, n, DIFFUSION["c_z"]), tm[None, None])
        call = model
    if case["graph"]:
        if case["kept"]:   # the pair tensor belongs to the rollout, not to the step
            z = args[2]
            step = lambda a, s, mask: model(a, s, z, mask)  # noqa: E731
            args = (args[0], args[1], args[3])
        else:
            step = model
        call = pkg.GraphedModule(step, *args)
        return call, args, step   # the graph reads the weights (and the pair tensor) that the step holds
    return call, args, None


def run(state):
    call, args = state[:2]
    with torch.no_grad():
        return call(*args)


def _pair_block_flops(n, c_z, c_hidden_mul, c_hidden_pair_att, no_heads_pair, transition_n):
    ch, d, h = c_hidden_mul, c_hidden_pair_att, no_heads_pair
    tri_mul = 2 * (2.0 * n**3 * ch + 2.0 * n * n * (4 * c_z * ch + ch * c_z + c_z * c_z))
    tri_att = 2 * (4.0 * n**3 * h * d + 2.0 * n * n * (5 * c_z * h * d + c_z * h))
    return tri_mul + tri_att + 2.0 * n * n * 3 * c_z * transition_n * c_z


def work(case):
    """Inputs and weights read once, outputs written once; the matrix products of the layers."""
    n, blocks, lead = case["n"], case["blocks"], case["lead"]
    size = 4 if case["dtype"] == "f32" else 2
    if case["kind"] in ("trunk", "pair"):
        flops, values = blocks * _pair_block_flops(n, **PAIR), 2 * n * n * 128 + n * n + blocks * 530e3
        if case["kind"] == "trunk":
            c = SINGLE["c_s"]
            flops += blocks * (2.0 * n * n * 128 * 16 + 2.0 * n * c * c * 5 + 4.0 * n * n * c + 2.0 * n * 12 * c * c)
            values += 2 * n * c + n + blocks * 17 * c * c
        return {"bytes": size * values, "flops": flops}
    if case["kind"] == "template":
        return {"bytes": size * lead * (2 * n * n * 64 + n * n), "flops": lead * blocks * _pair_block_flops(n, **TEMPLATE)}
    c, cs = DIFFUSION["c_a"], DIFFUSION["c_s"]
    flops = blocks * lead * n * (2.0 * 5 * c * c + 2.0 * 6 * cs * c + 4.0 * n * c + 2.0 * 3 * c * 2 * c)
    values = lead * n * (2 * c + cs) + n + blocks * (11 * c * c + 6 * cs * c)
    if case["kept"]:
        values += blocks * 16 * n * n   # the projected pair bias of every block
    else:
        flops += blocks * 2.0 * n * n * 128 * 16
        values += n * n * 128
    return {"bytes": size * values, "flops": flops}


def tolerance(case):
    """bf16 operands of every product and bf16 storage between layers: an RMS error of 4e-3 per block of the trunk, growing
    like the root of the depth, in each of two programs. The diffusion stack rounds its activations 48 times, each 1.1e-3,
    again in both. f32: sums of at most 2048 products."""
    if case["dtype"] == "f32":
        return {"rel": 1e-5}
    return {"rel": 0.016 if case["kind"] == "diffusion" else 0.006 * math.sqrt(case["blocks"])}
