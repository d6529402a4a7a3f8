"""The parameter structs and packed weights that the native block calls work from: built once, kept while what they were
built from stays the same, built again when it changes. Everything here runs without a GPU (no kernel is called)."""

import torch

CPU, BF = torch.device("cpu"), torch.bfloat16
DIFF = dict(c_a=128, c_s=64, c_z=128, c_hidden=8, no_heads=16, n_transition=2, use_ada_layer_norm=True, n_query=None,
            n_key=None, inf=1e9)


def diffusion(pkg, blocks=3):
    return pkg.DiffusionTransformer(**DIFF, no_blocks=blocks).eval().requires_grad_(False)


def params(stack, dtype=BF):
    return stack._plans.get(stack, dtype, CPU)


def test_packed_weights_survive_a_plan_that_is_built_again(pkg):
    """A captured graph reads the stacked conditioning weights by address: while no parameter changes they stay where they
    are, whatever else makes the structs be built again."""
    stack = diffusion(pkg)
    packed = stack._packed
    params(stack)
    cond = packed._val[3]
    stack.eval()
    pkg.LayerNorm(8)
    for b in stack.blocks:
        b.attention_pair_bias.inf = 1e8
    params(stack)
    assert packed._val[3] is cond
    stack.blocks[0].attention_pair_bias.linear_ada_out.weight.mul_(2)
    params(stack)
    assert packed._val[3] is not cond


def test_a_graph_holds_what_its_capture_read(pkg):
    stack = diffusion(pkg)
    with pkg.lib.holding() as held:
        params(stack)
        with pkg.lib.holding() as inner:
            pkg.lib.hold("inner")
    assert any(h is stack._packed._val for h in held) and inner == ["inner"] and "inner" not in held
    pkg.lib.hold("outside")
    assert "outside" not in held
