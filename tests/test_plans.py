"""The parameter structs and packed weights that the native block calls work from: built once, kept while what they were
built from stays the same, built again when it changes. Everything here runs without a GPU (no kernel is called)."""

import sys
import threading

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


def test_threads_that_share_a_module(pkg):
    """Two types in turn on several threads, from the first call on: every thread gets a whole plan of its own type."""
    blk = pkg.PairBlock(c_z=64, c_hidden_mul=64, c_hidden_pair_att=16, no_heads_pair=4, transition_type="swiglu",
                        transition_n=2, pair_dropout=0.25, fuse_projection_weights=False, inf=1e9).eval().requires_grad_(False)
    wrong, interval = [], sys.getswitchinterval()

    def work(dtype):
        try:
            for _ in range(60):
                plan = blk._plans.get(blk, dtype, CPU)
                pointers = [plan.params.tri_mul_in.w_z, plan.params.pair_transition.w_out]
                mine = [plan.keep[1][9], plan.keep[4][4]]
                if plan.dtype != dtype or any(t.dtype != dtype for t in mine) or pointers != [t.data_ptr() for t in mine]:
                    wrong.append("another thread's plan")
        except Exception as e:   # noqa: BLE001
            wrong.append(repr(e))

    sys.setswitchinterval(1e-6)
    try:
        threads = [threading.Thread(target=work, args=(d,)) for d in (BF, torch.float32) * 3]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
    finally:
        sys.setswitchinterval(interval)
    assert not wrong, wrong[:3]
