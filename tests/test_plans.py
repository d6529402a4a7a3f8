"""The parameter structs and packed weights that the native block calls work from: built once, kept while what they were
built from stays the same, built again when it changes. Everything here runs without a GPU (no kernel is called)."""

import copy
import gc
import pickle
import sys
import threading
import weakref

import pytest
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


def pair_block(pkg):
    return pkg.PairBlock(c_z=64, c_hidden_mul=64, c_hidden_pair_att=16, no_heads_pair=4, transition_type="swiglu",
                         transition_n=2, pair_dropout=0.25, fuse_projection_weights=False, inf=1e9).eval().requires_grad_(False)


def test_an_unchanged_module_keeps_its_plan(pkg):
    stack = diffusion(pkg)
    plan = params(stack)
    stack.eval()
    stack.hoist_pair_bias = False
    pkg.LayerNorm(8).eval()
    assert plan is not None and params(stack) is plan


EDITS = {
    "replaced block": lambda s, o: s.blocks.__setitem__(0, o.blocks[0]),
    "deleted block": lambda s, o: s.blocks.__delitem__(-1),
    "appended block": lambda s, o: s.blocks.append(o.blocks[0]),
    "inserted block": lambda s, o: s.blocks.insert(1, o.blocks[0]),
    "swapped blocks": lambda s, o: s._modules["blocks"]._modules.update({"0": s.blocks[1], "1": s.blocks[0]}),
    "another layer": lambda s, o: s.blocks[1].add_module("conditioned_transition", o.blocks[1].conditioned_transition),
    "another linear": lambda s, o: setattr(s.blocks[1].attention_pair_bias.mha, "linear_o",
                                           o.blocks[1].attention_pair_bias.mha.linear_o),
    "another parameter": lambda s, o: s.blocks[1].conditioned_transition.linear_out.register_parameter(
        "weight", torch.nn.Parameter(o.blocks[1].conditioned_transition.linear_out.weight.clone(), requires_grad=False)),
}


@pytest.mark.parametrize("edit", list(EDITS))
def test_edits_of_the_module_tree_are_seen(pkg, edit):
    """After the edit the structs say what those of a stack made that way say."""
    stack, other = diffusion(pkg), diffusion(pkg)
    params(stack, torch.float32)
    EDITS[edit](stack, other)
    plan = params(stack, torch.float32)
    assert len(plan.params[0]) == len(stack.blocks)
    for n, b in enumerate(stack.blocks):   # fp32 parameters are read where they are
        assert plan.params[0][n].w_o == b.attention_pair_bias.mha.linear_o.weight.data_ptr()
        assert plan.params[1][n].w_out == b.conditioned_transition.linear_out.weight.data_ptr()


@pytest.mark.parametrize("change", ["inf", "c_hidden", "training"])
def test_changed_constants_are_seen(pkg, change):
    blk = pair_block(pkg)
    plan = blk._plans.get(blk, BF, CPU)
    if change == "inf":
        blk.tri_att_start.inf = blk.tri_att_end.inf = 1e8
        assert blk._plans.get(blk, BF, CPU).shape(blk, 1, 8, 0, 0).dims.inf_pair == 1e8
    elif change == "c_hidden":   # the two directions no longer agree
        blk.tri_mul_in.c_hidden = 32
        assert blk._plans.get(blk, BF, CPU) is None
    else:
        blk.ps_dropout_row_layer.train()
        assert blk._plans.get(blk, BF, CPU) is None
    assert plan is not blk._plans._plan


@pytest.mark.parametrize("how", ["instance", "class", "hook", "global hook", "plain tensor", "computed"])
def test_what_the_native_call_would_pass_by_takes_the_layer_path(pkg, how, monkeypatch):
    blk = pair_block(pkg)
    assert blk._plans.get(blk, BF, CPU) is not None
    seen = lambda *a, **k: None  # noqa: E731
    if how == "instance":
        blk.tri_mul_in.forward = seen
    elif how == "class":
        monkeypatch.setattr(pkg.TriangleMultiplicationIncoming, "forward", seen)
    elif how == "hook":
        blk.tri_mul_out.register_forward_hook(seen)
    elif how == "global hook":
        handle = torch.nn.modules.module.register_module_forward_hook(seen)
    elif how == "plain tensor":   # may be written to without a trace in the module's parameters
        lin = blk.pair_transition.linear_out
        w = lin.weight.data
        del lin.weight
        lin.weight = w
    else:
        torch.nn.utils.parametrize.register_parametrization(blk.tri_att_end.linear_z, "weight", torch.nn.Identity())
    try:
        assert blk._plans.get(blk, BF, CPU) is None and blk._plans.get(blk, BF, CPU) is None
    finally:
        if how == "global hook":
            handle.remove()
            assert blk._plans.get(blk, BF, CPU) is not None



@pytest.mark.parametrize("change", ["layer_norm_z.weight", "layer_norm_z.bias", "linear_z.weight", "z", "data of z"])
def test_kept_pair_biases_are_projected_again(pkg, monkeypatch, change):
    """For new parameters (a new one starts at version 0, as the old one did) and new values of the pair tensor."""
    stack = diffusion(pkg)
    apb = stack.blocks[1].attention_pair_bias
    projected = []
    monkeypatch.setattr(pkg.AttentionPairBias, "can_hoist_pair_bias", lambda self, z: True)
    monkeypatch.setattr(pkg.AttentionPairBias, "project_pair_bias", lambda self, z: projected.append(self) or z)
    z = torch.zeros(1, 4, 4, 128)
    token = params(stack, torch.float32)
    first = stack._pair_biases(z, token)
    assert stack._pair_biases(z, token) is first and len(projected) == 3
    if change == "z":
        z.add_(1)
    elif change == "data of z":
        z.data = torch.ones(1, 4, 4, 128)
    else:
        layer, name = change.split(".")
        shape = (16, 128) if layer == "linear_z" else (128,)
        setattr(getattr(apb, layer), name, torch.nn.Parameter(torch.ones(shape), requires_grad=False))
    del projected[:]
    assert stack._pair_biases(z, params(stack, torch.float32)) is not first and len(projected) == 3
    assert stack._pair_biases(z) is not first and len(projected) == 3   # the layer path finds the new ones


@pytest.mark.parametrize("how", [copy.deepcopy, lambda m: pickle.loads(pickle.dumps(m))], ids=["deepcopy", "pickle"])
def test_a_used_module_can_be_copied(pkg, monkeypatch, how):
    """The copy packs its own weights, keeps no biases and has a plan of its own."""
    stack = diffusion(pkg)
    monkeypatch.setattr(pkg.AttentionPairBias, "can_hoist_pair_bias", lambda self, z: True)
    monkeypatch.setattr(pkg.AttentionPairBias, "project_pair_bias", lambda self, z: z)
    plan = params(stack)
    stack._pair_biases(torch.zeros(1, 4, 4, 128), plan)
    twin = how(stack)
    assert twin._bias_cache is None and stack._bias_cache is not None
    assert twin._packed._val is None and params(twin) is not plan and params(stack) is plan
    assert params(twin).params[1][0].w_out != plan.params[1][0].w_out


def test_modules_pickled_without_plans(pkg):
    """As a build that had no native calls pickled them."""
    stack = diffusion(pkg)
    for name in ("_plans", "_packed"):
        del stack.__dict__[name]
    blk = pair_block(pkg)
    del blk.__dict__["_plans"]
    assert params(pickle.loads(pickle.dumps(stack))) is not None
    blk = pickle.loads(pickle.dumps(blk))
    assert blk._plans.get(blk, BF, CPU) is not None


def test_projecting_pair_biases_packs_no_second_copy_of_the_layer(pkg, monkeypatch):
    stack = diffusion(pkg)
    monkeypatch.setattr(pkg.AttentionPairBias, "can_hoist_pair_bias", lambda self, z: True)
    got = []
    monkeypatch.setattr(pkg.lib, "pair_bias_project", lambda z, *prm: got.append(prm))
    stack._pair_biases(torch.zeros(1, 4, 4, 128), params(stack, torch.float32))
    for b, prm in zip(stack.blocks, got):
        apb = b.attention_pair_bias
        assert apb._packed._val is None
        assert all(torch.equal(x, y) for x, y in zip(prm, (apb.layer_norm_z.weight, apb.layer_norm_z.bias, apb.linear_z.weight))
                   if x is not None)


def test_parameters_of_a_flat_buffer(pkg):
    """Views at odd offsets, as a flattened or sharded model keeps them: the copies start where the kernels can read them."""
    stack = diffusion(pkg).to(BF)
    flat = torch.zeros(1 + sum(p.numel() + 1 for p in stack.parameters()), dtype=BF)
    at = 1
    for p in stack.parameters():
        flat[at:at + p.numel()].copy_(p.view(-1))
        p.data = flat[at:at + p.numel()].view(p.shape)
        at += p.numel() + 1
    plan = params(stack)
    assert any(p.data_ptr() % 16 for p in stack.parameters())
    pointers = [getattr(s, n) for array in plan.params for s in array for n, _ in s._fields_]
    assert pointers and all(p is None or p % 16 == 0 for p in pointers)
    assert torch.equal(plan.keep[11], stack.blocks[0].attention_pair_bias.mha.linear_q.weight)


def test_a_block_copies_no_weights_that_can_be_read_where_they_are(pkg):
    blk = pairformer_block(pkg).to(BF)
    plan = blk._plans.get(blk, BF, CPU)
    own = {p.data_ptr() for p in blk.parameters()}
    pair, attn, trans = plan.keep
    assert all(t is None or t.data_ptr() in own for ts in (*pair, attn, trans) for t in ts)


def pairformer_block(pkg):
    return pkg.PairFormerBlock(c_s=64, c_z=64, c_hidden_pair_bias=4, no_heads_pair_bias=16, c_hidden_mul=64, c_hidden_pair_att=16,
                               no_heads_pair=4, transition_type="swiglu", transition_n=2, pair_dropout=0.25,
                               fuse_projection_weights=False, inf=1e9).eval().requires_grad_(False)


@pytest.mark.parametrize("make", [pair_block, pairformer_block, diffusion])
def test_a_used_module_is_freed_with_its_last_reference(pkg, make):
    """Its weights with it, without waiting for the garbage collector: a plan does not refer to the module it belongs to."""
    m = make(pkg)
    assert m._plans.get(m, BF, CPU) is not None
    if make is pairformer_block:
        assert m.pair_stack._plans.get(m.pair_stack, BF, CPU) is not None
    gone = [weakref.ref(m), weakref.ref(next(m.parameters()))]
    gc.disable()
    try:
        del m
        assert all(r() is None for r in gone)
    finally:
        gc.enable()
