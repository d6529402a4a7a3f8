"""What the native block calls are given: tensors of other shapes or devices than the kernels read are refused on the host,
as the layers refuse them. The library calls are recorded instead of made; nothing here needs a GPU."""

import pytest
import torch

from cases import DIFF, OF3, PAIR, _PF_KW

BF = torch.bfloat16


class OnGpu(torch.Tensor):
    """A host tensor that passes for a CUDA one."""

    is_cuda = property(lambda self: True)


def gpu(*shape, dtype=BF):
    return torch.zeros(shape, dtype=dtype).as_subclass(OnGpu)


@pytest.fixture
def calls(pkg, monkeypatch):
    made = []
    for name in ("pair_block_forward", "pairformer_block_forward", "diffusion_stack_forward", "trimul_forward",
                 "triattn_forward", "transition_forward", "attn_pair_bias_forward", "attn_pair_bias_forward_pretiles",
                 "attn_pair_bias_forward_prebias", "cond_transition_forward"):
        monkeypatch.setattr(pkg.lib, name, lambda *a, _n=name, **k: made.append(_n))
    monkeypatch.setattr(pkg.lib, "pair_bias_project_tiles",
                        lambda z, *p: torch.zeros(z.shape[0], 16, (z.shape[1] + 31) // 32, z.shape[1], 32, dtype=BF))
    return made


@pytest.fixture(scope="module")
def block(pkg):
    return pkg.PairFormerBlock(**OF3, **_PF_KW).eval().to(BF).requires_grad_(False)


@pytest.fixture(scope="module")
def diffusion(pkg):
    return pkg.DiffusionTransformer(**DIFF, no_blocks=2, use_ada_layer_norm=True, n_query=None, n_key=None,
                                    inf=1e9).eval().to(BF).requires_grad_(False)


def test_good_shapes_take_one_native_call(block, diffusion, calls):
    with torch.no_grad():
        block.pair_stack(gpu(1, 20, 20, 128), None)
        block(gpu(2, 20, 384), gpu(2, 20, 20, 128), None, None)
        diffusion(gpu(1, 3, 20, 768), gpu(1, 3, 20, 384), gpu(1, 1, 20, 20, 128))
    assert calls == ["pair_block_forward", "pairformer_block_forward", "diffusion_stack_forward"]


@pytest.mark.parametrize("z", [(1, 20, 20, 64), (1, 30, 20, 128), (1, 20, 30, 128), (0, 20, 20, 128), (20, 128)])
def test_pair_block_refuses_other_pair_tensors(block, calls, z):
    with torch.no_grad():
        try:
            block.pair_stack(gpu(*z), None)
        except (RuntimeError, IndexError, AssertionError):
            pass
    assert "pair_block_forward" not in calls


@pytest.mark.parametrize("s,z", [((1, 20, 128), (1, 20, 20, 128)), ((1, 20, 384), (1, 20, 20, 64)),
                                 ((1, 20, 384), (1, 20, 40, 128)), ((1, 10, 384), (1, 20, 20, 128))])
def test_pairformer_block_refuses_other_tensors(block, calls, s, z):
    with torch.no_grad():
        try:
            block(gpu(*s), gpu(*z), None, None)
        except (RuntimeError, AssertionError):
            pass
    assert "pairformer_block_forward" not in calls


def test_kept_biases_of_another_batch_are_refused(diffusion, calls):
    """Samples [2, 5] with pair tensors [1, 5]: the expanded pair tensor has ten entries, the kept biases five."""
    with torch.no_grad(), pytest.raises(AssertionError):
        diffusion(gpu(2, 5, 20, 768), gpu(2, 5, 20, 384), gpu(1, 5, 20, 20, 128))
    assert calls == []


def test_tensors_of_another_device_are_refused(block, diffusion, calls):
    far = lambda *shape: torch.zeros(shape, dtype=BF, device="meta")  # noqa: E731
    a, s, z = gpu(1, 2, 20, 768), gpu(1, 2, 20, 384), gpu(1, 1, 20, 20, 128)
    with torch.no_grad():
        for call in (lambda: block(far(1, 20, 384), gpu(1, 20, 20, 128), None, None),
                     lambda: block(gpu(1, 20, 384), gpu(1, 20, 20, 128), far(1, 20), None),
                     lambda: block.pair_stack(gpu(1, 20, 20, 128), far(1, 20, 20)),
                     lambda: diffusion(a, far(1, 2, 20, 384), z),
                     lambda: diffusion(a, s, far(1, 1, 20, 20, 128)),
                     lambda: diffusion(a, s, z, mask=far(1, 2, 20))):
            with pytest.raises(RuntimeError, match="is on meta"):
                call()
    assert calls == []


@pytest.mark.parametrize("c_s,N,dtype", [(384, 20, BF), (384, 8192, BF), (384, 8193, BF), (2048, 20, BF), (2112, 20, BF),
                                         (100, 20, BF), (384, 20, torch.float32)])
def test_the_projected_bias_has_the_form_that_the_library_reads(pkg, monkeypatch, c_s, N, dtype):
    """Sizes around the limits of the tensor-core attention and of its adaptive LayerNorm: bias tiles read as fp32 biases are
    half as long as what is read."""
    apb = pkg.AttentionPairBias(c_q=768, c_k=768, c_v=768, c_s=c_s, c_z=128, c_hidden=48, no_heads=16,
                                use_ada_layer_norm=True)
    made = []
    monkeypatch.setattr(pkg.lib, "pair_bias_project_tiles", lambda *a: made.append("tiles"))
    monkeypatch.setattr(pkg.lib, "pair_bias_project", lambda *a: made.append("f32"))
    apb.project_pair_bias(torch.empty(1, N, N, 128, dtype=dtype, device="meta"))
    lib = pkg.lib.load()
    code, flags = pkg.lib.dtype_code(dtype), pkg.lib.FLAG_ADA_LN
    fast = dtype == BF and c_s % 64 == 0 and c_s <= 2048 and N <= 8192
    assert made == ["tiles" if fast else "f32"]
    assert lib.of3_pair_bias_takes_tiles(N, 768, c_s, 128, 16, 48, code, flags) == fast
    assert lib.of3_pair_bias_takes_tiles(N, 768, c_s, 128, 16, 48, code, flags | pkg.lib.FLAG_FORCE_GENERIC) == 0


def test_a_failed_stack_call_still_joins_the_second_stream(pkg, calls, monkeypatch):
    """The blocks before the failure have work on it that reads and writes tensors of the main stream."""
    stack = pkg.PairFormerStack(**OF3, **_PF_KW, no_blocks=3, blocks_per_ckpt=None).eval().to(BF).requires_grad_(False)
    waits = []
    monkeypatch.setattr(torch.cuda, "current_stream", lambda device=None: "main")
    monkeypatch.setattr(pkg.lib, "side_stream", lambda main: "side")
    monkeypatch.setattr(pkg.lib, "stream_wait", lambda waiter, signaler: waits.append((waiter, signaler)))

    def call(*args):
        calls.append("block")
        if len(calls) == 2:
            raise RuntimeError("second block")

    monkeypatch.setattr(pkg.lib, "pairformer_block_forward", call)
    with torch.no_grad(), pytest.raises(RuntimeError, match="second block"):
        stack(gpu(1, 20, 384), gpu(1, 20, 20, 128), None, None)
    assert calls == ["block", "block"] and waits == [("side", "main"), ("main", "side")]


def test_only_blocks_behind_a_block_continue(pkg, monkeypatch):
    """A block whose weights have just been packed, or written to, starts behind all work before it."""
    stack = pkg.PairFormerStack(**OF3, **_PF_KW, no_blocks=3, blocks_per_ckpt=None).eval().to(BF).requires_grad_(False)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda device=None: "main")
    monkeypatch.setattr(pkg.lib, "side_stream", lambda main: "side")
    monkeypatch.setattr(pkg.lib, "stream_wait", lambda *a: None)
    flags = []
    monkeypatch.setattr(pkg.lib, "pairformer_block_forward",
                        lambda s, z, sm, pm, plan, dt, f, prm, side: flags.append(bool(f & pkg.lib.FLAG_CONTINUES)))

    def call():
        del flags[:]
        with torch.no_grad():
            stack(gpu(1, 20, 384), gpu(1, 20, 20, 128), None, None)
        return flags

    assert call() == [False, False, False] and call() == [False, True, True]
    stack.blocks[1].single_transition.linear_out.weight.mul_(2)
    assert call() == [False, False, True] and call() == [False, True, True]


def test_a_pair_stack_continues_from_block_to_block(pkg, monkeypatch):
    """But not past a block that is run by a call of its own, with its hooks."""
    stack = pkg.PairStack(no_blocks=3, **{k: v for k, v in OF3.items() if k in PAIR}, **_PF_KW).eval().to(BF).requires_grad_(False)
    flags, hooked = [], []
    monkeypatch.setattr(pkg.lib, "pair_block_forward",
                        lambda z, pm, plan, dt, f, prm: flags.append(bool(f & pkg.lib.FLAG_CONTINUES)))

    def call():
        del flags[:]
        with torch.no_grad():
            stack(gpu(1, 20, 20, 128), None)
        return flags

    assert call() == [False, False, False] and call() == [False, True, True]
    hook = stack.blocks[1].register_forward_pre_hook(lambda m, args: hooked.append(m))
    assert call() == [False, False, False] and hooked == [stack.blocks[1]]
    hook.remove()
    assert call() == [False, True, True]


def test_a_replaced_step_of_a_pair_block_is_run(pkg, calls):
    blk = pkg.PairBlock(**{k: v for k, v in OF3.items() if k in PAIR}, **_PF_KW).eval().to(BF).requires_grad_(False)
    seen = []
    blk.tri_mul_out_in = lambda z, *a, **k: seen.append("step") or z
    with torch.no_grad():
        blk(gpu(1, 20, 20, 128), None)
    assert seen == ["step"] and "pair_block_forward" not in calls
