"""The native block entry points against the layer-by-layer path of the same modules: the same kernels in the same order,
so the same bits; parameters changed in place, replaced, or moved between calls are seen."""

import ctypes

import pytest
import torch

from cases import OF3, W, _PF_KW, pkg, token_pair_mask

pytestmark = pytest.mark.gpu


def _layers(stack, s, z, sm, pm):
    for b in stack.blocks:
        p = b.pair_stack
        z = p.tri_mul_out_in(z, pm, inplace_safe=False)
        z = p.tri_att_start_end(z, None, pm, False, False, False, inplace_safe=True)
        z = p.pair_transition._run(z, pm, in_place=True)
        s = b.attn_pair_bias._run(s.clone(), z, None, sm, in_place=True)
        s = b.single_transition._run(s, sm, in_place=True)
    return s, z


@pytest.mark.parametrize("dtype,B,N", [(torch.bfloat16, 1, 37), (torch.bfloat16, 2, 130), (torch.float32, 2, 19)])
def test_native_blocks_equal_the_layers(dtype, B, N):
    dev = torch.device("cuda:0")
    st = pkg.PairFormerStack(**OF3, **_PF_KW, no_blocks=2, blocks_per_ckpt=None)
    st.load_state_dict(W.pairformer_stack_params(seed=5, no_blocks=2, **OF3))
    st = st.to(dev, dtype).eval()
    g = torch.Generator().manual_seed(N)
    sm = torch.ones(B, N)
    sm[:, -3:] = 0
    s, z = torch.randn(B, N, 384, generator=g), torch.randn(B, N, N, 128, generator=g)
    s, z, sm, pm = (t.to(dev, dtype) for t in (s, z, sm, token_pair_mask(sm)))
    with torch.no_grad():
        for _ in range(2):   # the second time with other weights at the same addresses and at new ones
            ref = _layers(st, s, z, sm, pm)
            got = st(s, z, sm, pm)
            blk = st.blocks[0](s, z, sm, pm)
            one = _layers(type("S", (), {"blocks": [st.blocks[0]]}), s, z, sm, pm)
            for a, b in zip((*got, *blk), (*ref, *one)):
                assert torch.equal(a, b)
            st.blocks[0].pair_stack.tri_att_end.mha.linear_o.weight.mul_(1.5)
            lin = st.blocks[1].single_transition.linear_out
            lin.weight = torch.nn.Parameter(lin.weight.flip(0).contiguous(), requires_grad=False)


def test_a_hook_takes_the_layer_path():
    dev = torch.device("cuda:0")
    blk = pkg.PairFormerBlock(**OF3, **_PF_KW).to(dev, torch.bfloat16).eval()
    s, z = torch.randn(1, 20, 384, device=dev).bfloat16(), torch.randn(1, 20, 20, 128, device=dev).bfloat16()
    seen = []
    h = blk.pair_stack.tri_mul_in.register_forward_hook(lambda m, i, o: seen.append(o.shape))
    with torch.no_grad():
        blk(s, z, None, None)
        h.remove()
        blk(s, z, None, None)
    assert seen == [z.shape]


def test_kept_biases_where_the_attention_is_the_generic_one():
    """c_s beyond the tensor-core layer's limit: the kept biases are fp32 tensors, read as such. Against the call that projects
    its own: the same kernels but for the projection, whose operands are bf16 in one and fp32 in the other (2^-9 per product,
    on a bias of order one in front of a softmax; the update is some 0.3 of the output): the bar of one bf16 block, 8e-3."""
    dev, bf = torch.device("cuda:0"), torch.bfloat16
    g = torch.Generator().manual_seed(4)
    st = pkg.DiffusionTransformer(c_a=768, c_s=2112, c_z=128, c_hidden=48, no_heads=16, no_blocks=1, n_transition=2,
                                  use_ada_layer_norm=True, n_query=None, n_key=None, inf=1e9)
    with torch.no_grad():
        for p in st.parameters():
            p.copy_(torch.randn(p.shape, generator=g) * (p.shape[-1] ** -0.5 if p.dim() > 1 else 0.1))
    st = st.to(dev, bf).eval().requires_grad_(False)
    a, s, z = (torch.randn(sh, generator=g).to(dev, bf) for sh in ((1, 2, 33, 768), (1, 2, 33, 2112), (1, 1, 33, 33, 128)))
    with torch.no_grad():
        kept = st(a, s, z)
        assert st._bias_cache[3][0].dtype == torch.float32
        st.hoist_pair_bias = False
        own = st(a, s, z)
    pkg.lib.check_device_status()
    assert ((kept - own).float().norm() / own.float().norm()).item() < 8e-3


def test_the_first_launch_of_a_call_is_not_chained():
    """It stands behind whatever the caller enqueued, an update of the weights for instance, which its loads ahead of the wait
    must not overtake; all other launches of the tensor-core path are chained."""
    dev, bf = torch.device("cuda:0"), torch.bfloat16
    L = pkg.lib.load()

    def counts(call):
        pkg.lib.profile_begin(timing=False)
        with torch.no_grad():
            call()
        total = sum(n for n, _ in pkg.lib.profile_end().values())
        chained, ms = ctypes.c_longlong(0), ctypes.c_float(0)
        assert L.of3_profile_read(0, ctypes.byref(chained), ctypes.byref(ms)) == 0
        return total, total - chained.value

    st = pkg.PairFormerStack(**OF3, **_PF_KW, no_blocks=3, blocks_per_ckpt=None).to(dev, bf).eval().requires_grad_(False)
    s, z = torch.randn(1, 20, 384, device=dev).to(bf), torch.randn(1, 20, 20, 128, device=dev).to(bf)
    p = st.blocks[0].pair_stack
    for layer in (p.tri_mul_out, p.tri_att_start, p.pair_transition):
        assert counts(lambda: layer(z))[1] == 1
    assert counts(lambda: p(z, None))[1] == 1
    total, unchained = counts(lambda: st(s, z, None, None))   # the blocks' weights are packed in between
    assert unchained == 3 and counts(lambda: st(s, z, None, None)) == (total, 1)
    st.blocks[2].pair_stack.tri_att_end.mha.linear_o.weight.mul_(1.5)
    assert counts(lambda: st(s, z, None, None)) == (total, 2)


@pytest.mark.parametrize("offset", [1, 16, 255])
def test_a_workspace_may_start_anywhere(monkeypatch, offset):
    """A caller's workspace of exactly the bytes that were asked for, at any address: same bits."""
    dev, bf = torch.device("cuda:0"), torch.bfloat16
    g = torch.Generator().manual_seed(2)
    st = pkg.PairFormerStack(**OF3, **_PF_KW, no_blocks=2, blocks_per_ckpt=None)
    st.load_state_dict(W.pairformer_stack_params(seed=5, no_blocks=2, **OF3))
    diff = pkg.DiffusionTransformer(c_a=768, c_s=384, c_z=128, c_hidden=48, no_heads=16, no_blocks=1, n_transition=2,
                                    use_ada_layer_norm=True, n_query=None, n_key=None, inf=1e9)
    st, diff = (m.to(dev, bf).eval().requires_grad_(False) for m in (st, diff))
    diff.hoist_pair_bias = False
    s, z = torch.randn(1, 37, 384, generator=g).to(dev, bf), torch.randn(1, 37, 37, 128, generator=g).to(dev, bf)
    a = torch.randn(1, 37, 768, generator=g).to(dev, bf)

    def run():
        with torch.no_grad():
            blk = st.blocks[0]
            return (*st(s, z, None, None), *blk(s, z, None, None), blk.pair_stack(z, None), diff(a, s, z),
                    blk.attn_pair_bias(s, z), blk.single_transition(s), blk.pair_stack.tri_att_end(z))

    want, kept = run(), []

    def odd(nbytes, device, stream=None):
        torch.cuda.synchronize()   # (made anew per call)
        kept.append(torch.empty(nbytes + 512, dtype=torch.uint8, device=device))
        assert kept[-1].data_ptr() % 256 == 0
        return kept[-1][offset:offset + nbytes]

    monkeypatch.setattr(pkg.lib, "workspace", odd)
    got = run()
    torch.cuda.synchronize()
    pkg.lib.check_device_status()
    assert len(kept) > 5 and all(torch.equal(x, y) for x, y in zip(got, want))
