"""The native block entry points against the layer-by-layer path of the same modules: the same kernels in the same order,
so the same bits; parameters changed in place, replaced, or moved between calls are seen."""

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
