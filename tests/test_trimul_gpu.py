"""The triangle update at the edges of its line blocks (8), position tiles (128) and contraction tiles (128 x 256), with
several samples and both widths, against the fp32 oracle. Bars of tests/test_parity_gpu.py for one block of chained
layers: RMS error 8e-3, worst element 8e-2."""

import pytest
import torch

from cases import PAIR, W, _PF_KW, oracle, pkg, rand_mask, rel_err, rms_err

pytestmark = pytest.mark.gpu
TEMPLATE = dict(c_z=64, c_hidden_mul=64, c_hidden_pair_att=16, no_heads_pair=4, transition_n=2)


@pytest.mark.parametrize("dims,B,N", [(PAIR, 2, 7), (PAIR, 2, 8), (PAIR, 3, 9), (PAIR, 1, 120), (PAIR, 2, 129), (PAIR, 1, 257),
                                      (PAIR, 1, 264), (TEMPLATE, 3, 9), (TEMPLATE, 2, 129), (TEMPLATE, 1, 265)])
@pytest.mark.parametrize("outgoing", [True, False])
def test_triangle_update_matches_the_oracle(dims, B, N, outgoing):
    dev, bf = torch.device("cuda:0"), torch.bfloat16
    name = "tri_mul_out" if outgoing else "tri_mul_in"
    g = torch.Generator().manual_seed(N)
    P = {k: v.to(bf).float() for k, v in W.pair_block_params(seed=8, final_std=None, **dims).items()}
    z = torch.randn(B, N, N, dims["c_z"], generator=g).to(bf)
    m = rand_mask((B, N, N), g, 0.9)
    ref = z.float() + oracle.triangle_multiplicative_update(z.float(), m, P, name + ".", outgoing)
    blk = pkg.PairBlock(**dims, **_PF_KW)
    blk.load_state_dict(P, strict=True)
    blk = blk.to(dev, bf).eval()
    got = z.to(dev)
    with torch.no_grad():
        getattr(blk, name)(got, mask=m.to(dev, bf), inplace_safe=True, _add_with_inplace=True)
    pkg.lib.check_device_status()
    got = got.float().cpu()
    assert rms_err(got, ref) < 8e-3 and rel_err(got, ref) < 8e-2, (rms_err(got, ref), rel_err(got, ref))


@pytest.mark.parametrize("N", [8, 16, 20, 24, 40, 136, 200, 264])
def test_the_contraction_leaves_the_rest_of_the_pitch_alone(N):
    """Columns from N rounded up to 8 on belong to the caller (another result, or nothing: the last row may end the buffer),
    whatever width the pitch would allow a store."""
    dev, bf = torch.device("cuda:0"), torch.bfloat16
    g = torch.Generator().manual_seed(N)
    M, K, batch, used = 130, 72, 3, (N + 7) // 8 * 8
    ldo = (N + 15) // 16 * 16 + 16
    a = torch.randn(batch, M, K, generator=g).to(dev, bf)
    b = torch.randn(batch, N, K, generator=g).to(dev, bf)
    whole = torch.full((batch, M, ldo), 7.0, dtype=bf, device=dev)
    pkg.lib.contract_nt_bf16(a, b, whole)
    torch.cuda.synchronize()
    pkg.lib.check_device_status()
    assert (whole[..., used:] == 7).all()
    ref = torch.einsum("bik,bjk->bij", a.double(), b.double())
    # operands as given, fp32 sums of 72 products, one rounding to bf16: 2^-9 relative and some 1e-6 of the sum's terms
    assert ((whole[..., :N].double() - ref).abs() <= 2**-8 * ref.abs() + 1e-4).all()
