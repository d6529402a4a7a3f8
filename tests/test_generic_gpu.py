"""The fp32 GEMM and attention tiles of the shape-generic family at their edges (32- and 128-row tiles, 64 queries x 64 keys,
widths that no vector load divides), against the oracle: 1e-4 x RMS on the worst element, the bar of the validation mode."""

import pytest
import torch

from cases import OF3, W, _PF_KW, oracle, pkg, rand_mask, rel_err, token_pair_mask

pytestmark = pytest.mark.gpu
ODD = dict(c_s=36, c_z=20, c_hidden_pair_bias=9, no_heads_pair_bias=4, c_hidden_mul=19, c_hidden_pair_att=14,
           no_heads_pair=3, transition_n=2)


@pytest.mark.parametrize("dims,B,N", [(OF3, 1, 1), (OF3, 2, 33), (OF3, 1, 65), (ODD, 2, 31), (ODD, 1, 130)])
def test_fp32_block_matches_the_oracle(dims, B, N):
    dev = torch.device("cuda:0")
    g = torch.Generator().manual_seed(N)
    P = W.pairformer_block_params(seed=41, final_std=None, **dims)
    s, z = torch.randn(B, N, dims["c_s"], generator=g), torch.randn(B, N, N, dims["c_z"], generator=g)
    sm = rand_mask((B, N), g, 0.9)
    pm = token_pair_mask(sm)
    ref = oracle.pairformer_block(s, z, sm, pm, P, "", dims["no_heads_pair"], dims["no_heads_pair_bias"])
    blk = pkg.PairFormerBlock(**dims, **_PF_KW)
    blk.load_state_dict(P, strict=True)
    blk = blk.to(dev).eval()
    with torch.no_grad():
        got = blk(s.to(dev), z.to(dev), sm.to(dev), pm.to(dev))
    for a, b in zip(got, ref):
        assert rel_err(a.cpu(), b) < 1e-4, rel_err(a.cpu(), b)


@pytest.mark.parametrize("c_z,c_hidden_mul,heads,d,n,N", [(128, 128, 4, 32, 4, 101), (36, 20, 3, 12, 2, 141), (68, 36, 2, 18, 1, 139)])
def test_fp32_pair_block_on_large_tiles(c_z, c_hidden_mul, heads, d, n, N):
    """Enough rows for the 128 x 64 tiles, with a ragged last one; widths in whole vectors that divide neither a slab of 16 nor
    a tile."""
    dims = dict(c_z=c_z, c_hidden_mul=c_hidden_mul, c_hidden_pair_att=d, no_heads_pair=heads, transition_n=n)
    dev = torch.device("cuda:0")
    g = torch.Generator().manual_seed(N)
    P = W.pair_block_params(seed=43, final_std=None, **dims)
    z, m = torch.randn(1, N, N, c_z, generator=g), rand_mask((1, N, N), g, 0.9)
    ref = oracle.pair_block(z, m, P, "", heads)
    blk = pkg.PairBlock(**dims, **_PF_KW)
    blk.load_state_dict(P, strict=True)
    blk = blk.to(dev).eval()
    with torch.no_grad():
        got = blk(z.to(dev), m.to(dev)).cpu()
    assert rel_err(got, ref) < 1e-4, rel_err(got, ref)


@pytest.mark.parametrize("c_hidden_mul,B,N", [(128, 1, 68), (128, 2, 132), (36, 1, 140)])
def test_fp32_contraction_in_whole_vectors(c_hidden_mul, B, N):
    """N in whole vectors and enough planes for the 128 x 64 tiles: the outgoing update's N x N products, a plane per batch
    entry, read in vectors along k, with ragged row and column tiles and a ragged last slab of k."""
    dev = torch.device("cuda:0")
    g = torch.Generator().manual_seed(N)
    z, m = torch.randn(B, N, N, 32, generator=g), rand_mask((B, N, N), g, 0.9)
    for cls in (pkg.TriangleMultiplicationOutgoing, pkg.TriangleMultiplicationIncoming):
        layer = cls(32, c_hidden_mul)
        with torch.no_grad():
            for p in layer.parameters():
                p.copy_(torch.randn(p.shape, generator=g) * (p.shape[-1] ** -0.5 if p.dim() > 1 else 0.3))
            P = {"l." + k: v.clone() for k, v in layer.state_dict().items()}
            ref = oracle.triangle_multiplicative_update(z, m, P, "l.", outgoing=cls is pkg.TriangleMultiplicationOutgoing)
            got = layer.to(dev).eval()(z.to(dev), mask=m.to(dev)).cpu()
        assert rel_err(got, ref) < 1e-4, rel_err(got, ref)
