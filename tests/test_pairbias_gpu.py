"""Pair-bias projection for several layers in one pass: every layer's attention equals the one whose bias is projected
alone, bit for bit, at the edges of the projection's tiles (128 positions of a line, 32 keys, groups of 8 layers); and the
projected bias itself against fp64."""

import pytest
import torch

import cases
from cases import pkg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("blocks,N,samples", [(1, 5, 1), (3, 32, 2), (9, 33, 1), (17, 130, 2), (25, 64, 1)])
def test_blocks_projected_together_equal_blocks_projected_alone(blocks, N, samples):
    dev, bf = torch.device("cuda:0"), torch.bfloat16
    st = pkg.DiffusionTransformer(**cases.DIFF, no_blocks=blocks, use_ada_layer_norm=True, n_query=None, n_key=None, inf=1e9)
    g = torch.Generator().manual_seed(N)
    with torch.no_grad():
        for p in st.parameters():
            p.copy_(torch.randn(p.shape, generator=g) * (0.02 if p.dim() > 1 else 0.3) + (1.0 if p.dim() == 1 else 0.0))
    st = st.to(dev, bf).eval()
    a, s = (torch.randn(1, samples, N, c, generator=g).to(dev, bf) for c in (768, 384))
    z = torch.randn(1, 1, N, N, 128, generator=g).to(dev, bf)
    m = torch.ones(1, 1, N, device=dev, dtype=bf)
    with torch.no_grad():
        kept = st(a, s, z, mask=m)          # one projection launch per layer
        st.hoist_pair_bias = False
        assert torch.equal(st(a, s, z, mask=m), kept)
    pkg.lib.check_device_status()


@pytest.mark.parametrize("N,shift", [(3, 0.0), (129, 0.0), (160, 3.0)])
def test_projection_against_fp64(N, shift):
    dev, bf = torch.device("cuda:0"), torch.bfloat16
    g = torch.Generator().manual_seed(N)
    z = (torch.randn(1, N, N, 128, generator=g) + shift).to(bf)
    lw, lb = (1 + 0.2 * torch.randn(128, generator=g)).to(bf), (0.2 * torch.randn(128, generator=g)).to(bf)
    w = (torch.randn(16, 128, generator=g) / 128**0.5).to(bf)
    zz = z.double()
    zn = (zz - zz.mean(-1, keepdim=True)) / (zz.var(-1, unbiased=False, keepdim=True) + 1e-5).sqrt()
    ref = torch.einsum("bijc,hc->bhij", zn * lw.double() + lb.double(), w.double())
    got = pkg.lib.pair_bias_project(z.to(dev), lw.to(dev), lb.to(dev), w.to(dev))
    # W * gamma is rounded to bf16: unit roundoff u = 2^-8 (8 significand bits), so each weight is off by at most u of itself
    # and, evenly spread, by u / sqrt(3) in RMS. The error of a position is then that share of the output's RMS at most, and
    # the worst of up to 4e5 positions lies within 5 sigma (the same arithmetic in fp64 with rounded weights: 7.6e-3).
    bound = 5 * 2.0**-8 / 3**0.5
    assert cases.rel_err(got.cpu(), ref) < bound, cases.rel_err(got.cpu(), ref)
    pkg.lib.check_device_status()


@pytest.mark.parametrize("N", [5, 66, 130])
def test_bias_tiles_equal_a_converted_bias(N):
    """The two forms of a projected bias give the same attention, bit for bit: row-sharded callers project fp32 rows, whole
    tensors the tiles."""
    dev, bf = torch.device("cuda:0"), torch.bfloat16
    g = torch.Generator().manual_seed(N)
    apb = pkg.AttentionPairBias(c_q=384, c_k=384, c_v=384, c_s=384, c_z=128, c_hidden=24, no_heads=16)
    with torch.no_grad():
        for p in apb.parameters():
            p.copy_(torch.randn(p.shape, generator=g) * (p.shape[-1] ** -0.5 if p.dim() > 1 else 0.3) + (1.0 if p.dim() == 1 else 0.0))
    apb = apb.to(dev, bf).eval().requires_grad_(False)
    a, z = torch.randn(2, N, 384, generator=g).to(dev, bf), (1 + torch.randn(2, N, N, 128, generator=g)).to(dev, bf)
    prm = (apb.layer_norm_z.weight, apb.layer_norm_z.bias, apb.linear_z.weight)
    with torch.no_grad():
        outs = [apb._run(a, z, None, None, in_place=False, pair_bias=bias)
                for bias in (None, pkg.lib.pair_bias_project_tiles(z, *prm), pkg.lib.pair_bias_project(z, *prm))]
    pkg.lib.check_device_status()
    assert torch.equal(outs[0], outs[1]) and torch.equal(outs[1], outs[2])
