"""Kernels whose blocks have one tile each, which all of a block's warps share, against the same rows in a tensor of several tiles per
block: a pair block on one sample and on as many as give every block more than one tile (and the attention two lines per block), with and without a mask, both nodes of the
attention and both directions of the update, bit for bit. The output of the attention takes a view that is not transposed as one
line: its tiles cross lines and samples."""

import pytest
import torch

from cases import PAIR, _PF_KW, pkg

pytestmark = pytest.mark.gpu
TEMPLATE = dict(c_z=64, c_hidden_mul=64, c_hidden_pair_att=16, no_heads_pair=4, transition_n=2)


def _block(dims, g):
    blk = pkg.PairBlock(**dims, **_PF_KW)
    with torch.no_grad():
        for p in blk.parameters():
            p.copy_(torch.randn(p.shape, generator=g) * (p.shape[-1] ** -0.5 if p.dim() > 1 else 0.1) + (1.0 if p.dim() == 1 else 0.0))
    return blk.to("cuda:0", torch.bfloat16).eval().requires_grad_(False)


@pytest.mark.parametrize("dims", [PAIR, TEMPLATE], ids=["c128", "c64"])
@pytest.mark.parametrize("N", [1, 2, 17, 37, 38, 64, 75, 100, 111, 112, 127, 128, 129, 148])
@pytest.mark.parametrize("masked", [False, True])
def test_a_lone_tile_equals_one_of_several(dims, N, masked):
    g = torch.Generator().manual_seed(N)
    blk = _block(dims, g)
    samples = -(-400 // N) if N > 2 else 20000 // (N * N)   # more tiles than twice the SMs, of lines and of rows
    z = torch.randn(samples, N, N, dims["c_z"], generator=g).to("cuda:0", torch.bfloat16)
    m = (torch.rand(samples, N, N, generator=g) < 0.9).to("cuda:0", torch.bfloat16) if masked else torch.ones_like(z[..., 0])
    with torch.no_grad():
        want = blk(z, m)
        got = blk(z[:1].contiguous(), m[:1].contiguous())
        last = blk(z[-1:].contiguous(), m[-1:].contiguous())
    pkg.lib.check_device_status()
    assert torch.isfinite(got).all() and torch.equal(got, want[:1]) and torch.equal(last, want[-1:])
