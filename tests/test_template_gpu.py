"""The pair block at the template stack's widths (c = 64, 4 heads x 16, transition n = 2) on its tensor-core kernels, and the
attention core of both widths at the edges of its tiles (128 queries, 64 keys, pairs of lines, 32-key bias tiles), against
the fp32 oracle. Bars of tests/test_parity_gpu.py for one block of chained layers: RMS error 8e-3, worst element 8e-2."""

import pytest
import torch

from cases import PAIR, W, _PF_KW, oracle, pkg, rand_mask, rel_err, rms_err

pytestmark = pytest.mark.gpu
TEMPLATE = dict(c_z=64, c_hidden_mul=64, c_hidden_pair_att=16, no_heads_pair=4, transition_n=2)


@pytest.mark.parametrize("dims,B,N", [(TEMPLATE, 2, 1), (TEMPLATE, 2, 33), (TEMPLATE, 1, 64), (TEMPLATE, 3, 97),
                                      (TEMPLATE, 1, 161), (PAIR, 1, 1), (PAIR, 1, 63), (PAIR, 1, 97), (PAIR, 1, 129)])
def test_pair_block_matches_the_oracle(dims, B, N):
    dev, bf = torch.device("cuda:0"), torch.bfloat16
    g = torch.Generator().manual_seed(N)
    P = {k: v.to(bf).float() for k, v in W.pair_block_params(seed=31, final_std=None, **dims).items()}
    z = torch.randn(B, N, N, dims["c_z"], generator=g).to(bf)
    m = rand_mask((B, N, N), g, 0.9)
    assert pkg.lib.fast_path_available(pkg.lib.MODULE_TRIATTN, bf, dims["c_z"], 0, 4, dims["c_hidden_pair_att"])
    ref = oracle.pair_block(z.float(), m, P, "", 4)
    blk = pkg.PairBlock(**dims, **_PF_KW)
    blk.load_state_dict(P, strict=True)
    blk = blk.to(dev, bf).eval()
    with torch.no_grad():
        got = blk(z.to(dev), m.to(dev, bf)).float().cpu()
    pkg.lib.check_device_status()
    assert rms_err(got, ref) < 8e-3 and rel_err(got, ref) < 8e-2, (rms_err(got, ref), rel_err(got, ref))
