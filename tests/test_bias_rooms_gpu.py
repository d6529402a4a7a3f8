"""The rooms for the projected pair bias that the blocks of a trunk take in turn: more blocks than rooms, against the blocks one after
the other on one stream, and in a workspace that has one room only (what was asked for when there was one)."""

import pytest
import torch

from cases import PAIR, pkg

pytestmark = pytest.mark.gpu
SINGLE = dict(c_s=384, c_hidden_pair_bias=24, no_heads_pair_bias=16)
COMMON = dict(transition_type="swiglu", pair_dropout=0.25, fuse_projection_weights=False, inf=1e9, blocks_per_ckpt=None)


@pytest.mark.parametrize("N,blocks", [(40, 2), (40, 9), (200, 6)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_rooms_in_turn(N, blocks, dtype, monkeypatch):
    g = torch.Generator().manual_seed(N)
    st = pkg.PairFormerStack(**PAIR, **SINGLE, **COMMON, no_blocks=blocks)
    with torch.no_grad():
        for p in st.parameters():
            p.copy_(torch.randn(p.shape, generator=g) * (0.05 if p.dim() > 1 else 0.1) + (1.0 if p.dim() == 1 else 0.0))
    st = st.to("cuda:0", dtype).eval().requires_grad_(False)
    s = torch.randn(1, N, 384, generator=g).to("cuda:0", dtype)
    z = torch.randn(1, N, N, 128, generator=g).to("cuda:0", dtype)
    sm, pm = (torch.ones(1, *shape, dtype=dtype, device="cuda:0") for shape in ((N,), (N, N)))
    with torch.no_grad():
        got = [st(s, z, sm, pm) for _ in range(3)][-1]
        st.overlap_single_track = False
        want = st(s, z, sm, pm)
        st.overlap_single_track = True
        room = pkg.lib.load().of3_pair_bias_tiles_elems(N) * 2 if dtype == torch.bfloat16 else 16 * N * N * 4
        real = pkg.lib.workspace

        def short(n, device, stream=None):
            ws = real(n, device) if stream is None else real(n, device, stream)
            return ws if stream is not None else ws[: n - 3 * (-(-room // 256) * 256)]

        monkeypatch.setattr(pkg.lib, "workspace", short)
        old = st(s, z, sm, pm)
    pkg.lib.check_device_status()
    for a, b in zip(got, want):
        assert torch.isfinite(a).all() and torch.equal(a, b)
    for a, b in zip(old, want):
        assert torch.equal(a, b)
