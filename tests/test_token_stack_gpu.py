"""The diffusion token stack over the numbers of rows at which its launches change: blocks whose conditioning rows, and fewer
whose projections, share a launch (2000 rows: ten, then two, and one), key counts that are no multiple of a key block. The stack
against its blocks called one by one, bit for bit: there every block has launches of its own. The adaptive LayerNorm's rows
against the same rows in calls of a few. And the lone-tile instantiation of the pair transition against the other one, bit for
bit."""

import pytest
import torch

import cases
from cases import PAIR, W, _PF_KW, pkg

pytestmark = pytest.mark.gpu


def _stack(blocks, g):
    st = pkg.DiffusionTransformer(**cases.DIFF, no_blocks=blocks, use_ada_layer_norm=True, n_query=None, n_key=None, inf=1e9)
    with torch.no_grad():
        for p in st.parameters():
            p.copy_(torch.randn(p.shape, generator=g) * (0.02 if p.dim() > 1 else 0.3) + (1.0 if p.dim() == 1 else 0.0))
    return st.to("cuda:0", torch.bfloat16).eval().requires_grad_(False)


# 700 rows: projections of 5 blocks per launch, rows of 20, then 4; 900: 4 and 24; 1400: 2 and 14, then 10
@pytest.mark.parametrize("N,samples,blocks", [(1, 1, 2), (31, 3, 2), (148, 2, 2), (99, 3, 2), (119, 5, 2), (237, 5, 2), (400, 5, 12),
                                              (350, 2, 24), (300, 3, 24), (280, 5, 24)])
@pytest.mark.parametrize("packed", [True, False])
def test_stack_equals_its_blocks(N, samples, blocks, packed, monkeypatch):
    """``packed``: the stack's projections of s lie back to back, or each layer has launches of its own."""
    if not packed:
        for layer in (pkg.AttentionPairBias, pkg.ConditionedTransitionBlock):
            monkeypatch.setattr(layer, "_cond_group", ())
    g = torch.Generator().manual_seed(N)
    st = _stack(blocks, g)
    a, s = (torch.randn(1, samples, N, c, generator=g).to("cuda:0", torch.bfloat16) for c in (768, 384))
    z = torch.randn(1, 1, N, N, 128, generator=g).to("cuda:0", torch.bfloat16)
    m = (torch.rand(1, 1, N, generator=g) < 0.9).to("cuda:0", torch.bfloat16)
    m[..., 0] = 1
    with torch.no_grad():
        got = st(a, s, z, mask=m)
        want = a
        for blk in st.blocks:
            want = blk(want, s, z, mask=m)
    pkg.lib.check_device_status()
    assert torch.isfinite(got).all() and torch.equal(got, want)


@pytest.mark.parametrize("rows", [5, 111, 296, 301, 593, 1185, 1777, 2370])
def test_adaptive_rows_equal_those_of_short_calls(rows):
    """One to four blocks per SM, no limit; every seventh row's gates below -44, where the sigmoid's division is taken."""
    dev, bf = torch.device("cuda:0"), torch.bfloat16
    g = torch.Generator().manual_seed(rows)
    blk = _stack(1, g).blocks[0].conditioned_transition
    blk.layer_norm.linear_g.weight.zero_()
    blk.layer_norm.linear_g.weight[:, 0] = 20.0
    blk.layer_norm.layer_norm_s.weight.fill_(1.0)
    blk.layer_norm.linear_g.bias.zero_()
    a, s = (torch.randn(1, rows, c, generator=g) for c in (768, 384))
    s[..., 0] = 1.0
    s[:, ::7, 0] = -3.0
    a, s = a.to(dev, bf), s.to(dev, bf)
    with torch.no_grad():
        whole = blk(a, s, mask=None)
        parts = [blk(a[:, i:i + 67].contiguous(), s[:, i:i + 67].contiguous(), mask=None) for i in range(0, rows, 67)]
    pkg.lib.check_device_status()
    assert torch.isfinite(whole).all() and whole.any() and torch.equal(whole, torch.cat(parts, 1))


@pytest.mark.parametrize("rows", [1, 127, 128 * 147 + 1, 128 * 148])
def test_a_transition_of_lone_tiles_equals_that_of_several(rows):
    dev, bf = torch.device("cuda:0"), torch.bfloat16
    g = torch.Generator().manual_seed(rows)
    blk = pkg.PairBlock(**PAIR, **_PF_KW)
    blk.load_state_dict(W.pair_block_params(seed=5, final_std=None, **PAIR), strict=True)
    blk = blk.to(dev, bf).eval().requires_grad_(False)
    x = torch.randn(1, 1, 128 * 300, PAIR["c_z"], generator=g).to(dev, bf)
    m = (torch.rand(1, 1, 128 * 300, generator=g) < 0.9).to(dev, bf)
    with torch.no_grad():
        whole = blk.pair_transition(x, m)
        part = blk.pair_transition(x[:, :, :rows].contiguous(), m[:, :, :rows].contiguous())
    pkg.lib.check_device_status()
    assert torch.equal(part, whole[:, :, :rows])


def test_a_workspace_without_room_for_shared_launches_is_taken(monkeypatch):
    """The conditioning rows of three blocks (group of one: 1 + 2 slices of 2000 x 384) in a workspace short of the other two's;
    one that is shorter by 256 bytes (and the 256 of its alignment) more is refused."""
    N, samples, blocks = 400, 5, 3
    g = torch.Generator().manual_seed(1)
    st = _stack(blocks, g)
    a, s = (torch.randn(1, samples, N, c, generator=g).to("cuda:0", torch.bfloat16) for c in (768, 384))
    z = torch.randn(1, 1, N, N, 128, generator=g).to("cuda:0", torch.bfloat16)
    real, short = pkg.lib.workspace, 4 * N * samples * 384 * 2
    with torch.no_grad():
        want = st(a, s, z, mask=None)
        monkeypatch.setattr(pkg.lib, "workspace", lambda n, *k, **kw: real(n, *k, **kw)[: n - short])
        got = st(a, s, z, mask=None)
        monkeypatch.setattr(pkg.lib, "workspace", lambda n, *k, **kw: real(n, *k, **kw)[: n - short - 512])
        with pytest.raises(RuntimeError, match="workspace too small"):
            st(a, s, z, mask=None)
    pkg.lib.check_device_status()
    assert torch.equal(got, want)
