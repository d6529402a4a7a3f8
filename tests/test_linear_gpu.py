"""The linear layers of the single track and of the diffusion token stack in their several forms, bit for bit.

The output projections, whose gate, residual and result pass through shared memory where the caller's tensors start on 16 bytes,
against the same call on tensors that do not (every thread then reads and writes rows of its own): the same products, gates and
sums in the same order. Rows: part of a tile, its edges, several tiles per block. The launches for few tokens against those of
128-row tiles."""

import pytest
import torch

from cases import pkg

pytestmark = pytest.mark.gpu


def _at(x, offset):
    """``x`` as a dense tensor that starts ``offset`` bytes behind a 256-byte boundary."""
    buf = torch.zeros(x.numel() * 2 + 512, dtype=torch.uint8, device=x.device)
    start = -buf.data_ptr() % 256 + offset
    y = buf[start:start + 2 * x.numel()].view(torch.bfloat16).view(x.shape)
    return y.copy_(x)


# widths whose column tiles are 64, 128 and 192 wide; 128 x 38 + 5 rows of 768: more tiles than blocks
@pytest.mark.parametrize("rows,c", [(1, 768), (127, 768), (128, 768), (129, 320), (1153, 768), (2500, 768), (3840, 768),
                                    (128 * 38 + 5, 768), (128 * 75 + 1, 512)])
@pytest.mark.parametrize("gated,residual", [(True, True), (True, False), (False, True), (False, False)])
def test_staged_rows_equal_direct_ones(rows, c, gated, residual):
    dev, bf = torch.device("cuda:0"), torch.bfloat16
    g = torch.Generator().manual_seed(rows + c)
    n, c_s = 2, 384

    def w(*shape):
        return (torch.randn(shape, generator=g) * shape[-1] ** -0.5).to(dev, bf)

    x, s = (torch.randn(rows, k, generator=g).to(dev, bf) for k in (c, c_s))
    mask = torch.rand(rows, generator=g).to(dev, bf)
    ln = torch.rand(c_s, generator=g).to(dev, bf) + 0.5
    if gated:
        params = [ln, w(c, c_s), w(c), w(c, c_s), w(n * c, c), w(n * c, c), w(c, c_s), w(c), w(c, n * c)]
        run = lambda a, out: pkg.lib.cond_transition_forward(a, s, mask, out, params, n, residual)  # noqa: E731
    else:
        params = [w(c), w(c), w(n * c, c), w(n * c, c), w(c, n * c)]
        run = lambda a, out: pkg.lib.transition_forward(a, mask, out, params, n, residual)  # noqa: E731
    outs = []
    for offset in (0, 2, 16):
        a = _at(x, offset)
        out = a if residual else _at(torch.full_like(x, 7.0), offset)
        run(a, out)
        outs.append(out.clone())
    pkg.lib.check_device_status()
    assert torch.isfinite(outs[0]).all() and outs[0].any()
    assert torch.equal(outs[0], outs[1]) and torch.equal(outs[0], outs[2])


def _diffusion_block(g):
    blk = pkg.DiffusionTransformerBlock(c_a=768, c_s=384, c_z=128, c_hidden=48, no_heads=16, n_transition=2,
                                        use_ada_layer_norm=True, n_query=None, n_key=None, inf=1e9)
    with torch.no_grad():
        for p in blk.parameters():
            p.copy_(torch.randn(p.shape, generator=g) * (0.03 if p.dim() > 1 else 0.3) + (1.0 if p.dim() == 1 else 0.0))
    return blk.to("cuda:0", torch.bfloat16).eval().requires_grad_(False)


# Tiles of 16, 32 and 64 tokens, one and several of them, per sample and over the rows of all samples; key blocks that end inside,
# at and before a tile's end; 370: the last sizes that one wave of 64-token tiles takes (three launches, then two, then one)
@pytest.mark.parametrize("N,samples", [(1, 1), (1, 3), (15, 1), (16, 1), (17, 2), (31, 1), (32, 1), (33, 3), (48, 1), (64, 1), (65, 1),
                                       (75, 5), (96, 1), (111, 1), (129, 1), (185, 2), (192, 1), (193, 1), (370, 1), (384, 1),
                                       (385, 1), (768, 1), (769, 1)])
def test_few_tokens_equal_rows_of_a_larger_call(N, samples):
    """The launches for few tokens against the 128-row ones, which the same samples take in a call of many: the same products in the
    same order, so the same bits."""
    g = torch.Generator().manual_seed(N)
    blk = _diffusion_block(g)
    many = max(samples + 1, -(-800 // N))
    many += many % 2
    if N < 32:
        many = 60   # more samples than one wave of tiles
    a, s = (torch.randn(1, many, N, c, generator=g).to("cuda:0", torch.bfloat16) for c in (768, 384))
    z = torch.randn(1, 1, N, N, 128, generator=g).to("cuda:0", torch.bfloat16)
    m = (torch.rand(1, 1, N, generator=g) < 0.9).to("cuda:0", torch.bfloat16)
    m[..., 0] = 1
    with torch.no_grad():
        want = blk(a, s, z, mask=m)[:, :samples]
        got = blk(a[:, :samples].contiguous(), s[:, :samples].contiguous(), z, mask=m)
    pkg.lib.check_device_status()
    assert torch.isfinite(got).all() and got.any() and torch.equal(got, want)


# 12 column tiles of 256 (queries to gates; the hidden channels) times 14, 25, 30, 31 and 40 row tiles on 148 SMs: a last wave of 20
# tiles, of 4, of 64 and of 36, in halves, and one of 76, whole; the last row tile full and in part
@pytest.mark.parametrize("N,samples", [(350, 5), (1050, 3), (768, 5), (987, 4), (1024, 5)])
def test_halves_of_the_last_wave_equal_whole_tiles(N, samples):
    """A step whose last wave of wide tiles is half empty, its tiles in two, against every sample by itself."""
    g = torch.Generator().manual_seed(N)
    blk = _diffusion_block(g)
    a, s = (torch.randn(1, samples, N, c, generator=g).to("cuda:0", torch.bfloat16) for c in (768, 384))
    z = torch.randn(1, 1, N, N, 128, generator=g).to("cuda:0", torch.bfloat16)
    m = (torch.rand(1, 1, N, generator=g) < 0.9).to("cuda:0", torch.bfloat16)
    m[..., 0] = 1
    with torch.no_grad():
        got = blk(a, s, z, mask=m)
        want = torch.cat([blk(a[:, i:i + 1].contiguous(), s[:, i:i + 1].contiguous(), z, mask=m) for i in range(samples)], 1)
    pkg.lib.check_device_status()
    assert torch.isfinite(got).all() and got.any() and torch.equal(got, want)


@pytest.mark.parametrize("N,samples", [(1, 2), (7, 1), (16, 1), (33, 2), (64, 1), (100, 1), (129, 2), (500, 1), (768, 1)])
def test_few_tokens_of_the_single_track(N, samples):
    """The same for the attention of the trunk's single track (16 heads of 24, whose images pad k to 32)."""
    g = torch.Generator().manual_seed(N)
    layer = pkg.AttentionPairBias(c_q=384, c_k=384, c_v=384, c_s=None, c_z=128, c_hidden=24, no_heads=16)
    with torch.no_grad():
        for p in layer.parameters():
            p.copy_(torch.randn(p.shape, generator=g) * (0.05 if p.dim() > 1 else 0.3) + (1.0 if p.dim() == 1 else 0.0))
    layer = layer.to("cuda:0", torch.bfloat16).eval().requires_grad_(False)
    many = max(samples + 1, -(-1700 // N)) if N > 12 else 200   # more tiles than one wave takes
    a = torch.randn(many, N, 384, generator=g).to("cuda:0", torch.bfloat16)
    z = torch.randn(samples, N, N, 128, generator=g).to("cuda:0", torch.bfloat16)
    z = torch.cat([z, z[:1].expand(many - samples, -1, -1, -1)])
    m = (torch.rand(many, N, generator=g) < 0.9).to("cuda:0", torch.bfloat16)
    m[:, 0] = 1
    with torch.no_grad():
        want = layer(a, z, mask=m)[:samples]
        got = layer(a[:samples].contiguous(), z[:samples].contiguous(), mask=m[:samples].contiguous())
    pkg.lib.check_device_status()
    assert torch.isfinite(got).all() and got.any() and torch.equal(got, want)


# more rows than one wave of 64-token tiles takes in any of the products: 768 of 768 channels, 1536 of 384
@pytest.mark.parametrize("N,samples", [(1, 1), (1, 3), (7, 1), (15, 1), (16, 1), (17, 2), (31, 1)])
@pytest.mark.parametrize("track", ["diffusion", "single"])
def test_fewest_tokens_equal_rows_of_a_large_call(N, samples, track):
    """The smallest calls, all of whose products are launches for few tokens, against a call that has none of these."""
    g = torch.Generator().manual_seed(N + samples)
    many = (801 if track == "diffusion" else 1601) // N + 1
    c = 768 if track == "diffusion" else 384
    a, s = (torch.randn(many, N, k, generator=g).to("cuda:0", torch.bfloat16) for k in (c, 384))
    z = torch.randn(1, N, N, 128, generator=g).to("cuda:0", torch.bfloat16)
    m = (torch.rand(1, N, generator=g) < 0.9).to("cuda:0", torch.bfloat16)
    m[:, 0] = 1
    if track == "diffusion":
        blk = _diffusion_block(g)
        run = lambda k: blk(a[None, :k].contiguous(), s[None, :k].contiguous(), z[None], mask=m[None])[0]  # noqa: E731
    else:
        layer = pkg.AttentionPairBias(c_q=c, c_k=c, c_v=c, c_s=None, c_z=128, c_hidden=24, no_heads=16)
        up = pkg.SwiGLUTransition(c_in=c, n=4)
        with torch.no_grad():
            for p in (*layer.parameters(), *up.parameters()):
                p.copy_(torch.randn(p.shape, generator=g) * (0.05 if p.dim() > 1 else 0.3) + (1.0 if p.dim() == 1 else 0.0))
        layer, up = (x.to("cuda:0", torch.bfloat16).eval().requires_grad_(False) for x in (layer, up))

        def run(k):
            zk, mk = z.expand(k, -1, -1, -1).contiguous(), m.expand(k, -1).contiguous()
            x = a[:k] + layer(a[:k].contiguous(), zk, mask=mk)
            return x + up(x, mask=mk)
    with torch.no_grad():
        want, got = run(many)[:samples], run(samples)
    pkg.lib.check_device_status()
    assert torch.isfinite(got).all() and got.any() and torch.equal(got, want)
