"""The output projections of the single track, whose gate, residual and result pass through shared memory where the caller's
tensors start on 16 bytes, against the same call on tensors that do not (every thread then reads and writes rows of its own): the
same products, gates and sums in the same order, so the same bits. Rows: part of a tile, its edges, several tiles per block."""

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
