"""fp32 products on the tensor cores (as products of bf16 parts): ragged rows, columns and k, vectors that do not start on 16 bytes,
both orders of the triangle contraction, against fp64; and values that the parts cannot hold. An fp32 operand is the sum of its
parts, six of the nine products are kept (the others are below 2^-26 of the value), and sums are cut off at most every 64 products:
below 2^-22 of the RMS for two layers in a row."""

import pytest
import torch
import torch.nn.functional as F

from cases import oracle, pkg, rms_err

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")


def _params(c, n, g):
    w = lambda *shape: (torch.randn(shape, generator=g) * shape[-1] ** -0.5).to(DEV)  # noqa: E731
    return [w(c) + 1, w(c), w(n * c, c), w(n * c, c), w(c, n * c)]


def _reference(x, mask, p):
    y = F.layer_norm(x, (x.shape[-1],), p[0], p[1], 1e-5)
    return x + mask[:, None] * ((F.silu(y @ p[2].T) * (y @ p[3].T)) @ p[4].T)


# k of whole k-blocks, of whole vectors and odd; two k-blocks at most and more of the second product
@pytest.mark.parametrize("rows,c,n", [(20001, 128, 4), (9000, 64, 2), (12345, 36, 4), (16385, 37, 3), (7000, 200, 1), (5000, 256, 4)])
@pytest.mark.parametrize("offset", [0, 1])
def test_transition(rows, c, n, offset):
    g = torch.Generator().manual_seed(rows)
    p = _params(c, n, g)
    x = torch.randn(rows * c + 1, generator=g).to(DEV)[offset:offset + rows * c].view(rows, c)
    mask = torch.rand(rows, generator=g).to(DEV)
    out = x.clone() if offset == 0 else torch.empty(rows * c + 1, device=DEV)[1:].view(rows, c).copy_(x)
    pkg.lib.transition_forward(out, mask, out, p, n, True)
    pkg.lib.check_device_status()
    want = _reference(x.double(), mask.double(), [t.double() for t in p])
    assert rms_err(out, want) < 2.0 ** -22, rms_err(out, want)


@pytest.mark.parametrize("N,c", [(33, 128), (67, 96), (100, 128), (129, 64), (130, 40)])
@pytest.mark.parametrize("outgoing", [True, False])
def test_triangle_update(N, c, outgoing):
    g = torch.Generator().manual_seed(N)
    cls = pkg.TriangleMultiplicationOutgoing if outgoing else pkg.TriangleMultiplicationIncoming
    layer = cls(c, c)
    with torch.no_grad():
        for q in layer.parameters():
            q.copy_(torch.randn(q.shape, generator=g) * (q.shape[-1] ** -0.5 if q.dim() > 1 else 0.1) + (1.0 if q.dim() == 1 else 0.0))
    layer = layer.to(DEV).eval().requires_grad_(False)
    z = torch.randn(1, N, N, c, generator=g).to(DEV)
    mask = (torch.rand(1, N, N, generator=g) < 0.9).float().to(DEV)
    got = layer(z, mask=mask)
    pkg.lib.check_device_status()
    P = {k: v.double() for k, v in layer.named_parameters()}
    want = oracle.triangle_multiplicative_update(z.double(), mask.double(), P, "", outgoing)
    assert rms_err(got, want) < 2.0 ** -22, rms_err(got, want)


def test_values_that_bf16_parts_cannot_hold():
    """A row of infinities, a NaN, infinite and very large weights: what the FMA pipe gives, there and nowhere else."""
    rows, c, n = 20000, 128, 4
    g = torch.Generator().manual_seed(3)
    p = _params(c, n, g)
    x = torch.randn(rows, c, generator=g).to(DEV)
    mask = torch.ones(rows, device=DEV)
    x[300, 5], x[7000, 1] = float("inf"), float("nan")
    plain = x.clone()
    pkg.lib.transition_forward(plain, mask, plain, p, n, True)
    want = _reference(x.double(), mask.double(), [t.double() for t in p])
    bad = torch.zeros(rows, dtype=torch.bool, device=DEV)
    bad[300] = bad[7000] = True
    assert not torch.isfinite(plain[bad]).any() and rms_err(plain[~bad], want[~bad]) < 2.0 ** -22
    p[4][7, 11], p[4][90, 3], p[4][91, 3] = float("inf"), 3.4e38, -3.4e38
    x[300, 5], x[7000, 1] = 0.0, 0.0
    got = x.clone()
    pkg.lib.transition_forward(got, mask, got, p, n, True)
    pkg.lib.check_device_status()
    want = _reference(x.double(), mask.double(), [t.double() for t in p])
    cols = torch.ones(c, dtype=torch.bool, device=DEV)
    cols[7] = cols[90] = cols[91] = False
    assert torch.isinf(got[:, 7]).all() and torch.equal(got[:, 7] > 0, want[:, 7] > 0)
    assert rms_err(got[:, cols], want[:, cols]) < 2.0 ** -22
    for k in (90, 91):
        fits = want[:, k].abs() < 3.3e38
        # the hidden value's error: 2^-20 of the two sums it is made of (RMS 1), and of itself
        rms = want[fits, k].pow(2).mean().sqrt()
        assert fits.any() and ((got[:, k].double() - want[:, k]).abs()[fits] <= 2.0 ** -20 * (3 * rms + want[fits, k].abs())).all()
        assert torch.isinf(got[:, k][want[:, k].abs() > 3.5e38]).all()


# k of one k-block (whole, ragged) and of several; gate / up of 128 channels, the final product of 64 and 72, and both in each call
@pytest.mark.parametrize("c,n", [(64, 1), (36, 2), (128, 4)])
def test_special_values_in_every_tile(c, n):
    """An infinity or a NaN in every 128 rows, many tiles per block: only its own row is not finite. The others are sums in order on the
    FMA pipe: k roundings of at most 2^-24 of sums that grow to the last one, sqrt(k / 6) 2^-24 RMS, 9.2 x 2^-24 at k = 512, and as
    much again at most from the layer before and the residual."""
    rows = 45000
    g = torch.Generator().manual_seed(c)
    p = _params(c, n, g)
    x = torch.randn(rows, c, generator=g).to(DEV)
    bad = torch.zeros(rows, dtype=torch.bool, device=DEV)
    bad[torch.arange(5, rows, 128)] = True
    want = _reference(x.double(), torch.ones(rows, dtype=torch.double, device=DEV), [t.double() for t in p])
    x[bad, 3] = float("inf")
    x[133::256, 3] = float("nan")
    out = x.clone()
    pkg.lib.transition_forward(out, torch.ones(rows, device=DEV), out, p, n, True)
    pkg.lib.check_device_status()
    assert not torch.isfinite(out[bad]).any() and rms_err(out[~bad], want[~bad]) < 2.0 ** -20


# one k-block, ragged and whole, two of them, and many
@pytest.mark.parametrize("c,n", [(36, 1), (32, 2), (64, 2), (128, 4)])
def test_products_beyond_the_range(c, n):
    """Operands that bf16 parts hold, products that fp32 does not: infinities of their sign, and nothing else changes."""
    rows = 20001
    g = torch.Generator().manual_seed(c)
    p = _params(c, n, g)
    p[3] *= 2.0 ** 24
    p[4][7] = 0
    p[4][7, 11] = 1.003e38
    x = torch.randn(rows, c, generator=g).to(DEV)
    mask = torch.ones(rows, device=DEV)
    out = x.clone()
    pkg.lib.transition_forward(out, mask, out, p, n, True)
    pkg.lib.check_device_status()
    want = _reference(x.double(), mask.double(), [t.double() for t in p])
    beyond = want[:, 7].abs() > 3.5e38
    assert beyond.sum() > rows // 2 and torch.isinf(out[beyond, 7]).all()
    assert torch.equal(out[beyond, 7] > 0, want[beyond, 7] > 0)
    cols = torch.arange(c, device=DEV) != 7
    assert torch.isfinite(out[:, cols]).all() and rms_err(out[:, cols], want[:, cols]) < 2.0 ** -20   # (redone ones: see above)


# hidden values below and beside the parts' reach (2^-110) against weights that bring the sums back, at both ends of what the parts'
# products take; products whose parts are denormal; one k-block, ragged and whole, two of them, and many
@pytest.mark.parametrize("up,out", [(2.0 ** -118, 1.0), (2.0 ** -118, 2.0 ** 50), (2.0 ** -118, 2.0 ** 100), (2.0 ** -112, 2.0 ** 50),
                                    (2.0 ** -60, 2.0 ** -62), (2.0 ** -40, 2.0 ** -80), (2.0 ** -49, 2.0 ** -49)])
@pytest.mark.parametrize("c,n", [(36, 1), (32, 2), (64, 2), (128, 4)])
@pytest.mark.parametrize("mixed", [False, True])
def test_small_operands(up, out, c, n, mixed):
    """Products of small values are as good as those of ordinary ones, alone and beside them (mixed: half of the hidden channels are
    ordinary, and half of the output's columns are without them). As sums in order on the FMA pipe at most: see above."""
    rows = 20001
    g = torch.Generator().manual_seed(c)
    p = _params(c, n, g)
    half, rest = n * c // 2, c // 2
    p[3][:half if mixed else n * c] *= up
    p[4] *= out
    if mixed:
        p[4][:rest, half:] = 0
    x = torch.randn(rows, c, generator=g).to(DEV)
    mask = torch.ones(rows, device=DEV)
    got = torch.empty_like(x)
    pkg.lib.transition_forward(x, mask, got, p, n, False)
    pkg.lib.check_device_status()
    q = [t.double() for t in p]
    y = F.layer_norm(x.double(), (c,), q[0], q[1], 1e-5)
    want = (F.silu(y @ q[2].T) * (y @ q[3].T)) @ q[4].T
    for cols in ((slice(0, rest), slice(rest, c)) if mixed else (slice(0, c),)):
        y, w = got[:, cols].double(), want[:, cols]
        keep = 2.0 ** -149 / w.pow(2).mean().sqrt()   # (what fp32 itself does not hold)
        assert rms_err(y, w) < 2.0 ** -20 + keep, (rms_err(y, w), keep)
