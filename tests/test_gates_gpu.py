"""Gates of the single attention far outside the usual range: sigmoid(-100) is below the smallest float, and the update behind
such a gate is exactly zero; sigmoid(100) is one."""

import pytest
import torch

from cases import pkg

pytestmark = pytest.mark.gpu
N = 37


def _layer(ada: bool):
    """AttentionPairBias with 16 heads of 24 (plain) or 48 (adaptive), its adaptive inputs and attention gates zero."""
    c, d = (768, 48) if ada else (384, 24)
    layer = pkg.AttentionPairBias(c_q=c, c_k=c, c_v=c, c_s=384, c_z=128, c_hidden=d, no_heads=16, use_ada_layer_norm=ada)
    g = torch.Generator().manual_seed(5)
    with torch.no_grad():
        for p in layer.parameters():
            p.copy_(torch.randn(p.shape, generator=g) if p.dim() > 1 else torch.zeros(p.shape))
        layer.layer_norm_z.weight.fill_(1.0)
        layer.mha.linear_g.weight.zero_()
        if ada:
            layer.layer_norm_a.layer_norm_s.weight.fill_(1.0)
            layer.layer_norm_a.linear_g.weight.zero_()
            layer.layer_norm_a.linear_s.weight.zero_()
            layer.linear_ada_out.weight.zero_()
        else:
            layer.layer_norm_a.weight.fill_(1.0)
    return layer.to("cuda:0", torch.bfloat16).eval().requires_grad_(False)


def _inputs(ada: bool):
    g = torch.Generator().manual_seed(6)
    a = torch.randint(0, 2, (1, 3, N, 768 if ada else 384), generator=g) * 2.0 - 1.0
    a[..., 0] = 1.0   # normalised: within 0.8 .. 1.2
    z = torch.randn(1, 1 if ada else 3, N, N, 128, generator=g)
    s = torch.randn(1, 3, N, 384, generator=g) if ada else None
    return [None if t is None else t.to("cuda:0", torch.bfloat16) for t in (a, z, s)]


def _run(layer, a, z, s):
    with torch.no_grad():
        out = layer(a, z, s=s)
    pkg.lib.check_device_status()
    assert torch.isfinite(out).all()
    return out


@pytest.mark.parametrize("ada", [False, True])
def test_closed_and_open_attention_gates(ada):
    x, layer = _inputs(ada), _layer(ada)
    if ada:
        layer.layer_norm_a.linear_g.bias.fill_(100.0)
    half = _run(layer, *x)                                # gates of sigmoid(0)
    layer.mha.linear_g.weight[:, 0] = 128.0
    assert half.abs().max() > 0.1 and torch.equal(_run(layer, *x), 2 * half)
    layer.mha.linear_g.weight[:, 0] = -128.0
    assert not _run(layer, *x).any()


def test_closed_adaptive_gates():
    """sigmoid(-100) * LN(a) + 0: queries, keys and values are zeros, and so is the update."""
    x, layer = _inputs(True), _layer(True)
    layer.layer_norm_a.linear_g.bias.fill_(-100.0)
    assert not _run(layer, *x).any()
    layer.layer_norm_a.linear_g.bias.fill_(-3.0)
    assert _run(layer, *x).any()


def test_closed_and_open_output_gates():
    """The output projection's gate: one where open; closed, it leaves at most 1.6e-38 of the update."""
    x, layer = _inputs(True), _layer(True)
    layer.layer_norm_a.linear_g.bias.fill_(100.0)
    half = _run(layer, *x)
    layer.linear_ada_out.bias.fill_(100.0)
    assert half.any() and torch.equal(_run(layer, *x), 2 * half)
    layer.linear_ada_out.bias.fill_(-100.0)
    assert (_run(layer, *x).double().abs() <= 4e-38 * half.double().abs()).all()
