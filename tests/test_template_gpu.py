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


@pytest.mark.parametrize("c,N", [(128, 320), (64, 300)])
def test_numerator_and_denominator_of_the_softmax_round_alike(c, N):
    """Values near one and rows that few keys dominate, the largest logit as a rule not in the first key block, so that the
    probabilities of the dominant keys are rounded (2^-9): summed before that rounding, the row sum no longer cancels it. All
    else of the layer is made exact (gate 1/2, output projection the identity, no bias), so the error against a double softmax
    of the kernel's own bf16 operands is the final rounding of o and nothing more: 1.00 times it with matched sums, 1.13 with a
    row sum of unrounded probabilities (both simulated in double)."""
    dev, bf, H = torch.device("cuda:0"), torch.bfloat16, 4
    g = torch.Generator().manual_seed(c)
    wq, wk, wv = (torch.randn(c, c, generator=g) * (k * c ** -0.5) for k in (3.0, 1.0, 0.01))
    wq[:, 0] = wk[:, 0] = 0
    wv[:, 0] = 0.97
    att = pkg.TriangleAttention(c, c // H, H)
    with torch.no_grad():
        att.layer_norm.weight[0], att.layer_norm.bias[0] = 0, 1   # channel 0 of the normalised rows is one
        for lin, w in ((att.mha.linear_q, wq), (att.mha.linear_k, wk), (att.mha.linear_v, wv), (att.mha.linear_o, torch.eye(c)),
                       (att.mha.linear_g, torch.zeros(c, c)), (att.linear_z, torch.zeros(H, c))):
            lin.weight.copy_(w)
    att = att.to(dev, bf).eval().requires_grad_(False)
    z = torch.randn(N, N, c, generator=g).to(dev, bf)
    with torch.no_grad():
        got = 2 * att(z[None])[0, :4].double()
    pkg.lib.check_device_status()
    ln = torch.nn.functional.layer_norm(z[:4].float(), (c,)).to(bf).float()
    ln[..., 0] = 1
    q, k, v = (torch.nn.functional.linear(ln.double(), w.to(dev, bf).double()).float() for w in (wq, wk, wv))
    q = (q * (1.4426950408889634 / (c // H) ** 0.5)).to(bf)
    q, k, v = (t.to(bf).double().view(4, N, H, c // H) for t in (q, k, v))
    p = torch.softmax(torch.einsum("bqhd,bkhd->bhqk", q, k) * 0.6931471805599453, -1)
    exact = torch.einsum("bhqk,bkhd->bqhd", p, v).reshape(4, N, c)
    rounding = (exact.to(bf).double() - exact).norm()
    assert ((got - exact).norm() / rounding).item() < 1.04


@pytest.mark.parametrize("kind", ["template", "f32"])
def test_tensors_that_start_anywhere(kind):
    """A pair tensor one element into its buffer, in place and not: what a kernel cannot read where it lies is copied first.
    Same bits as for an aligned one."""
    dev, N = torch.device("cuda:0"), 20
    dt = torch.bfloat16 if kind == "template" else torch.float32
    dims = TEMPLATE if kind == "template" else PAIR
    g = torch.Generator().manual_seed(3)
    single = dict(c_s=384, c_hidden_pair_bias=24, no_heads_pair_bias=16)
    blk = pkg.PairBlock(**dims, **_PF_KW) if kind == "template" else pkg.PairFormerBlock(**dims, **single, **_PF_KW)
    with torch.no_grad():
        for p in blk.parameters():
            p.copy_(torch.randn(p.shape, generator=g) * (0.5 * p.shape[-1] ** -0.5 if p.dim() > 1 else 0.3))
    blk = blk.to(dev, dt).eval().requires_grad_(False)
    z, s = torch.randn(1, N, N, dims["c_z"], generator=g).to(dev, dt), torch.randn(1, N, 384, generator=g).to(dev, dt)
    pair = blk if kind == "template" else blk.pair_stack
    call = (lambda z, **k: (blk(z, None, **k),)) if kind == "template" else (lambda z, **k: blk(s.clone(), z, None, None, **k))
    layers = (pair.tri_mul_in, pair.tri_att_start, pair.tri_att_end, pair.pair_transition)

    def odd():
        buf = torch.empty(z.numel() + 1, dtype=dt, device=dev)
        return buf[1:].view(z.shape).copy_(z)

    with torch.no_grad():
        want, each = call(z.clone()), [m(z) for m in layers]
        inside = odd()
        assert inside.data_ptr() % 16
        got = call(inside, inplace_safe=True)
        assert got[-1].data_ptr() == inside.data_ptr()
        for x in (got, call(odd())):
            assert all(torch.equal(a, b) for a, b in zip(x, want))
        assert all(torch.equal(m(odd()), w) for m, w in zip(layers, each))
    pkg.lib.check_device_status()


@pytest.mark.parametrize("c,B,N", [(128, 1, 1), (128, 2, 37), (64, 2, 64), (128, 1, 65), (64, 1, 129), (128, 1, 200)])
def test_ending_node_is_the_starting_node_of_the_transposed_tensor(c, B, N):
    """The ending-node layer reads z and the mask in place, the mask through rows that its projection kernel writes: the same
    bits as the starting-node layer on transposed copies, with masks that are not symmetric and without one."""
    dev, bf = torch.device("cuda:0"), torch.bfloat16
    g = torch.Generator().manual_seed(N)
    end, start = (pkg.TriangleAttention(c, c // 4, 4, starting=s) for s in (False, True))
    with torch.no_grad():
        for p, q in zip(end.parameters(), start.parameters()):
            p.copy_(torch.randn(p.shape, generator=g) * (p.shape[-1] ** -0.5 if p.dim() > 1 else 0.3))
            q.copy_(p)
    end, start = (m.to(dev, bf).eval().requires_grad_(False) for m in (end, start))
    z = torch.randn(B, N, N, c, generator=g).to(dev, bf)
    m = rand_mask((B, N, N), g, 0.8).to(dev, bf)
    with torch.no_grad():
        for mask in (m, None):
            want = start(z.transpose(1, 2).contiguous(), mask=None if mask is None else mask.transpose(1, 2).contiguous())
            assert torch.equal(end(z, mask=mask), want.transpose(1, 2))
    pkg.lib.check_device_status()


def test_the_ending_node_in_a_workspace_of_the_starting_nodes_size(monkeypatch):
    """No room for mask rows: the mask is read in place, the same bits; without a mask there is nothing to make room for."""
    dev, bf = torch.device("cuda:0"), torch.bfloat16
    g = torch.Generator().manual_seed(3)
    layer = pkg.TriangleAttention(128, 32, 4, starting=False).to(dev, bf).eval().requires_grad_(False)
    for p in layer.parameters():
        p.copy_(torch.randn(p.shape, generator=g) * (p.shape[-1] ** -0.5 if p.dim() > 1 else 0.3))
    z, m = torch.randn(2, 70, 70, 128, generator=g).to(dev, bf), rand_mask((2, 70, 70), g, 0.8).to(dev, bf)
    want = [layer(z, mask=mask) for mask in (m, None)]
    size = pkg.lib.load().of3_triattn_workspace_bytes(2, 70, 128, 4, 32, 0, 0)
    monkeypatch.setattr(pkg.lib, "workspace", lambda nbytes, device, stream=None: torch.empty(size, dtype=torch.uint8, device=device))
    for mask, w in zip((m, None), want):
        assert torch.equal(layer(z, mask=mask), w)
    pkg.lib.check_device_status()
