"""The attention core of the single track with one and with two samples per block, bit for bit: samples that share a pair tensor,
together and one by one. Lines (samples x 16 heads x query tiles of 128) on 148 SMs: one per SM at most, two, three (the last that take
one line per block), more of an even and an odd number, two pair tensors, and keys that end inside a block. And calls of several
threads at once, whose launches ask for different shares of an SM."""

import threading

import pytest
import torch

from cases import pkg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,samples,pairs", [(1, 2, 1), (31, 9, 1), (64, 10, 1), (130, 3, 2), (129, 9, 1), (250, 13, 1), (128, 28, 1),
                                             (385, 5, 2), (100, 29, 1), (33, 31, 2), (640, 5, 1), (513, 6, 1), (768, 5, 1)])
def test_samples_together_equal_one_by_one(N, samples, pairs):
    g = torch.Generator().manual_seed(N + samples)
    blk = pkg.DiffusionTransformerBlock(c_a=768, c_s=384, c_z=128, c_hidden=48, no_heads=16, n_transition=2,
                                        use_ada_layer_norm=True, n_query=None, n_key=None, inf=1e9)
    with torch.no_grad():
        for p in blk.parameters():
            p.copy_(torch.randn(p.shape, generator=g) * (0.03 if p.dim() > 1 else 0.3) + (1.0 if p.dim() == 1 else 0.0))
    blk = blk.to("cuda:0", torch.bfloat16).eval().requires_grad_(False)
    a, s = (torch.randn(pairs, samples, N, c, generator=g).to("cuda:0", torch.bfloat16) for c in (768, 384))
    z = torch.randn(pairs, 1, N, N, 128, generator=g).to("cuda:0", torch.bfloat16)
    m = (torch.rand(pairs, 1, N, generator=g) < 0.9).to("cuda:0", torch.bfloat16)
    m[..., 0] = 1
    with torch.no_grad():
        got = blk(a, s, z, mask=m)
        for k in range(pairs):
            for i in (0, 1, samples // 2, samples - 1):
                want = blk(a[k:k + 1, i:i + 1].contiguous(), s[k:k + 1, i:i + 1].contiguous(), z[k:k + 1], mask=m[k:k + 1])
                assert torch.equal(got[k, i], want[0, 0]), (k, i)
    pkg.lib.check_device_status()
    assert torch.isfinite(got).all() and got.any()


def test_threads_whose_launches_differ():
    """One line per SM at most in one thread, two in the other: 114 and 76 KB of shared memory per block, of one kernel. Stacks, whose
    calls launch it time and again without Python in between."""
    g = torch.Generator().manual_seed(1)
    N = 200
    stack = pkg.DiffusionTransformer(c_a=768, c_s=384, c_z=128, c_hidden=48, no_heads=16, no_blocks=24, n_transition=2,
                                     use_ada_layer_norm=True, n_query=None, n_key=None, inf=1e9, blocks_per_ckpt=None)
    with torch.no_grad():
        for p in stack.parameters():
            p.copy_(torch.randn(p.shape, generator=g) * (0.03 if p.dim() > 1 else 0.3) + (1.0 if p.dim() == 1 else 0.0))
    stack = stack.to("cuda:0", torch.bfloat16).eval().requires_grad_(False)
    z = torch.randn(1, 1, N, N, 128, generator=g).to("cuda:0", torch.bfloat16)
    m = torch.ones(1, 1, N, dtype=torch.bfloat16, device="cuda:0")
    inputs = [[torch.randn(1, samples, N, c, generator=g).to("cuda:0", torch.bfloat16) for c in (768, 384)] for samples in (1, 5)]
    with torch.no_grad():
        want = [stack(a, s, z, mask=m) for a, s in inputs]
    torch.cuda.synchronize()
    start, got, errors = threading.Barrier(2), [None, None], []

    def work(k):
        try:
            with torch.no_grad(), torch.cuda.stream(torch.cuda.Stream()):
                for _ in range(60):
                    start.wait(60)
                    got[k] = stack(*inputs[k], z, mask=m)
                    torch.cuda.current_stream().synchronize()
        except Exception as e:  # noqa: BLE001
            errors.append(e)
            start.abort()

    threads = [threading.Thread(target=work, args=(k,)) for k in (0, 1)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    pkg.lib.check_device_status()
    assert not errors, errors
    assert all(torch.equal(x, y) for x, y in zip(got, want))
