"""The C-ABI library: builds for sm_100a, loads without a GPU, exports every symbol the public
header declares, and rejects bad arguments with error codes instead of crashing."""

import ctypes
import re
from pathlib import Path

import pytest
import torch

ROOT = Path(__file__).resolve().parent.parent


def declared_symbols():
    text = (ROOT / "include" / "of3b200.h").read_text()
    text = re.sub(r"/\*.*?\*/", "", text, flags=re.S)
    return sorted(set(re.findall(r"\b(of3_[a-z0-9_]+)\s*\(", text)))


def test_header_declares_entry_points():
    syms = declared_symbols()
    assert "of3_trimul_forward" in syms and "of3_triattn_forward" in syms and len(syms) >= 15


def test_library_exports_every_declared_symbol(pkg):
    lib = pkg.lib.load()
    for name in declared_symbols():
        assert hasattr(lib, name), f"{name} declared in include/of3b200.h but not exported"
    assert set(pkg.lib.SIGNATURES) == set(declared_symbols())


def test_bad_arguments_return_error_codes(pkg):
    lib = pkg.lib.load()
    p = pkg.lib.TrimulParams()
    rc = lib.of3_trimul_forward(None, None, None, 1, 8, 128, 128, 0, 0, ctypes.byref(p), None, 0, None)
    assert rc == -1 and b"null" in lib.of3_last_error_string()
    rc = lib.of3_trimul_forward(None, None, None, 1, 8, 128, 128, 7, 0, ctypes.byref(p), None, 0, None)
    assert rc == -1 and b"dtype" in lib.of3_last_error_string()
    t = pkg.lib.TransitionParams()
    assert lib.of3_transition_forward(None, None, None, 4, 128, 4, 1, 0, ctypes.byref(t), None, 0, None) == -1


def test_workspace_queries_need_no_gpu(pkg):
    lib = pkg.lib.load()
    for dt in (0, 1):
        assert lib.of3_trimul_workspace_bytes(1, 64, 128, 128, dt, 0) > 0
        assert lib.of3_triattn_workspace_bytes(1, 64, 128, 4, 32, dt, 0) > 0
        assert lib.of3_transition_workspace_bytes(4096, 128, 4, dt, 0) > 0
        assert lib.of3_attn_pair_bias_workspace_bytes(2, 1, 64, 384, 0, 128, 16, 24, dt, 0) > 0
        assert lib.of3_cond_transition_workspace_bytes(128, 768, 384, 2, dt, 0) > 0


@pytest.mark.parametrize("B,N,c", [(1, 1, 128), (2, 37, 64), (1, 2048, 128)])
def test_only_the_ending_node_asks_for_mask_rows(pkg, B, N, c):
    """Operand images, output and bias tiles are what both nodes need; a row of the mask per line, in whole blocks of 64 keys,
    the ending node's alone. (Each array starts on 256 bytes, and so does the first.)"""
    up = lambda x, to: (x + to - 1) // to * to  # noqa: E731
    start, end = (pkg.lib.load().of3_triattn_workspace_bytes(B, N, c, 4, c // 4, 0, flags)
                  for flags in (0, pkg.lib.FLAG_TRANSPOSED))
    images = 3 * B * up(N, 4) * up(N, 128) * c * 2
    rest = up(B * N * N * c * 2, 256) + B * 4 * up(N, 32) * N * 2
    assert start <= images + rest + 256
    assert up(start, 256) + B * N * up(N, 64) * 2 == end


@pytest.mark.parametrize("dt,bytes_per,N,rooms", [(0, 2, 512, 4), (0, 2, 544, 1), (0, 2, 768, 1), (0, 2, 2048, 1),
                                                  (1, 4, 362, 4), (1, 4, 363, 1), (1, 4, 1024, 1)])
def test_rooms_for_the_pair_bias_in_a_workspace(pkg, dt, bytes_per, N, rooms):
    """Beside the layers' own: four of 16 N^2 values up to 8 MB each, one above."""
    lib = pkg.lib
    d = lib.BlockDims(B=1, N=N, c_z=128, c_hidden_mul=128, no_heads_pair=4, c_hidden_pair_att=32, pair_transition_n=4, c_s=384,
                      no_heads_single=16, c_hidden_single=24, single_transition_n=4, inf_pair=1e9, inf_single=1e9)
    pair = lib.load().of3_pair_block_workspace_bytes(ctypes.byref(d), dt, 0)
    both = lib.load().of3_pairformer_block_workspace_bytes(ctypes.byref(d), dt, 0, 0)
    room = 16 * N * N * bytes_per
    assert pair > 0 and 0 <= both - pair - rooms * room < (rooms + 2) * 256


def test_no_cpu_fallback(pkg):
    """CPU tensors are refused: there is no path that avoids the CUDA library."""
    m = pkg.TriangleMultiplicationOutgoing(128, 128).eval()
    with torch.no_grad(), pytest.raises(RuntimeError, match="no CPU path"):
        m(torch.zeros(1, 4, 4, 128))


def test_forward_only(pkg):
    m = pkg.SwiGLUTransition(128, 4)
    with pytest.raises(NotImplementedError):
        m(torch.zeros(1, 4, 128, requires_grad=True))


def test_state_dict_keys_match_reference_layout(pkg):
    P = pkg.weights.pairformer_block_params(1)
    blk = pkg.PairFormerBlock(c_s=384, c_z=128, c_hidden_pair_bias=24, no_heads_pair_bias=16,
                              c_hidden_mul=128, c_hidden_pair_att=32, no_heads_pair=4,
                              transition_type="swiglu", transition_n=4, pair_dropout=0.25,
                              fuse_projection_weights=False, inf=1e9)
    assert len(P) == 57 and sum(v.numel() for v in P.values()) == 3070848
    blk.load_state_dict(P, strict=True)
    # a freshly constructed block is the identity on (s, z): its zero-initialised matrices
    zeros = [k for k, v in blk.state_dict().items() if v.abs().sum() == 0 and v.dim() == 2]
    assert len(zeros) == 0  # we just loaded random weights
    fresh = pkg.PairFormerBlock(c_s=384, c_z=128, c_hidden_pair_bias=24, no_heads_pair_bias=16,
                                c_hidden_mul=128, c_hidden_pair_att=32, no_heads_pair=4,
                                transition_type="swiglu", transition_n=4, pair_dropout=0.25,
                                fuse_projection_weights=False, inf=1e9)
    zeros = [k for k, v in fresh.state_dict().items() if v.dim() == 2 and v.abs().sum() == 0]
    assert len(zeros) == 16


def test_modules_pack_grouped_weights_back_to_back(pkg):
    """The projections of the conditioning run as one launch when their weights lie back to back in memory (the
    library compares addresses): the modules' parameter packer must lay them out that way, and q | g | k | v and the
    SwiGLU pair too, with unchanged values."""
    dt, dev = torch.bfloat16, torch.device("cpu")
    apb = pkg.AttentionPairBias(c_q=768, c_k=768, c_v=768, c_s=384, c_z=128, c_hidden=48, no_heads=16,
                                use_ada_layer_norm=True, inf=1e9)
    prm = apb._params(dt, dev)
    step = 768 * 768 * 2
    q, g, k, v = prm[11], prm[15], prm[13], prm[14]
    assert [t.data_ptr() - q.data_ptr() for t in (g, k, v)] == [step, 2 * step, 3 * step]
    assert torch.equal(q, apb.mha.linear_q.weight.to(dt)) and torch.equal(v, apb.mha.linear_v.weight.to(dt))
    assert torch.equal(g, apb.mha.linear_g.weight.to(dt)) and torch.equal(k, apb.mha.linear_k.weight.to(dt))
    assert prm[5].data_ptr() - prm[3].data_ptr() == 768 * 384 * 2          # AdaLN linear_g, linear_s
    ctb = pkg.ConditionedTransitionBlock(c_a=768, c_s=384, n=2)
    prm = ctb._params(dt, dev)
    assert prm[3].data_ptr() - prm[1].data_ptr() == 768 * 384 * 2          # AdaLN pair
    assert prm[5].data_ptr() - prm[4].data_ptr() == 2 * 768 * 768 * 2      # SwiGLU linear_a, linear_b
    tr = pkg.SwiGLUTransition(c_in=384, n=4)
    prm = tr._params(dt, dev)
    assert prm[3].data_ptr() - prm[2].data_ptr() == 4 * 384 * 384 * 2
    assert torch.equal(prm[3], tr.swiglu.linear_b.weight.to(dt))


def _filled(struct):
    """A parameter struct of addresses that nobody reads: the calls below are refused before the first launch."""
    s = struct()
    for name, kind in struct._fields_:
        setattr(s, name, 4096 if kind is ctypes.c_void_p else _filled(kind))
    return s


def _pointer_fields(struct, prefix=()):
    for name, kind in struct._fields_:
        if kind is ctypes.c_void_p:
            yield (*prefix, name)
        else:
            yield from _pointer_fields(kind, (*prefix, name))


def test_block_entry_points_refuse_null_parameters(pkg):
    """Every parameter that the kernels read without asking, as the layers' own entry points refuse them."""
    L, lib = pkg.lib, pkg.lib.load()
    dims = L.BlockDims(1, 8, 128, 128, 4, 32, 4, 384, 16, 24, 4, 1e9, 1e9)
    diff = L.DiffusionDims(1, 1, 8, 768, 384, 128, 16, 48, 2, 1e9)
    ref = ctypes.byref
    calls = {
        L.PairBlockParams: lambda p: lib.of3_pair_block_forward(4096, None, ref(dims), 0, 0, ref(p), 4096, 1 << 40, None),
        L.PairformerBlockParams: lambda p: lib.of3_pairformer_block_forward(4096, 4096, None, None, ref(dims), 0, 0, ref(p),
                                                                            4096, 1 << 40, 4096, 1 << 40, None, None),
        L.AttnPairBiasParams: lambda p: lib.of3_diffusion_stack_forward(
            4096, 4096, 4096, None, None, ref(diff), 0, L.FLAG_ADA_LN, 1, ref(p), ref(_filled(L.CondTransitionParams)), 4096,
            1 << 40, None),
        L.CondTransitionParams: lambda p: lib.of3_diffusion_stack_forward(
            4096, 4096, 4096, None, None, ref(diff), 0, L.FLAG_ADA_LN, 1, ref(_filled(L.AttnPairBiasParams)), ref(p), 4096,
            1 << 40, None),
    }
    optional = {"b_q", "ln_z_b"}
    for struct, call in calls.items():
        unused = optional | ({"ln_a_w", "ln_a_b"} if struct is L.AttnPairBiasParams else set())
        for path in _pointer_fields(struct):
            if path[-1] in unused or ("attn" in path and ("ada" in path[-1])):
                continue
            p = _filled(struct)
            owner = p
            for name in path[:-1]:
                owner = getattr(owner, name)
            setattr(owner, path[-1], None)
            assert call(p) == -1 and b"null parameter" in lib.of3_last_error_string(), path
