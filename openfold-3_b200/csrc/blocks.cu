// Whole blocks of the Pairformer, and the whole diffusion token stack, behind one C call each: the same layers in the
// same order as the module entry points of api.cu, issued by native code. A pair block is 13 launches and the single
// track of a block 8 more; from Python, one layer call at a time, a block cost about 400 us of host time (the 4-block trunk
// at N = 37 took 1.6 ms for 0.3 ms of device work, and so did N = 256).
#include "fast_pairbias.cuh"
#include "fast_single.cuh"
#include "generic_ops.cuh"
#include "modules.cuh"
#include "runtime.cuh"

#include <vector>

using namespace of3;

namespace {

// Layers of one stack call share the workspace: each starts at its beginning.
struct Scratch {
    void* base;
    size_t cap;
    size_t need = 0;
    template <typename F>
    int run(F&& f) {
        Arena ws(base, cap);
        const int rc = f(ws);
        if (ws.off > need) need = ws.off;
        return rc;
    }
};

int pair_block(void* z, const void* mask, const of3_block_dims& D, int dtype, int flags, const of3_pair_block_params* p,
               Scratch& ws, cudaStream_t st) {
    const int f = (flags & OF3_FLAG_FORCE_GENERIC) | OF3_FLAG_ADD_RESIDUAL;
    int rc;
    if ((rc = ws.run([&](Arena& a) {
             return trimul_dispatch(z, mask, z, D.B, D.N, D.c_z, D.c_hidden_mul, dtype, f | OF3_FLAG_OUTGOING,
                                    &p->tri_mul_out, a, st);
         })))
        return rc;
    if ((rc = ws.run([&](Arena& a) {
             return trimul_dispatch(z, mask, z, D.B, D.N, D.c_z, D.c_hidden_mul, dtype, f, &p->tri_mul_in, a, st);
         })))
        return rc;
    if ((rc = ws.run([&](Arena& a) {
             return triattn_dispatch(z, mask, z, D.B, D.N, D.c_z, D.no_heads_pair, D.c_hidden_pair_att, D.inf_pair, dtype,
                                     f, &p->tri_att_start, a, st);
         })))
        return rc;
    if ((rc = ws.run([&](Arena& a) {
             return triattn_dispatch(z, mask, z, D.B, D.N, D.c_z, D.no_heads_pair, D.c_hidden_pair_att, D.inf_pair, dtype,
                                     f | OF3_FLAG_TRANSPOSED, &p->tri_att_end, a, st);
         })))
        return rc;
    return ws.run([&](Arena& a) {
        return transition_dispatch(z, (flags & OF3_FLAG_NO_TRANSITION_MASK) ? nullptr : mask, z,
                                   (long long)D.B * D.N * D.N, D.c_z, D.pair_transition_n, dtype, f, &p->pair_transition, a,
                                   st);
    });
}

// How the single track gets its pair bias: projected ahead of it (bf16 bias tiles of the tensor-core attention, or an
// fp32 tensor), or by the attention layer itself.
enum BiasForm { kBiasInLayer, kBiasTiles, kBiasF32 };
BiasForm bias_form(const of3_block_dims& D, int dtype, int flags) {
    if (D.c_z != 128 || D.no_heads_single != 16 || (flags & OF3_FLAG_FORCE_GENERIC)) return kBiasInLayer;
    if (dtype == OF3_DTYPE_BF16)
        return fast::attn_pair_bias_supported(D.B, D.B, D.N, D.c_s, 0, D.c_z, D.no_heads_single, D.c_hidden_single, flags)
                   ? kBiasTiles
                   : kBiasInLayer;
    return kBiasF32;
}
// Rooms for the projected bias in a block's workspace. With one, every block's projection waits for the single track of the block
// ahead, which ended long before; but a wait for another stream takes the place of the chain between two kernels (N = 256: 5.9 instead
// of 1.1 us). Trunk, one room / four, us: 4 blocks of 128 474 / 460, 256 1229 / 1217, 384 2428 / 2407, 12 of 256 3562 / 3475, 8 of 320
// 3764 / 3748, 448 7326 / 7248, 512 8960 / 8856. Where a room is larger (16 N^2 values: 8 MB at 512) one: 640 15033 / 15041, 768 23017 /
// 23062, and three more would be 57 MB at 768, 0.4 GB at 2048.
constexpr int kBiasSlots = 4;
constexpr size_t kBiasSlotMost = 8 << 20;
size_t bias_bytes(const of3_block_dims& D, BiasForm f) {
    if (f == kBiasTiles) return (size_t)D.B * of3_pair_bias_tiles_elems(D.N) * sizeof(__nv_bfloat16);
    return f == kBiasF32 ? (size_t)D.B * D.no_heads_single * D.N * D.N * sizeof(float) : 0;
}
size_t rooms_bytes(size_t one) { return (one <= kBiasSlotMost ? kBiasSlots : 1) * align_up(one, 256); }

int project_bias(const void* z, void* bias, const of3_block_dims& D, BiasForm form, const of3_attn_pair_bias_params* p,
                 cudaStream_t st) {
    if (form == kBiasTiles)
        return fast::pair_bias_tiles_c128_h16((const __nv_bfloat16*)z, (const __nv_bfloat16*)p->ln_z_w,
                                              (const __nv_bfloat16*)p->ln_z_b, (const __nv_bfloat16*)p->w_z,
                                              (__nv_bfloat16*)bias, D.B, D.N, st);
    return generic::pair_bias_c128_h16<float>((const float*)z, (const float*)p->ln_z_w, (const float*)p->ln_z_b,
                                              (const float*)p->w_z, (float*)bias, D.B, (long long)D.N * D.N, st);
}

int single_track(void* s, const void* z, const void* bias, BiasForm form, const void* mask, const of3_block_dims& D,
                 int dtype, int flags, const of3_pairformer_block_params* p, Scratch& ws, cudaStream_t st) {
    const int f = (flags & (OF3_FLAG_FORCE_GENERIC | fast::kFlagBeside)) | OF3_FLAG_ADD_RESIDUAL;
    int rc = ws.run([&](Arena& a) {
        if (form == kBiasTiles)
            return fast::attn_pair_bias((const __nv_bfloat16*)s, nullptr, nullptr, (const __nv_bfloat16*)mask,
                                        (__nv_bfloat16*)s, D.B, D.B, D.N, D.c_s, 0, D.no_heads_single, D.c_hidden_single,
                                        D.inf_single, f, &p->attn, a, st, nullptr, (const __nv_bfloat16*)bias);
        if (form == kBiasF32)
            return generic::attn_pair_bias<float>((const float*)s, nullptr, nullptr, (const float*)mask, (float*)s, D.B,
                                                  D.B, D.N, D.c_s, 0, D.c_z, D.no_heads_single, D.c_hidden_single,
                                                  D.inf_single, f, &p->attn, a, st, (const float*)bias);
        return apb_dispatch(s, z, nullptr, mask, s, D.B, D.B, D.N, D.c_s, 0, D.c_z, D.no_heads_single, D.c_hidden_single,
                            D.inf_single, dtype, f, &p->attn, a, st);
    });
    if (rc) return rc;
    return ws.run([&](Arena& a) {
        return transition_dispatch(s, (flags & OF3_FLAG_NO_TRANSITION_MASK) ? nullptr : mask, s, (long long)D.B * D.N,
                                   D.c_s, D.single_transition_n, dtype, f, &p->single_transition, a, st);
    });
}

// ---------------------------------------------------------------- diffusion token stack
// Room for the conditioning projections of one group of blocks. s is the same for all blocks, so a launch can cover
// several of them: with few rows the projections of one block (6 matrices of c_a x c_s) fill a fraction of the chip and
// cost a launch each; with many rows one block fills it, and its planes should stay in L2 until they are read.
constexpr size_t kCondGroupBytes = 32u << 20;
// Room for the normalised rows of the conditioning ahead of those projections: one launch for several groups of blocks, of
// which each alone waits for the kernel ahead and for its own start (5 x 768 tokens: 24 launches of 5.1 us -> 5 of 13.8, 5 x 500:
// 24 of 5.1 -> 3 of 20.2).
constexpr size_t kCondRowsBytes = 32u << 20;
// Room for the bias images of the blocks whose pair bias one pass over z projects (24 blocks up to N = 1150): 24 x 18.9 MB
// of the workspace at N = 768, for 225 us instead of 24 passes of 56.
constexpr size_t kBiasGroupBytes = 1u << 30;

int diffusion_stack(void* a, const void* s, const void* z, const void* mask, const void* const* bias,
                    const of3_diffusion_dims& D, int dtype, int flags, int blocks, const of3_attn_pair_bias_params* pa,
                    const of3_cond_transition_params* pt, Scratch& ws, cudaStream_t st) {
    typedef __nv_bfloat16 bf16;
    const int f = (flags & (OF3_FLAG_FORCE_GENERIC | OF3_FLAG_ADA_LN)) | OF3_FLAG_ADD_RESIDUAL;
    const long long rows = (long long)D.Ba * D.N;
    const void* tmask = (flags & OF3_FLAG_NO_TRANSITION_MASK) ? nullptr : mask;
    const bool fast_attn = dtype == OF3_DTYPE_BF16 &&
                           fast::attn_pair_bias_supported(D.Ba, D.Bz, D.N, D.c_a, D.c_s, D.c_z, D.H, D.d, f);
    const bool fast_trans = dtype == OF3_DTYPE_BF16 && fast::cond_transition_supported(D.c_a, D.c_s, D.n, f);
    int rc;
    if (!(fast_attn && fast_trans && (flags & OF3_FLAG_ADA_LN))) {
        for (int b = 0; b < blocks; ++b) {
            rc = ws.run([&](Arena& A) {
                if (bias != nullptr && fast_attn)
                    return fast::attn_pair_bias((const bf16*)a, nullptr, (const bf16*)s, (const bf16*)mask, (bf16*)a, D.Ba,
                                                D.Bz, D.N, D.c_a, D.c_s, D.H, D.d, D.inf, f, pa + b, A, st, nullptr,
                                                (const bf16*)bias[b]);
                if (bias != nullptr && dtype == OF3_DTYPE_F32)
                    return generic::attn_pair_bias<float>((const float*)a, nullptr, (const float*)s, (const float*)mask,
                                                          (float*)a, D.Ba, D.Bz, D.N, D.c_a, D.c_s, D.c_z, D.H, D.d,
                                                          D.inf, f, pa + b, A, st, (const float*)bias[b]);
                if (bias != nullptr)
                    return generic::attn_pair_bias<bf16>((const bf16*)a, nullptr, (const bf16*)s, (const bf16*)mask,
                                                         (bf16*)a, D.Ba, D.Bz, D.N, D.c_a, D.c_s, D.c_z, D.H, D.d, D.inf,
                                                         f, pa + b, A, st, (const float*)bias[b]);
                return apb_dispatch(a, z, s, mask, a, D.Ba, D.Bz, D.N, D.c_a, D.c_s, D.c_z, D.H, D.d, D.inf, dtype, f,
                                    pa + b, A, st);
            });
            if (rc) return rc;
            rc = ws.run([&](Arena& A) {
                return cond_dispatch(a, s, tmask, a, rows, D.c_a, D.c_s, D.n, dtype, f & ~OF3_FLAG_ADA_LN, pt + b, A, st);
            });
            if (rc) return rc;
        }
        return OF3_OK;
    }
    // pair biases projected in the call: several blocks per pass over z, as many as fit kBiasGroupBytes
    const size_t per_bias = (size_t)D.Bz * of3_pair_bias_tiles_elems(D.N) * sizeof(bf16);
    int nbias = 0;
    if (bias == nullptr) {
        const size_t fit = kBiasGroupBytes / per_bias;
        nbias = fit < 1 ? 1 : (fit > (size_t)fast::kMaxBiasLayers ? fast::kMaxBiasLayers : (int)fit);
        if (nbias > blocks) nbias = blocks;
    }
    const size_t per_block = (size_t)rows * 6 * D.c_a * sizeof(bf16);
    int group = per_block ? (int)(kCondGroupBytes / per_block) : 1;
    if (group < 1) group = 1;
    if (group > blocks) group = blocks;
    if (group > fast::kMaxCondBatch / 2) group = fast::kMaxCondBatch / 2;
    int rows_group = (int)(kCondRowsBytes / ((size_t)rows * 2 * D.c_s * sizeof(bf16)));   // blocks per launch of the rows
    if (rows_group > fast::kMaxCondBatch / 2) rows_group = fast::kMaxCondBatch / 2;
    if (rows_group > blocks) rows_group = blocks;
    rows_group = rows_group < group ? group : rows_group / group * group;
    auto run = [&](Arena& A, int rows_group) -> int {
        bf16* planes = (bf16*)A.take(group * per_block);
        bf16* sn = (bf16*)A.take((size_t)(2 * rows_group + 1) * rows * D.c_s * sizeof(bf16));
        bf16* tiles = nbias ? (bf16*)A.take(nbias * per_bias) : nullptr;
        const size_t mark = A.off;
        size_t need = A.off;
        for (int b0 = 0; b0 < blocks; b0 += group) {
            const int nb = blocks - b0 < group ? blocks - b0 : group;
            if (A.base) {
                OF3_REQUIRE(A.ok(), OF3_ERR_WORKSPACE, "diffusion stack: workspace too small (%zu needed)", A.off);
                const int r0 = b0 / rows_group * rows_group, nr = blocks - r0 < rows_group ? blocks - r0 : rows_group;
                fast::CondLayer layer[fast::kMaxCondBatch];   // of the blocks [r0, r0 + nr)
                for (int i = 0; i < nr; ++i) {
                    layer[2 * i] = fast::cond_layer(pa + r0 + i);
                    layer[2 * i + 1] = fast::cond_layer(pt + r0 + i);
                }
                int rc = b0 == r0 ? fast::conditioning_rows((const bf16*)s, layer, 2 * nr, rows, D.c_s, sn, st) : OF3_OK;
                if (rc == OF3_OK)
                    rc = fast::conditioning_planes(sn, 2 * (b0 - r0), 2 * nr, layer + 2 * (b0 - r0), 2 * nb, rows, D.c_a, D.c_s,
                                                   planes, st);
                if (rc) return rc;
            }
            for (int i = 0; i < nb; ++i) {
                const int b = b0 + i;
                const bf16* cond = planes ? planes + (size_t)i * 6 * rows * D.c_a : (const bf16*)256;
                A.off = mark;
                const bf16* bt = bias ? (const bf16*)bias[b] : (const bf16*)256;
                if (bias == nullptr && A.base) {
                    if (b % nbias == 0) {
                        const int n = blocks - b < nbias ? blocks - b : nbias;
                        fast::BiasLayer bl[fast::kMaxBiasLayers];
                        for (int l = 0; l < n; ++l)
                            bl[l] = {(const bf16*)pa[b + l].ln_z_w, (const bf16*)pa[b + l].ln_z_b, (const bf16*)pa[b + l].w_z};
                        const int brc = fast::pair_bias_tiles((const bf16*)z, bl, n, tiles, D.Bz, D.N, st);
                        if (brc) return brc;
                    }
                    bt = tiles + (size_t)(b % nbias) * (per_bias / sizeof(bf16));
                }
                int rc = fast::attn_pair_bias((const bf16*)a, (const bf16*)z, (const bf16*)s, (const bf16*)mask, (bf16*)a,
                                              D.Ba, D.Bz, D.N, D.c_a, D.c_s, D.H, D.d, D.inf, f, pa + b, A, st, nullptr,
                                              bt, cond);
                if (rc) return rc;
                need = A.off > need ? A.off : need;
                A.off = mark;
                rc = fast::cond_transition((const bf16*)a, (const bf16*)s, (const bf16*)tmask, (bf16*)a, rows, D.c_a, D.c_s,
                                           D.n, f, pt + b, A, st, planes ? cond + 3 * rows * D.c_a : cond);
                if (rc) return rc;
                need = A.off > need ? A.off : need;
                if (!A.base) break;   // sizing: the blocks are alike
            }
            if (!A.base) break;
        }
        A.off = need;
        return OF3_OK;
    };
    return ws.run([&](Arena& A) -> int {
        if (!A.base) return run(A, rows_group);
        // A workspace without room for more takes the rows of one group at a time: a caller's buffer may be of the size that was
        // asked for before rows were shared. (The sizing of one block: under 1 us of a call's host time.)
        Arena whole(nullptr, 0);
        const int rc = run(whole, rows_group);
        return rc ? rc : run(A, whole.off <= A.cap ? rows_group : group);
    });
}

bool diffusion_dims_ok(const of3_diffusion_dims* d) {
    return d && d->Ba > 0 && d->Bz > 0 && d->Ba % d->Bz == 0 && d->N > 0 && d->c_a > 0 && d->c_s > 0 && d->c_z > 0 &&
           d->H > 0 && d->d > 0 && d->n > 0;
}

bool dims_ok(const of3_block_dims* d) {
    return d && d->B > 0 && d->N > 0 && d->c_z > 0 && d->c_hidden_mul > 0 && d->no_heads_pair > 0 &&
           d->c_hidden_pair_att > 0 && d->pair_transition_n > 0;
}
bool single_dims_ok(const of3_block_dims* d) {
    return d->c_s > 0 && d->no_heads_single > 0 && d->c_hidden_single > 0 && d->single_transition_n > 0;
}
bool complete_block(const of3_pair_block_params& p) {
    return complete(p.tri_mul_out) && complete(p.tri_mul_in) && complete(p.tri_att_start) && complete(p.tri_att_end) &&
           complete(p.pair_transition);
}
#define CHECK_BLOCK(what)                                                                                        \
    OF3_REQUIRE(dtype == OF3_DTYPE_BF16 || dtype == OF3_DTYPE_F32, OF3_ERR_ARG, what ": bad dtype %d", dtype);    \
    OF3_REQUIRE(dims_ok(dims), OF3_ERR_ARG, what ": non-positive size")

}  // namespace

extern "C" {

int of3_stream_wait(void* waiter, void* signaler) {
    return stream_wait((cudaStream_t)waiter, (cudaStream_t)signaler);
}

size_t of3_pair_block_workspace_bytes(const of3_block_dims* dims, int dtype, int flags) {
    if (!dims_ok(dims)) return 0;
    of3_pair_block_params p = {};
    Scratch ws{nullptr, 0};
    if (pair_block(nullptr, nullptr, *dims, dtype, flags, &p, ws, nullptr)) return 0;
    return ws.need + 256;
}

int of3_pair_block_forward(void* z, const void* pair_mask, const of3_block_dims* dims, int dtype, int flags,
                           const of3_pair_block_params* p, void* workspace, size_t workspace_bytes, void* stream) {
    CHECK_BLOCK("pair_block");
    OF3_REQUIRE(z && p && workspace, OF3_ERR_ARG, "pair_block: null pointer argument");
    OF3_REQUIRE(complete_block(*p), OF3_ERR_ARG, "pair_block: null parameter pointer");
    CallScope call((flags & OF3_FLAG_CONTINUES) != 0);
    Scratch ws{workspace, workspace_bytes};
    return pair_block(z, pair_mask, *dims, dtype, flags, p, ws, (cudaStream_t)stream);
}

// side = 0: the main stream's workspace: the largest layer, then the projected pair bias, which outlives the next
// block's layers; side = 1: the single track's.
size_t of3_pairformer_block_workspace_bytes(const of3_block_dims* dims, int dtype, int flags, int side) {
    if (!dims_ok(dims) || !single_dims_ok(dims)) return 0;
    of3_pairformer_block_params p = {};
    Scratch ws{nullptr, 0};
    const BiasForm form = bias_form(*dims, dtype, flags);
    if (side) {
        // a bias pointer that is never read: the projected form takes no room here
        if (single_track(nullptr, nullptr, form == kBiasTiles ? (const void*)256 : nullptr, form, nullptr, *dims, dtype, flags, &p, ws, nullptr)) return 0;
        return ws.need + 256;
    }
    if (pair_block(nullptr, nullptr, *dims, dtype, flags, &p.pair, ws, nullptr)) return 0;
    return align_up(ws.need, 256) + rooms_bytes(bias_bytes(*dims, form)) + 256;
}

int of3_pairformer_block_forward(void* s, void* z, const void* single_mask, const void* pair_mask,
                                 const of3_block_dims* dims, int dtype, int flags, const of3_pairformer_block_params* p,
                                 void* workspace, size_t workspace_bytes, void* side_workspace,
                                 size_t side_workspace_bytes, void* stream, void* side_stream) {
    CHECK_BLOCK("pairformer_block");
    OF3_REQUIRE(single_dims_ok(dims), OF3_ERR_ARG, "pairformer_block: non-positive single-track size");
    OF3_REQUIRE(s && z && p && workspace && side_workspace, OF3_ERR_ARG, "pairformer_block: null pointer argument");
    OF3_REQUIRE(complete_block(p->pair) && complete(p->attn, false, true) && complete(p->single_transition), OF3_ERR_ARG,
                "pairformer_block: null parameter pointer");
    cudaStream_t main = (cudaStream_t)stream;
    const BiasForm form = bias_form(*dims, dtype, flags);
    const size_t one = bias_bytes(*dims, form);
    const Arena whole(workspace, workspace_bytes);   // its start aligned
    OF3_REQUIRE(whole.cap >= one, OF3_ERR_WORKSPACE, "pairformer_block: workspace too small");
    // all rooms, where the layers have theirs beside them (a buffer may be of the size that was asked for when there was one)
    Scratch sizing{nullptr, 0};
    int slot = side_stream != nullptr ? (flags >> 8) & (kBiasSlots - 1) : 0;
    size_t tail = one;
    if (form != kBiasInLayer && one <= kBiasSlotMost &&
        pair_block(nullptr, nullptr, *dims, dtype, flags, &p->pair, sizing, nullptr) == OF3_OK &&
        whole.cap >= align_up(sizing.need, 256) + rooms_bytes(one))
        tail = rooms_bytes(one);
    else
        slot = 0;
    const size_t head = (whole.cap - tail) / 256 * 256;
    void* bias = whole.base + head + slot * align_up(one, 256);
    Scratch ws{whole.base, head}, ws_side{side_workspace, side_workspace_bytes};
    CallScope call((flags & OF3_FLAG_CONTINUES) != 0);
    int rc;
    if ((rc = pair_block(z, pair_mask, *dims, dtype, flags, &p->pair, ws, main))) return rc;
    if (form == kBiasInLayer || side_stream == nullptr) {
        if (form != kBiasInLayer && (rc = project_bias(z, bias, *dims, form, &p->attn, main))) return rc;
        return single_track(s, z, bias, form, single_mask, *dims, dtype, flags, p, ws_side, main);
    }
    // The pair stack never reads s, so the single track (a chain of small, launch-bound kernels) runs on the side
    // stream under the next block's pair stack. What it needs of z, the pair bias, is projected here, before the next
    // block overwrites z, into a room of its own, or into the first: behind the single tracks that read it.
    cudaStream_t side = (cudaStream_t)side_stream;
    if (slot == 0 && (rc = stream_wait(main, side))) return rc;
    if ((rc = project_bias(z, bias, *dims, form, &p->attn, main))) return rc;
    if ((rc = stream_wait(side, main))) return rc;
    const int beside = (flags & OF3_FLAG_LAST) ? 0 : fast::kFlagBeside;
    return single_track(s, nullptr, bias, form, single_mask, *dims, dtype, flags | beside, p, ws_side, side);
}

size_t of3_diffusion_stack_workspace_bytes(const of3_diffusion_dims* dims, int dtype, int flags, int blocks,
                                           int with_bias) {
    if (!diffusion_dims_ok(dims) || blocks <= 0) return 0;
    Scratch ws{nullptr, 0};
    const std::vector<of3_attn_pair_bias_params> pas(blocks, of3_attn_pair_bias_params{});
    const std::vector<of3_cond_transition_params> pts(blocks, of3_cond_transition_params{});
    const std::vector<const void*> bias(blocks, (const void*)256);   // never read: says that the bias takes no room here
    if (diffusion_stack(nullptr, nullptr, nullptr, nullptr, with_bias ? bias.data() : nullptr, *dims, dtype, flags, blocks,
                        pas.data(), pts.data(), ws, nullptr))
        return 0;
    return ws.need + 256;
}

int of3_diffusion_stack_forward(void* a, const void* s, const void* z, const void* mask, const void* const* bias,
                                const of3_diffusion_dims* dims, int dtype, int flags, int blocks,
                                const of3_attn_pair_bias_params* attn, const of3_cond_transition_params* transition,
                                void* workspace, size_t workspace_bytes, void* stream) {
    OF3_REQUIRE(dtype == OF3_DTYPE_BF16 || dtype == OF3_DTYPE_F32, OF3_ERR_ARG, "diffusion_stack: bad dtype %d", dtype);
    OF3_REQUIRE(diffusion_dims_ok(dims) && blocks > 0, OF3_ERR_ARG, "diffusion_stack: bad sizes");
    OF3_REQUIRE(a && s && (z || bias) && attn && transition && workspace, OF3_ERR_ARG,
                "diffusion_stack: null pointer argument");
    for (int b = 0; b < blocks; ++b)
        OF3_REQUIRE(complete(attn[b], (flags & OF3_FLAG_ADA_LN) != 0, bias == nullptr) && complete(transition[b]) &&
                        (bias == nullptr || bias[b] != nullptr),
                    OF3_ERR_ARG, "diffusion_stack: null parameter pointer (block %d)", b);
    CallScope call;
    Scratch ws{workspace, workspace_bytes};
    return diffusion_stack(a, s, z, mask, bias, *dims, dtype, flags, blocks, attn, transition, ws, (cudaStream_t)stream);
}

}  // extern "C"
