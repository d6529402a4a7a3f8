// Single-track layers (bf16; c_s = 384 in the trunk, c_a = 768 in the diffusion token stack): attention with pair bias
// (LayerNorm variant, and the conditioned variant with adaptive LayerNorm), the SwiGLU transition for widths without a
// fused row-tile kernel, and the conditioned transition.
//
// The token dimension is tiny next to the pair tensor (N x 384 against N x N x 128), so these are launch/latency-bound
// chains, not roofline kernels: four launches per attention layer (LayerNorm or AdaLN rows; q | k | v | g projection
// written as attention operand images; attention; output projection with gate and residual) and three per transition
// (rows; SwiGLU; output projection with gate, mask and residual), with the linears and their epilogues in linear.cu and
// the attention in fast_single_attn.cu. The conditioned layers add one launch for LN_s(s) and one for the three
// projections of s, which a stack computes for several layers at once (s is the same for all of them).
// Reference: openfold3/core/model/layers/attention_pair_bias.py:123-227,
//            openfold3/core/model/primitives/attention.py:94-135, 270-310,
//            openfold3/core/model/layers/transition.py:225-271, 274-380,
//            openfold3/core/model/primitives/normalization.py:89-140.
#include "fast_single.cuh"
#include "linear.cuh"
#include "modules.cuh"
#include "runtime.cuh"
#include "umma.cuh"

namespace of3 {
namespace fast {
namespace {

using namespace umma;
typedef __nv_bfloat16 bf16;
constexpr int kKidSingle = 8;
constexpr int kKidLinear = 10;  // linear layers, those on the contraction kernel too (accounted apart from the triangle einsum)
constexpr float kEps = 1e-5f;

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// ---------------------------------------------------------------- LayerNorm of rows, one warp per row
// The row stays in registers: NV vectors of 8 values per lane (lane, lane + 32, ...), one 16-byte load each. (Re-reading
// it three times with 2-byte loads took 8 - 20 us for 3840 rows.)
template <int NV>
struct Row {
    float x[NV * 8], mean, rstd;
    __device__ __forceinline__ void load(const bf16* p, int C, int lane) {
#pragma unroll
        for (int v = 0; v < NV; ++v) {
            const int c = (v * 32 + lane) * 8;
            uint32_t u[4] = {0u, 0u, 0u, 0u};
            if (c < C) ld_row8_any(p + c, u);
#pragma unroll
            for (int e = 0; e < 8; ++e) x[v * 8 + e] = (e & 1) ? bf16hi(u[e >> 1]) : bf16lo(u[e >> 1]);
        }
    }
    // x <- (x - mean) * rstd, zero past C
    __device__ __forceinline__ void normalize(int C, int lane) {
        float s = 0.f;
#pragma unroll
        for (int i = 0; i < NV * 8; ++i) s += x[i];
        mean = warp_sum(s) / (float)C;
        float q = 0.f;
#pragma unroll
        for (int v = 0; v < NV; ++v) {
            const bool in = (v * 32 + lane) * 8 < C;
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                const float d = in ? x[v * 8 + e] - mean : 0.f;
                x[v * 8 + e] = d;
                q = fmaf(d, d, q);
            }
        }
        rstd = rsqrtf(warp_sum(q) / (float)C + kEps);
#pragma unroll
        for (int i = 0; i < NV * 8; ++i) x[i] *= rstd;
    }
};
__device__ __forceinline__ void unpack8(const uint32_t (&u)[4], float (&f)[8]) {
#pragma unroll
    for (int e = 0; e < 8; ++e) f[e] = (e & 1) ? bf16hi(u[e >> 1]) : bf16lo(u[e >> 1]);
}
__device__ __forceinline__ uint4 pack8(const float (&f)[8]) {
    return make_uint4(pack_bf16x2(f[0], f[1]), pack_bf16x2(f[2], f[3]), pack_bf16x2(f[4], f[5]), pack_bf16x2(f[6], f[7]));
}

// y = LN(x) * gamma + beta
template <int NV>
__global__ void __launch_bounds__(256) ln_rows_kernel(const bf16* __restrict__ x, const bf16* __restrict__ gamma,
                                                      const bf16* __restrict__ beta, bf16* __restrict__ y,
                                                      long long rows, int C) {
    grid_trigger();
    grid_wait();
    const int lane = threadIdx.x & 31;
    const long long r = (long long)blockIdx.x * 8 + (threadIdx.x >> 5);
    if (r >= rows) return;
    Row<NV> row;
    row.load(x + r * C, C, lane);
    row.normalize(C, lane);
#pragma unroll
    for (int v = 0; v < NV; ++v) {
        const int c = (v * 32 + lane) * 8;
        if (c >= C) continue;
        uint32_t g[4], b[4];
        float gf[8], bf[8], o[8];
        ld_row8_any(gamma + c, g);
        ld_row8_any(beta + c, b);
        unpack8(g, gf);
        unpack8(b, bf);
#pragma unroll
        for (int e = 0; e < 8; ++e) o[e] = fmaf(row.x[v * 8 + e], gf[e], bf[e]);
        *reinterpret_cast<uint4*>(y + r * C + c) = pack8(o);
    }
}

// Conditioning inputs: y[l] = LN_s(s) * w[l] for the layers of one launch, then (by the last y block) s itself as slice
// `layers`, so that one batched GEMM reads both.
constexpr int kMaxCondLayers = 48;
struct CondWeights {
    const bf16* w[kMaxCondLayers];
};
template <int NV>
__global__ void __launch_bounds__(256) cond_rows_kernel(const bf16* __restrict__ s, const CondWeights cw, int layers,
                                                        bf16* __restrict__ y, long long rows, int C) {
    grid_trigger();
    grid_wait();
    const int lane = threadIdx.x & 31;
    const long long r = (long long)blockIdx.x * 8 + (threadIdx.x >> 5);
    if (r >= rows) return;
    Row<NV> row;
    row.load(s + r * C, C, lane);
    if (blockIdx.y == gridDim.y - 1) {
#pragma unroll
        for (int v = 0; v < NV; ++v) {
            const int c = (v * 32 + lane) * 8;
            float o[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) o[e] = row.x[v * 8 + e];
            if (c < C) *reinterpret_cast<uint4*>(y + (layers * rows + r) * C + c) = pack8(o);
        }
    }
    row.normalize(C, lane);
    for (int l = blockIdx.y; l < layers; l += gridDim.y) {
#pragma unroll
        for (int v = 0; v < NV; ++v) {
            const int c = (v * 32 + lane) * 8;
            if (c >= C) continue;
            uint32_t g[4];
            float gf[8], o[8];
            ld_row8_any(cw.w[l] + c, g);
            unpack8(g, gf);
#pragma unroll
            for (int e = 0; e < 8; ++e) o[e] = row.x[v * 8 + e] * gf[e];
            *reinterpret_cast<uint4*>(y + (l * rows + r) * C + c) = pack8(o);
        }
    }
}

// an = sigmoid(g_lin + b_g) * LN(a) + s_lin (normalization.py:121-140)
constexpr int kAdaRows = 4;   // per block
template <int NV>
__global__ void __launch_bounds__(32 * kAdaRows) ada_rows_kernel(const bf16* __restrict__ a, const bf16* __restrict__ g_lin,
                                                                 const bf16* __restrict__ b_g,
                                                                 const bf16* __restrict__ s_lin, bf16* __restrict__ an,
                                                                 long long rows, int C) {
    grid_trigger();
    grid_wait();
    const int lane = threadIdx.x & 31;
    const long long r = (long long)blockIdx.x * kAdaRows + (threadIdx.x >> 5);
    if (r >= rows) return;
    uint32_t g[NV][4], s[NV][4], b[NV][4];   // in flight together with the row
#pragma unroll
    for (int v = 0; v < NV; ++v) {
        const int c = (v * 32 + lane) * 8;
        if (c >= C) continue;
        const uint4 gv = *reinterpret_cast<const uint4*>(g_lin + r * C + c);
        const uint4 sv = *reinterpret_cast<const uint4*>(s_lin + r * C + c);
        g[v][0] = gv.x; g[v][1] = gv.y; g[v][2] = gv.z; g[v][3] = gv.w;
        ld_row8_any(b_g + c, b[v]);
        s[v][0] = sv.x; s[v][1] = sv.y; s[v][2] = sv.z; s[v][3] = sv.w;
    }
    Row<NV> row;
    row.load(a + r * C, C, lane);
    row.normalize(C, lane);
    auto store = [&](int c, const float (&x)[8], const uint32_t (&gv)[4], const uint32_t (&sv)[4], const uint32_t (&bv)[4],
                     auto divide) {
        float gf[8], sf[8], bf[8], o[8];
        unpack8(gv, gf);
        unpack8(sv, sf);
        unpack8(bv, bf);
#pragma unroll
        for (int e = 0; e < 8; ++e) o[e] = divide(x[e], 1.0f + __expf(-(gf[e] + bf[e]))) + sf[e];
        *reinterpret_cast<uint4*>(an + r * C + c) = pack8(o);
    };
    // quotient_of's range: gates above -44 (a normalised value is at most sqrt(C))
    float dmax = 1.0f;
    uint32_t xmin = 0xffffffffu;   // of the bits of |x|, doubled, minus one: zero is in the range
#pragma unroll
    for (int v = 0; v < NV; ++v) {
        const int c = (v * 32 + lane) * 8;
        if (c >= C) continue;
        float x[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) x[e] = row.x[v * 8 + e];
        store(c, x, g[v], s[v], b[v], [&](float xe, float d) {
            dmax = fmaxf(dmax, d);
            xmin = min(xmin, 2u * __float_as_uint(xe) - 1u);
            return quotient_of(xe, d);
        });
    }
    if (dmax <= 0x1p64f && xmin >= 2u * __float_as_uint(0x1p-60f) - 1u) return;
    // A closed gate, as a rule: the lane's values once more, by the division. Behind the loop and as one of its own, since
    // divisions between the vectors above cost a short call 3 us per launch in instructions fetched and never run.
#pragma unroll 1
    for (int c = lane * 8; c < C; c += 256) {
        uint32_t av[4], gv[4], sv[4], bv[4];
        ld_row8_any(a + r * C + c, av);
        ld_row8_any(g_lin + r * C + c, gv);
        ld_row8_any(s_lin + r * C + c, sv);
        ld_row8_any(b_g + c, bv);
        float x[8];
        unpack8(av, x);
#pragma unroll
        for (int e = 0; e < 8; ++e) x[e] = (x[e] - row.mean) * row.rstd;
        store(c, x, gv, sv, bv, [](float xe, float d) { return xe / d; });
    }
}

#define BY_WIDTH(C, CALL)                                   \
    do {                                                    \
        if ((C) <= 256) { constexpr int NV = 1; CALL; }     \
        else if ((C) <= 512) { constexpr int NV = 2; CALL; } \
        else if ((C) <= 768) { constexpr int NV = 3; CALL; } \
        else if ((C) <= 1024) { constexpr int NV = 4; CALL; } \
        else { constexpr int NV = 8; CALL; }                \
    } while (0)
constexpr int kMaxRowWidth = 2048;   // eight vectors per lane

unsigned row_blocks(long long rows) { return (unsigned)((rows + 7) / 8); }

int ln_rows(const bf16* x, const bf16* gamma, const bf16* beta, bf16* y, long long rows, int C, cudaStream_t st) {
    LaunchScope scope(kKidSingle, st);
    BY_WIDTH(C, OF3_CUDA_CHECK(launch_chained(ln_rows_kernel<NV>, row_blocks(rows), 256, 0, st, x, gamma, beta, y, rows, C)));
    return OF3_OK;
}
// How many blocks of the AdaLN rows an SM may hold: as many as spread them evenly over the SMs, by a request for shared memory
// that the kernel does not use. The blocks start while the kernel ahead drains, and without a limit they gather on the SMs that
// it has left first, where each then waits for the others' loads; the next kernel, one block per SM, starts behind the fullest.
// (Alone, unchained, the kernel takes the same time with and without.) Step of 24 blocks in a graph, c_a = 768, us, without a
// limit / at most 1 / 2 / 3 / 4 blocks per SM, medians whose runs differ by up to 0.3 %:
//   rows  111   867 /  911 /  866 /  860 /  873      rows 1184  1685 / 1720 / 1648 / 1655 / 1674
//         150   938 /  915 /  927 /  940 /  928           1300  1764 / 1846 / 1772 / 1738 / 1752
//         250   954 /  951 /  958 /  956 /  957           1500  1561 / 1657 / 1584 / 1533 / 1551
//         450  1152 / 1054 / 1064 / 1154 / 1160           1775  1859 / 1981 / 1890 / 1851 / 1851
//         592  1233 / 1223 / 1228 / 1239 / 1247           1900  1886 / 2061 / 1927 / 1916 / 1882
//         700  1281 / 1311 / 1261 / 1283 / 1291           2200  1970 / 2156 / 2025 / 2020 / 1977
//         900  1517 / 1528 / 1470 / 1480 / 1504           2750  2295 / 2580 / 2417 / 2370 / 2362
// c_a = 384: 450 rows 820 / - / 819 / 824 / 838, 1000 1176 / - / 1138 / 1141 / 1154, 1500 1113 / - / 1127 / 1083 / 1090, 2000
// 1307 / - / 1308 / 1304 / 1262, 3840 1954 / - / 2078 / 2016 / 1981. With fewer than two rows per SM a limit of one lost 5 % at
// 111 rows and gained 2 % at 150: two. Past four blocks per SM they fill the chip anyway: no limit.
int ada_blocks_per_sm(long long rows) {
    const long long sms = sm_count(), per_sm = (rows + kAdaRows * sms - 1) / (kAdaRows * sms);
    return rows < 2 * sms ? 2 : (per_sm <= 4 ? (int)per_sm : 0);
}
template <int NV>
int ada_rows_width(const bf16* a, const bf16* planes, const bf16* b_g, bf16* an, long long rows, int C, cudaStream_t st) {
    constexpr int kSmBytes = 228 << 10, kReserved = 1 << 10;   // shared memory of an SM; of it, the system's per block
    const int limit = ada_blocks_per_sm(rows);
    static PerDeviceOnce configured;
    if (!configured.done()) {
        OF3_CUDA_CHECK(cudaFuncSetAttribute(ada_rows_kernel<NV>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                            kSmBytes - kReserved));
        configured.mark();
    }
    OF3_CUDA_CHECK(launch_chained(ada_rows_kernel<NV>, (unsigned)((rows + kAdaRows - 1) / kAdaRows), 32 * kAdaRows,
                                  limit ? kSmBytes / limit - kReserved : 0, st, a, planes, b_g, planes + rows * C, an, rows,
                                  C));
    return OF3_OK;
}
int ada_rows(const bf16* a, const bf16* planes, const bf16* b_g, bf16* an, long long rows, int C, cudaStream_t st) {
    LaunchScope scope(kKidSingle, st);
    BY_WIDTH(C, return ada_rows_width<NV>(a, planes, b_g, an, rows, C, st));
}
// y = x w^T on the contraction kernel
int linear_bf16(const bf16* x, const bf16* w, bf16* y, long long rows, int out_dim, int in_dim, cudaStream_t st) {
    return contract_nt_bf16(x, w, y, 1, (int)rows, out_dim, in_dim, in_dim, in_dim, out_dim, rows * in_dim,
                            (long long)out_dim * in_dim, rows * out_dim, st, 0, 0, kKidLinear);
}

bool aligned16(const void* p) { return ((uintptr_t)p & 15) == 0; }
// Launches for few tokens fill the chip with short blocks. Beside a pair stack (kFlagBeside) each of these makes a block of it late,
// while a pair stack of few tokens leaves SMs idle. Trunk of four blocks, us, 128-row tiles in all blocks / in all but the last / in
// none: N = 24 408 / - / 399, 37 411 / - / 406, 64 417 / - / 409, 80 442 / 436 / 449, 96 450 / 444 / 458, 128 473 / 467 / 485.
bool alone(long long rows, int flags) { return !(flags & kFlagBeside) || rows <= kBesideRows; }
bool even(const void* p) { return ((uintptr_t)p & 3) == 0; }   // pairs of channels

}  // namespace

int conditioning_rows(const bf16* s, const CondLayer* layer, int layers, long long rows, int c_s, bf16* sn,
                      cudaStream_t st) {
    OF3_REQUIRE(layers >= 1 && layers <= kMaxCondLayers, OF3_ERR_ARG, "conditioning: %d layers", layers);
    CondWeights cw = {};
    for (int l = 0; l < layers; ++l) cw.w[l] = layer[l].ln_s_w;
    // few rows: the layers are spread over blocks too
    const unsigned gx = row_blocks(rows);
    const unsigned want = 2u * (unsigned)sm_count();
    unsigned gy = gx >= want ? 1u : want / gx + 1;
    if (gy > (unsigned)layers) gy = layers;
    LaunchScope scope(kKidSingle, st);
    BY_WIDTH(c_s, OF3_CUDA_CHECK(launch_chained(cond_rows_kernel<NV>, dim3(gx, gy), 256, 0, st, s, cw, layers, sn, rows,
                                                c_s)));
    return OF3_OK;
}

int conditioning_planes(const bf16* sn, int first, int raw_slice, const CondLayer* layer, int layers, long long rows,
                        int c_a, int c_s, bf16* planes, cudaStream_t st) {
    const bf16* x0 = sn + first * rows * c_s;
    const int raw_rel = raw_slice - first;
    const long long wsz = (long long)c_a * c_s, plane = rows * c_a;
    auto grouped = [&](int l) {   // the layer's own three matrices
        return layer[l].w_s == layer[l].w_g + wsz && layer[l].w_out == layer[l].w_g + 2 * wsz && aligned16(layer[l].w_g);
    };
    bool all = true;
    for (int l = 0; l < layers; ++l) all = all && grouped(l) && layer[l].w_g == layer[0].w_g + 3 * l * wsz;
    if (all) return linear_conditioning(x0, rows, c_s, c_a, layer[0].w_g, layers, raw_rel + 1, raw_rel, planes, st);
    for (int l = 0; l < layers; ++l) {
        const bf16 *x = x0 + l * rows * c_s, *raw = x0 + raw_rel * rows * c_s;
        bf16* y = planes + 3 * l * plane;
        int rc;
        if ((rc = linear_bf16(x, layer[l].w_g, y, rows, c_a, c_s, st))) return rc;
        if ((rc = linear_bf16(x, layer[l].w_s, y + plane, rows, c_a, c_s, st))) return rc;
        if ((rc = linear_bf16(raw, layer[l].w_out, y + 2 * plane, rows, c_a, c_s, st))) return rc;
    }
    return OF3_OK;
}

int conditioning(const bf16* s, const CondLayer* layer, int layers, long long rows, int c_a, int c_s, bf16* sn,
                 bf16* planes, cudaStream_t st) {
    const int rc = conditioning_rows(s, layer, layers, rows, c_s, sn, st);
    return rc ? rc : conditioning_planes(sn, 0, layers, layer, layers, rows, c_a, c_s, planes, st);
}

// bf16, one pair tensor per group of samples; c_a = H * d a multiple of 64; d in {24, 48}.
bool attn_pair_bias_supported(int Ba, int Bz, int N, int c_a, int c_s, int c_z, int H, int d, int flags) {
    if (flags & OF3_FLAG_FORCE_GENERIC) return false;
    if ((flags & OF3_FLAG_ADA_LN) && (c_s <= 0 || c_s % 64 != 0 || c_s > kMaxRowWidth)) return false;
    if (!(d == 24 || d == 48) || H * d != c_a || c_a % 64 != 0) return false;
    if (c_z != 128 || H != 16 || Bz <= 0 || Ba % Bz != 0) return false;
    return single_attn_tc_supported(N, H, d);
}

int attn_pair_bias(const bf16* a, const bf16* z, const bf16* s, const bf16* mask, bf16* out, int Ba, int Bz, int N,
                   int c_a, int c_s, int H, int d, float inf, int flags, const of3_attn_pair_bias_params* p, Arena& ws,
                   cudaStream_t st, const float* pair_bias, const bf16* bias_tiles, const bf16* cond) {
    const long long rows = (long long)Ba * N;
    const bool ada = (flags & OF3_FLAG_ADA_LN) != 0;
    bf16* an = (bf16*)ws.take(rows * c_a * sizeof(bf16));
    bf16* g = (bf16*)ws.take(rows * c_a * sizeof(bf16));
    bf16* og = an;   // the normalised rows are dead once projected
    const SingleImages im = take_single_images(ws, Ba, N, N, H, d);
    const bool own_cond = ada && cond == nullptr;
    bf16* sn = own_cond ? (bf16*)ws.take(2 * rows * c_s * sizeof(bf16)) : nullptr;
    bf16* planes = own_cond ? (bf16*)ws.take(3 * rows * c_a * sizeof(bf16)) : nullptr;
    bf16* tb = bias_tiles ? nullptr : (bf16*)ws.take((size_t)Bz * of3_pair_bias_tiles_elems(N) * sizeof(bf16));
    if (!ws.base) return OF3_OK;
    OF3_REQUIRE(ws.ok(), OF3_ERR_WORKSPACE, "attn_pair_bias: workspace too small (%zu needed)", ws.off);
    int rc;
    if (ada) {
        if (cond == nullptr) {
            const CondLayer l = cond_layer(p);
            if ((rc = conditioning(s, &l, 1, rows, c_a, c_s, sn, planes, st))) return rc;
            cond = planes;
        }
        if ((rc = ada_rows(a, cond, (const bf16*)p->ada_b_g, an, rows, c_a, st))) return rc;
    } else if ((rc = ln_rows(a, (const bf16*)p->ln_a_w, (const bf16*)p->ln_a_b, an, rows, c_a, st))) {
        return rc;
    }
    {
        const LinearIn in{an, rows, c_a, c_a,
                          {(const bf16*)p->w_q, (const bf16*)p->w_g, (const bf16*)p->w_k, (const bf16*)p->w_v}, 4};
        const LinearOut kinds[4] = {kOutQ, kOutG, kOutK, kOutV};
        const AttnImages images{im.q, im.k, im.v, g, (const bf16*)p->b_q, N, H, d};
        const bool few = token_images_supported(Ba, N, c_a, d) && alone(rows, flags);
        if ((rc = (few ? token_attn_images : linear_attn_images)(in, kinds, images, st))) return rc;
    }
    SingleBias bias;
    bias.tiles = bias_tiles;
    bias.f32 = pair_bias;
    bias.z = z;
    bias.ln_w = (const bf16*)p->ln_z_w;
    bias.ln_b = (const bf16*)p->ln_z_b;
    bias.w = (const bf16*)p->w_z;
    if ((rc = single_attn(im, g, bias, tb, mask, og, Ba, N, N, H, d, inf, Ba / Bz, !(flags & kFlagBeside), st))) return rc;
    const LinearIn in{og, rows, c_a, c_a, {(const bf16*)p->w_o}, 1};
    const bool few = token_residual_supported(rows, c_a) && alone(rows, flags) && even(a) && even(out);
    return (few ? token_residual : linear_residual)(in, (flags & OF3_FLAG_ADD_RESIDUAL) ? a : nullptr,
                                                    ada ? cond + 2 * rows * c_a : nullptr, (const bf16*)p->b_ada_out, nullptr, out,
                                                    st);
}

// ConditionedTransitionBlock (transition.py:325-339): AdaLN -> SwiGLU -> linear_out, gated by sigmoid(linear_g(s)).
bool cond_transition_supported(int c_a, int c_s, int n, int flags) {
    return !(flags & OF3_FLAG_FORCE_GENERIC) && c_a % 64 == 0 && c_s % 64 == 0 && c_a <= kMaxRowWidth &&
           c_s <= kMaxRowWidth;
}
int cond_transition(const bf16* a, const bf16* s, const bf16* mask, bf16* out, long long rows, int c_a, int c_s, int n,
                    int flags, const of3_cond_transition_params* p, Arena& ws, cudaStream_t st, const bf16* cond) {
    const int hid = n * c_a;
    bf16* an = (bf16*)ws.take(rows * c_a * sizeof(bf16));
    bf16* h = (bf16*)ws.take(rows * hid * sizeof(bf16));
    bf16* sn = cond ? nullptr : (bf16*)ws.take(2 * rows * c_s * sizeof(bf16));
    bf16* planes = cond ? nullptr : (bf16*)ws.take(3 * rows * c_a * sizeof(bf16));
    if (!ws.base) return OF3_OK;
    OF3_REQUIRE(ws.ok(), OF3_ERR_WORKSPACE, "cond_transition: workspace too small (%zu needed)", ws.off);
    int rc;
    if (cond == nullptr) {
        const CondLayer l = cond_layer(p);
        if ((rc = conditioning(s, &l, 1, rows, c_a, c_s, sn, planes, st))) return rc;
        cond = planes;
    }
    if ((rc = ada_rows(a, cond, (const bf16*)p->ada_b_g, an, rows, c_a, st))) return rc;
    const LinearIn up{an, rows, c_a, hid, {(const bf16*)p->w_a, (const bf16*)p->w_b}, 2};
    if ((rc = (token_swiglu_supported(rows, hid) ? token_swiglu : linear_swiglu)(up, h, st))) return rc;
    const LinearIn down{h, rows, hid, c_a, {(const bf16*)p->w_out}, 1};
    const bool few = token_residual_supported(rows, c_a) && even(a) && even(out);
    return (few ? token_residual : linear_residual)(down, (flags & OF3_FLAG_ADD_RESIDUAL) ? a : nullptr, cond + 2 * rows * c_a,
                           (const bf16*)p->b_g, mask, out, st);
}

// The same layer for a window of R query rows [row0, row0 + R) of one sample: keys and values come from
// all N rows of `a`, queries / gate / output only from the window; pair_bias_rows is [H][R][N] (the
// projected pair bias of exactly those rows) and out_rows is [R][c_a]. Used when the pair tensor, and
// with it the pair bias, is split by rows over several GPUs.
int attn_pair_bias_rows(const bf16* a, const float* pair_bias_rows, const bf16* mask, bf16* out_rows, int N, int row0,
                        int R, int c_a, int H, int d, float inf, int flags, const of3_attn_pair_bias_params* p,
                        Arena& ws, cudaStream_t st) {
    bf16* an = (bf16*)ws.take((size_t)N * c_a * sizeof(bf16));
    bf16* g = (bf16*)ws.take((size_t)R * c_a * sizeof(bf16));
    bf16* og = (bf16*)ws.take((size_t)R * c_a * sizeof(bf16));
    const SingleImages im = take_single_images(ws, 1, N, R, H, d);
    bf16* tb = (bf16*)ws.take((size_t)H * ceil_div(N, 32) * R * 32 * sizeof(bf16));
    if (!ws.base) return OF3_OK;
    OF3_REQUIRE(ws.ok(), OF3_ERR_WORKSPACE, "attn_pair_bias_rows: workspace too small (%zu needed)", ws.off);
    OF3_REQUIRE(row0 >= 0 && R > 0 && row0 + R <= N, OF3_ERR_ARG, "attn_pair_bias_rows: window [%d, %d) outside %d rows",
                row0, row0 + R, N);
    int rc;
    if ((rc = ln_rows(a, (const bf16*)p->ln_a_w, (const bf16*)p->ln_a_b, an, N, c_a, st))) return rc;
    {
        const LinearIn kv{an, N, c_a, c_a, {(const bf16*)p->w_k, (const bf16*)p->w_v}, 2};
        const LinearOut kvk[2] = {kOutK, kOutV};
        if ((rc = linear_attn_images(kv, kvk, AttnImages{im.q, im.k, im.v, g, nullptr, N, H, d}, st))) return rc;
        const LinearIn qg{an + (long long)row0 * c_a, R, c_a, c_a, {(const bf16*)p->w_q, (const bf16*)p->w_g}, 2};
        const LinearOut qgk[2] = {kOutQ, kOutG};
        if ((rc = linear_attn_images(qg, qgk, AttnImages{im.q, im.k, im.v, g, (const bf16*)p->b_q, R, H, d}, st)))
            return rc;
    }
    SingleBias bias;
    bias.f32 = pair_bias_rows;
    if ((rc = single_attn(im, g, bias, tb, mask, og, 1, N, R, H, d, inf, 1, false, st))) return rc;
    const LinearIn in{og, R, c_a, c_a, {(const bf16*)p->w_o}, 1};
    return linear_residual(in, (flags & OF3_FLAG_ADD_RESIDUAL) ? a + (long long)row0 * c_a : nullptr, nullptr, nullptr,
                           nullptr, out_rows, st);
}

// SwiGLU transition for widths without the fused row-tile kernel (bf16, c a multiple of 64).
bool transition_wide_supported(int c, int n) { return c % 64 == 0 && c <= kMaxRowWidth && !transition_supported(c, n); }

int transition_wide(const bf16* x, const bf16* mask, bf16* out, long long rows, int c, int n, int flags,
                    const of3_transition_params* p, Arena& ws, cudaStream_t st) {
    const int hid = n * c;
    bf16* xn = (bf16*)ws.take(rows * c * sizeof(bf16));
    bf16* h = (bf16*)ws.take(rows * hid * sizeof(bf16));
    if (!ws.base) return OF3_OK;
    OF3_REQUIRE(ws.ok(), OF3_ERR_WORKSPACE, "transition: workspace too small (%zu needed)", ws.off);
    OF3_REQUIRE(rows < (1LL << 31), OF3_ERR_SHAPE, "transition: too many rows");
    int rc;
    if ((rc = ln_rows(x, (const bf16*)p->ln_w, (const bf16*)p->ln_b, xn, rows, c, st))) return rc;
    const LinearIn up{xn, rows, c, hid, {(const bf16*)p->w_a, (const bf16*)p->w_b}, 2};
    if ((rc = (token_swiglu_supported(rows, hid) && alone(rows, flags) ? token_swiglu : linear_swiglu)(up, h, st))) return rc;
    const LinearIn down{h, rows, hid, c, {(const bf16*)p->w_out}, 1};
    const bool few = token_residual_supported(rows, c) && alone(rows, flags) && even(x) && even(out);
    return (few ? token_residual : linear_residual)(down, (flags & OF3_FLAG_ADD_RESIDUAL) ? x : nullptr, nullptr, nullptr, mask, out, st);
}

}  // namespace fast
}  // namespace of3
