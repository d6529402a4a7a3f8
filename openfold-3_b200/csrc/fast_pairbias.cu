// Pair-bias projection of the single track and of the diffusion token stack on the tensor pipe (bf16 z, c_z = 128, 16
// heads), for one layer or for several at once:
//   bias_l[h][pos] = sum_c LayerNorm_l(z[pos])[c] * W_l[h][c]          (attention_pair_bias.py:154-163)
// The layers differ in LayerNorm weights and projection only, so with W'_l = W_l * gamma_l (rounded to bf16 once per
// launch, in the prologue) and the row's mean and 1 / std
//   bias_l[h][pos] = rstd * (W'_l[h] . z[pos] - mean * sum_c W'_l[h][c]) + sum_c beta_l[c] W_l[h][c]
// and z itself, unnormalised and unrounded, is the GEMM's operand: one pass over z for all layers, and no normalised tile
// is written back to shared memory. (The operand error is one bf16 rounding per product, of the weight instead of the
// activation; sums and the mean correction are fp32.)
//
// Per tile of 128 positions of a line: TMA -> per group of 128 output channels (8 layers x 16 heads) one 128 x 128 x 128
// GEMM with the weights as the A operand, so that a TMEM lane is an output channel and its columns are consecutive
// keys: a thread stores 32 bytes of a bias row at a time. Eight warps take the row statistics meanwhile.
// Bound: HBM. 24 layers at N = 768 read 151 MB and write 453 MB, 94 us; one pass per layer (LayerNorm into the operand
// tile, 2-byte stores) took 24 x 56 us.
#include "fast_pairbias.cuh"
#include "modules.cuh"
#include "rowtile.cuh"
#include "runtime.cuh"

namespace of3 {
namespace fast {
namespace {

using namespace umma;
using namespace rowtile;

constexpr int kKidPairBias = 9;
constexpr int kHeads = 16;
constexpr int kZStages = 3;    // z tiles in flight
constexpr int kRing = 4;       // row statistics of the last tiles: the epilogue trails the loads
constexpr int kSlots = 4;      // TMEM slots of 128 columns
constexpr int kStatWarps = 8;
constexpr int kPbThreads = 32 * (2 + kStatWarps + 8);   // producer, MMA, statistics, two epilogue sets

template <int G>   // groups of 128 output channels
struct PbSmem {
    static constexpr uint32_t kW = 0;
    static constexpr uint32_t kZ = G * kTileBytes;
    static constexpr uint32_t kStat = kZ + kZStages * kTileBytes;    // ring x 2 x 128 floats: 1 / std, -mean / std
    static constexpr uint32_t kConst = kStat + kRing * 1024;         // per channel: sum of W', constant term
    static constexpr uint32_t kBars = kConst + G * 1024;
    static constexpr uint32_t kDyn = kBars + 256 + 1024;
};

struct PbWeights {
    const __nv_bfloat16 *ln_w[kMaxBiasLayers], *ln_b[kMaxBiasLayers], *w[kMaxBiasLayers];
};

// Output: with tiles != null the attention kernel's bias image of every layer (bf16, times log2(e), [layer][b*16 + h][key
// block of 32][query row][32 keys], each 64-byte row in the 64-byte swizzle of a K-major A operand, keys past the end
// zeros), lines = query rows; else (one layer) fp32 dst[line * 16 + h][position].
// kOne: a single layer. As the A operand its 16 channels leave seven eighths of the lanes empty and one warp per tile to write
// them out, 128 keys in a row; as the B operand a TMEM lane is a position, four warps take 32 keys each, and a store of a warp
// is the 64 bytes of a bias row: N = 768 69 -> 45 us (1.6 times the floor: z read, tiles written), N = 256 12.5 -> 8.9. The same
// sums, so the same bits.
template <int G, bool kOne>
__global__ void __launch_bounds__(kPbThreads, 1)
pair_bias_kernel(const __grid_constant__ CUtensorMap tmZ, const __grid_constant__ PbWeights wts, int layers,
                 float* __restrict__ dst, __nv_bfloat16* __restrict__ tiles, long long layer_stride, long long lines,
                 int N, int* status) {
    using Sm = PbSmem<G>;
    extern __shared__ uint8_t smem_raw[];
    const uint32_t sbase = (smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t* gbase = smem_raw + (sbase - smem_u32(smem_raw));
    float* stat = reinterpret_cast<float*>(gbase + Sm::kStat);
    float2* chan = reinterpret_cast<float2*>(gbase + Sm::kConst);
    const uint32_t bars = sbase + Sm::kBars;
    auto z_full = [&](int s) { return bars + 8u * s; };
    auto z_empty = [&](int s) { return bars + 8u * (kZStages + s); };
    auto st_ready = [&](int r) { return bars + 8u * (2 * kZStages + r); };
    auto st_free = [&](int r) { return bars + 8u * (2 * kZStages + kRing + r); };
    auto slot_full = [&](int q) { return bars + 8u * (2 * kZStages + 2 * kRing + q); };
    auto slot_empty = [&](int q) { return bars + 8u * (2 * kZStages + 2 * kRing + kSlots + q); };
    volatile uint32_t* tmem_ptr = reinterpret_cast<volatile uint32_t*>(gbase + Sm::kBars + 200);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(gbase + Sm::kBars + 208);
    static_assert(8 * (2 * kZStages + 2 * kRing + 2 * kSlots) <= 200, "barrier block");

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int tiles_per_line = (N + kRows - 1) / kRows;
    const long long num_tiles = lines * tiles_per_line;
    const int lines_per_sample = tiles != nullptr ? N : 1;
    constexpr float kLog2e = 1.4426950408889634f;

    if (threadIdx.x == 0) {
        for (int s = 0; s < kZStages; ++s) {
            mbar_init(z_full(s), 1);
            mbar_init(z_empty(s), 1 + kStatWarps);
        }
        for (int r = 0; r < kRing; ++r) {
            mbar_init(st_ready(r), kStatWarps);
            mbar_init(st_free(r), 4 * G);
        }
        for (int q = 0; q < kSlots; ++q) {
            mbar_init(slot_full(q), 1);
            mbar_init(slot_empty(q), 4);
        }
        *abort_flag = 0;
        mbar_fence_init();
        prefetch_tmap(&tmZ);
    }
    // W' as swizzled operand tiles, 16 threads per channel; channels past the last layer are zeros
    for (int idx = threadIdx.x; idx < G * 128 * 16; idx += kPbThreads) {
        const int n = idx >> 4, seg = idx & 15, l = n >> 4, h = n & 15;
        float cs = 0.f, cb = 0.f;
        uint32_t o[4] = {0u, 0u, 0u, 0u};
        if (l < layers) {
            uint32_t wv[4], gv[4] = {0x3F803F80u, 0x3F803F80u, 0x3F803F80u, 0x3F803F80u}, bv[4] = {0u, 0u, 0u, 0u};
            ld_row8_any(wts.w[l] + h * kC + seg * 8, wv);
            if (wts.ln_w[l]) ld_row8_any(wts.ln_w[l] + seg * 8, gv);
            if (wts.ln_b[l]) ld_row8_any(wts.ln_b[l] + seg * 8, bv);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                o[e] = pack_bf16x2(bf16lo(wv[e]) * bf16lo(gv[e]), bf16hi(wv[e]) * bf16hi(gv[e]));
                cs += bf16lo(o[e]) + bf16hi(o[e]);
                cb = fmaf(bf16lo(wv[e]), bf16lo(bv[e]), fmaf(bf16hi(wv[e]), bf16hi(bv[e]), cb));
            }
        }
        sts128(chunk_addr(sbase + Sm::kW + (n >> 7) * kTileBytes, n & 127, seg), make_uint4(o[0], o[1], o[2], o[3]));
#pragma unroll
        for (int w = 8; w > 0; w >>= 1) {
            cs += __shfl_xor_sync(0xffffffffu, cs, w);
            cb += __shfl_xor_sync(0xffffffffu, cb, w);
        }
        if (seg == 0) chan[n] = make_float2(cs, cb);
    }
    fence_proxy_async_smem();
    if (warp == 1) {
        tmem_alloc(smem_u32((const void*)tmem_ptr), 512);
        tmem_relinquish();
    }
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem_base = *tmem_ptr;
    grid_trigger();
    grid_wait();

    if (warp == 0) {
        // ---------------------------------------------------------------- TMA producer
        if (elect_one()) {
            uint32_t it = 0;
            TileWalk tw(blockIdx.x, gridDim.x, lines_per_sample, tiles_per_line);
            for (long long t = blockIdx.x; t < num_tiles; t += gridDim.x, ++it, tw.next()) {
                const int s = it % kZStages;
                if (!mbar_wait(z_empty(s), ((it / kZStages) & 1u) ^ 1u, abort_flag)) {
                    report_wait_failure(status, abort_flag, kKidPairBias, 1);
                    break;
                }
                mbar_arrive_expect_tx(z_full(s), kTileBytes);
                const uint32_t d = sbase + Sm::kZ + s * kTileBytes;
                for (int kb = 0; kb < 2; ++kb)
                    tma_load_3d(d + kb * kKBlockBytes, &tmZ, z_full(s), kb * 64, tw.tile * kRows,
                                tw.b * lines_per_sample + tw.line);
            }
        }
    } else if (warp == 1) {
        // ---------------------------------------------------------------- MMA issuer
        if (elect_one()) {
            constexpr uint32_t idesc = idesc_bf16_f32(128, kOne ? kHeads : 128);
            uint32_t it = 0, job = 0;
            bool ok = true;
            for (long long t = blockIdx.x; t < num_tiles && ok; t += gridDim.x, ++it) {
                const int s = it % kZStages;
                if (!mbar_wait(z_full(s), (it / kZStages) & 1u, abort_flag)) {
                    report_wait_failure(status, abort_flag, kKidPairBias, 2);
                    break;
                }
                for (int g = 0; g < G; ++g, ++job) {
                    const int q = job % kSlots;
                    if (!mbar_wait(slot_empty(q), ((job / kSlots) & 1u) ^ 1u, abort_flag)) {
                        report_wait_failure(status, abort_flag, kKidPairBias, 3);
                        ok = false;
                        break;
                    }
                    tc_fence_after_sync();
                    const uint32_t wt = sbase + Sm::kW + g * kTileBytes, zt = sbase + Sm::kZ + s * kTileBytes;
                    mma_rows<128>(tmem_base + q * 128, kOne ? zt : wt, kOne ? wt : zt, kKBlockBytes, idesc, false);
                    mma_commit(slot_full(q));
                }
                if (ok) mma_commit(z_empty(s));
            }
        }
    } else if (warp < 2 + kStatWarps) {
        // ---------------------------------------------------------------- row statistics: 16 positions per warp
        const int row = (warp - 2) * 16 + (lane & 15), half = lane >> 4;
        uint32_t it = 0;
        for (long long t = blockIdx.x; t < num_tiles; t += gridDim.x, ++it) {
            const int s = it % kZStages, r = it % kRing;
            if (!mbar_wait(z_full(s), (it / kZStages) & 1u, abort_flag) ||
                !mbar_wait(st_free(r), ((it / kRing) & 1u) ^ 1u, abort_flag)) {
                if (lane == 0) report_wait_failure(status, abort_flag, kKidPairBias, 4);
                break;
            }
            uint32_t raw[32];
            load_half_row(sbase + Sm::kZ + s * kTileBytes, row, half, raw);
            float mean, rstd;
            half_row_stats(raw, mean, rstd);
            if (half == 0) {
                stat[r * 256 + row] = rstd;
                stat[r * 256 + 128 + row] = -rstd * mean;
            }
            __syncwarp();
            if (lane == 0) {
                mbar_arrive(z_empty(s));
                mbar_arrive(st_ready(r));
            }
        }
    } else {
        // ---------------------------------------------------------------- epilogue: thread = output channel
        const int set = (warp - 2 - kStatWarps) >> 2, quad = warp & 3;
        const int nkb = (N + 31) >> 5;
        const long long hs = (long long)nkb * N * 32;   // elements per (sample, head) of the bias image
        uint32_t it = 0, job = 0;
        bool ok = true;
        TileWalk tw(blockIdx.x, gridDim.x, lines_per_sample, tiles_per_line);
        for (long long t = blockIdx.x; t < num_tiles && ok; t += gridDim.x, ++it, tw.next()) {
            const int t0 = tw.tile * kRows;
            const int live = N - t0 < kRows ? N - t0 : kRows;                       // positions that exist
            const int span = tiles != nullptr ? ((live + 31) & ~31) : live;         // positions to be written
            const int r = it % kRing;
            const float* p1 = stat + r * 256;
            for (int g = 0; g < G; ++g, ++job) {
                if ((int)(job & 1u) != set) continue;
                const int q = job % kSlots;
                if (!mbar_wait(st_ready(r), (it / kRing) & 1u, abort_flag) ||
                    !mbar_wait(slot_full(q), (job / kSlots) & 1u, abort_flag)) {
                    if (lane == 0) report_wait_failure(status, abort_flag, kKidPairBias, 5);
                    ok = false;
                    break;
                }
                tc_fence_after_sync();
                if constexpr (kOne) {
                    const int row = quad * 32 + lane, pos = t0 + row;   // (quad * 32 < span: the whole warp's key block)
                    uint32_t acc[16];
                    tmem_ld16(tmem_base + ((uint32_t)(quad * 32) << 16) + q * 128, acc);
                    const float rs = p1[row], nm = p1[128 + row];
                    tmem_ld_wait();
                    if (row < span) {
                        auto value = [&](int h) {
                            const float2 cc = chan[h];
                            return fmaf(rs, __uint_as_float(acc[h]), fmaf(nm, cc.x, cc.y));
                        };
                        if (tiles != nullptr) {
                            const int key = ((((row & 31) >> 3) ^ ((tw.line >> 1) & 3)) << 3) | (row & 7);
                            __nv_bfloat16* trow = tiles + (long long)tw.b * kHeads * hs + (long long)(pos >> 5) * N * 32 +
                                                  tw.line * 32 + key;
#pragma unroll
                            for (int h = 0; h < kHeads; ++h)
                                trow[h * hs] = __float2bfloat16_rn(pos < N ? value(h) * kLog2e : 0.f);
                        } else {
                            float* drow = dst + (long long)tw.b * kHeads * N + pos;
#pragma unroll
                            for (int h = 0; h < kHeads; ++h) drow[(long long)h * N] = value(h);
                        }
                    }
                    tc_fence_before_sync();
                    __syncwarp();
                    if (lane == 0) {
                        mbar_arrive(slot_empty(q));
                        mbar_arrive(st_free(r));
                    }
                    continue;
                }
                const int n = g * 128 + quad * 32 + lane, l = n >> 4, h = n & 15;
                if (g * 128 + quad * 32 < layers * kHeads) {   // the warp has a channel (a layer is half a warp)
                    const float2 cc = chan[n];
                    const int sw = (tw.line >> 1) & 3;
                    __nv_bfloat16* trow = tiles + l * layer_stride + ((long long)tw.b * kHeads + h) * hs + tw.line * 32;
                    const uint32_t taddr = tmem_base + ((uint32_t)(quad * 32) << 16) + q * 128;
#pragma unroll 2
                    for (int k0 = 0; k0 < span; k0 += 16) {
                        uint32_t acc[16];
                        tmem_ld16(taddr + k0, acc);
                        float v[16];
                        tmem_ld_wait();
#pragma unroll
                        for (int e = 0; e < 16; e += 4) {
                            const float4 a = *reinterpret_cast<const float4*>(p1 + k0 + e);
                            const float4 m = *reinterpret_cast<const float4*>(p1 + 128 + k0 + e);
                            v[e] = fmaf(a.x, __uint_as_float(acc[e]), fmaf(m.x, cc.x, cc.y));
                            v[e + 1] = fmaf(a.y, __uint_as_float(acc[e + 1]), fmaf(m.y, cc.x, cc.y));
                            v[e + 2] = fmaf(a.z, __uint_as_float(acc[e + 2]), fmaf(m.z, cc.x, cc.y));
                            v[e + 3] = fmaf(a.w, __uint_as_float(acc[e + 3]), fmaf(m.w, cc.x, cc.y));
                        }
                        if (l < layers) {
                            if (k0 + 16 > live) {   // keys past the end
#pragma unroll
                                for (int e = 0; e < 16; ++e)
                                    if (k0 + e >= live) v[e] = 0.f;
                            }
                            // chunks c2 and c2 + 1 of the row lie at c2 ^ sw and (c2 + 1) ^ sw: one aligned pair
                            const int c2 = (k0 >> 3) & 2;
                            uint32_t o[8], w[8];
                            // scaled last, as the conversion of an fp32 bias is: a row shard, which takes that, gives
                            // the same bits as the whole tensor
#pragma unroll
                            for (int e = 0; e < 8; ++e) o[e] = pack_bf16x2(v[2 * e] * kLog2e, v[2 * e + 1] * kLog2e);
#pragma unroll
                            for (int e = 0; e < 8; ++e) w[e] = (sw & 1) ? o[e ^ 4] : o[e];
                            stg256_or_2x128(trow + (long long)((t0 + k0) >> 5) * N * 32 + ((c2 ^ (sw & 2)) << 3), w,
                                            aligned32(tiles));
                        }
                        __syncwarp();
                    }
                }
                tc_fence_before_sync();
                __syncwarp();
                if (lane == 0) {
                    mbar_arrive(slot_empty(q));
                    mbar_arrive(st_free(r));
                }
            }
        }
    }

    tc_fence_before_sync();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after_sync();
        tmem_dealloc(tmem_base, 512);
    }
}

template <int G, bool kOne>
int launch_g(const CUtensorMap& tmZ, const PbWeights& wts, int layers, float* dst, __nv_bfloat16* tiles,
             long long layer_stride, long long lines, int N, cudaStream_t st) {
    static PerDeviceOnce configured;
    if (!configured.done()) {
        OF3_CUDA_CHECK(cudaFuncSetAttribute(pair_bias_kernel<G, kOne>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                            PbSmem<G>::kDyn));
        configured.mark();
    }
    const long long num_tiles = lines * ceil_div(N, kRows);
    const int grid = (int)(num_tiles < sm_count() ? num_tiles : sm_count());
    LaunchScope scope(kKidPairBias, st);
    OF3_CUDA_CHECK(launch_chained(pair_bias_kernel<G, kOne>, grid, kPbThreads, PbSmem<G>::kDyn, st, tmZ, wts, layers, dst, tiles,
                                  layer_stride, lines, N, device_status_ptr()));
    return OF3_OK;
}

int launch(const __nv_bfloat16* z, const BiasLayer* layer, int layers, float* dst, __nv_bfloat16* tiles,
           long long layer_stride, long long lines, int N, cudaStream_t st) {
    if (lines <= 0 || N <= 0) return OF3_OK;
    OF3_REQUIRE(((uintptr_t)z & 15) == 0, OF3_ERR_ALIGN, "pair_bias: z must be 16-byte aligned");
    OF3_REQUIRE(((uintptr_t)tiles & 15) == 0, OF3_ERR_ALIGN, "pair_bias: bias tiles must be 16-byte aligned");
    OF3_REQUIRE(lines < (1LL << 31), OF3_ERR_SHAPE, "pair_bias: too many pair positions");
    OF3_REQUIRE(layers >= 1 && layers <= kMaxBiasLayers, OF3_ERR_ARG, "pair_bias: %d layers", layers);
    OF3_REQUIRE(tiles != nullptr || layers == 1, OF3_ERR_ARG, "pair_bias: fp32 output of %d layers", layers);
    PbWeights wts = {};
    for (int l = 0; l < layers; ++l) {
        wts.ln_w[l] = layer[l].ln_w;
        wts.ln_b[l] = layer[l].ln_b;
        wts.w[l] = layer[l].w;
    }
    CUtensorMap tmZ;
    uint64_t dims[3] = {128, (uint64_t)N, (uint64_t)lines};
    uint64_t str[2] = {256, (uint64_t)N * 256};
    uint32_t box[3] = {64, 128, 1};
    const int rc = make_tmap_bf16(&tmZ, z, 3, dims, str, box, 1);
    if (rc) return rc;
    switch ((layers * kHeads + 127) / 128) {
        case 1:
            return layers == 1 ? launch_g<1, true>(tmZ, wts, layers, dst, tiles, layer_stride, lines, N, st)
                               : launch_g<1, false>(tmZ, wts, layers, dst, tiles, layer_stride, lines, N, st);
        case 2: return launch_g<2, false>(tmZ, wts, layers, dst, tiles, layer_stride, lines, N, st);
        default: return launch_g<3, false>(tmZ, wts, layers, dst, tiles, layer_stride, lines, N, st);
    }
}

}  // namespace

// dst[b][h][pos] (fp32) for B samples of nn pair positions each; z [B * nn][128] bf16.
int pair_bias_c128_h16(const __nv_bfloat16* z, const __nv_bfloat16* ln_w, const __nv_bfloat16* ln_b,
                       const __nv_bfloat16* w, float* dst, long long B, long long nn, cudaStream_t st) {
    OF3_REQUIRE(nn < (1LL << 31) - 256, OF3_ERR_SHAPE, "pair_bias: too many pair positions");
    const BiasLayer l{ln_w, ln_b, w};
    return launch(z, &l, 1, dst, nullptr, 0, B, (int)nn, st);
}

int pair_bias_tiles(const __nv_bfloat16* z, const BiasLayer* layer, int layers, __nv_bfloat16* tiles, long long B, int N,
                    cudaStream_t st) {
    const long long stride = B * kHeads * (long long)((N + 31) / 32) * N * 32;
    for (int l0 = 0; l0 < layers; l0 += kMaxBiasLayers) {
        const int n = layers - l0 < kMaxBiasLayers ? layers - l0 : kMaxBiasLayers;
        const int rc = launch(z, layer + l0, n, nullptr, tiles + l0 * stride, stride, B * N, N, st);
        if (rc) return rc;
    }
    return OF3_OK;
}

// One layer's bias image (z [B][N][N][128]).
int pair_bias_tiles_c128_h16(const __nv_bfloat16* z, const __nv_bfloat16* ln_w, const __nv_bfloat16* ln_b,
                             const __nv_bfloat16* w, __nv_bfloat16* tiles, long long B, int N, cudaStream_t st) {
    const BiasLayer l{ln_w, ln_b, w};
    return pair_bias_tiles(z, &l, 1, tiles, B, N, st);
}

}  // namespace fast
}  // namespace of3
