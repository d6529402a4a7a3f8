// Triangle multiplicative update, bf16 / tcgen05 family (c_z = c_hidden = 128, or 64 in the template stack).
//
// Three kernels per layer, all fed by TMA:
//   trimul_in   z tile -> LayerNorm_in (in place) -> the four projections a_p, a_g, b_p, b_g TRANSPOSED
//               (tcgen05: the weights are the A operand, the normalised tile the B operand, so a TMEM lane is an
//               output channel and its columns are the tile's 128 positions) -> mask * sigmoid(gate) * proj ->
//               a, b stored CHANNEL-MAJOR with the contracted index innermost, a_t[c][i][k], b_t[c][j][k]:
//               every epilogue thread writes its channel's 256 contiguous bytes with 32-byte stores.
//               For the incoming update the tile walks z along its first index instead, so that
//               both directions feed the same K-major x K-major contraction.
//   contract    x_t[c][i][j] = sum_k a_t[c][i][k] * b_t[c][j][k]      (contract.cu)
//   trimul_out  x tile (all channels of 128 positions) -> LayerNorm_out -> linear_z, and in the
//               same pass z tile -> LayerNorm_in -> linear_g (recomputing the gate is one more
//               128^3 MMA and saves writing and re-reading an N^2 x 128 gate tensor);
//               out = z + sigmoid(gate) * update, TMA-stored.
// Reference: openfold3/core/model/layers/triangular_multiplicative_update.py:421-503.
#include "modules.cuh"
#include "rowtile.cuh"
#include "runtime.cuh"

namespace of3 {
namespace fast {
namespace {

using namespace umma;
using namespace rowtile;

constexpr int kKidIn = 2;
constexpr int kKidOut = 3;

// Where the channel-major tensors a_t, b_t and x_t keep channel c of a line: at channel(c) + line(l), its positions behind
// one another. Planes: [c][line][ld], or one group of channels per destination rank when they are about to be exchanged.
// Blocked (a whole pair tensor on this GPU): [line / 8][c][8][ld], so that what the tiles in flight write and read at one
// time, all channels of some twenty lines, lies in a few megabytes. In planes the 32 channels of one store lie a plane
// apart, and from 2 MB per plane on in as many pages. trimul_in, planes -> blocked: N = 768 149 -> 142 us, N = 1003
// 369 -> 246, N = 2048 1.19 -> 1.01 ms; blocks of 32 lines are no faster.
struct PlaneLayout {
    int ld, group_shift, line_shift;
    long long group_stride, chan_stride, block_stride, sample_stride;   // elements
    __host__ __device__ long long channel(int c) const {
        return (long long)(c >> group_shift) * group_stride + (long long)(c & ((1 << group_shift) - 1)) * chan_stride;
    }
    __host__ __device__ long long line(int l) const {
        return (long long)(l >> line_shift) * block_stride + (long long)(l & (int)((1u << line_shift) - 1u)) * ld;
    }
};
PlaneLayout plane_layout(int R, int ld, int C, int groups, long long group_stride) {
    PlaneLayout pl;
    pl.ld = ld;
    pl.group_shift = C == 128 ? 7 : 6;
    for (int g = groups; g > 1; g >>= 1) --pl.group_shift;
    pl.line_shift = 31;
    pl.chan_stride = (long long)R * ld;
    pl.group_stride = groups == 1 ? C * pl.chan_stride : group_stride;
    pl.block_stride = 0;
    pl.sample_stride = groups * pl.group_stride;
    return pl;
}
constexpr int kLineBlock = 1 << kLineBlockShift;
PlaneLayout blocked_layout(int R, int ld, int C) {
    PlaneLayout pl;
    pl.ld = ld;
    pl.group_shift = C == 128 ? 7 : 6;
    pl.line_shift = kLineBlockShift;
    pl.group_stride = 0;
    pl.chan_stride = (long long)kLineBlock * ld;
    pl.block_stride = C * pl.chan_stride;
    pl.sample_stride = ceil_div(R, kLineBlock) * pl.block_stride;
    return pl;
}

// R = lines per sample (R == N for a whole pair tensor, N / P for a row shard)
// =====================================================================================
// trimul_in
// =====================================================================================
// 128 channels: the four weights are four A operands and a tile makes two jobs, its a and its b projection. 64
// channels: the A operands are [a_p; b_p] and [a_g; b_g], 128 rows each, and a tile is one job.
template <int C>
struct InSmem {
    static constexpr int kJobs = C / 64;                       // GEMM pairs (projection, gate) per tile
    static constexpr int kStages = C == 128 ? 2 : 4;           // z tiles in flight
    static constexpr uint32_t kW = 0;                          // C / 64 k-blocks x [4 C rows x 128 B]
    static constexpr uint32_t kWKb = 4 * C * 128;
    static constexpr uint32_t kZ = C / 64 * kWKb;              // stages of one tile
    static constexpr uint32_t kGamma = kZ + kStages * tile_bytes<C>();   // C floats
    static constexpr uint32_t kBeta = kGamma + 512;
    static constexpr uint32_t kMask = kBeta + 512;             // ring of 128 floats: 0.5 * mask of the tile's positions
    static constexpr int kMaskRing = C == 128 ? 4 : 8;
    static constexpr uint32_t kBars = kMask + kMaskRing * 512;
    static constexpr uint32_t kTotal = kBars + 192;
    static constexpr uint32_t kDyn = kTotal + 1024;
};

// outgoing: tmZ is 3-D {c, second index, b*N + first index}; incoming: 4-D {c, second, first, b}
constexpr int kInLnWarps = 8;    // two threads per position
constexpr int kInEpiSets = 2;    // epilogue warp sets, one per TMEM slot
// Warps per 32 channels of a set, each with its part of the positions: 64 channels have one job per tile, whose epilogue
// is the longest step (template stack, N = 300 x 4: 55 -> 47 us with two); with 128 channels a second one gives nothing
// (N = 768: 142 -> 150: registers).
template <int C>
constexpr int kInEpiParts = C == 128 ? 1 : 2;
template <int C>
constexpr int kInThreads = 32 * (2 + kInLnWarps + 4 * kInEpiSets * kInEpiParts<C>);  // producer, MMA, LayerNorm, epilogue

template <int C, bool kOutgoing>
__global__ void __launch_bounds__(kInThreads<C>, 1)
trimul_in_kernel(const __grid_constant__ CUtensorMap tmZ, const __grid_constant__ CUtensorMap tmWap,
                 const __grid_constant__ CUtensorMap tmWag, const __grid_constant__ CUtensorMap tmWbp,
                 const __grid_constant__ CUtensorMap tmWbg, const __nv_bfloat16* __restrict__ mask,
                 const __nv_bfloat16* __restrict__ ln_w, const __nv_bfloat16* __restrict__ ln_b,
                 __nv_bfloat16* __restrict__ a_t, __nv_bfloat16* __restrict__ b_t, int B, int R,
                 int N, PlaneLayout pl, int wide_stores, int* status) {
    using Sm = InSmem<C>;
    constexpr int kSt = Sm::kStages;
    extern __shared__ uint8_t smem_raw[];
    const uint32_t sbase = (smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t* gbase = smem_raw + (sbase - smem_u32(smem_raw));
    float* gamma = reinterpret_cast<float*>(gbase + Sm::kGamma);
    float* beta = reinterpret_cast<float*>(gbase + Sm::kBeta);
    float* mask05 = reinterpret_cast<float*>(gbase + Sm::kMask);
    const uint32_t bars = sbase + Sm::kBars;
    const uint32_t w_full = bars;
    auto z_full = [&](int s) { return bars + 8u * (1 + s); };
    auto z_empty = [&](int s) { return bars + 8u * (1 + kSt + s); };
    auto a_ready = [&](int s) { return bars + 8u * (1 + 2 * kSt + s); };
    auto slot_full = [&](int q) { return bars + 8u * (1 + 3 * kSt + q); };
    auto slot_empty = [&](int q) { return bars + 8u * (3 + 3 * kSt + q); };
    volatile uint32_t* tmem_ptr = reinterpret_cast<volatile uint32_t*>(gbase + Sm::kBars + 160);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(gbase + Sm::kBars + 168);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int tiles_per_line = (N + kRows - 1) / kRows;
    const long long num_tiles = (long long)B * R * tiles_per_line;

    if (threadIdx.x == 0) {
        mbar_init(w_full, 1);
        for (int s = 0; s < kSt; ++s) {
            mbar_init(z_full(s), 1);
            mbar_init(z_empty(s), 1);
            mbar_init(a_ready(s), kInLnWarps);
        }
        for (int q = 0; q < 2; ++q) {
            mbar_init(slot_full(q), 1);
            mbar_init(slot_empty(q), 4 * kInEpiParts<C>);
        }
        *abort_flag = 0;
        mbar_fence_init();
        prefetch_tmap(&tmZ);
    }
    if (threadIdx.x < C) {
        gamma[threadIdx.x] = __bfloat162float(ln_w[threadIdx.x]);
        beta[threadIdx.x] = __bfloat162float(ln_b[threadIdx.x]);
    }
    if (warp == 1) {
        tmem_alloc(smem_u32((const void*)tmem_ptr), 512);
        tmem_relinquish();
    }
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem_base = *tmem_ptr;
    grid_trigger();
    // 128 channels, lone tiles: the LayerNorm warps, done with theirs, take the second half of the positions. With the projections of
    // the attention shared likewise, four pair blocks of 120 tokens: 387.4 -> 384.8 us. (64 channels have twice the epilogue warps.)
    const bool solo = C == 128 && num_tiles <= (long long)gridDim.x;

    if (warp == 0) {
        // ---------------------------------------------------------------- TMA producer
        if (elect_one()) {
            mbar_arrive_expect_tx(w_full, C / 64 * Sm::kWKb);
            // slab order: C = 128: a_p, a_g, b_p, b_g; C = 64: a_p, b_p | a_g, b_g
            const CUtensorMap* wm[4] = {&tmWap, C == 128 ? &tmWag : &tmWbp, C == 128 ? &tmWbp : &tmWag, &tmWbg};
            for (int w = 0; w < 4; ++w)
                for (int kb = 0; kb < C / 64; ++kb)
                    tma_load_2d(sbase + Sm::kW + kb * Sm::kWKb + w * C * 128, wm[w], w_full, kb * 64, 0);
            grid_wait();
            uint32_t it = 0;
            TileWalk tw(blockIdx.x, gridDim.x, R, tiles_per_line);
            for (long long t = blockIdx.x; t < num_tiles; t += gridDim.x, ++it, tw.next()) {
                const int s = it % kSt;
                if (!mbar_wait(z_empty(s), ((it / kSt) & 1u) ^ 1u, abort_flag)) {
                    report_wait_failure(status, abort_flag, kKidIn, 1);
                    break;
                }
                const int t0 = tw.tile * kRows;
                mbar_arrive_expect_tx(z_full(s), tile_bytes<C>());
                const uint32_t dst = sbase + Sm::kZ + s * tile_bytes<C>();
                for (int kb = 0; kb < C / 64; ++kb) {
                    if (kOutgoing)
                        tma_load_3d(dst + kb * kKBlockBytes, &tmZ, z_full(s), kb * 64, t0,
                                    tw.b * R + tw.line);
                    else
                        tma_load_4d(dst + kb * kKBlockBytes, &tmZ, z_full(s), kb * 64, tw.line, t0,
                                    tw.b);
                }
            }
        }
    } else if (warp == 1) {
        // ---------------------------------------------------------------- MMA issuer
        if (elect_one()) {
            constexpr uint32_t idesc = idesc_bf16_f32(128, 128);
            bool ok = mbar_wait(w_full, 0, abort_flag);
            if (!ok) report_wait_failure(status, abort_flag, kKidIn, 2);
            uint32_t it = 0;
            for (long long t = blockIdx.x; t < num_tiles && ok; t += gridDim.x, ++it) {
                const int s = it % kSt;
                if (!mbar_wait(a_ready(s), (it / kSt) & 1u, abort_flag)) {
                    report_wait_failure(status, abort_flag, kKidIn, 3);
                    break;
                }
                const uint32_t ztile = sbase + Sm::kZ + s * tile_bytes<C>();
                for (int q = 0; q < Sm::kJobs; ++q) {
                    const uint32_t job = it * Sm::kJobs + q, slot = job & 1u;
                    if (!mbar_wait(slot_empty(slot), ((job >> 1) & 1u) ^ 1u, abort_flag)) {
                        report_wait_failure(status, abort_flag, kKidIn, 4);
                        ok = false;
                        break;
                    }
                    tc_fence_after_sync();
                    // D[channel][position] = W[channel][:] . LN(z)[position][:]: projection, then gate
                    for (int hg = 0; hg < 2; ++hg) {
                        const uint32_t w_tile = sbase + Sm::kW + (q * 2 + hg) * 128 * 128;
#pragma unroll
                        for (int kb = 0; kb < C / 64; ++kb) {
                            const uint64_t ad = smem_desc_k_sw128(w_tile + kb * Sm::kWKb);
                            const uint64_t bd = smem_desc_k_sw128(ztile + kb * kKBlockBytes);
#pragma unroll
                            for (int k4 = 0; k4 < 4; ++k4)
                                mma_bf16(tmem_base + slot * 256 + hg * 128, ad + 2u * k4, bd + 2u * k4, idesc,
                                         (kb != 0 || k4 != 0) ? 1u : 0u);
                        }
                    }
                    mma_commit(slot_full(slot));
                }
                if (ok) mma_commit(z_empty(s));
            }
        }
    } else if (warp < 2 + kInLnWarps) {
        // ---------------------------------------------------------------- LayerNorm warps: a warp takes 16 positions,
        // lanes 0..15 their first 64 channels, lanes 16..31 the other 64 (statistics joined by one shuffle)
        const int row = (warp - 2) * 16 + (lane & 15);
        const int half = lane >> 4;
        grid_wait();
        uint32_t it = 0;
        TileWalk tw(blockIdx.x, gridDim.x, R, tiles_per_line);
        for (long long t = blockIdx.x; t < num_tiles; t += gridDim.x, ++it, tw.next()) {
            const int s = it % kSt;
            if (!mbar_wait(z_full(s), (it / kSt) & 1u, abort_flag)) {
                if (lane == 0) report_wait_failure(status, abort_flag, kKidIn, 5);
                break;
            }
            const uint32_t tile = sbase + Sm::kZ + s * tile_bytes<C>();
            uint32_t raw[C / 4];
            load_half_row<C>(tile, row, half, raw);
            float mean, rstd;
            half_row_stats<C>(raw, mean, rstd);
            store_normalized_half_row<C>(tile, row, half, raw, mean, rstd, gamma, beta);
            const int t0 = tw.tile * kRows;
            const int k = t0 + row;
            float m = 0.f;   // positions past the end of the line are never stored
            if (k < N) {
                m = 0.5f;
                if (mask != nullptr) {
                    const long long lin = kOutgoing ? ((long long)(tw.b * R + tw.line) * N + k)
                                                    : ((long long)(tw.b * N + k) * R + tw.line);
                    m = 0.5f * __bfloat162float(mask[lin]);
                }
            }
            // The epilogue of tile `it` may still read its buffer while the next kStages tiles are normalised (and, with
            // one job per tile, one tile more waits for the other TMEM slot); by tile it + kMaskRing it has released
            // its slot
            if (half == 0) mask05[(it % Sm::kMaskRing) * 128 + row] = m;
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) mbar_arrive(a_ready(s));
        }
    }
    if (warp >= (solo ? 2 : 2 + kInLnWarps)) {
        // ---------------------------------------------------------------- epilogue warps: the first four take the a
        // projection (TMEM slot 0), the other four the b projection (slot 1); thread = output channel, columns =
        // positions
        constexpr int kParts = kInEpiParts<C>;
        const bool helper = C == 128 && warp < 2 + kInLnWarps;
        const int ew = helper ? warp - 2 : warp - 2 - kInLnWarps;
        const int set = ew / (4 * kParts);   // TMEM slot of this set's jobs
        const int quad = warp & 3;
        const int lch = quad * 32 + lane;
        const bool is_b = C == 128 ? set == 1 : lch >= 64;
        const int c = lch & (C - 1);
        __nv_bfloat16* plane = (is_b ? b_t : a_t) + pl.channel(c);
        const uint32_t taddr = tmem_base + ((uint32_t)(quad * 32) << 16) + set * 256;
        grid_wait();
        uint32_t it = 0, use = 0;
        TileWalk tw(blockIdx.x, gridDim.x, R, tiles_per_line);
        for (long long t = blockIdx.x; t < num_tiles; t += gridDim.x, ++it, tw.next()) {
            if (C == 64 && (it & 1u) != (uint32_t)set) continue;   // one job per tile: the sets take turns
            const int t0 = tw.tile * kRows;
            const int kmax = (N - t0 < kRows) ? N - t0 : kRows;   // positions of the tile that exist
            if (!mbar_wait(slot_full(set), use & 1u, abort_flag)) {
                if (lane == 0) report_wait_failure(status, abort_flag, kKidIn, 6);
                break;
            }
            ++use;
            tc_fence_after_sync();
            const int k_half = ((kmax + 31) >> 5) << 4;   // of lone tiles
            const int k_begin = helper ? k_half : ((ew >> 2) & (kParts - 1)) * (kRows / kParts);
            const float* mk = mask05 + (it % Sm::kMaskRing) * 128;
            // the line pitch ld is a multiple of 8 elements, so a 16-byte store that starts below N ends inside the
            // row; with a pitch that is a multiple of 16 (and 32-byte aligned planes) the same holds for 32 bytes
            __nv_bfloat16* dst = plane + tw.b * pl.sample_stride + pl.line(tw.line) + t0;
            // 16 positions per pass; the TMEM load of the next pass is in flight while this one is computed
            auto emit = [&](const uint32_t (&p)[16], const uint32_t (&g)[16], int k0) {
                uint32_t o[8];
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    const float4 m0 = *reinterpret_cast<const float4*>(mk + k0 + j * 8);
                    const float4 m1 = *reinterpret_cast<const float4*>(mk + k0 + j * 8 + 4);
                    const float mm[8] = {m0.x, m0.y, m0.z, m0.w, m1.x, m1.y, m1.z, m1.w};
                    float v[8];
#pragma unroll
                    for (int e = 0; e < 8; ++e) {
                        // mask * p * sigmoid(g) = pm * tanh(g / 2) + pm with pm = (mask / 2) * p
                        const float pm = mm[e] * __uint_as_float(p[j * 8 + e]);
                        v[e] = fmaf(tanh_approx(0.5f * __uint_as_float(g[j * 8 + e])), pm, pm);
                    }
#pragma unroll
                    for (int e = 0; e < 4; ++e) o[j * 4 + e] = pack_bf16x2(v[2 * e], v[2 * e + 1]);
                }
                if (wide_stores) {   // one full 32-byte sector per thread
                    asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(dst + k0), "r"(o[0]),
                                 "r"(o[1]), "r"(o[2]), "r"(o[3]), "r"(o[4]), "r"(o[5]), "r"(o[6]), "r"(o[7])
                                 : "memory");
                } else {
                    *reinterpret_cast<uint4*>(dst + k0) = make_uint4(o[0], o[1], o[2], o[3]);
                    if (k0 + 8 < kmax) *reinterpret_cast<uint4*>(dst + k0 + 8) = make_uint4(o[4], o[5], o[6], o[7]);
                }
            };
            const int k_end = solo && !helper ? k_half : min(kmax, k_begin + kRows / kParts);
            if constexpr (kParts > 1) {   // (the warps hide each other's loads)
#pragma unroll 1
                for (int k0 = k_begin; k0 < k_end; k0 += 16) {
                    uint32_t p[16], g[16];
                    tmem_ld16(taddr + k0, p);
                    tmem_ld16(taddr + 128 + k0, g);
                    tmem_ld_wait();
                    emit(p, g, k0);
                }
            } else {
                uint32_t pa[16], ga[16], pb[16], gb[16];
                if (k_begin < k_end) {
                    tmem_ld16(taddr + k_begin, pa);
                    tmem_ld16(taddr + 128 + k_begin, ga);
                }
#pragma unroll 1
                for (int k0 = k_begin; k0 < k_end; k0 += 32) {
                    tmem_ld_wait();
                    if (k0 + 16 < k_end) {
                        tmem_ld16(taddr + k0 + 16, pb);
                        tmem_ld16(taddr + 128 + k0 + 16, gb);
                    }
                    emit(pa, ga, k0);
                    if (k0 + 16 < k_end) {
                        tmem_ld_wait();
                        if (k0 + 32 < k_end) {
                            tmem_ld16(taddr + k0 + 32, pa);
                            tmem_ld16(taddr + 128 + k0 + 32, ga);
                        }
                        emit(pb, gb, k0 + 16);
                    }
                }
            }
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0 && !helper) mbar_arrive(slot_empty(set));
        }
    }

    tc_fence_before_sync();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after_sync();
        tmem_dealloc(tmem_base, 512);
    }
}

// The same layer with the projections the other way round (the normalised tile is the A operand, a TMEM lane is a
// position, its columns the output channels; N = 256 per MMA): a warp's store covers 32 consecutive positions of ONE
// channel plane. For planes only (row shards): slower than the kernel above while one stays within a 2 MB page or so (170
// against 151 us for the planes of a whole tensor at N = 768: one 2-byte store per value), faster beyond (1.13 against
// 2.02 ms at N = 2048, where the 32 planes that one store of the kernel above touches lie megabytes apart).
constexpr int kInRowsThreads = 448;  // producer, MMA, 4 LayerNorm warps, 2 x 4 epilogue warps

template <bool kOutgoing>
__global__ void __launch_bounds__(kInRowsThreads, 1)
trimul_in_rows_kernel(const __grid_constant__ CUtensorMap tmZ, const __grid_constant__ CUtensorMap tmWap,
                 const __grid_constant__ CUtensorMap tmWag, const __grid_constant__ CUtensorMap tmWbp,
                 const __grid_constant__ CUtensorMap tmWbg, const __nv_bfloat16* __restrict__ mask,
                 const __nv_bfloat16* __restrict__ ln_w, const __nv_bfloat16* __restrict__ ln_b,
                 __nv_bfloat16* __restrict__ a_t, __nv_bfloat16* __restrict__ b_t, int B, int R,
                 int N, PlaneLayout pl, int* status) {
    extern __shared__ uint8_t smem_raw[];
    const uint32_t sbase = (smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t* gbase = smem_raw + (sbase - smem_u32(smem_raw));
    float* gamma = reinterpret_cast<float*>(gbase + InSmem<128>::kGamma);
    float* beta = reinterpret_cast<float*>(gbase + InSmem<128>::kBeta);
    const uint32_t bars = sbase + InSmem<128>::kBars;
    const uint32_t w_full = bars;
    auto z_full = [&](int s) { return bars + 8u * (1 + s); };
    auto z_empty = [&](int s) { return bars + 8u * (3 + s); };
    auto a_ready = [&](int s) { return bars + 8u * (5 + s); };
    auto slot_full = [&](int q) { return bars + 8u * (7 + q); };
    auto slot_empty = [&](int q) { return bars + 8u * (9 + q); };
    volatile uint32_t* tmem_ptr = reinterpret_cast<volatile uint32_t*>(gbase + InSmem<128>::kBars + 96);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(gbase + InSmem<128>::kBars + 104);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int tiles_per_line = (N + kRows - 1) / kRows;
    const long long num_tiles = (long long)B * R * tiles_per_line;

    if (threadIdx.x == 0) {
        mbar_init(w_full, 1);
        for (int s = 0; s < 2; ++s) {
            mbar_init(z_full(s), 1);
            mbar_init(z_empty(s), 1);
            mbar_init(a_ready(s), 4);
            mbar_init(slot_full(s), 1);
            mbar_init(slot_empty(s), 4);
        }
        *abort_flag = 0;
        mbar_fence_init();
        prefetch_tmap(&tmZ);
    }
    if (threadIdx.x < 128) {
        gamma[threadIdx.x] = __bfloat162float(ln_w[threadIdx.x]);
        beta[threadIdx.x] = __bfloat162float(ln_b[threadIdx.x]);
    }
    if (warp == 1) {
        tmem_alloc(smem_u32((const void*)tmem_ptr), 512);
        tmem_relinquish();
    }
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem_base = *tmem_ptr;
    grid_trigger();
    if (warp != 0 && warp != 1) grid_wait();

    if (warp == 0) {
        // ---------------------------------------------------------------- TMA producer
        if (elect_one()) {
            mbar_arrive_expect_tx(w_full, 2 * InSmem<128>::kWKb);
            const CUtensorMap* wm[4] = {&tmWap, &tmWag, &tmWbp, &tmWbg};
            for (int w = 0; w < 4; ++w)
                for (int kb = 0; kb < 2; ++kb)
                    tma_load_2d(sbase + InSmem<128>::kW + kb * InSmem<128>::kWKb + w * 128 * 128, wm[w], w_full,
                                kb * 64, 0);
            grid_wait();
            uint32_t it = 0;
            TileWalk tw(blockIdx.x, gridDim.x, R, tiles_per_line);
            for (long long t = blockIdx.x; t < num_tiles; t += gridDim.x, ++it, tw.next()) {
                const int s = it & 1;
                if (!mbar_wait(z_empty(s), ((it >> 1) & 1u) ^ 1u, abort_flag)) {
                    report_wait_failure(status, abort_flag, kKidIn, 1);
                    break;
                }
                const int t0 = tw.tile * kRows;
                mbar_arrive_expect_tx(z_full(s), kTileBytes);
                const uint32_t dst = sbase + InSmem<128>::kZ + s * kTileBytes;
                for (int kb = 0; kb < 2; ++kb) {
                    if (kOutgoing)
                        tma_load_3d(dst + kb * kKBlockBytes, &tmZ, z_full(s), kb * 64, t0,
                                    tw.b * R + tw.line);
                    else
                        tma_load_4d(dst + kb * kKBlockBytes, &tmZ, z_full(s), kb * 64, tw.line, t0,
                                    tw.b);
                }
            }
        }
    } else if (warp == 1) {
        // ---------------------------------------------------------------- MMA issuer
        if (elect_one()) {
            constexpr uint32_t idesc = idesc_bf16_f32(128, 256);
            bool ok = mbar_wait(w_full, 0, abort_flag);
            if (!ok) report_wait_failure(status, abort_flag, kKidIn, 2);
            uint32_t it = 0;
            for (long long t = blockIdx.x; t < num_tiles && ok; t += gridDim.x, ++it) {
                const int s = it & 1;
                if (!mbar_wait(a_ready(s), (it >> 1) & 1u, abort_flag)) {
                    report_wait_failure(status, abort_flag, kKidIn, 3);
                    break;
                }
                for (int q = 0; q < 2; ++q) {
                    if (!mbar_wait(slot_empty(q), (it & 1u) ^ 1u, abort_flag)) {
                        report_wait_failure(status, abort_flag, kKidIn, 4);
                        ok = false;
                        break;
                    }
                    tc_fence_after_sync();
                    mma_k128(tmem_base + q * 256, sbase + InSmem<128>::kZ + s * kTileBytes,
                             sbase + InSmem<128>::kW + q * 256 * 128, InSmem<128>::kWKb, idesc, false);
                    mma_commit(slot_full(q));
                }
                if (ok) mma_commit(z_empty(s));
            }
        }
    } else if (warp < 6) {
        // ---------------------------------------------------------------- LayerNorm warps (2..5)
        const int row = (warp - 2) * 32 + lane;
        uint32_t it = 0;
        for (long long t = blockIdx.x; t < num_tiles; t += gridDim.x, ++it) {
            const int s = it & 1;
            if (!mbar_wait(z_full(s), (it >> 1) & 1u, abort_flag)) {
                if (lane == 0) report_wait_failure(status, abort_flag, kKidIn, 5);
                break;
            }
            const uint32_t tile = sbase + InSmem<128>::kZ + s * kTileBytes;
            uint32_t raw[64];
            load_row(tile, row, raw);
            float mean, rstd;
            row_stats(raw, mean, rstd);
            store_normalized_row(tile, row, raw, mean, rstd, gamma, beta);
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) mbar_arrive(a_ready(s));
        }
    } else {
        // ---------------------------------------------------------------- epilogue warps: 6..9 take the a
        // projection (TMEM slot 0), 10..13 the b projection (slot 1). One set of four warps doing both
        // (2 x 128 sigmoid / multiply / convert / store per row and tile on one thread) was the longest
        // chain of the kernel.
        const int qset = (warp - 6) >> 2;
        const int quad = warp & 3;
        const int row = quad * 32 + lane;
        uint32_t it = 0;
        bool ok = true;
        TileWalk tw(blockIdx.x, gridDim.x, R, tiles_per_line);
        for (long long t = blockIdx.x; t < num_tiles && ok; t += gridDim.x, ++it, tw.next()) {
            const int t0 = tw.tile * kRows;
            const int k = t0 + row;
            const bool valid = k < N;
            float m = 1.0f;
            if (valid && mask != nullptr) {
                const long long lin = kOutgoing ? ((long long)(tw.b * R + tw.line) * N + k)
                                                : ((long long)(tw.b * N + k) * R + tw.line);
                m = __bfloat162float(mask[lin]);
            }
            const float mh = 0.5f * m;
            for (int q = qset; q <= qset; ++q) {
                if (!mbar_wait(slot_full(q), it & 1u, abort_flag)) {
                    if (lane == 0) report_wait_failure(status, abort_flag, kKidIn, 6);
                    ok = false;
                    break;
                }
                tc_fence_after_sync();
                const long long cs = pl.chan_stride;
                __nv_bfloat16* dst = (q == 0 ? a_t : b_t) + tw.b * pl.sample_stride + pl.line(tw.line) + k;
                const uint32_t taddr = tmem_base + ((uint32_t)(quad * 32) << 16) + q * 256;
#pragma unroll 1
                for (int cb = 0; cb < 4; ++cb) {
                    uint32_t p[32], g[32];
                    tmem_ld32(taddr + cb * 32, p);
                    tmem_ld32(taddr + 128 + cb * 32, g);
                    tmem_ld_wait();
                    if (valid) {
#pragma unroll
                        for (int hf = 0; hf < 2; ++hf) {  // groups hold >= 16 channels: no boundary inside a half
                            const int c0 = cb * 32 + hf * 16;
                            __nv_bfloat16* d0 = dst + pl.channel(c0);
#pragma unroll
                            for (int e = 0; e < 16; ++e) {
                                // the same expression as the kernel above, so that both give the same bits:
                                // mask * p * sigmoid(g) = pm * tanh(g / 2) + pm with pm = (mask / 2) * p
                                const float pm = mh * __uint_as_float(p[hf * 16 + e]);
                                const float v = fmaf(tanh_approx(0.5f * __uint_as_float(g[hf * 16 + e])), pm, pm);
                                d0[(long long)e * cs] = __float2bfloat16_rn(v);
                            }
                        }
                    }
                }
                tc_fence_before_sync();
                __syncwarp();
                if (lane == 0) mbar_arrive(slot_empty(q));
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

// =====================================================================================
// trimul_out
// =====================================================================================
template <int C>
struct OutSmem {
    static constexpr uint32_t kWBytes = C * C * 2;            // a weight as C / 64 k-blocks of [C rows x 128 B]
    static constexpr uint32_t kWg = 0;
    static constexpr uint32_t kWz = kWBytes;
    static constexpr uint32_t kZ = 2 * kWBytes;                    // 2 groups: z tile, then output
    static constexpr uint32_t kX = kZ + 2 * tile_bytes<C>();       // 2 groups: x tile [c][j], then A
    static constexpr uint32_t kParams = kX + 2 * tile_bytes<C>();  // gamma_in, beta_in, gamma_out, beta_out
    static constexpr uint32_t kXch = kParams + 4 * 512;            // 2 groups x 512 floats: LayerNorm partial sums
    static constexpr uint32_t kBars = kXch + 4096;
    static constexpr uint32_t kTotal = kBars + 160;
    static constexpr uint32_t kDyn = kTotal + 1024;
};

// Warps: 0 producer, 1 and 2 issue the GEMMs and the stores of the two row groups, then 2 groups x 8 warps, which alternate
// tiles; two threads share a row, each with half of its channels. (One thread per row took 3400 + 4300 cycles for the two
// LayerNorms and 3900 for the output of a tile's 17400 at N = 768: latency, with one warp of a group per scheduler; and the
// row thread that waited for the store to leave its buffer another 1500.)
constexpr int kOutThreads = 32 * (4 + 2 * 8);
// registers: the block is launched with 96 per thread; the issuing warpgroup (its fourth warp is idle) gives up what the row
// warps take, which hold half a row of z under the statistics of x (N = 768: 127 -> 119 us, with the
// conversions for x and mixed adds for z that leave 20 bytes of spills; mixed adds for both: 122)
constexpr int kOutRegsLaunch = 96, kOutRegsIssue = 64, kOutRegsRows = 104;
static_assert(kOutRegsIssue + 4 * kOutRegsRows <= 5 * kOutRegsLaunch, "register split");

// CH channels of one position of an x tile [c][128 positions], as pairs
template <int CH>
__device__ __forceinline__ void gather_column(uint32_t col, uint32_t (&raw)[CH / 2]) {
#pragma unroll
    for (int i = 0; i < CH / 2; ++i) {
        uint32_t lo, hi;
        if ((i & 7) == 0) asm volatile("" ::: "memory");  // cap the loads in flight per batch
        asm volatile("ld.shared.u16 %0, [%1];" : "=r"(lo) : "r"(col + (2 * i) * 256));
        asm volatile("ld.shared.u16 %0, [%1];" : "=r"(hi) : "r"(col + (2 * i + 1) * 256));
        raw[i] = lo | (hi << 16);
    }
}
// z += sigmoid(gate) * update for 16 channels of a row, two chunks of the tile from `chunk` on
__device__ __forceinline__ void update_channels(uint32_t ztile, int row, int chunk, const uint32_t (&gate)[16], const uint32_t (&upd)[16],
                                                int add_residual) {
#pragma unroll
    for (int ch = 0; ch < 2; ++ch) {
        const uint32_t addr = chunk_addr(ztile, row, chunk + ch);
        const uint4 z = lds128(addr);
        const uint32_t zr[4] = {z.x, z.y, z.z, z.w};
        uint32_t o[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int e = ch * 8 + j * 2;
            float v0 = sigmoid_fast(__uint_as_float(gate[e])) * __uint_as_float(upd[e]);
            float v1 = sigmoid_fast(__uint_as_float(gate[e + 1])) * __uint_as_float(upd[e + 1]);
            if (add_residual) {
                v0 += bf16lo(zr[j]);
                v1 += bf16hi(zr[j]);
            }
            o[j] = pack_bf16x2(v0, v1);
        }
        sts128(addr, make_uint4(o[0], o[1], o[2], o[3]));
    }
}

// kSolo: one tile per CTA (a tensor of no more tiles than SMs). Both groups work on it: the first normalises x, the second z, into
// its own z buffer, so that the raw row is still there for the residual, and each takes half of every thread's output. The chain of
// one thread's steps is what such a launch takes: N = 37 / 128, in a block, 9.4 / 7.6 -> 5.7 / 6.1 us.
template <int C, bool kSolo>
__global__ void __launch_bounds__(kOutThreads, 1)
trimul_out_kernel(const __grid_constant__ CUtensorMap tmZ, const __grid_constant__ CUtensorMap tmX,
                  const __grid_constant__ CUtensorMap tmOut, const __grid_constant__ CUtensorMap tmWg,
                  const __grid_constant__ CUtensorMap tmWz, const __nv_bfloat16* __restrict__ ln_in_w,
                  const __nv_bfloat16* __restrict__ ln_in_b, const __nv_bfloat16* __restrict__ ln_out_w,
                  const __nv_bfloat16* __restrict__ ln_out_b, int B, int R, int N, int x_line_shift,
                  int add_residual, int* status) {
    using Sm = OutSmem<C>;
    constexpr int kTm = 2 * C;   // tensor-memory columns of a group: gate, update
    constexpr int CH = C / 2;   // channels per thread
    extern __shared__ uint8_t smem_raw[];
    const uint32_t sbase = (smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t* gbase = smem_raw + (sbase - smem_u32(smem_raw));
    float* prm = reinterpret_cast<float*>(gbase + Sm::kParams);
    const uint32_t bars = sbase + Sm::kBars;
    const uint32_t w_full = bars;
    // The x buffer is free as soon as the group's GEMMs have read it (the result goes over the z buffer), so
    // the next x tile is fetched during the epilogue; the z buffer is free once the output store has read it,
    // and its next tile lands while the group gathers and normalises x. Fetched together after the store,
    // the two loads cost every tile 2200 cycles of waiting.
    auto x_full = [&](int g) { return bars + 8u * (1 + g); };   // TMA landed: x tile
    auto z_empty = [&](int g) { return bars + 8u * (3 + g); };  // output store has read the z buffer
    auto a_ready = [&](int g) { return bars + 8u * (5 + g); };  // both A operands written
    auto d_full = [&](int g) { return bars + 8u * (7 + g); };   // MMAs of the group's tile done
    auto z_full = [&](int g) { return bars + 8u * (9 + g); };   // TMA landed: z tile
    auto x_empty = [&](int g) { return bars + 8u * (11 + g); };  // MMAs have read the x buffer
    auto out_ready = [&](int g) { return bars + 8u * (13 + g); };  // the group's result lies in the z buffer
    volatile uint32_t* tmem_ptr = reinterpret_cast<volatile uint32_t*>(gbase + Sm::kBars + 128);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(gbase + Sm::kBars + 132);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int tiles_per_line = (N + kRows - 1) / kRows;
    const long long num_tiles = (long long)B * R * tiles_per_line;
    // tiles of this CTA alternate between the two groups: local tile index lt -> group lt & 1
    const long long my_tiles = tiles_of_block(num_tiles);

    if (threadIdx.x == 0) {
        mbar_init(w_full, 1);
        for (int g = 0; g < 2; ++g) {
            mbar_init(x_full(g), 1);
            mbar_init(z_full(g), 1);
            mbar_init(x_empty(g), 1);
            mbar_init(z_empty(g), 1);
            mbar_init(a_ready(g), 8);
            mbar_init(d_full(g), 1);
            mbar_init(out_ready(g), kSolo ? 16 : 8);
        }
        *abort_flag = 0;
        mbar_fence_init();
        prefetch_tmap(&tmZ);
        prefetch_tmap(&tmX);
        prefetch_tmap(&tmOut);
    }
    if (threadIdx.x < C) {
        prm[threadIdx.x] = __bfloat162float(ln_in_w[threadIdx.x]);
        prm[128 + threadIdx.x] = __bfloat162float(ln_in_b[threadIdx.x]);
        prm[256 + threadIdx.x] = __bfloat162float(ln_out_w[threadIdx.x]);
        prm[384 + threadIdx.x] = __bfloat162float(ln_out_b[threadIdx.x]);
    }
    if (warp == 1) {
        tmem_alloc(smem_u32((const void*)tmem_ptr), 2 * kTm);
        tmem_relinquish();
    }
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem_base = *tmem_ptr;
    grid_trigger();
    if (warp >= 1) grid_wait();
    if (warp < 4) asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kOutRegsIssue));
    else asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kOutRegsRows));

    if (warp == 0) {
        // ---------------------------------------------------------------- TMA producer
        if (elect_one()) {
            mbar_arrive_expect_tx(w_full, 2 * Sm::kWBytes);
            for (int kb = 0; kb < C / 64; ++kb) {
                tma_load_2d(sbase + Sm::kWg + kb * C * 128, &tmWg, w_full, kb * 64, 0);
                tma_load_2d(sbase + Sm::kWz + kb * C * 128, &tmWz, w_full, kb * 64, 0);
            }
            grid_wait();
            TileWalk tw(blockIdx.x, gridDim.x, R, tiles_per_line);
            for (long long lt = 0; lt < my_tiles; ++lt, tw.next()) {
                const int g = (int)(lt & 1);
                const uint32_t use = (uint32_t)(lt >> 1);
                const int t0 = tw.tile * kRows;
                if (!mbar_wait(x_empty(g), (use & 1u) ^ 1u, abort_flag)) {
                    report_wait_failure(status, abort_flag, kKidOut, 1);
                    break;
                }
                // x tile: all 128 channels of positions (fixed, t0 .. t0+127), layout [c][j]
                mbar_arrive_expect_tx(x_full(g), tile_bytes<C>());
                tma_load_5d(sbase + Sm::kX + g * tile_bytes<C>(), &tmX, x_full(g), t0,
                            tw.line & (int)((1u << x_line_shift) - 1u), tw.line >> x_line_shift, 0, tw.b);
                if (!mbar_wait(z_empty(g), (use & 1u) ^ 1u, abort_flag)) {
                    report_wait_failure(status, abort_flag, kKidOut, 6);
                    break;
                }
                mbar_arrive_expect_tx(z_full(g), tile_bytes<C>());
                const uint32_t zdst = sbase + Sm::kZ + g * tile_bytes<C>();
                for (int kb = 0; kb < C / 64; ++kb)
                    tma_load_3d(zdst + kb * kKBlockBytes, &tmZ, z_full(g), kb * 64, t0, tw.b * R + tw.line);
            }
        }
    } else if (warp <= 2) {
        // ---------------------------------------------------------------- GEMMs and stores of row group g
        if (elect_one()) {
            const int g = warp - 1;
            constexpr uint32_t idesc = idesc_bf16_f32(128, C);
            const uint32_t ztile = sbase + Sm::kZ + g * tile_bytes<C>();
            bool ok = mbar_wait(w_full, 0, abort_flag);
            if (!ok) report_wait_failure(status, abort_flag, kKidOut, 2);
            TileWalk tw(blockIdx.x + g * gridDim.x, 2 * gridDim.x, R, tiles_per_line);
            for (long long lt = g; lt < my_tiles && ok; lt += 2, tw.next()) {
                const uint32_t par = (uint32_t)(lt >> 1) & 1u;
                if (kSolo && !mbar_wait(a_ready(1), 0, abort_flag)) {
                    report_wait_failure(status, abort_flag, kKidOut, 9);
                    break;
                }
                if (!kSolo && !mbar_wait(a_ready(g), par, abort_flag)) {
                    report_wait_failure(status, abort_flag, kKidOut, 3);
                    break;
                }
                tc_fence_after_sync();
                // gate = LN_in(z) W_g^T -> columns [0,C); update = LN_out(x) W_z^T -> [C,2C)
                mma_rows<C>(tmem_base + g * kTm, kSolo ? ztile + tile_bytes<C>() : ztile, sbase + Sm::kWg, C * 128, idesc, false);
                if (kSolo && !mbar_wait(a_ready(0), 0, abort_flag)) {
                    report_wait_failure(status, abort_flag, kKidOut, 3);
                    break;
                }
                tc_fence_after_sync();
                mma_rows<C>(tmem_base + g * kTm + C, sbase + Sm::kX + g * tile_bytes<C>(), sbase + Sm::kWz, C * 128, idesc,
                            false);
                mma_commit(d_full(g));
                mma_commit(x_empty(g));
                if (!mbar_wait(out_ready(g), par, abort_flag)) {
                    report_wait_failure(status, abort_flag, kKidOut, 8);
                    break;
                }
                for (int kb = 0; kb < C / 64; ++kb)
                    tma_store_3d(&tmOut, ztile + kb * kKBlockBytes, kb * 64, tw.tile * kRows, tw.b * R + tw.line);
                tma_store_commit();
                tma_store_wait_read<0>();
                mbar_arrive(z_empty(g));
            }
            tma_store_wait_all<0>();
        }
    } else if (warp >= 4) {
        // ---------------------------------------------------------------- two row groups
        const int g = (warp - 4) >> 3;
        const int quad = warp & 3;
        const int half = ((warp - 4) >> 2) & 1;   // which half of the row's channels
        const int row = quad * 32 + lane;
        const uint32_t ztile = sbase + Sm::kZ + g * tile_bytes<C>();
        const uint32_t xtile = sbase + Sm::kX + g * tile_bytes<C>();
        float* xch = reinterpret_cast<float*>(gbase + Sm::kXch) + g * 512;
        if constexpr (kSolo) {
            const uint32_t ztile0 = sbase + Sm::kZ, ztile1 = ztile0 + tile_bytes<C>();
            bool ok = mbar_wait(g == 0 ? x_full(0) : z_full(0), 0, abort_flag);
            if (!ok && lane == 0) report_wait_failure(status, abort_flag, kKidOut, g == 0 ? 4 : 7);
            float mean, rstd;
            if (g == 0) {
                uint32_t xraw[CH / 2];
                gather_column<CH>(xtile + row * 2 + half * (CH * 256), xraw);
                half_row_stats_xwarp<C, false>(xraw, row, half, xch, 1, 256, mean, rstd);
                store_normalized_half_row<C>(xtile, row, half, xraw, mean, rstd, prm + 256, prm + 384);
            } else {
                uint32_t zraw[CH / 2];
                load_half_row<C>(ztile0, row, half, zraw);
                half_row_stats_xwarp<C>(zraw, row, half, xch, 2, 256, mean, rstd);
                store_normalized_half_row<C>(ztile1, row, half, zraw, mean, rstd, prm, prm + 128);
            }
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) mbar_arrive(a_ready(g));
            if (ok && !(ok = mbar_wait(z_full(0), 0, abort_flag) && mbar_wait(d_full(0), 0, abort_flag)) && lane == 0)
                report_wait_failure(status, abort_flag, kKidOut, 5);
            if (ok) {
                tc_fence_after_sync();
                const int c0 = half * CH + g * (CH / 2);   // this thread's CH / 2 channels
                const uint32_t taddr = tmem_base + ((uint32_t)(quad * 32) << 16) + c0;
#pragma unroll
                for (int cb = 0; cb < CH / 32; ++cb) {
                    uint32_t gate[16], upd[16];
                    tmem_ld16(taddr + cb * 16, gate);
                    tmem_ld16(taddr + C + cb * 16, upd);
                    tmem_ld_wait();
                    update_channels(ztile0, row, c0 / 8 + cb * 2, gate, upd, add_residual);
                }
                tc_fence_before_sync();
                fence_proxy_async_smem();
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(out_ready(0));
        }
        for (long long lt = kSolo ? my_tiles : g; lt < my_tiles; lt += 2) {
            const uint32_t use = (uint32_t)(lt >> 1);
            if (!mbar_wait(x_full(g), use & 1u, abort_flag)) {
                if (lane == 0) report_wait_failure(status, abort_flag, kKidOut, 4);
                break;
            }
            float mean, rstd;
            // --- half of the x column of this position: [c][j] layout, stride 256 B
            {
                uint32_t xraw[CH / 2];
                gather_column<CH>(xtile + row * 2 + half * (CH * 256), xraw);
                // (behind its first barrier everyone has read its column: rows may overwrite the buffer)
                half_row_stats_xwarp<C, false>(xraw, row, half, xch, 1 + g, 256, mean, rstd);
                store_normalized_half_row<C>(xtile, row, half, xraw, mean, rstd, prm + 256, prm + 384);
            }
            // --- z row: keep the raw values for the residual, normalise in place (A operand 1)
            if (!mbar_wait(z_full(g), use & 1u, abort_flag)) {
                if (lane == 0) report_wait_failure(status, abort_flag, kKidOut, 7);
                break;
            }
            uint32_t zraw[CH / 2];
            load_half_row<C>(ztile, row, half, zraw);
            half_row_stats_xwarp<C>(zraw, row, half, xch, 1 + g, 256, mean, rstd);
            store_normalized_half_row<C>(ztile, row, half, zraw, mean, rstd, prm, prm + 128);
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) mbar_arrive(a_ready(g));
            // --- wait for both GEMMs, combine, write the output tile over the z buffer
            if (!mbar_wait(d_full(g), use & 1u, abort_flag)) {
                if (lane == 0) report_wait_failure(status, abort_flag, kKidOut, 5);
                break;
            }
            tc_fence_after_sync();
            const uint32_t taddr = tmem_base + ((uint32_t)(quad * 32) << 16) + g * kTm + half * CH;
#pragma unroll
            for (int cb = 0; cb < CH / 16; ++cb) {  // 16 channels per step
                uint32_t gate[16], upd[16];
                tmem_ld16(taddr + cb * 16, gate);
                tmem_ld16(taddr + C + cb * 16, upd);
                tmem_ld_wait();
#pragma unroll
                for (int ch = 0; ch < 2; ++ch) {
                    uint32_t o[4];
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const int e = ch * 8 + j * 2;
                        const uint32_t zr = zraw[cb * 8 + ch * 4 + j];
                        float v0 = sigmoid_fast(__uint_as_float(gate[e])) * __uint_as_float(upd[e]);
                        float v1 = sigmoid_fast(__uint_as_float(gate[e + 1])) * __uint_as_float(upd[e + 1]);
                        if (add_residual) {
                            v0 += bf16lo(zr);
                            v1 += bf16hi(zr);
                        }
                        o[j] = pack_bf16x2(v0, v1);
                    }
                    sts128(chunk_addr(ztile, row, half * (CH / 8) + cb * 2 + ch), make_uint4(o[0], o[1], o[2], o[3]));
                }
            }
            tc_fence_before_sync();
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) mbar_arrive(out_ready(g));
        }
    }

    tc_fence_before_sync();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after_sync();
        tmem_dealloc(tmem_base, 2 * kTm);
    }
}

int weight_tmap(CUtensorMap* m, const void* w, int C) {
    uint64_t dims[2] = {(uint64_t)C, (uint64_t)C};
    uint64_t str[1] = {(uint64_t)C * 2};
    uint32_t box[2] = {64, (uint32_t)C};
    return make_tmap_bf16(m, w, 2, dims, str, box, true);
}

// z as lines: {c, position, b*R + line}
int line_tmap(CUtensorMap* m, const void* z, int B, int R, int N, int C) {
    uint64_t dims[3] = {(uint64_t)C, (uint64_t)N, (uint64_t)B * R};
    uint64_t str[2] = {(uint64_t)C * 2, (uint64_t)N * C * 2};
    uint32_t box[3] = {64, 128, 1};
    return make_tmap_bf16(m, z, 3, dims, str, box, 1);
}

template <int C, bool kOutgoing>
int launch_in(int grid, cudaStream_t st, const CUtensorMap& tmZ, const CUtensorMap* w, const __nv_bfloat16* mask,
              const __nv_bfloat16* lw, const __nv_bfloat16* lb, __nv_bfloat16* a_t, __nv_bfloat16* b_t, int B, int R,
              int N, const PlaneLayout& pl, int wide) {
    static PerDeviceOnce configured;
    if (!configured.done()) {
        OF3_CUDA_CHECK(cudaFuncSetAttribute(trimul_in_kernel<C, kOutgoing>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                            InSmem<C>::kDyn));
        configured.mark();
    }
    LaunchScope scope(kKidIn, st);
    OF3_CUDA_CHECK(launch_chained(trimul_in_kernel<C, kOutgoing>, grid, kInThreads<C>, InSmem<C>::kDyn, st, tmZ, w[0], w[1],
                                  w[2], w[3], mask, lw, lb, a_t, b_t, B, R, N, pl, wide, device_status_ptr()));
    return OF3_OK;
}
template <bool kOutgoing>
int launch_in_rows(int grid, cudaStream_t st, const CUtensorMap& tmZ, const CUtensorMap* w, const __nv_bfloat16* mask,
                   const __nv_bfloat16* lw, const __nv_bfloat16* lb, __nv_bfloat16* a_t, __nv_bfloat16* b_t, int B, int R,
                   int N, const PlaneLayout& pl) {
    static PerDeviceOnce configured;
    if (!configured.done()) {
        OF3_CUDA_CHECK(cudaFuncSetAttribute(trimul_in_rows_kernel<kOutgoing>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                            InSmem<128>::kDyn));
        configured.mark();
    }
    LaunchScope scope(kKidIn, st);
    OF3_CUDA_CHECK(launch_chained(trimul_in_rows_kernel<kOutgoing>, grid, kInRowsThreads, InSmem<128>::kDyn, st, tmZ, w[0],
                                  w[1], w[2], w[3], mask, lw, lb, a_t, b_t, B, R, N, pl, device_status_ptr()));
    return OF3_OK;
}
template <int C, bool kSolo>
int launch_out(int grid, cudaStream_t st, const CUtensorMap& tmZ, const CUtensorMap& tmX, const CUtensorMap& tmOut,
               const CUtensorMap& tmWg, const CUtensorMap& tmWz, const of3_trimul_params* p, int B, int R, int N,
               int x_line_shift, int add_residual) {
    static PerDeviceOnce configured;
    if (!configured.done()) {
        cudaFuncAttributes fa;   // a block launched with fewer registers would wait for the split for good
        OF3_CUDA_CHECK(cudaFuncGetAttributes(&fa, trimul_out_kernel<C, kSolo>));
        OF3_REQUIRE(fa.numRegs == kOutRegsLaunch, OF3_ERR_DRIVER, "trimul_out is built with %d registers, not %d", fa.numRegs,
                    kOutRegsLaunch);
        OF3_CUDA_CHECK(cudaFuncSetAttribute(trimul_out_kernel<C, kSolo>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                            OutSmem<C>::kDyn));
        configured.mark();
    }
    typedef const __nv_bfloat16* P;
    LaunchScope scope(kKidOut, st);
    OF3_CUDA_CHECK(launch_chained(trimul_out_kernel<C, kSolo>, grid, kOutThreads, OutSmem<C>::kDyn, st, tmZ, tmX, tmOut, tmWg, tmWz,
                                  (P)p->ln_in_w, (P)p->ln_in_b, (P)p->ln_out_w, (P)p->ln_out_b, B, R, N, x_line_shift, add_residual,
                                  device_status_ptr()));
    return OF3_OK;
}

}  // namespace

bool trimul_supported(int c_z, int c_h) { return c_z == c_h && (c_z == 128 || c_z == 64); }

// a_t[(b*C + c)][line][k], b_t likewise, from R lines of N positions per sample: z is [B][R][N][C].
// transposed_walk: z is [B][N][R][C] and a line runs along its FIRST index (line = second index),
// which makes the incoming update the same K-major contraction as the outgoing one; with R != N this
// is a row shard of N rows seen as R lines of N positions each.
static int project(const __nv_bfloat16* z, const __nv_bfloat16* mask, __nv_bfloat16* a_t, __nv_bfloat16* b_t, int B, int R,
                   int N, const PlaneLayout& pl, bool transposed_walk, const of3_trimul_params* p, cudaStream_t st, int C) {
    OF3_REQUIRE(((uintptr_t)z & 15) == 0, OF3_ERR_ALIGN, "trimul: z must be 16-byte aligned");
    int rc;
    CUtensorMap tmZ, tmW[4];
    if (!transposed_walk) {
        if ((rc = line_tmap(&tmZ, z, B, R, N, C))) return rc;
    } else {  // {c, second (line), first (position), b}
        uint64_t dims[4] = {(uint64_t)C, (uint64_t)R, (uint64_t)N, (uint64_t)B};
        uint64_t str[3] = {(uint64_t)C * 2, (uint64_t)R * C * 2, (uint64_t)N * R * C * 2};
        uint32_t box[4] = {64, 1, 128, 1};
        if ((rc = make_tmap_bf16(&tmZ, z, 4, dims, str, box, 1))) return rc;
    }
    const void* w4[4] = {p->w_a_p, p->w_a_g, p->w_b_p, p->w_b_g};
    for (int i = 0; i < 4; ++i)
        if ((rc = weight_tmap(&tmW[i], w4[i], C))) return rc;
    const long long tiles = (long long)B * R * ceil_div(N, kRows);
    const int grid = (int)(tiles < sm_count() ? tiles : sm_count());
    // 32-byte stores need every channel row of a_t / b_t to start on a 32-byte boundary
    const int wide = (pl.ld % 16 == 0 && pl.group_stride % 16 == 0 && ((uintptr_t)a_t & 31) == 0 && ((uintptr_t)b_t & 31) == 0) ? 1 : 0;
    // a channel plane of R lines: beyond about one 2 MB page the kernel whose stores stay inside one plane wins
    const bool planes_far_apart = C == 128 && pl.chan_stride * (long long)sizeof(__nv_bfloat16) > (2LL << 20);
    const __nv_bfloat16* lw = (const __nv_bfloat16*)p->ln_in_w;
    const __nv_bfloat16* lb = (const __nv_bfloat16*)p->ln_in_b;
    if (planes_far_apart)
        return transposed_walk ? launch_in_rows<false>(grid, st, tmZ, tmW, mask, lw, lb, a_t, b_t, B, R, N, pl)
                               : launch_in_rows<true>(grid, st, tmZ, tmW, mask, lw, lb, a_t, b_t, B, R, N, pl);
    if (C == 128)
        return transposed_walk ? launch_in<128, false>(grid, st, tmZ, tmW, mask, lw, lb, a_t, b_t, B, R, N, pl, wide)
                               : launch_in<128, true>(grid, st, tmZ, tmW, mask, lw, lb, a_t, b_t, B, R, N, pl, wide);
    return transposed_walk ? launch_in<64, false>(grid, st, tmZ, tmW, mask, lw, lb, a_t, b_t, B, R, N, pl, wide)
                           : launch_in<64, true>(grid, st, tmZ, tmW, mask, lw, lb, a_t, b_t, B, R, N, pl, wide);
}

// groups > 1: the C channels are written as `groups` equal groups, group q of a_t at
// a_t + q * group_stride (b_t likewise), so that each group can be sent to another rank as one block.
int trimul_project(const __nv_bfloat16* z, const __nv_bfloat16* mask, __nv_bfloat16* a_t, __nv_bfloat16* b_t,
                   int B, int R, int N, int ld, bool transposed_walk, const of3_trimul_params* p,
                   cudaStream_t st, int groups, long long group_stride, int C) {
    OF3_REQUIRE(groups == 1 || groups == 2 || groups == 4 || groups == 8, OF3_ERR_ARG,
                "trimul: channel groups must be 1, 2, 4 or 8 (got %d)", groups);
    return project(z, mask, a_t, b_t, B, R, N, plane_layout(R, ld, C, groups, group_stride), transposed_walk, p, st, C);
}

// LN_out(x) -> linear_z, gate from LN_in(z), residual: the part of the update after the contraction,
// on R lines of z with x_t[b*C + c][line][j] (pitch ld)
static int output(const __nv_bfloat16* z, __nv_bfloat16* out, const __nv_bfloat16* x_t, int B, int R, int N,
                  const PlaneLayout& pl, int add_residual, const of3_trimul_params* p, cudaStream_t st, int C) {
    OF3_REQUIRE(((uintptr_t)z & 15) == 0 && ((uintptr_t)out & 15) == 0 && ((uintptr_t)x_t & 15) == 0, OF3_ERR_ALIGN,
                "trimul: z/out/x must be 16-byte aligned");
    int rc;
    CUtensorMap tmZ, tmOut, tmX, tmWg, tmWz;
    if ((rc = line_tmap(&tmZ, z, B, R, N, C))) return rc;
    if ((rc = line_tmap(&tmOut, out, B, R, N, C))) return rc;
    {   // {position j, line of its block, block, channel, sample}: box = 128 positions of one line x C channels, no swizzle
        const bool blocked = pl.line_shift == kLineBlockShift;
        uint64_t dims[5] = {(uint64_t)N, (uint64_t)(blocked ? kLineBlock : R), (uint64_t)(blocked ? ceil_div(R, kLineBlock) : 1),
                            (uint64_t)C, (uint64_t)B};
        uint64_t str[4] = {(uint64_t)pl.ld * 2, (uint64_t)(blocked ? pl.block_stride : pl.sample_stride) * 2,
                           (uint64_t)pl.chan_stride * 2, (uint64_t)pl.sample_stride * 2};
        uint32_t box[5] = {128, 1, 1, (uint32_t)C, 1};
        if ((rc = make_tmap_bf16(&tmX, x_t, 5, dims, str, box, 0))) return rc;
    }
    if ((rc = weight_tmap(&tmWg, p->w_g, C))) return rc;
    if ((rc = weight_tmap(&tmWz, p->w_z, C))) return rc;
    const long long tiles = (long long)B * R * ceil_div(N, kRows);
    const int grid = (int)(tiles < sm_count() ? tiles : sm_count());
    const bool solo = tiles <= grid;
    auto* launch = C == 128 ? (solo ? launch_out<128, true> : launch_out<128, false>) : (solo ? launch_out<64, true> : launch_out<64, false>);
    return launch(grid, st, tmZ, tmX, tmOut, tmWg, tmWz, p, B, R, N, pl.line_shift, add_residual);
}

// the same on planes [b*C + c][line][ld]
int trimul_output(const __nv_bfloat16* z, __nv_bfloat16* out, const __nv_bfloat16* x_t, int B, int R, int N, int ld,
                  int add_residual, const of3_trimul_params* p, cudaStream_t st, int C) {
    return output(z, out, x_t, B, R, N, plane_layout(R, ld, C, 1, 0), add_residual, p, st, C);
}

int trimul(const __nv_bfloat16* z, const __nv_bfloat16* mask, __nv_bfloat16* out, int B, int N, int C,
           int flags, const of3_trimul_params* p, Arena& ws, cudaStream_t st) {
    const int ld = (int)align_up(N, 16);   // (32-byte stores)
    const PlaneLayout pl = blocked_layout(N, ld, C);
    const size_t bytes = (size_t)B * pl.sample_stride * sizeof(__nv_bfloat16);
    __nv_bfloat16* a_t = (__nv_bfloat16*)ws.take(bytes);
    __nv_bfloat16* b_t = (__nv_bfloat16*)ws.take(bytes);
    __nv_bfloat16* x_t = (__nv_bfloat16*)ws.take(bytes);
    if (!ws.base) return OF3_OK;
    OF3_REQUIRE(ws.ok(), OF3_ERR_WORKSPACE, "trimul: workspace too small (%zu needed)", ws.off);
    const bool outgoing = (flags & OF3_FLAG_OUTGOING) != 0;
    int rc = project(z, mask, a_t, b_t, B, N, N, pl, !outgoing, p, st, C);
    if (rc) return rc;
    if ((rc = contract_blocked_bf16(a_t, b_t, x_t, B, C, N, ld, st))) return rc;
    return output(z, out, x_t, B, N, N, pl, (flags & OF3_FLAG_ADD_RESIDUAL) ? 1 : 0, p, st, C);
}

}  // namespace fast
}  // namespace of3
