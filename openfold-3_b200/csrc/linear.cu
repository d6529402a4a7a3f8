// Linear layers on tcgen05 with their consumers in the epilogue (bf16 operands, fp32 accumulation): the projections of
// the single track (c_s = 384) and of the diffusion token stack (c_a = 768, c_s = 384).
//
//   y = x W^T, x [rows][k], W [n][k], both K-major. Persistent CTA: warp 0 TMA producer (128-byte swizzled k-blocks of
//   64), warp 1 MMA issuer (128 x BN x 16, accumulators double-buffered in TMEM), warps 2..17 the epilogue (four per 32
//   rows, each a quarter of the columns; thread = row).
//
// What bounds them: a few hundred 128-row tiles with k = 384 .. 1536, and for short sequences launch and fill latency. At 3840
// rows of 768 a CTA has two to four tiles of the images, gate / up and conditioning projections, of which the epilogues are a
// quarter to a third (images 19.3 us, 14.2 with nothing computed or stored there; conditioning 16.0, 10.9 without stores), and
// one of the output projections (120 tiles of 192 columns), whose panels arrive at 115 GB/s per SM (64 bytes per cycle). The
// separate passes that would read the products back (attention operand images, silu * mul, gates, residuals) cost as much again
// as 11 launches per block.
// So the product leaves the SM in the form its consumer reads, and BN is chosen per call (pick_bn).
#include <type_traits>

#include "linear.cuh"
#include "modules.cuh"
#include "rowtile.cuh"
#include "runtime.cuh"
#include "single_attn.cuh"

namespace of3 {
namespace fast {
namespace {

using namespace umma;
typedef __nv_bfloat16 bf16;

constexpr int kKid = 10;
constexpr int kBM = 128, kBK = 64;
constexpr int kEpiParts = 4;   // epilogue warps per 32 rows, each with its part of the columns
constexpr int kThreads = 32 * (2 + 4 * kEpiParts);
constexpr float kLog2e = 1.4426950408889634f;

// kEpiStaged: kEpiResidual with the gate's, the residual's and the output's tile in shared memory, moved by TMA. Rows of the
// caller's tensors that lie in different lanes cost the memory pipe a line at a time, behind the operand panels: at 3840 rows of
// 768 the gates of a tile of 192 columns arrived 7.4 us after its start, when its product of k = 768 was done at 4.5 us. Staged,
// gates and product are there after 5 and 6 us, and the tile ends at 8.3 instead of 11.9 us (k = 1536: 12.3 instead of 15.2).
// Step of 24 blocks, c_a = 768: 5 x 1024 tokens 4334 -> 4225 us, 5 x 768 2995 -> 2924, 5 x 500 2249 -> 2214, 3 x 300 1403 ->
// 1390, 111 923 both. With BN = 256 two stages of operands would be left: at most 192.
enum Epi { kEpiStore, kEpiImages, kEpiSwiglu, kEpiResidual, kEpiStaged };

template <int BN, int EPI>
struct LinCfg {
    static constexpr int kABytes = kBM * kBK * 2;
    static constexpr int kStageBytes = kABytes + BN * kBK * 2;
    static constexpr int kPlaneBytes = EPI == kEpiStaged ? kBM * BN * 2 : 0;   // a tile of the gate, and one of the residual / output
    static constexpr int kStages = EPI == kEpiStaged ? (BN == 192 ? 3 : (BN == 128 ? 5 : 8))
                                                     : (BN == 256 ? 4 : (BN == 192 ? 5 : (BN == 128 ? 6 : 8)));
    static constexpr int kAccStride = BN <= 64 ? 64 : (BN <= 128 ? 128 : 256);
    static constexpr int kTmemCols = 2 * kAccStride;
    static constexpr int kPlanes = kStages * kStageBytes;            // offsets
    static constexpr int kBars = kPlanes + 2 * kPlaneBytes;
    static constexpr int kSmemBytes = kBars + 1024 + 256;
    static_assert(kSmemBytes <= 227 * 1024, "shared memory of a block");
};

struct LinMaps {
    CUtensorMap a, w[4];
};
struct StagedMaps : LinMaps {
    CUtensorMap gate, residual, out;   // boxes of 64 columns and 128 rows
};
struct EpiArgs {
    // kEpiStore
    bf16* y;
    int raw_slice;
    // kEpiImages
    AttnImages im;
    int kind[4];
    float qscale;
    // kEpiSwiglu, kEpiResidual
    bf16* out;
    const bf16 *residual, *gate, *gate_bias, *mask;
};

// One column group of 16 of this thread's row as attention operand images; `kind` is uniform over the tile.
template <int D>
__device__ __forceinline__ void store_images(const AttnImages& im, int kind, float qscale, const uint32_t (&r)[16],
                                             int col0, long long row, long long bb, int pos) {
    constexpr int KD = SingleImage<D>::kKD, DV = SingleImage<D>::kDV;
    const int HD = im.H * D;
    if (kind == kOutG) {
        uint32_t o[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) o[e] = pack_bf16x2(__uint_as_float(r[2 * e]), __uint_as_float(r[2 * e + 1]));
        stg256(im.g + row * HD + col0, o);
        return;
    }
    const int n = im.rows_per_sample;
    const int nkb = (n + kSingleBK - 1) / kSingleBK, n_qt = (n + kSingleBQ - 1) / kSingleBQ;
    const int pad = nkb * kSingleBK - n;   // keys past the end of the last block: zeros, written by the first rows
    if constexpr (D % 16 == 0 && KD == 64) {
        // 16 channels of one head: two neighbouring chunks of the row, which the swizzle keeps inside one 32-byte sector. Rows of
        // different lanes are different lines, and the memory pipe takes a line at a time: two stores of 16 bytes cost twice
        // one of 32 (5 x 768 tokens: 21.5 -> 19.2 us per launch).
        if (kind != kOutV) {
            const int h = col0 / D, c = (col0 - h * D) >> 3;
            float f[16];
#pragma unroll
            for (int e = 0; e < 16; ++e) f[e] = __uint_as_float(r[e]);
            if (kind == kOutQ) {
                if (im.q_bias) {
                    uint32_t b[8];
                    ld_row16_any(im.q_bias + col0, b);
#pragma unroll
                    for (int e = 0; e < 16; ++e) f[e] += (e & 1) ? bf16hi(b[e >> 1]) : bf16lo(b[e >> 1]);
                }
#pragma unroll
                for (int e = 0; e < 16; ++e) f[e] *= qscale;
            }
            uint32_t o[8];
#pragma unroll
            for (int e = 0; e < 4; ++e) {   // odd rows: the chunks change places
                const uint32_t lo = pack_bf16x2(f[2 * e], f[2 * e + 1]), hi = pack_bf16x2(f[8 + 2 * e], f[9 + 2 * e]);
                o[e] = pos & 1 ? hi : lo;
                o[4 + e] = pos & 1 ? lo : hi;
            }
            if (kind == kOutQ) {
                uint8_t* t = reinterpret_cast<uint8_t*>(im.q) +
                             ((bb * im.H + h) * n_qt + (pos >> 7)) * (long long)(kSingleBQ * KD * 2);
                stg256(t + (single_chunk_off<KD>(pos & 127, c) & ~31u), o);
            } else {
                uint8_t* t0 = reinterpret_cast<uint8_t*>(im.k) + (bb * im.H + h) * nkb * (long long)(kSingleBK * KD * 2);
                stg256(t0 + (pos >> 5) * (long long)(kSingleBK * KD * 2) + (single_chunk_off<KD>(pos & 31, c) & ~31u), o);
                const uint32_t zero[8] = {};
                for (int p = n + pos; p < n + pad; p += n)
                    stg256(t0 + (p >> 5) * (long long)(kSingleBK * KD * 2) + (single_chunk_off<KD>(p & 31, c) & ~31u), zero);
            }
            return;
        }
    }
#pragma unroll
    for (int half = 0; half < 2; ++half) {
        const int col = col0 + half * 8;
        const int h = col / D, d0 = col - h * D;
        if (kind == kOutV) {
            // tile [DV][32 keys], 64-byte rows: a warp's 32 consecutive keys fill one row of one tile
            auto put = [&](int p, bool live) {
                const int kc = (p & 31) >> 3;
                bf16* tile = im.v + (((bb * im.H + h) * nkb + (p >> 5)) * (long long)DV) * kSingleBK;
#pragma unroll
                for (int e = 0; e < 8; ++e) {
                    const int dd = d0 + e;
                    tile[dd * kSingleBK + (((kc ^ ((dd >> 1) & 3)) << 3) | (p & 7))] =
                        __float2bfloat16_rn(live ? __uint_as_float(r[half * 8 + e]) : 0.f);
                }
            };
            put(pos, true);
            for (int p = n + pos; p < n + pad; p += n) put(p, false);
            continue;
        }
        float f[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) f[e] = __uint_as_float(r[half * 8 + e]);
        if (kind == kOutQ) {
            if (im.q_bias) {
                uint32_t b[4];
                ld_row8_any(im.q_bias + col, b);
                #pragma unroll
                for (int e = 0; e < 8; ++e) f[e] += (e & 1) ? bf16hi(b[e >> 1]) : bf16lo(b[e >> 1]);
            }
#pragma unroll
            for (int e = 0; e < 8; ++e) f[e] *= qscale;
        }
        const uint4 v = make_uint4(pack_bf16x2(f[0], f[1]), pack_bf16x2(f[2], f[3]), pack_bf16x2(f[4], f[5]),
                                   pack_bf16x2(f[6], f[7]));
        const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
        const int c = d0 >> 3;
        const bool last = D < KD && D <= 32 && c == D / 8 - 1;   // 24 channels: chunk 3 of the row pads K with zeros
        if (kind == kOutQ) {
            uint8_t* t = reinterpret_cast<uint8_t*>(im.q) +
                         ((bb * im.H + h) * n_qt + (pos >> 7)) * (long long)(kSingleBQ * KD * 2);
            *reinterpret_cast<uint4*>(t + single_chunk_off<KD>(pos & 127, c)) = v;
            if (last) *reinterpret_cast<uint4*>(t + single_chunk_off<KD>(pos & 127, c + 1)) = zero;
        } else {
            uint8_t* t0 = reinterpret_cast<uint8_t*>(im.k) + (bb * im.H + h) * nkb * (long long)(kSingleBK * KD * 2);
            uint8_t* t = t0 + (pos >> 5) * (long long)(kSingleBK * KD * 2);
            *reinterpret_cast<uint4*>(t + single_chunk_off<KD>(pos & 31, c)) = v;
            if (last) *reinterpret_cast<uint4*>(t + single_chunk_off<KD>(pos & 31, c + 1)) = zero;
            for (int p = n + pos; p < n + pad; p += n) {
                uint8_t* tp = t0 + (p >> 5) * (long long)(kSingleBK * KD * 2);
                *reinterpret_cast<uint4*>(tp + single_chunk_off<KD>(p & 31, c)) = zero;
                if (last) *reinterpret_cast<uint4*>(tp + single_chunk_off<KD>(p & 31, c + 1)) = zero;
            }
        }
    }
}

// A last wave of 256-wide tiles that takes at most half of the SMs runs as twice as many tiles of half the columns: a half tile takes
// about 0.6 of a whole one, whose time the wave otherwise costs. A step of 24 blocks whose wave has 64 tiles (5 x 768 tokens) 2959 ->
// 2920 us, 36 (5 x 1024) 4287 -> 4234, 20 (5 x 350) 1833 -> 1798; fuller waves stay whole and as fast (92 tiles, 5 x 500: 2231).
template <int BN, int EPI>
__host__ __device__ constexpr bool has_halves() { return BN == 256 && (EPI == kEpiImages || EPI == kEpiSwiglu); }

template <int BN, int EPI, int D>
__global__ void __launch_bounds__(kThreads, 1)
linear_kernel(const __grid_constant__ std::conditional_t<EPI == kEpiStaged, StagedMaps, LinMaps> maps, const EpiArgs ep,
              long long rows, int K, int n, int num_mats, int whole_tiles, int* status) {
    using Cfg = LinCfg<BN, EPI>;
    constexpr int S = Cfg::kStages;
    constexpr int kWRows = EPI == kEpiSwiglu ? BN / 2 : BN;   // rows of each weight matrix in a tile
    extern __shared__ uint8_t smem_raw[];
    const uint32_t sbase = (smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t* gbase = smem_raw + (sbase - smem_u32(smem_raw));
    const uint32_t bars = sbase + Cfg::kBars;
    auto full = [&](int s) { return bars + 8u * s; };
    auto empty = [&](int s) { return bars + 8u * (S + s); };
    auto tfull = [&](int a) { return bars + 8u * (2 * S + a); };
    auto tempty = [&](int a) { return bars + 8u * (2 * S + 2 + a); };
    const uint32_t planes_full = bars + 8u * (2 * S + 4);
    volatile uint32_t* tmem_ptr = reinterpret_cast<volatile uint32_t*>(gbase + Cfg::kBars + 8 * (2 * S + 5));
    volatile int* abort_flag = reinterpret_cast<volatile int*>(gbase + Cfg::kBars + 8 * (2 * S + 5) + 8);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int num_mt = (int)((rows + kBM - 1) / kBM);
    const int nt_per_mat = n / kWRows;
    // kEpiSwiglu: matrices 0 and 1 share a tile; otherwise a tile lies inside one matrix
    const int num_nt = EPI == kEpiSwiglu ? nt_per_mat : nt_per_mat * num_mats;
    const int num_kb = K / kBK;
    // The tiles from whole_tiles on come in two halves of their columns (kHalves)
    constexpr bool kHalves = has_halves<BN, EPI>();
    const int num_tiles = kHalves ? 2 * num_mt * num_nt - whole_tiles : num_mt * num_nt;
    // a tile: row tile mt (innermost: concurrent CTAs share the weight panel), matrix g, column tile inside it; which half
    struct Tile { int mt, g, nt, half; bool whole; };
    auto tile_of = [&](int t) {
        Tile c;
        c.whole = !kHalves || t < whole_tiles;
        c.half = 0;
        if (!c.whole) {
            c.half = (t - whole_tiles) & 1;
            t = whole_tiles + ((t - whole_tiles) >> 1);
        }
        c.mt = t % num_mt;
        const int q = t / num_mt;
        c.g = EPI == kEpiSwiglu ? 0 : q / nt_per_mat;
        c.nt = EPI == kEpiSwiglu ? q : q % nt_per_mat;
        return c;
    };

    if (threadIdx.x == 0) {
        for (int s = 0; s < S; ++s) {
            mbar_init(full(s), 1);
            mbar_init(empty(s), 1);
        }
        for (int a = 0; a < 2; ++a) {
            mbar_init(tfull(a), 1);
            mbar_init(tempty(a), 4 * kEpiParts);
        }
        mbar_init(planes_full, 1);
        *abort_flag = 0;
        mbar_fence_init();
        prefetch_tmap(&maps.a);
        prefetch_tmap(&maps.w[0]);
    }
    if (warp == 1) {
        tmem_alloc(smem_u32((const void*)tmem_ptr), Cfg::kTmemCols);
        tmem_relinquish();
    }
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    grid_trigger();
    const uint32_t tmem_base = *tmem_ptr;

    if (warp == 0) {
        // ---------------------------------------------------------------- TMA producer
        if (elect_one()) {
            auto load_w = [&](const Tile& c, int kb, int s) {
                const uint32_t sw = sbase + s * Cfg::kStageBytes + Cfg::kABytes;
                if constexpr (kHalves) {   // boxes of half a tile's rows
                    const int mats = EPI == kEpiSwiglu ? 2 : 1, boxes = c.whole ? 2 : 1;
                    for (int m = 0; m < mats; ++m)
                        for (int b = 0; b < boxes; ++b)
                            tma_load_2d(sw + (m * boxes + b) * (kWRows / 2) * 128, &maps.w[EPI == kEpiSwiglu ? m : c.g], full(s), kb * kBK,
                                        c.nt * kWRows + (b + c.half) * (kWRows / 2));
                } else if constexpr (EPI == kEpiSwiglu) {
                    tma_load_2d(sw, &maps.w[0], full(s), kb * kBK, c.nt * kWRows);
                    tma_load_2d(sw + kWRows * 128, &maps.w[1], full(s), kb * kBK, c.nt * kWRows);
                } else if constexpr (EPI == kEpiStore) {
                    tma_load_2d(sw, &maps.w[0], full(s), kb * kBK, c.g * n + c.nt * BN);
                } else {
                    tma_load_2d(sw, &maps.w[c.g], full(s), kb * kBK, c.nt * BN);
                }
            };
            auto load_a = [&](const Tile& c, int kb, int s) {
                const int slice = EPI == kEpiStore ? (c.g % 3 == 2 ? ep.raw_slice : c.g / 3) : 0;
                tma_load_3d(sbase + s * Cfg::kStageBytes, &maps.a, full(s), kb * kBK, c.mt * kBM, slice);
            };
            // the weight panels of the first stages do not depend on the kernel before this one
            const Tile first = tile_of(blockIdx.x);
            const int ahead = num_kb < S ? num_kb : S;
            for (int kb = 0; kb < ahead; ++kb) {
                mbar_arrive_expect_tx(full(kb), Cfg::kStageBytes);   // (a CTA's first tile is a whole one)
                load_w(first, kb, kb);
            }
            grid_wait();
            for (int kb = 0; kb < ahead; ++kb) load_a(first, kb, kb);
            uint32_t it = 0;
            bool ok = true;
            for (int t = blockIdx.x; t < num_tiles && ok; t += gridDim.x) {
                const Tile c = tile_of(t);
                for (int kb = 0; kb < num_kb; ++kb, ++it) {
                    if (it < (uint32_t)ahead) continue;
                    const int s = it % S;
                    if (!mbar_wait(empty(s), ((it / S) & 1u) ^ 1u, abort_flag)) {
                        report_wait_failure(status, abort_flag, kKid, 1);
                        ok = false;
                        break;
                    }
                    mbar_arrive_expect_tx(full(s), c.whole ? Cfg::kStageBytes : Cfg::kABytes + BN / 2 * kBK * 2);
                    load_a(c, kb, s);
                    load_w(c, kb, s);
                }
            }
        }
    } else if (warp == 1) {
        // ---------------------------------------------------------------- MMA issuer
        if (elect_one()) {
            uint32_t it = 0, tc = 0;
            bool ok = true;
            for (int t = blockIdx.x; t < num_tiles && ok; t += gridDim.x, ++tc) {
                const uint32_t acc = tc & 1u;
                if (!mbar_wait(tempty(acc), ((tc >> 1) & 1u) ^ 1u, abort_flag)) {
                    report_wait_failure(status, abort_flag, kKid, 2);
                    break;
                }
                tc_fence_after_sync();
                const uint32_t d = tmem_base + acc * Cfg::kAccStride;
                const uint32_t idesc = !kHalves || t < whole_tiles ? idesc_bf16_f32(kBM, BN) : idesc_bf16_f32(kBM, BN / 2);
                for (int kb = 0; kb < num_kb; ++kb, ++it) {
                    const int s = it % S;
                    if (!mbar_wait(full(s), (it / S) & 1u, abort_flag)) {
                        report_wait_failure(status, abort_flag, kKid, 3);
                        ok = false;
                        break;
                    }
                    tc_fence_after_sync();
                    const uint32_t sa = sbase + s * Cfg::kStageBytes;
                    const uint64_t ad = smem_desc_k_sw128(sa), bd = smem_desc_k_sw128(sa + Cfg::kABytes);
#pragma unroll
                    for (int k4 = 0; k4 < kBK / 16; ++k4)
                        mma_bf16(d, ad + 2u * k4, bd + 2u * k4, idesc, (kb | k4) != 0 ? 1u : 0u);
                    mma_commit(empty(s));
                }
                if (ok) mma_commit(tfull(acc));
            }
        }
    } else {
        // ---------------------------------------------------------------- epilogue: thread = row, a part of the columns
        // With two warps per 32 rows an epilogue took 7700 (images), 8900 (silu * mul) and 18100 (gate and residual) cycles
        // for tiles whose GEMMs take 8300, 8300 and 14000 (in-kernel clock, 3840 rows of 768): latency, two warps per
        // scheduler, and the divisions of the sigmoids.
        const int quad = warp & 3, part = (warp - 2) >> 2;
        constexpr int kCols = (EPI == kEpiSwiglu ? BN / 2 : BN) / kEpiParts;   // result columns per thread and tile
        grid_wait();
        // kEpiStaged: a tile's gate and residual, by one thread, which also stores the tile ahead
        [[maybe_unused]] auto load_planes = [&](int t) {
            if constexpr (EPI == kEpiStaged) {
                const Tile c = tile_of(t);
                const bool gate = ep.gate != nullptr, residual = ep.residual != nullptr;
                mbar_arrive_expect_tx(planes_full, (gate + residual) * Cfg::kPlaneBytes);
                for (int b = 0; b < BN / 64; ++b) {
                    if (gate) tma_load_2d(sbase + Cfg::kPlanes + b * (kBM * 128), &maps.gate, planes_full, c.nt * BN + b * 64, c.mt * kBM);
                }
                for (int b = 0; b < BN / 64; ++b) {
                    if (residual)
                        tma_load_2d(sbase + Cfg::kPlanes + Cfg::kPlaneBytes + b * (kBM * 128), &maps.residual, planes_full,
                                    c.nt * BN + b * 64, c.mt * kBM);
                }
            }
        };
        if (EPI == kEpiStaged && threadIdx.x == 64) load_planes(blockIdx.x);
        uint32_t tc = 0;
        bool ok = true;   // kEpiStaged: a warp whose wait ran out still takes part in the barriers of the tiles that are left
        for (int t = blockIdx.x; t < num_tiles; t += gridDim.x, ++tc) {
            const Tile c = tile_of(t);
            const uint32_t acc = tc & 1u;
            const long long row = (long long)c.mt * kBM + quad * 32 + lane;
            const bool live = row < rows;
            const int cols = c.whole ? kCols : kCols / 2;
            const int colb = c.nt * kWRows + c.half * (kWRows / 2) + part * cols;   // first column of this thread, inside the matrix
            // The gate and residual values of the tile, all of them on their way under its GEMM: fetched 16 columns at a time
            // between the TMEM loads, their latency was what a tile took (six times 1 us at BN = 192)
            constexpr int kPre = EPI == kEpiResidual ? kCols / 16 : 1;
            [[maybe_unused]] uint32_t gv[kPre][8], zv[kPre][8];
            [[maybe_unused]] float mk = 1.0f, bias0 = 0.f, bias1 = 0.f;   // gate biases of columns lane and 32 + lane
            [[maybe_unused]] float sg[EPI == kEpiStaged ? kCols : 1];
            // this thread's eight columns from `col` (of the tile) on in a plane
            [[maybe_unused]] auto plane = [&](int which, int col) {
                return reinterpret_cast<uint4*>(gbase + Cfg::kPlanes + which * Cfg::kPlaneBytes + (col >> 6) * (kBM * 128) +
                                                sw128_offset(quad * 32 + lane, col & 63));
            };
            if constexpr (EPI == kEpiResidual || EPI == kEpiStaged) {
                if (ep.gate != nullptr) {
                    if (lane < kCols) bias0 = __bfloat162float(ep.gate_bias[colb + lane]);
                    if (32 + lane < kCols) bias1 = __bfloat162float(ep.gate_bias[colb + 32 + lane]);
                }
            }
            if constexpr (EPI == kEpiStaged) {
                if (live && ep.mask != nullptr) mk = __bfloat162float(ep.mask[row]);
                if (ok && !mbar_wait(planes_full, tc & 1u, abort_flag)) {
                    if (lane == 0) report_wait_failure(status, abort_flag, kKid, 5);
                    ok = false;
                }
                // the gates' sigmoids, under the product: two special-function results per value, 1.7 us of a tile of 192 columns
                if (ep.gate != nullptr && ok) {
#pragma unroll
                    for (int e0 = 0; e0 < kCols; e0 += 8) {
                        const uint4 g = *plane(0, part * kCols + e0);
                        const uint32_t gw[4] = {g.x, g.y, g.z, g.w};
#pragma unroll
                        for (int e = 0; e < 8; ++e) {
                            const float ge = e & 1 ? bf16hi(gw[e >> 1]) : bf16lo(gw[e >> 1]);
                            sg[e0 + e] = sigmoid_of(ge + __shfl_sync(0xffffffffu, e0 < 32 ? bias0 : bias1, (e0 + e) & 31));
                            asm volatile("" : "+f"(sg[e0 + e]));   // not behind the wait
                        }
                    }
                }
            }
            if constexpr (EPI == kEpiResidual) {
                if (live) {
                    if (ep.mask != nullptr) mk = __bfloat162float(ep.mask[row]);
#pragma unroll
                    for (int p = 0; p < kPre; ++p) {
                        if (ep.gate != nullptr) ld_row16_wide(ep.gate + row * n + colb + p * 16, gv[p]);
                        if (ep.residual != nullptr) ld_row16_wide(ep.residual + row * n + colb + p * 16, zv[p]);
                    }
                }
            }
            if (ok && !mbar_wait(tfull(acc), (tc >> 1) & 1u, abort_flag)) {
                if (lane == 0) report_wait_failure(status, abort_flag, kKid, 4);
                ok = false;
            }
            if (EPI != kEpiStaged && !ok) break;
            tc_fence_after_sync();
            const uint32_t taddr = tmem_base + ((uint32_t)(quad * 32) << 16) + acc * Cfg::kAccStride + part * cols;
            const uint32_t second = c.whole ? BN / 2 : BN / 4;   // kEpiSwiglu: the other matrix' columns
            [[maybe_unused]] int bb = 0, pos = 0;   // sample and position of the row
            if constexpr (EPI == kEpiImages) {
                bb = (int)((uint32_t)row / (uint32_t)ep.im.rows_per_sample);
                pos = (int)row - bb * ep.im.rows_per_sample;
            }
#pragma unroll(EPI == kEpiResidual ? kPre : (EPI == kEpiStaged ? kCols / 16 : 1))
            for (int c0 = 0; c0 < (kHalves ? cols : kCols); c0 += 16) {
                if (EPI == kEpiStaged && !ok) break;
                uint32_t r[16], r2[16];
                tmem_ld16(taddr + c0, r);
                if constexpr (EPI == kEpiSwiglu) tmem_ld16(taddr + second + c0, r2);
                tmem_ld_wait();
                const int col = colb + c0;
                if (EPI != kEpiResidual && EPI != kEpiStaged && !live) continue;   // (its gate biases are shared by shuffles)
                if constexpr (EPI == kEpiImages) {
                    store_images<D>(ep.im, ep.kind[c.g], ep.qscale, r, col, row, bb, pos);
                } else if constexpr (EPI == kEpiStaged) {
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        uint4* p = plane(1, part * kCols + c0 + h * 8);
                        float v[8];
#pragma unroll
                        for (int e = 0; e < 8; ++e) {
                            v[e] = __fmul_rn(mk, __uint_as_float(r[h * 8 + e]));
                            if (ep.gate != nullptr) v[e] = __fmul_rn(v[e], sg[c0 + h * 8 + e]);   // not one fma with the residual
                        }
                        if (ep.residual != nullptr) {
                            const uint4 z = *p;
                            const uint32_t zw[4] = {z.x, z.y, z.z, z.w};
#pragma unroll
                            for (int e = 0; e < 8; ++e) v[e] += e & 1 ? bf16hi(zw[e >> 1]) : bf16lo(zw[e >> 1]);
                        }
                        *p = make_uint4(pack_bf16x2(v[0], v[1]), pack_bf16x2(v[2], v[3]), pack_bf16x2(v[4], v[5]),
                                        pack_bf16x2(v[6], v[7]));
                    }
                } else {
                    uint32_t o[8];
                    if constexpr (EPI == kEpiStore) {
#pragma unroll
                        for (int e = 0; e < 8; ++e)
                            o[e] = pack_bf16x2(__uint_as_float(r[2 * e]), __uint_as_float(r[2 * e + 1]));
                        stg256(ep.y + ((long long)c.g * rows + row) * n + col, o);
                    } else if constexpr (EPI == kEpiSwiglu) {
#pragma unroll
                        for (int e = 0; e < 8; ++e) {
                            const float a0 = __uint_as_float(r[2 * e]), a1 = __uint_as_float(r[2 * e + 1]);
                            o[e] = pack_bf16x2(a0 * sigmoid_of(a0) * __uint_as_float(r2[2 * e]),
                                               a1 * sigmoid_of(a1) * __uint_as_float(r2[2 * e + 1]));
                        }
                        stg256(ep.out + row * n + col, o);
                    } else {
                        float v[16];
#pragma unroll
                        for (int e = 0; e < 16; ++e) v[e] = mk * __uint_as_float(r[e]);
                        if (ep.gate != nullptr) {
                            const uint32_t (&g)[8] = gv[c0 / 16];
                            const float bias = c0 < 32 ? bias0 : bias1;
#pragma unroll
                            for (int e = 0; e < 8; ++e) {
                                const int src = (c0 & 31) + 2 * e;
                                v[2 * e] *= sigmoid_of(bf16lo(g[e]) + __shfl_sync(0xffffffffu, bias, src));
                                v[2 * e + 1] *= sigmoid_of(bf16hi(g[e]) + __shfl_sync(0xffffffffu, bias, src + 1));
                            }
                        }
                        if (ep.residual != nullptr) {
                            const uint32_t (&z)[8] = zv[c0 / 16];
#pragma unroll
                            for (int e = 0; e < 8; ++e) {
                                v[2 * e] += bf16lo(z[e]);
                                v[2 * e + 1] += bf16hi(z[e]);
                            }
                        }
#pragma unroll
                        for (int e = 0; e < 8; ++e) o[e] = pack_bf16x2(v[2 * e], v[2 * e + 1]);
                        if (live) st_row16_any(ep.out + row * n + col, o);
                    }
                }
            }
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive(tempty(acc));
            if constexpr (EPI == kEpiStaged) {
                fence_proxy_async_smem();
                rowtile::group_sync(1, 128 * kEpiParts);
                if (threadIdx.x == 64 && ok) {
                    for (int b = 0; b < BN / 64; ++b)
                        tma_store_2d(&maps.out, sbase + Cfg::kPlanes + Cfg::kPlaneBytes + b * (kBM * 128), c.nt * BN + b * 64, c.mt * kBM);
                    tma_store_commit();
                    if (t + (int)gridDim.x < num_tiles) {
                        tma_store_wait_read<0>();
                        load_planes(t + gridDim.x);
                    }
                }
            }
        }
        if (EPI == kEpiStaged && threadIdx.x == 64) tma_store_wait_all<0>();
    }

    tc_fence_before_sync();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after_sync();
        tmem_dealloc(tmem_base, Cfg::kTmemCols);
    }
}

// Column tile: the number of waves of 148 CTAs times the panels a tile streams (128 rows of x and BN of the weights per
// k-block, plus a constant for its fill and epilogue). Wide tiles move fewer bytes, narrow ones fill the chip when there
// are few rows; a BN that does not divide the matrix is out. (A last wave of halves counted as one of half the width picks 256
// where 192 ties: 5 x 350, 4 x 500 and 5 x 450 tokens within 0.2% of each other.)
int pick_bn(long long rows, int n, int mats, bool swiglu, int widest = 256) {
    const long long sms = sm_count(), mt = (rows + kBM - 1) / kBM;
    const int cand[4] = {256, 192, 128, 64};
    int best = 0;
    long long best_cost = 0;
    for (int bn : cand) {
        const int wr = swiglu ? bn / 2 : bn;
        if (bn > widest || n % wr != 0 || (swiglu && (bn == 64 || bn == 192))) continue;
        const long long tiles = mt * (n / wr) * (swiglu ? 1 : mats);
        const long long cost = (tiles + sms - 1) / sms * (128 + bn + 64);
        if (best == 0 || cost < best_cost) {
            best = bn;
            best_cost = cost;
        }
    }
    return best;
}

template <int BN, int EPI, int D>
int launch(const LinearIn& in, const EpiArgs& ep, int slices, int w_rows, cudaStream_t st) {
    using Cfg = LinCfg<BN, EPI>;
    constexpr int kWRows = EPI == kEpiSwiglu ? BN / 2 : BN;
    std::conditional_t<EPI == kEpiStaged, StagedMaps, LinMaps> maps;
    int rc;
    {
        uint64_t dims[3] = {(uint64_t)in.k, (uint64_t)in.rows, (uint64_t)slices};
        uint64_t str[2] = {(uint64_t)in.k * 2, (uint64_t)in.rows * in.k * 2};
        uint32_t box[3] = {kBK, kBM, 1};
        if ((rc = make_tmap_bf16(&maps.a, in.x, 3, dims, str, box, 1))) return rc;
    }
    const int tensors = EPI == kEpiStore ? 1 : in.num_w;
    for (int i = 0; i < tensors; ++i) {
        uint64_t dims[2] = {(uint64_t)in.k, (uint64_t)w_rows};
        uint64_t str[1] = {(uint64_t)in.k * 2};
        uint32_t box[2] = {kBK, (uint32_t)(has_halves<BN, EPI>() ? kWRows / 2 : kWRows)};
        if ((rc = make_tmap_bf16(&maps.w[i], in.w[i], 2, dims, str, box, 1))) return rc;
    }
    for (int i = tensors; i < 4; ++i) maps.w[i] = maps.w[0];
    if constexpr (EPI == kEpiStaged) {
        const uint64_t dims[2] = {(uint64_t)in.n, (uint64_t)in.rows};
        const uint64_t str[1] = {(uint64_t)in.n * 2};
        const uint32_t box[2] = {64, kBM};
        if ((rc = make_tmap_bf16(&maps.out, ep.out, 2, dims, str, box, 1))) return rc;
        maps.gate = maps.residual = maps.out;
        if (ep.gate && (rc = make_tmap_bf16(&maps.gate, ep.gate, 2, dims, str, box, 1))) return rc;
        if (ep.residual && (rc = make_tmap_bf16(&maps.residual, ep.residual, 2, dims, str, box, 1))) return rc;
    }
    static PerDeviceOnce configured;
    if (!configured.done()) {
        OF3_CUDA_CHECK(cudaFuncSetAttribute(linear_kernel<BN, EPI, D>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                            Cfg::kSmemBytes));
        configured.mark();
    }
    const long long tiles = ((in.rows + kBM - 1) / kBM) * (in.n / kWRows) * (EPI == kEpiSwiglu ? 1 : in.num_w);
    OF3_REQUIRE(tiles < (1LL << 30) && in.rows < (1LL << 31), OF3_ERR_SHAPE, "linear: too many rows");
    const int grid = (int)(tiles < sm_count() ? tiles : sm_count());
    const int rest = (int)(tiles % grid), whole = (int)tiles - (has_halves<BN, EPI>() && 2 * rest <= grid ? rest : 0);
    LaunchScope scope(kKid, st);
    OF3_CUDA_CHECK(launch_chained(linear_kernel<BN, EPI, D>, grid, kThreads, Cfg::kSmemBytes, st, maps, ep, in.rows, in.k,
                                  in.n, in.num_w, whole, device_status_ptr()));
    return OF3_OK;
}

template <int EPI, int D>
int dispatch(const LinearIn& in, const EpiArgs& ep, int slices, int w_rows, cudaStream_t st) {
    OF3_REQUIRE(in.k % kBK == 0 && in.n % 64 == 0, OF3_ERR_SHAPE, "linear: widths %d x %d are not multiples of 64", in.n,
                in.k);
    switch (pick_bn(in.rows, in.n, in.num_w, EPI == kEpiSwiglu, EPI == kEpiResidual || EPI == kEpiStaged ? 192 : 256)) {
        case 256:
            if constexpr (EPI != kEpiResidual && EPI != kEpiStaged) return launch<256, EPI, D>(in, ep, slices, w_rows, st);
        case 192:
            if constexpr (EPI != kEpiSwiglu) return launch<192, EPI, D>(in, ep, slices, w_rows, st);
        case 128: return launch<128, EPI, D>(in, ep, slices, w_rows, st);
        default:
            if constexpr (EPI != kEpiSwiglu) return launch<64, EPI, D>(in, ep, slices, w_rows, st);
            return OF3_ERR_SHAPE;
    }
}

}  // namespace

int linear_conditioning(const bf16* x, long long rows, int k, int n, const bf16* w, int layers, int slices,
                        int raw_slice, bf16* y, cudaStream_t st) {
    LinearIn in{x, rows, k, n, {w}, 3 * layers};
    EpiArgs ep = {};
    ep.y = y;
    ep.raw_slice = raw_slice;
    return dispatch<kEpiStore, 0>(in, ep, slices, 3 * layers * n, st);
}

int linear_attn_images(const LinearIn& in, const LinearOut* kinds, const AttnImages& im, cudaStream_t st) {
    EpiArgs ep = {};
    ep.im = im;
    for (int i = 0; i < in.num_w; ++i) ep.kind[i] = kinds[i];
    ep.qscale = kLog2e * (1.0f / sqrtf((float)im.D));
    return im.D == 24 ? dispatch<kEpiImages, 24>(in, ep, 1, in.n, st) : dispatch<kEpiImages, 48>(in, ep, 1, in.n, st);
}

int linear_swiglu(const LinearIn& in, bf16* h, cudaStream_t st) {
    EpiArgs ep = {};
    ep.out = h;
    return dispatch<kEpiSwiglu, 0>(in, ep, 1, in.n, st);
}

int linear_residual(const LinearIn& in, const bf16* residual, const bf16* gate, const bf16* gate_bias, const bf16* mask,
                    bf16* out, cudaStream_t st) {
    EpiArgs ep = {};
    ep.out = out;
    ep.residual = residual;
    ep.gate = gate;
    ep.gate_bias = gate_bias;
    ep.mask = mask;
    const bool tma = (((uintptr_t)residual | (uintptr_t)gate | (uintptr_t)out) & 15) == 0;
    return tma ? dispatch<kEpiStaged, 0>(in, ep, 1, in.n, st) : dispatch<kEpiResidual, 0>(in, ep, 1, in.n, st);
}

}  // namespace fast
}  // namespace of3
