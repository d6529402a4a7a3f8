// SwiGLU pair transition, bf16 / tcgen05 family (c = 128, expansion 4 -> hidden 512).
//
// One fused kernel: x tile -> LayerNorm (in place in the A operand) -> per 64-wide hidden chunk
//   G1: [a|b] = LN(x) [W_a;W_b]_chunk^T  (128x128x128, accumulators in TMEM)
//   h  = silu(a) * b  -> bf16 -> shared memory as the next A operand (never leaves the SM)
//   G2: y += h W_out[:, chunk]^T         (128x128x64, accumulated over the 8 chunks in TMEM)
// then out = x + mask * y, TMA-stored. The 512-wide hidden activation (604 MB at N = 768 in the
// reference's unfused path) never touches HBM. Two row groups of 128 rows share every weight chunk (streamed from L2
// by TMA, double-buffered), which halves the weight traffic per row.
// Reference: openfold3/core/model/layers/transition.py:225-271,
//            openfold3/core/model/primitives/activations.py:33-61.
#include "modules.cuh"
#include "rowtile.cuh"
#include "runtime.cuh"

namespace of3 {
namespace fast {
namespace {

using namespace umma;
using namespace rowtile;

constexpr int kKidTrans = 4;
constexpr int kHidden = 512;
constexpr int kChunk = 64;
constexpr int kNumChunks = kHidden / kChunk;  // 8


// v[0..3]: partial sums of 4 rows, spread over the 16 lanes of a half warp -> the rows' sums, in every lane. The first
// steps of the tree send the rows that the lane does not go on with: 3 + 2 + 4 shuffles instead of 4 x 4.
__device__ __forceinline__ void row_sums(float (&v)[4], int lane) {
#pragma unroll
    for (int w = 2; w >= 1; w >>= 1) {   // w rows kept; the partner is 4 w lanes away
        const bool up = lane & (4 * w);
#pragma unroll
        for (int r = 0; r < w; ++r) {
            const float keep = up ? v[r + w] : v[r], send = up ? v[r] : v[r + w];
            v[r] = keep + __shfl_xor_sync(0xffffffffu, send, 4 * w);
        }
    }
    float sum = v[0];   // of row (lane & 12) >> 2
    sum += __shfl_xor_sync(0xffffffffu, sum, 2);
    sum += __shfl_xor_sync(0xffffffffu, sum, 1);
#pragma unroll
    for (int r = 0; r < 4; ++r) v[r] = __shfl_sync(0xffffffffu, sum, (lane & 16) + 4 * r);
}

// Keeps the compiler from carrying values computed from v[first .. first + 15] over this point.
template <int N>
__device__ __forceinline__ void opaque(uint32_t (&v)[N], int first) {
#pragma unroll
    for (int i = 0; i < 16; ++i) asm volatile("" : "+r"(v[first + i]));
}

// LN of rows 0, 2, .. 2 (NR - 1) from src on, of which those below `left` exist: eight channels of each, packed. A half warp reads a
// row (coalesced).
template <int NR>
__device__ __forceinline__ void normalize_rows(const __nv_bfloat16* src, int left, int ch, int lane, const float* prm,
                                               uint32_t (&raw)[NR * 4]) {
#pragma unroll
    for (int h = 0; h < NR; h += 4) {   // four rows at a time (registers)
        float mean[4], rstd[4];
        asm volatile("" ::: "memory");
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            uint4 v = make_uint4(0u, 0u, 0u, 0u);
            if (2 * (h + r) < left) v = *reinterpret_cast<const uint4*>(src + 2 * (h + r) * kC);
            uint32_t* o = &raw[(h + r) * 4];
            o[0] = v.x; o[1] = v.y; o[2] = v.z; o[3] = v.w;
        }
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            float a = 0.f, b = 0.f;
#pragma unroll
            for (int i = 0; i < 4; ++i) { a = add_lo(raw[(h + r) * 4 + i], a); b = add_hi(raw[(h + r) * 4 + i], b); }
            mean[r] = a + b;
        }
        row_sums(mean, lane);
        opaque(raw, h * 4);   // unpack again rather than keep 32 floats
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            mean[r] *= 1.0f / kC;
            float a = 0.f, b = 0.f;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const float x0 = add_lo(raw[(h + r) * 4 + i], -mean[r]), x1 = add_hi(raw[(h + r) * 4 + i], -mean[r]);
                a = fmaf(x0, x0, a);
                b = fmaf(x1, x1, b);
            }
            rstd[r] = a + b;
        }
        row_sums(rstd, lane);
        opaque(raw, h * 4);
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            rstd[r] = rsqrtf(rstd[r] * (1.0f / kC) + kLnEps);
            mean[r] *= -rstd[r];
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float2 ga = *reinterpret_cast<const float2*>(prm + ch * 8 + i * 2);
            const float2 be = *reinterpret_cast<const float2*>(prm + 128 + ch * 8 + i * 2);
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                uint32_t& v = raw[(h + r) * 4 + i];
                v = pack_bf16x2(fmaf(fmaf(bf16lo(v), rstd[r], mean[r]), ga.x, be.x),
                                fmaf(fmaf(bf16hi(v), rstd[r], mean[r]), ga.y, be.y));
            }
        }
    }
}

struct TrSmem {
    static constexpr uint32_t kWStage = 49152;                 // [Wa|Wb] slab 32 KB + Wout chunk 16 KB
    static constexpr uint32_t kW = 0;                          // 2 stages
    static constexpr uint32_t kX = 2 * kWStage;                // 3 x 32 KB (x tile / LN(x) / x again / output)
    static constexpr uint32_t kH = kX + 3 * kTileBytes;        // 2 groups x 16 KB
    static constexpr uint32_t kParams = kH + 2 * kKBlockBytes; // gamma, beta
    static constexpr uint32_t kBars = kParams + 1024;
    static constexpr uint32_t kTotal = kBars + 256;
    static constexpr uint32_t kDyn = kTotal + 1024;
};

// warps: 0 weight producer, 1 and 2 the MMA issuers of row group 0 and 1, 3 the results' stores, 4..11 LayerNorm,
// 12..19 and 20..27 the two row groups: two threads share a row (TMEM lane) and take half of every hidden chunk through
// silu * mul, and half of the output row each.
//
// The tensor work of a tile is 6100 cycles; what kept a pair of tiles at 34400 (in-kernel clock phases at N = 768) was
// what both groups did between two tiles at the same time, with the tensor pipe idle: store 2100, wait for the next x
// 2600, LayerNorm 5300, output 1200. So the tiles are prepared ahead, by warps of their own: these hold the next tile,
// normalised, in registers until one of the three x buffers is free (the CTA's tile t uses buffer t mod 3). The residual
// is fetched once more from L2 into the buffer that the last G1 has released instead of staying in 32 registers of
// every row thread.
// What is left is near the shared memory's limit: a 128 x 128 x 16 MMA reads 8 KB in its 64 cycles, which is all that
// the memory gives, and the weights, LN(x), h and the result are written beside it.
// Both groups take the chunks in the same order, so that a row's result does not depend on where in the tensor it lies
// (half a tile apart, with the cyclic sequence entered where it is, they would never wait for a buffer: 234 us instead
// of 250). N = 768: 316 -> 250 us, N = 37: 25.8 -> 20.9.
constexpr int kTrThreads = 32 * 28;

// kSolo: one tile per CTA (a tensor of no more tiles than SMs), whose chunks alternate between both groups' D1 and h buffers, so
// that G1 runs two chunks ahead of the silu pass instead of one: N = 24 / 37 / 64 / 111 / 137, unchained, 14.1 / 14.2 / 14.3 / 14.7 /
// 15.0 -> 12.7 / 12.8 / 13.0 / 13.6 / 14.0 us. The LayerNorm of its tile is shared by the LayerNorm warps and the first row group,
// four rows per half warp instead of eight in two turns, each of which waited for its loads (N = 37, four pair blocks: 349 -> 344). An instantiation of its own: with
// the choice made in the kernel N = 768 took 241 instead of 224 us (registers).
template <bool kSolo>
__global__ void __launch_bounds__(kTrThreads, 1)
transition_kernel(const __grid_constant__ CUtensorMap tmX, const __grid_constant__ CUtensorMap tmOut,
                  const __grid_constant__ CUtensorMap tmWa, const __grid_constant__ CUtensorMap tmWb,
                  const __grid_constant__ CUtensorMap tmWo, const __nv_bfloat16* x,   // x may be the output
                  const __nv_bfloat16* __restrict__ mask,
                  const __nv_bfloat16* __restrict__ ln_w, const __nv_bfloat16* __restrict__ ln_b,
                  long long rows, int add_residual, int* status) {
    extern __shared__ uint8_t smem_raw[];
    const uint32_t sbase = (smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t* gbase = smem_raw + (sbase - smem_u32(smem_raw));
    float* prm = reinterpret_cast<float*>(gbase + TrSmem::kParams);
    const uint32_t bars = sbase + TrSmem::kBars;
    auto w_full = [&](int s) { return bars + 8u * (0 + s); };
    auto w_empty = [&](int s) { return bars + 8u * (2 + s); };
    auto wo_full = [&](int s) { return bars + 8u * (4 + s); };    // W_out chunk of a weight stage (its own ring:
    auto wo_empty = [&](int s) { return bars + 8u * (6 + s); };   // the slab is free long before the chunk's 2nd GEMM)
    auto a_ready = [&](int b) { return bars + 8u * (8 + b); };
    auto x_empty = [&](int b) { return bars + 8u * (11 + b); };
    auto d1_full = [&](int g) { return bars + 8u * (14 + g); };
    auto d1_empty = [&](int g) { return bars + 8u * (16 + g); };
    auto h_ready = [&](int g) { return bars + 8u * (18 + g); };
    auto h_free = [&](int g) { return bars + 8u * (20 + g); };
    auto d2_full = [&](int g) { return bars + 8u * (22 + g); };
    auto d2_empty = [&](int g) { return bars + 8u * (24 + g); };
    auto res_full = [&](int g) { return bars + 8u * (26 + g); };   // x is back in the tile's buffer
    auto out_ready = [&](int g) { return bars + 8u * (28 + g); };  // the group's result lies in the tile's buffer
    volatile uint32_t* tmem_ptr = reinterpret_cast<volatile uint32_t*>(gbase + TrSmem::kBars + 240);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(gbase + TrSmem::kBars + 248);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int my_tiles = (int)tiles_of_block((rows + kRows - 1) / kRows);
    // group g's tiles are the CTA's tiles g, g + 2, ...
    // One tile only (kSolo, or a CTA with one where others have two): both groups work on it, each on half of every chunk's
    // columns and of the output's. The silu pass is the longest link of a lone tile's chain. (The last of three tiles or more
    // is its group's alone.)
    const bool solo = kSolo || my_tiles == 1;
    const int num_chunks = ((my_tiles + 1) >> 1) * kNumChunks;

    if (threadIdx.x == 0) {
        for (int i = 0; i < 2; ++i) {
            mbar_init(w_full(i), 1);
            mbar_init(w_empty(i), 2);  // both groups' issuers have consumed the [W_a|W_b] slab
            mbar_init(wo_full(i), 1);
            mbar_init(wo_empty(i), 2);
            mbar_init(d1_full(i), 1);
            mbar_init(d1_empty(i), solo ? 16 : 8);
            mbar_init(h_ready(i), solo ? 16 : 8);
            mbar_init(h_free(i), 1);
            mbar_init(d2_full(i), 1);
            mbar_init(d2_empty(i), 8);
            mbar_init(res_full(i), 1);
            mbar_init(out_ready(i), solo ? 16 : 8);
        }
        for (int i = 0; i < 3; ++i) {
            mbar_init(x_empty(i), 1);
            mbar_init(a_ready(i), kSolo ? 16 : 8);
        }
        *abort_flag = 0;
        mbar_fence_init();
        prefetch_tmap(&tmX);
        prefetch_tmap(&tmWa);
        prefetch_tmap(&tmWb);
        prefetch_tmap(&tmWo);
    }
    if (threadIdx.x < 128) {
        prm[threadIdx.x] = __bfloat162float(ln_w[threadIdx.x]);
        prm[128 + threadIdx.x] = __bfloat162float(ln_b[threadIdx.x]);
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
    if (warp != 0) grid_wait();   // (the weights do not depend on the kernel before this one)
    // TMEM columns: group g -> D1 at g*256 + [0,128) ([a 64 | b 64]), D2 at g*256 + [128,256)

    if (warp == 0) {
        // ---------------------------------------------------------------- weight producer
        if (elect_one()) {
            bool ok = true;
            auto load_slab = [&](int wi) -> bool {
                const int s = wi & 1, c = wi & (kNumChunks - 1);
                if (!mbar_wait(w_empty(s), ((uint32_t)(wi >> 1) & 1u) ^ 1u, abort_flag)) {
                    report_wait_failure(status, abort_flag, kKidTrans, 2);
                    return false;
                }
                mbar_arrive_expect_tx(w_full(s), 2 * kKBlockBytes);
                const uint32_t w = sbase + TrSmem::kW + s * TrSmem::kWStage;
                for (int kb = 0; kb < 2; ++kb) {
                    // slab k-block kb: rows [0,64) = W_a chunk, rows [64,128) = W_b chunk
                    tma_load_2d(w + kb * kKBlockBytes, &tmWa, w_full(s), kb * 64, c * kChunk);
                    tma_load_2d(w + kb * kKBlockBytes + 64 * 128, &tmWb, w_full(s), kb * 64, c * kChunk);
                }
                return true;
            };
            ok = load_slab(0);
            for (int wi = 0; wi < num_chunks && ok; ++wi) {
                // a slab's stage is released by the G1 two chunks before, and that comes before the G2 which releases
                // this chunk's W_out stage
                if (wi + 1 < num_chunks && !load_slab(wi + 1)) break;
                const int s = wi & 1, c = wi & (kNumChunks - 1);
                if (!mbar_wait(wo_empty(s), ((uint32_t)(wi >> 1) & 1u) ^ 1u, abort_flag)) {
                    report_wait_failure(status, abort_flag, kKidTrans, 12);
                    break;
                }
                mbar_arrive_expect_tx(wo_full(s), kKBlockBytes);
                tma_load_2d(sbase + TrSmem::kW + s * TrSmem::kWStage + 2 * kKBlockBytes, &tmWo, wo_full(s), c * kChunk, 0);
            }
        }
    } else if (warp <= 2) {
        // ---------------------------------------------------------------- MMA issuer of row group g
        if (elect_one()) {
            const int g = warp - 1;
            constexpr uint32_t idesc = idesc_bf16_f32(128, 128);
            bool ok = true;
            auto fail = [&](int site) {
                report_wait_failure(status, abort_flag, kKidTrans, site);
                ok = false;
            };
            auto skip_chunk = [&](int wi) {   // the other group's alone: keep both weight rings moving
                const int s = wi & 1;
                const uint32_t par = (uint32_t)(wi >> 1) & 1u;
                if (!mbar_wait(w_full(s), par, abort_flag)) return fail(3);
                mbar_arrive(w_empty(s));
                if (!mbar_wait(wo_full(s), par, abort_flag)) return fail(13);
                mbar_arrive(wo_empty(s));
            };
            // Software-pipelined: G1 of chunk i + 1 is issued as soon as the row group has read D1 of chunk i, BEFORE
            // waiting for that chunk's silu pass and its G2, so the row group finds its next accumulator ready when it
            // comes back; across the tiles' boundary too, if the next tile's LN(x) is there by then.
            int t = g, buf = g;   // the CTA's tile that G1 is at, and its x buffer (t mod 3)
            uint32_t use = 0;     // t / 3: how often the buffer has been used before
            auto issue_g1 = [&](int i) -> bool {   // i: chunk, counted over the group's tiles
                const int s = i & 1, c = i & (kNumChunks - 1);
                if (c == 0 && !mbar_wait(a_ready(buf), use & 1u, abort_flag)) { fail(4); return false; }
                if (!mbar_wait(w_full(s), (uint32_t)(i >> 1) & 1u, abort_flag)) { fail(3); return false; }
                const int d = kSolo ? i & 1 : g;
                if (!mbar_wait(d1_empty(d), ((uint32_t)(kSolo ? i >> 1 : i) & 1u) ^ 1u, abort_flag)) { fail(5); return false; }
                tc_fence_after_sync();
                mma_k128(tmem_base + d * 256, sbase + TrSmem::kX + buf * kTileBytes,
                         sbase + TrSmem::kW + s * TrSmem::kWStage, kKBlockBytes, idesc, false);
                mma_commit(d1_full(d));
                mma_commit(w_empty(s));
                return true;
            };
            const int n = ((my_tiles + 1 - g) >> 1) * kNumChunks;
            const int ahead = kSolo ? 2 : 1;
            if (ok && n > 0) ok = issue_g1(0);
            if (ok && n > 0 && kSolo) ok = issue_g1(1);
            for (int i = 0; i < n && ok; ++i) {
                const int s = i & 1, c = i & (kNumChunks - 1);
                const int d = kSolo ? i & 1 : g;                        // D1 and h buffers of the chunk
                const uint32_t dpar = (uint32_t)(kSolo ? i >> 1 : i) & 1u;
                bool late = false;    // the next tile's LN(x) is not there yet: its first G1 does not hold up this tile's last G2
                if (c == kNumChunks - 1) {
                    // the last G1 has read LN(x): fetch x once more (from L2) for the residual, under the silu pass
                    if (!mbar_wait(d1_full(d), dpar, abort_flag)) { fail(15); break; }
                    if (add_residual) {
                        const uint32_t xtile = sbase + TrSmem::kX + buf * kTileBytes;
                        const int row0 = (int)((blockIdx.x + (long long)t * gridDim.x) * kRows);
                        mbar_arrive_expect_tx(res_full(g), kTileBytes);
                        tma_load_2d(xtile, &tmX, res_full(g), 0, row0);
                        tma_load_2d(xtile + kKBlockBytes, &tmX, res_full(g), 64, row0);
                    } else {
                        mbar_arrive(res_full(g));
                    }
                    t += 2;
                    buf += 2;
                    if (buf >= 3) { buf -= 3; ++use; }
                    late = i + 1 < n && !mbar_try_wait(a_ready(buf), use & 1u);
                }
                if (i + ahead < n && !late && !issue_g1(i + ahead)) break;
                if (c == 0 && !mbar_wait(d2_empty(g), ((uint32_t)(i / kNumChunks) & 1u) ^ 1u, abort_flag)) { fail(6); break; }
                if (!mbar_wait(wo_full(s), (uint32_t)(i >> 1) & 1u, abort_flag)) { fail(13); break; }
                if (!mbar_wait(h_ready(d), dpar, abort_flag)) { fail(7); break; }
                tc_fence_after_sync();
                const uint64_t ad = smem_desc_k_sw128(sbase + TrSmem::kH + d * kKBlockBytes);
                const uint64_t bd = smem_desc_k_sw128(sbase + TrSmem::kW + s * TrSmem::kWStage + 2 * kKBlockBytes);
#pragma unroll
                for (int k4 = 0; k4 < 4; ++k4)
                    mma_bf16(tmem_base + g * 256 + 128, ad + 2u * k4, bd + 2u * k4, idesc, (c != 0 || k4 != 0) ? 1u : 0u);
                mma_commit(h_free(d));
                if (c == kNumChunks - 1) mma_commit(d2_full(g));
                mma_commit(wo_empty(s));
                if (late && !issue_g1(i + 1)) break;   // (several tiles: one chunk ahead)
            }
            for (int i = n; i < num_chunks && ok; ++i) skip_chunk(i);
        }
    } else if (warp == 3) {
        // ---------------------------------------------------------------- results out
        if (elect_one()) {
            uint32_t buf = 0;
            for (int t = 0; t < my_tiles; ++t) {
                if (!mbar_wait(out_ready(t & 1), (uint32_t)(t >> 1) & 1u, abort_flag)) {
                    report_wait_failure(status, abort_flag, kKidTrans, 14);
                    break;
                }
                const uint32_t xtile = sbase + TrSmem::kX + buf * kTileBytes;
                const int row0 = (int)((blockIdx.x + (long long)t * gridDim.x) * kRows);
                tma_store_3d(&tmOut, xtile, 0, row0, 0);
                tma_store_3d(&tmOut, xtile + kKBlockBytes, 64, row0, 0);
                tma_store_commit();
                if (t + 3 < my_tiles) {
                    tma_store_wait_read<0>();
                    mbar_arrive(x_empty(buf));
                }
                if (++buf == 3) buf = 0;
            }
            tma_store_wait_all<0>();
        }
    } else if (!kSolo && warp < 12) {
        // ---------------------------------------------------------------- LayerNorm: 16 rows per warp and tile
        // A half warp reads a row (coalesced), so that a thread holds 8 channels of 8 rows; see row_sums.
        const int ch = lane & 15, sub = lane >> 4;
        const int row0 = (warp - 4) * 16 + sub;
        uint32_t buf = 0, use = 0;
        for (int t = 0; t < my_tiles; ++t) {
            const uint32_t xtile = sbase + TrSmem::kX + buf * kTileBytes;
            const long long base = (blockIdx.x + (long long)t * gridDim.x) * kRows + row0;
            const __nv_bfloat16* src = x + base * kC + ch * 8;
            const int left = (int)min(rows - base, 16LL);   // rows 0, 2, ... 14 from here; the tensor may end before
            uint32_t raw[32];
            normalize_rows<8>(src, left, ch, lane, prm, raw);
            if (!mbar_wait(x_empty(buf), (use & 1u) ^ 1u, abort_flag)) {
                if (lane == 0) report_wait_failure(status, abort_flag, kKidTrans, 8);
                break;
            }
#pragma unroll
            for (int r = 0; r < 8; ++r)
                sts128(chunk_addr(xtile, row0 + 2 * r, ch), make_uint4(raw[r * 4], raw[r * 4 + 1], raw[r * 4 + 2], raw[r * 4 + 3]));
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) mbar_arrive(a_ready(buf));
            if (++buf == 3) { buf = 0; ++use; }
        }
    } else {
        // ---------------------------------------------------------------- two row groups
        if constexpr (kSolo) {
            // the tile's LayerNorm, eight rows per warp: by the LayerNorm warps and the first row group, which has no row yet
            if (warp < 20) {
                const int ch = lane & 15, row0 = (warp - 4) * 8 + (lane >> 4);
                const long long base = blockIdx.x * (long long)kRows + row0;
                uint32_t raw[16];
                normalize_rows<4>(x + base * kC + ch * 8, (int)min(rows - base, 8LL), ch, lane, prm, raw);
#pragma unroll
                for (int r = 0; r < 4; ++r)
                    sts128(chunk_addr(sbase + TrSmem::kX, row0 + 2 * r, ch),
                           make_uint4(raw[r * 4], raw[r * 4 + 1], raw[r * 4 + 2], raw[r * 4 + 3]));
                fence_proxy_async_smem();
                __syncwarp();
                if (lane == 0) mbar_arrive(a_ready(0));
            }
        }
        const int own = (warp - 12) >> 3;      // group of these warps
        const int g = solo ? 0 : own;          // group whose tile they work on
        const int quad = warp & 3;
        const int half = ((warp - 12) >> 2) & 1;
        const int row = quad * 32 + lane;
        const uint32_t t_lane = tmem_base + ((uint32_t)(quad * 32) << 16);
        const uint32_t t_d2 = t_lane + g * 256 + 128;
        bool ok = !kSolo || warp >= 12;
        uint32_t ppar = 0;
        int buf = g;
        for (int t = g; t < my_tiles && ok; t += 2, ppar ^= 1u) {
            const uint32_t xtile = sbase + TrSmem::kX + buf * kTileBytes;
            buf += 2;
            if (buf >= 3) buf -= 3;
            const long long grow = (blockIdx.x + (long long)t * gridDim.x) * kRows + row;
            float m = 1.0f;
            if (mask != nullptr && grow < rows) m = __bfloat162float(mask[grow]);

            for (int c = 0; c < kNumChunks; ++c) {
                const int d = kSolo ? c & 1 : g;
                const uint32_t cpar = (uint32_t)(kSolo ? c >> 1 : c) & 1u;
                const uint32_t htile = sbase + TrSmem::kH + d * kKBlockBytes;
                const uint32_t t_d1 = t_lane + d * 256;
                if (!mbar_wait(d1_full(d), cpar, abort_flag)) {
                    if (lane == 0) report_wait_failure(status, abort_flag, kKidTrans, 9);
                    ok = false;
                    break;
                }
                tc_fence_after_sync();
                uint32_t hpk[16];  // 32 of the chunk's 64 hidden values of this row, packed bf16x2
#pragma unroll
                for (int q = 0; q < 2; ++q) {
                    if (solo && q != own) continue;
                    uint32_t a[16], b[16];
                    tmem_ld16(t_d1 + half * 32 + q * 16, a);
                    tmem_ld16(t_d1 + 64 + half * 32 + q * 16, b);
                    tmem_ld_wait();
                    if (q == 1 || solo) {   // D1 is in registers: the next chunk's G1 may run under the rest of this pass
                        tc_fence_before_sync();
                        __syncwarp();
                        if (lane == 0) mbar_arrive(d1_empty(d));
                    }
#pragma unroll
                    for (int e = 0; e < 16; e += 2) {
                        const float a0 = __uint_as_float(a[e]), a1 = __uint_as_float(a[e + 1]);
                        const float h0 = a0 * sigmoid_fast(a0) * __uint_as_float(b[e]);
                        const float h1 = a1 * sigmoid_fast(a1) * __uint_as_float(b[e + 1]);
                        hpk[q * 8 + e / 2] = pack_bf16x2(h0, h1);
                    }
                }
                // the previous chunk's G2 must have consumed the H buffer before it is overwritten
                if (!mbar_wait(h_free(d), cpar ^ 1u, abort_flag)) {
                    if (lane == 0) report_wait_failure(status, abort_flag, kKidTrans, 10);
                    ok = false;
                    break;
                }
#pragma unroll
                for (int ch = 0; ch < 4; ++ch) {
                    if (solo && ch >> 1 != own) continue;
                    sts128(chunk_addr(htile, row, half * 4 + ch),
                           make_uint4(hpk[ch * 4], hpk[ch * 4 + 1], hpk[ch * 4 + 2], hpk[ch * 4 + 3]));
                }
                fence_proxy_async_smem();
                __syncwarp();
                if (lane == 0) mbar_arrive(h_ready(d));
            }
            if (!ok) break;
            if (!mbar_wait(d2_full(g), ppar, abort_flag)) {
                if (lane == 0) report_wait_failure(status, abort_flag, kKidTrans, 11);
                break;
            }
            if (!mbar_wait(res_full(g), ppar, abort_flag)) {
                if (lane == 0) report_wait_failure(status, abort_flag, kKidTrans, 16);
                break;
            }
            tc_fence_after_sync();
#pragma unroll
            for (int cb = 0; cb < 4; ++cb) {
                if (solo && cb >> 1 != own) continue;
                uint32_t y[16];
                tmem_ld16(t_d2 + half * 64 + cb * 16, y);
                tmem_ld_wait();
                if (cb == 3) {
                    tc_fence_before_sync();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(d2_empty(g));
                }
#pragma unroll
                for (int ch = 0; ch < 2; ++ch) {
                    const uint32_t xa = chunk_addr(xtile, row, half * 8 + cb * 2 + ch);
                    const uint4 xv = lds128(xa);
                    const uint32_t xw[4] = {xv.x, xv.y, xv.z, xv.w};
                    uint32_t o[4];
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const int e = ch * 8 + j * 2;
                        float v0 = m * __uint_as_float(y[e]);
                        float v1 = m * __uint_as_float(y[e + 1]);
                        if (add_residual) {
                            v0 += bf16lo(xw[j]);
                            v1 += bf16hi(xw[j]);
                        }
                        o[j] = pack_bf16x2(v0, v1);
                    }
                    sts128(xa, make_uint4(o[0], o[1], o[2], o[3]));
                }
            }
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) mbar_arrive(out_ready(g));
        }
    }

    tc_fence_before_sync();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after_sync();
        tmem_dealloc(tmem_base, 512);
    }
}

// ------------------------------------------------------------------------------------------------ c = 64, n = 2
// The template stack's widths: the hidden layer is one chunk of 128, all weights (48 KB) stay resident and a tile is two
// GEMMs. Bound by HBM and by the hand-offs of a tile (16 KB in, 16 KB out); two row groups per SM are in flight (their
// accumulators fill the tensor memory), each with a second x buffer, so that its next tile lands while this one is
// computed.
struct Tr64Smem {
    static constexpr uint32_t kWab = 0;                          // [W_a; W_b]: 256 rows x 128 B
    static constexpr uint32_t kWo = 32768;                       // W_out: 2 k-blocks x [64 rows x 128 B]
    static constexpr uint32_t kX = kWo + 16384;                  // 2 groups x 2 buffers x 16 KB
    static constexpr uint32_t kH = kX + 4 * kKBlockBytes;        // 2 groups x 2 k-blocks x 16 KB
    static constexpr uint32_t kParams = kH + 4 * kKBlockBytes;   // gamma, beta
    static constexpr uint32_t kXch = kParams + 1024;
    static constexpr uint32_t kBars = kXch + 4096;
    static constexpr uint32_t kTotal = kBars + 192;
    static constexpr uint32_t kDyn = kTotal + 1024;
};

constexpr int kTr64Threads = 32 * (3 + 2 * 8);

__global__ void __launch_bounds__(kTr64Threads, 1)
transition64_kernel(const __grid_constant__ CUtensorMap tmX, const __grid_constant__ CUtensorMap tmOut,
                    const __grid_constant__ CUtensorMap tmWa, const __grid_constant__ CUtensorMap tmWb,
                    const __grid_constant__ CUtensorMap tmWo, const __nv_bfloat16* __restrict__ mask,
                    const __nv_bfloat16* __restrict__ ln_w, const __nv_bfloat16* __restrict__ ln_b,
                    long long rows, int add_residual, int* status) {
    using Sm = Tr64Smem;
    constexpr int C = 64;
    extern __shared__ uint8_t smem_raw[];
    const uint32_t sbase = (smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t* gbase = smem_raw + (sbase - smem_u32(smem_raw));
    float* prm = reinterpret_cast<float*>(gbase + Sm::kParams);
    const uint32_t bars = sbase + Sm::kBars;
    const uint32_t w_full = bars;
    auto x_full = [&](int g, int b) { return bars + 8u * (1 + g * 2 + b); };
    auto x_empty = [&](int g, int b) { return bars + 8u * (5 + g * 2 + b); };
    auto a_ready = [&](int g) { return bars + 8u * (9 + g); };
    auto d1_full = [&](int g) { return bars + 8u * (11 + g); };
    auto h_ready = [&](int g) { return bars + 8u * (13 + g); };
    auto d2_full = [&](int g) { return bars + 8u * (15 + g); };
    auto out_ready = [&](int g) { return bars + 8u * (17 + g); };   // the group's result lies in the x buffer
    volatile uint32_t* tmem_ptr = reinterpret_cast<volatile uint32_t*>(gbase + Sm::kBars + 160);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(gbase + Sm::kBars + 168);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const long long num_tiles = (rows + kRows - 1) / kRows;
    const long long my_tiles = tiles_of_block(num_tiles);

    if (threadIdx.x == 0) {
        mbar_init(w_full, 1);
        for (int g = 0; g < 2; ++g) {
            for (int b = 0; b < 2; ++b) {
                mbar_init(x_full(g, b), 1);
                mbar_init(x_empty(g, b), 1);
            }
            mbar_init(a_ready(g), 8);
            mbar_init(d1_full(g), 1);
            mbar_init(h_ready(g), 8);
            mbar_init(d2_full(g), 1);
            mbar_init(out_ready(g), 8);
        }
        *abort_flag = 0;
        mbar_fence_init();
        prefetch_tmap(&tmX);
    }
    if (threadIdx.x < C) {
        prm[threadIdx.x] = __bfloat162float(ln_w[threadIdx.x]);
        prm[128 + threadIdx.x] = __bfloat162float(ln_b[threadIdx.x]);
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
    // TMEM: group g: D1 = [a 128 | b 128] at g * 256; D2 (64 columns) over the a half once D1 has been read

    if (warp == 0) {
        if (elect_one()) {
            mbar_arrive_expect_tx(w_full, 49152);
            tma_load_2d(sbase + Sm::kWab, &tmWa, w_full, 0, 0);
            tma_load_2d(sbase + Sm::kWab + 16384, &tmWb, w_full, 0, 0);
            for (int kb = 0; kb < 2; ++kb) tma_load_2d(sbase + Sm::kWo + kb * 8192, &tmWo, w_full, kb * 64, 0);
            grid_wait();
            for (long long lt = 0; lt < my_tiles; ++lt) {
                const int g = (int)(lt & 1), b = (int)((lt >> 1) & 1);
                const long long tile = blockIdx.x + lt * gridDim.x;
                if (!mbar_wait(x_empty(g, b), ((uint32_t)(lt >> 2) & 1u) ^ 1u, abort_flag)) {
                    report_wait_failure(status, abort_flag, kKidTrans, 21);
                    break;
                }
                mbar_arrive_expect_tx(x_full(g, b), kKBlockBytes);
                tma_load_2d(sbase + Sm::kX + (g * 2 + b) * kKBlockBytes, &tmX, x_full(g, b), 0, (int)(tile * kRows));
            }
        }
    } else if (warp <= 2) {
        if (elect_one()) {
            const int g = warp - 1;
            grid_wait();   // (the stores)
            bool ok = mbar_wait(w_full, 0, abort_flag);
            if (!ok) report_wait_failure(status, abort_flag, kKidTrans, 22);
            for (long long lt = g; lt < my_tiles && ok; lt += 2) {
                const uint32_t ph = (uint32_t)(lt >> 1) & 1u;
                const uint32_t xtile = sbase + Sm::kX + (g * 2 + ph) * kKBlockBytes;
                if (!mbar_wait(a_ready(g), ph, abort_flag)) {
                    report_wait_failure(status, abort_flag, kKidTrans, 23);
                    break;
                }
                tc_fence_after_sync();
                mma_rows<64>(tmem_base + g * 256, xtile, sbase + Sm::kWab, 0, idesc_bf16_f32(128, 256), false);
                mma_commit(d1_full(g));
                if (!mbar_wait(h_ready(g), ph, abort_flag)) {
                    report_wait_failure(status, abort_flag, kKidTrans, 24);
                    break;
                }
                tc_fence_after_sync();
                mma_rows<128>(tmem_base + g * 256, sbase + Sm::kH + g * 2 * kKBlockBytes, sbase + Sm::kWo, 8192,
                              idesc_bf16_f32(128, 64), false);
                mma_commit(d2_full(g));
                if (!mbar_wait(out_ready(g), ph, abort_flag)) {
                    report_wait_failure(status, abort_flag, kKidTrans, 28);
                    break;
                }
                tma_store_3d(&tmOut, xtile, 0, (int)((blockIdx.x + lt * gridDim.x) * kRows), 0);
                tma_store_commit();
                tma_store_wait_read<0>();
                mbar_arrive(x_empty(g, (int)ph));
            }
            tma_store_wait_all<0>();
        }
    } else {
        const int g = (warp - 3) >> 3;
        const int quad = warp & 3;
        const int half = ((warp - 3) >> 2) & 1;
        const int row = quad * 32 + lane;
        float* xch = reinterpret_cast<float*>(gbase + Sm::kXch) + g * 512;
        const uint32_t htile = sbase + Sm::kH + g * 2 * kKBlockBytes;
        const uint32_t td = tmem_base + ((uint32_t)(quad * 32) << 16) + g * 256;
        grid_wait();
        for (long long lt = g; lt < my_tiles; lt += 2) {
            const uint32_t ph = (uint32_t)(lt >> 1) & 1u;
            const int b = (int)ph;
            const long long tile = blockIdx.x + lt * gridDim.x;
            const long long grow = tile * kRows + row;
            const uint32_t xtile = sbase + Sm::kX + (g * 2 + b) * kKBlockBytes;
            if (!mbar_wait(x_full(g, b), (uint32_t)(lt >> 2) & 1u, abort_flag)) {
                if (lane == 0) report_wait_failure(status, abort_flag, kKidTrans, 25);
                break;
            }
            uint32_t raw[C / 4];
            load_half_row<C>(xtile, row, half, raw);
            {
                float mean, rstd;
                half_row_stats_xwarp<C>(raw, row, half, xch, 1 + g, 256, mean, rstd);
                store_normalized_half_row<C>(xtile, row, half, raw, mean, rstd, prm, prm + 128);
            }
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) mbar_arrive(a_ready(g));
            float m = 1.0f;
            if (mask != nullptr && grow < rows) m = __bfloat162float(mask[grow]);
            if (!mbar_wait(d1_full(g), ph, abort_flag)) {
                if (lane == 0) report_wait_failure(status, abort_flag, kKidTrans, 26);
                break;
            }
            tc_fence_after_sync();
#pragma unroll
            for (int q = 0; q < 4; ++q) {   // this thread's 64 hidden values: k-block `half` of the h tile
                uint32_t a[16], bb[16], o[8];
                tmem_ld16(td + half * 64 + q * 16, a);
                tmem_ld16(td + 128 + half * 64 + q * 16, bb);
                tmem_ld_wait();
#pragma unroll
                for (int e = 0; e < 16; e += 2) {
                    const float a0 = __uint_as_float(a[e]), a1 = __uint_as_float(a[e + 1]);
                    o[e / 2] = pack_bf16x2(a0 * sigmoid_fast(a0) * __uint_as_float(bb[e]),
                                           a1 * sigmoid_fast(a1) * __uint_as_float(bb[e + 1]));
                }
                sts128(chunk_addr(htile, row, half * 8 + q * 2), make_uint4(o[0], o[1], o[2], o[3]));
                sts128(chunk_addr(htile, row, half * 8 + q * 2 + 1), make_uint4(o[4], o[5], o[6], o[7]));
            }
            tc_fence_before_sync();
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) mbar_arrive(h_ready(g));
            if (!mbar_wait(d2_full(g), ph, abort_flag)) {
                if (lane == 0) report_wait_failure(status, abort_flag, kKidTrans, 27);
                break;
            }
            tc_fence_after_sync();
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                uint32_t y[16];
                tmem_ld16(td + half * 32 + q * 16, y);
                tmem_ld_wait();
#pragma unroll
                for (int ch = 0; ch < 2; ++ch) {
                    uint32_t o[4];
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const int e = ch * 8 + j * 2;
                        const uint32_t xr = raw[q * 8 + ch * 4 + j];
                        float v0 = m * __uint_as_float(y[e]), v1 = m * __uint_as_float(y[e + 1]);
                        if (add_residual) {
                            v0 += bf16lo(xr);
                            v1 += bf16hi(xr);
                        }
                        o[j] = pack_bf16x2(v0, v1);
                    }
                    sts128(chunk_addr(xtile, row, half * 4 + q * 2 + ch), make_uint4(o[0], o[1], o[2], o[3]));
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
        tmem_dealloc(tmem_base, 512);
    }
}

}  // namespace

bool transition_supported(int c, int n) { return (c == 128 && n == 4) || (c == 64 && n == 2); }

int transition(const __nv_bfloat16* x, const __nv_bfloat16* mask, __nv_bfloat16* out, long long rows, int c,
               int flags, const of3_transition_params* p, Arena& ws, cudaStream_t st) {
    (void)ws.take(16);
    if (!ws.base) return OF3_OK;
    OF3_REQUIRE(rows < (1LL << 31) - 256, OF3_ERR_SHAPE, "transition: too many rows");
    int rc;
    const uint64_t hidden = c == 128 ? kHidden : 128;
    CUtensorMap tmX, tmOut, tmWa, tmWb, tmWo;
    {
        uint64_t dims[2] = {(uint64_t)c, (uint64_t)rows};
        uint64_t str[1] = {(uint64_t)c * 2};
        uint32_t box[2] = {64, 128};
        if ((rc = make_tmap_bf16(&tmX, x, 2, dims, str, box, true))) return rc;
        // the store map is 3-D only to share tma_store_3d with the other kernels
        uint64_t dims3[3] = {(uint64_t)c, (uint64_t)rows, 1};
        uint64_t str3[2] = {(uint64_t)c * 2, (uint64_t)rows * c * 2};
        uint32_t box3[3] = {64, 128, 1};
        if ((rc = make_tmap_bf16(&tmOut, out, 3, dims3, str3, box3, true))) return rc;
    }
    {
        uint64_t dims[2] = {(uint64_t)c, hidden};
        uint64_t str[1] = {(uint64_t)c * 2};
        uint32_t box[2] = {64, c == 128 ? (uint32_t)kChunk : 128u};
        if ((rc = make_tmap_bf16(&tmWa, p->w_a, 2, dims, str, box, true))) return rc;
        if ((rc = make_tmap_bf16(&tmWb, p->w_b, 2, dims, str, box, true))) return rc;
        uint64_t dimo[2] = {hidden, (uint64_t)c};
        uint64_t stro[1] = {hidden * 2};
        uint32_t boxo[2] = {kChunk, (uint32_t)c};
        if ((rc = make_tmap_bf16(&tmWo, p->w_out, 2, dimo, stro, boxo, true))) return rc;
    }
    if (!device_configured(4)) {
        OF3_CUDA_CHECK(cudaFuncSetAttribute(transition_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                            TrSmem::kDyn));
        OF3_CUDA_CHECK(cudaFuncSetAttribute(transition_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                            TrSmem::kDyn));
        OF3_CUDA_CHECK(cudaFuncSetAttribute(transition64_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                            Tr64Smem::kDyn));
        device_mark_configured(4);
    }
    const long long tiles = (rows + kRows - 1) / kRows;
    // Two tiles per CTA share each weight chunk: an even number of tiles per CTA, once every SM has one (with fewer tiles
    // than SMs a tile has its SM's pipes to itself).
    long long grid = sm_count();
    if (tiles <= grid) grid = tiles;
    else if (tiles < 2 * grid) grid = (tiles + 1) / 2;
    if (grid < 1) grid = 1;
    LaunchScope scope(kKidTrans, st);
    typedef const __nv_bfloat16* P;
    const int residual = (flags & OF3_FLAG_ADD_RESIDUAL) ? 1 : 0;
    if (c == 128)
        OF3_CUDA_CHECK(launch_chained(tiles <= grid ? transition_kernel<true> : transition_kernel<false>, dim3((unsigned)grid),
                                      kTrThreads, TrSmem::kDyn, st, tmX, tmOut, tmWa, tmWb, tmWo, x, mask, (P)p->ln_w,
                                      (P)p->ln_b, rows, residual, device_status_ptr()));
    else
        OF3_CUDA_CHECK(launch_chained(transition64_kernel, dim3((unsigned)grid), kTr64Threads, Tr64Smem::kDyn, st, tmX, tmOut,
                                      tmWa, tmWb, tmWo, mask, (P)p->ln_w, (P)p->ln_b, rows, residual, device_status_ptr()));
    return OF3_OK;
}

}  // namespace fast
}  // namespace of3
