// Triangle attention, bf16 / tcgen05 family (c_z = 128 with 4 heads x 32, c_z = 64 with 4 heads x 16).
//
//   triattn_proj   z tile -> LayerNorm (in place in the A operand) -> [q|k|v] projection on
//                  tcgen05; the 4-wide triangle-bias projection is a fourth small GEMM. q is
//                  stored pre-scaled by log2(e)/sqrt(d), the bias pre-scaled by log2(e), so the
//                  softmax runs on exp2. Layouts: q, k, v as pre-swizzled operand tiles (see the
//                  epilogue), bias as bf16 tiles [head][key block of 32][q][32].
//   triattn_core   streaming attention for (2 lines, head, 128 queries): S = Q K^T + bias on tcgen05 into
//                  TMEM, online softmax (fp32, exp2) by one thread per query row, P written back
//                  to TMEM as bf16 and used from there as the A operand of O += P V. N^3 logits are
//                  never materialised.
//   triattn_out    z tile -> LayerNorm -> linear_g (gate recomputed instead of stored), o tile
//                  * sigmoid(gate) -> linear_o -> + z, TMA-stored.
// "line" is the leading index of the (possibly transposed) pair tensor: with kTransposed the
// kernels read and write z through transposed TMA boxes, which gives the ending-node layer
// (and PairBlock's transpose / tri_att_end / transpose) without moving z.
// Reference: openfold3/core/model/layers/triangular_attention.py:102-167,
//            openfold3/core/model/primitives/attention.py:94-135, 270-310.
#include "modules.cuh"
#include "rowtile.cuh"
#include "runtime.cuh"

namespace of3 {
namespace fast {
namespace {

using namespace umma;
using namespace rowtile;

constexpr int kH = 4;   // heads; the head dimension is D = C / 4: 32, or 16 in the template stack
constexpr int kKidProj = 5;
constexpr int kKidCore = 6;
constexpr int kKidOut = 7;
constexpr float kLog2e = 1.4426950408889634f;

// R = lines per sample (R == N for a whole pair tensor, N / P for a row shard)
// z tile of a line: rows (line, t0..t0+127) of the view; transposed view = z[b, t, line, :]
template <int C, bool kTransposed>
__device__ __forceinline__ void load_z_tile(uint32_t dst, const CUtensorMap* tm, uint32_t bar,
                                            const TileWalk& c, int R) {
    for (int kb = 0; kb < C / 64; ++kb) {
        if (kTransposed)
            tma_load_4d(dst + kb * kKBlockBytes, tm, bar, kb * 64, c.line, c.tile * kRows, c.b);
        else
            tma_load_3d(dst + kb * kKBlockBytes, tm, bar, kb * 64, c.tile * kRows, c.b * R + c.line);
    }
}

// =====================================================================================
// triattn_proj
// =====================================================================================
template <int C>
struct ProjSmem {
    static constexpr int kStages = C == 128 ? 3 : 4;           // z tiles in flight
    static constexpr uint32_t kWKb = 3 * C * 128;             // one k-block of [q|k|v]
    static constexpr uint32_t kW = 0;
    static constexpr uint32_t kZ = C / 64 * kWKb;
    static constexpr uint32_t kGamma = kZ + kStages * tile_bytes<C>();
    static constexpr uint32_t kBeta = kGamma + 512;
    static constexpr uint32_t kWb = kBeta + 512;              // bias weight as a B operand: k-blocks of [16 x 128 B]
    static constexpr uint32_t kBars = kWb + 4096;
    static constexpr uint32_t kTotal = kBars + 192;
    static constexpr uint32_t kDyn = kTotal + 1024;
};

// Operand images of the attention core: per (sample, head) tiles that hold a line each, the tiles of neighbouring lines
// contiguous (the two lines of a CTA arrive with one bulk copy), every tile the shared-memory image of a K-major
// tcgen05 operand:
//   q [b*4 + h][query tile of 128][line < rpad][128][D]   rows of 64 bytes (64-byte swizzle) or, D = 16, of 32 bytes
//   k [b*4 + h][key block of 64  ][line < rpad][64][D]    likewise
//   v [b*4 + h][key block of 64  ][line < rpad][D][64]    128-byte rows, 128-byte swizzle
// 16-byte chunk c of row r of a q / k tile lies at chunk c ^ qk_xor(r).
constexpr int kBK = 64;  // keys per key block = per attention step
template <int D>
__device__ __forceinline__ int qk_xor(int r) { return D == 32 ? (r >> 1) & 3 : (r >> 2) & 1; }

// warps: 0 producer, 1 MMA issuer, 2..9 LayerNorm (two threads per row), 10..13 epilogue of TMEM slot 0 (q, k), 14..17 of
// slot 1 (v and the 4-wide triangle bias): the epilogue is the longest part of a tile's chain. The bias projection is a fourth GEMM (N = 16 with 12 zero rows)
// instead of 1024 FMAs per row inside the LayerNorm pass.
constexpr int kProjLnWarps = 8;
constexpr int kProjThreads = 32 * (2 + kProjLnWarps + 8);
constexpr int kBiasK = 32;  // keys per bias row
// Pair-bias image: bf16, pre-scaled by log2(e), [b*4 + head][key block of 32][query row][32 keys]: the 128 rows
// of a query tile and one key block are contiguous (one untiled bulk copy) and each 64-byte row is stored in the
// 64-byte swizzle of a K-major tcgen05 A operand (16-byte chunk c of query row q at chunk c ^ ((q / 2) % 4)),
// because the attention kernel adds the bias on the tensor pipe: S += bias_tile * I_32^T.

// 64 channels: two CTAs share an SM (template stack, N = 300 x 4: 58 -> 49 us)
template <int C, bool kTransposed>
__global__ void __launch_bounds__(kProjThreads, C == 64 ? 2 : 1)
triattn_proj_kernel(const __grid_constant__ CUtensorMap tmZ, const __grid_constant__ CUtensorMap tmWq,
                    const __grid_constant__ CUtensorMap tmWk, const __grid_constant__ CUtensorMap tmWv,
                    const __grid_constant__ CUtensorMap tmWb,
                    const __nv_bfloat16* __restrict__ ln_w, const __nv_bfloat16* __restrict__ ln_b,
                    __nv_bfloat16* __restrict__ q_out,
                    __nv_bfloat16* __restrict__ k_out, __nv_bfloat16* __restrict__ vt_out,
                    __nv_bfloat16* __restrict__ tb_out, const __nv_bfloat16* __restrict__ mask,
                    __nv_bfloat16* __restrict__ mask_t, int B, int R, int N, int npad, int row0, int* status) {
    using Sm = ProjSmem<C>;
    constexpr int kSt = Sm::kStages, D = C / kH;
    extern __shared__ uint8_t smem_raw[];
    const uint32_t sbase = (smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t* gbase = smem_raw + (sbase - smem_u32(smem_raw));
    float* gamma = reinterpret_cast<float*>(gbase + Sm::kGamma);
    float* beta = reinterpret_cast<float*>(gbase + Sm::kBeta);
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
            mbar_init(a_ready(s), kProjLnWarps);
        }
        for (int q = 0; q < 2; ++q) {
            mbar_init(slot_full(q), 1);
            mbar_init(slot_empty(q), 4);
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
        tmem_alloc(smem_u32((const void*)tmem_ptr), 4 * C);
        tmem_relinquish();
    }
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem_base = *tmem_ptr;
    grid_trigger();
    if (warp >= 2) grid_wait();
    // 128 channels, lone tiles: the LayerNorm warps, done with theirs, take k and half of v's heads. With trimul_in's share of the
    // positions, four blocks of the trunk: N = 37 408.1 -> 404.7 us, 64 406.9 -> 402.8, 100 447.9 -> 445.8. (64 channels: registers.)
    const bool solo = C == 128 && num_tiles <= (long long)gridDim.x;
    // TMEM: slot 0 = [q|k] columns [0,2C), slot 1 = v columns [2C,3C) + triangle bias [3C,3C+16)

    if (warp == 0) {
        if (elect_one()) {
            mbar_arrive_expect_tx(w_full, C / 64 * (Sm::kWKb + 2048));
            const CUtensorMap* wm[3] = {&tmWq, &tmWk, &tmWv};
            for (int w = 0; w < 3; ++w)
                for (int kb = 0; kb < C / 64; ++kb)
                    tma_load_2d(sbase + Sm::kW + kb * Sm::kWKb + w * C * 128, wm[w], w_full, kb * 64, 0);
            // rows 4..15 of the box lie outside the [4 x C] weight: the copy fills them with zeros
            for (int kb = 0; kb < C / 64; ++kb) tma_load_2d(sbase + Sm::kWb + kb * 2048, &tmWb, w_full, kb * 64, 0);
            grid_wait();
            uint32_t it = 0;
            TileWalk tc(blockIdx.x, gridDim.x, R, tiles_per_line);
            for (long long t = blockIdx.x; t < num_tiles; t += gridDim.x, ++it, tc.next()) {
                const int s = it % kSt;
                if (!mbar_wait(z_empty(s), ((it / kSt) & 1u) ^ 1u, abort_flag)) {
                    report_wait_failure(status, abort_flag, kKidProj, 1);
                    break;
                }
                mbar_arrive_expect_tx(z_full(s), tile_bytes<C>());
                load_z_tile<C, kTransposed>(sbase + Sm::kZ + s * tile_bytes<C>(), &tmZ, z_full(s), tc, R);
            }
        }
    } else if (warp == 1) {
        if (elect_one()) {
            bool ok = mbar_wait(w_full, 0, abort_flag);
            if (!ok) report_wait_failure(status, abort_flag, kKidProj, 2);
            uint32_t it = 0;
            for (long long t = blockIdx.x; t < num_tiles && ok; t += gridDim.x, ++it) {
                const int s = it % kSt;
                if (!mbar_wait(a_ready(s), (it / kSt) & 1u, abort_flag)) {
                    report_wait_failure(status, abort_flag, kKidProj, 3);
                    break;
                }
                for (int q = 0; q < 2; ++q) {
                    if (!mbar_wait(slot_empty(q), (it & 1u) ^ 1u, abort_flag)) {
                        report_wait_failure(status, abort_flag, kKidProj, 4);
                        ok = false;
                        break;
                    }
                    tc_fence_after_sync();
                    const uint32_t ztile = sbase + Sm::kZ + s * tile_bytes<C>();
                    mma_rows<C>(tmem_base + q * 2 * C, ztile, sbase + Sm::kW + q * 2 * C * 128, Sm::kWKb,
                                q == 0 ? idesc_bf16_f32(128, 2 * C) : idesc_bf16_f32(128, C), false);
                    if (q == 1)
                        mma_rows<C>(tmem_base + 3 * C, ztile, sbase + Sm::kWb, 2048, idesc_bf16_f32(128, 16), false);
                    mma_commit(slot_full(q));
                }
                if (ok) mma_commit(z_empty(s));
            }
        }
    } else if (warp < 2 + kProjLnWarps) {
        // LayerNorm warps: normalise in place (the A operand of all four GEMMs); a warp takes 16 positions, lanes 0..15
        // their first half of the channels, lanes 16..31 the other half
        const int row = (warp - 2) * 16 + (lane & 15), half = lane >> 4;
        uint32_t it = 0;
        TileWalk tc(blockIdx.x, gridDim.x, R, tiles_per_line);
        for (long long t = blockIdx.x; t < num_tiles; t += gridDim.x, ++it, tc.next()) {
            const int s = it % kSt;
            // The transposed view's mask column, as a row for the attention core: there every block of 128 queries and every
            // head of a line would fetch a sector per key (N = 768: 85 of 762 us).
            const int pos = tc.tile * kRows + row;
            const bool copy_mask = kTransposed && mask_t != nullptr && half == 0 && pos < N;
            __nv_bfloat16 mv = __float2bfloat16_rn(1.0f);
            if (copy_mask) mv = mask[((long long)tc.b * N + pos) * N + tc.line];
            if (!mbar_wait(z_full(s), (it / kSt) & 1u, abort_flag)) {
                if (lane == 0) report_wait_failure(status, abort_flag, kKidProj, 5);
                break;
            }
            const uint32_t tile = sbase + Sm::kZ + s * tile_bytes<C>();
            uint32_t raw[C / 4];
            load_half_row<C>(tile, row, half, raw);
            float mean, rstd;
            half_row_stats<C>(raw, mean, rstd);
            store_normalized_half_row<C>(tile, row, half, raw, mean, rstd, gamma, beta);
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) mbar_arrive(a_ready(s));
            if (copy_mask) mask_t[((long long)tc.b * R + tc.line) * npad + pos] = mv;
        }
    }
    if (warp >= (solo ? 2 : 2 + kProjLnWarps)) {
        // epilogue warps
        const bool helper = C == 128 && warp < 2 + kProjLnWarps, shared = solo && !helper;
        const int set = ((warp - 2) >> 2) & 1;
        const int qk_end = shared ? 1 : 2, h_end = shared ? kH / 2 : kH;
        const int quad = warp & 3;
        const int row = quad * 32 + lane;
        const float qscale = kLog2e * rsqrtf((float)D);
        const int rpad = (R + 3) & ~3;
        const int nkb = npad >> 6;
        const uint32_t taddr = tmem_base + ((uint32_t)(quad * 32) << 16);
        uint32_t it = 0;
        TileWalk tc(blockIdx.x, gridDim.x, R, tiles_per_line);
        for (long long t = blockIdx.x; t < num_tiles; t += gridDim.x, ++it, tc.next()) {
            const int pos = tc.tile * kRows + row;
            const bool valid = pos < npad;   // positions in [N, npad) are written as zeros (key padding)
            const bool live = pos < N;
            if (!mbar_wait(slot_full(set), it & 1u, abort_flag)) {
                if (lane == 0) report_wait_failure(status, abort_flag, kKidProj, 6 + set);
                break;
            }
            tc_fence_after_sync();
            if (set == 0) {
                // ---- slot 0: q (columns [0, C)) and k ([C, 2C))
#pragma unroll 1
                for (int qk = helper ? 1 : 0; qk < qk_end; ++qk) {
                    __nv_bfloat16* base = qk == 0 ? q_out : k_out;
                    const float sl = live ? (qk == 0 ? qscale : 1.0f) : 0.f;
#pragma unroll 1
                    for (int h = 0; h < kH; ++h) {
                        uint32_t r[D];
                        if constexpr (D == 32) tmem_ld32(taddr + qk * C + h * D, r);
                        else tmem_ld16(taddr + qk * C + h * D, r);
                        tmem_ld_wait();
                        if (valid || qk == 0) {
                            const long long bh = (long long)tc.b * kH + h;
                            const long long rowidx = qk == 0
                                ? ((bh * tiles_per_line + tc.tile) * rpad + tc.line) * 128 + row
                                : ((bh * nkb + (pos >> 6)) * rpad + tc.line) * kBK + (pos & 63);
                            __nv_bfloat16* dst = base + rowidx * D;
                            // 32 bytes at a time: chunks c2 and c2 + 1 of the row lie at c2 ^ x and (c2 + 1) ^ x
                            const int x = qk_xor<D>(pos);
#pragma unroll
                            for (int c2 = 0; c2 < D / 8; c2 += 2) {
                                uint32_t o[8], w[8];
#pragma unroll
                                for (int e = 0; e < 8; ++e)
                                    o[e] = pack_bf16x2(sl * __uint_as_float(r[c2 * 8 + 2 * e]),
                                                       sl * __uint_as_float(r[c2 * 8 + 2 * e + 1]));
#pragma unroll
                                for (int e = 0; e < 8; ++e) w[e] = (x & 1) ? o[e ^ 4] : o[e];
                                stg256_or_2x128(dst + ((c2 ^ (x & 2)) << 3), w, aligned32(base));
                            }
                        }
                    }
                }
                tc_fence_before_sync();
                __syncwarp();
                if (lane == 0 && !helper) mbar_arrive(slot_empty(0));
            } else {
                // ---- slot 1: v, transposed; the triangle bias
#pragma unroll 1
                for (int h = helper ? kH / 2 : 0; h < h_end; ++h) {
                    uint32_t r[D];
                    if constexpr (D == 32) tmem_ld32(taddr + 2 * C + h * D, r);
                    else tmem_ld16(taddr + 2 * C + h * D, r);
                    tmem_ld_wait();
                    if (valid) {
                        __nv_bfloat16* tile = vt_out + ((((long long)tc.b * kH + h) * nkb + (pos >> 6)) * rpad + tc.line) *
                                                           (long long)(D * kBK);
                        const int c = (pos & 63) >> 3, w = pos & 7;
#pragma unroll
                        for (int e = 0; e < D; ++e)
                            tile[e * kBK + (((c ^ (e & 7)) << 3) | w)] =
                                __float2bfloat16_rn(live ? __uint_as_float(r[e]) : 0.f);
                    }
                }
                if (helper) break;
                uint32_t tbr[16];  // triangle bias of this position: columns 3C..3C+3, pre-scaled for exp2
                tmem_ld16(taddr + 3 * C, tbr);
                tmem_ld_wait();
                tc_fence_before_sync();
                __syncwarp();
                if (lane == 0) mbar_arrive(slot_empty(1));
                const int nkb32 = (N + kBiasK - 1) / kBiasK;
                if (pos < nkb32 * kBiasK) {  // the key padding of the last row is read by the attention kernel: zeros
                    // row0 = index of this shard's first line among all query rows (the swizzle follows the global row)
                    const int kc = (((pos & 31) >> 3) ^ (((row0 + tc.line) >> 1) & 3)) * 8 + (pos & 7);
#pragma unroll
                    for (int h = 0; h < kH; ++h)
                        tb_out[((((long long)tc.b * kH + h) * nkb32 + (pos >> 5)) * R + tc.line) * kBiasK + kc] =
                            __float2bfloat16_rn(live ? __uint_as_float(tbr[h]) * kLog2e : 0.f);
                }
            }
        }
    }

    tc_fence_before_sync();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after_sync();
        tmem_dealloc(tmem_base, 4 * C);
    }
}

// =====================================================================================
// triattn_core
// =====================================================================================
// One CTA = one head, 128 queries and TWO lines of the pair tensor, 64 keys per step; two CTAs share an SM
// (their prologues, epilogues and waits interleave). Few lines: ONE per CTA, up to three CTAs per SM (finish_impl).
// Per line and step j:
//   S warp        S_j = Q K_j^T + Tb_j I^T: 128 x 64 logits in TMEM, issued as soon as the softmax warps have S_{j-1} in
//                 registers. The pair-bias tiles [128 q x 32 k] (bf16, shared by both lines) are a second A operand
//                 against a 32 x 32 identity: a bf16 value times 1.0 accumulated in fp32 is exact.
//   softmax warps thread = query row = TMEM lane: S -> registers [+ mask bias where the block has masked keys], row
//                 maximum, P = exp2(S - m) rounded to bf16, sum of the rounded values, P into TMEM columns of its own
//   PV warp       O[128 x D] += P_j V_j with P read from TMEM as the A operand
// What bounds it: one exponential per logit (N = 768: 1.8e9 per launch, 402 us of the MUFU pipe at 1.9 GHz), and the latency
// of a step's hand-offs: polls, TMEM loads and stores, MMAs and commits go through the same queue as the exponentials of the
// four softmax warps of a scheduler and take 50 - 100 cycles each behind them (a step of a line: 3260 cycles, of which 1790
// exponentials, 940 waits for S and P V, 380 the load of S). The tensor pipe is not the limit: 298 cycles per line and step
// in a loop of the same MMAs, of 815. Hence few such instructions in a row per warp: a warp per line issues S, a third one P V
// (one warp for both: the next S queued behind P V); a K / bias stage is handed back by a commit behind S, not by the softmax
// warps once they have read S (675 -> 660 us at N = 768, together 652); P V of the step before is awaited before the
// exponentials, so that nothing divides these (644). Measured and worse: persistent blocks with 128 keys per step, two lines
// per SM and the row sum on the tensor pipe 774 (two softmax warps per scheduler do not hide the hand-offs); no row maximum,
// the block taken again where its sum overflows 733; all of P stored at the end of a step 701; S loaded in two halves 662.
// Earlier steps, N = 768: 32 keys per step, two S buffers, P over S, row sum as a column of O: 759. 64 keys per step, P over
// S: a step waits 1100 of its 3500 cycles for P V and the next S. P beside S, so that S_{j+1} is computed under the
// softmax of S_j (the column of O for the row sum no longer fits, the threads take it: 28 us): with the bias added by
// the threads 805 (it costs them 160), on the tensor pipe 682 (12.2).
// TMEM columns of a line (128): S [0,64), P [64,96), O [96, 96 + D).
// The running maximum m used for scaling is only raised when the row maximum exceeds it by more than 32
// (2^32 head room in P, in bf16 as precise as below 1): then, and only then, the thread rescales its O row in TMEM and
// its row sum. The result is exact: numerator and denominator always share one scale, and one rounding of P: the row sum
// adds the bf16 values that the GEMM reads (mixed-precision adds, N = 768 649 -> 666 us, N = 2048 11.07 -> 11.25 ms;
// unpacking them for packed adds 681, 11.66). Summed before the rounding, what it does to the dominant keys of a row, up to
// 2^-9, no longer cancels: 13 % more error in o where the values are alike.
constexpr int kBQ = 128;      // queries per CTA
constexpr int kMaxKeys = 2048;   // one CTA keeps a mask-bias row per line in shared memory
constexpr int kKvStages = 2;     // ring of K + bias tiles, ring of V tiles
constexpr int kLinePad = 4;   // the operand images pad the line count of a sample to a multiple of this
// three warpgroups: producer, S of line 0, S of line 1, P V of both; the softmax warps of line 0; of line 1 (one line: producer, S,
// P V and an idle warp; the softmax warps)
template <int kLines>
constexpr int kCoreThreads = 128 * (1 + kLines);
template <int kLines>
constexpr int kCorePerSm = kLines == 1 ? 3 : 2;
// registers: the block is launched with 80 per thread (two blocks of 384 threads per SM, or three of 256); the issuing warpgroup gives up
// what the softmax warpgroups, which hold a row of 64 logits, take. (The issuing warps need more than 32; with 96 for
// the softmax warps it is no faster.)
constexpr int kCoreRegsLaunch = 80, kCoreRegsIssue = 64, kCoreRegsSoftmax = 88;
static_assert(kCoreRegsIssue + 2 * kCoreRegsSoftmax <= 3 * kCoreRegsLaunch && kCoreRegsIssue + kCoreRegsSoftmax <= 2 * kCoreRegsLaunch,
              "register split");
constexpr float kRescaleThreshold = 32.0f;
constexpr uint32_t kTbTileBytes = kBQ * kBiasK * 2;    // 8192: 128 query rows x 32 keys
constexpr uint32_t kColP = 64, kColO = 96;

template <int D, int kLines>
struct CoreSmem {
    static constexpr uint32_t kQBytes = kBQ * D * 2;
    static constexpr uint32_t kKBytes = kBK * D * 2;
    static constexpr uint32_t kVBytes = D * kBK * 2;
    static constexpr uint32_t kQ = 0;                                     // lines
    static constexpr uint32_t kK = kQ + kLines * kQBytes;                 // stages x lines
    static constexpr uint32_t kTb = kK + kKvStages * kLines * kKBytes;    // stages x 2 bias tiles [128 q][32 k] bf16
    static constexpr uint32_t kV = kTb + kKvStages * 2 * kTbTileBytes;    // stages x lines
    static constexpr uint32_t kIdent = kV + kKvStages * kLines * kVBytes; // 2 KB: 32 x 32 identity (B operand)
    static constexpr uint32_t kBars = kIdent + 2048;
    static constexpr uint32_t kFlags = kBars + 256;                       // lines x 32 block flags (bytes)
    static constexpr uint32_t kMb = kFlags + kLines * 32;                 // lines x nkeys_pad floats
    static uint32_t dyn_bytes(int nblk) { return kMb + kLines * nblk * kBK * 4 + 1024; }
};

// kColumns: where the mask of a transposed view is read in place (strides that are not constants cost the short calls 0.3 %)
template <int D, bool kColumns, int kLines>
__global__ void __launch_bounds__(kCoreThreads<kLines>, kCorePerSm<kLines>)
triattn_core_kernel(const __nv_bfloat16* __restrict__ q_img, const __nv_bfloat16* __restrict__ k_img,
                    const __nv_bfloat16* __restrict__ v_img, const __nv_bfloat16* __restrict__ tb_img,
                    const __nv_bfloat16* __restrict__ mask, int mask_pitch, __nv_bfloat16* __restrict__ o_out, int R,
                    int N, float inf, int* status) {
    using Sm = CoreSmem<D, kLines>;
    extern __shared__ uint8_t smem_raw[];
    const uint32_t sbase = (smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t* gbase = smem_raw + (sbase - smem_u32(smem_raw));
    float* mbs = reinterpret_cast<float*>(gbase + Sm::kMb);
    volatile uint8_t* mbflag = gbase + Sm::kFlags;
    const uint32_t bars = sbase + Sm::kBars;
    constexpr int kSt = kKvStages;
    const uint32_t q_full = bars;
    auto kb_full = [&](int s) { return bars + 8u * (1 + s); };             // K tiles + bias tiles landed
    auto kb_empty = [&](int s) { return bars + 8u * (1 + kSt + s); };
    auto v_full = [&](int s) { return bars + 8u * (1 + 2 * kSt + s); };
    auto v_empty = [&](int s) { return bars + 8u * (1 + 3 * kSt + s); };
    constexpr int kB1 = 1 + 4 * kSt;
    auto s_full = [&](int L) { return bars + 8u * (kB1 + L); };
    auto p_ready = [&](int L) { return bars + 8u * (kB1 + kLines + L); };
    auto pv_done = [&](int L) { return bars + 8u * (kB1 + 2 * kLines + L); };
    auto s_read = [&](int L) { return bars + 8u * (kB1 + 3 * kLines + L); };  // S is in the softmax warps' registers
    constexpr int kNumBars = kB1 + 4 * kLines;
    static_assert(8 * kNumBars + 16 <= 256, "barrier block");
    volatile uint32_t* tmem_ptr = reinterpret_cast<volatile uint32_t*>(gbase + Sm::kBars + 8 * kNumBars);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(gbase + Sm::kBars + 8 * kNumBars + 8);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int n_qt = (N + kBQ - 1) / kBQ;
    const int groups_per_b = (R + kLines - 1) / kLines;
    const int qt = blockIdx.x % n_qt;
    const int h = (blockIdx.x / n_qt) % kH;
    const int lg = blockIdx.x / (n_qt * kH);
    const int b = lg / groups_per_b;
    const int line0 = (lg % groups_per_b) * kLines;
    const int q0 = qt * kBQ;
    const int nblk = (N + kBK - 1) / kBK;
    const int nkp = nblk * kBK;
    // (a line past the end of the sample: the images' padding line, unwritten, with the mask of the group's first; not stored)
    auto line_of = [&](int L) { return (line0 + L < R) ? line0 + L : line0; };

    if (threadIdx.x == 0) {
        mbar_init(q_full, 1);
        for (int s = 0; s < kSt; ++s) {
            mbar_init(kb_full(s), 1);
            mbar_init(kb_empty(s), kLines);      // each line's commit after the S that read the stage
            mbar_init(v_full(s), 1);
            mbar_init(v_empty(s), kLines);       // each line's commit after the P V that read the stage
        }
        for (int L = 0; L < kLines; ++L) {
            mbar_init(s_full(L), 1);
            mbar_init(p_ready(L), 4);
            mbar_init(pv_done(L), 1);
            mbar_init(s_read(L), 4);
        }
        *abort_flag = 0;
        mbar_fence_init();
    }
    // 32 x 32 identity, bf16, K-major with the 64-byte swizzle: element (n, n) of row n
    for (int idx = threadIdx.x; idx < 32 * 16; idx += kCoreThreads<kLines>) {
        const int n = idx >> 4, w = idx & 15;  // row, 32-bit word of the row (2 elements)
        const int k = w * 2;                   // first element of the word
        uint32_t v = 0;
        if (k == n) v = 0x00003F80u;
        if (k + 1 == n) v = 0x3F800000u;
        const int chunk = (k >> 3) ^ ((n >> 1) & 3);
        *reinterpret_cast<uint32_t*>(gbase + Sm::kIdent + n * 64 + chunk * 16 + (w & 3) * 4) = v;
    }
    fence_proxy_async_smem();
    if (warp == 0) {
        tmem_alloc(smem_u32((const void*)tmem_ptr), kLines * 128);
        tmem_relinquish();
    }
    tc_fence_before_sync();
    __syncthreads();  // the only CTA-wide barrier before the teardown: the copies and GEMMs start right behind it
    tc_fence_after_sync();
    const uint32_t tmem_base = *tmem_ptr;
    grid_trigger();
    grid_wait();

    if (warp < 4) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kCoreRegsIssue));
        if (warp == 0) {
            if (lane == 0) {
                const int rpad = (R + kLinePad - 1) / kLinePad * kLinePad;
                const int nkb32 = (N + kBiasK - 1) / kBiasK;
                const long long bh = (long long)b * kH + h;
                mbar_arrive_expect_tx(q_full, kLines * Sm::kQBytes);
                bulk_load(sbase + Sm::kQ, q_img + (((bh * n_qt + qt) * rpad + line0) * kBQ) * (long long)D,
                          kLines * Sm::kQBytes, q_full);
                const int q_rows = (N - q0 < kBQ) ? N - q0 : kBQ;  // rows of the bias tiles that exist
                const uint32_t tb_bytes = (uint32_t)q_rows * kBiasK * 2;
                for (int j = 0; j < nblk; ++j) {
                    const long long tile0 = ((bh * nblk + j) * rpad + line0) * (long long)(kBK * D);
                    const int s = j % kSt;
                    const uint32_t ph = ((j / kSt) & 1u) ^ 1u;
                    if (!mbar_wait(kb_empty(s), ph, abort_flag)) {
                        report_wait_failure(status, abort_flag, kKidCore, 1);
                        break;
                    }
                    const int nt = (2 * j + 1 < nkb32) ? 2 : 1;
                    mbar_arrive_expect_tx(kb_full(s), kLines * Sm::kKBytes + nt * tb_bytes);
                    bulk_load(sbase + Sm::kK + s * kLines * Sm::kKBytes, k_img + tile0, kLines * Sm::kKBytes, kb_full(s));
                    for (int t = 0; t < nt; ++t)
                        bulk_load(sbase + Sm::kTb + (s * 2 + t) * kTbTileBytes,
                                  tb_img + ((bh * nkb32 + 2 * j + t) * (long long)N + q0) * kBiasK, tb_bytes, kb_full(s));
                    if (!mbar_wait(v_empty(s), ph, abort_flag)) {
                        report_wait_failure(status, abort_flag, kKidCore, 11);
                        break;
                    }
                    mbar_arrive_expect_tx(v_full(s), kLines * Sm::kVBytes);
                    bulk_load(sbase + Sm::kV + s * kLines * Sm::kVBytes, v_img + tile0, kLines * Sm::kVBytes, v_full(s));
                }
            }
        } else if (warp <= kLines) {
            // ------------------------------------------------------------ one MMA-issuing warp per line
            // The whole warp walks the loop and lane 0 issues: with warp-uniform control flow and operands (the
            // shuffles tell the compiler so) descriptors and addresses live in uniform registers, instead of being
            // moved there one by one in front of every tcgen05.mma of a single-lane loop. (With elect_one() in these loops,
            // where an MMA costs the warp 40 instead of 50 - 65 cycles and a commit 4 instead of 46: N = 768 683 us against 670.)
            const int L = __shfl_sync(0xffffffffu, warp, 0) - 1;
            const uint32_t tm = __shfl_sync(0xffffffffu, tmem_base, 0);
            const uint32_t sb = __shfl_sync(0xffffffffu, sbase, 0);
            constexpr uint32_t idesc_s = idesc_bf16_f32(128, kBK);       // S: 128 x 64, K = D
            constexpr uint32_t idesc_b = idesc_bf16_f32(128, kBiasK);    // + bias: 128 x 32, K = 32
            auto qk_desc = [](uint32_t a) { return D == 32 ? smem_desc_k_sw64(a) : smem_desc_k_sw32(a); };
            const bool q_ok = mbar_wait(q_full, 0, abort_flag);
            if (!q_ok && lane == 0) report_wait_failure(status, abort_flag, kKidCore, 2);
            const uint64_t qdesc = qk_desc(sb + Sm::kQ + L * Sm::kQBytes);
            const uint64_t identdesc = smem_desc_k_sw64(sb + Sm::kIdent);
            const uint32_t t_line = tm + L * 128;
            const int nkb32 = (N + kBiasK - 1) / kBiasK;
            for (int i = 0; i < nblk && q_ok; ++i) {   // S_i, once S_{i-1} is in registers
                const int ks = i % kSt;
                if (!mbar_wait(kb_full(ks), (i / kSt) & 1u, abort_flag)) {
                    if (lane == 0) report_wait_failure(status, abort_flag, kKidCore, 3);
                    break;
                }
                if (i > 0 && !mbar_wait(s_read(L), (i - 1) & 1u, abort_flag)) {
                    if (lane == 0) report_wait_failure(status, abort_flag, kKidCore, 4);
                    break;
                }
                tc_fence_after_sync();
                const uint64_t kdesc = qk_desc(sb + Sm::kK + (ks * kLines + L) * Sm::kKBytes);
                if (lane == 0) {
#pragma unroll
                    for (int kk = 0; kk < D / 16; ++kk)
                        mma_bf16(t_line, qdesc + 2u * kk, kdesc + 2u * kk, idesc_s, kk != 0 ? 1u : 0u);
                    const int nt = (2 * i + 1 < nkb32) ? 2 : 1;
                    for (int t = 0; t < nt; ++t) {
                        const uint64_t tbdesc = smem_desc_k_sw64(sb + Sm::kTb + (ks * 2 + t) * kTbTileBytes);
                        mma_bf16(t_line + t * kBiasK, tbdesc, identdesc, idesc_b, 1u);
                        mma_bf16(t_line + t * kBiasK, tbdesc + 2u, identdesc + 2u, idesc_b, 1u);
                    }
                    mma_commit(s_full(L));
                    mma_commit(kb_empty(ks));
                }
                __syncwarp();
            }
        } else if (warp == kLines + 1) {
            // ------------------------------------------------------------ the warp that issues O += P_j V_j of all lines
            const uint32_t tm = __shfl_sync(0xffffffffu, tmem_base, 0);
            const uint32_t sb = __shfl_sync(0xffffffffu, sbase, 0);
            constexpr uint32_t idesc_o = idesc_bf16_f32(128, D);   // O: 128 x D, K = 64
            bool ok = true;
            for (int j = 0; j < nblk && ok; ++j) {
                const int vs = j % kSt;
                if (!mbar_wait(v_full(vs), (j / kSt) & 1u, abort_flag)) {
                    if (lane == 0) report_wait_failure(status, abort_flag, kKidCore, 12);
                    break;
                }
                for (int L = 0; L < kLines; ++L) {
                    if (!mbar_wait(p_ready(L), j & 1u, abort_flag)) {
                        if (lane == 0) report_wait_failure(status, abort_flag, kKidCore, 5);
                        ok = false;
                        break;
                    }
                    tc_fence_after_sync();
                    const uint32_t t_line = tm + L * 128;
                    const uint64_t vdesc = smem_desc_k_sw128(sb + Sm::kV + (vs * kLines + L) * Sm::kVBytes);
                    if (lane == 0) {
#pragma unroll
                        for (int kk = 0; kk < kBK / 16; ++kk)
                            mma_bf16_ts(t_line + kColO, t_line + kColP + kk * 8u, vdesc + 2u * kk, idesc_o,
                                        (j | kk) != 0 ? 1u : 0u);
                        mma_commit(pv_done(L));
                        mma_commit(v_empty(vs));
                    }
                    __syncwarp();
                }
            }
        }
    } else {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kCoreRegsSoftmax));
        // ---------------------------------------------------------------- softmax warpgroups
        const int L = (warp >> 2) - 1;
        const int quad = warp & 3;
        const int row = quad * 32 + lane;
        const int qpos = q0 + row;
        const bool line_valid = line0 + L < R;
        const long long bl = (long long)b * R + line_of(L);
        const uint32_t trow = tmem_base + ((uint32_t)(quad * 32) << 16) + L * 128;
        float* mbl = mbs + L * nkp;
        // Additive key mask of this line, pre-scaled for exp2: inf * (mask - 1) * log2(e), -inf beyond N. The four
        // warps of the line prepare it for themselves (eight keys per thread and pass, the loads of a pass
        // independent of each other) while the first copies and GEMMs are already under way.
        {
            const int gt = quad * 32 + lane;  // 0..127 within the line's warps
            const int line = line_of(L);
            for (int base = 0; base < nkp; base += 128 * 8) {   // warp-uniform trip count (ballot below)
                const int c0 = base + gt * 8;
                const bool active = c0 < nkp;
                float v[8];
#pragma unroll
                for (int e = 0; e < 8; ++e) {
                    const int k = c0 + e;
                    float m = 1.0f;
                    if (mask != nullptr && k < N) {
                        const long long mi = kColumns ? ((long long)b * mask_pitch + k) * mask_pitch + line
                                                      : ((long long)b * R + line) * mask_pitch + k;
                        m = __bfloat162float(mask[mi]);
                    }
                    v[e] = (k < N) ? inf * (m - 1.0f) * kLog2e : -INFINITY;
                }
                bool any = false;
#pragma unroll
                for (int e = 0; e < 8; ++e) any |= (v[e] != 0.f);
                if (active) {
                    *reinterpret_cast<float4*>(mbl + c0) = make_float4(v[0], v[1], v[2], v[3]);
                    *reinterpret_cast<float4*>(mbl + c0 + 4) = make_float4(v[4], v[5], v[6], v[7]);
                }
                // a key block of 64 = eight consecutive threads: does any of its keys carry a non-zero bias?
                const unsigned bal = __ballot_sync(0xffffffffu, any);
                if (active && (lane & 7) == 0) mbflag[L * 32 + (c0 >> 6)] = ((bal >> lane) & 0xFFu) ? 1 : 0;
            }
            group_sync(1 + L, 128);
        }
        // bit j: key block j of this line has a masked (or padding) key
        const unsigned mflags = __ballot_sync(0xffffffffu, lane < nblk && mbflag[L * 32 + lane]);
        float m_used = 0.f, lsum = 0.f;
        bool ok = true;
        // A warp whose 32 queries all lie past the end (the last query tile) only keeps the hand-offs going: what P and O
        // hold in its lanes reaches no other lane. N = 300, 16-wide heads, four samples: 267 -> 261 us.
        const bool idle = q0 + quad * 32 >= N;
        for (int j = 0; j < nblk && idle; ++j) {
            bool waited = mbar_wait(s_full(L), j & 1u, abort_flag);
            __syncwarp();
            if (waited && lane == 0) mbar_arrive(s_read(L));
            // (its arrival for step j must not count for step j - 1)
            if (waited && j > 0) waited = mbar_wait(pv_done(L), (j - 1) & 1u, abort_flag);
            if (!waited) {
                if (lane == 0) report_wait_failure(status, abort_flag, kKidCore, 14);
                break;
            }
            if (lane == 0) mbar_arrive(p_ready(L));
        }
        if (idle) ok = false;   // nothing to store
        for (int j = 0; j < nblk && ok; ++j) {
            if (!mbar_wait(s_full(L), j & 1u, abort_flag)) {
                if (lane == 0) report_wait_failure(status, abort_flag, kKidCore, 7);
                ok = false;
                break;
            }
            tc_fence_after_sync();
            uint32_t sr[64];
            tmem_ld32(trow, *reinterpret_cast<uint32_t(*)[32]>(sr));
            tmem_ld32(trow + 32, *reinterpret_cast<uint32_t(*)[32]>(sr + 32));
            tmem_ld_wait();
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive(s_read(L));
            float* sv = reinterpret_cast<float*>(sr);
            // + mask bias (blocks without a masked key skip it): (q.k + pair bias) + inf * (mask - 1); a masked
            // key ends at the same -1.44e9 in either order of the two additions, an unmasked one adds exactly 0
            if ((mflags >> j) & 1u) {
                const int k0 = j * kBK;
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                    const float4 mb = *reinterpret_cast<const float4*>(mbl + k0 + i * 4);
                    add2(sv[i * 4], sv[i * 4 + 1], mb.x, mb.y);
                    add2(sv[i * 4 + 2], sv[i * 4 + 3], mb.z, mb.w);
                }
            }
            float mx0 = max3(sv[0], sv[1], sv[2]), mx1 = max3(sv[3], sv[4], sv[5]);
            float mx2 = max3(sv[6], sv[7], sv[8]), mx3 = max3(sv[9], sv[10], sv[11]);
#pragma unroll
            for (int e = 12; e < 60; e += 8) {
                mx0 = max3(mx0, sv[e], sv[e + 1]);
                mx1 = max3(mx1, sv[e + 2], sv[e + 3]);
                mx2 = max3(mx2, sv[e + 4], sv[e + 5]);
                mx3 = max3(mx3, sv[e + 6], sv[e + 7]);
            }
            mx0 = max3(mx0, sv[60], sv[61]);
            mx1 = max3(mx1, sv[62], sv[63]);
            const float mx = max3(fmaxf(mx0, mx1), mx2, mx3);
            bool rescale = false;
            if (j == 0) {
                m_used = mx;  // finite: block 0 always holds a key < N, masked keys are -1e9-ish, not -inf
            } else {
                rescale = __any_sync(0xffffffffu, mx - m_used > kRescaleThreshold);
            }
            if (rescale) {
                float f = 1.0f;
                if (mx - m_used > kRescaleThreshold) {
                    f = ex2_approx(m_used - mx);
                    m_used = mx;
                }
                lsum *= f;
                if (!mbar_wait(pv_done(L), (j - 1) & 1u, abort_flag)) {   // every P V so far has landed in O
                    if (lane == 0) report_wait_failure(status, abort_flag, kKidCore, 8);
                    ok = false;
                    break;
                }
                tc_fence_after_sync();
#pragma unroll
                for (int part = 0; part < D / 16; ++part) {
                    uint32_t orow[16];
                    tmem_ld16(trow + kColO + part * 16, orow);
                    tmem_ld_wait();
#pragma unroll
                    for (int e = 0; e < 16; ++e) orow[e] = __float_as_uint(__uint_as_float(orow[e]) * f);
                    tmem_st16(trow + kColO + part * 16, orow);
                }
            }
            const float nm = -m_used;
            float l0 = 0.f, l1 = 0.f, l2 = 0.f, l3 = 0.f;
            uint32_t pk[16];
            auto exps = [&](int hf) {
#pragma unroll
                for (int e = 0; e < 32; e += 4) {
                    float* x = sv + hf * 32 + e;
                    add2(x[0], x[1], nm, nm);
                    add2(x[2], x[3], nm, nm);
                    const float p0 = ex2_approx(x[0]), p1 = ex2_approx(x[1]), p2 = ex2_approx(x[2]), p3 = ex2_approx(x[3]);
                    pk[e >> 1] = pack_bf16x2(p0, p1);
                    pk[(e >> 1) + 1] = pack_bf16x2(p2, p3);
                    add_bf16x2(l0, l1, pk[e >> 1]);
                    add_bf16x2(l2, l3, pk[(e >> 1) + 1]);
                }
            };
            if (j > 0) {   // P_{j-1} has been read
                if (!mbar_wait(pv_done(L), (j - 1) & 1u, abort_flag)) {
                    if (lane == 0) report_wait_failure(status, abort_flag, kKidCore, 9);
                    ok = false;
                    break;
                }
                tc_fence_after_sync();
            }
            exps(0);
            tmem_st16(trow + kColP, pk);
            exps(1);
            tmem_st16(trow + kColP + 16, pk);
            lsum += (l0 + l1) + (l2 + l3);
            tmem_st_wait();
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive(p_ready(L));
        }

        if (ok) {
            if (mbar_wait(pv_done(L), (nblk - 1) & 1u, abort_flag)) {
                tc_fence_after_sync();
                const float inv = 1.0f / lsum;
                __nv_bfloat16* dst = o_out + (bl * N + qpos) * (long long)(kH * D) + h * D;
#pragma unroll
                for (int part = 0; part < D / 16; ++part) {
                    uint32_t r[16], o[8];
                    tmem_ld16(trow + kColO + part * 16, r);
                    tmem_ld_wait();
#pragma unroll
                    for (int e = 0; e < 8; ++e)
                        o[e] = pack_bf16x2(__uint_as_float(r[2 * e]) * inv, __uint_as_float(r[2 * e + 1]) * inv);
                    if (qpos < N && line_valid) stg256_or_2x128(dst + part * 16, o, aligned32(o_out));
                }
            } else if (lane == 0) {
                report_wait_failure(status, abort_flag, kKidCore, 10);
            }
        }
    }

    tc_fence_before_sync();
    __syncthreads();
    if (warp == 0) {
        tc_fence_after_sync();
        tmem_dealloc(tmem_base, kLines * 128);
    }
}

// =====================================================================================
// triattn_out
// =====================================================================================
template <int C>
struct AOutSmem {
    static constexpr uint32_t kWBytes = C * C * 2;
    static constexpr uint32_t kWg = 0;
    static constexpr uint32_t kWo = kWBytes;
    static constexpr uint32_t kZ = 2 * kWBytes;                    // 2 groups: z tile
    static constexpr uint32_t kO = kZ + 2 * tile_bytes<C>();       // 2 groups: o tile, gated in place, then output
    static constexpr uint32_t kParams = kO + 2 * tile_bytes<C>();  // gamma, beta
    static constexpr uint32_t kXch = kParams + 1024;          // 2 groups x 512 floats: LayerNorm partial sums
    static constexpr uint32_t kBars = kXch + 4096;
    static constexpr uint32_t kTotal = kBars + 192;
    static constexpr uint32_t kDyn = kTotal + 1024;
};

// Warps: 0 producer, 1 and 2 issue the GEMMs and the stores of the two row groups, then 2 groups x 8 warps: a group alternates
// tiles with the other one; inside a group two threads share a row (TMEM lane), each with half of its channels through
// LayerNorm, gating and the output pass. Each group has its own issuer: with one for both a group's output GEMM waited 5500
// of a tile's 15300 cycles (N = 768) for the other group's next LayerNorm, and a row thread that waited for its TMA store to
// leave the buffer held its group up for 2000; the issuer has that time, between a tile's last GEMM and the next LayerNorm.
constexpr int kAOutThreads = 32 * (3 + 2 * 8);

// o <- o * sigmoid(gate) for the eight channels at addr
__device__ __forceinline__ void gate_chunk(uint32_t addr, const uint32_t* gate) {
    const uint4 ov = lds128(addr);
    const uint32_t w[4] = {ov.x, ov.y, ov.z, ov.w};
    uint32_t o[4];
#pragma unroll
    for (int j = 0; j < 4; ++j)
        o[j] = pack_bf16x2(bf16lo(w[j]) * sigmoid_fast(__uint_as_float(gate[2 * j])),
                           bf16hi(w[j]) * sigmoid_fast(__uint_as_float(gate[2 * j + 1])));
    sts128(addr, make_uint4(o[0], o[1], o[2], o[3]));
}
// the update of eight channels, with the residual z (pairs), to addr
__device__ __forceinline__ void add_chunk(uint32_t addr, const uint32_t* upd, const uint32_t* z, int add_residual) {
    uint32_t o[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        float v0 = __uint_as_float(upd[2 * j]), v1 = __uint_as_float(upd[2 * j + 1]);
        if (add_residual) {
            v0 = add_lo(z[j], v0);
            v1 = add_hi(z[j], v1);
        }
        o[j] = pack_bf16x2(v0, v1);
    }
    sts128(addr, make_uint4(o[0], o[1], o[2], o[3]));
}

// kSolo: one tile per CTA (a tensor of no more tiles than SMs). Both groups work on it: each takes the statistics of its half rows,
// and half of a thread's channels from there on. N = 37, in a block: 6.3 -> 5.4 us.
template <int C, bool kTransposed, bool kSolo>
__global__ void __launch_bounds__(kAOutThreads, 1)
triattn_out_kernel(const __grid_constant__ CUtensorMap tmZ, const __grid_constant__ CUtensorMap tmO,
                   const __grid_constant__ CUtensorMap tmOut, const __grid_constant__ CUtensorMap tmWg,
                   const __grid_constant__ CUtensorMap tmWo, const __nv_bfloat16* __restrict__ ln_w,
                   const __nv_bfloat16* __restrict__ ln_b, int B, int R, int N, int add_residual, int* status) {
    using Sm = AOutSmem<C>;
    extern __shared__ uint8_t smem_raw[];
    const uint32_t sbase = (smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t* gbase = smem_raw + (sbase - smem_u32(smem_raw));
    float* prm = reinterpret_cast<float*>(gbase + Sm::kParams);
    const uint32_t bars = sbase + Sm::kBars;
    const uint32_t w_full = bars;
    // The z buffer is free once the gate GEMM has read it (the result goes over the o buffer), so the next
    // z tile is fetched while this one is still being gated and projected; the o buffer is free once the output
    // store has read it, and its next tile lands during the next LayerNorm + gate GEMM.
    auto z_full = [&](int g) { return bars + 8u * (1 + g); };
    auto o_empty = [&](int g) { return bars + 8u * (3 + g); };
    auto o_full = [&](int g) { return bars + 8u * (13 + g); };
    auto z_empty = [&](int g) { return bars + 8u * (15 + g); };
    auto a1_ready = [&](int g) { return bars + 8u * (5 + g); };
    auto g_full = [&](int g) { return bars + 8u * (7 + g); };
    auto a2_ready = [&](int g) { return bars + 8u * (9 + g); };
    auto d_full = [&](int g) { return bars + 8u * (11 + g); };
    auto out_ready = [&](int g) { return bars + 8u * (17 + g); };   // the group's result lies in the o buffer
    volatile uint32_t* tmem_ptr = reinterpret_cast<volatile uint32_t*>(gbase + Sm::kBars + 160);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(gbase + Sm::kBars + 164);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int tiles_per_line = (N + kRows - 1) / kRows;
    const long long num_tiles = (long long)B * R * tiles_per_line;
    const long long my_tiles = tiles_of_block(num_tiles);

    if (threadIdx.x == 0) {
        mbar_init(w_full, 1);
        for (int g = 0; g < 2; ++g) {
            mbar_init(z_full(g), 1);
            mbar_init(o_full(g), 1);
            mbar_init(z_empty(g), 1);
            mbar_init(o_empty(g), 1);
            mbar_init(a1_ready(g), kSolo ? 16 : 8);
            mbar_init(g_full(g), 1);
            mbar_init(a2_ready(g), kSolo ? 16 : 8);
            mbar_init(d_full(g), 1);
            mbar_init(out_ready(g), kSolo ? 16 : 8);
        }
        *abort_flag = 0;
        mbar_fence_init();
        prefetch_tmap(&tmZ);
        prefetch_tmap(&tmO);
        prefetch_tmap(&tmOut);
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
    if (warp >= 3) grid_wait();

    if (warp == 0) {
        if (elect_one()) {
            mbar_arrive_expect_tx(w_full, 2 * Sm::kWBytes);
            for (int kb = 0; kb < C / 64; ++kb) {
                tma_load_2d(sbase + Sm::kWg + kb * C * 128, &tmWg, w_full, kb * 64, 0);
                tma_load_2d(sbase + Sm::kWo + kb * C * 128, &tmWo, w_full, kb * 64, 0);
            }
            grid_wait();
            TileWalk tc(blockIdx.x, gridDim.x, R, tiles_per_line);
            for (long long lt = 0; lt < my_tiles; ++lt, tc.next()) {
                const int g = (int)(lt & 1);
                const uint32_t use = (uint32_t)(lt >> 1);
                if (!mbar_wait(z_empty(g), (use & 1u) ^ 1u, abort_flag)) {
                    report_wait_failure(status, abort_flag, kKidOut, 1);
                    break;
                }
                mbar_arrive_expect_tx(z_full(g), tile_bytes<C>());
                load_z_tile<C, kTransposed>(sbase + Sm::kZ + g * tile_bytes<C>(), &tmZ, z_full(g), tc, R);
                if (!mbar_wait(o_empty(g), (use & 1u) ^ 1u, abort_flag)) {
                    report_wait_failure(status, abort_flag, kKidOut, 8);
                    break;
                }
                mbar_arrive_expect_tx(o_full(g), tile_bytes<C>());
                const uint32_t odst = sbase + Sm::kO + g * tile_bytes<C>();
                for (int kb = 0; kb < C / 64; ++kb)
                    tma_load_3d(odst + kb * kKBlockBytes, &tmO, o_full(g), kb * 64, tc.tile * kRows, tc.b * R + tc.line);
            }
        }
    } else if (warp <= 2) {
        // ---------------------------------------------------------------- MMA issuer of row group g
        if (elect_one()) {
            const int g = warp - 1;
            constexpr uint32_t idesc = idesc_bf16_f32(128, C);
            bool ok = mbar_wait(w_full, 0, abort_flag);
            if (!ok) report_wait_failure(status, abort_flag, kKidOut, 2);
            grid_wait();   // (the stores)
            const uint32_t otile = sbase + Sm::kO + g * tile_bytes<C>();
            TileWalk tc(blockIdx.x + g * gridDim.x, 2 * gridDim.x, R, tiles_per_line);
            for (long long lt = g; lt < my_tiles && ok; lt += 2, tc.next()) {
                const uint32_t par = (uint32_t)(lt >> 1) & 1u;
                if (!mbar_wait(a1_ready(g), par, abort_flag)) {
                    report_wait_failure(status, abort_flag, kKidOut, 3);
                    break;
                }
                tc_fence_after_sync();
                mma_rows<C>(tmem_base + g * 256, sbase + Sm::kZ + g * tile_bytes<C>(), sbase + Sm::kWg, C * 128, idesc,
                            false);
                mma_commit(g_full(g));
                mma_commit(z_empty(g));
                if (!mbar_wait(a2_ready(g), par, abort_flag)) {
                    report_wait_failure(status, abort_flag, kKidOut, 4);
                    break;
                }
                tc_fence_after_sync();
                mma_rows<C>(tmem_base + g * 256 + 128, sbase + Sm::kO + g * tile_bytes<C>(), sbase + Sm::kWo, C * 128,
                            idesc, false);
                mma_commit(d_full(g));
                if (!mbar_wait(out_ready(g), par, abort_flag)) {
                    report_wait_failure(status, abort_flag, kKidOut, 10);
                    break;
                }
                for (int kb = 0; kb < C / 64; ++kb) {
                    if (kTransposed) {
                        asm volatile(
                            "cp.async.bulk.tensor.4d.global.shared::cta.tile.bulk_group [%0, {%2, %3, %4, %5}], [%1];" ::
                                "l"(reinterpret_cast<uint64_t>(&tmOut)),
                            "r"(otile + kb * kKBlockBytes), "r"(kb * 64), "r"(tc.line), "r"(tc.tile * kRows), "r"(tc.b)
                            : "memory");
                    } else {
                        tma_store_3d(&tmOut, otile + kb * kKBlockBytes, kb * 64, tc.tile * kRows, tc.b * R + tc.line);
                    }
                }
                tma_store_commit();
                tma_store_wait_read<0>();
                mbar_arrive(o_empty(g));
            }
            tma_store_wait_all<0>();
        }
    } else {
        const int g = (warp - 3) >> 3;
        const int quad = warp & 3;
        const int half = ((warp - 3) >> 2) & 1;   // half of the row's channels
        const int row = quad * 32 + lane;
        float* xch = reinterpret_cast<float*>(gbase + Sm::kXch) + g * 512;
        const uint32_t ztile = sbase + Sm::kZ + g * tile_bytes<C>();
        const uint32_t otile = sbase + Sm::kO + g * tile_bytes<C>();
        const uint32_t taddr = tmem_base + ((uint32_t)(quad * 32) << 16) + g * 256 + half * (C / 2);
        if constexpr (kSolo) {
            const uint32_t z0 = sbase + Sm::kZ, o0 = sbase + Sm::kO;
            const int chunk = half * (C / 16) + g * (C / 32);   // this thread's C / 4 channels
            const uint32_t t0 = tmem_base + ((uint32_t)(quad * 32) << 16) + chunk * 8;
            bool ok = true;
            auto wait = [&](uint32_t bar, int site) {
                if (ok && !(ok = mbar_wait(bar, 0, abort_flag)) && lane == 0) report_wait_failure(status, abort_flag, kKidOut, site);
            };
            wait(z_full(0), 5);
            uint32_t zq[C / 8];
            {
                uint32_t zraw[C / 4];
                load_half_row<C>(z0, row, half, zraw);
                float mean, rstd;
                half_row_stats_xwarp<C>(zraw, row, half, xch, 1, 512, mean, rstd);   // (its barrier: everyone has read the row)
#pragma unroll
                for (int i = 0; i < C / 8; ++i) zq[i] = g ? zraw[C / 8 + i] : zraw[i];
                store_normalized_chunks<C / 32>(z0, row, chunk, zq, mean, rstd, prm, prm + 128);
            }
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) mbar_arrive(a1_ready(0));
            wait(g_full(0), 6);
            wait(o_full(0), 9);
            tc_fence_after_sync();
#pragma unroll
            for (int cb = 0; cb < C / 64 && ok; ++cb) {
                uint32_t gate[16];
                tmem_ld16(t0 + cb * 16, gate);
                tmem_ld_wait();
#pragma unroll
                for (int ch = 0; ch < 2; ++ch) gate_chunk(chunk_addr(o0, row, chunk + cb * 2 + ch), gate + ch * 8);
            }
            tc_fence_before_sync();
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) mbar_arrive(a2_ready(0));
            wait(d_full(0), 7);
            tc_fence_after_sync();
#pragma unroll
            for (int cb = 0; cb < C / 64 && ok; ++cb) {
                uint32_t upd[16];
                tmem_ld16(t0 + 128 + cb * 16, upd);
                tmem_ld_wait();
#pragma unroll
                for (int ch = 0; ch < 2; ++ch)
                    add_chunk(chunk_addr(o0, row, chunk + cb * 2 + ch), upd + ch * 8, zq + cb * 8 + ch * 4, add_residual);
            }
            tc_fence_before_sync();
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) mbar_arrive(out_ready(0));
        }
        for (long long lt = kSolo ? my_tiles : g; lt < my_tiles; lt += 2) {
            const uint32_t use = (uint32_t)(lt >> 1);
            if (!mbar_wait(z_full(g), use & 1u, abort_flag)) {
                if (lane == 0) report_wait_failure(status, abort_flag, kKidOut, 5);
                break;
            }
            uint32_t zraw[C / 4];
            load_half_row<C>(ztile, row, half, zraw);
            {
                float mean, rstd;
                half_row_stats_xwarp<C>(zraw, row, half, xch, 1 + g, 256, mean, rstd);
                store_normalized_half_row<C>(ztile, row, half, zraw, mean, rstd, prm, prm + 128);
            }
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) mbar_arrive(a1_ready(g));
            // ---- gate: o <- o * sigmoid(LN(z) W_g^T), in place in the o tile
            if (!mbar_wait(g_full(g), use & 1u, abort_flag)) {
                if (lane == 0) report_wait_failure(status, abort_flag, kKidOut, 6);
                break;
            }
            tc_fence_after_sync();
            if (!mbar_wait(o_full(g), use & 1u, abort_flag)) {
                if (lane == 0) report_wait_failure(status, abort_flag, kKidOut, 9);
                break;
            }
#pragma unroll
            for (int cb = 0; cb < C / 32; ++cb) {
                uint32_t gate[16];
                tmem_ld16(taddr + cb * 16, gate);
                tmem_ld_wait();
#pragma unroll
                for (int ch = 0; ch < 2; ++ch) gate_chunk(chunk_addr(otile, row, half * (C / 16) + cb * 2 + ch), gate + ch * 8);
            }
            tc_fence_before_sync();
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) mbar_arrive(a2_ready(g));
            // ---- output projection + residual, written over the o tile (its GEMM is done) and TMA-stored
            if (!mbar_wait(d_full(g), use & 1u, abort_flag)) {
                if (lane == 0) report_wait_failure(status, abort_flag, kKidOut, 7);
                break;
            }
            tc_fence_after_sync();
#pragma unroll
            for (int cb = 0; cb < C / 32; ++cb) {
                uint32_t upd[16];
                tmem_ld16(taddr + 128 + cb * 16, upd);
                tmem_ld_wait();
#pragma unroll
                for (int ch = 0; ch < 2; ++ch)
                    add_chunk(chunk_addr(otile, row, half * (C / 16) + cb * 2 + ch), upd + ch * 8, zraw + cb * 8 + ch * 4, add_residual);
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

int weight_tmap(CUtensorMap* m, const void* w, int C) {
    uint64_t dims[2] = {(uint64_t)C, (uint64_t)C};
    uint64_t str[1] = {(uint64_t)C * 2};
    uint32_t box[2] = {64, (uint32_t)C};
    return make_tmap_bf16(m, w, 2, dims, str, box, 1);
}

int z_tmap(CUtensorMap* m, const void* z, int B, int R, int N, int C, bool transposed) {
    const uint64_t row = (uint64_t)C * 2;
    if (!transposed) {
        uint64_t dims[3] = {(uint64_t)C, (uint64_t)N, (uint64_t)B * R};
        uint64_t str[2] = {row, (uint64_t)N * row};
        uint32_t box[3] = {64, 128, 1};
        return make_tmap_bf16(m, z, 3, dims, str, box, 1);
    }
    uint64_t dims[4] = {(uint64_t)C, (uint64_t)N, (uint64_t)N, (uint64_t)B};
    uint64_t str[3] = {row, (uint64_t)N * row, (uint64_t)N * N * row};
    uint32_t box[4] = {64, 1, 128, 1};
    return make_tmap_bf16(m, z, 4, dims, str, box, 1);
}

// Shared memory of which an SM (228 KB, 1 KB of them the system's per block) has per_sm shares and no more
constexpr uint32_t core_share(int per_sm) { return 228 * 1024 / (uint32_t)(per_sm + 1); }

template <int C, bool kT>
int set_attrs() {
    static PerDeviceOnce configured;
    if (!configured.done()) {
        OF3_CUDA_CHECK(cudaFuncSetAttribute(triattn_proj_kernel<C, kT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                            ProjSmem<C>::kDyn));
        for (auto* core : {triattn_core_kernel<C / kH, false, 1>, triattn_core_kernel<C / kH, true, 1>,
                           triattn_core_kernel<C / kH, false, 2>, triattn_core_kernel<C / kH, true, 2>}) {
            cudaFuncAttributes fa;   // a block launched with fewer registers would wait for the split for good
            OF3_CUDA_CHECK(cudaFuncGetAttributes(&fa, core));
            OF3_REQUIRE(fa.numRegs == kCoreRegsLaunch, OF3_ERR_DRIVER, "triattn_core is built with %d registers, not %d",
                        fa.numRegs, kCoreRegsLaunch);
            OF3_CUDA_CHECK(cudaFuncSetAttribute(core, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                max(CoreSmem<C / kH, 2>::dyn_bytes(kMaxKeys / kBK), core_share(1))));
        }
        for (auto* out : {triattn_out_kernel<C, kT, false>, triattn_out_kernel<C, kT, true>})
            OF3_CUDA_CHECK(cudaFuncSetAttribute(out, cudaFuncAttributeMaxDynamicSharedMemorySize, AOutSmem<C>::kDyn));
        configured.mark();
    }
    return OF3_OK;
}

template <int C, bool kT>
int project_impl(const __nv_bfloat16* z, __nv_bfloat16* q, __nv_bfloat16* k, __nv_bfloat16* vt,
                 __nv_bfloat16* tb, const __nv_bfloat16* mask, __nv_bfloat16* mask_t, int B, int R, int N, int row0,
                 const of3_triattn_params* p, cudaStream_t st) {
    int rc;
    CUtensorMap tmZ, tmW[3], tmWb;
    if ((rc = z_tmap(&tmZ, z, B, R, N, C, kT))) return rc;
    const void* w3[3] = {p->w_q, p->w_k, p->w_v};
    for (int i = 0; i < 3; ++i)
        if ((rc = weight_tmap(&tmW[i], w3[i], C))) return rc;
    {   // linear_z.weight [4, C]: box of 16 rows, the 12 rows past the end are zero-filled
        OF3_REQUIRE(((uintptr_t)p->w_bias & 15) == 0, OF3_ERR_ALIGN, "triattn: linear_z.weight must be 16-byte aligned");
        uint64_t dims[2] = {(uint64_t)C, (uint64_t)kH};
        uint64_t str[1] = {(uint64_t)C * 2};
        uint32_t box[2] = {64, 16};
        if ((rc = make_tmap_bf16(&tmWb, p->w_bias, 2, dims, str, box, 1))) return rc;
    }
    if ((rc = set_attrs<C, kT>())) return rc;
    const long long tiles = (long long)B * R * ceil_div(N, kRows);
    const int slots = sm_count() * (C == 128 ? 1 : 2);
    const int grid = (int)(tiles < slots ? tiles : slots);
    typedef const __nv_bfloat16* P;
    LaunchScope scope(kKidProj, st);
    OF3_CUDA_CHECK(launch_chained(triattn_proj_kernel<C, kT>, grid, kProjThreads, ProjSmem<C>::kDyn, st, tmZ, tmW[0],
                                  tmW[1], tmW[2], tmWb, (P)p->ln_w, (P)p->ln_b, q, k, vt, tb, mask, mask_t, B,
                                  R, N, triattn_mask_pitch(N), row0, device_status_ptr()));
    return OF3_OK;
}

template <int C, bool kT>
int finish_impl(const __nv_bfloat16* z, const MaskView& mask, __nv_bfloat16* out, const __nv_bfloat16* q,
                const __nv_bfloat16* k, const __nv_bfloat16* vt, const __nv_bfloat16* tb, __nv_bfloat16* o, int B,
                int R, int N, float inf, int add_residual, const of3_triattn_params* p, cudaStream_t st) {
    int rc;
    CUtensorMap tmZ, tmOut, tmO, tmWg, tmWo;
    // The output kernel takes a view that is not transposed as one line: its tiles end with the tensor, not with every line (N = 37:
    // 11 tiles instead of 37, 300: 704 instead of 900)
    const bool flat = !kT && (long long)B * R * N < (1LL << 31);
    const int oB = flat ? 1 : B, oR = flat ? 1 : R, oN = flat ? B * R * N : N;
    if ((rc = z_tmap(&tmZ, z, oB, oR, oN, C, kT))) return rc;
    if ((rc = z_tmap(&tmOut, out, oB, oR, oN, C, kT))) return rc;
    if ((rc = z_tmap(&tmO, o, oB, oR, oN, C, false))) return rc;  // o is [line][pos][C] in view order
    if ((rc = weight_tmap(&tmWg, p->w_g, C))) return rc;
    if ((rc = weight_tmap(&tmWo, p->w_o, C))) return rc;
    if ((rc = set_attrs<C, kT>())) return rc;
    int* status = device_status_ptr();
    const long long lines = (long long)B * R * kH * ceil_div(N, kBQ), pairs = (long long)B * ceil_div(R, 2) * kH * ceil_div(N, kBQ);
    OF3_REQUIRE(pairs < (1LL << 31), OF3_ERR_SHAPE, "triattn: too many attention tiles");
    // One line per block where the chip takes all lines at once, and room for as many blocks per SM as spread them evenly: blocks start
    // while the projections drain, and gathered on the SMs that these had left first; the launch ends with its fullest SM. Trunk of
    // four blocks, us, two lines per block / also with a share of the SM where there are no more blocks than SMs / one line: N = 37
    // (one line per SM) 403.8 / 400.0 / 375.5, 50 409 / 395 / 392, 64 (two) 403 / 391.0 / 387.4, 80 (three) - / 430.4 / 420.1, 111 - /
    // 451.5 / 449.7; pair stack of 37 343.6 / 316.9 with one line, template of 60 134.3 / 127.9 / 126.8.
    // Past three lines per SM two per block: N = 112 447 us against 465 with one, 128 457 / 477, 148 711 / 728, 4 x 60 template 172 / 178.
    const bool one = lines <= kCorePerSm<1> * (long long)sm_count();
    const long long ctas = one ? lines : pairs;
    const int nblk = ceil_div(N, kBK);
    uint32_t smem = one ? CoreSmem<C / kH, 1>::dyn_bytes(nblk) : CoreSmem<C / kH, 2>::dyn_bytes(nblk);
    if (one) smem = max(smem, core_share((int)((lines + sm_count() - 1) / sm_count())));
    {
        LaunchScope scope(kKidCore, st);
        auto* core = mask.columns ? (one ? triattn_core_kernel<C / kH, true, 1> : triattn_core_kernel<C / kH, true, 2>)
                                  : (one ? triattn_core_kernel<C / kH, false, 1> : triattn_core_kernel<C / kH, false, 2>);
        OF3_CUDA_CHECK(launch_chained(core, (unsigned)ctas, one ? kCoreThreads<1> : kCoreThreads<2>, smem, st, q, k, vt, tb, mask.p,
                                      mask.pitch, o, R, N, inf, status));
    }
    const long long tiles = (long long)oB * oR * ceil_div(oN, kRows);
    const int grid = (int)(tiles < sm_count() ? tiles : sm_count());
    typedef const __nv_bfloat16* P;
    LaunchScope scope(kKidOut, st);
    OF3_CUDA_CHECK(launch_chained(tiles <= grid ? triattn_out_kernel<C, kT, true> : triattn_out_kernel<C, kT, false>, grid,
                                  kAOutThreads, AOutSmem<C>::kDyn, st, tmZ, tmO, tmOut, tmWg, tmWo, (P)p->ln_w, (P)p->ln_b, oB, oR,
                                  oN, add_residual, status));
    return OF3_OK;
}

}  // namespace

bool triattn_supported(int c_z, int H, int d, int N) {
    return H == kH && ((c_z == 128 && d == 32) || (c_z == 64 && d == 16)) && N <= kMaxKeys;
}

// Elements of each of the q / k / v image buffers for B samples of R lines and N positions: 4 heads x
// (query tiles of 128) x (R rounded up to 4 lines) x 128 x D; the k / v images need no more than that.
size_t triattn_image_elems(int B, int R, int N, int C) {
    return (size_t)B * ceil_div(N, kBQ) * align_up(R, kLinePad) * kBQ * C;
}

// Elements (bf16) of the pair-bias image of B samples with R query rows and N keys: [B*4][key blocks of 32][R][32].
size_t triattn_bias_elems(int B, int R, int N) {
    return (size_t)B * kH * ceil_div(N, kBiasK) * R * kBiasK;
}

int triattn_mask_pitch(int N) { return (int)align_up(N, kBK); }

// q, k, v operand images and this shard's rows of the pair-bias image tb[(b*H + h)][key block][line][32]
// from R lines of N positions; row0 = index of the shard's first line among all N query rows (0 for a whole
// tensor). transposed: whole square tensors only; where mask_t is given, their mask [B, N, N] goes there with the view's lines
// as rows of triattn_mask_pitch elements.
int triattn_project(const __nv_bfloat16* z, __nv_bfloat16* q, __nv_bfloat16* k, __nv_bfloat16* vt,
                    __nv_bfloat16* tb, int B, int R, int N, int row0, bool transposed,
                    const of3_triattn_params* p, cudaStream_t st, int C, const __nv_bfloat16* mask,
                    __nv_bfloat16* mask_t) {
    OF3_REQUIRE(((uintptr_t)z & 15) == 0, OF3_ERR_ALIGN, "triattn: z must be 16-byte aligned");
    OF3_REQUIRE((((uintptr_t)q | (uintptr_t)k | (uintptr_t)vt) & 15) == 0, OF3_ERR_ALIGN,
                "triattn: q / k / v images must be 16-byte aligned");
    OF3_REQUIRE(!transposed || R == N, OF3_ERR_SHAPE, "triattn: transposed view needs the whole tensor");
    OF3_REQUIRE(mask_t == nullptr || mask != nullptr, OF3_ERR_ARG, "triattn: mask rows without a mask");
    if (C == 128)
        return transposed ? project_impl<128, true>(z, q, k, vt, tb, mask, mask_t, B, R, N, row0, p, st)
                          : project_impl<128, false>(z, q, k, vt, tb, mask, mask_t, B, R, N, row0, p, st);
    return transposed ? project_impl<64, true>(z, q, k, vt, tb, mask, mask_t, B, R, N, row0, p, st)
                      : project_impl<64, false>(z, q, k, vt, tb, mask, mask_t, B, R, N, row0, p, st);
}

// attention over the R lines with the pair-bias image of all N query rows (tb [(b*H + h)][key block][N][32]),
// gate, output projection, residual.
int triattn_finish(const __nv_bfloat16* z, const MaskView& mask, __nv_bfloat16* out,
                   const __nv_bfloat16* q, const __nv_bfloat16* k, const __nv_bfloat16* vt,
                   const __nv_bfloat16* tb, __nv_bfloat16* o, int B, int R, int N, float inf,
                   bool transposed, int add_residual, const of3_triattn_params* p, cudaStream_t st, int C) {
    OF3_REQUIRE(((uintptr_t)tb & 15) == 0, OF3_ERR_ALIGN, "triattn: the pair-bias image must be 16-byte aligned");
    OF3_REQUIRE((((uintptr_t)o | (uintptr_t)q | (uintptr_t)k | (uintptr_t)vt) & 15) == 0, OF3_ERR_ALIGN,
                "triattn: the attention's output and operand images must be 16-byte aligned");
    OF3_REQUIRE(((uintptr_t)z & 15) == 0 && ((uintptr_t)out & 15) == 0, OF3_ERR_ALIGN,
                "triattn: z/out must be 16-byte aligned");
    OF3_REQUIRE(N <= kMaxKeys, OF3_ERR_SHAPE, "triattn: N %d above the %d keys one CTA keeps a mask row for", N,
                kMaxKeys);
    OF3_REQUIRE(!transposed || R == N, OF3_ERR_SHAPE, "triattn: transposed view needs the whole tensor");
    OF3_REQUIRE(!mask.columns || transposed, OF3_ERR_ARG, "triattn: mask by columns of a view that is not transposed");
    if (C == 128)
        return transposed ? finish_impl<128, true>(z, mask, out, q, k, vt, tb, o, B, R, N, inf, add_residual, p, st)
                          : finish_impl<128, false>(z, mask, out, q, k, vt, tb, o, B, R, N, inf, add_residual, p, st);
    return transposed ? finish_impl<64, true>(z, mask, out, q, k, vt, tb, o, B, R, N, inf, add_residual, p, st)
                      : finish_impl<64, false>(z, mask, out, q, k, vt, tb, o, B, R, N, inf, add_residual, p, st);
}

int triattn(const __nv_bfloat16* z, const __nv_bfloat16* mask, __nv_bfloat16* out, int B, int N, int C,
            float inf, int flags, const of3_triattn_params* p, Arena& ws, cudaStream_t st) {
    const size_t plane = (size_t)B * N * N * C * sizeof(__nv_bfloat16);
    const size_t img = triattn_image_elems(B, N, N, C) * sizeof(__nv_bfloat16);
    __nv_bfloat16* q = (__nv_bfloat16*)ws.take(img);
    __nv_bfloat16* k = (__nv_bfloat16*)ws.take(img);
    __nv_bfloat16* vt = (__nv_bfloat16*)ws.take(img);
    __nv_bfloat16* o = (__nv_bfloat16*)ws.take(plane);
    __nv_bfloat16* tb = (__nv_bfloat16*)ws.take(triattn_bias_elems(B, N, N) * sizeof(__nv_bfloat16));
    const bool tr = (flags & OF3_FLAG_TRANSPOSED) != 0;
    if (!ws.base && !tr) return OF3_OK;
    OF3_REQUIRE(!ws.base || ws.ok(), OF3_ERR_WORKSPACE, "triattn: workspace too small (%zu needed)", ws.off);
    // Mask rows of the ending node, 0.1 % of the workspace: where they do not fit (a workspace of the starting node's size),
    // the attention reads the mask in place (N = 768: 85 us more).
    const int pitch = triattn_mask_pitch(N);
    __nv_bfloat16* mask_t = (__nv_bfloat16*)ws.take((size_t)B * N * pitch * sizeof(__nv_bfloat16));
    if (!ws.base) return OF3_OK;
    if (!tr || mask == nullptr || !ws.ok()) mask_t = nullptr;
    int rc = triattn_project(z, q, k, vt, tb, B, N, N, 0, tr, p, st, C, mask, mask_t);
    if (rc) return rc;
    const MaskView view = mask_t != nullptr ? MaskView{mask_t, pitch, false} : MaskView{mask, N, tr && mask != nullptr};
    return triattn_finish(z, view, out, q, k, vt, tb, o, B, N, N, inf, tr, (flags & OF3_FLAG_ADD_RESIDUAL) ? 1 : 0, p, st, C);
}

}  // namespace fast
}  // namespace of3
