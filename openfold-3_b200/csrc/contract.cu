// Batched NT contraction on tcgen05:  X[b][i][j] = sum_k A[b][i][k] * B[b][j][k]
// (bf16 operands, fp32 accumulation in TMEM, bf16 result).
//
// This is the N^3*c part of the triangle multiplicative update: one "batch" entry per
// (sample, hidden channel); the prologue kernel writes the gated projections a, b
// channel-major with the contracted index innermost, so the outgoing and the incoming
// update are the same K-major x K-major GEMM
// (reference: openfold3/core/model/layers/triangular_multiplicative_update.py:71-97).
//
// Persistent, warp-specialised CTA (one per SM):
//   warp 0     TMA producer     A tile 128x64, B tile BNx64 per k-block, 128B swizzle
//   warp 1     MMA issuer       tcgen05.mma 128 x BN x 16, accumulators double-buffered in TMEM
//   warps 2-5  epilogue         tcgen05.ld -> bf16 -> global (overlaps the next tile's main loop); 32 bytes per store
//                               where the pitch allows it (16-byte halves of a sector reach L2 one by one: N = 384 39 -> 29 us,
//                               N = 768 114 -> 107)
#include "modules.cuh"
#include "rowtile.cuh"
#include "runtime.cuh"

namespace of3 {
namespace {

using namespace umma;

constexpr int kBM = 128;
constexpr int kBK = 64;
constexpr int kKernelIdContract = 1;

template <int BN>
struct ContractCfg {
    static constexpr int kStages = (BN == 256) ? 4 : 6;
    static constexpr int kABytes = kBM * kBK * 2;
    static constexpr int kBBytes = BN * kBK * 2;
    static constexpr int kStageBytes = kABytes + kBBytes;
    static constexpr int kTmemCols = 2 * BN;
    static constexpr int kSmemBytes = kStages * kStageBytes + 1024 /*align slack*/ + 256 /*barriers*/;
};

template <int BN>
__global__ void __launch_bounds__(192, 1)
contract_nt_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                   __nv_bfloat16* __restrict__ out, int M, int N, int K, int batch,
                   long long out_batch_stride, int ldo, int rows_per_block, long long row_block_stride,
                   int a_shared, int chan_shift, long long out_sample_stride, int wide_cols, int* status) {
    using Cfg = ContractCfg<BN>;
    constexpr int S = Cfg::kStages;
    extern __shared__ uint8_t smem_raw[];
    const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    const uint32_t bar_base = smem_base + S * Cfg::kStageBytes;
    // barrier block: full[S], empty[S], tmem_full[2], tmem_empty[2] (8 B each), then tmem ptr, abort
    auto full_bar = [&](int s) { return bar_base + 8u * s; };
    auto empty_bar = [&](int s) { return bar_base + 8u * (S + s); };
    auto tfull_bar = [&](int a) { return bar_base + 8u * (2 * S + a); };
    auto tempty_bar = [&](int a) { return bar_base + 8u * (2 * S + 2 + a); };
    uint8_t* gen_base = smem_raw + (smem_base - smem_u32(smem_raw));
    volatile uint32_t* tmem_ptr_smem =
        reinterpret_cast<volatile uint32_t*>(gen_base + S * Cfg::kStageBytes + 8 * (2 * S + 4));
    volatile int* abort_flag =
        reinterpret_cast<volatile int*>(gen_base + S * Cfg::kStageBytes + 8 * (2 * S + 4) + 8);

    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;

    const int num_mt = (M + kBM - 1) / kBM;
    const int num_nt = (N + BN - 1) / BN;
    const int num_kb = (K + kBK - 1) / kBK;
    const long long num_tiles = (long long)batch * num_mt * num_nt;

    if (threadIdx.x == 0) {
        for (int s = 0; s < S; ++s) {
            mbar_init(full_bar(s), 1);
            mbar_init(empty_bar(s), 1);
        }
        for (int a = 0; a < 2; ++a) {
            mbar_init(tfull_bar(a), 1);
            mbar_init(tempty_bar(a), 4);
        }
        *abort_flag = 0;
        mbar_fence_init();
        prefetch_tmap(&tmA);
        prefetch_tmap(&tmB);
    }
    if (warp == 1) {
        tmem_alloc(smem_u32((const void*)tmem_ptr_smem), Cfg::kTmemCols);
        tmem_relinquish();
    }
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem_base = *tmem_ptr_smem;
    grid_trigger();
    grid_wait();

    if (warp == 0) {
        // ------------------------------------------------ TMA producer
        if (elect_one()) {
            uint32_t it = 0;
            bool ok = true;
            rowtile::TileWalk tw(blockIdx.x, gridDim.x, num_mt, num_nt);
            for (long long t = blockIdx.x; t < num_tiles && ok; t += gridDim.x, tw.next()) {
                // maps: {k, row, 1, batch entry, 1}, or {k, row of its block, block, channel, sample}
                const int a0 = tw.line * kBM, b0 = tw.tile * BN;
                const int b = tw.b & (int)((1u << chan_shift) - 1u), smp = tw.b >> chan_shift;
                const bool blocked = chan_shift != 31;
                const int a_row = blocked ? 0 : a0, a_blk = blocked ? a0 >> kLineBlockShift : 0;
                const int b_row = blocked ? 0 : b0, b_blk = blocked ? b0 >> kLineBlockShift : 0;
                for (int kb = 0; kb < num_kb; ++kb, ++it) {
                    const int s = it % S;
                    const uint32_t ph = (it / S) & 1u;
                    if (!mbar_wait(empty_bar(s), ph ^ 1u, abort_flag)) {
                        report_wait_failure(status, abort_flag, kKernelIdContract, 1);
                        ok = false;
                        break;
                    }
                    mbar_arrive_expect_tx(full_bar(s), Cfg::kStageBytes);
                    const uint32_t sa = smem_base + s * Cfg::kStageBytes;
                    tma_load_5d(sa, &tmA, full_bar(s), kb * kBK, a_row, a_blk, a_shared ? 0 : b, smp);
                    tma_load_5d(sa + Cfg::kABytes, &tmB, full_bar(s), kb * kBK, b_row, b_blk, b, smp);
                }
            }
        }
    } else if (warp == 1) {
        // ------------------------------------------------ MMA issuer
        if (elect_one()) {
            constexpr uint32_t idesc = idesc_bf16_f32(kBM, BN);
            uint32_t it = 0, tcount = 0;
            bool ok = true;
            for (long long t = blockIdx.x; t < num_tiles && ok; t += gridDim.x, ++tcount) {
                const uint32_t acc = tcount & 1u;
                const uint32_t acc_ph = (tcount >> 1) & 1u;
                if (!mbar_wait(tempty_bar(acc), acc_ph ^ 1u, abort_flag)) {
                    report_wait_failure(status, abort_flag, kKernelIdContract, 2);
                    ok = false;
                    break;
                }
                tc_fence_after_sync();
                const uint32_t d_tmem = tmem_base + acc * BN;
                for (int kb = 0; kb < num_kb; ++kb, ++it) {
                    const int s = it % S;
                    const uint32_t ph = (it / S) & 1u;
                    if (!mbar_wait(full_bar(s), ph, abort_flag)) {
                        report_wait_failure(status, abort_flag, kKernelIdContract, 3);
                        ok = false;
                        break;
                    }
                    tc_fence_after_sync();
                    const uint32_t sa = smem_base + s * Cfg::kStageBytes;
                    const uint64_t adesc = smem_desc_k_sw128(sa);
                    const uint64_t bdesc = smem_desc_k_sw128(sa + Cfg::kABytes);
#pragma unroll
                    for (int k4 = 0; k4 < kBK / 16; ++k4) {
                        // +32 B per 16-element K step == +2 in the 16-byte-unit address field
                        mma_bf16(d_tmem, adesc + 2u * k4, bdesc + 2u * k4, idesc,
                                 (kb | k4) != 0 ? 1u : 0u);
                    }
                    mma_commit(empty_bar(s));
                }
                if (ok) mma_commit(tfull_bar(acc));
            }
        }
    } else {
        // ------------------------------------------------ epilogue (warps 2..5)
        const int quad = warp & 3;  // TMEM lane quarter this warp may read
        uint32_t tcount = 0;
        bool ok = true;
        rowtile::TileWalk tw(blockIdx.x, gridDim.x, num_mt, num_nt);
        for (long long t = blockIdx.x; t < num_tiles && ok; t += gridDim.x, ++tcount, tw.next()) {
            const int nt = tw.tile, mt = tw.line, b = tw.b;
            const uint32_t acc = tcount & 1u;
            const uint32_t acc_ph = (tcount >> 1) & 1u;
            if (!mbar_wait(tfull_bar(acc), acc_ph, abort_flag)) {
                if (lane == 0) report_wait_failure(status, abort_flag, kKernelIdContract, 4);
                ok = false;
                break;
            }
            tc_fence_after_sync();
            const int row = mt * kBM + quad * 32 + lane;
            // rows_per_block > 0: output rows are grouped in blocks of that many rows and block q starts
            // at q * row_block_stride (the layout a row-sharding all-to-all sends without a repack, and the blocked one)
            long long roff = (long long)row * ldo;
            if (rows_per_block > 0) {
                const int q = (uint32_t)row / (uint32_t)rows_per_block;
                roff = (long long)q * row_block_stride + (long long)(row - q * rows_per_block) * ldo;
            }
            __nv_bfloat16* orow = out + (long long)(b >> chan_shift) * out_sample_stride +
                                  (long long)(b & (int)((1u << chan_shift) - 1u)) * out_batch_stride + roff;
            const uint32_t taddr = tmem_base + ((uint32_t)(quad * 32) << 16) + acc * BN;
#pragma unroll 1
            for (int c = 0; c < BN / 32; ++c) {
                uint32_t r[32];
                tmem_ld32(taddr + c * 32, r);
                tmem_ld_wait();
                const int col0 = nt * BN + c * 32;
                if (row < M) {
#pragma unroll
                    for (int g = 0; g < 2; ++g) {   // 16 columns: a sector of 32 bytes, whole where the pitch allows it
                        const int col = col0 + g * 16;
                        uint32_t o[8];
#pragma unroll
                        for (int e = 0; e < 8; ++e)
                            o[e] = pack_bf16x2(__uint_as_float(r[g * 16 + 2 * e]), __uint_as_float(r[g * 16 + 2 * e + 1]));
                        if (col < N) {
                            if (col + 16 <= wide_cols) {
                                stg256(orow + col, o);
                            } else {
                                *reinterpret_cast<uint4*>(orow + col) = make_uint4(o[0], o[1], o[2], o[3]);
                                if (col + 8 < N) *reinterpret_cast<uint4*>(orow + col + 8) = make_uint4(o[4], o[5], o[6], o[7]);
                            }
                        }
                    }
                }
            }
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive(tempty_bar(acc));
        }
    }

    // ---------------------------------------------------- teardown
    tc_fence_before_sync();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after_sync();
        tmem_dealloc(tmem_base, Cfg::kTmemCols);
    }
}

// rows of `lines` lines in the blocked layout of contract_blocked_bf16, `box_rows` of them per copy
int blocked_tmap(CUtensorMap* m, const __nv_bfloat16* x, int samples, int channels, int lines, int K, int ld, int box_rows) {
    const uint64_t row = (uint64_t)ld * 2, chan = row << kLineBlockShift, blk = chan * channels;
    const uint64_t blocks = (uint64_t)ceil_div(lines, 1 << kLineBlockShift);
    uint64_t dims[5] = {(uint64_t)K, 1ull << kLineBlockShift, blocks, (uint64_t)channels, (uint64_t)samples};
    uint64_t str[4] = {row, blk, chan, blk * blocks};
    uint32_t box[5] = {kBK, 1u << kLineBlockShift, (uint32_t)box_rows >> kLineBlockShift, 1, 1};
    return make_tmap_bf16(m, x, 5, dims, str, box, true);
}
// entries of `rows` rows, `entry` elements apart
int plane_tmap(CUtensorMap* m, const __nv_bfloat16* x, int entries, int rows, int K, int ld, long long entry, int box_rows) {
    uint64_t dims[5] = {(uint64_t)K, (uint64_t)rows, 1, (uint64_t)entries, 1};
    uint64_t str[4] = {(uint64_t)ld * 2, (uint64_t)entry * 2, (uint64_t)entry * 2, (uint64_t)entry * 2};
    uint32_t box[5] = {kBK, (uint32_t)box_rows, 1, 1, 1};
    return make_tmap_bf16(m, x, 5, dims, str, box, true);
}

struct ContractOut {
    __nv_bfloat16* out;
    int ld, rows_per_block, chan_shift;   // chan_shift 31: the batch entries are not split into samples
    long long batch_stride, row_block_stride, sample_stride;
};

template <int BN>
int launch_contract(const CUtensorMap& tmA, const CUtensorMap& tmB, const ContractOut& o, int batch, int M, int N, int K,
                    bool a_shared, cudaStream_t stream, int account_as) {
    using Cfg = ContractCfg<BN>;
    constexpr int kAttrKey = BN == 256 ? 0 : (BN == 128 ? 1 : 2);  // per-device function attributes
    if (!device_configured(kAttrKey)) {
        OF3_CUDA_CHECK(cudaFuncSetAttribute(contract_nt_kernel<BN>,
                                            cudaFuncAttributeMaxDynamicSharedMemorySize,
                                            Cfg::kSmemBytes));
        device_mark_configured(kAttrKey);
    }
    const long long tiles = (long long)batch * ceil_div(M, kBM) * ceil_div(N, BN);
    const int grid = (int)(tiles < sm_count() ? tiles : sm_count());
    int* status = device_status_ptr();
    LaunchScope scope(account_as, stream);  // launch accounting: the triangle einsum or a plain linear layer
    // 16 columns per store, up to the last column that is the output's: a general output ends at N rounded up to 8 (what lies
    // behind it in the pitch is the caller's), the blocked one has its whole pitch to itself
    const bool wide = o.ld % 16 == 0 && o.batch_stride % 16 == 0 && o.row_block_stride % 16 == 0 &&
                      o.sample_stride % 16 == 0 && ((uintptr_t)o.out & 31) == 0;
    const int wide_cols = !wide ? 0 : (o.chan_shift == 31 ? (int)align_up(N, 8) : o.ld);
    OF3_CUDA_CHECK(launch_chained(contract_nt_kernel<BN>, grid, 192, Cfg::kSmemBytes, stream, tmA, tmB, o.out, M, N, K, batch,
                                  o.batch_stride, o.ld, o.rows_per_block, o.row_block_stride, a_shared ? 1 : 0, o.chan_shift,
                                  o.sample_stride, wide_cols, status));
    return OF3_OK;
}

}  // namespace

int contract_nt_bf16(const __nv_bfloat16* a, const __nv_bfloat16* b, __nv_bfloat16* out, int batch,
                     int M, int N, int K, int lda, int ldb, int ldo, long long a_bs, long long b_bs,
                     long long o_bs, cudaStream_t stream, int rows_per_block, long long row_block_stride,
                     int account_as) {
    OF3_REQUIRE(a && b && out, OF3_ERR_ARG, "contract: null pointer");
    OF3_REQUIRE(batch > 0 && M > 0 && N > 0 && K > 0, OF3_ERR_ARG, "contract: non-positive size");
    OF3_REQUIRE(lda % 8 == 0 && ldb % 8 == 0 && ldo % 8 == 0 && a_bs % 8 == 0 && b_bs % 8 == 0 &&
                    o_bs % 8 == 0,
                OF3_ERR_ALIGN, "contract: pitches must be multiples of 8 elements");
    OF3_REQUIRE(ldo >= (int)align_up(N, 8), OF3_ERR_ALIGN, "contract: ldo < round_up(N, 8)");
    OF3_REQUIRE(((uintptr_t)out & 15) == 0, OF3_ERR_ALIGN, "contract: out not 16-byte aligned");
    OF3_REQUIRE(rows_per_block >= 0 && row_block_stride % 8 == 0, OF3_ERR_ALIGN,
                "contract: row block stride must be a multiple of 8 elements");
    const ContractOut o = {out, ldo, rows_per_block, 31, o_bs, row_block_stride, 0};
    const int bn = N > 128 ? 256 : 128;
    CUtensorMap tmA, tmB;
    int rc;
    // a_bs == 0: every batch entry multiplies the same A (several linear layers on one input)
    if ((rc = plane_tmap(&tmA, a, a_bs == 0 ? 1 : batch, M, K, lda, a_bs == 0 ? (long long)lda * M : a_bs, kBM))) return rc;
    if ((rc = plane_tmap(&tmB, b, batch, N, K, ldb, b_bs, bn))) return rc;
    return bn == 256 ? launch_contract<256>(tmA, tmB, o, batch, M, N, K, a_bs == 0, stream, account_as)
                     : launch_contract<128>(tmA, tmB, o, batch, M, N, K, a_bs == 0, stream, account_as);
}

// X = A B^T per sample and channel, all three as [sample][line / 8][channel][8][ld] with N lines of N positions.
int contract_blocked_bf16(const __nv_bfloat16* a, const __nv_bfloat16* b, __nv_bfloat16* out, int samples, int channels,
                          int N, int ld, cudaStream_t stream) {
    OF3_REQUIRE(a && b && out && samples > 0 && N > 0, OF3_ERR_ARG, "contract: bad argument");
    OF3_REQUIRE((channels & (channels - 1)) == 0, OF3_ERR_SHAPE, "contract: channels must be a power of two");
    OF3_REQUIRE(ld % 8 == 0 && ld >= (int)align_up(N, 8) && ((uintptr_t)out & 15) == 0, OF3_ERR_ALIGN,
                "contract: pitch or alignment");
    int shift = 0;
    while ((1 << shift) < channels) ++shift;
    const long long chan = (long long)ld << kLineBlockShift, blk = chan * channels;
    const ContractOut o = {out, ld, 1 << kLineBlockShift, shift, chan, blk, ceil_div(N, 1 << kLineBlockShift) * blk};
    const int bn = N > 128 ? 256 : 128;
    CUtensorMap tmA, tmB;
    int rc;
    if ((rc = blocked_tmap(&tmA, a, samples, channels, N, N, ld, kBM))) return rc;
    if ((rc = blocked_tmap(&tmB, b, samples, channels, N, N, ld, bn))) return rc;
    return bn == 256 ? launch_contract<256>(tmA, tmB, o, samples * channels, N, N, N, false, stream, 1)
                     : launch_contract<128>(tmA, tmB, o, samples * channels, N, N, N, false, stream, 1);
}

}  // namespace of3

// X[b][i][j] = sum_k A[b][i][k] * B[b][j][k]; element pitches lda/ldb/ldo, batch strides in elements.
extern "C" int of3_contract_nt_bf16(const void* a, const void* b, void* out, int batch, int M, int N,
                                    int K, int lda, int ldb, int ldo, long long a_batch_stride,
                                    long long b_batch_stride, long long out_batch_stride,
                                    void* stream) {
    of3::CallScope call;
    return of3::contract_nt_bf16((const __nv_bfloat16*)a, (const __nv_bfloat16*)b,
                                 (__nv_bfloat16*)out, batch, M, N, K, lda, ldb, ldo, a_batch_stride,
                                 b_batch_stride, out_batch_stride, (cudaStream_t)stream, 0, 0, 1);
}
