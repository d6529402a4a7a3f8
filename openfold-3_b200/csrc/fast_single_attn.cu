// Attention of the single track and of the diffusion token stack on the tensor pipe (bf16, 16 heads of 24 or 48):
// the streaming core of the triangle attention (csrc/fast_triattn.cu) with one (pair tensor, head, 128 queries) and
// one or two samples per CTA.
//
//   operand images  q / k / v projections as pre-swizzled operand tiles (linear.cu): q with its bias added and scaled
//                   by log2(e)/sqrt(d), K-dim padded with zeros to 32 (d = 24) or 64 (d = 48); k likewise per key
//                   block of 32; v transposed [d rows][32 keys]; keys >= N are zeros
//   single_bias     pair bias fp32 [zh][nq][N] -> bf16 tiles [zh][key block][nq][32], pre-scaled by log2(e), each
//                   64-byte row in the 64-byte swizzle of a K-major A operand (callers that project the bias
//                   themselves get these tiles straight from csrc/fast_pairbias.cu and skip this kernel)
//   single_core     a CTA takes one or two samples; per CTA and 32-key step: S = Q K^T + bias I^T (tcgen05, TMEM), online softmax by one thread per
//                   query row (exp2, lazy rescaling), P (bf16) back into TMEM over S as the A operand of
//                   O += P [V; 1] (the row of ones makes the tensor pipe accumulate the row sum l); epilogue
//                   O / l * sigmoid(gate) -> og [rows, H*d]
// Queries may be a window of nq rows of the sample (row-sharded callers); keys and values are always all N rows.
// Reference: openfold3/core/model/layers/attention_pair_bias.py:123-227,
//            openfold3/core/model/primitives/attention.py:94-135, 270-310.
#include "fast_single.cuh"
#include "modules.cuh"
#include "rowtile.cuh"
#include "runtime.cuh"
#include "single_attn.cuh"

namespace of3 {
namespace fast {
namespace {

using namespace umma;
using namespace rowtile;
typedef __nv_bfloat16 bf16;

constexpr int kKidSingleAttn = 8;    // bias conversion: accounted with the single track's small kernels
constexpr int kKidSingleCore = 11;   // the attention core
constexpr float kLog2e = 1.4426950408889634f;
constexpr int kBQ = kSingleBQ;   // queries per CTA and line
constexpr int kBK = kSingleBK;   // keys per step
// Lines (samples) per CTA: two share the pair-bias tiles; one where that leaves fewer lines per SM (core_impl)
template <int kLines>
constexpr int kThreads = 32 * (1 + kLines + 4 * kLines);  // producer, one MMA warp per line, softmax warps
template <int kLines>
constexpr int kCtasPerSm = kLines == 1 ? 3 : 2;
constexpr float kRescaleThreshold = 8.0f;
constexpr int kMaxKeysSingle = 8192;  // one flag byte per key block, 256 of them
constexpr int kMaxSmem = 227 * 1024;  // shared memory of a CTA

template <int D, int kLines>
struct Cfg {
    static constexpr int kKD = SingleImage<D>::kKD;
    static constexpr int kKSteps = (D + 15) / 16;        // K = 16 steps that hold data
    static constexpr int kDV = SingleImage<D>::kDV;
    static constexpr int kStages = (D <= 32) ? 4 : 3;    // ring of K + bias tiles
    static constexpr int kVStages = (D <= 32) ? 4 : 2;   // ring of V tiles (two CTAs of 16 x 48 heads must fit an SM)
    static constexpr uint32_t kQBytes = kBQ * kKD * 2;   // 8 or 16 KB
    static constexpr uint32_t kKBytes = kBK * kKD * 2;   // 2 or 4 KB
    static constexpr uint32_t kVBytes = kDV * kBK * 2;   // 2 or 3 KB: the tile a bulk copy brings
    static constexpr int kON = kDV + 16;                 // N of the P V GEMM: channels, a row of ones (-> row sum), padding
    static constexpr uint32_t kVSlot = kON * kBK * 2;    // 3 or 4 KB: rows kDV .. kDV + 15 are written once per CTA
    static constexpr uint32_t kTbBytes = kBQ * kBK * 2;  // 8 KB
    // shared memory (offsets from a 1024-byte boundary)
    static constexpr uint32_t kQ = 0;
    static constexpr uint32_t kK = kQ + kLines * kQBytes;
    static constexpr uint32_t kTb = kK + kStages * kLines * kKBytes;
    static constexpr uint32_t kV = kTb + kStages * kTbBytes;
    static constexpr uint32_t kIdent = kV + kVStages * kLines * kVSlot;
    static constexpr uint32_t kBars = kIdent + 2048;
    static constexpr uint32_t kFlags = kBars + 320;       // lines x 256 key-block flags (bytes)
    static constexpr uint32_t kMb = kFlags + kLines * 256;
    static uint32_t dyn_bytes(int nkp) { return kMb + kLines * nkp * 4 + 1024; }
    // TMEM columns of a line (128): S slots [0,32) [32,64), each taking the step's P (16 columns of bf16 pairs)
    // in place once S has been read out; O [64, 64 + kON): kDV channels, then the sum of the row's P
    static constexpr uint32_t kColO = 64;
};

// pair bias fp32 [zh][nq][N] -> bf16 tiles [zh][key block][nq][32], times log2(e); block = (query row, zh)
__global__ void __launch_bounds__(256)
single_bias_kernel(const float* __restrict__ pair_bias, bf16* __restrict__ tb_img, int N, int nq, int nkb) {
    const int qrow = blockIdx.x;
    const long long zh = blockIdx.y;
    const float* src = pair_bias + (zh * nq + qrow) * (long long)N;
    for (int key = threadIdx.x; key < nkb * kBK; key += 256) {
        const float val = key < N ? src[key] * kLog2e : 0.f;
        const int kb = key >> 5, kk = key & 31;
        const int c = (kk >> 3) ^ ((qrow >> 1) & 3);
        tb_img[((zh * nkb + kb) * (long long)nq + qrow) * kBK + c * 8 + (kk & 7)] = __float2bfloat16_rn(val);
    }
}

// V consecutive channels of the caller's row: 32 bytes where V = 16 and the address allows it
template <int V>
__device__ __forceinline__ void load_row(const bf16* p, uint32_t (&o)[V / 2]) {
    if constexpr (V == 16) {
        if (aligned32(p)) ldg256(p, o);
        else ld_row16(p, o);
    } else {
        const uint4 v = *reinterpret_cast<const uint4*>(p);
        o[0] = v.x; o[1] = v.y; o[2] = v.z; o[3] = v.w;
    }
}
template <int V>
__device__ __forceinline__ void store_row(bf16* p, const uint32_t (&o)[V / 2]) {
    if constexpr (V == 16) stg256_or_2x128(p, o, aligned32(p));
    else *reinterpret_cast<uint4*>(p) = make_uint4(o[0], o[1], o[2], o[3]);
}

// ---------------------------------------------------------------- single_core
// One CTA = (pair tensor z, head, 128 queries) for ONE sample ("line"), three CTAs per SM, or for TWO that share the pair bias
// (the last of an odd number of samples: one, and nothing is done for the other), two CTAs per SM; core_impl chooses.
// Per line and 32-key step j:
//   MMA warp      S_j = Q K_j^T + Tb_j I^T into TMEM slot j % 2 (the bias tile is a second A operand against a
//                 32 x 32 identity: the tensor pipe adds it, exactly, in fp32)
//   softmax warps thread = query row = TMEM lane: S -> registers [+ key-mask bias], row maximum, P = exp2(S - m),
//                 P rounded to bf16 into the first 16 columns of the slot S_j came from
//   MMA warp      O += P_j V_j with P read from TMEM as the A operand; when that GEMM is done the slot takes S_{j+2}
// The running maximum m used for scaling is only raised when a row maximum exceeds it by more than 8 (2^8 head
// room in P): then the thread rescales its O row in TMEM and its running sum. Numerator and denominator always
// share one scale, so the result is exact.
// What bounds it: one wave of blocks, each a chain of steps, and at both ends what no other block covers. Gate values fetched
// behind the last P V, 16 bytes at a time, and divisions in the sigmoids made the epilogue 11000 cycles of some 60000 (5 x 768
// tokens, 24 layers: 3630 -> 3456 us). Measured and not kept: 64 keys per step as in the triangle attention (with 48 channels
// P then has one block of columns and two hand-offs per step: 3505 us), three V slots (one block per SM at N = 768: 3773).
template <int D, int kLines>
__global__ void __launch_bounds__(kThreads<kLines>, kCtasPerSm<kLines>)
single_core_kernel(const bf16* __restrict__ q_img, const bf16* __restrict__ k_img, const bf16* __restrict__ v_img,
                   const bf16* __restrict__ tb_img, const bf16* __restrict__ mask, const bf16* __restrict__ gate,
                   bf16* __restrict__ out, int N, int nq, int H, int rpb, int pairs, float inf, int* status) {
    using C = Cfg<D, kLines>;
    constexpr int KD = C::kKD, DV = C::kDV, kSt = C::kStages, kVSt = C::kVStages;
    extern __shared__ uint8_t smem_raw[];
    const uint32_t sbase = (smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t* gbase = smem_raw + (sbase - smem_u32(smem_raw));
    float* mbs = reinterpret_cast<float*>(gbase + C::kMb);
    volatile uint8_t* mbflag = gbase + C::kFlags;
    const uint32_t bars = sbase + C::kBars;
    const uint32_t q_full = bars;
    auto kb_full = [&](int s) { return bars + 8u * (1 + s); };
    auto kb_empty = [&](int s) { return bars + 8u * (1 + kSt + s); };
    constexpr int kB1 = 1 + 2 * kSt;
    auto v_full = [&](int s) { return bars + 8u * (kB1 + s); };
    auto v_empty = [&](int s) { return bars + 8u * (kB1 + kVSt + s); };
    constexpr int kB2 = kB1 + 2 * kVSt;
    auto s_full = [&](int L, int s) { return bars + 8u * (kB2 + L * 2 + s); };
    auto p_ready = [&](int L, int s) { return bars + 8u * (kB2 + 2 * kLines + L * 2 + s); };
    auto pv_done = [&](int L, int s) { return bars + 8u * (kB2 + 4 * kLines + L * 2 + s); };
    constexpr int kNumBars = kB2 + 6 * kLines;
    static_assert(8 * kNumBars + 16 <= 320, "barrier block");
    volatile uint32_t* tmem_ptr = reinterpret_cast<volatile uint32_t*>(gbase + C::kBars + 8 * kNumBars);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(gbase + C::kBars + 8 * kNumBars + 8);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int n_qt = (nq + kBQ - 1) / kBQ;
    // CTAs of kLines samples first, `pairs` of them; then those of the last sample of an odd number
    const bool odd = kLines == 2 && (int)blockIdx.x >= pairs;
    const int b = odd ? (int)blockIdx.x - pairs : (int)blockIdx.x;
    const int gpz = odd ? 1 : rpb / kLines;   // CTAs of the kind per (z, head, query tile)
    const int grp = odd ? rpb / kLines : b % gpz;
    const int qt = (b / gpz) % n_qt;
    const int h = (b / (gpz * n_qt)) % H;
    const int z = b / (gpz * n_qt * H);
    const int q0 = qt * kBQ;
    const int nblk = (N + kBK - 1) / kBK;
    const int nkp = nblk * kBK;
    const int lines = odd ? 1 : kLines;   // samples of this group
    auto sample_of = [&](int L) { return (long long)z * rpb + grp * kLines + L; };

    if (threadIdx.x == 0) {
        mbar_init(q_full, 1);
        for (int s = 0; s < kSt; ++s) {
            mbar_init(kb_full(s), 1);
            mbar_init(kb_empty(s), lines);       // each line's commit after the S that read the stage
        }
        for (int s = 0; s < kVSt; ++s) {
            mbar_init(v_full(s), 1);
            mbar_init(v_empty(s), lines);        // each line's commit after the P V that read the stage
        }
        for (int L = 0; L < kLines; ++L) {
            for (int s = 0; s < 2; ++s) {
                mbar_init(s_full(L, s), 1);
                mbar_init(p_ready(L, s), 4);
                mbar_init(pv_done(L, s), 1);
            }
        }
        *abort_flag = 0;
        mbar_fence_init();
    }
    // 32 x 32 identity, bf16, K-major with the 64-byte swizzle
    for (int idx = threadIdx.x; idx < 32 * 16; idx += blockDim.x) {
        const int n = idx >> 4, w = idx & 15;
        const int k = w * 2;
        uint32_t v = 0;
        if (k == n) v = 0x00003F80u;
        if (k + 1 == n) v = 0x3F800000u;
        const int chunk = (k >> 3) ^ ((n >> 1) & 3);
        *reinterpret_cast<uint32_t*>(gbase + C::kIdent + n * 64 + chunk * 16 + (w & 3) * 4) = v;
    }
    // rows kDV .. kDV + 15 of every V slot: a row of ones (column kDV of O then accumulates the row sum of P on the
    // tensor pipe, rounded exactly like the numerator) and 15 rows of zeros; the bulk copies write rows 0 .. kDV - 1
    for (int idx = threadIdx.x; idx < kVSt * kLines * 64; idx += blockDim.x) {
        const int slot = idx >> 6, w = idx & 63;   // 64 uint4 = 1 KB per slot
        const uint32_t v = (w < 4) ? 0x3F803F80u : 0u;
        *reinterpret_cast<uint4*>(gbase + C::kV + slot * C::kVSlot + C::kVBytes + w * 16) = make_uint4(v, v, v, v);
    }
    fence_proxy_async_smem();
    if (warp == 1) {
        tmem_alloc(smem_u32((const void*)tmem_ptr), kLines * 128);
        tmem_relinquish();
    }
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem_base = *tmem_ptr;
    grid_trigger();
    grid_wait();

    if (warp == 0) {
        if (elect_one()) {
            const long long zh = (long long)z * H + h;
            mbar_arrive_expect_tx(q_full, lines * C::kQBytes);
            for (int L = 0; L < lines; ++L)
                bulk_load(sbase + C::kQ + L * C::kQBytes,
                          q_img + (((sample_of(L) * H + h) * n_qt + qt) * kBQ) * (long long)KD, C::kQBytes, q_full);
            const int q_rows = (nq - q0 < kBQ) ? nq - q0 : kBQ;   // rows of the bias tile that exist
            const uint32_t tb_bytes = (uint32_t)q_rows * kBK * 2;
            auto load_kb = [&](int j) {
                const int s = j % kSt;
                if (!mbar_wait(kb_empty(s), ((j / kSt) & 1u) ^ 1u, abort_flag)) {
                    report_wait_failure(status, abort_flag, kKidSingleCore, 1);
                    return false;
                }
                mbar_arrive_expect_tx(kb_full(s), lines * C::kKBytes + tb_bytes);
                for (int L = 0; L < lines; ++L)
                    bulk_load(sbase + C::kK + (s * kLines + L) * C::kKBytes,
                              k_img + (((sample_of(L) * H + h) * nblk + j) * kBK) * (long long)KD, C::kKBytes,
                              kb_full(s));
                bulk_load(sbase + C::kTb + s * C::kTbBytes, tb_img + ((zh * nblk + j) * (long long)nq + q0) * kBK,
                          tb_bytes, kb_full(s));
                return true;
            };
            auto load_v = [&](int j) {
                const int s = j % kVSt;
                if (!mbar_wait(v_empty(s), ((j / kVSt) & 1u) ^ 1u, abort_flag)) {
                    report_wait_failure(status, abort_flag, kKidSingleCore, 11);
                    return false;
                }
                mbar_arrive_expect_tx(v_full(s), lines * C::kVBytes);
                for (int L = 0; L < lines; ++L)
                    bulk_load(sbase + C::kV + (s * kLines + L) * C::kVSlot,
                              v_img + (((sample_of(L) * H + h) * nblk + j) * (long long)DV) * kBK, C::kVBytes,
                              v_full(s));
                return true;
            };
            // K and bias run two blocks ahead of V: a V slot waits for P V, and what is behind it in this loop for as long
            // (5 samples of 768 tokens, 24 layers: 3456 -> 3420 us)
            for (int j = 0; j < nblk + 2; ++j) {
                if (j < nblk && !load_kb(j)) break;
                if (j >= 2 && !load_v(j - 2)) break;
            }
        }
    } else if (warp <= kLines) {
        // ---------------------------------------------------------------- one MMA-issuing warp per line
        // The whole warp walks the loop and an elected lane issues: with warp-uniform control flow and operands
        // descriptors and addresses live in uniform registers.
        const int L = __shfl_sync(0xffffffffu, warp, 0) - 1;
        const uint32_t tm = __shfl_sync(0xffffffffu, tmem_base, 0);
        const uint32_t sb = __shfl_sync(0xffffffffu, sbase, 0);
        constexpr uint32_t idesc_s = idesc_bf16_f32(128, kBK);
        constexpr uint32_t idesc_o = idesc_bf16_f32(128, C::kON);
        auto kdesc_of = [](uint32_t a) { return KD == 32 ? smem_desc_k_sw64(a) : smem_desc_k_sw128(a); };
        bool ok = L < lines;
        if (ok) ok = mbar_wait(q_full, 0, abort_flag);
        if (!ok && L < lines && lane == 0) report_wait_failure(status, abort_flag, kKidSingleCore, 2);
        const uint64_t qdesc = kdesc_of(sb + C::kQ + L * C::kQBytes);
        const uint64_t identdesc = smem_desc_k_sw64(sb + C::kIdent);
        const uint32_t t_line = tm + L * 128;
        // S_i = Q K_i^T + Tb_i into slot i % 2, free once P_{i-2} V_{i-2} (which read P out of it) is done
        auto issue_s = [&](int i) -> bool {
            const int s = i & 1;
            const int ks = i % kSt;
            if (i >= 2 && !mbar_wait(pv_done(L, s), ((i - 2) >> 1) & 1u, abort_flag)) {
                if (lane == 0) report_wait_failure(status, abort_flag, kKidSingleCore, 4);
                return false;
            }
            if (!mbar_wait(kb_full(ks), (i / kSt) & 1u, abort_flag)) {
                if (lane == 0) report_wait_failure(status, abort_flag, kKidSingleCore, 3);
                return false;
            }
            tc_fence_after_sync();
            const uint64_t kdesc = kdesc_of(sb + C::kK + (ks * kLines + L) * C::kKBytes);
            const uint64_t tbdesc = smem_desc_k_sw64(sb + C::kTb + ks * C::kTbBytes);
            const uint32_t d = t_line + s * kBK;
            if (elect_one()) {
#pragma unroll
                for (int kk = 0; kk < C::kKSteps; ++kk)
                    mma_bf16(d, qdesc + 2u * kk, kdesc + 2u * kk, idesc_s, kk ? 1u : 0u);
                mma_bf16(d, tbdesc, identdesc, idesc_s, 1u);            // + pair bias
                mma_bf16(d, tbdesc + 2u, identdesc + 2u, idesc_s, 1u);
                mma_commit(s_full(L, s));
                mma_commit(kb_empty(ks));
            }
            __syncwarp();
            return true;
        };
        ok = ok && issue_s(0);
        if (ok && nblk > 1) ok = issue_s(1);
        for (int j = 0; j < nblk && ok; ++j) {
            const int vs = j % kVSt;
            if (!mbar_wait(v_full(vs), (j / kVSt) & 1u, abort_flag)) {
                if (lane == 0) report_wait_failure(status, abort_flag, kKidSingleCore, 12);
                break;
            }
            if (!mbar_wait(p_ready(L, j & 1), (j >> 1) & 1u, abort_flag)) {
                if (lane == 0) report_wait_failure(status, abort_flag, kKidSingleCore, 5);
                break;
            }
            tc_fence_after_sync();
            const uint64_t vdesc = smem_desc_k_sw64(sb + C::kV + (vs * kLines + L) * C::kVSlot);
            if (elect_one()) {
                const uint32_t a_p = t_line + (j & 1) * kBK;
                mma_bf16_ts(t_line + C::kColO, a_p, vdesc, idesc_o, j != 0 ? 1u : 0u);
                mma_bf16_ts(t_line + C::kColO, a_p + 8u, vdesc + 2u, idesc_o, 1u);
                mma_commit(pv_done(L, j & 1));
                mma_commit(v_empty(vs));
            }
            __syncwarp();
            if (j + 2 < nblk && !issue_s(j + 2)) break;
        }
    } else {
        // ---------------------------------------------------------------- softmax warpgroups
        const int L = (warp - 1 - kLines) >> 2;
        const int quad = warp & 3;
        const int row = quad * 32 + lane;
        const int qpos = q0 + row;
        bool ok = L < lines;
        const long long bb = sample_of(L);
        const uint32_t trow = tmem_base + ((uint32_t)(quad * 32) << 16) + L * 128;
        float* mbl = mbs + L * nkp;
        // Additive key mask of this sample, pre-scaled for exp2: inf * (mask - 1) * log2(e), -inf beyond N; one flag
        // per key block tells whether the block has any non-zero entry.
        if (ok) {
            const int gt = (warp - 1 - kLines - 4 * L) * 32 + lane;  // 0..127 within the line's warps
            for (int base = 0; base < nkp; base += 128 * 8) {        // warp-uniform trip count (ballot below)
                const int c0 = base + gt * 8;
                const bool active = c0 < nkp;
                float v[8];
#pragma unroll
                for (int e = 0; e < 8; ++e) {
                    const int k = c0 + e;
                    float m = 1.0f;
                    if (mask != nullptr && k < N) m = __bfloat162float(mask[bb * N + k]);
                    v[e] = (k < N) ? inf * (m - 1.0f) * kLog2e : -INFINITY;
                }
                bool any = false;
#pragma unroll
                for (int e = 0; e < 8; ++e) any |= (v[e] != 0.f);
                if (active) {
                    *reinterpret_cast<float4*>(mbl + c0) = make_float4(v[0], v[1], v[2], v[3]);
                    *reinterpret_cast<float4*>(mbl + c0 + 4) = make_float4(v[4], v[5], v[6], v[7]);
                }
                const unsigned bal = __ballot_sync(0xffffffffu, any);
                if (active && (lane & 3) == 0) mbflag[L * 256 + (c0 >> 5)] = ((bal >> lane) & 0xFu) ? 1 : 0;
            }
            group_sync(1 + L, 128);
        }
        float m_used = 0.f;
        for (int j = 0; j < nblk && ok; ++j) {
            const int s = j & 1;
            if (!mbar_wait(s_full(L, s), (j >> 1) & 1u, abort_flag)) {
                if (lane == 0) report_wait_failure(status, abort_flag, kKidSingleCore, 7);
                ok = false;
                break;
            }
            tc_fence_after_sync();
            uint32_t sr[32];
            tmem_ld32(trow + s * kBK, sr);
            tmem_ld_wait();
            float sv[kBK];
#pragma unroll
            for (int e = 0; e < 32; ++e) sv[e] = __uint_as_float(sr[e]);
            if (mbflag[L * 256 + j]) {
                const int k0 = j * kBK;
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const float4 mb = *reinterpret_cast<const float4*>(mbl + k0 + i * 4);
                    sv[i * 4] += mb.x;
                    sv[i * 4 + 1] += mb.y;
                    sv[i * 4 + 2] += mb.z;
                    sv[i * 4 + 3] += mb.w;
                }
            }
            float mx0 = max3(sv[0], sv[1], sv[2]), mx1 = max3(sv[3], sv[4], sv[5]);
#pragma unroll
            for (int e = 6; e < 30; e += 4) {
                mx0 = max3(mx0, sv[e], sv[e + 1]);
                mx1 = max3(mx1, sv[e + 2], sv[e + 3]);
            }
            const float mx = max3(mx0, mx1, fmaxf(sv[30], sv[31]));
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
                // every P V issued so far must have landed in O before it is rescaled
                if (!mbar_wait(pv_done(L, (j - 1) & 1), ((j - 1) >> 1) & 1u, abort_flag)) {
                    if (lane == 0) report_wait_failure(status, abort_flag, kKidSingleCore, 8);
                    ok = false;
                    break;
                }
                tc_fence_after_sync();
                uint32_t orow[32];
                tmem_ld32(trow + C::kColO, orow);
                tmem_ld_wait();
#pragma unroll
                for (int e = 0; e < 32; ++e) orow[e] = __float_as_uint(__uint_as_float(orow[e]) * f);
                tmem_st32(trow + C::kColO, orow);
                if (DV > 32) {
                    uint32_t o2[16];
                    tmem_ld16(trow + C::kColO + 32, o2);
                    tmem_ld_wait();
#pragma unroll
                    for (int e = 0; e < 16; ++e) o2[e] = __float_as_uint(__uint_as_float(o2[e]) * f);
                    tmem_st16(trow + C::kColO + 32, o2);
                }
                const uint32_t lsum = tmem_ld1(trow + C::kColO + DV);   // the row sum rides in column kDV of O
                tmem_ld_wait();
                tmem_st1(trow + C::kColO + DV, __float_as_uint(__uint_as_float(lsum) * f));
                tmem_st_wait();
            }
            uint32_t pk[16];
            const float nm = -m_used;
#pragma unroll
            for (int e = 0; e < 32; e += 2) {
                add2(sv[e], sv[e + 1], nm, nm);
                pk[e >> 1] = pack_bf16x2(ex2_approx(sv[e]), ex2_approx(sv[e + 1]));
            }
            // P_j goes where S_j was: every thread of the warp has its S row in registers (the load above is
            // warp-wide), other warps own other lanes; the row sum is taken by the tensor pipe from the rounded P
            tmem_st16(trow + s * kBK, pk);
            tmem_st_wait();
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive(p_ready(L, s));
        }
        if (ok) {
            const bool store = qpos < nq;
            const long long off = (bb * nq + qpos) * (long long)(H * D) + h * D;
            // The row's gate, on its way under the last P V; whole sectors in and out (rows of heads of 48 are 96 bytes)
            constexpr int kV = D % 16 == 0 ? 16 : 8;   // channels per access
            uint32_t gw[D / kV][kV / 2];
            if (store && gate != nullptr) {
#pragma unroll
                for (int c = 0; c < D / kV; ++c) load_row<kV>(gate + off + c * kV, gw[c]);
            }
            if (mbar_wait(pv_done(L, (nblk - 1) & 1), ((nblk - 1) >> 1) & 1u, abort_flag)) {
                tc_fence_after_sync();
                const uint32_t lsum = tmem_ld1(trow + C::kColO + DV);
                tmem_ld_wait();
                const float inv = 1.0f / __uint_as_float(lsum);
                float gmin = 0.f;
#pragma unroll
                for (int part = 0; part < DV / 16; ++part) {
                    uint32_t r[16];
                    tmem_ld16(trow + C::kColO + part * 16, r);
                    tmem_ld_wait();
#pragma unroll
                    for (int c = part * 16 / kV; c < (part + 1) * 16 / kV && c < D / kV; ++c) {
                        float f[kV];
#pragma unroll
                        for (int e = 0; e < kV; ++e) f[e] = __uint_as_float(r[c * kV % 16 + e]) * inv;
                        if (gate != nullptr) {
#pragma unroll
                            for (int e = 0; e < kV; ++e) {
                                const float ge = (e & 1) ? bf16hi(gw[c][e >> 1]) : bf16lo(gw[c][e >> 1]);
                                gmin = fminf(gmin, ge);
                                f[e] *= rcp_of(1.0f + __expf(-ge));
                            }
                        }
                        uint32_t o[kV / 2];
#pragma unroll
                        for (int e = 0; e < kV / 2; ++e) o[e] = pack_bf16x2(f[2 * e], f[2 * e + 1]);
                        if (store) store_row<kV>(out + off + c * kV, o);
                    }
                }
                // A row with a closed gate, past the range of rcp_of: once more by the division (exactly 0 where the
                // exponential overflows). A loop of its own, which costs nothing where it is not run.
                if (__any_sync(0xffffffffu, store && gate != nullptr && gmin < kSigmoidMin)) {
#pragma unroll 1
                    for (int c = 0; c < D; ++c) {
                        const uint32_t acc = tmem_ld1(trow + C::kColO + c);
                        tmem_ld_wait();
                        if (store)
                            out[off + c] = __float2bfloat16_rn(__uint_as_float(acc) * inv * sigmoidf_fast(__bfloat162float(gate[off + c])));
                    }
                }
            } else if (lane == 0) {
                report_wait_failure(status, abort_flag, kKidSingleCore, 10);
            }
        }
    }

    tc_fence_before_sync();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after_sync();
        tmem_dealloc(tmem_base, kLines * 128);
    }
}

template <int D, int kLines>
int launch_core(const SingleImages& im, const bf16* g, const bf16* tb, const bf16* mask, bf16* out, int BB, int N, int nq,
                int H, float inf, int rpb, uint32_t smem, cudaStream_t st) {
    // Sizes depend on N and on the lines of a call, and the limit is the kernel's, for all threads of the process: the largest, once
    static PerDeviceOnce configured;
    if (!configured.done()) {
        OF3_CUDA_CHECK(cudaFuncSetAttribute(single_core_kernel<D, kLines>, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxSmem));
        configured.mark();
    }
    const long long each = (long long)(BB / rpb) * H * ceil_div(nq, kBQ), pairs = each * (rpb / kLines);
    const long long grid = pairs + (rpb % kLines ? each : 0);
    LaunchScope scope(kKidSingleCore, st);
    OF3_CUDA_CHECK(launch_chained(single_core_kernel<D, kLines>, dim3((unsigned)grid), kThreads<kLines>, smem, st, im.q, im.k,
                                  im.v, tb, mask, g, out, N, nq, H, rpb, (int)pairs, inf, device_status_ptr()));
    return OF3_OK;
}

// One line per CTA where the chip takes all lines at once (three per SM), two above. A line's step is a chain of hand-offs: an SM
// with four lines needs some 1900 cycles for a step of each, with fewer up to half of that, so the launch takes as long as its
// fullest SM. Under the launch before, whose blocks end one by one, the SMs that are free first took two CTAs of two lines each
// while others stayed empty. So a CTA takes shared memory of which an SM has only as many shares as the lines need (not beside
// another stack, whose blocks want to share the SM). Steps of 24 blocks, two lines per CTA -> this: 111 tokens 759 -> 755 us,
// 5 x 111 1046 -> 959, 1024 1571 -> 1480, 3 x 300 1393 -> 1241, 2 x 700 1797 -> 1597, 5 x 500 2225 -> 2108, 5 x 640 2634 -> 2539
// (lines per SM of the last four: 1, 2, 3, 3). Without the shares 3 x 300 1293, 3 x 400 1599 (with 1436). More lines, two per CTA:
// the pairs first and the odd samples behind them, which end the launch sooner than pairs do (5 x 1024: 4214 -> 4091).
template <int D>
int core_impl(const SingleImages& im, const bf16* g, const bf16* tb, const bf16* mask, bf16* out, int BB, int N, int nq,
              int H, float inf, int rpb, bool spread, cudaStream_t st) {
    const int nkp = ceil_div(N, kBK) * kBK;
    const long long lines = (long long)BB * H * ceil_div(nq, kBQ), sms = sm_count();
    uint32_t smem = Cfg<D, 1>::dyn_bytes(nkp);
    constexpr uint32_t kSmBytes = 228 * 1024, kReserved = 1024;   // shared memory of an SM, of it per CTA
    int fit = (int)(kSmBytes / (smem + kReserved));
    if (fit > kCtasPerSm<1>) fit = kCtasPerSm<1>;
    if (rpb > 1 && lines > fit * sms)
        return launch_core<D, 2>(im, g, tb, mask, out, BB, N, nq, H, inf, rpb, Cfg<D, 2>::dyn_bytes(nkp), st);
    const long long per_sm = (lines + sms - 1) / sms;
    if (spread && per_sm < fit) {
        const uint32_t more = kSmBytes / (uint32_t)(per_sm + 1) - kReserved + 1024;   // one more would not fit
        smem = smem > more ? smem : more;
    }
    return launch_core<D, 1>(im, g, tb, mask, out, BB, N, nq, H, inf, rpb, smem, st);
}

}  // namespace

// d in {24, 48}; H * d a multiple of 8 (16-byte rows per head); N within the mask row a CTA keeps.
bool single_attn_tc_supported(int N, int H, int d) {
    if (!(d == 24 || d == 48) || N < 1 || N > kMaxKeysSingle || H * d % 64 != 0) return false;
    const size_t smem = d == 24 ? Cfg<24, 2>::dyn_bytes(ceil_div(N, kBK) * kBK) : Cfg<48, 2>::dyn_bytes(ceil_div(N, kBK) * kBK);
    return smem <= kMaxSmem;
}

SingleImages take_single_images(Arena& ws, int BB, int N, int nq, int H, int d) {
    const size_t n_qt = ceil_div(nq, kBQ), nkb = ceil_div(N, kBK), bh = (size_t)BB * H;
    SingleImages im;
    im.q = (bf16*)ws.take(bh * n_qt * (d == 24 ? Cfg<24, 1>::kQBytes : Cfg<48, 1>::kQBytes));
    im.k = (bf16*)ws.take(bh * nkb * (d == 24 ? Cfg<24, 1>::kKBytes : Cfg<48, 1>::kKBytes));
    im.v = (bf16*)ws.take(bh * nkb * (d == 24 ? Cfg<24, 1>::kVBytes : Cfg<48, 1>::kVBytes));
    return im;
}

// Gated attention with pair bias over BB samples of N keys and nq query rows each:
//   out[bb, i, h, :] = sigmoid(g[bb, i, h, :]) * softmax_j((q[bb, i, h] + q_bias[h]) . k[bb, j, h] / sqrt(d)
//                                                       + inf * (mask[bb, j] - 1) + pair_bias[bb / rpb, h, i, j]) v
// g, out: [BB, nq, H*d]; mask [BB, N] or null; tb: room for the bias tiles where they are not given.
int single_attn(const SingleImages& im, const bf16* g, const SingleBias& bias, bf16* tb, const bf16* mask, bf16* out,
                int BB, int N, int nq, int H, int d, float inf, int rows_per_bias, bool spread, cudaStream_t st) {
    OF3_REQUIRE(single_attn_tc_supported(N, H, d), OF3_ERR_SHAPE, "single attention: N %d, H %d, d %d not supported",
                N, H, d);
    OF3_REQUIRE(rows_per_bias > 0 && BB % rows_per_bias == 0, OF3_ERR_SHAPE,
                "single attention: %d samples do not divide into groups of %d", BB, rows_per_bias);
    const int Bz = BB / rows_per_bias;
    const bf16* tiles = tb;
    if (bias.tiles != nullptr) {
        tiles = bias.tiles;   // projected earlier, in this kernel's layout
    } else if (bias.f32 != nullptr) {
        LaunchScope scope(kKidSingleAttn, st);
        single_bias_kernel<<<dim3(nq, Bz * H), 256, 0, st>>>(bias.f32, tb, N, nq, ceil_div(N, kBK));
        OF3_CUDA_CHECK(cudaGetLastError());
    } else {   // straight from the pair tensor: no fp32 bias in between
        OF3_REQUIRE(bias.z != nullptr && bias.w != nullptr && nq == N && H == 16, OF3_ERR_ARG,
                    "single attention: neither a pair bias nor a whole pair tensor to project it from");
        const int rc = pair_bias_tiles_c128_h16(bias.z, bias.ln_w, bias.ln_b, bias.w, tb, Bz, N, st);
        if (rc) return rc;
    }
    return d == 24 ? core_impl<24>(im, g, tiles, mask, out, BB, N, nq, H, inf, rows_per_bias, spread, st)
                   : core_impl<48>(im, g, tiles, mask, out, BB, N, nq, H, inf, rows_per_bias, spread, st);
}

}  // namespace fast
}  // namespace of3
