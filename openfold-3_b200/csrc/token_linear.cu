// Linear layers of few tokens on tcgen05 (bf16 operands, fp32 accumulation): the projections of the diffusion token stack
// (c_a = 768) where a call has too few 128-row tiles to fill the chip.
//
// The roles of linear.cu's operands change places: a tile is 128 output channels (the weights are the A operand, a TMEM lane is
// a channel) by NT tokens (the B operand, a TMEM column is a token). A CTA then waits for NT rows of x instead of 128, which
// come from the kernel ahead, while most of its weights, which do not, are in shared memory before that kernel has ended; and
// a tile has NT columns to hand on instead of 64.
//
// 576 threads: warp 0 TMA producer (128-byte swizzled k-blocks of 64), warp 1 MMA issuer (128 x NT x 16), warps 2..17 the epilogue
// (four per 32 channels, each a quarter of the tokens; thread = channel).
//
// What bounds them: latency. Of a launch of 111 tokens 0.9 us pass from the last store of the kernel ahead to the end of the wait
// for it, 0.6 until x is there, 1.2 (k = 768) for the product, whose instructions take 25 (64 channels) or 41 (128) cycles each,
// 0.2 - 0.9 for the epilogue. Step of 24 blocks, linear.cu -> here, us: 40 tokens 867 -> 655, 111 923 -> 757, 190 976 -> 846, 380
// 1092 -> 1013, 600 1272 -> 1207, 768 1350 -> 1288, 5 x 75 1021 -> 925. Half an SM's shared memory, so that a CTA starts beside
// one that has yet to end: 111 tokens 854 instead of 789 (with one k-block per stage). The adaptive LayerNorm in these kernels,
// a tile's rows in each of its CTAs: 111 tokens 964, 380 1676 (some 35 instructions per value, 24 times).
// Reference: openfold3/core/model/layers/attention_pair_bias.py:123-227, openfold3/core/model/layers/transition.py:325-339.
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
constexpr int kBK = 64;              // k-block
constexpr int kParts = 4;            // epilogue warps per quarter of the channels, each with its part of the tokens
constexpr int kThreads = 32 * (2 + 4 * kParts);
constexpr int kGroup = 3;            // k-blocks of a stage
constexpr int kMaxStages = 8;
constexpr float kLog2e = 1.4426950408889634f;

enum Epi { kImages, kSwiglu, kResidual };

// BF channels by NT tokens
template <int BF, int NT>
struct Cfg {
    // a stage: kGroup k-blocks of the weights, then of the tokens. A wait of the issuing thread costs its next instructions 120
    // cycles and more, as much as a k-block's four products take: with one per k-block they took 282 cycles (64 x 16 channels and
    // tokens) and 315 (128 x 32), with one per three 182 and 238.
    static constexpr int kWBlock = BF * kBK * 2, kXBlock = NT * kBK * 2;
    static constexpr int kWBytes = kGroup * kWBlock;
    static constexpr int kStageBytes = kWBytes + kGroup * kXBlock;
    static constexpr int kFixed = 1024 + 256;
    static constexpr int kFit = (227 * 1024 - kFixed) / kStageBytes;
    static constexpr int kStages = kFit < kMaxStages ? kFit : kMaxStages;
    static constexpr int kTmemCols = NT < 32 ? 32 : NT;
};

struct TokMaps {
    CUtensorMap x, w[4];
};
struct TokArgs {
    // kImages
    AttnImages im;
    int kind[4];
    float qscale;
    // kSwiglu, kResidual
    bf16* out;
    const bf16 *residual, *gate, *gate_bias, *mask;
};

// v0, v1: this lane's channel for tokens t and t + 1. The bf16 pair of channels (lane & ~1, lane | 1) of token t + (lane & 1).
__device__ __forceinline__ uint32_t pair_channels(float v0, float v1, int lane) {
    const float other = __shfl_xor_sync(0xffffffffu, lane & 1 ? v0 : v1, 1);
    return lane & 1 ? pack_bf16x2(other, v1) : pack_bf16x2(v0, other);
}

template <int N>
__device__ __forceinline__ void tmem_ld_cols(uint32_t taddr, uint32_t (&r)[N]) {
    if constexpr (N == 16) tmem_ld16(taddr, r);
    else if constexpr (N == 8) tmem_ld8(taddr, r);
    else tmem_ld4(taddr, r);
}

// D: channels per head (kImages)
template <int BF, int NT, int EPI, int D>
__global__ void __launch_bounds__(kThreads, 1)
token_linear_kernel(const __grid_constant__ TokMaps maps, const TokArgs ar, int rows, int K, int n, int tok_tiles,
                    int* status) {
    using C = Cfg<BF, NT>;
    constexpr int kTok = NT / kParts;                       // tokens per thread
    constexpr int kOut = EPI == kSwiglu ? BF / 2 : BF;      // result channels of a tile
    constexpr int stages = C::kStages;
    extern __shared__ uint8_t smem_raw[];
    const uint32_t sbase = (smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t* gbase = smem_raw + (sbase - smem_u32(smem_raw));
    const uint32_t bars = sbase + stages * C::kStageBytes;
    auto full = [&](int s) { return bars + 8u * s; };
    auto empty = [&](int s) { return bars + 8u * (kMaxStages + s); };
    const uint32_t done = bars + 8u * (2 * kMaxStages);
    uint8_t* tail = gbase + stages * C::kStageBytes + 8 * (2 * kMaxStages + 1);
    volatile uint32_t* tmem_ptr = reinterpret_cast<volatile uint32_t*>(tail);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tail + 8);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int num_groups = (K / kBK + kGroup - 1) / kGroup;   // (of the last one, k-blocks past the end are zeros)
    // token tiles innermost: CTAs that run at the same time share the weights
    const int tt = blockIdx.x % tok_tiles, ft = blockIdx.x / tok_tiles;
    const int per_mat = n / kOut;
    const int g = EPI == kImages ? ft / per_mat : 0, nt = EPI == kImages ? ft - g * per_mat : ft;
    // kImages: a tile lies in one sample, so that its keys fill whole chunks of the V image
    const int ns = EPI == kImages ? ar.im.rows_per_sample : rows;
    const int per_sample = tok_tiles / (EPI == kImages ? rows / ns : 1), bb = EPI == kImages ? tt / per_sample : 0;
    const int pos0 = (EPI == kImages ? tt - bb * per_sample : tt) * NT;   // first token, in its sample

    if (threadIdx.x == 0) {
        for (int s = 0; s < stages; ++s) {
            mbar_init(full(s), 1);
            mbar_init(empty(s), 1);
        }
        mbar_init(done, 1);
        *abort_flag = 0;
        mbar_fence_init();
        prefetch_tmap(&maps.w[g]);
        prefetch_tmap(&maps.x);
    }
    if (warp == 1) {
        tmem_alloc(smem_u32((const void*)tmem_ptr), C::kTmemCols);
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
            auto load_w = [&](int gr, int s) {
                const uint32_t dst = sbase + s * C::kStageBytes;
                if constexpr (EPI == kSwiglu) {
                    // a warp's 32 lanes: 16 channels of the first matrix, the same 16 of the second
                    for (int kb = 0; kb < kGroup; ++kb)
#pragma unroll
                        for (int b = 0; b < BF / 16; ++b)
                            tma_load_3d(dst + kb * C::kWBlock + b * 2048, &maps.w[b & 1], full(s), 0, nt * kOut + (b >> 1) * 16,
                                        gr * kGroup + kb);
                } else {
                    tma_load_3d(dst, &maps.w[g], full(s), 0, nt * BF, gr * kGroup);
                }
            };
            auto load_x = [&](int gr, int s) {
                tma_load_3d(sbase + s * C::kStageBytes + C::kWBytes, &maps.x, full(s), 0, bb * ns + pos0, gr * kGroup);
            };
            const int ahead = num_groups < stages ? num_groups : stages;
            for (int gr = 0; gr < ahead; ++gr) {
                mbar_arrive_expect_tx(full(gr), C::kStageBytes);
                load_w(gr, gr);
            }
            grid_wait();
            for (int gr = 0; gr < ahead; ++gr) load_x(gr, gr);
            uint32_t ph = 0;
            for (int gr = ahead, s = 0; gr < num_groups; ++gr) {
                if (!mbar_wait(empty(s), ph, abort_flag)) {
                    report_wait_failure(status, abort_flag, kKid, 11);
                    break;
                }
                mbar_arrive_expect_tx(full(s), C::kStageBytes);
                load_x(gr, s);
                load_w(gr, s);
                if (++s == stages) {
                    s = 0;
                    ph ^= 1u;
                }
            }
        }
    } else if (warp == 1) {
        // ---------------------------------------------------------------- MMA issuer
        if (elect_one()) {
            constexpr uint32_t idesc = idesc_bf16_f32(BF, NT);
            bool ok = true;
            uint32_t ph = 0;
            for (int gr = 0, s = 0; gr < num_groups; ++gr) {
                if (!mbar_wait(full(s), ph, abort_flag)) {
                    report_wait_failure(status, abort_flag, kKid, 12);
                    ok = false;
                    break;
                }
                tc_fence_after_sync();
                const uint32_t sw = sbase + s * C::kStageBytes;
#pragma unroll
                for (int kb = 0; kb < kGroup; ++kb) {
                    const uint64_t wd = smem_desc_k_sw128(sw + kb * C::kWBlock);
                    const uint64_t xd = smem_desc_k_sw128(sw + C::kWBytes + kb * C::kXBlock);
#pragma unroll
                    for (int k4 = 0; k4 < kBK / 16; ++k4)
                        mma_bf16(tmem_base, wd + 2u * k4, xd + 2u * k4, idesc, (gr | kb | k4) != 0 ? 1u : 0u);
                }
                mma_commit(empty(s));
                if (++s == stages) {
                    s = 0;
                    ph ^= 1u;
                }
            }
            if (ok) mma_commit(done);
        }
    } else {
        // ---------------------------------------------------------------- epilogue: thread = channel, kTok tokens
        const int quad = warp & 3, part = (warp - 2) >> 2;
        grid_wait();
        const int tok = pos0 + part * kTok;                    // first token of this thread, in its sample
        const uint32_t taddr = tmem_base + ((uint32_t)(quad * 32) << 16) + part * kTok;
        if constexpr (EPI == kResidual) {
            // 64 channels: rows 16 q .. 16 q + 15 of the tile in the first lanes of warp q. A lane finishes two of them (one
            // 4-byte access) for a quarter of the thread's tokens: t = 4 i + cls.
            static_assert(BF == 64, "lanes of the tile");
            const int cls = (lane & 1) + 2 * (lane >> 4), c = nt * BF + quad * 16 + (lane & 14);
            uint32_t zv[kTok / 4], gv[kTok / 4];
            float s0[kTok / 4], s1[kTok / 4], mk[kTok / 4];
            const float b0 = ar.gate ? __bfloat162float(ar.gate_bias[c]) : 0.f;
            const float b1 = ar.gate ? __bfloat162float(ar.gate_bias[c + 1]) : 0.f;
#pragma unroll
            for (int i = 0; i < kTok / 4; ++i) {
                const int t = tok + 4 * i + cls;
                zv[i] = gv[i] = 0u;
                mk[i] = 1.0f;
                if (t >= rows) continue;
                const long long off = (long long)t * n + c;
                if (ar.gate) gv[i] = *reinterpret_cast<const uint32_t*>(ar.gate + off);
                if (ar.residual) zv[i] = *reinterpret_cast<const uint32_t*>(ar.residual + off);
                if (ar.mask) mk[i] = __bfloat162float(ar.mask[t]);
            }
#pragma unroll
            for (int i = 0; i < kTok / 4; ++i) {
                s0[i] = ar.gate ? sigmoid_of(bf16lo(gv[i]) + b0) : 1.0f;
                s1[i] = ar.gate ? sigmoid_of(bf16hi(gv[i]) + b1) : 1.0f;
                asm volatile("" : "+f"(s0[i]), "+f"(s1[i]));   // not behind the wait
            }
            if (!mbar_wait(done, 0, abort_flag)) {
                if (lane == 0) report_wait_failure(status, abort_flag, kKid, 13);
            } else {
                tc_fence_after_sync();
                uint32_t r[kTok];
                tmem_ld_cols(taddr, r);
                tmem_ld_wait();
#pragma unroll
                for (int i = 0; i < kTok / 4; ++i) {
                    const uint32_t u0 = __shfl_sync(0xffffffffu, r[4 * i + 2], lane & 15);
                    const uint32_t u1 = __shfl_sync(0xffffffffu, r[4 * i + 3], lane & 15);
                    const float v0 = __uint_as_float(lane < 16 ? r[4 * i] : u0), v1 = __uint_as_float(lane < 16 ? r[4 * i + 1] : u1);
                    const float other = __shfl_xor_sync(0xffffffffu, lane & 1 ? v0 : v1, 1);
                    float lo = lane & 1 ? other : v0, hi = lane & 1 ? v1 : other;
                    lo = __fmul_rn(__fmul_rn(mk[i], lo), s0[i]);   // not one fma with the residual
                    hi = __fmul_rn(__fmul_rn(mk[i], hi), s1[i]);
                    if (ar.residual) {
                        lo += bf16lo(zv[i]);
                        hi += bf16hi(zv[i]);
                    }
                    const int t = tok + 4 * i + cls;
                    if (t < rows) *reinterpret_cast<uint32_t*>(ar.out + (long long)t * n + c) = pack_bf16x2(lo, hi);
                }
                tc_fence_before_sync();
            }
        } else if (!mbar_wait(done, 0, abort_flag)) {
            if (lane == 0) report_wait_failure(status, abort_flag, kKid, 14);
        } else {
            tc_fence_after_sync();
            uint32_t r[kTok];
            tmem_ld_cols(taddr, r);
            tmem_ld_wait();
            float v[kTok];
#pragma unroll
            for (int e = 0; e < kTok; ++e) v[e] = __uint_as_float(r[e]);
            if constexpr (EPI == kSwiglu) {
                static_assert(EPI != kSwiglu || BF == 128, "lanes of the tile");
                const bool up = lane >= 16;
                const int f = nt * kOut + quad * 16 + (lane & 15);
#pragma unroll
                for (int i = 0; i < kTok; i += 2) {   // lanes 0..15: token i, 16..31: token i + 1
                    const float other = __shfl_xor_sync(0xffffffffu, up ? v[i] : v[i + 1], 16);
                    const float a = up ? other : v[i], b = up ? v[i + 1] : other;
                    const int t = tok + i + up;
                    if (t < rows) ar.out[(long long)t * n + f] = __float2bfloat16_rn(a * sigmoid_of(a) * b);
                }
            } else {
                static_assert(EPI != kImages || BF == 128, "lanes of the tile");
                const AttnImages& im = ar.im;
                constexpr int KD = SingleImage<D>::kKD, DV = SingleImage<D>::kDV;
                const int kind = ar.kind[g], HD = im.H * D;
                const int nkb = (ns + kSingleBK - 1) / kSingleBK, n_qt = (ns + kSingleBQ - 1) / kSingleBQ;
                const int f = nt * kOut + quad * 32 + lane;   // channel, in its matrix
                const int h = f / D, d = f - h * D;
                const long long bh = (long long)bb * im.H + h;
                if (kind == kOutV) {
                    // tile [DV channels][32 keys], 64-byte rows: this channel's keys, a chunk of eight (or half a one) at a time;
                    // keys past the end of the last block are zeros
                    constexpr int kRun = kTok < 8 ? kTok : 8;
#pragma unroll
                    for (int i = 0; i < kTok; i += kRun) {
                        const int p = tok + i;
                        if (p >= nkb * kSingleBK) break;
                        uint32_t o[kRun / 2];
#pragma unroll
                        for (int e = 0; e < kRun; e += 2)
                            o[e / 2] = pack_bf16x2(p + e < ns ? v[i + e] : 0.f, p + e + 1 < ns ? v[i + e + 1] : 0.f);
                        bf16* t = im.v + ((bh * nkb + (p >> 5)) * DV + d) * kSingleBK +
                                  (((((p & 31) >> 3) ^ ((d >> 1) & 3)) << 3) | (p & 7));
                        if constexpr (kRun == 8) *reinterpret_cast<uint4*>(t) = make_uint4(o[0], o[1], o[2], o[3]);
                        else *reinterpret_cast<uint2*>(t) = make_uint2(o[0], o[1]);
                    }
                } else {
                    const float qb = kind == kOutQ && im.q_bias ? __bfloat162float(im.q_bias[f]) : 0.f;
                    const int dp = d & ~1;   // (an even channel and the next one lie in one head and chunk)
                    constexpr int kRow = KD * 2;   // bytes of an image's row
                    const bool last = D < KD && D <= 32 && dp >= D - 8;   // 24 channels: chunk 3 of the row pads K with zeros
                    uint8_t* const q = reinterpret_cast<uint8_t*>(im.q) + bh * n_qt * (long long)(kSingleBQ * kRow);
                    uint8_t* const k = reinterpret_cast<uint8_t*>(im.k) + bh * nkb * (long long)(kSingleBK * kRow);
#pragma unroll
                    for (int i = 0; i < kTok; i += 2) {
                        float v0 = v[i], v1 = v[i + 1];
                        if (kind == kOutQ) {
                            if (im.q_bias) {
                                v0 += qb;
                                v1 += qb;
                            }
                            v0 *= ar.qscale;
                            v1 *= ar.qscale;
                        }
                        const uint32_t o = pair_channels(v0, v1, lane);
                        const int p = tok + i + (lane & 1);
                        auto in_row = [&](int c) {   // chunk c of row p, from the row's start
                            return single_chunk_off<KD>(p & 7, c) - (p & 7) * kRow + (dp & 7) * 2;
                        };
                        if (kind == kOutG) {
                            if (p < ns) *reinterpret_cast<uint32_t*>(im.g + ((long long)bb * ns + p) * HD + (f & ~1)) = o;
                        } else {   // tiles of 128 (32) rows, one behind the other
                            const bool is_q = kind == kOutQ;
                            uint8_t* const row = (is_q ? q : k) + (long long)p * kRow;
                            if (p < (is_q ? ns : nkb * kSingleBK)) {
                                *reinterpret_cast<uint32_t*>(row + in_row(dp >> 3)) = p < ns ? o : 0u;
                                if (last) *reinterpret_cast<uint32_t*>(row + in_row((dp >> 3) + 1)) = 0u;
                            }
                        }
                    }
                }
            }
            tc_fence_before_sync();
        }
    }

    tc_fence_before_sync();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after_sync();
        tmem_dealloc(tmem_base, C::kTmemCols);
    }
}

template <int BF, int NT, int EPI, int D>
int launch(const TokArgs& ar, const LinearIn& in, int tok_tiles, int grid, cudaStream_t st) {
    using C = Cfg<BF, NT>;
    TokMaps maps;
    int rc;
    // k in blocks, the third dimension: a box is the k-blocks of a stage
    const uint64_t str[2] = {(uint64_t)in.k * 2, kBK * 2};
    for (int i = 0; i < in.num_w; ++i) {
        const uint64_t dims[3] = {kBK, (uint64_t)in.n, (uint64_t)in.k / kBK};
        const uint32_t box[3] = {kBK, EPI == kSwiglu ? 16u : (uint32_t)BF, EPI == kSwiglu ? 1u : (uint32_t)kGroup};
        if ((rc = make_tmap_bf16(&maps.w[i], in.w[i], 3, dims, str, box, 1))) return rc;
    }
    for (int i = in.num_w; i < 4; ++i) maps.w[i] = maps.w[0];
    {
        const uint64_t dims[3] = {kBK, (uint64_t)in.rows, (uint64_t)in.k / kBK};
        const uint32_t box[3] = {kBK, NT, kGroup};
        if ((rc = make_tmap_bf16(&maps.x, in.x, 3, dims, str, box, 1))) return rc;
    }
    constexpr int smem = C::kStages * C::kStageBytes + C::kFixed;
    static PerDeviceOnce configured;
    if (!configured.done()) {
        OF3_CUDA_CHECK(cudaFuncSetAttribute(token_linear_kernel<BF, NT, EPI, D>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
        configured.mark();
    }
    LaunchScope scope(kKid, st);
    OF3_CUDA_CHECK(launch_chained(token_linear_kernel<BF, NT, EPI, D>, grid, kThreads, smem, st, maps, ar, (int)in.rows, in.k, in.n,
                                  tok_tiles, device_status_ptr()));
    return OF3_OK;
}

// Tokens per tile: the fewest that one wave of CTAs covers, since a tile's loads and epilogue grow with them and its products
// hardly do. `samples`: tiles lie in one sample each.
template <int BF, int EPI, int D = 0>
int by_tokens(const TokArgs& ar, const LinearIn& in, int samples, int channel_tiles, cudaStream_t st) {
    // (kImages: whole key blocks of 32, of which the tiles write the end as zeros)
    const int ns = EPI == kImages ? ((int)(in.rows / samples) + 31) / 32 * 32 : (int)in.rows;
    auto tiles = [&](int nt) { return samples * ((ns + nt - 1) / nt); };
    auto fits = [&](int nt) { return tiles(nt) * channel_tiles <= sm_count(); };
    if (fits(16)) return launch<BF, 16, EPI, D>(ar, in, tiles(16), tiles(16) * channel_tiles, st);
    if (fits(32)) return launch<BF, 32, EPI, D>(ar, in, tiles(32), tiles(32) * channel_tiles, st);
    return launch<BF, 64, EPI, D>(ar, in, tiles(64), tiles(64) * channel_tiles, st);
}

}  // namespace

// One wave of tiles of 64 tokens. (Two and three waves of the projections of 768 to 3072 channels: 500 tokens 1352 us per step
// against 1201 by 128-row tiles, 780 1817 against 1484.)
static bool one_wave(long long samples, long long tokens, int channel_tiles) {
    return samples * ((tokens + 63) / 64) * channel_tiles <= sm_count();
}
bool token_images_supported(int samples, int tokens, int c, int d) {
    return c % 128 == 0 && (d == 24 || d == 48) && one_wave(samples, tokens, 4 * c / 128);
}
bool token_swiglu_supported(long long rows, int hidden) { return hidden % 64 == 0 && one_wave(1, rows, hidden / 64); }
bool token_residual_supported(long long rows, int c) { return c % 64 == 0 && one_wave(1, rows, c / 64); }

int token_attn_images(const LinearIn& in, const LinearOut* kinds, const AttnImages& im, cudaStream_t st) {
    TokArgs ar = {};
    ar.im = im;
    for (int i = 0; i < in.num_w; ++i) ar.kind[i] = kinds[i];
    ar.qscale = kLog2e * (1.0f / sqrtf((float)im.D));
    const int samples = (int)(in.rows / im.rows_per_sample), tiles = in.n / 128 * in.num_w;
    return im.D == 24 ? by_tokens<128, kImages, 24>(ar, in, samples, tiles, st) : by_tokens<128, kImages, 48>(ar, in, samples, tiles, st);
}

int token_swiglu(const LinearIn& in, bf16* h, cudaStream_t st) {
    TokArgs ar = {};
    ar.out = h;
    return by_tokens<128, kSwiglu>(ar, in, 1, in.n / 64, st);
}

int token_residual(const LinearIn& in, const bf16* residual, const bf16* gate, const bf16* gate_bias, const bf16* mask, bf16* out,
                   cudaStream_t st) {
    TokArgs ar = {};
    ar.out = out;
    ar.residual = residual;
    ar.gate = gate;
    ar.gate_bias = gate_bias;
    ar.mask = mask;
    return by_tokens<64, kResidual>(ar, in, 1, in.n / 64, st);
}

}  // namespace fast
}  // namespace of3
