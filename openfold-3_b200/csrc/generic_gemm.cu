// fp32 GEMMs of the shape-generic family, with the element-wise step that follows in the epilogue.
//
// Large layers of fp32 operands run on the tensor cores as products of three bf16 parts (gemm_split_kernel): below the FMA pipe's
// error, and past its 75 TFLOP/s. Few rows, and bf16 weights, stay on the FMA pipe: tiles of 128 x 64 with 8 x 8 products per
// thread (packed fma.f32x2; the next k-slab is in registers while this one is multiplied), and where there are few of these, or
// the operands are fp32, 32 x 32 tiles whose k-slab is split over four groups of threads (the chain over k = 1536 on 24 large tiles
// is what such a layer waits for). Fp32 trunk block, FMA pipe alone / as here, us: N = 48 429 / 369, 64 520 / 434, 128 955 / 695, 250
// 3310 / 2246.
#include "generic_ops.cuh"
#include "runtime.cuh"
#include "umma.cuh"
#include <type_traits>

namespace of3 {
namespace generic {
namespace {

typedef unsigned long long u64;

__device__ __forceinline__ float sigmoid_acc(float x) { return 1.0f / (1.0f + expf(-x)); }
__device__ __forceinline__ u64 dup2(float a) {
    u64 d;
    asm("mov.b64 %0, {%1, %1};" : "=l"(d) : "f"(a));
    return d;
}
__device__ __forceinline__ void fma2(u64& acc, u64 a, u64 b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b));
}
__device__ __forceinline__ float2 unpack2(u64 v) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
// four consecutive elements, `n` of which exist (n <= 0: none)
__device__ __forceinline__ float4 load4(const float* p, int n, bool vec) {
    if (vec && n >= 4) return *reinterpret_cast<const float4*>(p);
    return make_float4(n > 0 ? p[0] : 0.f, n > 1 ? p[1] : 0.f, n > 2 ? p[2] : 0.f, n > 3 ? p[3] : 0.f);
}
__device__ __forceinline__ float4 load4(const __nv_bfloat16* p, int n, bool vec) {
    if (vec && n >= 4) {
        const uint2 v = *reinterpret_cast<const uint2*>(p);
        return make_float4(bf16lo(v.x), bf16hi(v.x), bf16lo(v.y), bf16hi(v.y));
    }
    return make_float4(n > 0 ? __bfloat162float(p[0]) : 0.f, n > 1 ? __bfloat162float(p[1]) : 0.f,
                       n > 2 ? __bfloat162float(p[2]) : 0.f, n > 3 ? __bfloat162float(p[3]) : 0.f);
}
template <typename T>
__device__ __forceinline__ bool vec_ok(const T* p, long long ld) {
    return (reinterpret_cast<uintptr_t>(p) & (4 * sizeof(T) - 1)) == 0 && (ld & 3) == 0;
}

__device__ __forceinline__ void store4(__nv_bfloat16* p, const float (&o)[4]) {
    *reinterpret_cast<uint2*>(p) = make_uint2(pack_bf16x2(o[0], o[1]), pack_bf16x2(o[2], o[3]));
}
enum Epi { kStore, kGatedPlanes, kSwiglu, kFinal };

template <typename T>
struct Args {
    const float* a;          // [M][K], pitch K (k_outer: [K][M], pitch M)
    const T* w[8];           // [n][K], pitch K (k_outer: [K][n], pitch n)
    const T* bias[4];
    float* out[4];
    long long M, a_batch;    // a_batch: plane stride of a, w[0] and out[0] (batched products only)
    int n, K;
    const T* mask;
    const float* gate;
    const T* residual;
    T* final_out;
    RowMap map;
};

// What follows the product of a thread's TM x TN values: row_of(i), col_of(j) say where they lie.
template <int BM, int BN, int TM, int TN, int EPI, typename T>
__device__ __forceinline__ void epilogue(const Args<T>& p, const float (&v)[TM][TN], long long m0, int n0, int grp,
                                         long long boff, int tx, int ty) {
    constexpr int HN = BN / 2, HM = BM / 2, TN2 = TN / 2, TM2 = TM / 2;
    const int n = p.n;
    const long long M = p.M;
    auto row_of = [&](int i) { return m0 + (i / TM2) * HM + ty * TM2 + i % TM2; };
    auto col_of = [&](int j) { return n0 + (j / TN2) * HN + tx * TN2 + j % TN2; };   // kPaired: j < TN / 2 only
    if constexpr (EPI == kGatedPlanes) {
        float* out = p.out[grp];
        const bool vo = vec_ok(out, M);
#pragma unroll
        for (int hf = 0; hf < 2; ++hf) {
            const long long r = row_of(hf * TM2);
            float mk[TM2];
#pragma unroll
            for (int i = 0; i < TM2; ++i) mk[i] = (p.mask && r + i < M) ? ld_as_float(p.mask + r + i) : 1.0f;
#pragma unroll
            for (int j = 0; j < TN2; ++j) {
                const int c = col_of(j);
                if (c >= n) continue;
                float o[TM2];
#pragma unroll
                for (int i = 0; i < TM2; ++i)
                    o[i] = mk[i] * sigmoid_acc(v[hf * TM2 + i][TN2 + j]) * v[hf * TM2 + i][j];
                float* d = out + (long long)c * M + r;
                if (TM2 == 4 && vo && r + 3 < M) {
                    *reinterpret_cast<float4*>(d) = make_float4(o[0], o[1], o[TM2 - 2], o[TM2 - 1]);
                } else {
#pragma unroll
                    for (int i = 0; i < TM2; ++i)
                        if (r + i < M) d[i] = o[i];
                }
            }
        }
        return;
    }
    if constexpr (EPI == kFinal && TN2 == 4) {
        // Whole vectors, the gate and residual of TM2 rows ahead of the first store: the output may be the residual's
        // own tensor, so that a load behind a store waits for it (with vector LayerNorm rows, one fp32 trunk block at
        // N = 128: 1077 -> 1011 us).
        const bool vec = (n & 3) == 0 && (p.map.inner_stride & 3) == 0 && (p.map.outer_stride & 3) == 0 &&
                         vec_ok(p.final_out, 0) && (!p.residual || vec_ok(p.residual, 0)) && (!p.gate || vec_ok(p.gate, n));
        if (vec) {
#pragma unroll
            for (int hm = 0; hm < 2; ++hm) {
                float4 gt[TM2][2], rs[TM2][2];
                float mk[TM2];
                long long off[TM2];
#pragma unroll
                for (int i = 0; i < TM2; ++i) {
                    const long long r = row_of(hm * TM2 + i);
                    off[i] = r < M ? row_offset(p.map, r) : -1;
                    mk[i] = (p.mask && r < M) ? ld_as_float(p.mask + r) : 1.0f;
#pragma unroll
                    for (int hf = 0; hf < 2; ++hf) {
                        const int c = col_of(hf * TN2), left = r < M ? n - c : 0;
                        gt[i][hf] = p.gate ? load4(p.gate + r * n + c, left, true) : make_float4(0.f, 0.f, 0.f, 0.f);
                        rs[i][hf] = p.residual ? load4(p.residual + off[i] + c, left, true) : make_float4(0.f, 0.f, 0.f, 0.f);
                    }
                }
#pragma unroll
                for (int i = 0; i < TM2; ++i) {
#pragma unroll
                    for (int hf = 0; hf < 2; ++hf) {
                        const int c = col_of(hf * TN2);
                        if (off[i] < 0 || c >= n) continue;
                        const float ge[4] = {gt[i][hf].x, gt[i][hf].y, gt[i][hf].z, gt[i][hf].w};
                        const float re[4] = {rs[i][hf].x, rs[i][hf].y, rs[i][hf].z, rs[i][hf].w};
                        float o[4];
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
                            o[j] = v[hm * TM2 + i][hf * TN2 + j];
                            if (p.gate) o[j] *= sigmoid_acc(ge[j]);
                            if (p.mask) o[j] *= mk[i];
                            if (p.residual) o[j] += re[j];
                        }
                        store4(p.final_out + off[i] + c, o);
                    }
                }
            }
            return;
        }
    }
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const long long r = row_of(i);
        if (r >= M) continue;
        if constexpr (EPI == kSwiglu) {
            float* d = p.out[0] + r * n;
            const int c = col_of(0);
            float o[TN2];
#pragma unroll
            for (int j = 0; j < TN2; ++j) o[j] = v[i][j] * sigmoid_acc(v[i][j]) * v[i][TN2 + j];
            if (TN2 == 4 && vec_ok(p.out[0], n) && c + 3 < n) {
                *reinterpret_cast<float4*>(d + c) = make_float4(o[0], o[1], o[TN2 - 2], o[TN2 - 1]);
            } else {
#pragma unroll
                for (int j = 0; j < TN2; ++j)
                    if (c + j < n) d[c + j] = o[j];
            }
        } else if constexpr (EPI == kStore) {
            float* d = p.out[grp] + boff + r * n;
            const bool vo = TN2 == 4 && vec_ok(p.out[grp] + boff, n);
#pragma unroll
            for (int hf = 0; hf < 2; ++hf) {
                const int c = col_of(hf * TN2);
                float o[TN2];
#pragma unroll
                for (int j = 0; j < TN2; ++j)
                    o[j] = v[i][hf * TN2 + j] + ((p.bias[grp] && c + j < n) ? ld_as_float(p.bias[grp] + c + j) : 0.f);
                if (vo && c + 3 < n) {
                    *reinterpret_cast<float4*>(d + c) = make_float4(o[0], o[1], o[TN2 - 2], o[TN2 - 1]);
                } else {
#pragma unroll
                    for (int j = 0; j < TN2; ++j)
                        if (c + j < n) d[c + j] = o[j];
                }
            }
        } else if constexpr (EPI == kFinal) {
            const float mk = p.mask ? ld_as_float(p.mask + r) : 1.0f;
            const long long off = row_offset(p.map, r);
#pragma unroll
            for (int j = 0; j < TN; ++j) {
                const int c = col_of(j);
                if (c >= n) continue;
                float o = v[i][j];
                if (p.gate) o *= sigmoid_acc(p.gate[r * n + c]);
                if (p.mask) o *= mk;
                if (p.residual) o += ld_as_float(p.residual + off + c);
                st_from_float(p.final_out + off + c, o);
            }
        }
    }
}

// BM x BN tile; G groups of (BM / TM) x (BN / TN) threads, group g multiplies k = g (mod G quarters) of each slab. A
// thread's rows are TM / 2 consecutive ones in each half of the tile, its columns TN / 2 in each half of the tile's BN;
// for the paired epilogues the left half of the columns comes from one weight and the right half from another.
template <int BM, int BN, int TM, int TN, int G, int EPI, bool K_OUTER, typename T>
__global__ void __launch_bounds__(G* BM / TM * BN / TN) gemm_kernel(const Args<T> p) {
    constexpr int BK = 16 * G;
    constexpr int kThreads = G * BM / TM * BN / TN;
    constexpr bool kPaired = EPI == kGatedPlanes || EPI == kSwiglu;
    constexpr int HN = BN / 2, HM = BM / 2, TN2 = TN / 2, TM2 = TM / 2;
    constexpr int LA = BM * BK / 4 / kThreads, LW = BN * BK / 4 / kThreads;   // vectors per thread and slab
    static_assert(BM * BK % (4 * kThreads) == 0 && BN * BK % (4 * kThreads) == 0, "slab loads");
    constexpr int PA = BM + 4, PW = BN + 4;
    __shared__ __align__(16) float As[2][BK][PA];
    __shared__ __align__(16) float Ws[2][BK][PW];
    umma::grid_trigger();
    umma::grid_wait();

    const int K = p.K, n = p.n;
    const long long M = p.M;
    const long long m0 = (long long)blockIdx.x * BM;   // row tiles innermost: CTAs side by side share the weight panel
    const int tiles_n = (n + (kPaired ? HN : BN) - 1) / (kPaired ? HN : BN);
    const int grp = blockIdx.y / tiles_n;                       // weight (or pair of weights) of this tile
    const int n0 = (blockIdx.y % tiles_n) * (kPaired ? HN : BN);
    const long long boff = (long long)blockIdx.z * p.a_batch;
    const float* a = p.a + boff;
    const T* w0 = (kPaired ? p.w[2 * grp] : p.w[grp]) + boff;
    const T* w1 = kPaired ? p.w[2 * grp + 1] : w0;
    const bool va = vec_ok(a, K_OUTER ? M : K), vw = vec_ok(w0, K_OUTER ? n : K) && vec_ok(w1, K_OUTER ? n : K);

    float4 ra[LA], rw[LW];
    auto fetch = [&](int k0) {
#pragma unroll
        for (int i = 0; i < LA; ++i) {
            const int idx = threadIdx.x + i * kThreads;
            if (K_OUTER) {   // four consecutive rows of one k
                const int kk = idx / (BM / 4), mm = idx % (BM / 4) * 4;
                const long long left = k0 + kk < K ? M - (m0 + mm) : 0;
                ra[i] = load4(a + (long long)(k0 + kk) * M + m0 + mm, left > 4 ? 4 : (int)left, va);
            } else {
                const int mm = idx / (BK / 4), kk = idx % (BK / 4) * 4;
                ra[i] = load4(a + (m0 + mm) * K + k0 + kk, m0 + mm < M ? K - (k0 + kk) : 0, va);
            }
        }
#pragma unroll
        for (int i = 0; i < LW; ++i) {
            const int idx = threadIdx.x + i * kThreads;
            if (K_OUTER) {
                const int kk = idx / (BN / 4), nn = idx % (BN / 4) * 4;
                rw[i] = load4(w0 + (long long)(k0 + kk) * n + n0 + nn, k0 + kk < K ? n - (n0 + nn) : 0, vw);
            } else {
                const int nn = idx / (BK / 4), kk = idx % (BK / 4) * 4;
                const int col = n0 + (kPaired ? nn % HN : nn);
                const T* w = kPaired && nn >= HN ? w1 : w0;
                rw[i] = load4(w + (long long)col * K + k0 + kk, col < n ? K - (k0 + kk) : 0, vw);
            }
        }
    };
    auto put = [&](int buf) {
#pragma unroll
        for (int i = 0; i < LA; ++i) {
            const int idx = threadIdx.x + i * kThreads;
            if (K_OUTER) {
                *reinterpret_cast<float4*>(&As[buf][idx / (BM / 4)][idx % (BM / 4) * 4]) = ra[i];
            } else {
                const int mm = idx / (BK / 4), kk = idx % (BK / 4) * 4;
                As[buf][kk][mm] = ra[i].x;
                As[buf][kk + 1][mm] = ra[i].y;
                As[buf][kk + 2][mm] = ra[i].z;
                As[buf][kk + 3][mm] = ra[i].w;
            }
        }
#pragma unroll
        for (int i = 0; i < LW; ++i) {
            const int idx = threadIdx.x + i * kThreads;
            if (K_OUTER) {
                *reinterpret_cast<float4*>(&Ws[buf][idx / (BN / 4)][idx % (BN / 4) * 4]) = rw[i];
            } else {
                const int nn = idx / (BK / 4), kk = idx % (BK / 4) * 4;
                Ws[buf][kk][nn] = rw[i].x;
                Ws[buf][kk + 1][nn] = rw[i].y;
                Ws[buf][kk + 2][nn] = rw[i].z;
                Ws[buf][kk + 3][nn] = rw[i].w;
            }
        }
    };

    constexpr int kGroupThreads = kThreads / G;
    const int g = threadIdx.x / kGroupThreads, gt = threadIdx.x % kGroupThreads;
    const int tx = gt % (BN / TN), ty = gt / (BN / TN);
    u64 acc[TM][TN2];   // pairs of columns
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN2; ++j) acc[i][j] = 0ull;

    fetch(0);
    put(0);
    __syncthreads();
    int buf = 0;
    for (int k0 = 0; k0 < K; k0 += BK, buf ^= 1) {
        if (k0 + BK < K) fetch(k0 + BK);
#pragma unroll
        for (int q = 0; q < 16; ++q) {
            const int kk = g * 16 + q;
            float av[TM];
            u64 wv[TN2];
#pragma unroll
            for (int hf = 0; hf < 2; ++hf) {
                if constexpr (TM2 == 4) {
                    const float4 v = *reinterpret_cast<const float4*>(&As[buf][kk][hf * HM + ty * 4]);
                    av[hf * 4] = v.x; av[hf * 4 + 1] = v.y; av[hf * 4 + 2] = v.z; av[hf * 4 + 3] = v.w;
                } else {
                    const float2 v = *reinterpret_cast<const float2*>(&As[buf][kk][hf * HM + ty * 2]);
                    av[hf * 2] = v.x; av[hf * 2 + 1] = v.y;
                }
                if constexpr (TN2 == 4) {
                    const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(&Ws[buf][kk][hf * HN + tx * 4]);
                    wv[hf * 2] = v.x; wv[hf * 2 + 1] = v.y;
                } else {
                    wv[hf] = *reinterpret_cast<const u64*>(&Ws[buf][kk][hf * HN + tx * 2]);
                }
            }
#pragma unroll
            for (int i = 0; i < TM; ++i) {
                const u64 ad = dup2(av[i]);
#pragma unroll
                for (int j = 0; j < TN2; ++j) fma2(acc[i][j], ad, wv[j]);
            }
        }
        if (k0 + BK < K) put(buf ^ 1);
        __syncthreads();
    }

    float v[TM][TN];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN2; ++j) {
            const float2 f = unpack2(acc[i][j]);
            v[i][2 * j] = f.x;
            v[i][2 * j + 1] = f.y;
        }
    if constexpr (G > 1) {   // the groups' partial sums, through the (now idle) slab buffers
        float* red = &As[0][0][0];
        static_assert(sizeof(As) >= sizeof(float) * (G - 1) * kGroupThreads * TM * TN, "reduction space");
        if (g > 0) {
#pragma unroll
            for (int i = 0; i < TM * TN; ++i) red[((g - 1) * TM * TN + i) * kGroupThreads + gt] = v[i / TN][i % TN];
        }
        __syncthreads();
        if (g > 0) return;
#pragma unroll
        for (int i = 0; i < TM * TN; ++i)
#pragma unroll
            for (int q = 0; q < G - 1; ++q) v[i / TN][i % TN] += red[(q * TM * TN + i) * kGroupThreads + gt];
    }

    epilogue<BM, BN, TM, TN, EPI, T>(p, v, m0, n0, grp, boff, tx, ty);
}

// ---------------------------------------------------------------- fp32 products on the tensor cores
// An fp32 value of 2^-110 and more is the sum of three bf16 values of 8 bits each, and a product of two such values the sum of the six
// of their products that are above 2^-26 of it (G. Henry, P. T. P. Tang, A. Heinecke, "Leveraging the bfloat16 Artificial Intelligence
// Datatype For Higher-Precision Computations", 2019). The products of the leading parts are summed by the tensor core over 64 k at a
// time, each such sum is added up in fp32 by the epilogue's threads; the other five, 2^-8 of them and less, have an accumulator of
// their own. (The tensor core cuts sums off instead of rounding them: in one accumulator over all of k the error grows to 1e-5 at
// k = 1536.) RMS error of 128 x 64 products against fp64, normal
// operands, FFMA in order / as pairs along k / this: k = 64 1.5e-7 / 1.1e-7 / 7.1e-8, 128 2.0e-7 / 1.5e-7 / 7.4e-8, 512 4.0e-7 /
// 2.9e-7 / 8.9e-8, 1536 7.0e-7 / 4.9e-7 / 1.2e-7; operands around 1: k = 128 1.7e-7 / 9.2e-8 / 3.3e-8.
// A tile with a value of 2^127 and more, an infinity or a NaN is computed once more on the FMA pipe. Where a product of two values may
// be beyond fp32's range (2^55 of one of them and more, for k below 2^17) its parts can be infinities of either sign: of a tile with
// such values the rows are computed once more where a sum of their warp is not finite. At the other end the parts miss up to 2^-134 of
// a value below 2^-110, and of products below 2^-126 more is cut off than an fma rounds away (31 x 2^-149 against 6.5, RMS, k = 512).
// Values that are zero or 2^-50 and more have neither. A tile with others, and with none of 2^55 and more, misses at most 2^-61 in a
// sum: its rows are computed once more where a sum of their warp is below 2^-34. (An addition and half a minimum per value: fp32 trunk
// block N = 128 683.6 -> 692 us. From the bf16 parts' remainder, which is zero where nothing is missed, 703; a minimum of all values
// first, and zeros told apart behind it, 696.)
//
// Tiles of 128 rows by BN columns; warps 0..7 convert (loads of the next k-block are on their way under this one's conversions),
// 8..15 the epilogue (two per 32 rows, thread = row), 16 issues the MMAs.
constexpr int kSplitThreads = 32 * 20;
// registers: the block is launched with 96 per thread; the issuing warpgroup gives up what the epilogue takes, which holds 64 sums
// beside the gates and residuals that are on their way
constexpr int kSplitRegsLaunch = 96, kSplitRegsIssue = 32, kSplitRegsConvert = 104, kSplitRegsEpi = 120;
static_assert(2 * kSplitRegsConvert + 2 * kSplitRegsEpi + kSplitRegsIssue <= 5 * kSplitRegsLaunch, "register split");
// kFinal: gate, residual and output in whole vectors of four columns (an absent one is aligned)
__host__ __device__ inline bool final_vec(const Args<float>& p) {
    const uintptr_t bits = reinterpret_cast<uintptr_t>(p.final_out) | reinterpret_cast<uintptr_t>(p.residual) | reinterpret_cast<uintptr_t>(p.gate);
    return (bits & 15) == 0 && (p.n & 3) == 0 && (p.map.inner_stride & 3) == 0 && (p.map.outer_stride & 3) == 0;
}

template <int BN>
struct SplitCfg {
    static constexpr int kAPlane = 128 * 128, kWPlane = BN * 128;   // bytes: 64 bf16 per row, 128-byte swizzle
    static constexpr int kStage = 3 * (kAPlane + kWPlane);
    static constexpr int kBars = 2 * kStage;
    static constexpr int kSmem = kBars + 256 + 1024;
    static_assert(kSmem <= 227 * 1024, "shared memory of a block");
    static constexpr int kTmem = 4 * BN;   // leading sums of even and odd k-blocks; small sums of even and odd tiles
};

// x0 and x1 less the halves of v, a pair of bf16 values
__device__ __forceinline__ void sub_pair(float& x0, float& x1, uint32_t v) {
    const uint32_t neg = v ^ 0x80008000u;
    asm("{\n.reg .b16 lo, hi;\nmov.b32 {lo, hi}, %2;\nadd.rn.f32.bf16 %0, lo, %0;\nadd.rn.f32.bf16 %1, hi, %1;\n}\n"
        : "+f"(x0), "+f"(x1)
        : "r"(neg));
}
// The largest of the magnitudes; NaN of a NaN
__device__ __forceinline__ float max_abs(float m, float x0, float x1) {
    asm("max.NaN.abs.f32 %0, %0, %1, %2;" : "+f"(m) : "f"(x0), "f"(x1));
    return m;
}
// Orders the magnitudes of values, with zero behind all others
__host__ __device__ constexpr uint32_t nonzero_order(uint32_t bits) { return bits + bits - 1u; }
// Eight values into three planes of a stage, at d; their largest magnitude, and the order of the smallest that is not zero
__device__ __forceinline__ void split8(float (&x)[8], uint8_t* d, int plane, float& largest, uint32_t& smallest) {
    uint32_t u[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        largest = max_abs(largest, x[2 * i], x[2 * i + 1]);
        smallest = __vimin3_u32(smallest, nonzero_order(__float_as_uint(x[2 * i])), nonzero_order(__float_as_uint(x[2 * i + 1])));
    }
#pragma unroll
    for (int q = 0; q < 3; ++q) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            u[i] = pack_bf16x2(x[2 * i], x[2 * i + 1]);
            if (q < 2) sub_pair(x[2 * i], x[2 * i + 1], u[i]);
        }
        *reinterpret_cast<uint4*>(d + q * plane) = make_uint4(u[0], u[1], u[2], u[3]);
    }
}

// eight consecutive values, `n` of which exist
__device__ __forceinline__ void load8(const float* p, int n, bool vec, float (&x)[8]) {
    const float4 a = load4(p, n, vec), b = load4(p + 4, n - 4, vec);
    x[0] = a.x; x[1] = a.y; x[2] = a.z; x[3] = a.w;
    x[4] = b.x; x[5] = b.y; x[6] = b.z; x[7] = b.w;
}
__device__ __forceinline__ void load8(const float* p, int n, float (&x)[8]) {   // n a multiple of four, p on 16 bytes
    float4 a = make_float4(0.f, 0.f, 0.f, 0.f), b = a;
    if (n >= 4) a = reinterpret_cast<const float4*>(p)[0];
    if (n >= 8) b = reinterpret_cast<const float4*>(p)[1];
    x[0] = a.x; x[1] = a.y; x[2] = a.z; x[3] = a.w;
    x[4] = b.x; x[5] = b.y; x[6] = b.z; x[7] = b.w;
}
__device__ __forceinline__ void store8(float* p, const float (&o)[8], int n) {   // the first n
    if (n >= 8 && umma::aligned32(p)) {
        uint32_t u[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) u[i] = __float_as_uint(o[i]);
        umma::stg256(p, u);
    } else if (n >= 8 && (reinterpret_cast<uintptr_t>(p) & 15) == 0) {
        reinterpret_cast<float4*>(p)[0] = make_float4(o[0], o[1], o[2], o[3]);
        reinterpret_cast<float4*>(p)[1] = make_float4(o[4], o[5], o[6], o[7]);
    } else {
#pragma unroll
        for (int i = 0; i < 8; ++i)
            if (i < n) p[i] = o[i];
    }
}

// kWhole: k in whole k-blocks, and operands in whole vectors along it. kShort (kFinal): at most two k-blocks, and gate, residual and
// output in whole vectors (an instantiation of its own: both forms in one kernel spilled 1100 bytes of registers)
template <int BN, int EPI, bool K_OUTER, bool kWhole, bool kShort>
__global__ void __launch_bounds__(kSplitThreads, 1)
gemm_split_kernel(const Args<float> p, int batch, int groups, int* status) {
    using namespace umma;
    using C = SplitCfg<BN>;
    constexpr bool kPaired = EPI == kGatedPlanes || EPI == kSwiglu;
    constexpr int HN = BN / 2, kCols = kPaired ? HN : BN;   // columns of the result per tile
    constexpr int kRun = BN / 4;                            // an epilogue thread's columns: kRun in each half of the tile
    constexpr int kItemsA = 4, kItemsW = BN / 32;           // vectors of eight k per converting thread and k-block
    constexpr int kKid = 20;
    extern __shared__ uint8_t smem_raw[];
    const uint32_t sbase = (smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t* gbase = smem_raw + (sbase - smem_u32(smem_raw));
    const uint32_t bars = sbase + C::kBars;
    auto full = [&](int s) { return bars + 8u * s; };             // a stage is converted
    auto empty = [&](int s) { return bars + 8u * (2 + s); };      // its products are done
    auto main_full = [&](int s) { return bars + 8u * (4 + s); };  // leading sums of a k-block
    auto main_free = [&](int s) { return bars + 8u * (6 + s); };
    auto small_full = [&](int s) { return bars + 8u * (8 + s); };   // small sums of a tile
    auto small_free = [&](int s) { return bars + 8u * (10 + s); };
    volatile uint32_t* tmem_ptr = reinterpret_cast<volatile uint32_t*>(gbase + C::kBars + 96);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(gbase + C::kBars + 104);
    // marks of tiles: [4] tile numbers (of this CTA, from 1). Values that the parts do not hold; large and small ones, whose sums are to
    // be looked at
    volatile int* special = reinterpret_cast<volatile int*>(gbase + C::kBars + 112);
    volatile int *large = special + 4, *small = special + 8;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int K = p.K, n = p.n;
    const long long M = p.M;
    const int num_kb = (K + 63) / 64;
    const uint32_t row_tiles = (uint32_t)((M + 127) / 128), col_tiles = (uint32_t)(n + kCols - 1) / kCols;
    const uint32_t num_tiles = row_tiles * col_tiles * (uint32_t)(groups * batch);   // (below 2^31)
    struct Tile {
        long long m0, boff;
        int grp, n0;
    };
    auto tile_of = [&](uint32_t t) {   // row tiles innermost: CTAs that run at the same time share the weights
        Tile c;
        uint32_t q = t / row_tiles;
        c.m0 = (t - q * row_tiles) * 128LL;
        const uint32_t q2 = q / col_tiles;
        c.n0 = (int)(q - q2 * col_tiles) * kCols;
        q = q2 / (uint32_t)groups;
        c.grp = (int)(q2 - q * groups);
        c.boff = q * p.a_batch;
        return c;
    };
    auto weight_row = [&](const Tile& c, int j, int& col) {   // row j of the weight tile: its matrix, and its row there
        col = c.n0 + (kPaired ? j % HN : j);
        return kPaired ? (j < HN ? p.w[2 * c.grp] : p.w[2 * c.grp + 1]) : p.w[c.grp] + c.boff;
    };

    if (threadIdx.x == 0) {
        for (int s = 0; s < 2; ++s) {
            mbar_init(full(s), 8);
            mbar_init(empty(s), 1);
            mbar_init(main_full(s), 1);
            mbar_init(main_free(s), 8);
            mbar_init(small_full(s), 1);
            mbar_init(small_free(s), 8);
        }
        for (int i = 0; i < 12; ++i) special[i] = 0;
        *abort_flag = 0;
        mbar_fence_init();
    }
    if (warp == 16) {
        tmem_alloc(smem_u32((const void*)tmem_ptr), C::kTmem);
        tmem_relinquish();
    }
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem_base = *tmem_ptr;
    grid_trigger();
    if (warp >= 8) grid_wait();

    if (warp < 8) {
        // ---------------------------------------------------------------- conversion
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kSplitRegsConvert));
        const long long step_a = K_OUTER ? M : 1, step_w = K_OUTER ? n : 1;   // from one k to the next
        // the tile's operands, and where the thread's vectors of the first k-block lie; rows past the end: the last one
        const float *a0 = nullptr, *w0 = nullptr, *w1 = nullptr;
        uint32_t oa[kItemsA] = {}, ow[kItemsW] = {};
        static_assert(!kPaired || (!K_OUTER && kItemsW % 2 == 0), "the second half of the vectors is of the second weight");
        bool va = kWhole, vw = kWhole;
        float xa[kItemsA][8], xw[kItemsW][8];
        // a k-block's vector v: rows of k next to one another: eight lanes per row; K_OUTER: a row per lane
        auto row_of = [&](int v, int rows) { return K_OUTER ? v % rows : v >> 3; };
        auto chunk_of = [&](int v, int rows) { return K_OUTER ? v / rows : v & 7; };
        auto fetch = [&](const float* src, long long step, bool vec, int k, float (&x)[8]) {
            if constexpr (K_OUTER) {
#pragma unroll
                for (int e = 0; e < 8; ++e) x[e] = kWhole || k + e < K ? src[e * step] : 0.f;
            } else if constexpr (kWhole) {
                const float4 u = reinterpret_cast<const float4*>(src)[0], w = reinterpret_cast<const float4*>(src)[1];
                x[0] = u.x; x[1] = u.y; x[2] = u.z; x[3] = u.w;
                x[4] = w.x; x[5] = w.y; x[6] = w.z; x[7] = w.w;
            } else {
                load8(src, K - k, vec, x);
            }
        };
        auto fetch_a = [&](int i, int kb) {
            const int v = threadIdx.x + i * 256;
            fetch(a0 + kb * 64 * step_a + oa[i], step_a, va, kb * 64 + chunk_of(v, 128) * 8, xa[i]);
        };
        auto fetch_w = [&](int i, int kb) {
            const int v = threadIdx.x + i * 256;
            fetch((kPaired && i >= kItemsW / 2 ? w1 : w0) + kb * 64 * step_w + ow[i], step_w, vw, kb * 64 + chunk_of(v, BN) * 8, xw[i]);
        };
        auto open = [&](uint32_t t) {
            const Tile c = tile_of(t);
            int col;
            a0 = p.a + c.boff + (K_OUTER ? c.m0 : c.m0 * K);
            w0 = weight_row(c, 0, col);
            w1 = weight_row(c, BN - 1, col);
            if (!kWhole && !K_OUTER) {
                va = vec_ok(a0, K);
                vw = vec_ok(w0, K) && vec_ok(w1, K);
            }
            const uint32_t last_row = (uint32_t)min(M - 1 - c.m0, 127LL);
#pragma unroll
            for (int i = 0; i < kItemsA; ++i) {
                const int v = threadIdx.x + i * 256;
                const uint32_t r = min((uint32_t)row_of(v, 128), last_row);
                oa[i] = r * (K_OUTER ? 1u : (uint32_t)K) + chunk_of(v, 128) * 8 * (uint32_t)step_a;
            }
#pragma unroll
            for (int i = 0; i < kItemsW; ++i) {
                const int v = threadIdx.x + i * 256;
                weight_row(c, row_of(v, BN), col);
                ow[i] = (uint32_t)min(col, n - 1) * (K_OUTER ? 1u : (uint32_t)K) + chunk_of(v, BN) * 8 * (uint32_t)step_w;
            }
        };
        bool ok = true;
        uint32_t it = 0;
        int seq = 0;
        open(blockIdx.x);
        if (p.a_batch != 0) grid_wait();   // (batched products: no weights)
#pragma unroll
        for (int i = 0; i < kItemsW; ++i) fetch_w(i, 0);
        if (p.a_batch == 0) grid_wait();
#pragma unroll
        for (int i = 0; i < kItemsA; ++i) fetch_a(i, 0);
        for (uint32_t t = blockIdx.x; t < num_tiles && ok; t += gridDim.x, ++seq) {
            float largest = 0.f;
            uint32_t smallest = ~0u;
            for (int kb = 0; kb < num_kb; ++kb, ++it) {
                const int s = it & 1;
                if (!mbar_wait(empty(s), ((it >> 1) & 1u) ^ 1u, abort_flag)) {
                    if (lane == 0) report_wait_failure(status, abort_flag, kKid, 1);
                    ok = false;
                    break;
                }
                uint8_t* const stage = gbase + s * C::kStage;
                const bool last = kb + 1 == num_kb, more = !last || t + gridDim.x < num_tiles;
                const int next = last ? 0 : kb + 1;
                if (last && more) open(t + gridDim.x);
#pragma unroll
                for (int i = 0; i < kItemsA; ++i) {
                    const int v = threadIdx.x + i * 256;
                    split8(xa[i], stage + sw128_offset(row_of(v, 128), chunk_of(v, 128) * 8), C::kAPlane, largest, smallest);
                    if (more) fetch_a(i, next);
                }
#pragma unroll
                for (int i = 0; i < kItemsW; ++i) {
                    const int v = threadIdx.x + i * 256;
                    split8(xw[i], stage + 3 * C::kAPlane + sw128_offset(row_of(v, BN), chunk_of(v, BN) * 8), C::kWPlane, largest, smallest);
                    if (more) fetch_w(i, next);
                }
                if (!(largest < 0x1p55f)) {
                    large[seq & 3] = seq + 1;
                    if (!(largest < 0x1p127f)) special[seq & 3] = seq + 1;
                }
                if (smallest < nonzero_order(0x26800000u)) small[seq & 3] = seq + 1;   // 2^-50
                fence_proxy_async_smem();
                __syncwarp();
                if (lane == 0) mbar_arrive(full(s));
            }
        }
    } else if (warp >= 16) {
        // ---------------------------------------------------------------- MMA issuer
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kSplitRegsIssue));
        if (warp == 16 && elect_one()) {
            constexpr uint32_t idesc = idesc_bf16_f32(128, BN);
            uint32_t it = 0, tc = 0;
            bool ok = true;
            for (uint32_t t = blockIdx.x; t < num_tiles && ok; t += gridDim.x, ++tc) {
                const uint32_t d_small = tmem_base + 2 * BN + (tc & 1u) * BN;
                for (int kb = 0; kb < num_kb; ++kb, ++it) {
                    const int s = it & 1;
                    if (!mbar_wait(full(s), (it >> 1) & 1u, abort_flag) || !mbar_wait(main_free(s), ((it >> 1) & 1u) ^ 1u, abort_flag) ||
                        (kb == 0 && !mbar_wait(small_free(tc & 1u), ((tc >> 1) & 1u) ^ 1u, abort_flag))) {
                        report_wait_failure(status, abort_flag, kKid, 2);
                        ok = false;
                        break;
                    }
                    tc_fence_after_sync();
                    const uint32_t sa = sbase + s * C::kStage, sw = sa + 3 * C::kAPlane;
                    auto products = [&](int pa, int pw, uint32_t d, bool fresh) {
                        const uint64_t ad = smem_desc_k_sw128(sa + pa * C::kAPlane), wd = smem_desc_k_sw128(sw + pw * C::kWPlane);
#pragma unroll
                        for (int k4 = 0; k4 < 4; ++k4) mma_bf16(d, ad + 2u * k4, wd + 2u * k4, idesc, fresh && k4 == 0 ? 0u : 1u);
                    };
                    products(0, 0, tmem_base + s * BN, true);
                    mma_commit(main_full(s));
                    products(2, 0, d_small, kb == 0);
                    products(1, 1, d_small, false);
                    products(0, 2, d_small, false);
                    products(1, 0, d_small, false);
                    products(0, 1, d_small, false);
                    mma_commit(empty(s));
                }
                if (ok) mma_commit(small_full(tc & 1u));
            }
        }
    } else {
        // ---------------------------------------------------------------- epilogue: thread = row, kRun columns of each half
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kSplitRegsEpi));
        const int quad = warp & 3, part = (warp - 8) >> 2;
        const uint32_t taddr = tmem_base + ((uint32_t)(quad * 32) << 16) + part * kRun;
        uint32_t it = 0, tc = 0;
        for (uint32_t t = blockIdx.x; t < num_tiles; t += gridDim.x, ++tc) {
            __syncwarp();   // (lanes part where rows end, and in redo)
            const Tile c = tile_of(t);
            const long long r = c.m0 + quad * 32 + lane;
            const bool live = r < M;
            const float mk = (EPI == kGatedPlanes || EPI == kFinal) && p.mask && live ? p.mask[r] : 1.0f;
            const uint32_t t_small = 2 * BN + (tc & 1u) * BN;
            auto col_of = [&](int e) { return c.n0 + part * kRun + (e < kRun ? e : HN + e - kRun); };
            auto add16 = [&](uint32_t col, float (&v)[16]) {
                uint32_t u[16];
                tmem_ld16(taddr + col, u);
                tmem_ld_wait();
#pragma unroll
                for (int e = 0; e < 16; ++e) v[e] += __uint_as_float(u[e]);
            };
            auto wait_main = [&] {
                if (mbar_wait(main_full(it & 1), (it >> 1) & 1u, abort_flag)) return true;
                if (lane == 0) report_wait_failure(status, abort_flag, kKid, 3);
                return false;
            };
            auto wait_small = [&] {
                if (mbar_wait(small_full(tc & 1u), (tc >> 1) & 1u, abort_flag)) return true;
                if (lane == 0) report_wait_failure(status, abort_flag, kKid, 4);
                return false;
            };
            auto free_main = [&](uint32_t s) {
                tc_fence_before_sync();
                __syncwarp();
                if (lane == 0) mbar_arrive(main_free(s));
            };
            // one value of the result from its product (and that of the paired weight)
            auto result = [&](int e, float x, float y) {
                const int col = col_of(e);
                if (!live || col >= n) return;
                if constexpr (EPI == kGatedPlanes) {
                    p.out[c.grp][(long long)col * M + r] = mk * sigmoid_acc(y) * x;
                } else if constexpr (EPI == kSwiglu) {
                    p.out[0][r * n + col] = x * sigmoid_acc(x) * y;
                } else if constexpr (EPI == kFinal) {
                    if (p.gate) x *= sigmoid_acc(p.gate[r * n + col]);
                    if (p.mask) x *= mk;
                    const long long at = row_offset(p.map, r) + col;
                    p.final_out[at] = x + (p.residual ? p.residual[at] : 0.f);
                } else {
                    p.out[c.grp][c.boff + r * n + col] = x + (p.bias[c.grp] ? p.bias[c.grp][col] : 0.f);
                }
            };
            struct Marks {
                bool all, look;   // compute the tile once more; look at its sums
                float least;      // the smallest magnitude of a sound one
            };
            auto marks = [&] {
                const int id = (int)tc + 1;
                const bool l = large[tc & 3] == id, s = small[tc & 3] == id;
                return Marks{special[tc & 3] == id || (l && s), l || s, s ? 0x1p-34f : 0.f};
            };
            auto sound = [](const float (&v)[16], float least) {
                float chk = 0.f, mn = v[0];
#pragma unroll
                for (int e = 0; e < 16; ++e) {
                    chk = fmaf(v[e], 0.f, chk);
                    mn = fminf(fabsf(mn), fabsf(v[e]));
                }
                return chk == 0.f && fabsf(mn) >= least;
            };
            // columns of a tile that the split does not take: their products on the FMA pipe
            auto redo = [&](int first, int end) {
                auto dot = [&](int e) {
                    int col;
                    const float* w = weight_row(c, part * kRun + (e < kRun ? e : HN + e - kRun), col);
                    float x = 0.f;
                    if (live && col < n)
                        for (int k = 0; k < K; ++k)
                            x = K_OUTER ? fmaf(p.a[c.boff + (long long)k * M + r], w[(long long)k * n + col], x)
                                        : fmaf(p.a[c.boff + r * K + k], w[(long long)col * K + k], x);
                    return x;
                };
#pragma unroll 1
                for (int e = first; e < end; ++e) result(e, dot(e), kPaired ? dot(kRun + e) : 0.f);
            };
            // all of the thread's columns, 16 by 16. The marks are read ahead of the arrivals (of one k-block each, the tile after next
            // could otherwise be multiplied and the one behind it, whose marks take the same place, be converted)
            auto sum_up = [&](float (&v)[2 * kRun / 16][16], bool& again) {
                auto add = [&](uint32_t col) {
#pragma unroll
                    for (int e0 = 0; e0 < 2 * kRun; e0 += 16) add16(col + (e0 < kRun ? e0 : HN + e0 - kRun), v[e0 / 16]);
                };
#pragma unroll
                for (int e = 0; e < 2 * kRun; ++e) v[e / 16][e % 16] = 0.f;
                for (int kb = 0; kb < num_kb; ++kb, ++it) {
                    if (!wait_main()) return false;
                    tc_fence_after_sync();
                    add((it & 1) * BN);
                    free_main(it & 1);
                }
                if (!wait_small()) return false;
                const Marks m = marks();
                again = m.all;
                tc_fence_after_sync();
                add(t_small);
                tc_fence_before_sync();
                __syncwarp();
                if (lane == 0) mbar_arrive(small_free(tc & 1u));
                if (m.look) {
#pragma unroll
                    for (int q = 0; q < 2 * kRun / 16; ++q) again |= !sound(v[q], m.least);
                    again = __any_sync(0xffffffffu, again);
                }
                return true;
            };
            if constexpr (EPI == kFinal) {
                const long long off = live ? row_offset(p.map, r) : 0;
                const bool vec = kShort || final_vec(p);
                // Gates and residuals of 16 columns from e0 on: ahead of the stores before them, which may be to the residual's own rows
                struct Ahead {
                    float gate[2][8], residual[2][8];
                };
                auto fetch = [&](int e0, Ahead& a) {
#pragma unroll
                    for (int q = 0; q < 2; ++q) {
                        const int col = col_of(e0 + 8 * q), left = live ? n - col : 0;
                        if (p.gate) load8(p.gate + r * n + col, left, a.gate[q]);
                        if (p.residual) load8(p.residual + off + col, left, a.residual[q]);
                    }
                };
                auto finish = [&](float (&v)[16], const Ahead& a) {
#pragma unroll
                    for (int j = 0; j < 16; ++j) {
                        if (p.gate) v[j] *= sigmoid_acc(a.gate[j >> 3][j & 7]);
                        if (p.mask) v[j] *= mk;
                        if (p.residual) v[j] += a.residual[j >> 3][j & 7];
                    }
                };
                auto put = [&](int e0, const float (&v)[16]) {
#pragma unroll
                    for (int q = 0; q < 2; ++q) {
                        const int col = col_of(e0 + 8 * q);
                        float o[8];
#pragma unroll
                        for (int j = 0; j < 8; ++j) o[j] = v[8 * q + j];
                        if (live) store8(p.final_out + off + col, o, n - col);
                    }
                };
                if constexpr (kShort) {
                    // both leading sums stay where they are until they are added up, 16 columns at a time
                    Ahead a[2];
                    fetch(0, a[0]);
                    fetch(16, a[1]);
                    bool ok = wait_main();
                    const uint32_t s0 = it++ & 1;
                    if (ok && num_kb == 2) {
                        ok = wait_main();
                        ++it;
                    }
                    if (!ok || !wait_small()) break;
                    tc_fence_after_sync();
                    const Marks m = marks();
                    uint32_t again = 0;   // a bit per 16 columns
#pragma unroll
                    for (int e0 = 0; e0 < 2 * kRun; e0 += 16) {
                        const uint32_t at = e0 < kRun ? e0 : HN + e0 - kRun;
                        float v[16];
#pragma unroll
                        for (int e = 0; e < 16; ++e) v[e] = 0.f;
                        add16(s0 * BN + at, v);
                        if (num_kb == 2) add16((s0 ^ 1u) * BN + at, v);
                        add16(t_small + at, v);
                        if (e0 + 16 == 2 * kRun) {
                            free_main(s0);
                            if (num_kb == 2) free_main(s0 ^ 1u);
                            if (lane == 0) mbar_arrive(small_free(tc & 1u));
                        }
                        const bool bad = m.look && __any_sync(0xffffffffu, m.all || !sound(v, m.least));
                        finish(v, a[e0 / 16 % 2]);
                        if (e0 + 32 < 2 * kRun) fetch(e0 + 32, a[e0 / 16 % 2]);
                        if (bad) again |= 1u << (e0 / 16);
                        else put(e0, v);
                    }
#pragma unroll 1
                    for (int q = 0; again >> q; ++q)
                        if (again >> q & 1u) redo(16 * q, 16 * q + 16);
                } else {
                    float v[2 * kRun / 16][16];
                    bool again;
                    if (!sum_up(v, again)) break;
                    if (again) {
                        redo(0, 2 * kRun);
                    } else if (!vec) {
#pragma unroll
                        for (int e = 0; e < 2 * kRun; ++e) result(e, v[e / 16][e % 16], 0.f);
                    } else {
                        Ahead a;
                        fetch(0, a);
#pragma unroll
                        for (int e0 = 0; e0 < 2 * kRun; e0 += 16) {
                            finish(v[e0 / 16], a);
                            if (e0 + 16 < 2 * kRun) fetch(e0 + 16, a);
                            put(e0, v[e0 / 16]);
                        }
                    }
                }
            } else {
                float v[2 * kRun / 16][16];
                bool again;
                if (!sum_up(v, again)) break;
                if (again) {
                    redo(0, kPaired ? kRun : 2 * kRun);
                    continue;
                }
                if (!live) continue;
                auto at = [&](int e) { return v[e / 16][e % 16]; };
                if constexpr (EPI == kGatedPlanes) {
                    float* out = p.out[c.grp];
#pragma unroll
                    for (int j = 0; j < kRun; ++j)
                        if (col_of(j) < n) out[(long long)col_of(j) * M + r] = mk * sigmoid_acc(at(kRun + j)) * at(j);
                } else {
#pragma unroll
                    for (int e0 = 0; e0 < (EPI == kSwiglu ? kRun : 2 * kRun); e0 += 8) {
                        const int col = col_of(e0);
                        float o[8];
#pragma unroll
                        for (int j = 0; j < 8; ++j) {
                            const float x = at(e0 + j);
                            if constexpr (EPI == kSwiglu) o[j] = x * sigmoid_acc(x) * at(kRun + e0 + j);
                            else o[j] = x + (p.bias[c.grp] && col + j < n ? p.bias[c.grp][col + j] : 0.f);
                        }
                        store8((EPI == kSwiglu ? p.out[0] : p.out[c.grp] + c.boff) + r * n + col, o, n - col);
                    }
                }
            }
        }
    }

    tc_fence_before_sync();
    __syncthreads();
    if (warp == 16) {
        tc_fence_after_sync();
        tmem_dealloc(tmem_base, C::kTmem);
    }
}

template <int BN, int EPI, bool K_OUTER, bool kWhole, bool kShort = false>
int launch_split(const Args<float>& p, int groups, int batch, cudaStream_t st) {
    using C = SplitCfg<BN>;
    constexpr int kCols = EPI == kGatedPlanes || EPI == kSwiglu ? BN / 2 : BN;
    static PerDeviceOnce configured;
    if (!configured.done()) {
        cudaFuncAttributes fa;   // a block launched with fewer registers would wait for the split for good
        OF3_CUDA_CHECK(cudaFuncGetAttributes(&fa, gemm_split_kernel<BN, EPI, K_OUTER, kWhole, kShort>));
        OF3_REQUIRE(fa.numRegs == kSplitRegsLaunch, OF3_ERR_DRIVER, "the split product is built with %d registers, not %d", fa.numRegs,
                    kSplitRegsLaunch);
        OF3_CUDA_CHECK(cudaFuncSetAttribute(gemm_split_kernel<BN, EPI, K_OUTER, kWhole, kShort>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                            C::kSmem));
        configured.mark();
    }
    const long long tiles = (p.M + 127) / 128 * ((p.n + kCols - 1) / kCols) * groups * batch;
    OF3_REQUIRE(tiles < (1LL << 31), OF3_ERR_SHAPE, "gemm: %lld rows, %d columns, batch %d", p.M, p.n, batch);
    LaunchScope scope(20, st);
    OF3_CUDA_CHECK(launch_chained(gemm_split_kernel<BN, EPI, K_OUTER, kWhole, kShort>, (unsigned)(tiles < sm_count() ? tiles : sm_count()),
                                  kSplitThreads, C::kSmem, st, p, batch, groups, device_status_ptr()));
    return OF3_OK;
}

template <int EPI, bool K_OUTER, typename T>
int launch(Args<T> p, int groups, int batch, cudaStream_t st) {
    constexpr bool kPaired = EPI == kGatedPlanes || EPI == kSwiglu;
    if (p.M <= 0 || p.n <= 0 || batch <= 0) return OF3_OK;
    const long long M = p.M;
    auto tiles = [&](int bm, int bn) {
        return ((M + bm - 1) / bm) * ((p.n + bn - 1) / bn) * groups * (long long)batch;
    };
    if constexpr (std::is_same<T, float>::value) {
        // Tensor cores once the small tiles of the FMA kernel would come in more than four waves. Device time, us, FMA / tensor, cold:
        // 576 rows: 4 x 128 columns 7.8 / 11.9; 2304 rows: 128 columns 8.0 / 12.4 (two waves), 4 x 128 22.3 / 12.5 (eight)
        // (silu * up of short k later, for the sake of blocks: trunk of 25 tokens (k = 128, 640 tiles) 310.3 / 317.6, 26 (704) 305.8 / 309.0,
        // template of 49 (k = 64, 608) 350 / 352, but 51 (656) 348 / 344. Of longer k not: a transition alone of 192 channels, 445 rows,
        // 51.5 / 33.8; 256, 317 50.7 / 39.3; 384, 200 90.7 / 54.1; 768, 221 125.2 / 108.7)
        if (5 * tiles(32, kPaired ? 16 : 32) > (EPI == kSwiglu && p.K <= 128 ? 24 : 20) * sm_count() && p.K < 1 << 17) {
            bool whole = p.K % 64 == 0;
            if (!K_OUTER) {
                whole = whole && (reinterpret_cast<uintptr_t>(p.a) & 15) == 0 && (p.a_batch & 3) == 0;
                for (int i = 0; i < groups * (kPaired ? 2 : 1); ++i) whole = whole && (reinterpret_cast<uintptr_t>(p.w[i]) & 15) == 0;
            }
            if constexpr (EPI == kFinal) {
                if (whole && p.K <= 128 && final_vec(p)) return launch_split<128, EPI, K_OUTER, true, true>(p, groups, batch, st);
            }
            return whole ? launch_split<128, EPI, K_OUTER, true>(p, groups, batch, st)
                         : launch_split<128, EPI, K_OUTER, false>(p, groups, batch, st);
        }
    }
    // Otherwise small tiles; with bf16 weights, large ones once they give every SM at least one
    const bool large = !std::is_same<T, float>::value && tiles(128, kPaired ? 32 : 64) >= sm_count();
    const int bm = large ? 128 : 32, bn = large ? (kPaired ? 32 : 64) : (kPaired ? 16 : 32);
    const long long gx = (M + bm - 1) / bm, gy = (long long)((p.n + bn - 1) / bn) * groups;
    OF3_REQUIRE(batch <= 65535 && gy <= 65535 && gx < (1LL << 31), OF3_ERR_SHAPE, "gemm: %lld rows, %d columns, batch %d",
                M, p.n, batch);
    const dim3 grid((unsigned)gx, (unsigned)gy, batch);
    LaunchScope scope(20, st);
    if constexpr (!std::is_same<T, float>::value) {
        if (large) {
            OF3_CUDA_CHECK(launch_chained(gemm_kernel<128, 64, 8, 8, 1, EPI, K_OUTER, T>, grid, 128, 0, st, p));
            return OF3_OK;
        }
    }
    OF3_CUDA_CHECK(launch_chained(gemm_kernel<32, 32, 4, 4, 4, EPI, K_OUTER, T>, grid, 256, 0, st, p));
    return OF3_OK;
}

}  // namespace

template <typename T>
int linear_multi(const float* x, int count, const T* const* w, const T* const* bias, float* const* out, long long rows,
                 int n, int k, cudaStream_t st) {
    Args<T> p = {};
    p.a = x;
    for (int i = 0; i < count; ++i) {
        p.w[i] = w[i];
        p.bias[i] = bias ? bias[i] : nullptr;
        p.out[i] = out[i];
    }
    p.M = rows;
    p.n = n;
    p.K = k;
    return launch<kStore, false, T>(p, count, 1, st);
}
template <typename T>
int linear_gated_planes(const float* x, int count, const T* const* wp, const T* const* wg, const T* mask,
                        float* const* out, long long rows, int n, int k, cudaStream_t st) {
    Args<T> p = {};
    p.a = x;
    for (int i = 0; i < count; ++i) {
        p.w[2 * i] = wp[i];
        p.w[2 * i + 1] = wg[i];
        p.out[i] = out[i];
    }
    p.mask = mask;
    p.M = rows;
    p.n = n;
    p.K = k;
    return launch<kGatedPlanes, false, T>(p, count, 1, st);
}
template <typename T>
int linear_swiglu(const float* x, const T* wa, const T* wb, float* h, long long rows, int n, int k, cudaStream_t st) {
    Args<T> p = {};
    p.a = x;
    p.w[0] = wa;
    p.w[1] = wb;
    p.out[0] = h;
    p.M = rows;
    p.n = n;
    p.K = k;
    return launch<kSwiglu, false, T>(p, 1, 1, st);
}
template <typename T>
int linear_final(const float* x, const T* w, const float* gate, const T* residual, const T* mask, T* out, long long rows,
                 int n, int k, RowMap map, cudaStream_t st) {
    Args<T> p = {};
    p.a = x;
    p.w[0] = w;
    p.gate = gate;
    p.residual = residual;
    p.mask = mask;
    p.final_out = out;
    p.map = map;
    p.M = rows;
    p.n = n;
    p.K = k;
    return launch<kFinal, false, T>(p, 1, 1, st);
}
int contract_planes(const float* a, const float* b, float* x, int batch, int N, long long a_batch, bool k_outer,
                    cudaStream_t st) {
    for (int c0 = 0; c0 < batch; c0 += 32768) {
        const int nb = batch - c0 < 32768 ? batch - c0 : 32768;
        Args<float> p = {};
        p.a = a + c0 * a_batch;
        p.w[0] = b + c0 * a_batch;
        p.out[0] = x + c0 * a_batch;
        p.M = N;
        p.n = N;
        p.K = N;
        p.a_batch = a_batch;
        const int rc = k_outer ? launch<kStore, true, float>(p, 1, nb, st) : launch<kStore, false, float>(p, 1, nb, st);
        if (rc) return rc;
    }
    return OF3_OK;
}

#define INSTANTIATE(T)                                                                                             \
    template int linear_multi<T>(const float*, int, const T* const*, const T* const*, float* const*, long long, int, \
                                 int, cudaStream_t);                                                               \
    template int linear_gated_planes<T>(const float*, int, const T* const*, const T* const*, const T*, float* const*, \
                                        long long, int, int, cudaStream_t);                                        \
    template int linear_swiglu<T>(const float*, const T*, const T*, float*, long long, int, int, cudaStream_t);     \
    template int linear_final<T>(const float*, const T*, const float*, const T*, const T*, T*, long long, int, int, \
                                 RowMap, cudaStream_t);
INSTANTIATE(float)
INSTANTIATE(__nv_bfloat16)

}  // namespace generic
}  // namespace of3
