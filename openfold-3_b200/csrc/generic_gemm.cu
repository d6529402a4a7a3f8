// fp32 GEMMs of the shape-generic family on the FMA pipe, with the element-wise step that follows in the epilogue.
//
// Bound: 128 fp32 FMA per SM and clock (75 TFLOP/s); the operands of these layers sit in L2. Tiles of 128 x 64 with 8 x 8
// products per thread read 16 values from shared memory per 64 FMA (packed fma.f32x2: half the issue slots), the next
// k-slab is in registers while this one is multiplied. Layers with few rows take 32 x 32 tiles whose k-slab is split over
// four groups of threads (the chain over k = 1536 on 24 large tiles is what such a layer waits for).
// The 64 x 64 kernel with 4 x 4 products, scalar shared-memory reads and separate element-wise kernels ran the 128-token
// trunk block at 8.5 TFLOP/s.
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

__device__ __forceinline__ void store4(float* p, const float (&o)[4]) {
    *reinterpret_cast<float4*>(p) = make_float4(o[0], o[1], o[2], o[3]);
}
__device__ __forceinline__ void store4(__nv_bfloat16* p, const float (&o)[4]) {
    *reinterpret_cast<uint2*>(p) = make_uint2(pack_bf16x2(o[0], o[1]), pack_bf16x2(o[2], o[3]));
}
__device__ __forceinline__ void cp_async16(void* dst, const void* src, bool exists) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(umma::smem_u32(dst)), "l"(src), "r"(exists ? 16 : 0)
                 : "memory");
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

// The same product for fp32 operands in whole 16-byte vectors along k: slabs by cp.async as they lie, a thread's 8 x 8
// products in pairs (even k, odd k), whose halves are added at the end: operands come from shared memory as the pairs that
// fma.f32x2 takes, none is duplicated in registers. A row of a slab lies at the place that lets the lanes of a load, which
// own rows 4 apart, hit neighbouring ones: pitch 20 floats, no bank conflict. Two blocks per SM, since a thread holds 128
// sums: for the plain and the final epilogue the better kernel (one fp32 trunk block at N = 128: 1011 -> 978 us), for the
// paired ones, whose exponentials three blocks of the kernel above overlap with products, the worse (swiglu 107 -> 119 us).
// Both read 16 values per 64 products from shared memory, whose bandwidth (16 bytes x 32 lanes in four clocks) that takes
// whole; 16 x 8 products per thread leave two blocks per SM and are slower (122 us).
template <int EPI>
__global__ void __launch_bounds__(128, 2) gemm_pairs_kernel(const Args<float> p) {
    constexpr int BM = 128, BN = 64, TM = 8, TN = 8, BK = 16, kStages = 4, kPitch = BK + 4;
    static_assert(EPI == kStore || EPI == kFinal, "one weight per group");
    extern __shared__ __align__(16) float slabs[];   // stages x (BM + BN) rows
    umma::grid_trigger();
    umma::grid_wait();
    const int K = p.K, n = p.n;
    const long long M = p.M, m0 = (long long)blockIdx.x * BM;
    const int tiles_n = (n + BN - 1) / BN;
    const int grp = blockIdx.y / tiles_n;
    const int n0 = (blockIdx.y % tiles_n) * BN;
    const long long boff = (long long)blockIdx.z * p.a_batch;
    const float* a = p.a + boff;
    const float* w = p.w[grp] + boff;

    // this thread's 16-byte vectors of a slab: row t / 4 + 32 i, k offset 4 (t % 4)
    const int kc = (threadIdx.x & 3) * 4, lr = threadIdx.x >> 2;
    const float* src[6];
    float* dst[6];
    bool in[6];
#pragma unroll
    for (int i = 0; i < 6; ++i) {
        if (i < 4) {
            const int r = lr + 32 * i;                     // 64 hm + 4 ty + e -> slot 64 hm + 16 e + ty
            in[i] = m0 + r < M;
            src[i] = a + (in[i] ? m0 + r : 0) * K + kc;
            dst[i] = slabs + ((r & 64) + (r & 3) * 16 + ((r & 63) >> 2)) * kPitch + kc;
        } else {
            const int c = lr + 32 * (i - 4);               // 32 hf + 4 tx + e -> slot 32 hf + 8 e + tx
            in[i] = n0 + c < n;
            src[i] = w + (long long)(in[i] ? n0 + c : 0) * K + kc;
            dst[i] = slabs + (BM + (c & 32) + (c & 3) * 8 + ((c & 31) >> 2)) * kPitch + kc;
        }
    }
    const int slabs_k = (K + BK - 1) / BK;
    auto fetch = [&](int ks) {
        if (ks < slabs_k) {
            const bool kin = ks * BK + kc < K;
#pragma unroll
            for (int i = 0; i < 6; ++i)
                cp_async16(dst[i] + (ks % kStages) * ((BM + BN) * kPitch), kin ? src[i] + ks * BK : src[i] - kc, kin && in[i]);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    const int tx = threadIdx.x & 7, ty = threadIdx.x >> 3;
    u64 acc[TM][TN];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = 0ull;
#pragma unroll
    for (int ks = 0; ks < kStages - 1; ++ks) fetch(ks);
    for (int ks = 0; ks < slabs_k; ++ks) {
        asm volatile("cp.async.wait_group %0;" ::"n"(kStages - 2) : "memory");
        __syncthreads();
        fetch(ks + kStages - 1);
        const float* as = slabs + (ks % kStages) * ((BM + BN) * kPitch) + ty * kPitch;
        const float* ws = slabs + (ks % kStages) * ((BM + BN) * kPitch) + (BM + tx) * kPitch;
#pragma unroll
        for (int q = 0; q < BK / 4; ++q) {
            ulonglong2 av[TM];
#pragma unroll
            for (int i = 0; i < TM; ++i)
                av[i] = *reinterpret_cast<const ulonglong2*>(as + ((i >> 2) * 64 + (i & 3) * 16) * kPitch + q * 4);
#pragma unroll
            for (int j = 0; j < TN; ++j) {
                const ulonglong2 wv = *reinterpret_cast<const ulonglong2*>(ws + ((j >> 2) * 32 + (j & 3) * 8) * kPitch + q * 4);
#pragma unroll
                for (int i = 0; i < TM; ++i) {
                    fma2(acc[i][j], av[i].x, wv.x);
                    fma2(acc[i][j], av[i].y, wv.y);
                }
            }
        }
    }
    float v[TM][TN];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) {
            const float2 f = unpack2(acc[i][j]);
            v[i][j] = f.x + f.y;
        }
    epilogue<BM, BN, TM, TN, EPI, float>(p, v, m0, n0, grp, boff, tx, ty);
}
constexpr int kPairsSmem = 4 * (128 + 64) * 20 * 4;

template <int EPI>
int launch_pairs(const Args<float>& p, dim3 grid, cudaStream_t st) {
    static PerDeviceOnce configured;
    if (!configured.done()) {
        OF3_CUDA_CHECK(cudaFuncSetAttribute(gemm_pairs_kernel<EPI>, cudaFuncAttributeMaxDynamicSharedMemorySize, kPairsSmem));
        configured.mark();
    }
    OF3_CUDA_CHECK(launch_chained(gemm_pairs_kernel<EPI>, grid, 128, kPairsSmem, st, p));
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
    // large tiles once they give every SM at least one
    const bool large = tiles(128, kPaired ? 32 : 64) >= sm_count();
    const int bm = large ? 128 : 32, bn = large ? (kPaired ? 32 : 64) : (kPaired ? 16 : 32);
    const long long gx = (M + bm - 1) / bm, gy = (long long)((p.n + bn - 1) / bn) * groups;
    OF3_REQUIRE(batch <= 65535 && gy <= 65535 && gx < (1LL << 31), OF3_ERR_SHAPE, "gemm: %lld rows, %d columns, batch %d",
                M, p.n, batch);
    const dim3 grid((unsigned)gx, (unsigned)gy, batch);
    LaunchScope scope(20, st);
    if constexpr (std::is_same<T, float>::value && !K_OUTER && !kPaired) {
        // where every operand, and every plane of a batch, comes in whole vectors along k
        uintptr_t bits = reinterpret_cast<uintptr_t>(p.a) | (uintptr_t)(p.K & 3) << 2 | (uintptr_t)(p.a_batch & 3) << 2;
        for (int i = 0; i < groups; ++i) bits |= reinterpret_cast<uintptr_t>(p.w[i]);
        if (large && (bits & 15) == 0) return launch_pairs<EPI>(p, grid, st);
    }
    if (large)
        OF3_CUDA_CHECK(launch_chained(gemm_kernel<128, 64, 8, 8, 1, EPI, K_OUTER, T>, grid, 128, 0, st, p));
    else
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
