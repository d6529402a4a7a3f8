// Shape-generic SIMT kernels: see generic_ops.cuh. True fp32 arithmetic throughout.
#include "generic_ops.cuh"
#include "runtime.cuh"
#include "umma.cuh"
#include <type_traits>

namespace of3 {
namespace generic {
namespace {

constexpr int kThreads = 256;

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
__device__ __forceinline__ float sigmoid_acc(float x) { return 1.0f / (1.0f + expf(-x)); }

inline unsigned grid_for(long long n, int per_block) {
    long long g = (n + per_block - 1) / per_block;
    return (unsigned)(g < 1 ? 1 : g);
}

// ------------------------------------------------------------------ LayerNorm
// One warp per row; the row stays in registers up to 512 channels.
constexpr int kLnRegs = 16;
template <typename TX, typename TP>
__global__ void __launch_bounds__(kThreads) layernorm_kernel(const TX* __restrict__ x, const TP* __restrict__ gamma,
                                                             const TP* __restrict__ beta, float* __restrict__ y,
                                                             long long rows, int C, float eps, RowMap map,
                                                             const TP* __restrict__ proj_w, int H,
                                                             float* __restrict__ proj) {
    umma::grid_trigger();
    umma::grid_wait();
    const int lane = threadIdx.x & 31;
    const long long r = (long long)blockIdx.x * (kThreads / 32) + (threadIdx.x >> 5);
    if (r >= rows) return;
    const TX* xr = x + row_offset(map, r);
    float* yr = y + r * C;
    const bool in_regs = C <= 32 * kLnRegs;
    float v[kLnRegs];
    float s = 0.f;
    if (in_regs) {
#pragma unroll
        for (int i = 0; i < kLnRegs; ++i) {
            v[i] = lane + 32 * i < C ? ld_as_float(xr + lane + 32 * i) : 0.f;
            s += v[i];
        }
    } else {
        for (int c = lane; c < C; c += 32) s += ld_as_float(xr + c);
    }
    const float mean = warp_sum(s) / (float)C;
    float q = 0.f;
    if (in_regs) {
#pragma unroll
        for (int i = 0; i < kLnRegs; ++i) {
            const float d = lane + 32 * i < C ? v[i] - mean : 0.f;
            q += d * d;
        }
    } else {
        for (int c = lane; c < C; c += 32) {
            const float d = ld_as_float(xr + c) - mean;
            q += d * d;
        }
    }
    const float rstd = 1.0f / sqrtf(warp_sum(q) / (float)C + eps);
    auto norm = [&](float xv, int c) {
        float o = (xv - mean) * rstd;
        if (gamma) o *= ld_as_float(gamma + c);
        if (beta) o += ld_as_float(beta + c);
        return o;
    };
    if (in_regs) {
#pragma unroll
        for (int i = 0; i < kLnRegs; ++i) {
            const int c = lane + 32 * i;
            if (c < C) {
                v[i] = norm(v[i], c);
                if (y) yr[c] = v[i];
            }
        }
    } else if (y) {
        for (int c = lane; c < C; c += 32) yr[c] = norm(ld_as_float(xr + c), c);
    }
    for (int h = 0; h < H; ++h) {
        float d = 0.f;
        if (in_regs) {
#pragma unroll
            for (int i = 0; i < kLnRegs; ++i)
                if (lane + 32 * i < C) d = fmaf(v[i], ld_as_float(proj_w + (long long)h * C + lane + 32 * i), d);
        } else {
            for (int c = lane; c < C; c += 32)
                d = fmaf(norm(ld_as_float(xr + c), c), ld_as_float(proj_w + (long long)h * C + c), d);
        }
        d = warp_sum(d);
        if (lane == 0) proj[(long long)h * rows + r] = d;
    }
}

// The same for fp32 rows in whole 16-byte vectors, V of them per lane (C <= 128 V): at C = 128 a lane's loads, statistics and
// stores are one of each instead of sixteen guarded passes.
template <int V>
__global__ void __launch_bounds__(kThreads) layernorm_vec_kernel(const float* __restrict__ x, const float* __restrict__ gamma,
                                                                 const float* __restrict__ beta, float* __restrict__ y,
                                                                 long long rows, int C, float eps, RowMap map,
                                                                 const float* __restrict__ proj_w, int H,
                                                                 float* __restrict__ proj) {
    umma::grid_trigger();
    umma::grid_wait();
    const int lane = threadIdx.x & 31;
    const long long r = (long long)blockIdx.x * (kThreads / 32) + (threadIdx.x >> 5);
    if (r >= rows) return;
    const float* xr = x + row_offset(map, r);
    auto vec = [&](const float* p, int i, float fill) {
        const int c = 4 * (lane + 32 * i);
        return (p != nullptr && c < C) ? *reinterpret_cast<const float4*>(p + c) : make_float4(fill, fill, fill, fill);
    };
    float4 v[V], gm[V], bt[V];
    float s = 0.f;
#pragma unroll
    for (int i = 0; i < V; ++i) v[i] = vec(xr, i, 0.f);
#pragma unroll
    for (int i = 0; i < V; ++i) {
        gm[i] = vec(gamma, i, 1.f);
        bt[i] = vec(beta, i, 0.f);
    }
#pragma unroll
    for (int i = 0; i < V; ++i) s += (v[i].x + v[i].y) + (v[i].z + v[i].w);
    const float mean = warp_sum(s) / (float)C;
    float q = 0.f;
#pragma unroll
    for (int i = 0; i < V; ++i) {
        if (4 * (lane + 32 * i) < C) {
            v[i].x -= mean; v[i].y -= mean; v[i].z -= mean; v[i].w -= mean;
            q += (v[i].x * v[i].x + v[i].y * v[i].y) + (v[i].z * v[i].z + v[i].w * v[i].w);
        }
    }
    const float rstd = 1.0f / sqrtf(warp_sum(q) / (float)C + eps);
#pragma unroll
    for (int i = 0; i < V; ++i) {
        const int c = 4 * (lane + 32 * i);
        if (c >= C) continue;
        v[i].x = v[i].x * rstd * gm[i].x + bt[i].x;
        v[i].y = v[i].y * rstd * gm[i].y + bt[i].y;
        v[i].z = v[i].z * rstd * gm[i].z + bt[i].z;
        v[i].w = v[i].w * rstd * gm[i].w + bt[i].w;
        if (y) *reinterpret_cast<float4*>(y + r * C + c) = v[i];
    }
    for (int h = 0; h < H; ++h) {
        float d = 0.f;
#pragma unroll
        for (int i = 0; i < V; ++i) {
            const float4 w = vec(proj_w + (long long)h * C, i, 0.f);
            d = fmaf(v[i].x, w.x, d);
            d = fmaf(v[i].y, w.y, d);
            d = fmaf(v[i].z, w.z, d);
            d = fmaf(v[i].w, w.w, d);
        }
        d = warp_sum(d);
        if (lane == 0) proj[(long long)h * rows + r] = d;
    }
}

// Rows of channel planes: a block takes 32 rows, passes of 32 x 32 values through shared memory.
template <typename TP>
__global__ void __launch_bounds__(kThreads) layernorm_planes_kernel(const float* __restrict__ x,
                                                                    const TP* __restrict__ gamma,
                                                                    const TP* __restrict__ beta, float* __restrict__ y,
                                                                    long long rows, int C, float eps) {
    __shared__ float part[8][33], mean_s[32], rstd_s[32], tile[32][33];
    umma::grid_trigger();
    umma::grid_wait();
    const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
    const long long r0 = (long long)blockIdx.x * 32, r = r0 + lane;
    auto reduce = [&](float v) {   // sum over the 8 warps, per lane
        part[wp][lane] = v;
        __syncthreads();
        float s = 0.f;
#pragma unroll
        for (int i = 0; i < 8; ++i) s += part[i][lane];
        __syncthreads();
        return s;
    };
    float s = 0.f;
    for (int c = wp; c < C; c += 8) s += r < rows ? x[(long long)c * rows + r] : 0.f;
    const float mean = reduce(s) / (float)C;
    float q = 0.f;
    for (int c = wp; c < C; c += 8) {
        const float d = (r < rows ? x[(long long)c * rows + r] : 0.f) - mean;
        q += d * d;
    }
    const float rstd = 1.0f / sqrtf(reduce(q) / (float)C + eps);
    if (wp == 0) {
        mean_s[lane] = mean;
        rstd_s[lane] = rstd;
    }
    for (int c0 = 0; c0 < C; c0 += 32) {
        __syncthreads();
        for (int c = wp; c < 32; c += 8)
            tile[c][lane] = (c0 + c < C && r < rows) ? x[(long long)(c0 + c) * rows + r] : 0.f;
        __syncthreads();
        const int c = c0 + lane;
        if (c < C) {
            const float gm = gamma ? ld_as_float(gamma + c) : 1.f, bt = beta ? ld_as_float(beta + c) : 0.f;
            for (int i = wp; i < 32; i += 8)
                if (r0 + i < rows) y[(r0 + i) * C + c] = (tile[lane][i] - mean_s[i]) * rstd_s[i] * gm + bt;
        }
    }
}

// ------------------------------------------------------------------ streaming attention
// Block = 64 queries of one (bb, head), 256 threads as 16 x 16: thread (ty, tx) holds the 4 x 4 logits of queries 4 ty..
// and keys 4 tx.., and DC = DP / 16 output channels of its four queries. Q and K lie transposed in shared memory, P goes
// through it; a row's maximum and sum are joined over the 16 threads of a half warp. FMA-pipe bound: 16 FMA per two
// 16-byte shared-memory reads. (One warp per query, two shared-memory reads per FMA: 121 us per layer at N = 128, 4 x 32.)
constexpr int kAttMaxD = 64;
constexpr int kAttQ = 64, kAttK = 64, kAttP = 68;   // pitch: 16-byte aligned rows
template <int DP>
constexpr int att_smem_floats() { return 2 * DP * kAttP + kAttK * DP + kAttK * kAttP + kAttK; }

template <int DP, typename T>
__global__ void __launch_bounds__(256, DP <= 32 ? 3 : 2) attention_kernel(const float* __restrict__ q, const float* __restrict__ k,
                                                        const float* __restrict__ v, const float* g,
                                                        const T* __restrict__ mask, long long mask_row,
                                                        long long mask_k, float inf, const float* __restrict__ pair_bias,
                                                        float* out, int N, int H, int d, float scale,
                                                        long long rows_per_bias) {
    constexpr int DC = DP / 16;
    extern __shared__ __align__(16) float att_smem[];
    float* Qs = att_smem;                     // [DP][kAttP]
    float* Ks = Qs + DP * kAttP;              // [DP][kAttP]
    float* Vs = Ks + DP * kAttP;              // [64][DP]
    float* Ps = Vs + kAttK * DP;              // [64 keys][kAttP]
    float* Ms = Ps + kAttK * kAttP;           // [64]
    umma::grid_trigger();
    umma::grid_wait();
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    const long long bb = blockIdx.x;
    const int h = blockIdx.y, q0 = blockIdx.z * kAttQ;
    const long long pitch = (long long)H * d, base = bb * N * pitch + (long long)h * d;
    for (int idx = threadIdx.x; idx < kAttQ * DP; idx += 256) {
        const int i = idx / DP, c = idx % DP;
        Qs[c * kAttP + i] = (q0 + i < N && c < d) ? q[base + (q0 + i) * pitch + c] : 0.f;
    }
    const float* pb = pair_bias ? pair_bias + ((bb / rows_per_bias) * H + h) * (long long)N * N : nullptr;
    float m[4], l[4], o[4][DC];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        m[i] = -INFINITY;
        l[i] = 0.f;
#pragma unroll
        for (int c = 0; c < DC; ++c) o[i][c] = 0.f;
    }
    // A key block's keys and values, in registers while the block before them is multiplied: fetched between the barriers they, and
    // the pair bias fetched where it is added, were most of a block's time (fp32 trunk block: N = 128 695 -> 677 us, 250 2246 -> 2143, with three blocks per SM)
    constexpr int kVecs = kAttK * DP / 256;
    float rk[kVecs], rv[kVecs], rm = 0.f;
    auto fetch = [&](int k0) {
#pragma unroll
        for (int u = 0; u < kVecs; ++u) {
            const int i = (threadIdx.x + u * 256) / DP, c = (threadIdx.x + u * 256) % DP;
            const bool in = k0 + i < N && c < d;
            const long long off = base + (k0 + i) * pitch + c;
            rk[u] = in ? k[off] : 0.f;
            rv[u] = in ? v[off] : 0.f;
        }
        if (threadIdx.x < kAttK) {
            const int kk = k0 + threadIdx.x;
            rm = kk >= N ? -INFINITY : (mask ? inf * (ld_as_float(mask + bb * mask_row + kk * mask_k) - 1.0f) : 0.f);
        }
    };
    fetch(0);
    for (int k0 = 0; k0 < N; k0 += kAttK) {
        __syncthreads();
#pragma unroll
        for (int u = 0; u < kVecs; ++u) {
            const int i = (threadIdx.x + u * 256) / DP, c = (threadIdx.x + u * 256) % DP;
            Ks[c * kAttP + i] = rk[u];
            Vs[i * DP + c] = rv[u];
        }
        if (threadIdx.x < kAttK) Ms[threadIdx.x] = rm;
        __syncthreads();
        float bias[4][4];
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int qi = q0 + ty * 4 + i, kk = k0 + tx * 4 + j;
                bias[i][j] = pb && qi < N && kk < N ? pb[(long long)qi * N + kk] : 0.f;
            }
        if (k0 + kAttK < N) fetch(k0 + kAttK);
        float s[4][4];
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) s[i][j] = 0.f;
#pragma unroll 8
        for (int c = 0; c < DP; ++c) {
            const float4 a = *reinterpret_cast<const float4*>(&Qs[c * kAttP + ty * 4]);
            const float4 b = *reinterpret_cast<const float4*>(&Ks[c * kAttP + tx * 4]);
            const float av[4] = {a.x, a.y, a.z, a.w}, bv[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) s[i][j] = fmaf(av[i], bv[j], s[i][j]);
        }
        float p[4][4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            float mx = -INFINITY;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float x = s[i][j] * scale + Ms[tx * 4 + j] + bias[i][j];
                s[i][j] = x;
                mx = fmaxf(mx, x);
            }
#pragma unroll
            for (int w = 8; w > 0; w >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, w));
            const float m_new = fmaxf(m[i], mx);   // finite: the first block holds a key < N
            const float corr = expf(m[i] - m_new);
            m[i] = m_new;
            float sum = 0.f;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                p[i][j] = expf(s[i][j] - m_new);
                sum += p[i][j];
            }
#pragma unroll
            for (int w = 8; w > 0; w >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, w);
            l[i] = l[i] * corr + sum;
#pragma unroll
            for (int c = 0; c < DC; ++c) o[i][c] *= corr;
        }
#pragma unroll
        for (int j = 0; j < 4; ++j)
            *reinterpret_cast<float4*>(&Ps[(tx * 4 + j) * kAttP + ty * 4]) = make_float4(p[0][j], p[1][j], p[2][j], p[3][j]);
        __syncthreads();
#pragma unroll 8
        for (int kk = 0; kk < kAttK; ++kk) {
            const float4 a = *reinterpret_cast<const float4*>(&Ps[kk * kAttP + ty * 4]);
            const float av[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
            for (int c = 0; c < DC; ++c) {
                const float vv = Vs[kk * DP + tx * DC + c];
#pragma unroll
                for (int i = 0; i < 4; ++i) o[i][c] = fmaf(av[i], vv, o[i][c]);
            }
        }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int qi = q0 + ty * 4 + i;
        if (qi >= N) continue;
        const float inv = 1.0f / l[i];
        const long long off = base + qi * pitch;
#pragma unroll
        for (int c = 0; c < DC; ++c) {
            const int cc = tx * DC + c;
            if (cc < d) out[off + cc] = o[i][c] * inv * sigmoid_acc(g[off + cc]);
        }
    }
}

// ------------------------------------------------------------------ fused pair-bias projection
// LN(x).w_h = rstd * sum_c (x_c - mean) * (gamma_c w_hc) + sum_c beta_c w_hc
template <typename T>
__global__ void __launch_bounds__(128) pair_bias_c128_h16_kernel(const T* __restrict__ z,
                                                                 const T* __restrict__ gamma,
                                                                 const T* __restrict__ beta,
                                                                 const T* __restrict__ w,
                                                                 float* __restrict__ dst, long long rows,
                                                                 long long nn) {
    __shared__ float ws[16][128];
    __shared__ float cs[16];
    umma::grid_trigger();
    umma::grid_wait();
    for (int i = threadIdx.x; i < 16 * 128; i += 128) {
        const int c = i & 127;
        ws[i >> 7][c] = ld_as_float(w + i) * (gamma ? ld_as_float(gamma + c) : 1.0f);
    }
    if (threadIdx.x < 16) {
        float a = 0.f;
        if (beta)
            for (int c = 0; c < 128; ++c) a += ld_as_float(beta + c) * ld_as_float(w + threadIdx.x * 128 + c);
        cs[threadIdx.x] = a;
    }
    __syncthreads();
    const long long r = (long long)blockIdx.x * 128 + threadIdx.x;
    if (r >= rows) return;
    float x[128];
    const T* zr = z + r * 128;
    if constexpr (sizeof(T) == 2) {
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            const uint4 v = __ldg(reinterpret_cast<const uint4*>(zr) + i);
            const uint32_t u[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                x[i * 8 + j * 2] = bf16lo(u[j]);
                x[i * 8 + j * 2 + 1] = bf16hi(u[j]);
            }
        }
    } else {
#pragma unroll
        for (int i = 0; i < 32; ++i) {
            const float4 v = __ldg(reinterpret_cast<const float4*>(zr) + i);
            x[i * 4] = v.x; x[i * 4 + 1] = v.y; x[i * 4 + 2] = v.z; x[i * 4 + 3] = v.w;
        }
    }
    // four independent partial sums / four heads at a time: the single chains of 128 dependent
    // operations were the critical path at the 8-12 warps per SM that 128 row registers allow
    float s4[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int c = 0; c < 128; c += 4) {
        s4[0] += x[c]; s4[1] += x[c + 1]; s4[2] += x[c + 2]; s4[3] += x[c + 3];
    }
    const float mean = ((s4[0] + s4[1]) + (s4[2] + s4[3])) * (1.0f / 128.0f);
    float v4[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int c = 0; c < 128; c += 4) {
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            x[c + e] -= mean;
            v4[e] = fmaf(x[c + e], x[c + e], v4[e]);
        }
    }
    const float rstd = 1.0f / sqrtf(((v4[0] + v4[1]) + (v4[2] + v4[3])) * (1.0f / 128.0f) + 1e-5f);
    const long long b = r / nn;
    const long long qk = r % nn;
#pragma unroll 1
    for (int h = 0; h < 16; h += 4) {
        float acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int c = 0; c < 128; c += 4) {
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const float4 wv = *reinterpret_cast<const float4*>(&ws[h + e][c]);
                acc[e] = fmaf(x[c], wv.x, acc[e]);
                acc[e] = fmaf(x[c + 1], wv.y, acc[e]);
                acc[e] = fmaf(x[c + 2], wv.z, acc[e]);
                acc[e] = fmaf(x[c + 3], wv.w, acc[e]);
            }
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) dst[(b * 16 + h + e) * nn + qk] = fmaf(acc[e], rstd, cs[h + e]);
    }
}

// ------------------------------------------------------------------ elementwise
__global__ void ada_combine_kernel(const float* __restrict__ g, const float* __restrict__ a,
                                   const float* __restrict__ s, float* __restrict__ dst,
                                   long long n) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) dst[i] = sigmoid_acc(g[i]) * a[i] + s[i];
}
__global__ void swap_heads_kernel(const float* __restrict__ src, float* __restrict__ dst, long long B, long long nn, int H) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= B * H * nn) return;
    const long long h = (i / nn) % H, b = i / (nn * H);
    dst[i] = src[(h * B + b) * nn + i % nn];
}
template <typename T>
__global__ void to_f32_kernel(const T* __restrict__ src, float* __restrict__ dst, long long n) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) dst[i] = ld_as_float(src + i);
}

}  // namespace

// ------------------------------------------------------------------ host wrappers
template <typename TX, typename TP>
int layernorm(const TX* x, const TP* gamma, const TP* beta, float* y, long long rows, int C, float eps, RowMap map,
              cudaStream_t stream, const TP* proj_w, int H, float* proj) {
    if (rows <= 0) return OF3_OK;
    LaunchScope scope(20, stream);
    if constexpr (std::is_same<TX, float>::value) {
        const uintptr_t bits = (uintptr_t)x | (uintptr_t)gamma | (uintptr_t)beta | (uintptr_t)y | (uintptr_t)proj_w;
        const bool vec = (bits & 15) == 0 && ((C | map.inner_stride | map.outer_stride) & 3) == 0;
        if (vec && C <= 512) {
            OF3_CUDA_CHECK(launch_chained(C <= 128 ? layernorm_vec_kernel<1> : layernorm_vec_kernel<4>,
                                          grid_for(rows, kThreads / 32), kThreads, 0, stream, x, gamma, beta, y, rows, C, eps,
                                          map, proj_w, H, proj));
            return OF3_OK;
        }
    }
    OF3_CUDA_CHECK(launch_chained(layernorm_kernel<TX, TP>, grid_for(rows, kThreads / 32), kThreads, 0, stream, x, gamma,
                                  beta, y, rows, C, eps, map, proj_w, H, proj));
    return OF3_OK;
}
#define INSTANTIATE_LN(TX, TP)                                                                                       \
    template int layernorm<TX, TP>(const TX*, const TP*, const TP*, float*, long long, int, float, RowMap, cudaStream_t, \
                                   const TP*, int, float*);
INSTANTIATE_LN(float, float)
INSTANTIATE_LN(__nv_bfloat16, __nv_bfloat16)

template <typename TP>
int layernorm_planes(const float* x, const TP* gamma, const TP* beta, float* y, long long rows, int C, float eps,
                     cudaStream_t stream) {
    if (rows <= 0) return OF3_OK;
    LaunchScope scope(20, stream);
    OF3_CUDA_CHECK(launch_chained(layernorm_planes_kernel<TP>, grid_for(rows, 32), kThreads, 0, stream, x, gamma, beta, y,
                                  rows, C, eps));
    return OF3_OK;
}
template int layernorm_planes<float>(const float*, const float*, const float*, float*, long long, int, float, cudaStream_t);
template int layernorm_planes<__nv_bfloat16>(const float*, const __nv_bfloat16*, const __nv_bfloat16*, float*, long long,
                                             int, float, cudaStream_t);

template <int DP, typename T>
static int attention_launch(const float* q, const float* k, const float* v, const float* g, const T* mask,
                            long long mask_row, long long mask_k, float inf, const float* pair_bias, float* out,
                            long long BB, int N, int H, int d, float scale, long long rows_per_bias, cudaStream_t st) {
    constexpr int smem = att_smem_floats<DP>() * 4;
    static PerDeviceOnce configured;
    if (!configured.done()) {
        OF3_CUDA_CHECK(cudaFuncSetAttribute(attention_kernel<DP, T>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
        configured.mark();
    }
    LaunchScope scope(20, st);
    OF3_CUDA_CHECK(launch_chained(attention_kernel<DP, T>, dim3((unsigned)BB, H, ceil_div(N, kAttQ)), 256, smem, st, q, k,
                                  v, g, mask, mask_row, mask_k, inf, pair_bias, out, N, H, d, scale, rows_per_bias));
    return OF3_OK;
}
template <typename T>
int attention(const float* q, const float* k, const float* v, const float* g, const T* mask, long long mask_row,
              long long mask_k, float inf, const float* pair_bias, float* out, long long BB, int N, int H, int d,
              float scale, long long rows_per_bias, cudaStream_t st) {
    OF3_REQUIRE(d >= 1 && d <= kAttMaxD, OF3_ERR_SHAPE, "attention: head dim %d not in [1, %d]", d, kAttMaxD);
    OF3_REQUIRE(H <= 65535, OF3_ERR_SHAPE, "attention: too many heads");
    OF3_REQUIRE(ceil_div(N, kAttQ) <= 65535, OF3_ERR_SHAPE, "attention: N %d too large", N);
    if (BB <= 0) return OF3_OK;
#define ATT(DP) attention_launch<DP, T>(q, k, v, g, mask, mask_row, mask_k, inf, pair_bias, out, BB, N, H, d, scale, \
                                        rows_per_bias, st)
    return d <= 16 ? ATT(16) : (d <= 32 ? ATT(32) : (d <= 48 ? ATT(48) : ATT(64)));
#undef ATT
}
template int attention<float>(const float*, const float*, const float*, const float*, const float*, long long, long long,
                              float, const float*, float*, long long, int, int, int, float, long long, cudaStream_t);
template int attention<__nv_bfloat16>(const float*, const float*, const float*, const float*, const __nv_bfloat16*,
                                      long long, long long, float, const float*, float*, long long, int, int, int, float,
                                      long long, cudaStream_t);

int ada_combine(const float* g, const float* a, const float* s, float* dst, long long n,
                cudaStream_t stream) {
    if (n <= 0) return OF3_OK;
    LaunchScope scope(20, stream);
    ada_combine_kernel<<<grid_for(n, kThreads), kThreads, 0, stream>>>(g, a, s, dst, n);
    OF3_CUDA_CHECK(cudaGetLastError());
    return OF3_OK;
}
template <typename T>
int pair_bias_c128_h16(const T* z, const T* gamma, const T* beta, const T* w, float* dst, long long B,
                       long long positions_per_sample, cudaStream_t stream) {
    const long long nn = positions_per_sample;
    const long long rows = B * nn;
    if (rows <= 0) return OF3_OK;
    OF3_REQUIRE(((uintptr_t)z & 15) == 0, OF3_ERR_ALIGN, "pair_bias: z must be 16-byte aligned");
    LaunchScope scope(20, stream);
    OF3_CUDA_CHECK(launch_chained(pair_bias_c128_h16_kernel<T>, grid_for(rows, 128), 128, 0, stream, z, gamma, beta, w,
                                  dst, rows, nn));
    return OF3_OK;
}
template int pair_bias_c128_h16<float>(const float*, const float*, const float*, const float*, float*,
                                       long long, long long, cudaStream_t);
template int pair_bias_c128_h16<__nv_bfloat16>(const __nv_bfloat16*, const __nv_bfloat16*, const __nv_bfloat16*,
                                               const __nv_bfloat16*, float*, long long, long long, cudaStream_t);

int swap_heads(const float* src, float* dst, long long B, int N, int H, cudaStream_t stream) {
    const long long nn = (long long)N * N, total = B * H * nn;
    if (total <= 0) return OF3_OK;
    LaunchScope scope(20, stream);
    swap_heads_kernel<<<grid_for(total, kThreads), kThreads, 0, stream>>>(src, dst, B, nn, H);
    OF3_CUDA_CHECK(cudaGetLastError());
    return OF3_OK;
}

template <typename T>
int to_f32(const T* src, float* dst, long long n, cudaStream_t stream) {
    if (n <= 0) return OF3_OK;
    LaunchScope scope(20, stream);
    to_f32_kernel<T><<<grid_for(n, kThreads), kThreads, 0, stream>>>(src, dst, n);
    OF3_CUDA_CHECK(cudaGetLastError());
    return OF3_OK;
}
template int to_f32<float>(const float*, float*, long long, cudaStream_t);
template int to_f32<__nv_bfloat16>(const __nv_bfloat16*, float*, long long, cudaStream_t);

}  // namespace generic
}  // namespace of3
