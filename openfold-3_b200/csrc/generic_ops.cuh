// Shape-generic SIMT kernels (any channel width, head count, sequence length).
//
// They back (1) the fp32 validation mode, where every product and sum is fp32 or nearer to the exact value (large matrix
// products as sums of bf16 products on the tensor cores, generic_gemm.cu; no TF32), and (2) bf16 storage with shapes the tcgen05 kernels do not
// cover. Storage type T is float or __nv_bfloat16; intermediates are always fp32.
#pragma once
#include "common.cuh"

namespace of3 {
namespace generic {

// Where row r of a caller's tensor lies: (r / inner) * outer_stride + (r % inner) * inner_stride (elements), so that a
// transposed [N, N, C] view is read and written without materialising it.
struct RowMap {
    long long inner, outer_stride, inner_stride;
};
#ifdef __CUDACC__
__device__ __forceinline__ long long row_offset(const RowMap& m, long long r) {
    if (((r | m.inner) >> 32) == 0) {   // a 64-bit division costs some 500 cycles
        const uint32_t q = (uint32_t)r / (uint32_t)m.inner;
        return q * m.outer_stride + (uint32_t)(r - (long long)q * m.inner) * m.inner_stride;
    }
    return (r / m.inner) * m.outer_stride + (r % m.inner) * m.inner_stride;
}
#endif
inline RowMap dense_rows(long long rows, int C) { return RowMap{rows > 0 ? rows : 1, 0, C}; }

// y[r, :] = LN(x[r, :]) * gamma + beta (gamma / beta may be null); y dense fp32 [rows, C] or null. With proj_w
// [H, C] also proj[h * rows + r] = sum_c y[r, c] * proj_w[h, c].
template <typename TX, typename TP>
int layernorm(const TX* x, const TP* gamma, const TP* beta, float* y, long long rows, int C, float eps, RowMap map,
              cudaStream_t stream, const TP* proj_w = nullptr, int H = 0, float* proj = nullptr);
// y[r, :] = LN(x[:, r]) * gamma + beta for channel-major x [C][rows] (fp32); y dense fp32 [rows, C].
template <typename TP>
int layernorm_planes(const float* x, const TP* gamma, const TP* beta, float* y, long long rows, int C, float eps,
                     cudaStream_t stream);

// Linear layers y = x W^T of fp32 rows x [rows, k], dense, with weights [n, k] of the storage type.
// plain: out[i][rows, n] = x w[i]^T + bias[i], i < count <= 4, one launch
template <typename T>
int linear_multi(const float* x, int count, const T* const* w, const T* const* bias, float* const* out, long long rows,
                 int n, int k, cudaStream_t stream);
template <typename T>
inline int linear(const float* x, const T* w, const T* bias, float* out, long long rows, int n, int k, cudaStream_t st) {
    return linear_multi<T>(x, 1, &w, &bias, &out, rows, n, k, st);
}
// gated, channel-major: out[i][c * rows + r] = (mask ? mask[r] : 1) * sigmoid(x wg[i]^T)[r][c] * (x wp[i]^T)[r][c]
template <typename T>
int linear_gated_planes(const float* x, int count, const T* const* wp, const T* const* wg, const T* mask,
                        float* const* out, long long rows, int n, int k, cudaStream_t stream);
// h[rows, n] = silu(x wa^T) * (x wb^T)
template <typename T>
int linear_swiglu(const float* x, const T* wa, const T* wb, float* h, long long rows, int n, int k, cudaStream_t stream);
// out_row(r) = (residual ? residual_row(r) : 0) + (x w^T)[r] * (gate ? sigmoid(gate[r]) : 1) * (mask ? mask[r] : 1);
// gate dense fp32 [rows, n], mask [rows]; residual / out rows at `map` (they may alias)
template <typename T>
int linear_final(const float* x, const T* w, const float* gate, const T* residual, const T* mask, T* out, long long rows,
                 int n, int k, RowMap map, cudaStream_t stream);
// Batched products of fp32 planes, x[c][i][j] = sum_k a(c, i, k) b(c, j, k): a(c, i, k) = a[c * a_batch + i * N + k], or
// with k_outer a[c * a_batch + k * N + i] (b likewise); out[c * a_batch + i * N + j].
int contract_planes(const float* a, const float* b, float* x, int batch, int N, long long a_batch, bool k_outer,
                    cudaStream_t stream);

// Streaming (online-softmax) attention, gated:
//   o[bb, q, h, :] = sigmoid(g[bb, q, h, :]) * softmax_k( scale * q.k + inf * (mask(bb, k) - 1)
//                                                         + pair_bias[bb / rows_per_bias, h, q, k] ) v
// q, k, v, g, out: [BB, N, H*d] fp32 (out may be g); mask(bb, k) = mask[bb * mask_row + k * mask_k] or null;
// pair_bias [BB / rows_per_bias, H, N, N] fp32 or null. d <= 64.
template <typename T>
int attention(const float* q, const float* k, const float* v, const float* g, const T* mask, long long mask_row,
              long long mask_k, float inf, const float* pair_bias, float* out, long long BB, int N, int H, int d,
              float scale, long long rows_per_bias, cudaStream_t stream);

// dst = sigmoid(g) * a + s   (adaptive LayerNorm combine), all dense, n elements.
int ada_combine(const float* g, const float* a, const float* s, float* dst, long long n,
                cudaStream_t stream);
// Fused pair-bias projection for 128-channel pair tensors and 16 heads:
// dst[b][h][pos] = sum_c LN(z[b, pos, :])[c] * w[h][c] for pos < positions_per_sample (N*N for a whole
// tensor, R*N for a row shard), one thread per pair position, one pass over z.
// gamma/beta may be null. Returns OF3_ERR_SHAPE for other widths (callers fall back to the chain).
template <typename T>
int pair_bias_c128_h16(const T* z, const T* gamma, const T* beta, const T* w, float* dst, long long B,
                       long long positions_per_sample, cudaStream_t stream);
// dst[b][h][q][k] = src[h][b][q][k]
int swap_heads(const float* src, float* dst, long long B, int N, int H, cudaStream_t stream);
// dense fp32 copy of a storage-type tensor
template <typename T>
int to_f32(const T* src, float* dst, long long n, cudaStream_t stream);

}  // namespace generic
}  // namespace of3
