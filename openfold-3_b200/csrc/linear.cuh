// Linear layers of the single track and of the diffusion token stack with their consumers in the epilogue (linear.cu).
#pragma once
#include "common.cuh"

namespace of3 {
namespace fast {

// y[g][row][:] = x[a_index(g)][row][:] W_g^T for `groups` weights [n, k]
struct LinearIn {
    const __nv_bfloat16* x;    // [slices][rows][k]
    long long rows;
    int k;
    int n;                     // rows of one weight matrix
    const __nv_bfloat16* w[4]; // up to four weight matrices; or one base pointer and `groups` matrices back to back
    int num_w;
};

// plain store. Layers of three projections each (the adaptive LayerNorm's gate and shift from the normalised
// conditioning, the output gate from the raw one): layer l's matrices 0 and 1 multiply slice l of x, matrix 2 slice
// `raw_slice`. Weights back to back [layers][3][n][k], y [layers][3][rows][n].
int linear_conditioning(const __nv_bfloat16* x, long long rows, int k, int n, const __nv_bfloat16* w, int layers,
                        int slices, int raw_slice, __nv_bfloat16* y, cudaStream_t st);

// The operand images of the single-track attention (single_attn.cuh) straight from the projections of x:
// kinds[i] says what weight w[i] produces.
enum LinearOut { kOutQ = 0, kOutG = 1, kOutK = 2, kOutV = 3 };
struct AttnImages {
    __nv_bfloat16 *q, *k, *v, *g;   // q, k, v images and the gate rows [rows][H * D]
    const __nv_bfloat16* q_bias;    // [H * D] or null
    int rows_per_sample;            // rows of x per sample: query rows for q / g, keys for k / v
    int H, D;
};
int linear_attn_images(const LinearIn& in, const LinearOut* kinds, const AttnImages& im, cudaStream_t st);

// h[row][j] = silu(x w[0]^T) * (x w[1]^T)
int linear_swiglu(const LinearIn& in, __nv_bfloat16* h, cudaStream_t st);

// out[row][j] = (residual ? residual[row][j] : 0)
//               + (gate ? sigmoid(gate[row][j] + gate_bias[j]) : 1) * (mask ? mask[row] : 1) * (x w[0]^T)
// out may alias residual
int linear_residual(const LinearIn& in, const __nv_bfloat16* residual, const __nv_bfloat16* gate,
                    const __nv_bfloat16* gate_bias, const __nv_bfloat16* mask, __nv_bfloat16* out, cudaStream_t st);

// The same where a call has few tokens (token_linear.cu): tiles of 64 or 128 output channels by 16 to 64 tokens. residual and out
// start on 4 bytes.
bool token_images_supported(int samples, int tokens, int c, int d);
bool token_swiglu_supported(long long rows, int hidden);
bool token_residual_supported(long long rows, int c);
int token_attn_images(const LinearIn& in, const LinearOut* kinds, const AttnImages& im, cudaStream_t st);
int token_swiglu(const LinearIn& in, __nv_bfloat16* h, cudaStream_t st);
int token_residual(const LinearIn& in, const __nv_bfloat16* residual, const __nv_bfloat16* gate,
                   const __nv_bfloat16* gate_bias, const __nv_bfloat16* mask, __nv_bfloat16* out, cudaStream_t st);

}  // namespace fast
}  // namespace of3
