// Single-track layers behind the stack entry points: conditioning computed ahead for several layers.
#pragma once
#include "modules.cuh"

namespace of3 {
namespace fast {

// Internal flag of the single-track layers, beside the public ones: other kernels run at the same time (the next block's pair stack).
constexpr int kFlagBeside = 1 << 20;
constexpr int kBesideRows = 64;

// The three projections of the conditioning s that an AdaLN layer needs, planes [3][rows][c_a]: gate and shift of the
// adaptive LayerNorm (without the gate's bias), output gate (without its bias).
struct CondLayer {
    const __nv_bfloat16 *ln_s_w, *w_g, *w_s, *w_out;
};
inline CondLayer cond_layer(const of3_attn_pair_bias_params* p) {
    typedef const __nv_bfloat16* P;
    return {(P)p->ada_ln_s_w, (P)p->ada_w_g, (P)p->ada_w_s, (P)p->w_ada_out};
}
inline CondLayer cond_layer(const of3_cond_transition_params* p) {
    typedef const __nv_bfloat16* P;
    return {(P)p->ada_ln_s_w, (P)p->ada_w_g, (P)p->ada_w_s, (P)p->w_g};
}
// planes [layers][3][rows][c_a] for `layers` layers of one s [rows][c_s]; sn: scratch [layers + 1][rows][c_s]. One launch
// for the normalised rows and one GEMM launch when the layers' weights [3][c_a][c_s] lie back to back.
constexpr int kMaxCondBatch = 48;
int conditioning(const __nv_bfloat16* s, const CondLayer* layer, int layers, long long rows, int c_a, int c_s,
                 __nv_bfloat16* sn, __nv_bfloat16* planes, cudaStream_t st);
// The two launches apart: the normalised rows of `layers` layers (and s itself, slice `layers`) into sn; the planes of
// `layers` of them, from slice `first` on, where s is slice `raw`.
int conditioning_rows(const __nv_bfloat16* s, const CondLayer* layer, int layers, long long rows, int c_s, __nv_bfloat16* sn,
                      cudaStream_t st);
int conditioning_planes(const __nv_bfloat16* sn, int first, int raw, const CondLayer* layer, int layers, long long rows,
                        int c_a, int c_s, __nv_bfloat16* planes, cudaStream_t st);

// operand images of the attention kernel in the workspace
struct SingleImages {
    __nv_bfloat16 *q, *k, *v;
};
SingleImages take_single_images(Arena& ws, int BB, int N, int nq, int H, int d);
// pair bias of the attention: tiles (projected), fp32 [zh][nq][N] to be converted into tb, or z to be projected into tb
struct SingleBias {
    const __nv_bfloat16* tiles = nullptr;
    const float* f32 = nullptr;
    const __nv_bfloat16 *z = nullptr, *ln_w = nullptr, *ln_b = nullptr, *w = nullptr;
};
int single_attn(const SingleImages& im, const __nv_bfloat16* gate, const SingleBias& bias, __nv_bfloat16* tb,
                const __nv_bfloat16* mask, __nv_bfloat16* out, int BB, int N, int nq, int H, int d, float inf,
                int rows_per_bias, bool spread, cudaStream_t st);

}  // namespace fast
}  // namespace of3
