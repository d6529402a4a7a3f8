// Pair-bias projections of several layers of one pair tensor in one pass.
#pragma once
#include "common.cuh"

namespace of3 {
namespace fast {

constexpr int kMaxBiasLayers = 24;   // per launch: 3 groups of 128 output channels
struct BiasLayer {
    const __nv_bfloat16 *ln_w, *ln_b, *w;   // LayerNorm weight and bias (or null), linear_z.weight [16][128]
};
// z [B][N][N][128] -> the attention kernel's bias image of each layer, tiles [layer][B * 16][ceil(N / 32)][N][32] bf16
int pair_bias_tiles(const __nv_bfloat16* z, const BiasLayer* layer, int layers, __nv_bfloat16* tiles, long long B, int N,
                    cudaStream_t st);

}  // namespace fast
}  // namespace of3
