// Operand-image layout shared by the producers (linear.cu) and the reader (fast_single_attn.cu) of the single-track
// attention: q [bh][query tile of 128][128][KD], k [bh][key block of 32][32][KD], v [bh][key block][DV][32 keys].
#pragma once
#include "common.cuh"

namespace of3 {
namespace fast {

constexpr int kSingleBQ = 128;  // queries per tile
constexpr int kSingleBK = 32;   // keys per block
template <int D>
struct SingleImage {
    static constexpr int kKD = (D <= 32) ? 32 : 64;  // K dim of Q K^T after zero padding
    static constexpr int kDV = (D <= 32) ? 32 : 48;  // rows of the V^T tile = columns of O
};

#ifdef __CUDACC__
// 16-byte chunk c of row r inside a K-major tile with rows of KD bf16: 64-byte rows use the 64-byte swizzle,
// 128-byte rows the 128-byte swizzle (what the tcgen05 descriptors of umma.cuh expect).
template <int KD>
__device__ __forceinline__ uint32_t single_chunk_off(int r, int c) {
    return KD == 32 ? (uint32_t)(r * 64 + ((c ^ ((r >> 1) & 3)) << 4)) : (uint32_t)(r * 128 + ((c ^ (r & 7)) << 4));
}
#endif

}  // namespace fast
}  // namespace of3
