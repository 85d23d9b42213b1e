// K-quant matrices against token rows (kernels_kqt.cu): the activation image they read and the matrix handle.
//
// Activation image of a row, 544 bytes per superblock: 256 halves, then sixteen for the minima.  Halves: sub-block j (32 values) at
// 64 j, in groups of eight values in the order 0 2 1 3 4 6 5 7 - the order in which two 32-bit masks pull a word's nibbles apart.
// Minima: the eight 32-sums bs = 64 h + l with l in [-32, 31] as l[0..7], h[0..7] (both exact halves; a sum has 13 bits).
#pragma once
#include <cuda.h>
#include "brrr_kq.cuh"

namespace brrr {

constexpr int KIMG_SB = 544;

// Q8_K quantisation of one superblock by one warp (the arithmetic of warp_quant_q8k), straight into the image.
__device__ __forceinline__ void warp_quant_q8k_image(const float (&v)[8], int lane, uint8_t *img_sb, float *s) {
    float amax = 1e-12f;
#pragma unroll
    for (int i = 0; i < 8; i++) amax = fmaxf(amax, fabsf(v[i]));
#pragma unroll
    for (int o = 16; o; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
    const float sc = __fdiv_rn(amax, 127.0f);
    int q[8], sum = 0;
#pragma unroll
    for (int i = 0; i < 8; i++) { q[i] = brrr_q8_round(v[i], sc); sum += q[i]; }
    const int order[8] = {0, 2, 1, 3, 4, 6, 5, 7};
    uint32_t w[4];
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const __half2 h = __halves2half2(__int2half_rn(q[order[2 * i]]), __int2half_rn(q[order[2 * i + 1]]));
        w[i] = *reinterpret_cast<const uint32_t *>(&h);
    }
    *reinterpret_cast<uint4 *>(img_sb + lane * 16) = make_uint4(w[0], w[1], w[2], w[3]);
    sum += __shfl_xor_sync(0xffffffffu, sum, 1);
    sum += __shfl_xor_sync(0xffffffffu, sum, 2);
    const int h = (sum + 32) >> 6, l = sum - 64 * h;
    if ((lane & 3) < 2) *reinterpret_cast<__half *>(img_sb + 512 + (lane & 1) * 16 + 2 * (lane >> 2)) = __int2half_rn((lane & 1) ? h : l);
    if (lane == 0) *s = sc;
}

// A matrix of 128-row tiles: its bytes as tensors [row][byte] for the copies (Q4_K: boxes of 128 x 144; Q6_K planes: 128 x 128, 64, 16).
struct alignas(64) KqtMat {
    CUtensorMap map[3];
    int type, rows, cols;
};

}  // namespace brrr
