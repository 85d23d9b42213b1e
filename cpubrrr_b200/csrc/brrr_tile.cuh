// Activation images of the token-row matmuls (kernels_tile.cu): the quantised activation of a row in
// the number format and order of tcgen05 operand B, written once by whichever kernel quantises it.
// Per block pair p (32-blocks 2p and 2p + 1):
//
//   half image (Q8 matrices, kind::f16), 128 bytes:        [lane chain j][block q of the pair][8 halves]
//     the 8 values of lane j in block q: elements 4j .. 4j+3, then 16+4j .. 16+4j+3 (the order of a Q8 unit)
//   plane image (MXFP4 matrices, kind::f8f6f4), 256 bytes: [lane chain j][plane][block q][16 bytes]
//     an activation byte x = 16 a + c with a, c in [-8, 8]; plane 0 holds 32 a, plane 1 holds 2 c (twice the value,
//     so a sum with the true e2m1 weights is the sum with the doubled ones), both exact in e4m3; the 8 values in the
//     nibble order of a weight word (4j, 16+4j, 4j+1, 16+4j+1, ...) at bytes 8q .. 8q+7 of the 16, zero elsewhere: the
//     row of operand B for (token, block q).  Producers write the values only; the rest is zero from the allocation.
#pragma once
#include "brrr_dev.cuh"

#include <cuda_fp16.h>

namespace brrr {

enum { TI_HALF = 0, TI_PLANES = 1 };
__host__ __device__ constexpr int ti_pair(int image) { return image == TI_HALF ? 128 : 256; }

// A 32-block held one quantised value per lane: its 32 (x 2) values of image `img` of the row.
template <int IMG>
__device__ __forceinline__ void ti_emit_block(int qv, int lane, int b, uint8_t *img) {
    const int j = (lane & 15) >> 2, q = b & 1;
    uint8_t *base = img + (size_t)(b >> 1) * ti_pair(IMG);
    if (IMG == TI_HALF) {
        *reinterpret_cast<__half *>(base + j * 32 + q * 16 + ((lane & 3) + (lane >= 16 ? 4 : 0)) * 2) = __int2half_rn(qv);
    } else {
        const int a = (qv + 8) >> 4, c = qv - 16 * a;
        unsigned short codes;      // plane 0 in the upper byte
        asm("cvt.rn.satfinite.e4m3x2.f32 %0, %1, %2;" : "=h"(codes) : "f"((float)(32 * a)), "f"((float)(2 * c)));
        uint8_t *o = base + j * 64 + q * 24 + 2 * (lane & 3) + (lane >> 4);      // q * 16 + q * 8
        o[0] = (uint8_t)(codes >> 8);
        o[32] = (uint8_t)codes;
    }
}

}  // namespace brrr
