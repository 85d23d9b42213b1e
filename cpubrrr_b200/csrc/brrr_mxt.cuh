// Operand B of the fp4 tensor-core expert matvecs (kernels_mxt.cu): the digit planes of a Q8
// activation, written by whichever kernel quantises the activation.
//
// An activation byte x in [-127, 127] is 64 a + 8 b + c with digits in [-4, 4]; half a digit is an e2m1 value and its code is the digit's
// magnitude with the sign in bit 3.  In memory, per 32-block 48 bytes: for digit plane t = 0..2 (a, b, c) and lane chain j one
// word at t * 16 + j * 4, byte i holding the codes of positions 4 j + i (low nibble) and 16 + 4 j + i (high nibble).
//
// Operand image of one block pair (768 bytes of shared memory): for kc = 0, 1 (the block of the pair), column n = h * 12 + t * 4 + q * 2 + i
// (lane chain j = 2 h + i, plane t, q = block of the pair): 16 bytes at kc * 384 + n * 16, byte i holding the codes of positions i and
// 16 + i.  A column is non-zero only for kc = q and bytes 4 j .. 4 j + 3: the digits' words spread over a zeroed image.
#pragma once
#include "brrr_dev.cuh"

namespace brrr {

constexpr int XT_N = 24;                 // MMA N: 3 digit planes x 2 blocks x 4 lanes
constexpr int XT_B_PAIR = XT_N * 32;     // operand B bytes per block pair
constexpr int XT_DIG_BLOCK = 48;         // bytes of digits per 32-block

// e2m1 codes of half the digits of x: a | b << 4 | c << 8
__device__ __forceinline__ uint32_t xt_digits(int x) {
    const int a = (x + 36 + 256) / 64 - 4;
    const int r = x - 64 * a;            // -36 .. 27
    const int b = (r + 4 + 64) / 8 - 8;
    const int c = r - 8 * b;             // -4 .. 3
    auto code = [](int v) -> uint32_t { return v < 0 ? (uint32_t)-v | 8u : (uint32_t)v; };
    return code(a) | (code(b) << 4) | (code(c) << 8);
}

// One 32-block held one quantised value per lane: writes the block's 12 words.
// Must be called by all 32 lanes.
__device__ __forceinline__ void xt_emit_digits(int qv, int lane, int b, uint8_t *dig) {
    const uint32_t codes = xt_digits(qv);
    uint32_t *out = reinterpret_cast<uint32_t *>(dig + (size_t)b * XT_DIG_BLOCK) + ((lane & 15) >> 2);
#pragma unroll
    for (int t = 0; t < 3; t++) {
        const uint32_t nib = (codes >> (4 * t)) & 15u;
        const uint32_t other = __shfl_xor_sync(0xffffffffu, nib, 16);
        uint32_t w = (nib | (other << 4)) << (8 * (lane & 3));     // lanes < 16: byte i = code(i) | code(16 + i) << 4
        w |= __shfl_xor_sync(0xffffffffu, w, 1);
        w |= __shfl_xor_sync(0xffffffffu, w, 2);
        if (lane < 16 && (lane & 3) == 0) out[t * 4] = w;
    }
}

// Plane t of block b (i = 3 b + t) as read from the digits: its four words into the operand image.
__device__ __forceinline__ void xt_spread_digits(uint4 w, int i, unsigned char *bimg) {
    const int b = i / 3, t = i - 3 * b, q = b & 1;
    uint32_t *o = reinterpret_cast<uint32_t *>(bimg + (size_t)(b >> 1) * XT_B_PAIR + q * (XT_B_PAIR / 2) + t * 64 + q * 32);
    o[0] = w.x; o[5] = w.y; o[50] = w.z; o[55] = w.w;              // lane j: (j >> 1) * 192 + (j & 1) * 16 + 4 j bytes on
}

}  // namespace brrr
