// K-quant matrices against token rows (kernels_kqt.cu): the activation image they read and the matrix handle.
//
// Activation images are written as operand B of the products, so that one bulk copy brings a superblock of up to 32 tokens.  Tokens
// come in chunks of at most 32 (rows 32 c .. of a prompt tile, or tokens of one expert in the order of a KqPlan); a chunk of n has room
// for kq_cap(n) tokens.  Block (chunk, superblock), KIMG_BLOCK bytes apart: [34 pieces][kq_cap(n) tokens][16 bytes].  Piece 4 j + i:
// values 8 i .. 8 i + 7 of sub-block j (32 values) as halves in the order 0 2 1 3 4 6 5 7 - the order in which two 32-bit masks pull a
// word's nibbles apart.  Pieces 32, 33: the eight 32-sums bs = 64 h + l, l in [-32, 31], as l[0..7] and h[0..7] (halves are exact up to
// 2048, a sum has 13 bits).  The scales of block (chunk, superblock): 32 floats.
#pragma once
#include <cuda.h>
#include "brrr_kq.cuh"

namespace brrr {

constexpr int KT_NT = 32;                                 // tokens per chunk
constexpr int KIMG_BLOCK = 34 * KT_NT * 16;
constexpr int KT_MAXCHUNK = 512;
__host__ __device__ __forceinline__ int kq_cap(int n) { return n <= 8 ? 8 : n <= 16 ? 16 : KT_NT; }
__host__ __device__ __forceinline__ size_t kimg_bytes(int chunks, int nsb) { return (size_t)chunks * nsb * KIMG_BLOCK; }

// Tokens of every expert, cut into chunks: chunk c serves expert e[c] with n[c] entries (token * topk + slot) ent[32 c ..].
struct KqPlan {
    int nchunk;
    int e[KT_MAXCHUNK], n[KT_MAXCHUNK];
    int ent[KT_MAXCHUNK * KT_NT];
};

// where token `t` of a chunk keeps superblock sb
struct KimgSlot {
    uint8_t *p;      // its 16 bytes of piece 0
    int step;        // bytes from piece to piece
    float *ys;
};
__device__ __forceinline__ KimgSlot kimg_slot(uint8_t *img, float *ys, int chunk, int n, int i, int nsb, int sb) {
    const size_t b = (size_t)chunk * nsb + sb;
    return KimgSlot{img + b * KIMG_BLOCK + i * 16, kq_cap(n) * 16, ys + b * KT_NT + i};
}
// row t of a tile of `rows` rows
__device__ __forceinline__ KimgSlot kimg_row(uint8_t *img, float *ys, int t, int rows, int nsb, int sb) {
    return kimg_slot(img, ys, t / KT_NT, min(KT_NT, rows - t / KT_NT * KT_NT), t % KT_NT, nsb, sb);
}

// Q8_K quantisation of one superblock by one warp (the arithmetic of warp_quant_q8k), straight into the image.
__device__ __forceinline__ void warp_quant_q8k_image(const float (&v)[8], int lane, const KimgSlot &o) {
    uint32_t b[2];
    int sum, q[8];
    const float sc = warp_q8k(v, b, sum);
#pragma unroll
    for (int i = 0; i < 8; i++) q[i] = (int)(int8_t)(b[i >> 2] >> (8 * (i & 3)));
    const int order[8] = {0, 2, 1, 3, 4, 6, 5, 7};
    uint32_t w[4];
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const __half2 h = __halves2half2(__int2half_rn(q[order[2 * i]]), __int2half_rn(q[order[2 * i + 1]]));
        w[i] = *reinterpret_cast<const uint32_t *>(&h);
    }
    *reinterpret_cast<uint4 *>(o.p + lane * o.step) = make_uint4(w[0], w[1], w[2], w[3]);
    sum += __shfl_xor_sync(0xffffffffu, sum, 1);
    sum += __shfl_xor_sync(0xffffffffu, sum, 2);
    const int h = (sum + 32) >> 6, l = sum - 64 * h;
    if ((lane & 3) < 2) *reinterpret_cast<__half *>(o.p + (32 + (lane & 1)) * o.step + 2 * (lane >> 2)) = __int2half_rn((lane & 1) ? h : l);
    if (lane == 0) *o.ys = sc;
}

// K and V of a layer, [kv head][position][128], and as tensors for the decode attention's copies
struct alignas(64) QwCache {
    CUtensorMap km, vm;
    float *k, *v;
};

// A matrix of 128-row tiles: its bytes as tensors [row][byte] for the copies (Q4_K: boxes of 128 x 144; Q6_K planes: 128 x 128, 64, 16).
struct alignas(64) KqtMat {
    CUtensorMap map[3];
    int type, rows, cols;
};

}  // namespace brrr
