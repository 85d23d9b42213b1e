// Warp-level building blocks of the K-quant path (Q8_K activations, Q4_K / Q6_K weight rows in the
// GGUF byte layout), shared by the stage kernels and the qwen3moe decode kernels.
//
// Reference arithmetic (src/bin/engine_qwen2.rs:84-114, 164-200, 287-300): per 256-value
// superblock the dot is an exact integer sum scaled once, sumf += (ys*d)*acc - (ys*dmin)*mint
// (Q4_K) or sumf += (ys*d)*acc (Q6_K), unfused, superblocks in order.  The integer sum is
// order-free, so one warp owns a row, its lanes split each superblock (one 32-bit word of nibbles
// per lane for Q4_K, one byte pair of each field for Q6_K), the partial sums meet in a warp
// integer reduction and every lane carries the same float chain.
#pragma once
#include "brrr_dev.cuh"
#include "brrr_tma.cuh"

#include <cuda_fp16.h>

namespace brrr {

__device__ __forceinline__ float half_bits_to_f32(uint32_t h) { return __half2float(__ushort_as_half((unsigned short)h)); }

// byte i (0..11) of the 12 packed scale bytes held in three words
__device__ __forceinline__ uint32_t k4_byte(uint32_t s0, uint32_t s1, uint32_t s2, int i) {
    uint32_t w = i < 4 ? s0 : (i < 8 ? s1 : s2);
    return (w >> ((i & 3) * 8)) & 0xffu;
}

// 6-bit scale and min of sub-block j (src/bin/engine_qwen2.rs:52-56)
__device__ __forceinline__ void k4_scale_min(uint32_t s0, uint32_t s1, uint32_t s2, int j, int &sc, int &mn) {
    if (j < 4) {
        sc = (int)(k4_byte(s0, s1, s2, j) & 63u);
        mn = (int)(k4_byte(s0, s1, s2, j + 4) & 63u);
    } else {
        uint32_t hi = k4_byte(s0, s1, s2, j + 4);
        sc = (int)((hi & 0xFu) | ((k4_byte(s0, s1, s2, j - 4) >> 6) << 4));
        mn = (int)((hi >> 4) | ((k4_byte(s0, s1, s2, j) >> 6) << 4));
    }
}

// Q8_K quantisation of one 256-value superblock by one warp: lane l holds values 8l..8l+7 (so
// sub-block j is lanes 4j..4j+3).  Writes the quants, the scale and the eight 32-sums.
__device__ __forceinline__ void warp_quant_q8k(const float (&v)[8], int lane, int8_t *q, float *s, int32_t *bsum) {
    float amax = 1e-12f;
#pragma unroll
    for (int i = 0; i < 8; i++) amax = fmaxf(amax, fabsf(v[i]));
#pragma unroll
    for (int o = 16; o; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
    float sc = __fdiv_rn(amax, 127.0f);
    int qi[8], sum = 0;
#pragma unroll
    for (int i = 0; i < 8; i++) { qi[i] = brrr_q8_round(v[i], sc); sum += qi[i]; }
    uint32_t lo = (qi[0] & 0xff) | ((qi[1] & 0xff) << 8) | ((qi[2] & 0xff) << 16) | ((uint32_t)(qi[3] & 0xff) << 24);
    uint32_t hi = (qi[4] & 0xff) | ((qi[5] & 0xff) << 8) | ((qi[6] & 0xff) << 16) | ((uint32_t)(qi[7] & 0xff) << 24);
    *reinterpret_cast<uint2 *>(q + lane * 8) = make_uint2(lo, hi);
    sum += __shfl_xor_sync(0xffffffffu, sum, 1);
    sum += __shfl_xor_sync(0xffffffffu, sum, 2);
    if ((lane & 3) == 0) bsum[lane >> 2] = sum;
    if (lane == 0) *s = sc;
}

// Q4_K row x Q8_K activation by one warp; the result is valid in every lane.  Superblock: f16 d,
// f16 dmin, 12 scale bytes, 128 nibble bytes.  Lane l owns word l of the nibble bytes: bytes
// 4l..4l+3 of 32-byte chunk jj = l/8, whose low nibbles belong to sub-block 2jj and high nibbles to
// sub-block 2jj+1.  dbg (nullable): {scaled quant sum, min sum} per superblock.
__device__ __forceinline__ float q4k_row_dot(const uint8_t *row, int nsb, const int8_t *xq, const float *ys, const int32_t *bsum,
                                             int lane, int32_t *dbg = nullptr) {
    const uint32_t *b32 = reinterpret_cast<const uint32_t *>(row);
    const int jj = lane >> 3, k4 = (lane & 7) * 4;
    float sumf = 0.0f;
#pragma unroll 4
    for (int sb = 0; sb < nsb; sb++, b32 += 36) {
        uint32_t dd = __ldg(b32), s0 = __ldg(b32 + 1), s1 = __ldg(b32 + 2), s2 = __ldg(b32 + 3);
        uint32_t qv = __ldg(b32 + 4 + lane);
        int x0 = *reinterpret_cast<const int *>(xq + (sb * 8 + 2 * jj) * 32 + k4);
        int x1 = *reinterpret_cast<const int *>(xq + (sb * 8 + 2 * jj + 1) * 32 + k4);
        int sc0, mn0, sc1, mn1;
        k4_scale_min(s0, s1, s2, 2 * jj, sc0, mn0);
        k4_scale_min(s0, s1, s2, 2 * jj + 1, sc1, mn1);
        int a = __dp4a((int)(qv & 0x0F0F0F0Fu), x0, 0) * sc0 + __dp4a((int)((qv >> 4) & 0x0F0F0F0Fu), x1, 0) * sc1;
        int mt = 0;
        if (lane < 8) {
            int scj, mnj;
            k4_scale_min(s0, s1, s2, lane, scj, mnj);
            mt = mnj * bsum[sb * 8 + lane];
        }
        a = __reduce_add_sync(0xffffffffu, a);
        mt = __reduce_add_sync(0xffffffffu, mt);
        float ysb = ys[sb];
        float d = half_bits_to_f32(dd & 0xffffu), dmin = half_bits_to_f32(dd >> 16);
        float pos = __fmul_rn(__fmul_rn(ysb, d), (float)a);
        float neg = __fmul_rn(__fmul_rn(ysb, dmin), (float)mt);
        sumf = __fadd_rn(sumf, __fsub_rn(pos, neg));
        if (dbg && lane == 0) { dbg[sb * 2] = a; dbg[sb * 2 + 1] = mt; }
    }
    return sumf;
}

// Q6_K row x Q8_K activation by one warp; the result is valid in every lane.  Superblock: 128 B low
// nibbles (ql), 64 B 2-bit fields (qh), 16 int8 scales, f16 d; 210 bytes, so rows are only 2-byte
// aligned and fields are read as byte pairs.  Lane (h = l/16, pp = l%16) owns positions p = 2pp,
// 2pp+1 of half h: with la = ql[64h+p], lb = ql[64h+32+p], hv = qh[32h+p] the four values at
// 128h + {0,32,64,96} + p are (la&15 | (hv&3)<<4), (lb&15 | (hv>>2&3)<<4), (la>>4 | (hv>>4&3)<<4),
// (lb>>4 | (hv>>6)<<4), each - 32.  dbg (nullable): the integer accumulator per superblock.
__device__ __forceinline__ float q6k_row_dot(const uint8_t *row, int nsb, const int8_t *xq, const float *ys, int lane, int32_t *dbg = nullptr) {
    const uint8_t *b = row;
    const int h = lane >> 4, pp = lane & 15;
    float sumf = 0.0f;
#pragma unroll 2
    for (int sb = 0; sb < nsb; sb++, b += 210) {
        uint32_t la2 = __ldg(reinterpret_cast<const unsigned short *>(b + h * 64 + 2 * pp));
        uint32_t lb2 = __ldg(reinterpret_cast<const unsigned short *>(b + h * 64 + 32 + 2 * pp));
        uint32_t hv2 = __ldg(reinterpret_cast<const unsigned short *>(b + 128 + h * 32 + 2 * pp));
        const signed char *scp = reinterpret_cast<const signed char *>(b + 192) + h * 8 + (pp >> 3);
        const int8_t *xb = xq + sb * 256 + h * 128 + 2 * pp;
        int a = 0;
#pragma unroll
        for (int qd = 0; qd < 4; qd++) {
            uint32_t x2 = *reinterpret_cast<const unsigned short *>(xb + qd * 32);
            int part = 0;
#pragma unroll
            for (int e = 0; e < 2; e++) {
                uint32_t la = (la2 >> (8 * e)) & 0xffu, lb = (lb2 >> (8 * e)) & 0xffu, hv = (hv2 >> (8 * e)) & 0xffu;
                uint32_t lowsrc = (qd & 1) ? lb : la;
                uint32_t low = (qd & 2) ? (lowsrc >> 4) : (lowsrc & 0xFu);
                uint32_t high = (hv >> (2 * qd)) & 3u;
                int val = (int)(low | (high << 4)) - 32;
                int xv = (int)(signed char)((x2 >> (8 * e)) & 0xffu);
                part += val * xv;
            }
            a += part * (int)__ldg(scp + qd * 2);
        }
        a = __reduce_add_sync(0xffffffffu, a);
        float d = half_bits_to_f32(__ldg(reinterpret_cast<const unsigned short *>(b + 208)));
        sumf = __fadd_rn(sumf, __fmul_rn(__fmul_rn(ys[sb], d), (float)a));
        if (dbg && lane == 0) dbg[sb] = a;
    }
    return sumf;
}

// A K-quant matrix on the device, type 12 (Q4_K) or 14 (Q6_K).  Q4_K rows stay in the GGUF byte
// layout (144-byte superblocks, 16-byte aligned).  Q6_K rows are either in the GGUF layout (210-byte
// superblocks, 2-byte aligned: planes == 0) or re-laid at load time into four aligned planes per row
// (planes == 1): ql [nsb][128] | qh [nsb][64] | scales [nsb][16] | d [nsb] f16, padded to 16 bytes -
// a byte permutation, so every integer of the dot is unchanged.
struct KMatDev {
    const uint8_t *p;
    int type, rows, cols;
    int planes;
    __host__ __device__ size_t bpr() const {
        const size_t nsb = (size_t)(cols / 256);
        if (type == 12) return nsb * 144;
        return planes ? nsb * 208 + ((nsb * 2 + 15) & ~(size_t)15) : nsb * 210;
    }
};
// bytes of a row in the GGUF layout (the algorithmic figure, whatever the device layout)
__host__ __device__ __forceinline__ size_t kq_gguf_row_bytes(int type, int cols) { return (size_t)(cols / 256) * (type == 12 ? 144 : 210); }
__host__ __device__ __forceinline__ size_t q6k_plane_row_bytes(int nsb) { return (size_t)nsb * 208 + (((size_t)nsb * 2 + 15) & ~(size_t)15); }

// The qwen3moe RMS norm sums squares in 12 contiguous slices (the reference's 12 workers), each
// serially and unfused, and adds the partial sums in worker order (engine_qwen2.rs:15, 453-465).
constexpr int QW_NT = 12;
// worker w's contiguous slice of n items (engine_qwen2.rs:246-252)
__device__ __forceinline__ void qw_slice(int w, int n, int &a, int &b) {
    int base = n / QW_NT, rem = n % QW_NT;
    a = w * base + min(w, rem);
    b = a + base + (w < rem ? 1 : 0);
}

// ---------------------------------------------------------------- rows in shared memory (decode kernels)
// Eight values per lane of a superblock, one warp -> quants packed four to a word, their sum, the scale (the arithmetic of warp_quant_q8k).
// The quotient v / scale is formed as v (127 / amax) with an approximate reciprocal, which is within 1e-4 of it; rounding by adding
// 1.5 x 2^23 then gives the same integer unless the value lies that close to a half, where (and for scales out of range) the lane divides.
// Every lane returns the same scale.  350 cycles with eight warps at work; dividing each value: 1220.
__device__ __forceinline__ float warp_q8k(const float (&v)[8], uint32_t (&w)[2], int &sum) {
    float m = 1e-12f;
#pragma unroll
    for (int i = 0; i < 8; i++) m = fmaxf(m, fabsf(v[i]));
    const float amax = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(m)));      // not negative: ordered as integers
    const float sc = __fdiv_rn(amax, 127.0f), inv = __fdividef(127.0f, amax);
    uint32_t b[8], unsure = 0;
#pragma unroll
    for (int i = 0; i < 8; i++) {
        const float t = __fmul_rn(v[i], inv), r = __fadd_rn(t, 12582912.0f);
        b[i] = __float_as_uint(r);
        unsure |= (uint32_t)!(fabsf(__fsub_rn(t, __fsub_rn(r, 12582912.0f))) < 0.4999f) << i;
    }
    if (!(amax < 1e30f)) unsure = 0xFFu;
    if (unsure) {
#pragma unroll
        for (int i = 0; i < 8; i++) if (unsure & (1u << i)) b[i] = (uint32_t)brrr_q8_round(v[i], sc);
    }
#pragma unroll
    for (int i = 0; i < 2; i++) w[i] = __byte_perm(__byte_perm(b[4 * i], b[4 * i + 1], 0x0040), __byte_perm(b[4 * i + 2], b[4 * i + 3], 0x0040), 0x5410);
    sum = __dp4a((int)w[0], 0x01010101, __dp4a((int)w[1], 0x01010101, 0));
    return sc;
}
// Q8_K activation of the decode kernels: quants, one scale per 256 values, and the sums of every 16 quants (Q4_K minima need pairs of
// them, the -32 of Q6_K each).  CHUNK: bytes from one run of 64 quants to the next - 64 in global memory, 80 in shared memory, where four
// lanes per superblock then read theirs from different banks.
constexpr int KQ_SM_CHUNK = 80;
template <int CHUNK>
__device__ __forceinline__ void warp_quant_q8k16(const float (&v)[8], int lane, int sb, int8_t *q, float *s, int32_t *b16) {
    uint32_t w[2];
    int sum;
    const float sc = warp_q8k(v, w, sum);
    *reinterpret_cast<uint2 *>(q + (4 * sb + (lane >> 3)) * CHUNK + (lane & 7) * 8) = make_uint2(w[0], w[1]);
    sum += __shfl_xor_sync(0xffffffffu, sum, 1);
    if (!(lane & 1)) b16[sb * 16 + (lane >> 1)] = sum;
    if (lane == 0) s[sb] = sc;
}

// Four lanes own one superblock (a warp covers eight at a time); lane l4 holds the 64 activations that meet its 32 bytes of quants.
//   Q4_K: nibble bytes 32 l4 ..: x[0..1] for the low nibbles (sub-block 2 l4), x[2..3] for the high (2 l4 + 1); b[0], b[1] their sums
//   Q6_K planes: ql bytes 32 l4 ..: x[0..1] / x[2..3] for the low / high nibbles; b: 32 times the sums of the four sixteens.  Lanes with
//   sw = 1 (every other superblock) hold and read the two sixteens of each in the other order, so that neighbours do not meet in a bank.
struct KAct { int4 x[4]; int b[4]; };
template <int TYPE, int CHUNK>
__device__ __forceinline__ void kact_load(const int8_t *q, const int32_t *b16, int sb, int l4, int sw, KAct &a) {
    b16 += sb * 16;
    if (TYPE == 12) {
        const int4 *p = reinterpret_cast<const int4 *>(q + (4 * sb + l4) * CHUNK);
        a.x[0] = p[0]; a.x[1] = p[1]; a.x[2] = p[2]; a.x[3] = p[3];
        const int4 s = *reinterpret_cast<const int4 *>(b16 + 4 * l4);
        a.b[0] = s.x + s.y; a.b[1] = s.z + s.w; a.b[2] = a.b[3] = 0;
    } else {
        const int h = l4 >> 1, b = l4 & 1;
        const int4 *p = reinterpret_cast<const int4 *>(q + (4 * sb + 2 * h) * CHUNK + 32 * b), *r = reinterpret_cast<const int4 *>(q + (4 * sb + 2 * h + 1) * CHUNK + 32 * b);
        a.x[0] = p[sw]; a.x[1] = p[sw ^ 1]; a.x[2] = r[sw]; a.x[3] = r[sw ^ 1];
        const int2 s = *reinterpret_cast<const int2 *>(b16 + 8 * h + 2 * b), t = *reinterpret_cast<const int2 *>(b16 + 8 * h + 4 + 2 * b);
        a.b[0] = 32 * (sw ? s.y : s.x); a.b[1] = 32 * (sw ? s.x : s.y); a.b[2] = 32 * (sw ? t.y : t.x); a.b[3] = 32 * (sw ? t.x : t.y);
    }
}
__device__ __forceinline__ int dp4a_us(uint32_t u, int s, int c) {      // unsigned bytes x signed bytes
    int r;
    asm("dp4a.u32.s32 %0, %1, %2, %3;" : "=r"(r) : "r"(u), "r"(s), "r"(c));
    return r;
}

__device__ __forceinline__ uint32_t kq_lds16(uint32_t a) {
    unsigned short r;
    asm volatile("ld.shared.u16 %0, [%1];" : "=h"(r) : "r"(a));
    return r;
}

// Term of a superblock in the row sum: (ys d) a - (ys dmin) mt for Q4_K, (ys d) a for Q6_K, every product rounded on its own as in
// q4k_row_dot / q6k_row_dot; valid in the first of its four lanes.  row: address of the matrix row in shared memory.  All 32 lanes must
// call it.  About 100 instructions; 120 cycles per warp and scheduler.
template <int TYPE>
__device__ __forceinline__ float kq_term(int nsb, uint32_t row, int sb, const KAct &x, float ys, int l4, int sw) {
    const uint32_t M4 = 0x0F0F0F0Fu;
    const int lo4[8] = {x.x[0].x, x.x[0].y, x.x[0].z, x.x[0].w, x.x[1].x, x.x[1].y, x.x[1].z, x.x[1].w};
    const int hi4[8] = {x.x[2].x, x.x[2].y, x.x[2].z, x.x[2].w, x.x[3].x, x.x[3].y, x.x[3].z, x.x[3].w};
    if (TYPE == 12) {
        const uint32_t p = row + sb * 144;
        const uint4 h = lds128(p), u = lds128(p + 16 + 32 * l4), v = lds128(p + 32 + 32 * l4);
        const bool upper = l4 >= 2;                  // sub-blocks 4 .. 7: six bits in two fields
        const uint32_t sc = (upper ? (h.w & M4) | ((h.y >> 2) & 0x30303030u) : h.y & 0x3F3F3F3Fu) >> ((l4 & 1) * 16);
        const uint32_t mn = (upper ? ((h.w >> 4) & M4) | ((h.z >> 2) & 0x30303030u) : h.z & 0x3F3F3F3Fu) >> ((l4 & 1) * 16);
        const uint32_t w[8] = {u.x, u.y, u.z, u.w, v.x, v.y, v.z, v.w};
        int lo[2] = {0, 0}, hi[2] = {0, 0};
#pragma unroll
        for (int i = 0; i < 8; i++) { lo[i & 1] = dp4a_us(w[i] & M4, lo4[i], lo[i & 1]); hi[i & 1] = dp4a_us(w[i] & 0xF0F0F0F0u, hi4[i], hi[i & 1]); }      // hi: sixteen times its sum
        const int a = (lo[0] + lo[1]) * (int)(sc & 0xFFu) + ((hi[0] + hi[1]) >> 4) * (int)((sc >> 8) & 0xFFu);
        const int m = (int)(mn & 0xFFu) * x.b[0] + (int)((mn >> 8) & 0xFFu) * x.b[1];
        // two shuffles for both sums: even lanes keep a, odd lanes the minima
        const bool odd = l4 & 1;
        int r = odd ? m : a;
        r += __shfl_xor_sync(0xffffffffu, odd ? a : m, 1);
        r += __shfl_xor_sync(0xffffffffu, r, 2);
        const float f = __fmul_rn(__fmul_rn(ys, half_bits_to_f32(odd ? h.x >> 16 : h.x & 0xffffu)), (float)r);
        return __fsub_rn(f, __shfl_xor_sync(0xffffffffu, f, 1));
    }
    const int h = l4 >> 1, b = l4 & 1;
    const uint32_t lp = row + sb * 128 + 32 * l4, up = row + nsb * 128 + sb * 64 + 32 * h;
    const int o = sw * 16;
    const uint4 l0 = lds128(lp + o), l1 = lds128(lp + 16 - o), u0 = lds128(up + o), u1 = lds128(up + 16 - o);
    const uint2 s8 = lds64(row + nsb * 192 + sb * 16 + 8 * h);
    const float d = half_bits_to_f32(kq_lds16(row + nsb * 208 + sb * 2));
    const uint32_t order = (b ? 0x32u : 0x10u), pick = sw ? (order >> 4) | ((order & 15u) << 4) : order;
    const uint32_t slo = __byte_perm(s8.x, 0, pick), shi = __byte_perm(s8.y, 0, pick), M2 = 0x30303030u;
    const uint32_t l[8] = {l0.x, l0.y, l0.z, l0.w, l1.x, l1.y, l1.z, l1.w}, u[8] = {u0.x, u0.y, u0.z, u0.w, u1.x, u1.y, u1.z, u1.w};
    int a = 0;
#pragma unroll
    for (int g = 0; g < 2; g++) {                    // sixteen values share a scale
        int lo = 0, hi = 0;
#pragma unroll
        for (int i = 4 * g; i < 4 * g + 4; i++) {
            const uint32_t t = u[i] >> (2 * b);      // 2-bit fields: 0 and 4, or 2 and 6
            lo = dp4a_us((l[i] & M4) | ((t << 4) & M2), lo4[i], lo);
            hi = dp4a_us(((l[i] >> 4) & M4) | (t & M2), hi4[i], hi);
        }
        a += (lo - x.b[g]) * (int)(signed char)(slo >> (8 * g)) + (hi - x.b[2 + g]) * (int)(signed char)(shi >> (8 * g));
    }
    a += __shfl_xor_sync(0xffffffffu, a, 1);
    a += __shfl_xor_sync(0xffffffffu, a, 2);
    return __fmul_rn(__fmul_rn(ys, d), (float)a);
}

// Sum of squares of x[lo .. hi) in order by one thread, x 16-byte aligned: whole float4s, what lies outside the range counted as +0 (which
// changes no sum), the next sixteen values read while sixteen squares are added (5 cycles a value; scalar reads 8).
__device__ __forceinline__ float chain_squares(const float *x, int lo, int hi) {
    const float4 *p = reinterpret_cast<const float4 *>(x) + (lo >> 2);
    const int head = lo & 3, n = hi - (lo & ~3), n4 = (n + 3) >> 2;      // values from the aligned start, float4s
    float4 b[4];
    float ps = 0.0f;
#pragma unroll
    for (int k = 0; k < 4; k++) b[k] = p[min(k, n4 - 1)];
    if (head > 0) b[0].x = 0.0f;
    if (head > 1) b[0].y = 0.0f;
    if (head > 2) b[0].z = 0.0f;
    int i = 0;                               // float4s that b starts at
#pragma unroll 2
    for (; i + 4 < n4; i += 4) {
        float s[16];
#pragma unroll
        for (int k = 0; k < 4; k++) {
            s[4 * k] = __fmul_rn(b[k].x, b[k].x); s[4 * k + 1] = __fmul_rn(b[k].y, b[k].y);
            s[4 * k + 2] = __fmul_rn(b[k].z, b[k].z); s[4 * k + 3] = __fmul_rn(b[k].w, b[k].w);
        }
#pragma unroll
        for (int k = 0; k < 4; k++) b[k] = p[min(i + 4 + k, n4 - 1)];
#pragma unroll
        for (int k = 0; k < 16; k++) ps = __fadd_rn(ps, s[k]);
    }
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const int at = (i + k) * 4;
        if (at < n) ps = __fadd_rn(ps, __fmul_rn(b[k].x, b[k].x));
        if (at + 1 < n) ps = __fadd_rn(ps, __fmul_rn(b[k].y, b[k].y));
        if (at + 2 < n) ps = __fadd_rn(ps, __fmul_rn(b[k].z, b[k].z));
        if (at + 3 < n) ps = __fadd_rn(ps, __fmul_rn(b[k].w, b[k].w));
    }
    return ps;
}

// 1 / sqrt(sum / n + eps); a power of two divides exactly as its reciprocal multiplies
__device__ __forceinline__ float rms_inv(float sum, int n, float eps) {
    const float mean = (n & (n - 1)) ? __fdiv_rn(sum, (float)n) : __fmul_rn(sum, __int_as_float((127 - (31 - __clz(n))) << 23));
    return __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(mean, eps)));
}

}  // namespace brrr
