// Warp- and block-level building blocks shared by several kernels.
#pragma once
#include "brrr_dev.cuh"

namespace brrr {

// order-preserving map float -> uint32 (larger float = larger uint)
__device__ __forceinline__ uint32_t float_orderable(float v) {
    uint32_t b = __float_as_uint(v);
    return b ^ ((b >> 31) ? 0xFFFFFFFFu : 0x80000000u);
}

__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

// Quantise one 32-block held one element per lane; writes 32 int8 and the block scale.
// scale = max(1e-12, amax) / 127 (true division); q = round-half-away(v / scale) clamped +-127.
__device__ __forceinline__ void warp_quant_block(float v, int lane, int8_t *q, float *s) {
    float amax = fmaxf(warp_max(fabsf(v)), 1e-12f);
    float sc = __fdiv_rn(amax, 127.0f);
    if (lane == 0) *s = sc;
    q[lane] = (int8_t)brrr_q8_round_inv(v, sc, brrr_q8_inv(amax));
}

// Sum of squares in the 16-chain order: chain c (0..15) accumulates x[c], x[c+16], ... with fused
// multiply-adds; chains combine as ((a0+a1)+(a2+a3)) per lane, then (l0+l1)+(l2+l3); a scalar
// unfused tail covers n % 16.  Returns 1 / sqrt(ss / n + eps) to every thread of the block.
// Must be called by all threads; x must be visible to warp 0 (shared or global).
__device__ __forceinline__ float block_rms_inv(const float *x, int n, float eps, float *sh_out) {
    if (threadIdx.x < 32) {
        int c = threadIdx.x;
        float acc = 0.0f;
        int n16 = n & ~15;
        if (c < 16) {
            // chain c: x[c], x[c+16], ... in order; the next 12 values are on their way while 12 are added up, so that only
            // the fused multiply-adds sit on the dependent path
            int i = c;
            float v[12];
#pragma unroll
            for (int k = 0; k < 12; k++) v[k] = i + 16 * k < n16 ? x[i + 16 * k] : 0.0f;
#pragma unroll 2
            for (; i + 16 * 11 < n16; i += 16 * 12) {
                const float *w = x + min(i + 16 * 12, max(n16 - 16 * 12, 0) + c);      // past the last whole twelve: the end, read again below
                float u[12];
#pragma unroll
                for (int k = 0; k < 12; k++) u[k] = v[k];
#pragma unroll
                for (int k = 0; k < 12; k++) v[k] = w[16 * k];
#pragma unroll
                for (int k = 0; k < 12; k++) acc = __fmaf_rn(u[k], u[k], acc);
            }
            for (; i < n16; i += 16) { float t = x[i]; acc = __fmaf_rn(t, t, acc); }
        }
        acc = __fadd_rn(acc, __shfl_xor_sync(0xffffffffu, acc, 4));
        acc = __fadd_rn(acc, __shfl_xor_sync(0xffffffffu, acc, 8));
        acc = __fadd_rn(acc, __shfl_xor_sync(0xffffffffu, acc, 1));
        acc = __fadd_rn(acc, __shfl_xor_sync(0xffffffffu, acc, 2));
        if (c == 0) {
            for (int i = n16; i < n; i++) acc = __fadd_rn(acc, __fmul_rn(x[i], x[i]));
            *sh_out = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(__fdiv_rn(acc, (float)n), eps)));
        }
    }
    __syncthreads();
    return *sh_out;
}

// Block-wide RMSNorm + per-32 Q8 quantisation of x[0..n) into a staged activation image.
// Each thread owns 4 consecutive elements (one 32-bit word of quants), 8 consecutive threads own
// a 32-block, so a block's amax needs three shuffles.  norm_w == nullptr: quantise x as it is.
//   NQ_Q8:      xp[b*4+j] = {elements 4j..4j+3, elements 16+4j..16+4j+3}   (Q8 GEMV image)
//   NQ_MX:      xp[b*4+j] = the same two words byte-interleaved for the MXFP4 lane dot
//   NQ_NATURAL: quants in element order to (int8_t*)xp, scales to xsc       (global buffers)
// xf: n floats of shared scratch.  The static norm weights of the first MAXG passes are taken
// from wreg[], which the caller fills with norm_prefetch() before it waits on the previous
// kernel, so no cold global load sits on the critical path; later passes read norm_w directly.
// Must be called by all threads; nthreads % 32 == 0, n % 32 == 0, x and norm_w 16-byte aligned.
// Ends with the image complete but NOT yet synchronised.
enum { NQ_Q8 = 0, NQ_MX = 1, NQ_NATURAL = 2 };
// global -> shared copy of n floats (n % 4 == 0, 16-byte aligned).  Up to eight loads are issued before the first
// store: a store to shared memory between them would keep the compiler from overlapping the loads
// (it cannot rule out aliasing), and every load is a full round trip to L2.
__device__ __forceinline__ void stage_vec4(const float *__restrict__ src, float *dst, int n, int tid, int nthreads) {
    const int groups = n >> 2;
    const float4 *s4 = reinterpret_cast<const float4 *>(src);
    float4 *d4 = reinterpret_cast<float4 *>(dst);
    for (int g0 = tid; g0 < groups; g0 += 8 * nthreads) {
        float4 v[8];
#pragma unroll
        for (int k = 0; k < 8; k++) if (g0 + k * nthreads < groups) v[k] = s4[g0 + k * nthreads];
#pragma unroll
        for (int k = 0; k < 8; k++) if (g0 + k * nthreads < groups) d4[g0 + k * nthreads] = v[k];
    }
}

template <int MAXG>
__device__ __forceinline__ void norm_prefetch(const float *__restrict__ norm_w, int n, float4 (&wreg)[MAXG], int tid, int nthreads) {
#pragma unroll
    for (int p = 0; p < MAXG; p++) {
        const int g = tid + p * nthreads;
        wreg[p] = (norm_w && g < (n >> 2)) ? reinterpret_cast<const float4 *>(norm_w)[g] : make_float4(0.f, 0.f, 0.f, 0.f);
    }
}

template <int LAYOUT, int MAXG>
__device__ __forceinline__ void block_norm_quant_staged(const float *norm_w, const float4 (&wreg)[MAXG], float eps, int n,
                                                        float *xf, int2 *xp, float *xsc, float *inv_sh, int tid, int nthreads);

template <int LAYOUT, int MAXG>
__device__ __forceinline__ void block_norm_quant(const float *__restrict__ x, const float *norm_w, const float4 (&wreg)[MAXG], float eps, int n,
                                                 float *xf, int2 *xp, float *xsc, float *inv_sh, int tid, int nthreads) {
    stage_vec4(x, xf, n, tid, nthreads);
    __syncthreads();
    block_norm_quant_staged<LAYOUT, MAXG>(norm_w, wreg, eps, n, xf, xp, xsc, inv_sh, tid, nthreads);
}

// The same with x already in xf (shared memory) and visible to the whole block.
template <int LAYOUT, int MAXG>
__device__ __forceinline__ void block_norm_quant_staged(const float *norm_w, const float4 (&wreg)[MAXG], float eps, int n,
                                                        float *xf, int2 *xp, float *xsc, float *inv_sh, int tid, int nthreads) {
    const int groups = n >> 2;
    float4 *xf4 = reinterpret_cast<float4 *>(xf);
    float inv = 1.0f;
    if (norm_w) inv = block_rms_inv(xf, n, eps, inv_sh);
    const int npass = (groups + nthreads - 1) / nthreads;
    // The passes are independent; unrolling lets their divisions and shuffles overlap.
#pragma unroll
    for (int p = 0; p < 8; p++) {
        if (p >= npass) break;
        const int g = tid + p * nthreads;
        const bool live = g < groups;
        float4 v = live ? xf4[g] : make_float4(0.f, 0.f, 0.f, 0.f);
        if (norm_w && live) {
            float4 w;
            if (p < MAXG) w = wreg[p < MAXG ? p : 0];
            else w = reinterpret_cast<const float4 *>(norm_w)[g];
            v.x = __fmul_rn(__fmul_rn(v.x, inv), w.x); v.y = __fmul_rn(__fmul_rn(v.y, inv), w.y);
            v.z = __fmul_rn(__fmul_rn(v.z, inv), w.z); v.w = __fmul_rn(__fmul_rn(v.w, inv), w.w);
        }
        float amax = fmaxf(fmaxf(fabsf(v.x), fabsf(v.y)), fmaxf(fabsf(v.z), fabsf(v.w)));
        amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 1));
        amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 2));
        amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 4));
        amax = fmaxf(amax, 1e-12f);
        const float sc = __fdiv_rn(amax, 127.0f), qi = brrr_q8_inv(amax);
        uint32_t word = (uint32_t)(brrr_q8_round_inv(v.x, sc, qi) & 0xFF) | ((uint32_t)(brrr_q8_round_inv(v.y, sc, qi) & 0xFF) << 8) |
                        ((uint32_t)(brrr_q8_round_inv(v.z, sc, qi) & 0xFF) << 16) | ((uint32_t)(brrr_q8_round_inv(v.w, sc, qi) & 0xFF) << 24);
        const int t = g & 7, b = g >> 3;
        if (LAYOUT == NQ_MX) {
            uint32_t other = __shfl_xor_sync(0xffffffffu, word, 4);
            if (live && t < 4)
                xp[b * 4 + t] = make_int2((int)brrr_prmt(word, other, 0x5140u), (int)brrr_prmt(word, other, 0x7362u));
        } else if (LAYOUT == NQ_Q8) {
            if (live) reinterpret_cast<int *>(&xp[b * 4 + (t & 3)])[t >> 2] = (int)word;
        } else {
            if (live) reinterpret_cast<uint32_t *>(xp)[g] = word;
        }
        if (live && t == 0) xsc[b] = sc;
    }
}

// The largest entries of est[0 .. ne), ne <= 256: lane r < turns gets the expert of rank r (the larger first, the lower index among equals), by one
// warp without shared memory or barriers: each warp that needs the experts picks them itself.  All 32 lanes call it; every entry is a valid
// index whatever the values are (a NaN counts as larger than +inf or smaller than -inf, by its sign).  A lane holds PER consecutive experts as
// order-preserving keys; a turn is a maximum over the lane's keys and one reduction over the warp, the index travels beside the next turn.
// Used by every kernel that needs the speculative expert set (the set comes from an order-free router estimate; correctness never depends on
// it).  Ranking every expert against every other, block-wide with barriers, took 2300 cycles at 32 experts; at 128 the qwen3moe gate/up had its experts
// 2400 cycles after its dependency wait (64 + 128 tokens of the 30b-a3b shape: 209.2 ms, 206.5 with the warps picking and the copies spread over them).
template <int PER>
__device__ __forceinline__ int spec_pick_n(const float *est, int ne, int turns, int lane) {
    uint32_t key[PER];
#pragma unroll
    for (int i = 0; i < PER; i++) {
        const int e = lane * PER + i;
        key[i] = e < ne ? max(float_orderable(__fadd_rn(__ldcg(est + e), 0.0f)), 1u) : 0u;       // +0 for -0; 0: absent or taken
    }
    int mine = 0;
#pragma unroll 1
    for (int r = 0; r < turns; r++) {
        uint32_t m = key[0];
#pragma unroll
        for (int i = 1; i < PER; i++) m = max(m, key[i]);
        const uint32_t best = __reduce_max_sync(0xffffffffu, m);
        const int from = __ffs(__ballot_sync(0xffffffffu, m == best)) - 1;
        int at = PER - 1;
#pragma unroll
        for (int i = PER - 2; i >= 0; i--) if (key[i] == best) at = i;
        const int e = PER == 1 ? from : __shfl_sync(0xffffffffu, lane * PER + at, from);
        if (lane == r) mine = e;
#pragma unroll
        for (int i = 0; i < PER; i++) if (lane == from && i == at) key[i] = 0u;
    }
    return mine;
}
// turns <= topk ranks.  Builds with BRRR_TEST_HOOKS only: when the state's test_hooks word has bit 0 set, the last of the topk picks is replaced on every
// third position (the tests use it to force a missed speculation).
__device__ __forceinline__ int spec_pick(const float *est, int ne, int topk, int turns, const DevState *state, int lane) {
    const int e = ne <= 32 ? spec_pick_n<1>(est, ne, turns, lane) : ne <= 128 ? spec_pick_n<4>(est, ne, turns, lane) : spec_pick_n<8>(est, ne, turns, lane);
#ifdef BRRR_TEST_HOOKS
    if (state && (state->test_hooks & 1u) && state->pos % 3 == 0 && lane == topk - 1) return (e + 1) % ne;
#else
    (void)topk; (void)state;
#endif
    return e;
}

// gpt-oss clamped SwiGLU: xg = min(g, 7), yu = clamp(u, -7, 7), (xg / (1 + exp(-1.702 xg))) (yu + 1)
__device__ __forceinline__ float swiglu_oai(float g, float u) {
    float xg = fminf(g, 7.0f);
    float yu = fminf(fmaxf(u, -7.0f), 7.0f);
    float den = __fadd_rn(1.0f, brrr_expf_dev(__fmul_rn(-1.702f, xg)));
    return __fmul_rn(__fdiv_rn(xg, den), __fadd_rn(yu, 1.0f));
}


}  // namespace brrr
