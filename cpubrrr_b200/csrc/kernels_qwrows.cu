// Token rows of the qwen3moe engine: the stages between the K-quant products (kernels_kqt.cu) for up to 512 consecutive positions of
// a prompt.  Every row's numbers are those of the one-token kernels (kernels_qwen.cu): same operations in the same order.
#include "brrr_kernels.h"
#include "brrr_kqt.cuh"
#include "brrr_block.cuh"
#include "brrr_tma.cuh"
#include "brrr_tc.cuh"

namespace brrr {

namespace {

constexpr int QR_HD = 128;

// ---------------------------------------------------------------- embedding (engine_qwen2.rs:310-330)
__global__ void __launch_bounds__(256) qr_embed_kernel(const uint8_t *__restrict__ embd, int d, const uint32_t *__restrict__ toks, float *__restrict__ x) {
    pdl_wait();
    pdl_trigger();
    const int sb = blockIdx.x, t = blockIdx.y, i = threadIdx.x;
    const uint32_t *b32 = reinterpret_cast<const uint32_t *>(embd + (toks[t] * (size_t)(d / 256) + sb) * 144);
    const uint32_t dd = b32[0];
    const int j = i >> 5, l = i & 31;
    int sc, mn;
    k4_scale_min(b32[1], b32[2], b32[3], j, sc, mn);
    const uint32_t byte = reinterpret_cast<const uint8_t *>(b32 + 4)[(j >> 1) * 32 + l];
    const uint32_t q = (j & 1) ? (byte >> 4) : (byte & 0xFu);
    const float dv = half_bits_to_f32(dd & 0xffffu), dmin = half_bits_to_f32(dd >> 16);
    x[(size_t)t * d + sb * 256 + i] = __fsub_rn(__fmul_rn(__fmul_rn(dv, (float)sc), (float)q), __fmul_rn(dmin, (float)mn));
}

// ---------------------------------------------------------------- expert combine, RMS norm, Q8_K image (engine_qwen2.rs:432-465, 287-300)
// One CTA per row.  part: x += w[k] part[row topk + k], slots in order.  The norm's 12 slices are serial chains of d / 12 adds (the
// bound of this kernel: 171 dependent adds at d = 2048, ~0.7 us); rows run beside each other on the SM.
struct QrNormArgs {
    float *x;
    int d;
    const float *part, *wts;        // nullable: [row * topk + k][d], [row][8]
    int topk;
    const float *w;                 // nullable: combine only
    float eps;
    float *xn;                      // nullable: the normalised floats
    uint8_t *img;
    float *ys;
};

__global__ void __launch_bounds__(256) qr_norm_kernel(QrNormArgs a) {
    extern __shared__ __align__(16) float xs_sh[];
    __shared__ float part[QW_NT];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, d = a.d, t = blockIdx.x;
    pdl_wait();
    pdl_trigger();
    float4 *x4 = reinterpret_cast<float4 *>(a.x + (size_t)t * d);
    for (int g = tid; g < d / 4; g += 256) {
        float4 v = x4[g];
        if (a.part) {
            float4 pv[8];
#pragma unroll
            for (int k = 0; k < 8; k++) if (k < a.topk) pv[k] = reinterpret_cast<const float4 *>(a.part + ((size_t)t * a.topk + k) * d)[g];
#pragma unroll
            for (int k = 0; k < 8; k++)
                if (k < a.topk) {
                    const float w = a.wts[t * 8 + k];
                    v.x = __fadd_rn(v.x, __fmul_rn(w, pv[k].x)); v.y = __fadd_rn(v.y, __fmul_rn(w, pv[k].y));
                    v.z = __fadd_rn(v.z, __fmul_rn(w, pv[k].z)); v.w = __fadd_rn(v.w, __fmul_rn(w, pv[k].w));
                }
            x4[g] = v;
        }
        reinterpret_cast<float4 *>(xs_sh)[g] = v;
    }
    if (!a.w) return;
    __syncthreads();
    if (tid < QW_NT) {
        int lo, hi;
        qw_slice(tid, d, lo, hi);
        part[tid] = chain_squares(xs_sh, lo, hi);
    }
    __syncthreads();
    float tot = 0.0f;
#pragma unroll
    for (int k = 0; k < QW_NT; k++) tot = __fadd_rn(tot, part[k]);
    const float inv = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(__fdiv_rn(tot, (float)d), a.eps)));
    const int nsb = d / 256;
    for (int sb = warp; sb < nsb; sb += 8) {
        float v[8];
#pragma unroll
        for (int i = 0; i < 8; i++) {
            const int idx = sb * 256 + lane * 8 + i;
            v[i] = __fmul_rn(__fmul_rn(xs_sh[idx], inv), a.w[idx]);
        }
        if (a.xn) {
            float4 *dst = reinterpret_cast<float4 *>(a.xn + (size_t)t * d + sb * 256 + lane * 8);
            dst[0] = make_float4(v[0], v[1], v[2], v[3]);
            dst[1] = make_float4(v[4], v[5], v[6], v[7]);
        }
        warp_quant_q8k_image(v, lane, kimg_row(a.img, a.ys, t, gridDim.x, nsb, sb));
    }
}

// ---------------------------------------------------------------- QK norm + RoPE + cache append (engine_qwen2.rs:353-362, 466-482)
// One CTA per row: the mean squares are one serial chain per head, so each head is a lane's (all heads at once, rows padded to 132
// floats so that the lanes' 16-byte reads fall on different banks); the rest is elementwise.
constexpr int QR_PAD = 132;
__global__ void __launch_bounds__(256) qr_qknorm_kernel(float *__restrict__ q, const float *__restrict__ k, const float *__restrict__ v, const float *__restrict__ q_norm,
                                                        const float *__restrict__ k_norm, const float *__restrict__ rope, float eps, int nh, int nkv, int pos0,
                                                        float *__restrict__ kc, float *__restrict__ vc) {
    extern __shared__ __align__(16) float qk_sh[];      // [nh + nkv][QR_PAD], then [nh + nkv] inverses
    const int t = blockIdx.x, tid = threadIdx.x, pos = pos0 + t, heads = nh + nkv;
    float *inv_sh = qk_sh + heads * QR_PAD;
    pdl_wait();
    pdl_trigger();
    q += (size_t)t * nh * QR_HD;
    k += (size_t)t * nkv * QR_HD;
    v += (size_t)t * nkv * QR_HD;
    for (int i = tid; i < heads * 32; i += 256) {
        const int h = i >> 5, c = i & 31;
        reinterpret_cast<float4 *>(qk_sh + h * QR_PAD)[c] = reinterpret_cast<const float4 *>(h < nh ? q + h * QR_HD : k + (h - nh) * QR_HD)[c];
    }
    __syncthreads();
    for (int h = tid; h < heads; h += 256) {
        float ms = 0.0f;
#pragma unroll 8
        for (int i = 0; i < QR_HD / 4; i++) {
            const float4 r = reinterpret_cast<const float4 *>(qk_sh + h * QR_PAD)[i];
            ms = __fadd_rn(ms, __fmul_rn(r.x, r.x)); ms = __fadd_rn(ms, __fmul_rn(r.y, r.y));
            ms = __fadd_rn(ms, __fmul_rn(r.z, r.z)); ms = __fadd_rn(ms, __fmul_rn(r.w, r.w));
        }
        inv_sh[h] = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(__fdiv_rn(ms, (float)QR_HD), eps)));
    }
    __syncthreads();
    for (int i = tid; i < heads * 64; i += 256) {
        const int h = i >> 6, c = i & 63;
        const float inv = inv_sh[h], *w = h < nh ? q_norm : k_norm;
        const float aa = __fmul_rn(__fmul_rn(qk_sh[h * QR_PAD + c], inv), w[c]), bb = __fmul_rn(__fmul_rn(qk_sh[h * QR_PAD + 64 + c], inv), w[64 + c]);
        const float2 cs = reinterpret_cast<const float2 *>(rope)[(size_t)pos * 64 + c];
        const float o0 = __fsub_rn(__fmul_rn(aa, cs.x), __fmul_rn(bb, cs.y)), o1 = __fadd_rn(__fmul_rn(bb, cs.x), __fmul_rn(aa, cs.y));
        float *dst = h < nh ? q + h * QR_HD : kc + ((size_t)(h - nh) * BRRR_MAXSEQ + pos) * QR_HD;
        dst[c] = o0;
        dst[64 + c] = o1;
    }
    for (int i = tid; i < nkv * 32; i += 256)
        reinterpret_cast<float4 *>(vc + ((size_t)(i >> 5) * BRRR_MAXSEQ + pos) * QR_HD)[i & 31] = reinterpret_cast<const float4 *>(v)[i];
}

// ---------------------------------------------------------------- attention (engine_qwen2.rs:365-389)
// A CTA serves one KV head and R = group x queries (query head, row) pairs, which share every K and V tile it brings into shared
// memory; the scores of all keys stay in shared memory (R x keys floats), so each is computed once.  R is the largest of 32, 16, 8
// whose scores fit: 32 up to 1280 keys, 16 up to 2304, 8 up to the whole context.  Per pair, as qw_attn_kernel: score = 8 fused chains
// (dims c, c + 8, ...), (c + c+4), then (l0 + l1) + (l2 + l3), times 1 / sqrt(128); maximum over all keys; denominator (a warp of its
// own, lane = pair) and the output sums serial over the keys.  Keys past a pair's position carry p = +0, which leaves its sums as they
// are (they start at +0 and never become -0).
// Bound: shared-memory reads.  Score: lane = key, RP pairs per thread, two chains per packed multiply-add; p.V: lane = 4 dims.
constexpr int QA_THREADS = 288;
constexpr int QA_KPAD = 132;
template <int R> __host__ __device__ constexpr int qa_kt() { return R == 32 ? 32 : 64; }        // keys per tile
template <int R> __host__ __device__ constexpr int qa_max_keys() { return R == 32 ? 1280 : R == 16 ? 2304 : BRRR_MAXSEQ; }
__host__ __device__ constexpr int qa_stride(int n) { return ((n + 63) & ~63) + 4; }             // floats per pair: tail of the last tile, lanes' rows on different banks
template <int R> size_t qa_smem(int n) { return ((size_t)R * qa_stride(n) + R * QR_HD + 2 * qa_kt<R>() * QA_KPAD) * 4; }

struct QaArgs {
    const float *q, *kc, *vc;
    int nh, nkv, rows, pos0;
    uint8_t *img;
    float *ys;
};

template <int R>
__global__ void __launch_bounds__(QA_THREADS) qr_attn_kernel(QaArgs a) {
    constexpr int KT = qa_kt<R>(), RP = R == 8 ? 2 : 4, RG = R / RP, PV = R / 8;       // pairs per thread, groups of pairs; pairs per warp in p.V
    static_assert(RG * (KT / 32) == 8, "eight warps cover a tile");
    extern __shared__ __align__(16) float asm_[];
    const int group = a.nh / a.nkv, nq = R / group;
    const int kvh = blockIdx.y, r0 = (gridDim.x - 1 - blockIdx.x) * nq;                 // the longest rows first
    const int nrows = min(nq, a.rows - r0), n = a.pos0 + r0 + nrows, np = qa_stride(n);
    float *sc = asm_, *qs = sc + R * np, *tile = qs + R * QR_HD;
    __shared__ float den_sm[R];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const float *kbase = a.kc + (size_t)kvh * BRRR_MAXSEQ * QR_HD, *vbase = a.vc + (size_t)kvh * BRRR_MAXSEQ * QR_HD;
    const int ntile = (n + KT - 1) / KT;
    pdl_wait();
    pdl_trigger();
    for (int i = tid; i < R * 32; i += QA_THREADS) {      // pair p: row p / group, head p % group of the KV head's
        const int p = i >> 5, rr = p / group;
        reinterpret_cast<float4 *>(qs)[i] = rr < nrows ? reinterpret_cast<const float4 *>(a.q + ((size_t)(r0 + rr) * a.nh + kvh * group + p % group) * QR_HD)[i & 31]
                                                       : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    auto load = [&](const float *base, int t) {           // tile t into buffer t & 1 (compute warps); keys past n: the last one again
        const uint32_t dst = smem_u32(tile + (t & 1) * KT * QA_KPAD);
#pragma unroll
        for (int i = tid; i < KT * 32; i += 256) {
            const int key = i >> 5, c = i & 31;
            cp_async16(dst + (key * QA_KPAD + c * 4) * 4, base + (size_t)min(t * KT + key, n - 1) * QR_HD + c * 4);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    auto bar = [&]() { asm volatile("bar.sync 1, 256;" ::: "memory"); };
    if (warp < 8) load(kbase, 0);
    __syncthreads();
    if (warp < 8) {
        const int rg = warp % RG, sub = warp / RG;
        const float scale = __fdiv_rn(1.0f, __fsqrt_rn((float)QR_HD));
        for (int t = 0; t < ntile; t++) {
            if (t + 1 < ntile) { load(kbase, t + 1); asm volatile("cp.async.wait_group 1;" ::: "memory"); }
            else asm volatile("cp.async.wait_group 0;" ::: "memory");
            bar();
            const uint32_t ka = smem_u32(tile + (t & 1) * KT * QA_KPAD + (sub * 32 + lane) * QA_KPAD), qa = smem_u32(qs + rg * RP * QR_HD);
            f32x2 s[RP][4];
#pragma unroll
            for (int j = 0; j < RP; j++)
#pragma unroll
                for (int c = 0; c < 4; c++) s[j][c] = 0ull;
#pragma unroll 4
            for (int i = 0; i < 16; i++) {
                f32x2 kk[4];
                lds_pairs(ka + i * 32, kk[0], kk[1]);
                lds_pairs(ka + i * 32 + 16, kk[2], kk[3]);
#pragma unroll
                for (int j = 0; j < RP; j++) {
                    f32x2 qq[4];
                    lds_pairs(qa + j * 512 + i * 32, qq[0], qq[1]);
                    lds_pairs(qa + j * 512 + i * 32 + 16, qq[2], qq[3]);
#pragma unroll
                    for (int c = 0; c < 4; c++) s[j][c] = tl_fma2(kk[c], qq[c], s[j][c]);
                }
            }
#pragma unroll
            for (int j = 0; j < RP; j++) {
                float c[8];
#pragma unroll
                for (int i = 0; i < 4; i++) tl_unpack2(s[j][i], c[2 * i], c[2 * i + 1]);
                const float b0 = __fadd_rn(c[0], c[4]), b1 = __fadd_rn(c[1], c[5]), b2 = __fadd_rn(c[2], c[6]), b3 = __fadd_rn(c[3], c[7]);
                sc[(rg * RP + j) * np + t * KT + sub * 32 + lane] = __fmul_rn(__fadd_rn(__fadd_rn(b0, b1), __fadd_rn(b2, b3)), scale);
            }
            bar();
        }
        load(vbase, 0);
        // maximum and probabilities: a warp's own pairs
#pragma unroll
        for (int j = 0; j < PV; j++) {
            const int p = warp * PV + j, pn = a.pos0 + r0 + p / group + 1;
            float *row = sc + p * np;
            float mx = -3.402823466e+38f;
            for (int t = lane; t < min(pn, n); t += 32) mx = fmaxf(mx, row[t]);
            mx = warp_max(mx);
            for (int t = lane; t < ntile * KT; t += 32) row[t] = t < pn ? brrr_expf_dev(__fsub_rn(row[t], mx)) : 0.0f;
        }
    }
    __syncthreads();
    float acc[PV][4];
    if (warp == 8) {
        float den = 0.0f;
        if (lane < R) {
            const float *row = sc + lane * np;
#pragma unroll 4
            for (int t = 0; t < n; t += 4) {              // the tail of the last four is +0
                const float4 p = *reinterpret_cast<const float4 *>(row + t);
                den = __fadd_rn(den, p.x); den = __fadd_rn(den, p.y); den = __fadd_rn(den, p.z); den = __fadd_rn(den, p.w);
            }
            den_sm[lane] = den;
        }
    } else {
#pragma unroll
        for (int j = 0; j < PV; j++)
#pragma unroll
            for (int c = 0; c < 4; c++) acc[j][c] = 0.0f;
        for (int t = 0; t < ntile; t++) {
            if (t + 1 < ntile) { load(vbase, t + 1); asm volatile("cp.async.wait_group 1;" ::: "memory"); }
            else asm volatile("cp.async.wait_group 0;" ::: "memory");
            bar();
            const float *vt = tile + (t & 1) * KT * QA_KPAD + lane * 4, *pt = sc + warp * PV * np + t * KT;
#pragma unroll 2
            for (int k0 = 0; k0 < KT; k0 += 4) {
                float4 pp[PV];
#pragma unroll
                for (int j = 0; j < PV; j++) pp[j] = *reinterpret_cast<const float4 *>(pt + j * np + k0);
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    const float4 v = *reinterpret_cast<const float4 *>(vt + (k0 + k) * QA_KPAD);
#pragma unroll
                    for (int j = 0; j < PV; j++) {
                        const float p = k == 0 ? pp[j].x : k == 1 ? pp[j].y : k == 2 ? pp[j].z : pp[j].w;
                        acc[j][0] = __fmaf_rn(v.x, p, acc[j][0]); acc[j][1] = __fmaf_rn(v.y, p, acc[j][1]);
                        acc[j][2] = __fmaf_rn(v.z, p, acc[j][2]); acc[j][3] = __fmaf_rn(v.w, p, acc[j][3]);
                    }
                }
            }
            bar();
        }
    }
    __syncthreads();
    if (warp < 8) {
#pragma unroll
        for (int j = 0; j < PV; j++) {
            const int p = warp * PV + j;
            const float inv = __fdiv_rn(1.0f, den_sm[p]);
            reinterpret_cast<float4 *>(qs)[p * 32 + lane] = make_float4(__fmul_rn(acc[j][0], inv), __fmul_rn(acc[j][1], inv), __fmul_rn(acc[j][2], inv), __fmul_rn(acc[j][3], inv));
        }
    }
    __syncthreads();
    // two heads of a row are one superblock of the o-proj's activation (engine_qwen2.rs:390)
    for (int u = warp; u < R / 2; u += 9) {
        const int rr = 2 * u / group;
        if (rr >= nrows) break;
        const float4 v0 = reinterpret_cast<const float4 *>(qs)[u * 64 + lane * 2], v1 = reinterpret_cast<const float4 *>(qs)[u * 64 + lane * 2 + 1];
        const float v[8] = {v0.x, v0.y, v0.z, v0.w, v1.x, v1.y, v1.z, v1.w};
        warp_quant_q8k_image(v, lane, kimg_row(a.img, a.ys, r0 + rr, a.rows, a.nh / 2, (kvh * group + 2 * u % group) / 2));
    }
}

// ---------------------------------------------------------------- tokens of every expert, in chunks
// One CTA.  Counts, the chunks (experts in order; ceil(entries / 32) each, of equal size in whole groups of eight), then every entry to
// the next free place of its expert.  Which of an expert's places an entry takes changes no result: entries do not meet before the
// combine, which goes by token and slot.
__global__ void __launch_bounds__(1024) qr_plan_kernel(const int32_t *__restrict__ top, int ntok, int topk, int ne, KqPlan *__restrict__ plan) {
    __shared__ int cnt[256], chunk0[256], step[256], fill[256], wsum[8];
    const int tid = threadIdx.x, lane = tid & 31;
    if (tid < 256) { cnt[tid] = 0; fill[tid] = 0; }
    __syncthreads();
    pdl_wait();
    pdl_trigger();
    int mine[(BRRR_TILE_MAX * 8 + 1023) / 1024];
#pragma unroll
    for (int k = 0; k < BRRR_TILE_MAX * 8 / 1024; k++) {
        const int i = tid + k * 1024, t = i >> 3, s = i & 7;
        mine[k] = t < ntok && s < topk ? top[i] : -1;
        if (mine[k] >= 0) atomicAdd(&cnt[mine[k]], 1);
    }
    __syncthreads();
    int c = 0, nc = 0, incl = 0;
    if (tid < 256) {
        c = tid < ne ? cnt[tid] : 0;
        nc = (c + KT_NT - 1) / KT_NT;
        incl = nc;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) { const int v = __shfl_up_sync(0xffffffffu, incl, o); if (lane >= o) incl += v; }
        if (lane == 31) wsum[tid >> 5] = incl;
    }
    __syncthreads();
    if (tid < 256) {
        for (int w = 0; w < (tid >> 5); w++) incl += wsum[w];
        const int at = incl - nc, st = nc ? ((c + nc - 1) / nc + 7) & ~7 : 0;
        chunk0[tid] = at; step[tid] = st;
        for (int k = 0; k < nc; k++)
            if (at + k < KT_MAXCHUNK) { plan->e[at + k] = tid; plan->n[at + k] = max(min(st, c - k * st), 0); }
        if (tid == 255) plan->nchunk = min(incl, KT_MAXCHUNK);
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < BRRR_TILE_MAX * 8 / 1024; k++) {
        const int i = tid + k * 1024, e = mine[k];
        if (e < 0) continue;
        const int p = atomicAdd(&fill[e], 1), ch = chunk0[e] + p / step[e];
        if (ch < KT_MAXCHUNK) plan->ent[ch * KT_NT + p % step[e]] = (i >> 3) * topk + (i & 7);
    }
}

// images of the rows -> images of the chunks: a CTA per (chunk, superblock) at a time
__global__ void __launch_bounds__(256) qr_gather_kernel(const KqPlan *__restrict__ plan, const uint8_t *__restrict__ img, const float *__restrict__ ys, int rows, int topk,
                                                        int nsb, uint8_t *__restrict__ out, float *__restrict__ out_ys) {
    __shared__ int src[KT_NT];
    const int tid = threadIdx.x;
    pdl_wait();
    pdl_trigger();
    const int total = plan->nchunk * nsb;
    for (int u = blockIdx.x; u < total; u += gridDim.x) {
        const int ch = u / nsb, sb = u % nsb, n = plan->n[ch], cap = kq_cap(n), lg = cap == 8 ? 3 : cap == 16 ? 4 : 5;
        if (tid < n) {
            const int t = plan->ent[ch * KT_NT + tid] / topk;
            src[tid] = t;
            out_ys[(size_t)u * KT_NT + tid] = ys[((size_t)(t / KT_NT) * nsb + sb) * KT_NT + t % KT_NT];
        }
        __syncthreads();
        for (int i = tid; i < 34 << lg; i += 256) {
            const int piece = i >> lg, k = i & (cap - 1);
            if (k < n) {
                const int t = src[k], c0 = t / KT_NT, step = kq_cap(min(KT_NT, rows - c0 * KT_NT)) * 16;
                *reinterpret_cast<uint4 *>(out + (size_t)u * KIMG_BLOCK + i * 16) =
                    *reinterpret_cast<const uint4 *>(img + ((size_t)c0 * nsb + sb) * KIMG_BLOCK + piece * step + (t % KT_NT) * 16);
            }
        }
        __syncthreads();
    }
}

// ---------------------------------------------------------------- SiLU-GLU and Q8_K of h (engine_qwen2.rs:419-431): one warp per superblock
// of a position (32 chunk + i); g, u: [position][ff]
__global__ void __launch_bounds__(256) qr_glu_kernel(const KqPlan *__restrict__ plan, const float *__restrict__ g, const float *__restrict__ u, int nsb,
                                                     uint8_t *__restrict__ img, float *__restrict__ ys) {
    const int lane = threadIdx.x & 31;
    pdl_wait();
    pdl_trigger();
    const int total = plan->nchunk * KT_NT * nsb;
    for (int w = blockIdx.x * 8 + (threadIdx.x >> 5); w < total; w += gridDim.x * 8) {
        const int pos = w / nsb, sb = w % nsb, ch = pos / KT_NT, i = pos % KT_NT, n = plan->n[ch];
        if (i >= n) continue;
        const float4 *gp = reinterpret_cast<const float4 *>(g + (size_t)w * 256 + lane * 8), *up = reinterpret_cast<const float4 *>(u + (size_t)w * 256 + lane * 8);
        const float4 g0 = gp[0], g1 = gp[1], u0 = up[0], u1 = up[1];
        const float gv[8] = {g0.x, g0.y, g0.z, g0.w, g1.x, g1.y, g1.z, g1.w}, uv[8] = {u0.x, u0.y, u0.z, u0.w, u1.x, u1.y, u1.z, u1.w};
        float h[8];
#pragma unroll
        for (int k = 0; k < 8; k++) h[k] = __fmul_rn(__fdiv_rn(gv[k], __fadd_rn(1.0f, brrr_expf_dev(-gv[k]))), uv[k]);
        warp_quant_q8k_image(h, lane, kimg_slot(img, ys, ch, n, i, nsb, sb));
    }
}

// rows of floats -> images
__global__ void __launch_bounds__(256) qr_image_kernel(const float *__restrict__ x, int rows, int nsb, uint8_t *__restrict__ img, float *__restrict__ ys) {
    const int w = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (w >= rows * nsb) return;
    const float4 *p = reinterpret_cast<const float4 *>(x + (size_t)w * 256 + lane * 8);
    const float4 a = p[0], b = p[1];
    const float v[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
    warp_quant_q8k_image(v, lane, kimg_row(img, ys, w / nsb, rows, nsb, w % nsb));
}

template <int R>
cudaError_t qa_launch(const QaArgs &a, bool pdl, cudaStream_t st) {
    static unsigned long long configured = 0;      // one bit per device
    cudaError_t e = smem_optin(qr_attn_kernel<R>, 226 * 1024, configured);
    if (e != cudaSuccess) return e;
    const int nq = R / (a.nh / a.nkv);
    return launch_k(qr_attn_kernel<R>, dim3((a.rows + nq - 1) / nq, a.nkv), dim3(QA_THREADS), qa_smem<R>(a.pos0 + a.rows), st, pdl, a);
}

}  // namespace

cudaError_t launch_qr_embed(const uint8_t *embd, int d, const uint32_t *toks, int rows, float *x, bool pdl, cudaStream_t st) {
    return launch_k(qr_embed_kernel, dim3(d / 256, rows), dim3(256), 0, st, pdl, embd, d, toks, x);
}

cudaError_t launch_qr_norm(float *x, int rows, int d, const float *part, const float *wts, int topk, const float *w, float eps, float *xn, uint8_t *img, float *ys, bool pdl,
                           cudaStream_t st) {
    if (topk > 8) return cudaErrorInvalidValue;
    QrNormArgs a{x, d, part, wts, topk, w, eps, xn, img, ys};
    return launch_k(qr_norm_kernel, dim3(rows), dim3(256), (size_t)d * 4, st, pdl, a);
}

cudaError_t launch_qr_qknorm(float *q, const float *k, const float *v, const float *q_norm, const float *k_norm, const float *rope, float eps, int nh, int nkv, int pos0,
                             int rows, float *kc, float *vc, bool pdl, cudaStream_t st) {
    static unsigned long long configured = 0;      // one bit per device
    const size_t smem = (size_t)(nh + nkv) * (QR_PAD + 1) * 4;
    cudaError_t e = smem_optin(qr_qknorm_kernel, 200 * 1024, configured);
    if (e != cudaSuccess) return e;
    return launch_k(qr_qknorm_kernel, dim3(rows), dim3(256), smem, st, pdl, q, k, v, q_norm, k_norm, rope, eps, nh, nkv, pos0, kc, vc);
}

bool qr_attn_fits(int nh, int nkv) {
    const int group = nkv > 0 ? nh / nkv : 0;
    return (group == 2 || group == 4 || group == 8) && nh + nkv <= 256;
}

cudaError_t launch_qr_attn(const float *q, const float *kc, const float *vc, int nh, int nkv, int pos0, int rows, uint8_t *img, float *ys, bool pdl, cudaStream_t st) {
    if (!qr_attn_fits(nh, nkv)) return cudaErrorInvalidValue;
    QaArgs a{q, kc, vc, nh, nkv, rows, pos0, img, ys};
    const int n = pos0 + rows;
    if (n <= qa_max_keys<32>()) return qa_launch<32>(a, pdl, st);
    if (n <= qa_max_keys<16>()) return qa_launch<16>(a, pdl, st);
    return qa_launch<8>(a, pdl, st);
}

cudaError_t launch_qr_plan(const int32_t *top, int ntok, int topk, int ne, KqPlan *plan, bool pdl, cudaStream_t st) {
    if (ne > 256 || topk > 8 || ntok > BRRR_TILE_MAX) return cudaErrorInvalidValue;
    return launch_k(qr_plan_kernel, dim3(1), dim3(1024), 0, st, pdl, top, ntok, topk, ne, plan);
}

cudaError_t launch_qr_gather(const KqPlan *plan, const uint8_t *img, const float *ys, int rows, int topk, int ne, int nsb, uint8_t *out, float *out_ys, bool pdl,
                             cudaStream_t st) {
    const int blocks = kqt_max_chunks(rows * topk, ne) * nsb;
    return launch_k(qr_gather_kernel, dim3(blocks < 148 * 8 ? blocks : 148 * 8), dim3(256), 0, st, pdl, plan, img, ys, rows, topk, nsb, out, out_ys);
}

cudaError_t launch_qr_glu(const KqPlan *plan, const float *g, const float *u, int entries, int ne, int ff, uint8_t *img, float *ys, bool pdl, cudaStream_t st) {
    const int warps = kqt_max_chunks(entries, ne) * KT_NT * (ff / 256), blocks = (warps + 7) / 8;
    return launch_k(qr_glu_kernel, dim3(blocks < 148 * 8 ? blocks : 148 * 8), dim3(256), 0, st, pdl, plan, g, u, ff / 256, img, ys);
}

void launch_qr_image(const float *x, int rows, int cols, uint8_t *img, float *ys, cudaStream_t st) {
    const int nblk = rows * (cols / 256);
    if (nblk > 0) qr_image_kernel<<<(nblk + 7) / 8, 256, 0, st>>>(x, rows, cols / 256, img, ys);
}

}  // namespace brrr
