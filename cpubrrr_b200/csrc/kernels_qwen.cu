// Decode kernels of the qwen3moe engine (src/bin/engine_qwen2.rs:302-451): Q4_K embedding row, RMS norm with the reference's 12
// partial sums + Q8_K quantisation, K-quant matrix-vector products, per-head QK norm + RoPE + cache append, full causal GQA attention
// (head_dim 128), SiLU-GLU experts, weighted down-projection and the vocabulary argmax.
//
// Float order: every sum the reference forms serially is formed serially by one thread here (norm partials, head mean square, softmax
// denominator, probability-weighted values, superblock terms, the expert combine); integer sums are exact and split across lanes.
//
// A step is bound by latency: 36 MB of weights per layer are 5.6 us of memory time, the serial chains and hand-overs more.  So
// every kernel brings its matrix rows into shared memory with bulk copies, before its dependency wait wherever the rows are known by
// then (q|k|v, o-proj, down, the first rows of the head; K and V of the cached positions), and the layer is the chain
//   q|k|v (prologue: expert combine of the layer before, norm, Q8_K - every CTA its own: 64 KB from L2 cost less than a kernel)
//   -> attention (prologue: QK norm, RoPE, cache append) -> o-proj (prologue: Q8_K) -> routing hint (norm, Q8_K, estimate of the router)
//   -> gate/up + SiLU-GLU of the estimated experts -> down of the same
// joined by programmatic dependent launch, while the exact router - a chain of d dependent adds, 4.3 us at best at d = 2048 - runs
// beside the last three on another stream and publishes its choice to the next combine, which takes the weights and the order from
// it and flags the step if the estimate missed an expert (the host runs that step again without the estimate).
#include "brrr_kernels.h"
#include "brrr_kq.cuh"
#include "brrr_block.cuh"
#include "brrr_tma.cuh"

namespace brrr {

namespace {

constexpr int QW_HD = 128;
constexpr int QG_WARPS = 16, QG_THREADS = QG_WARPS * 32;
constexpr size_t QG_ROW_BYTES = 100 * 1024;      // shared memory for rows per CTA (two kernels share an SM)

// ---------------------------------------------------------------- embedding (engine_qwen2.rs:310-330)
__global__ void __launch_bounds__(256) qw_embed_kernel(const uint8_t *__restrict__ embd, int d, DevState *__restrict__ state,
                                                       float *__restrict__ x) {
    pdl_wait();
    pdl_trigger();
    if (blockIdx.x == 0 && threadIdx.x == 0) state->fold_seq = state->router_seq;      // routings published before this step (no router runs now)
    const size_t tok = state->tok;
    const int sb = blockIdx.x, i = threadIdx.x;
    const uint32_t *b32 = reinterpret_cast<const uint32_t *>(embd + (tok * (size_t)(d / 256) + sb) * 144);
    uint32_t dd = b32[0], s0 = b32[1], s1 = b32[2], s2 = b32[3];
    int j = i >> 5, l = i & 31, sc, mn;
    k4_scale_min(s0, s1, s2, j, sc, mn);
    uint32_t byte = reinterpret_cast<const uint8_t *>(b32 + 4)[(j >> 1) * 32 + l];
    uint32_t q = (j & 1) ? (byte >> 4) : (byte & 0xFu);
    float dv = half_bits_to_f32(dd & 0xffffu), dmin = half_bits_to_f32(dd >> 16);
    x[sb * 256 + i] = __fsub_rn(__fmul_rn(__fmul_rn(dv, (float)sc), (float)q), __fmul_rn(dmin, (float)mn));
}

// ---------------------------------------------------------------- expert selection
// sel[r] = expert of rank r of est[0 .. ne) (the larger first, the lower index among equals).  Block-wide; ends synchronised.
struct alignas(16) SelectScratch { float lg[256]; int rank[256]; };
__device__ __forceinline__ void qw_select(const float *est, int ne, int topk, const DevState *state, SelectScratch &w, int *sel, int tid, int nthreads) {
#ifdef BRRR_TEST_HOOKS
    const bool spoil = state && (state->test_hooks & 1u) && state->pos % 3 == 0;
#else
    constexpr bool spoil = false;
    (void)state;
#endif
    for (int e = tid; e < 256; e += nthreads) { w.lg[e] = e < ne ? __ldcg(est + e) : -INFINITY; w.rank[e] = 0; }
    if (tid < 8) sel[tid] = 0;
    __syncthreads();
    const int quarter = ((ne + 15) / 16) * 4;
    for (int i = tid; i < 4 * ne; i += nthreads) {
        const int p = i / ne, e = i - p * ne, o0 = p * quarter;
        const float v = w.lg[e];
        int r = 0;
        for (int o = o0; o < min(o0 + quarter, 256); o += 4) {
            const float4 u = *reinterpret_cast<const float4 *>(w.lg + o);
            r += (u.x > v || (u.x == v && o < e)) + (u.y > v || (u.y == v && o + 1 < e)) + (u.z > v || (u.z == v && o + 2 < e)) + (u.w > v || (u.w == v && o + 3 < e));
        }
        if (r) atomicAdd(&w.rank[e], r);
    }
    __syncthreads();
    for (int e = tid; e < ne; e += nthreads)
        if (w.rank[e] < topk) sel[w.rank[e]] = (spoil && w.rank[e] == topk - 1) ? (e + 1) % ne : e;
    __syncthreads();
}

// ---------------------------------------------------------------- expert combine + RMS norm + Q8_K (engine_qwen2.rs:432-465, 287-300)
// x += w[k] part[slot of k], exact experts in rank order (part == nullptr: nothing to add); then norm and quants.
struct QFold {
    const float *x_in, *part;        // residual; [slot][d]
    float *x_out;                    // the new residual (CTA 0 writes it; never x_in: other CTAs may still read that)
    const float *est;                // slot s of part belongs to rank s of the estimate; nullptr: of top
    const int32_t *top;              // exact routing (est == nullptr)
    const float *wts;
    int ne, topk, d;
    uint32_t seq;                    // est: this step's seq-th routing is awaited from the router
    const float *norm_w;             // nullable: combine only
    float eps;
    DevState *state;
};
struct QFoldShared {
    SelectScratch sel_ws;
    int sel[8], slot_of[8];
    float wts[8], part[QW_NT];
};

// Before the dependency wait: the estimate's experts and the exact routing, a bounded wait for the router's words (it does not depend on
// any kernel that waits here, and this kernel leaves it room on every SM).
__device__ __forceinline__ void qw_fold_routing(const QFold &a, QFoldShared &w, int tid) {
    if (!a.part) return;
    if (a.est) qw_select(a.est, a.ne, a.topk, a.state, w.sel_ws, w.sel, tid, QG_THREADS);
    if (tid < 32) {
        uint32_t payload = 0u;
        if (a.est) {
            if (tid < 16 && (tid & 7) < a.topk) {
                const uint32_t want = __ldcg(&a.state->fold_seq) + a.seq;
                const volatile unsigned long long *p = a.state->route_pub + tid;
                bool ok = false;
                const long long t0 = clock64();
                do {
                    for (int i = 0; i < 64 && !ok; i++) {
                        const unsigned long long v = *p;
                        ok = (uint32_t)(v >> 32) == want;
                        payload = (uint32_t)v;
                    }
                } while (!ok && clock64() - t0 < WAIT_CYCLES && *reinterpret_cast<volatile uint32_t *>(&a.state->err) == 0u);
                if (!ok) {               // the step is void from here: the host runs it again without the estimate
                    atomicCAS(&a.state->err, (uint32_t)DEV_ERR_NONE, (uint32_t)DEV_ERR_PEER_TIMEOUT);
                    atomicMin(&a.state->spec_fail_step, a.state->n_out);
                }
            }
        } else if (tid < 16 && (tid & 7) < a.topk) payload = tid < 8 ? (uint32_t)__ldcg(a.top + tid) : __float_as_uint(__ldcg(a.wts + (tid - 8)));
        if (tid >= 8 && tid < 8 + a.topk) w.wts[tid - 8] = __uint_as_float(payload);
        if (tid < a.topk) {
            int slot = tid;
            if (a.est) {
                slot = -1;
                for (int s = 0; s < a.topk; s++) if (w.sel[s] == (int)payload) slot = s;
                if (slot < 0) { slot = 0; atomicMin(&a.state->spec_fail_step, a.state->n_out); }      // the estimate missed this expert
            }
            w.slot_of[tid] = slot;
        }
    }
    __syncthreads();
}

// The 12-slice norm of xf (shared memory, synchronised): 1 / sqrt(mean + eps) in every thread.
__device__ __forceinline__ float qw_norm_inv(const float *xf, int d, float eps, float *part, int tid) {
    if (tid < QW_NT) {
        int lo, hi;
        qw_slice(tid, d, lo, hi);
        float ps = 0.0f;
#pragma unroll 8
        for (int i = lo; i < hi; i++) { const float v = xf[i]; ps = __fadd_rn(ps, __fmul_rn(v, v)); }
        part[tid] = ps;
    }
    __syncthreads();
    float tot = 0.0f;
#pragma unroll
    for (int k = 0; k < QW_NT; k++) tot = __fadd_rn(tot, part[k]);
    return __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(__fdiv_rn(tot, (float)d), eps)));
}

// After the wait.  xf: d floats of shared memory; q, s, b16: the Q8_K image (shared or global).
__device__ __forceinline__ void qw_fold_norm(const QFold &a, QFoldShared &w, float *xf, int8_t *q, float *s, int32_t *b16, bool store, int tid) {
    const int d = a.d, warp = tid >> 5, lane = tid & 31;
    for (int g = tid; g < d / 4; g += QG_THREADS) {
        float4 x = reinterpret_cast<const float4 *>(a.x_in)[g];
        if (a.part) {
            float4 p[8];
#pragma unroll
            for (int k = 0; k < 8; k++) if (k < a.topk) p[k] = __ldcg(reinterpret_cast<const float4 *>(a.part + (size_t)w.slot_of[k] * d) + g);
#pragma unroll
            for (int k = 0; k < 8; k++)
                if (k < a.topk) {
                    const float t = w.wts[k];
                    x.x = __fadd_rn(x.x, __fmul_rn(t, p[k].x)); x.y = __fadd_rn(x.y, __fmul_rn(t, p[k].y));
                    x.z = __fadd_rn(x.z, __fmul_rn(t, p[k].z)); x.w = __fadd_rn(x.w, __fmul_rn(t, p[k].w));
                }
        }
        reinterpret_cast<float4 *>(xf)[g] = x;
        if (store) reinterpret_cast<float4 *>(a.x_out)[g] = x;
    }
    if (!a.norm_w) return;
    __syncthreads();
    const float inv = qw_norm_inv(xf, d, a.eps, w.part, tid);
    for (int sb = warp; sb < d / 256; sb += QG_WARPS) {
        float v[8];
        const float4 w0 = reinterpret_cast<const float4 *>(a.norm_w + sb * 256)[lane * 2], w1 = reinterpret_cast<const float4 *>(a.norm_w + sb * 256)[lane * 2 + 1];
        const float nw[8] = {w0.x, w0.y, w0.z, w0.w, w1.x, w1.y, w1.z, w1.w};
#pragma unroll
        for (int i = 0; i < 8; i++) v[i] = __fmul_rn(__fmul_rn(xf[sb * 256 + lane * 8 + i], inv), nw[i]);
        warp_quant_q8k16(v, lane, q + sb * 256, s + sb, b16 + sb * 16);
    }
}

// the same as a kernel of its own, for the vocabulary head: one CTA, image to global memory
__global__ void __launch_bounds__(QG_THREADS) qw_fold_kernel(QFold a, int8_t *q, float *s, int32_t *b16) {
    extern __shared__ __align__(16) unsigned char qsm[];
    __shared__ QFoldShared w;
    qw_fold_routing(a, w, threadIdx.x);
    pdl_wait();
    pdl_trigger();
    qw_fold_norm(a, w, reinterpret_cast<float *>(qsm), q, s, b16, true, threadIdx.x);
}

// ---------------------------------------------------------------- matrix rows x one activation (q|k|v, o-proj)
// Lane group g = lane / 8 takes superblocks g, g + 4, ... of every row.  Up to eight superblocks the activation stays in registers from row
// to row; of wider rows a warp has one or two, and it is read per pair of superblocks (64 registers: two CTAs per SM).
template <int UPL> struct QLane {
    KAct x[2];
    float ys[2];
    const int8_t *q;
    const float *s;
    const int32_t *b16;
};
__device__ __forceinline__ void qw_lane_pair(int type, int nsb, const int8_t *q, const float *s, const int32_t *b16, int lane, int i0, KAct (&x)[2], float (&ys)[2]) {
#pragma unroll
    for (int i = 0; i < 2; i++) {
        const int sb = min((lane >> 3) + 4 * (i0 + i), nsb - 1);
        kact_load(type, q + sb * 256, b16 + sb * 16, lane & 7, x[i]);
        ys[i] = s[sb];
    }
}
template <int UPL>
__device__ __forceinline__ void qw_lane_load(int type, int nsb, const int8_t *q, const float *s, const int32_t *b16, int lane, QLane<UPL> &a) {
    if (UPL == 2) qw_lane_pair(type, nsb, q, s, b16, lane, 0, a.x, a.ys);
    else { a.q = q; a.s = s; a.b16 = b16; }
}
// superblock terms of a row -> terms[0 .. nsb)
template <int UPL>
__device__ __forceinline__ void qw_row_terms(int type, int nsb, const unsigned char *row, QLane<UPL> &a, int lane, float *terms) {
    const int g = lane >> 3, l8 = lane & 7;
#pragma unroll 1
    for (int i = 0; i < UPL; i += 2) {
        const int sb0 = g + 4 * i, sb1 = sb0 + 4;
        if (UPL > 2) qw_lane_pair(type, nsb, a.q, a.s, a.b16, lane, i, a.x, a.ys);
        const float t = kq_pair_term(type, nsb, row, min(sb0, nsb - 1), a.x[0], a.ys[0], row, min(sb1, nsb - 1), a.x[1], a.ys[1], l8);
        const int sb = l8 ? sb1 : sb0;
        if (!(l8 & 3) && sb < nsb) terms[sb] = t;
    }
}
__device__ __forceinline__ float qw_terms_sum(const float *t, int nsb) {      // superblocks in order, from zero
    float v = 0.0f;
    for (int i = 0; i < nsb; i++) v = __fadd_rn(v, t[i]);
    return v;
}
// up to three matrices of equal width, stacked
struct KStack {
    KMatDev m[3];
    float *y[3];
    int n, rows, per_cta, stride;      // rows in all, rows per CTA, bytes per row in shared memory
    __device__ int find(int row, int &local) const {
        int i = 0;
        while (i < n - 1 && row >= m[i].rows) { row -= m[i].rows; i++; }
        local = row;
        return i;
    }
};

struct QGemvArgs {
    KStack k;
    QFold f;                 // FOLD: the activation is the combined, normalised residual
    const float *act;        // else: these floats, as they are; outputs are added to y
    DevState *state;
};

// Shared memory: rows | xf (FOLD: d floats) | q | scales | 16-sums | terms.
// Bound: the hand-over, the prologue (combine, norm: 1.3 us) and one pass over rows that are already on chip (35 rows of 8 superblocks on
// 16 warps: 0.7 us).
template <int UPL, bool FOLD>
__global__ void __launch_bounds__(QG_THREADS, 2) qw_gemv_kernel(const __grid_constant__ QGemvArgs a) {
    extern __shared__ __align__(16) unsigned char qsm[];
    __shared__ QFoldShared w;
    __shared__ __align__(8) uint64_t bar;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int K = a.k.m[0].cols, nsb = K / 256, row0 = blockIdx.x * a.k.per_cta, n = min(a.k.per_cta, a.k.rows - row0);
    unsigned char *rows = qsm;
    float *xf = reinterpret_cast<float *>(qsm + (size_t)a.k.per_cta * a.k.stride);
    int8_t *q = reinterpret_cast<int8_t *>(xf + (FOLD ? K : 0));
    float *s = reinterpret_cast<float *>(q + K);
    int32_t *b16 = reinterpret_cast<int32_t *>(s + ((nsb + 3) & ~3));
    float *terms = reinterpret_cast<float *>(b16 + nsb * 16);
    Waiter waiter(a.state ? &a.state->err : nullptr);
    if (warp == 0) {
        if (lane == 0) {
            mbar_init(&bar, 1);
            mbar_fence_init();
            uint32_t bytes = 0;
            for (int i = 0, r = row0, l; i < n;) {           // whole runs of a matrix
                const int mi = a.k.find(r, l), run = min(n - i, a.k.m[mi].rows - l);
                bytes += (uint32_t)run * (uint32_t)a.k.m[mi].bpr();
                i += run; r += run;
            }
            mbar_expect_tx(&bar, bytes);
        }
        __syncwarp();
        for (int i = lane; i < n; i += 32) {
            int l;
            const KMatDev &m = a.k.m[a.k.find(row0 + i, l)];
            bulk_g2s(rows + (size_t)i * a.k.stride, m.p + (size_t)l * m.bpr(), (uint32_t)m.bpr(), &bar);
        }
    }
    float resid = 0.0f;
    int my_l = 0;
    const int my_m = tid < n ? a.k.find(row0 + tid, my_l) : 0;
    if (!FOLD && tid < n) resid = a.k.y[my_m][my_l];         // written two kernels back
    if (FOLD) qw_fold_routing(a.f, w, tid);
    pdl_wait();
    pdl_trigger();
    if (FOLD) qw_fold_norm(a.f, w, xf, q, s, b16, blockIdx.x == 0, tid);
    else
        for (int sb = warp; sb < nsb; sb += QG_WARPS) {
            const float4 *src = reinterpret_cast<const float4 *>(a.act + sb * 256 + lane * 8);
            const float4 p0 = src[0], p1 = src[1];
            const float v[8] = {p0.x, p0.y, p0.z, p0.w, p1.x, p1.y, p1.z, p1.w};
            warp_quant_q8k16(v, lane, q + sb * 256, s + sb, b16 + sb * 16);
        }
    __syncthreads();
    waiter.wait(&bar, 0u);
    QLane<UPL> x;
    int type = 0;
    for (int i = warp; i < n; i += QG_WARPS) {
        int l;
        const int t = a.k.m[a.k.find(row0 + i, l)].type;
        if (t != type) { type = t; qw_lane_load<UPL>(type, nsb, q, s, b16, lane, x); }
        qw_row_terms<UPL>(type, nsb, rows + (size_t)i * a.k.stride, x, lane, terms + i * nsb);
    }
    __syncthreads();
    if (tid < n) {
        const float v = qw_terms_sum(terms + tid * nsb, nsb);
        a.k.y[my_m][my_l] = FOLD ? v : __fadd_rn(resid, v);
    }
}

// ---------------------------------------------------------------- attention (engine_qwen2.rs:353-389, 466-482)
// One CTA per query head.  Prologue: QK norm (serial mean square) and RoPE of q and of the position's own k; the first head of a KV group
// appends k and v to the cache.  score(t): 8 chains (chain c covers dims c, c+8, ..., fused), (c + c+4) per lane, (l0+l1)+(l2+l3), times
// 1/sqrt(128); maximum over all keys; denominator and the 128 output sums serial over t.
// K, then V of the cached positions run through one ring of 64-position tiles, a copy per position (rows 136 floats apart: the score
// threads - (key, half of the chains) - read 16 bytes each from different banks).  The ring starts before the dependency wait.
// Bound: the chains over the keys (4 cycles each) and 5 cycles of shared-memory reads per key; at 100 positions the prologue.
constexpr int QA_TILE = 64, QA_STRIDE = 136, QA_SLOTS = 5, QA_THREADS = 288;
constexpr size_t QA_SMEM = (size_t)QA_SLOTS * QA_TILE * QA_STRIDE * 4 + (size_t)BRRR_MAXSEQ * 4;

struct QAttnArgs {
    const float *q, *k, *v, *q_norm, *k_norm, *rope;
    float eps;
    float *kc, *vc;              // [nkv][MAXSEQ][128]
    int nh, nkv;
    DevState *state;
    float *out;                  // [nh][128]
};

__device__ __forceinline__ float qa_half_score(const float *kp, const float *qp) {       // four chains of a key, then (c + c+4) with the other half's
    float s0 = 0.0f, s1 = 0.0f, s2 = 0.0f, s3 = 0.0f;
#pragma unroll
    for (int i = 0; i < 16; i++) {
        const float4 k = *reinterpret_cast<const float4 *>(kp + 8 * i), q = *reinterpret_cast<const float4 *>(qp + 8 * i);
        s0 = __fmaf_rn(k.x, q.x, s0); s1 = __fmaf_rn(k.y, q.y, s1); s2 = __fmaf_rn(k.z, q.z, s2); s3 = __fmaf_rn(k.w, q.w, s3);
    }
    s0 = __fadd_rn(s0, __shfl_xor_sync(0xffffffffu, s0, 1)); s1 = __fadd_rn(s1, __shfl_xor_sync(0xffffffffu, s1, 1));
    s2 = __fadd_rn(s2, __shfl_xor_sync(0xffffffffu, s2, 1)); s3 = __fadd_rn(s3, __shfl_xor_sync(0xffffffffu, s3, 1));
    return __fadd_rn(__fadd_rn(s0, s1), __fadd_rn(s2, s3));
}

__global__ void __launch_bounds__(QA_THREADS) qw_attn_kernel(QAttnArgs a) {
    extern __shared__ __align__(16) float asm_[];
    float *ring = asm_, *sc = asm_ + QA_SLOTS * QA_TILE * QA_STRIDE;
    __shared__ __align__(8) uint64_t full[QA_SLOTS], empty[QA_SLOTS];
    __shared__ __align__(16) float raw[2][QW_HD], nv[2][QW_HD], qs[QW_HD], ks[QW_HD], vs[QW_HD];
    __shared__ float red[8], inv_sh[2], den_sh;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int h = blockIdx.x, group = a.nh / a.nkv, kvh = h / group;
    const int pos = (int)a.state->pos, n = pos + 1, nt = (pos + QA_TILE - 1) / QA_TILE;        // the position is an input of the step
    float *kbase = a.kc + (size_t)kvh * BRRR_MAXSEQ * QW_HD, *vbase = a.vc + (size_t)kvh * BRRR_MAXSEQ * QW_HD;
    Waiter waiter(&a.state->err);
    if (tid == 256) {
        for (int i = 0; i < QA_SLOTS; i++) { mbar_init(&full[i], 1); mbar_init(&empty[i], 4); }
        mbar_fence_init();
    }
    float wv = 0.0f, co = 0.0f, si = 0.0f;
    if (tid < 256) {
        wv = (tid < QW_HD ? a.q_norm : a.k_norm)[tid & (QW_HD - 1)];
        const float2 cs = reinterpret_cast<const float2 *>(a.rope)[(size_t)pos * (QW_HD / 2) + (tid & 63)];
        co = cs.x; si = cs.y;
    }
    __syncthreads();
    if (warp == 8) {
        // ---- copies: K tiles, then V tiles
        bool waited = false;
        for (int t = 0; t < 2 * nt; t++) {
            const int slot = t % QA_SLOTS, k0 = (t < nt ? t : t - nt) * QA_TILE, cnt = min(QA_TILE, pos - k0);
            if (t >= QA_SLOTS) {
                if (!waited) { pdl_wait(); pdl_trigger(); waiter.poison_if_failed(); waited = true; }      // with the others: the next kernel may start
                waiter.wait(&empty[slot], (uint32_t)(t / QA_SLOTS - 1) & 1u);
            }
            if (lane == 0) mbar_expect_tx(&full[slot], (uint32_t)cnt * QW_HD * 4);
            __syncwarp();
            const float *src = (t < nt ? kbase : vbase) + (size_t)k0 * QW_HD;
            for (int i = lane; i < cnt; i += 32) bulk_g2s(ring + (size_t)(slot * QA_TILE + i) * QA_STRIDE, src + (size_t)i * QW_HD, QW_HD * 4, &full[slot]);
        }
        if (!waited) { pdl_wait(); pdl_trigger(); }
        return;
    }
    pdl_wait();
    pdl_trigger();
    waiter.poison_if_failed();
    auto bar = [&]() { asm volatile("bar.sync 1, 256;" ::: "memory"); };
    {
        const int u = tid & (QW_HD - 1);
        raw[tid >> 7][u] = tid < QW_HD ? a.q[h * QW_HD + u] : a.k[kvh * QW_HD + u];
        if (tid < QW_HD) vs[u] = a.v[kvh * QW_HD + u];
    }
    bar();
    if (tid == 0 || tid == 32) {
        const float4 *r = reinterpret_cast<const float4 *>(raw[tid >> 5]);
        float ms = 0.0f;
#pragma unroll 8
        for (int i = 0; i < QW_HD / 4; i++) {
            const float4 t = r[i];
            ms = __fadd_rn(ms, __fmul_rn(t.x, t.x)); ms = __fadd_rn(ms, __fmul_rn(t.y, t.y));
            ms = __fadd_rn(ms, __fmul_rn(t.z, t.z)); ms = __fadd_rn(ms, __fmul_rn(t.w, t.w));
        }
        inv_sh[tid >> 5] = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(__fdiv_rn(ms, (float)QW_HD), a.eps)));
    }
    bar();
    nv[tid >> 7][tid & (QW_HD - 1)] = __fmul_rn(__fmul_rn(raw[tid >> 7][tid & (QW_HD - 1)], inv_sh[tid >> 7]), wv);
    bar();
    {
        const int u = tid & (QW_HD - 1), c = u & 63;
        const float aa = nv[tid >> 7][c], bb = nv[tid >> 7][64 + c];
        const float o = u < 64 ? __fsub_rn(__fmul_rn(aa, co), __fmul_rn(bb, si)) : __fadd_rn(__fmul_rn(bb, co), __fmul_rn(aa, si));
        (tid < QW_HD ? qs : ks)[u] = o;
        if (h % group == 0) {
            if (tid >= QW_HD) kbase[(size_t)pos * QW_HD + u] = o;
            else vbase[(size_t)pos * QW_HD + u] = vs[u];
        }
    }
    bar();
    // ---- scores: a group of four warps per tile, thread = (key, half of the chains)
    const float scale = __fdiv_rn(1.0f, __fsqrt_rn((float)QW_HD));
    const int hf = lane & 1, key = (warp & 3) * 16 + (lane >> 1);
    for (int t = warp >> 2; t < nt; t += 2) {
        const int slot = t % QA_SLOTS;
        waiter.wait(&full[slot], (uint32_t)(t / QA_SLOTS) & 1u);
        const float s = qa_half_score(ring + (size_t)(slot * QA_TILE + key) * QA_STRIDE + 4 * hf, qs + 4 * hf);
        if (hf == 0 && t * QA_TILE + key < pos) sc[t * QA_TILE + key] = __fmul_rn(s, scale);
        __syncwarp();
        if (lane == 0) mbar_arrive(&empty[slot]);
    }
    if (warp == 7) {                 // the position itself
        const float s = qa_half_score(ks + 4 * hf, qs + 4 * hf);
        if (lane == 0) sc[pos] = __fmul_rn(s, scale);
    }
    bar();
    float mx = -3.402823466e+38f;
    for (int t = tid; t < n; t += 256) mx = fmaxf(mx, sc[t]);
    mx = warp_max(mx);
    if (lane == 0) red[warp] = mx;
    bar();
    mx = red[0];
#pragma unroll
    for (int w = 1; w < 8; w++) mx = fmaxf(mx, red[w]);
    for (int t = tid; t < ((n + 3) & ~3); t += 256) sc[t] = t < n ? brrr_expf_dev(__fsub_rn(sc[t], mx)) : 0.0f;      // +0 past the end changes no sum
    bar();
    float acc = 0.0f;
    if (warp < 4) {
        for (int t = 0; t < nt; t++) {
            const int u = nt + t, slot = u % QA_SLOTS, cnt = min(QA_TILE, pos - t * QA_TILE);
            waiter.wait(&full[slot], (uint32_t)(u / QA_SLOTS) & 1u);
            const float *vt = ring + (size_t)slot * QA_TILE * QA_STRIDE + tid, *pt = sc + t * QA_TILE;
            int k = 0;
#pragma unroll 4
            for (; k + 4 <= cnt; k += 4) {
                const float4 p = *reinterpret_cast<const float4 *>(pt + k);
                acc = __fmaf_rn(vt[k * QA_STRIDE], p.x, acc); acc = __fmaf_rn(vt[(k + 1) * QA_STRIDE], p.y, acc);
                acc = __fmaf_rn(vt[(k + 2) * QA_STRIDE], p.z, acc); acc = __fmaf_rn(vt[(k + 3) * QA_STRIDE], p.w, acc);
            }
            for (; k < cnt; k++) acc = __fmaf_rn(vt[k * QA_STRIDE], pt[k], acc);
            __syncwarp();
            if (lane == 0) mbar_arrive(&empty[slot]);
        }
        acc = __fmaf_rn(vs[tid], sc[pos], acc);
    } else if (tid == 128) {
        float den = 0.0f;
#pragma unroll 4
        for (int t = 0; t < n; t += 4) {
            const float4 p = *reinterpret_cast<const float4 *>(sc + t);
            den = __fadd_rn(den, p.x); den = __fadd_rn(den, p.y); den = __fadd_rn(den, p.z); den = __fadd_rn(den, p.w);
        }
        den_sh = den;
    }
    bar();
    if (tid < QW_HD) a.out[h * QW_HD + tid] = __fmul_rn(acc, __fdiv_rn(1.0f, den_sh));
}

// ---------------------------------------------------------------- routing hint
// One CTA per expert: an order-free estimate of its router logit (a few ulps from the serial chain), which only decides whose weights start
// moving (see qw_fold_routing), and a share of the normalised token's Q8_K.  The router row and the norm weights are in registers before
// the dependency wait.
constexpr int QH_THREADS = 128, QH_MAXG = 8;
struct QHintArgs {
    const float *x, *norm_w;
    float eps;
    int d, ne;
    const float *Wt;             // tiled router matrix
    float *est;
    int8_t *q;
    float *s;
    int32_t *b16;
};

__global__ void __launch_bounds__(QH_THREADS) qw_hint_kernel(QHintArgs a) {
    extern __shared__ __align__(16) float xf[];
    __shared__ float part[QW_NT], red[QH_THREADS / 32];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, e = blockIdx.x, d = a.d, groups = d >> 2;
    const int ntiles = (d + RT_TJ - 1) / RT_TJ;
    const float *wrow = a.Wt + ((size_t)(e >> 5) * ntiles * 32 + (e & 31)) * RT_STRIDE;
    float4 w[QH_MAXG];           // router weight x norm weight
#pragma unroll
    for (int p = 0; p < QH_MAXG; p++) {
        const int g = tid + p * QH_THREADS;
        w[p] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (g < groups) {
            const int j = g * 4, t = j / RT_TJ, jj = j % RT_TJ;
            const float4 r = *reinterpret_cast<const float4 *>(wrow + (size_t)t * RT_TILE_FLOATS + jj), n = reinterpret_cast<const float4 *>(a.norm_w)[g];
            w[p] = make_float4(r.x * n.x, r.y * n.y, r.z * n.z, r.w * n.w);
        }
    }
    pdl_wait();
    pdl_trigger();
    stage_vec4(a.x, xf, d, tid, QH_THREADS);
    __syncthreads();
    float dot = 0.0f;
#pragma unroll
    for (int p = 0; p < QH_MAXG; p++) {
        const int g = tid + p * QH_THREADS;
        if (g < groups) {
            const float4 x = reinterpret_cast<const float4 *>(xf)[g];
            dot += w[p].x * x.x + w[p].y * x.y + w[p].z * x.z + w[p].w * x.w;
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) dot += __shfl_xor_sync(0xffffffffu, dot, o);
    if (lane == 0) red[warp] = dot;
    const float inv = qw_norm_inv(xf, d, a.eps, part, tid);
    if (tid == 0) a.est[e] = inv * (red[0] + red[1] + red[2] + red[3]);
    for (int sb = e + warp * gridDim.x; sb < d / 256; sb += gridDim.x * (QH_THREADS / 32)) {
        float v[8];
#pragma unroll
        for (int i = 0; i < 8; i++) v[i] = __fmul_rn(__fmul_rn(xf[sb * 256 + lane * 8 + i], inv), a.norm_w[sb * 256 + lane * 8 + i]);
        warp_quant_q8k16(v, lane, a.q + sb * 256, a.s + sb, a.b16 + sb * 16);
    }
}

// ---------------------------------------------------------------- experts: gate/up + SiLU-GLU (engine_qwen2.rs:419-426)
// The (slot, row) pairs of gate and up rows are dealt out in runs, so that every SM streams the same bytes (42 pairs, 97 KB); the rows land
// in groups of sixteen, a row of each matrix per warp.  Nothing is known before the wait: est picks the experts here.
struct QGateUpArgs {
    KMatDev gate, up;
    const float *est;            // nullptr: top
    const int32_t *top;
    int ne, topk, ff, per_cta, stride_g, stride_u;
    const int8_t *q;
    const float *s;
    const int32_t *b16;
    float *hbuf;                 // [slot][ff]
    DevState *state;
};

template <int UPL>
__global__ void __launch_bounds__(QG_THREADS, 2) qw_gate_up_kernel(const __grid_constant__ QGateUpArgs a) {
    extern __shared__ __align__(16) unsigned char qsm[];
    __shared__ SelectScratch ws;
    __shared__ int sel[8];
    __shared__ __align__(8) uint64_t bar[16];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, K = a.gate.cols, nsb = K / 256;
    const int i0 = blockIdx.x * a.per_cta, n = min(a.per_cta, a.topk * a.ff - i0), groups = (n + QG_WARPS - 1) / QG_WARPS;
    unsigned char *rg = qsm, *ru = qsm + (size_t)a.per_cta * a.stride_g;
    int8_t *q = reinterpret_cast<int8_t *>(ru + (size_t)a.per_cta * a.stride_u);
    float *s = reinterpret_cast<float *>(q + K);
    int32_t *b16 = reinterpret_cast<int32_t *>(s + ((nsb + 3) & ~3));
    float *terms = reinterpret_cast<float *>(b16 + nsb * 16);      // [row][gate, up][nsb]
    Waiter waiter(a.state ? &a.state->err : nullptr);
    if (tid == 0) {
        for (int i = 0; i < groups; i++) mbar_init(&bar[i], 1);
        mbar_fence_init();
    }
    pdl_wait();
    pdl_trigger();
    waiter.poison_if_failed();
    for (int i = tid; i < K / 16; i += QG_THREADS) reinterpret_cast<int4 *>(q)[i] = reinterpret_cast<const int4 *>(a.q)[i];
    for (int i = tid; i < nsb; i += QG_THREADS) s[i] = a.s[i];
    for (int i = tid; i < nsb * 16; i += QG_THREADS) b16[i] = a.b16[i];
    if (a.est) qw_select(a.est, a.ne, a.topk, a.state, ws, sel, tid, QG_THREADS);
    else { if (tid < a.topk) sel[tid] = a.top[tid]; __syncthreads(); }
    if (tid < groups) mbar_expect_tx(&bar[tid], (uint32_t)min(QG_WARPS, n - tid * QG_WARPS) * (uint32_t)(a.stride_g + a.stride_u));
    for (int i = tid; i < 2 * n; i += QG_THREADS) {
        const int r = i >> 1, it = i0 + r, ei = it / a.ff;
        const size_t row = (size_t)sel[ei] * a.ff + (it - ei * a.ff);
        if (i & 1) bulk_g2s(ru + (size_t)r * a.stride_u, a.up.p + row * a.stride_u, (uint32_t)a.stride_u, &bar[r / QG_WARPS]);
        else bulk_g2s(rg + (size_t)r * a.stride_g, a.gate.p + row * a.stride_g, (uint32_t)a.stride_g, &bar[r / QG_WARPS]);
    }
    QLane<UPL> x;
    qw_lane_load<UPL>(a.gate.type, nsb, q, s, b16, lane, x);
    for (int k = 0; k < groups; k++) {
        const int i = k * QG_WARPS + warp;
        if (i >= n) break;
        waiter.wait(&bar[k], 0u);
        qw_row_terms<UPL>(a.gate.type, nsb, rg + (size_t)i * a.stride_g, x, lane, terms + (size_t)i * 2 * nsb);
        if (a.up.type != a.gate.type) qw_lane_load<UPL>(a.up.type, nsb, q, s, b16, lane, x);
        qw_row_terms<UPL>(a.up.type, nsb, ru + (size_t)i * a.stride_u, x, lane, terms + (size_t)i * 2 * nsb + nsb);
        if (a.up.type != a.gate.type) qw_lane_load<UPL>(a.gate.type, nsb, q, s, b16, lane, x);
    }
    __syncthreads();
    if (tid < n) {
        const float g = qw_terms_sum(terms + (size_t)tid * 2 * nsb, nsb), u = qw_terms_sum(terms + (size_t)tid * 2 * nsb + nsb, nsb);
        a.hbuf[i0 + tid] = __fmul_rn(__fdiv_rn(g, __fadd_rn(1.0f, brrr_expf_dev(-g))), u);
    }
}

// ---------------------------------------------------------------- down projection of every slot (engine_qwen2.rs:432-441)
// A CTA owns per_cta rows of each of the slots' matrices: contiguous in memory, fetched before the wait (the routing is two kernels
// old).  Prologue: Q8_K of h (every CTA all of it: 24 KB from L2).  part[slot][row] = dot; the weights and the order of the combine come
// later (QFold).
struct QDownArgs {
    KMatDev down;
    const float *est;
    const int32_t *top;
    int ne, topk, d, ff, per_cta;
    const float *hbuf;
    float *part;
    DevState *state;
};

__global__ void __launch_bounds__(QG_THREADS, 2) qw_down_kernel(const __grid_constant__ QDownArgs a) {
    extern __shared__ __align__(16) unsigned char qsm[];
    __shared__ SelectScratch ws;
    __shared__ int sel[8];
    __shared__ __align__(8) uint64_t bar;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 3, l8 = lane & 7;
    const int nsb = a.ff / 256, nun = a.topk * nsb, rb = (int)a.down.bpr(), r0 = blockIdx.x * a.per_cta, n = min(a.per_cta, a.d - r0);
    unsigned char *rows = qsm;                                         // [slot][row]
    int8_t *q = reinterpret_cast<int8_t *>(rows + (size_t)a.topk * a.per_cta * rb);
    float *s = reinterpret_cast<float *>(q + nun * 256);
    int32_t *b16 = reinterpret_cast<int32_t *>(s + ((nun + 3) & ~3));
    float *terms = reinterpret_cast<float *>(b16 + nun * 16);          // [row][slot][nsb]
    Waiter waiter(a.state ? &a.state->err : nullptr);
    if (tid == 0) { mbar_init(&bar, 1); mbar_fence_init(); }
    if (a.est) qw_select(a.est, a.ne, a.topk, a.state, ws, sel, tid, QG_THREADS);
    else { if (tid < a.topk) sel[tid] = a.top[tid]; __syncthreads(); }
    if (tid == 0) mbar_expect_tx(&bar, (uint32_t)a.topk * n * rb);
    if (tid < a.topk) bulk_g2s(rows + (size_t)tid * a.per_cta * rb, a.down.p + ((size_t)sel[tid] * a.d + r0) * rb, (uint32_t)n * rb, &bar);
    pdl_wait();          // h is complete
    pdl_trigger();
    waiter.poison_if_failed();
    for (int sb = warp; sb < nun; sb += QG_WARPS) {
        const float4 *src = reinterpret_cast<const float4 *>(a.hbuf + (size_t)sb * 256 + lane * 8);
        const float4 p0 = src[0], p1 = src[1];
        const float v[8] = {p0.x, p0.y, p0.z, p0.w, p1.x, p1.y, p1.z, p1.w};
        warp_quant_q8k16(v, lane, q + sb * 256, s + sb, b16 + sb * 16);
    }
    __syncthreads();
    waiter.wait(&bar, 0u);
    // (row, eight units) at a time: unit = slot * nsb + superblock
    const int per_row = (nun + 7) / 8, type = a.down.type;
    for (int it = warp; it < n * per_row; it += QG_WARPS) {
        const int r = it / per_row, u0 = (it - r * per_row) * 8 + g, u1 = u0 + 4, c0 = min(u0, nun - 1), c1 = min(u1, nun - 1);
        KAct x0, x1;
        kact_load(type, q + c0 * 256, b16 + c0 * 16, l8, x0);
        kact_load(type, q + c1 * 256, b16 + c1 * 16, l8, x1);
        const int e0 = c0 / nsb, e1 = c1 / nsb;
        const float t = kq_pair_term(type, nsb, rows + ((size_t)e0 * a.per_cta + r) * rb, c0 - e0 * nsb, x0, s[c0], rows + ((size_t)e1 * a.per_cta + r) * rb, c1 - e1 * nsb, x1,
                                     s[c1], l8);
        const int u = l8 ? u1 : u0;
        if (!(l8 & 3) && u < nun) terms[r * nun + u] = t;
    }
    __syncthreads();
    for (int i = tid; i < n * a.topk; i += QG_THREADS) {
        const int slot = i / n, r = i - slot * n;
        a.part[(size_t)slot * a.d + r0 + r] = qw_terms_sum(terms + r * nun + slot * nsb, nsb);
    }
}

// ---------------------------------------------------------------- vocabulary projection + argmax (engine_qwen2.rs:436-448)
// Persistent: a CTA streams its run of rows through a ring of 16-row stages, a row per warp; the ring fills before the dependency wait.
// Bound: HBM (255 MB at 151936 x 2048).
struct QHeadArgs {
    KMatDev m;
    const int8_t *q;
    const float *s;
    const int32_t *b16;
    float *logits;
    DevState *state;
    int per_cta, depth;
};

template <int UPL>
__global__ void __launch_bounds__(QG_THREADS + 32) qw_head_kernel(const __grid_constant__ QHeadArgs a) {
    extern __shared__ __align__(16) unsigned char qsm[];
    __shared__ __align__(8) uint64_t full[8], empty[8];
    __shared__ unsigned long long wbest[QG_WARPS];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, nsb = a.m.cols / 256, rb = (int)a.m.bpr(), depth = a.depth;
    const int row0 = blockIdx.x * a.per_cta, n = min(a.per_cta, a.m.rows - row0), stages = (n + QG_WARPS - 1) / QG_WARPS;
    Waiter waiter(&a.state->err);
    if (tid == 0) {
        for (int i = 0; i < depth; i++) { mbar_init(&full[i], 1); mbar_init(&empty[i], QG_WARPS); }
        mbar_fence_init();
    }
    __syncthreads();
    if (warp == QG_WARPS) {
        if (lane == 0) {
            pdl_trigger();
            for (int t = 0; t < stages; t++) {
                const int slot = t % depth;
                if (t >= depth) waiter.wait(&empty[slot], (uint32_t)(t / depth - 1) & 1u);
                const uint32_t bytes = (uint32_t)min(QG_WARPS, n - t * QG_WARPS) * rb;
                mbar_expect_tx(&full[slot], bytes);
                bulk_g2s(qsm + (size_t)slot * QG_WARPS * rb, a.m.p + (size_t)(row0 + t * QG_WARPS) * rb, bytes, &full[slot]);
            }
        }
        return;
    }
    pdl_wait();
    pdl_trigger();
    waiter.poison_if_failed();
    QLane<UPL> x;
    qw_lane_load<UPL>(a.m.type, nsb, a.q, a.s, a.b16, lane, x);
    float *terms = reinterpret_cast<float *>(qsm + (size_t)depth * QG_WARPS * rb) + warp * 2 * nsb;      // the warp's own, two rows
    unsigned long long best = 0ull;
    for (int t = 0; t < stages; t++) {
        const int slot = t % depth, i = t * QG_WARPS + warp;
        waiter.wait(&full[slot], (uint32_t)(t / depth) & 1u);
        float *tr = terms + (t & 1) * nsb;
        if (i < n) qw_row_terms<UPL>(a.m.type, nsb, qsm + (size_t)(slot * QG_WARPS + warp) * rb, x, lane, tr);
        __syncwarp();
        if (lane == 0) {
            mbar_arrive(&empty[slot]);
            if (i < n) {
                const float v = qw_terms_sum(tr, nsb);
                a.logits[row0 + i] = v;
                const unsigned long long key = ((unsigned long long)float_orderable(v) << 32) | (0xFFFFFFFFu - (uint32_t)(row0 + i));
                best = key > best ? key : best;
            }
        }
    }
    if (lane == 0) wbest[warp] = best;
    asm volatile("bar.sync 1, %0;" ::"r"(QG_THREADS) : "memory");
    if (tid == 0) {
#pragma unroll
        for (int w = 1; w < QG_WARPS; w++) best = wbest[w] > best ? wbest[w] : best;
        if (best) atomicMax(&a.state->best, best);
    }
}

// ---------------------------------------------------------------- load-time re-layout of Q6_K rows into aligned planes
__global__ void q6k_planes_kernel(const uint8_t *__restrict__ src, size_t rows, int nsb, uint8_t *__restrict__ dst) {
    const size_t rb = q6k_plane_row_bytes(nsb), total = rows * rb;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x) {
        const size_t row = i / rb;
        const int o = (int)(i % rb);
        const uint8_t *r = src + row * (size_t)nsb * 210;
        uint8_t v = 0;
        if (o < nsb * 128) v = r[(o / 128) * 210 + o % 128];
        else if (o < nsb * 192) { const int k = o - nsb * 128; v = r[(k / 64) * 210 + 128 + k % 64]; }
        else if (o < nsb * 208) { const int k = o - nsb * 192; v = r[(k / 16) * 210 + 192 + k % 16]; }
        else if (o < nsb * 210) { const int k = o - nsb * 208; v = r[(k / 2) * 210 + 208 + k % 2]; }
        dst[i] = v;
    }
}

// units per lane for rows of nsb superblocks: 2 or 4 (nsb <= 16)
int qw_upl(int nsb) { return nsb <= 8 ? 2 : nsb <= 16 ? 4 : 0; }
size_t qw_act_bytes(int nsb) { return (size_t)nsb * 256 + (size_t)((nsb + 3) & ~3) * 4 + (size_t)nsb * 64; }
bool qw_type_ok(const KMatDev &m) { return m.type == 12 || (m.type == 14 && m.planes); }
int qw_rows_per_cta(int rows, size_t bytes_per_row) {      // an even share of 148 SMs, unless that takes more shared memory than two kernels can share
    const int share = (rows + 147) / 148, fit = (int)(QG_ROW_BYTES / bytes_per_row);
    return share < fit ? share : fit;
}
constexpr int QG_SMEM_MAX = 200 * 1024;

template <int UPL, bool FOLD>
cudaError_t qw_gemv_launch(const QGemvArgs &a, size_t smem, bool pdl, cudaStream_t st) {
    static unsigned long long configured = 0;      // one bit per device
    cudaError_t e = smem_optin(qw_gemv_kernel<UPL, FOLD>, QG_SMEM_MAX, configured);
    if (e != cudaSuccess) return e;
    return launch_k(qw_gemv_kernel<UPL, FOLD>, dim3((a.k.rows + a.k.per_cta - 1) / a.k.per_cta), dim3(QG_THREADS), smem, st, pdl, a);
}

cudaError_t qw_gemv(const KMatDev *mats, float *const *ys_out, int n, const QFold *f, const float *act, DevState *state, bool pdl, cudaStream_t st) {
    QGemvArgs a{};
    a.k.n = n;
    size_t stride = 0;
    for (int i = 0; i < n; i++) {
        a.k.m[i] = mats[i]; a.k.y[i] = ys_out[i]; a.k.rows += mats[i].rows;
        if (mats[i].bpr() > stride) stride = mats[i].bpr();
        if (mats[i].cols != mats[0].cols || !qw_type_ok(mats[i])) return cudaErrorInvalidValue;
    }
    const int K = mats[0].cols, nsb = K / 256, upl = qw_upl(nsb);
    if (!upl || (f && (f->d != K || f->topk > 8 || f->ne > 256))) return cudaErrorInvalidValue;
    a.k.stride = (int)stride;
    a.k.per_cta = qw_rows_per_cta(a.k.rows, stride + nsb * 4);
    if (f) a.f = *f;
    a.act = act; a.state = state;
    const size_t smem = (size_t)a.k.per_cta * (stride + nsb * 4) + qw_act_bytes(nsb) + (f ? (size_t)K * 4 : 0);
    if (f) return upl == 2 ? qw_gemv_launch<2, true>(a, smem, pdl, st) : qw_gemv_launch<4, true>(a, smem, pdl, st);
    return upl == 2 ? qw_gemv_launch<2, false>(a, smem, pdl, st) : qw_gemv_launch<4, false>(a, smem, pdl, st);
}

template <int UPL>
cudaError_t qw_gate_up_launch(const QGateUpArgs &a, size_t smem, bool pdl, cudaStream_t st) {
    static unsigned long long configured = 0;      // one bit per device
    cudaError_t e = smem_optin(qw_gate_up_kernel<UPL>, QG_SMEM_MAX, configured);
    if (e != cudaSuccess) return e;
    return launch_k(qw_gate_up_kernel<UPL>, dim3((a.topk * a.ff + a.per_cta - 1) / a.per_cta), dim3(QG_THREADS), smem, st, pdl, a);
}
template <int UPL>
cudaError_t qw_head_launch(const QHeadArgs &a, size_t smem, bool pdl, cudaStream_t st) {
    static unsigned long long configured = 0;      // one bit per device
    cudaError_t e = smem_optin(qw_head_kernel<UPL>, 224 * 1024, configured);
    if (e != cudaSuccess) return e;
    return launch_k(qw_head_kernel<UPL>, dim3((a.m.rows + a.per_cta - 1) / a.per_cta), dim3(QG_THREADS + 32), smem, st, pdl, a);
}
QFold qw_fold_args(const QwCombine &c) { return QFold{c.x_in, c.part, c.x_out, c.est, c.top, c.wts, c.ne, c.topk, c.d, c.seq, c.norm_w, c.eps, c.state}; }

}  // namespace

// ---------------------------------------------------------------- launchers
cudaError_t launch_qw_embed(const uint8_t *embd, int d, DevState *state, float *x, bool pdl, cudaStream_t st) {
    return launch_k(qw_embed_kernel, dim3(d / 256), dim3(256), 0, st, pdl, embd, d, state, x);
}

cudaError_t launch_qw_fold(const QwCombine &c, int8_t *q, float *s, int32_t *b16, bool pdl, cudaStream_t st) {
    if (c.topk > 8 || c.ne > 256 || c.d > 8192) return cudaErrorInvalidValue;
    return launch_k(qw_fold_kernel, dim3(1), dim3(QG_THREADS), (size_t)c.d * 4, st, pdl, qw_fold_args(c), q, s, b16);
}

cudaError_t launch_qw_qkv(const KMatDev *mats, float *const *ys_out, const QwCombine &c, bool pdl, cudaStream_t st) {
    const QFold f = qw_fold_args(c);
    return qw_gemv(mats, ys_out, 3, &f, nullptr, c.state, pdl, st);
}

cudaError_t launch_qw_oproj(const KMatDev &wo, const float *act, float *x, DevState *state, bool pdl, cudaStream_t st) {
    return qw_gemv(&wo, &x, 1, nullptr, act, state, pdl, st);
}

cudaError_t launch_qw_attn(const float *q, const float *k, const float *v, const float *q_norm, const float *k_norm, const float *rope, float eps, float *kc, float *vc,
                           int nh, int nkv, DevState *state, float *out, bool pdl, cudaStream_t st) {
    static unsigned long long configured = 0;      // one bit per device
    cudaError_t e = smem_optin(qw_attn_kernel, (int)QA_SMEM, configured);
    if (e != cudaSuccess) return e;
    QAttnArgs a{q, k, v, q_norm, k_norm, rope, eps, kc, vc, nh, nkv, state, out};
    return launch_k(qw_attn_kernel, dim3(nh), dim3(QA_THREADS), QA_SMEM, st, pdl, a);
}

cudaError_t launch_qw_hint(const float *x, const float *norm_w, float eps, int d, const float *Wt, int ne, float *est, int8_t *q, float *s, int32_t *b16, bool pdl,
                           cudaStream_t st) {
    if (d > QH_MAXG * QH_THREADS * 4) return cudaErrorInvalidValue;
    QHintArgs a{x, norm_w, eps, d, ne, Wt, est, q, s, b16};
    return launch_k(qw_hint_kernel, dim3(ne), dim3(QH_THREADS), (size_t)d * 4, st, pdl, a);
}

cudaError_t launch_qw_gate_up(const KMatDev &gate, const KMatDev &up, const float *est, const int32_t *top, int ne, int topk, int ff, const int8_t *q, const float *s,
                              const int32_t *b16, float *hbuf, DevState *state, bool pdl, cudaStream_t st) {
    const int nsb = gate.cols / 256, upl = qw_upl(nsb);
    if (gate.cols != up.cols || !qw_type_ok(gate) || !qw_type_ok(up) || !upl || ne > 256 || topk > 8) return cudaErrorInvalidValue;
    QGateUpArgs a{gate, up, est, top, ne, topk, ff, 0, (int)gate.bpr(), (int)up.bpr(), q, s, b16, hbuf, state};
    const size_t row = (size_t)a.stride_g + a.stride_u + nsb * 8;
    a.per_cta = qw_rows_per_cta(topk * ff, row);
    if (a.per_cta > 256) return cudaErrorInvalidValue;
    const size_t smem = a.per_cta * row + qw_act_bytes(nsb);
    return upl == 2 ? qw_gate_up_launch<2>(a, smem, pdl, st) : qw_gate_up_launch<4>(a, smem, pdl, st);
}

cudaError_t launch_qw_down(const KMatDev &down, const float *est, const int32_t *top, int ne, int topk, int d, int ff, const float *hbuf, float *part, DevState *state,
                           bool pdl, cudaStream_t st) {
    if (!qw_type_ok(down) || ff % 256 || ff > 1024 || topk > 8 || ne > 256) return cudaErrorInvalidValue;
    QDownArgs a{down, est, top, ne, topk, d, ff, 0, hbuf, part, state};
    const int nun = topk * (ff / 256);
    const size_t row = (size_t)topk * down.bpr() + nun * 4;
    a.per_cta = qw_rows_per_cta(d, row);
    static unsigned long long configured = 0;      // one bit per device
    cudaError_t e = smem_optin(qw_down_kernel, QG_SMEM_MAX, configured);
    if (e != cudaSuccess) return e;
    return launch_k(qw_down_kernel, dim3((d + a.per_cta - 1) / a.per_cta), dim3(QG_THREADS), a.per_cta * row + qw_act_bytes(nun), st, pdl, a);
}

cudaError_t launch_qw_head(const KMatDev &head, const int8_t *q, const float *s, const int32_t *b16, float *logits, DevState *state, bool pdl, cudaStream_t st) {
    const int nsb = head.cols / 256, upl = qw_upl(nsb);
    if (!qw_type_ok(head) || !upl) return cudaErrorInvalidValue;
    const size_t stage = QG_WARPS * head.bpr(), terms = (size_t)QG_WARPS * 2 * nsb * 4;
    const int depth = (int)((220 * 1024 - terms) / stage);
    QHeadArgs a{head, q, s, b16, logits, state, (head.rows + 147) / 148, depth < 8 ? depth : 8};
    a.per_cta = (a.per_cta + QG_WARPS - 1) / QG_WARPS * QG_WARPS;
    const size_t smem = a.depth * stage + terms;
    return upl == 2 ? qw_head_launch<2>(a, smem, pdl, st) : qw_head_launch<4>(a, smem, pdl, st);
}

void launch_q6k_planes(const uint8_t *src, size_t rows, int cols, uint8_t *dst, cudaStream_t st) {
    if (rows) q6k_planes_kernel<<<1184, 256, 0, st>>>(src, rows, cols / 256, dst);
}

}  // namespace brrr
