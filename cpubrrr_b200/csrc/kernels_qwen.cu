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
//   q|k|v (prologue: norm, Q8_K) -> attention (prologue: QK norm, RoPE, cache append) -> o-proj (prologue: Q8_K) -> routing hint (norm,
//   Q8_K, estimate of the router) -> gate/up + SiLU-GLU of the estimated experts -> down of the same (prologue: Q8_K of h) + combine
// joined by programmatic dependent launch, while the exact router - a chain of d dependent adds, 4.3 us at best at d = 2048 - runs
// beside the last three on another stream and publishes its choice to the combine, which takes the weights and the order from it and
// flags the step if the estimate missed an expert (the host runs that step again without the estimate).
#include "brrr_kernels.h"
#include "brrr_kqt.cuh"
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
// The exact routing a step's combine uses, by one warp: slot_of[k] = slot (rank of the estimate) of the expert of rank k, wts[k] its weight.
// est: the words of the step's seq-th publication by the router, awaited with a bound (the router does not depend on any kernel that waits
// here, and the waiting kernels leave it room on an SM); picked: the estimate's expert of slot `lane`.  Else top and weights as they are.
__device__ __forceinline__ void qw_routing(bool est, int picked, const int32_t *top, const float *weights, int topk, uint32_t seq, DevState *state, int *slot_of, float *wts,
                                           int lane) {
    uint32_t payload = 0u;
    if (lane < 16 && (lane & 7) < topk) {
        if (est) {
            const uint32_t want = __ldcg(&state->fold_seq) + seq;
            const volatile unsigned long long *p = state->route_pub + lane;
            bool ok = false;
            const long long t0 = clock64();
            do {
                for (int i = 0; i < 64 && !ok; i++) {
                    const unsigned long long v = *p;
                    ok = (uint32_t)(v >> 32) == want;
                    payload = (uint32_t)v;
                }
            } while (!ok && clock64() - t0 < WAIT_CYCLES && *reinterpret_cast<volatile uint32_t *>(&state->err) == 0u);
            if (!ok) {               // the step is void from here: the host runs it again without the estimate
                atomicCAS(&state->err, (uint32_t)DEV_ERR_NONE, (uint32_t)DEV_ERR_PEER_TIMEOUT);
                atomicMin(&state->spec_fail_step, state->n_out);
            }
        } else payload = lane < 8 ? (uint32_t)__ldcg(top + lane) : __float_as_uint(__ldcg(weights + (lane - 8)));
    }
    if (lane >= 8 && lane < 8 + topk) wts[lane - 8] = __uint_as_float(payload);
    int found = -1;
    for (int s = 0; s < topk; s++) if (__shfl_sync(0xffffffffu, picked, s) == (int)payload) found = s;
    if (lane < topk) {
        int slot = lane;
        if (est) {
            slot = found;
            if (slot < 0) { slot = 0; atomicMin(&state->spec_fail_step, state->n_out); }      // the estimate missed this expert
        }
        slot_of[lane] = slot;
    }
}

// The 12-slice norm (engine_qwen2.rs:453-465) of xf (shared memory, synchronised): 1 / sqrt(mean + eps) in every thread.  beside(): run by every warp
// before the slices meet.
template <typename F>
__device__ __forceinline__ float qw_norm_inv(const float *xf, int d, float eps, float *part, int tid, F beside) {
    if (tid < QW_NT) {
        int lo, hi;
        qw_slice(tid, d, lo, hi);
        part[tid] = chain_squares(xf, lo, hi);
    }
    beside();
    __syncthreads();
    const float4 p0 = reinterpret_cast<const float4 *>(part)[0], p1 = reinterpret_cast<const float4 *>(part)[1], p2 = reinterpret_cast<const float4 *>(part)[2];
    const float p[QW_NT] = {p0.x, p0.y, p0.z, p0.w, p1.x, p1.y, p1.z, p1.w, p2.x, p2.y, p2.z, p2.w};
    float tot = 0.0f;
#pragma unroll
    for (int k = 0; k < QW_NT; k++) tot = __fadd_rn(tot, p[k]);
    return rms_inv(tot, d, eps);
}
__device__ __forceinline__ void qw_load8(const float *p, float (&v)[8]) {
    const float4 a = reinterpret_cast<const float4 *>(p)[0], b = reinterpret_cast<const float4 *>(p)[1];
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
}
// Norm and Q8_K of x (global) by a CTA of QG_THREADS, d <= 4096: warp w owns superblock w, whose norm weights it holds in nw.
template <int CHUNK>
__device__ __forceinline__ void qw_norm_image(const float *x, const float (&nw)[8], int d, float eps, float *xf, float *part, int8_t *q, float *s, int32_t *b16, int tid) {
    const int warp = tid >> 5, lane = tid & 31;
    for (int g = tid; g < d / 4; g += QG_THREADS) reinterpret_cast<float4 *>(xf)[g] = reinterpret_cast<const float4 *>(x)[g];
    __syncthreads();
    const float inv = qw_norm_inv(xf, d, eps, part, tid, []() {});
    if (warp < d / 256) {
        float v[8];
        qw_load8(xf + warp * 256 + lane * 8, v);
#pragma unroll
        for (int i = 0; i < 8; i++) v[i] = __fmul_rn(__fmul_rn(v[i], inv), nw[i]);
        warp_quant_q8k16<CHUNK>(v, lane, warp, q, s, b16);
    }
}

// the same as a kernel of its own, one CTA, image to global memory (the vocabulary head); x_copy (nullable): x as well
__global__ void __launch_bounds__(QG_THREADS) qw_norm_kernel(const float *__restrict__ x, const float *__restrict__ w, float eps, int d, int8_t *q, float *s, int32_t *b16,
                                                             float *x_copy) {
    extern __shared__ __align__(16) float xf[];
    __shared__ __align__(16) float part[QW_NT];
    const int tid = threadIdx.x;
    float nw[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    if ((tid >> 5) < d / 256) qw_load8(w + tid * 8, nw);
    pdl_wait_cta();
    pdl_trigger();
    qw_norm_image<64>(x, nw, d, eps, xf, part, q, s, b16, tid);
    if (x_copy)
        for (int i = tid; i < d; i += QG_THREADS) x_copy[i] = xf[i];
}

// ---------------------------------------------------------------- matrix rows x one activation (q|k|v, o-proj)
// Lane group g = lane / 4 takes superblocks g, g + 8 of every row.  Up to eight superblocks the activation stays in registers from row to row;
// of wider rows a warp has one or two, and it is read per eight superblocks (64 registers: two CTAs per SM).
template <int PASSES> struct QLane {
    KAct x;
    float ys;
    const int8_t *q;
    const float *s;
    const int32_t *b16;
};
template <int TYPE, int CHUNK, int PASSES>
__device__ __forceinline__ void qw_lane_load(int nsb, const int8_t *q, const float *s, const int32_t *b16, int lane, QLane<PASSES> &a) {
    if (PASSES == 1) {
        const int sb = min(lane >> 2, nsb - 1);
        kact_load<TYPE, CHUNK>(q, b16, sb, lane & 3, sb & 1, a.x);
        a.ys = s[sb];
    } else { a.q = q; a.s = s; a.b16 = b16; }
}
// superblock terms of a row (address in shared memory) -> terms[0 .. nsb)
template <int TYPE, int CHUNK, int PASSES>
__device__ __forceinline__ void qw_row_terms(int nsb, uint32_t row, QLane<PASSES> &a, int lane, float *terms) {
#pragma unroll 1
    for (int i = 0; i < PASSES; i++) {
        const int sb = (lane >> 2) + 8 * i, c = min(sb, nsb - 1);
        if (PASSES > 1) {
            kact_load<TYPE, CHUNK>(a.q, a.b16, c, lane & 3, c & 1, a.x);
            a.ys = a.s[c];
        }
        const float t = kq_term<TYPE>(nsb, row, c, a.x, a.ys, lane & 3, c & 1);
        if (!(lane & 3) && sb < nsb) terms[sb] = t;
    }
}
// rows [i0, i1) of a matrix, in shared memory from address rows on, a warp each
template <int TYPE, int PASSES>
__device__ __forceinline__ void qw_rows(int nsb, uint32_t rows, int stride, int i0, int i1, int8_t *q, const float *s, const int32_t *b16, float *terms, int warp, int lane) {
    QLane<PASSES> x;
    qw_lane_load<TYPE, KQ_SM_CHUNK>(nsb, q, s, b16, lane, x);
#pragma unroll 1
    for (int i = i0 + warp; i < i1; i += QG_WARPS) qw_row_terms<TYPE, KQ_SM_CHUNK>(nsb, rows + i * stride, x, lane, terms + i * nsb);
}
__device__ __forceinline__ float qw_terms_sum(const float *t, int nsb) {      // superblocks in order, from zero
    float v = 0.0f;
    int i = 0;
#pragma unroll 1
    for (; i + 8 <= nsb; i += 8) {
        float b[8];
#pragma unroll
        for (int k = 0; k < 8; k++) b[k] = t[i + k];
#pragma unroll
        for (int k = 0; k < 8; k++) v = __fadd_rn(v, b[k]);
    }
#pragma unroll 1
    for (; i < nsb; i++) v = __fadd_rn(v, t[i]);
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
    const float *x, *norm_w;     // NORM: the activation is the normalised residual x
    float eps;
    // else: x as it is; outputs are added to y
    DevState *state;
};

// Shared memory: rows | xf (NORM: K floats) | q | scales | 16-sums | terms.
// Bound: the hand-over, the prologue (norm: a chain of K / 12 adds) and one pass over rows that are already on chip.
template <int PASSES, bool NORM>
__global__ void __launch_bounds__(QG_THREADS, 2) qw_gemv_kernel(const __grid_constant__ QGemvArgs a) {
    extern __shared__ __align__(16) unsigned char qsm[];
    __shared__ __align__(16) float part[QW_NT];
    __shared__ __align__(8) uint64_t bar;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int K = a.k.m[0].cols, nsb = K / 256, row0 = blockIdx.x * a.k.per_cta, n = min(a.k.per_cta, a.k.rows - row0);
    unsigned char *rows = qsm;
    float *xf = reinterpret_cast<float *>(qsm + (size_t)a.k.per_cta * a.k.stride);
    int8_t *q = reinterpret_cast<int8_t *>(xf + (NORM ? K : 0));
    float *s = reinterpret_cast<float *>(q + nsb * 4 * KQ_SM_CHUNK);
    int32_t *b16 = reinterpret_cast<int32_t *>(s + ((nsb + 3) & ~3));
    float *terms = reinterpret_cast<float *>(b16 + nsb * 16);
    Waiter waiter(a.state ? &a.state->err : nullptr);
    if (tid == 0) {
        // whole runs of a matrix's rows; rows narrower than the stride (a stack of both types) one by one
        mbar_init(&bar, 1);
        mbar_fence_init();
        uint32_t bytes = 0;
        for (int pass = 0; pass < 2; pass++) {
            for (int i = 0, l; i < n;) {
                const KMatDev &m = a.k.m[a.k.find(row0 + i, l)];
                const int run = min(n - i, m.rows - l), rb = (int)m.bpr();
                if (pass == 0) bytes += (uint32_t)run * rb;
                else if (rb == a.k.stride) bulk_g2s(rows + (size_t)i * rb, m.p + (size_t)l * rb, (uint32_t)run * rb, &bar);
                else
                    for (int r = 0; r < run; r++) bulk_g2s(rows + (size_t)(i + r) * a.k.stride, m.p + (size_t)(l + r) * rb, (uint32_t)rb, &bar);
                i += run;
            }
            if (pass == 0) mbar_expect_tx(&bar, bytes);
        }
    }
    float resid = 0.0f, nw[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    int my_l = 0;
    const int my_m = tid < n ? a.k.find(row0 + tid, my_l) : 0;
    if (!NORM && tid < n) resid = a.k.y[my_m][my_l];         // written several kernels back
    if (NORM && warp < nsb) qw_load8(a.norm_w + tid * 8, nw);
    pdl_wait_cta();
    pdl_trigger();
    if (NORM) qw_norm_image<KQ_SM_CHUNK>(a.x, nw, K, a.eps, xf, part, q, s, b16, tid);
    else if (warp < nsb) {
        float v[8];
        qw_load8(a.x + tid * 8, v);
        warp_quant_q8k16<KQ_SM_CHUNK>(v, lane, warp, q, s, b16);
    }
    __syncthreads();
    waiter.wait(&bar, 0u);
    const uint32_t rows0 = smem_u32(rows);
#pragma unroll 1
    for (int i = 0, l; i < n;) {                 // one matrix of the stack after the other
        const int mi = a.k.find(row0 + i, l), end = i + min(n - i, a.k.m[mi].rows - l);
        if (a.k.m[mi].type == 12) qw_rows<12, PASSES>(nsb, rows0, a.k.stride, i, end, q, s, b16, terms, warp, lane);
        else qw_rows<14, PASSES>(nsb, rows0, a.k.stride, i, end, q, s, b16, terms, warp, lane);
        i = end;
    }
    __syncthreads();
    if (tid < n) {
        const float v = qw_terms_sum(terms + tid * nsb, nsb);
        a.k.y[my_m][my_l] = NORM ? v : __fadd_rn(resid, v);
    }
}

// ---------------------------------------------------------------- attention (engine_qwen2.rs:353-389, 466-482)
// One CTA per query head.  Prologue: QK norm (serial mean square) and RoPE of q and of the position's own k; the first head of a KV group
// appends k and v to the cache.  score(t): 8 chains (chain c covers dims c, c+8, ..., fused), (c + c+4) per lane, (l0+l1)+(l2+l3), times
// 1/sqrt(128); maximum over all keys; denominator and the 128 output sums serial over t.
// K, then V of the cached positions run through one ring of 64-position tiles that starts before the dependency wait: four tensor copies
// per tile, 32 dims each, their 16-byte chunks swizzled over the banks (chunk ^ position & 7) - 16-byte copies by the threads took 1000
// cycles of the load/store pipe per tile, a bulk copy per position 3400.
// Score threads are (key, two chains), keys of a phase two apart; p.V threads are the dims.
// Bound: at 100 positions the prologue's and softmax's latencies; then the chains over the keys (4 cycles each).
constexpr int QA_TILE = 64, QA_SLOTS = 5, QA_THREADS = 256, QA_ISSUER = 224;      // the issuer refills the ring: of the last warp, which carries no serial sum
constexpr uint32_t QA_BOX = QA_TILE * 128, QA_TILE_BYTES = 4 * QA_BOX;
constexpr size_t QA_SMEM = (size_t)QA_SLOTS * QA_TILE_BYTES + (size_t)BRRR_MAXSEQ * 4 + 1024;

struct alignas(64) QAttnArgs {
    CUtensorMap km, vm;          // the caches as [nkv * MAXSEQ][128], boxes of 64 positions x 32 dims
    const float *q, *k, *v, *q_norm, *k_norm, *rope;
    float eps;
    float *kc, *vc;              // [nkv][MAXSEQ][128]
    int nh, nkv;
    DevState *state;
    float *out;                  // [nh][128]
};

__device__ __forceinline__ void qa_box(uint32_t dst, const CUtensorMap *map, int x, int row, uint64_t *bar) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(dst), "l"(map), "r"(x), "r"(row),
                 "r"(smem_u32(bar))
                 : "memory");
}
__device__ __forceinline__ float2 qa_lds2(uint32_t a) {
    float2 r;
    asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(r.x), "=f"(r.y) : "r"(a));
    return r;
}
__device__ __forceinline__ float qa_lds(uint32_t a) {
    float r;
    asm volatile("ld.shared.f32 %0, [%1];" : "=f"(r) : "r"(a));
    return r;
}
// two chains of a key, then the others' in the four threads of a key: (c + c+4), (l0 + l1) + (l2 + l3)
__device__ __forceinline__ float qa_combine(float s0, float s1) {
    s0 = __fadd_rn(s0, __shfl_xor_sync(0xffffffffu, s0, 2));
    s1 = __fadd_rn(s1, __shfl_xor_sync(0xffffffffu, s1, 2));
    const float l = __fadd_rn(s0, s1);
    return __fadd_rn(l, __shfl_xor_sync(0xffffffffu, l, 1));
}

__global__ void __launch_bounds__(QA_THREADS) qw_attn_kernel(const __grid_constant__ QAttnArgs a) {
    extern __shared__ __align__(16) unsigned char asm_[];
    unsigned char *ring = asm_ + ((1024u - (smem_u32(asm_) & 1023u)) & 1023u);          // swizzled copies want 1024-byte alignment
    float *sc = reinterpret_cast<float *>(ring + QA_SLOTS * QA_TILE_BYTES);
    __shared__ __align__(16) float raw[2][QW_HD], nv[2][QW_HD], qs[QW_HD], ks[QW_HD], vs[QW_HD];
    __shared__ float red[8], inv_sh[2], den_sh;
    __shared__ __align__(8) uint64_t full[QA_SLOTS];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, u = tid & (QW_HD - 1), qk = tid >> 7;
    const int h = blockIdx.x, group = a.nh / a.nkv, kvh = h / group;
    const int pos = (int)a.state->pos, n = pos + 1, nt = (pos + QA_TILE - 1) / QA_TILE;        // the position is an input of the step
    const uint32_t ring0 = smem_u32(ring);
    Waiter waiter(&a.state->err);
    auto issue = [&](int t) {            // one thread: tile t of 2 nt, K then V (positions past the last cached one come along unused)
        const int slot = t % QA_SLOTS, row = kvh * BRRR_MAXSEQ + (t < nt ? t : t - nt) * QA_TILE;
        mbar_expect_tx(&full[slot], QA_TILE_BYTES);
#pragma unroll
        for (int b = 0; b < 4; b++) qa_box(ring0 + slot * QA_TILE_BYTES + b * QA_BOX, t < nt ? &a.km : &a.vm, b * 32, row, &full[slot]);
    };
    if (tid == 0) {
        for (int i = 0; i < QA_SLOTS; i++) mbar_init(&full[i], 1);
        mbar_fence_init();
        for (int t = 0; t < min(QA_SLOTS, 2 * nt); t++) issue(t);      // written in earlier steps
    }
    const float wv = (qk ? a.k_norm : a.q_norm)[u];
    const float2 cs = reinterpret_cast<const float2 *>(a.rope)[(size_t)pos * (QW_HD / 2) + (tid & 63)];
    pdl_wait_cta();
    pdl_trigger();
    raw[qk][u] = qk ? a.k[kvh * QW_HD + u] : a.q[h * QW_HD + u];
    if (!qk) vs[u] = a.v[kvh * QW_HD + u];
    waiter.poison_if_failed();
    __syncthreads();
    if (u == 0) inv_sh[qk] = rms_inv(chain_squares(raw[qk], 0, QW_HD), QW_HD, a.eps);
    __syncthreads();
    nv[qk][u] = __fmul_rn(__fmul_rn(raw[qk][u], inv_sh[qk]), wv);
    __syncthreads();
    {
        const int c = u & 63;
        const float aa = nv[qk][c], bb = nv[qk][64 + c];
        const float o = u < 64 ? __fsub_rn(__fmul_rn(aa, cs.x), __fmul_rn(bb, cs.y)) : __fadd_rn(__fmul_rn(bb, cs.x), __fmul_rn(aa, cs.y));
        (qk ? ks : qs)[u] = o;
        if (h % group == 0) {
            const size_t at = ((size_t)kvh * BRRR_MAXSEQ + pos) * QW_HD + u;
            if (qk) a.kc[at] = o;
            else a.vc[at] = vs[u];
        }
    }
    __syncthreads();
    // ---- scores: thread = (key, two chains)
    const float scale = __fdiv_rn(1.0f, __fsqrt_rn((float)QW_HD));
    const int c2 = (lane & 3) * 2, k8 = lane >> 2, key = warp * 8 + ((k8 & 3) * 2 | k8 >> 2);        // keys 0 2 4 6 1 3 5 7 of eight
    float2 qr[16];
#pragma unroll
    for (int i = 0; i < 16; i++) qr[i] = *reinterpret_cast<const float2 *>(qs + 8 * i + c2);
    float s0 = 0.0f, s1 = 0.0f;
#pragma unroll
    for (int i = 0; i < 16; i++) {
        const float2 k = *reinterpret_cast<const float2 *>(ks + 8 * i + c2);
        s0 = __fmaf_rn(k.x, qr[i].x, s0); s1 = __fmaf_rn(k.y, qr[i].y, s1);
    }
    float mx = __fmul_rn(qa_combine(s0, s1), scale);  // the position's own score, in every thread
    if (tid == 0) sc[pos] = mx;
    // chunk 2 (i & 3) + (c2 >> 2) of the key's row in box i >> 2
    uint32_t off[4];
#pragma unroll
    for (int i = 0; i < 4; i++) off[i] = (uint32_t)(key * 128 + (((2 * i + (c2 >> 2)) ^ (key & 7)) << 4) + (c2 & 2) * 4);
#pragma unroll 1
    for (int t = 0; t < nt; t++) {
        const int slot = t % QA_SLOTS;
        const uint32_t base = ring0 + slot * QA_TILE_BYTES;
        waiter.wait(&full[slot], (uint32_t)(t / QA_SLOTS) & 1u);
        s0 = s1 = 0.0f;
#pragma unroll
        for (int i = 0; i < 16; i++) {
            const float2 k = qa_lds2(base + (i >> 2) * QA_BOX + off[i & 3]);
            s0 = __fmaf_rn(k.x, qr[i].x, s0); s1 = __fmaf_rn(k.y, qr[i].y, s1);
        }
        const float s = __fmul_rn(qa_combine(s0, s1), scale);
        if (t * QA_TILE + key < pos) {
            mx = fmaxf(mx, s);
            if (!(lane & 3)) sc[t * QA_TILE + key] = s;
        }
        if (t + QA_SLOTS < 2 * nt) {
            __syncthreads();
            if (tid == QA_ISSUER) { fence_proxy_async(); issue(t + QA_SLOTS); }
        }
    }
    mx = warp_max(mx);
    if (lane == 0) red[warp] = mx;
    __syncthreads();
    mx = red[0];
#pragma unroll
    for (int w = 1; w < 8; w++) mx = fmaxf(mx, red[w]);
#pragma unroll 1
    for (int t = tid; t < ((n + 3) & ~3); t += QA_THREADS) sc[t] = t < n ? brrr_expf_dev(__fsub_rn(sc[t], mx)) : 0.0f;      // +0 past the end changes no sum
    __syncthreads();
    float acc = 0.0f;
    float den = 0.0f;
    auto add_den = [&](int t0, int t1) {      // probabilities t0 .. t1 - 1, t0 a multiple of 4, the last four padded with +0 (tile by tile: this warp takes part in the barriers)
        float4 p = *reinterpret_cast<const float4 *>(sc + t0);
#pragma unroll 4
        for (int t = t0 + 4; t < t1 + 4; t += 4) {
            const float4 c = p;
            p = *reinterpret_cast<const float4 *>(sc + (t < t1 ? t : t0));
            den = __fadd_rn(den, c.x); den = __fadd_rn(den, c.y); den = __fadd_rn(den, c.z); den = __fadd_rn(den, c.w);
        }
    };
    // chunk lane / 4 of the position's row in box `warp`
    uint32_t voff[8];
#pragma unroll
    for (int i = 0; i < 8; i++) voff[i] = (uint32_t)((warp & 3) * QA_BOX + i * 128 + (((lane >> 2) ^ i) << 4) + (lane & 3) * 4);
#pragma unroll 1
    for (int t = 0; t < nt; t++) {
        const int slot = (nt + t) % QA_SLOTS;
        if (tid < QW_HD) {
            waiter.wait(&full[slot], (uint32_t)((nt + t) / QA_SLOTS) & 1u);
            // sixteen positions at a time, the next sixteen's values on the way (two sets of registers: reloading one set in place exposed
            // every load's latency); then the rest
            const int cnt = min(QA_TILE, pos - t * QA_TILE);
            const uint32_t vt = ring0 + slot * QA_TILE_BYTES;
            const float *pt = sc + t * QA_TILE;
            float v0[16], v1[16];
            float4 p0[4], p1[4];
            auto load = [&](float (&v)[16], float4 (&p)[4], int k) {
                const uint32_t w = vt + (k & (QA_TILE - 1)) * 128;
                const float *o = pt + (k & (QA_TILE - 1));
#pragma unroll
                for (int i = 0; i < 16; i++) v[i] = qa_lds(w + voff[i & 7] + (i >> 3) * 1024);
#pragma unroll
                for (int i = 0; i < 4; i++) p[i] = *reinterpret_cast<const float4 *>(o + 4 * i);
            };
            auto add = [&](const float (&v)[16], const float4 (&p)[4], int left) {
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    if (4 * i < left) acc = __fmaf_rn(v[4 * i], p[i].x, acc);
                    if (4 * i + 1 < left) acc = __fmaf_rn(v[4 * i + 1], p[i].y, acc);
                    if (4 * i + 2 < left) acc = __fmaf_rn(v[4 * i + 2], p[i].z, acc);
                    if (4 * i + 3 < left) acc = __fmaf_rn(v[4 * i + 3], p[i].w, acc);
                }
            };
            load(v0, p0, 0);
            int k = 0;
#pragma unroll 1
            for (; k + 32 <= cnt; k += 32) {
                load(v1, p1, k + 16);
                add(v0, p0, 16);
                load(v0, p0, k + 32);
                add(v1, p1, 16);
            }
            if (k < cnt) {
                load(v1, p1, k + 16);
                add(v0, p0, cnt - k);
                add(v1, p1, cnt - k - 16);
            }
        }
        if (tid == 128) add_den(t * QA_TILE, t + 1 < nt ? (t + 1) * QA_TILE : n);
        if (nt + t + QA_SLOTS < 2 * nt) {
            __syncthreads();
            if (tid == QA_ISSUER) { fence_proxy_async(); issue(nt + t + QA_SLOTS); }
        }
    }
    if (tid == 128) {
        if (nt == 0) add_den(0, n);
        den_sh = den;
    }
    __syncthreads();
    if (tid < QW_HD) a.out[h * QW_HD + tid] = __fmul_rn(__fmaf_rn(vs[tid], sc[pos], acc), __fdiv_rn(1.0f, den_sh));
}

// ---------------------------------------------------------------- routing hint
// One CTA per expert: an order-free estimate of its router logit (a few ulps from the serial chain), which only decides whose weights start
// moving (see qw_routing), and a share of the normalised token's Q8_K.  The router row and the norm weights are in registers before
// the dependency wait; the dot runs beside the norm's chains.
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
    __shared__ __align__(16) float part[QW_NT], red[QH_THREADS / 32];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, e = blockIdx.x, d = a.d, groups = d >> 2;
    const int ntiles = (d + RT_TJ - 1) / RT_TJ;
    const float *wrow = a.Wt + ((size_t)(e >> 5) * ntiles * 32 + (e & 31)) * RT_STRIDE;
    const int sb = e + warp * gridDim.x;         // this warp's superblock, if any (further ones: at the end)
    float4 w[QH_MAXG];           // router weight x norm weight
    float nw[8] = {0, 0, 0, 0, 0, 0, 0, 0};
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
    if (sb < d / 256) qw_load8(a.norm_w + sb * 256 + lane * 8, nw);
    pdl_wait_cta();
    pdl_trigger();
    float4 x[QH_MAXG];
#pragma unroll
    for (int p = 0; p < QH_MAXG; p++) {
        const int g = tid + p * QH_THREADS;
        x[p] = g < groups ? reinterpret_cast<const float4 *>(a.x)[g] : make_float4(0.f, 0.f, 0.f, 0.f);
    }
#pragma unroll
    for (int p = 0; p < QH_MAXG; p++) if (tid + p * QH_THREADS < groups) reinterpret_cast<float4 *>(xf)[tid + p * QH_THREADS] = x[p];
    __syncthreads();
    float dot = 0.0f;            // beside the norm's chains, which the twelve threads of warp 0 begin with
    const float inv = qw_norm_inv(xf, d, a.eps, part, tid, [&]() {
#pragma unroll
        for (int p = 0; p < QH_MAXG; p++) dot += w[p].x * x[p].x + w[p].y * x[p].y + w[p].z * x[p].z + w[p].w * x[p].w;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) dot += __shfl_xor_sync(0xffffffffu, dot, o);
        if (lane == 0) red[warp] = dot;
    });
    if (tid == 0) a.est[e] = inv * (red[0] + red[1] + red[2] + red[3]);
    for (int b = sb; b < d / 256; b += gridDim.x * (QH_THREADS / 32)) {
        float v[8];
        if (b != sb) qw_load8(a.norm_w + b * 256 + lane * 8, nw);
        qw_load8(xf + b * 256 + lane * 8, v);
#pragma unroll
        for (int i = 0; i < 8; i++) v[i] = __fmul_rn(__fmul_rn(v[i], inv), nw[i]);
        warp_quant_q8k16<64>(v, lane, b, a.q, a.s, a.b16);
    }
}

// ---------------------------------------------------------------- experts: gate/up + SiLU-GLU (engine_qwen2.rs:419-426)
// The (slot, row) pairs of gate and up rows are dealt out in runs, so that every SM streams the same bytes (42 pairs, 97 KB); they land in
// groups of sixteen, a row of each matrix per warp.  Nothing is known before the wait: the experts are picked here, then the copies start,
// one per run of rows (a bulk copy costs its SM about 50 cycles).
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

template <int G, int U> struct KPair { static constexpr int gate = G, up = U; };

template <int PASSES>
__global__ void __launch_bounds__(QG_THREADS, 2) qw_gate_up_kernel(const __grid_constant__ QGateUpArgs a) {
    extern __shared__ __align__(16) unsigned char qsm[];
    __shared__ __align__(8) uint64_t bar[16];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, nsb = a.gate.cols / 256;
    const int i0 = blockIdx.x * a.per_cta, n = min(a.per_cta, a.topk * a.ff - i0), groups = (n + QG_WARPS - 1) / QG_WARPS;
    unsigned char *rg = qsm, *ru = qsm + (size_t)a.per_cta * a.stride_g;
    float *terms = reinterpret_cast<float *>(ru + (size_t)a.per_cta * a.stride_u);      // [row][gate, up][nsb]
    Waiter waiter(a.state ? &a.state->err : nullptr);
    // copy = (group, matrix, first or second run: a group of sixteen pairs touches two slots at most), at most four per warp: a copy
    // costs the warp that issues it about 100 cycles, so they are spread over the warps
    const int copy = warp + QG_WARPS * lane, grp = copy >> 2;
    if (copy < 4 * groups && !(copy & 3)) {
        mbar_init(&bar[grp], 1);
        mbar_fence_init();
    }
    int run = 0, slot = 0;
    uint32_t bytes = 0, expert_bytes = 0;
    const uint8_t *src = nullptr;
    unsigned char *dst = nullptr;
    if (copy < 4 * groups) {
        const int up = (copy >> 1) & 1, r0 = grp * QG_WARPS, cnt = min(QG_WARPS, n - r0), stride = up ? a.stride_u : a.stride_g;
        int it = i0 + r0, r = r0;
        slot = it / a.ff;
        run = min(cnt, (slot + 1) * a.ff - it);
        if (copy & 1) { r += run; it += run; run = cnt - run; slot++; }
        dst = (up ? ru : rg) + (size_t)r * stride;
        src = (up ? a.up.p : a.gate.p) + (size_t)(it - slot * a.ff) * stride;
        bytes = (uint32_t)run * stride;
        expert_bytes = (uint32_t)a.ff * stride;
        if ((copy & 3) == 0) mbar_expect_tx(&bar[grp], (uint32_t)cnt * (uint32_t)(a.stride_g + a.stride_u));
    }
    pdl_wait_cta();
    if (__any_sync(0xffffffffu, run > 0)) {
        const int e = a.est ? spec_pick(a.est, a.ne, a.topk, a.topk, a.state, lane) : a.top[min(lane, a.topk - 1)];
        const int mine = __shfl_sync(0xffffffffu, e, slot);
        if (run > 0) bulk_g2s(dst, src + (size_t)mine * expert_bytes, bytes, &bar[grp]);
        if (warp == 0) pdl_trigger();           // only now (warp 0 always has a copy): the down projection fetches its rows at once, and these come first
    }
    waiter.poison_if_failed();
    // the activation from global memory (L1 after the first warp)
    const uint32_t rg0 = smem_u32(rg), ru0 = smem_u32(ru);
    auto walk = [&](auto types) {
        constexpr int TG = decltype(types)::gate, TU = decltype(types)::up;
        QLane<PASSES> x;
        qw_lane_load<TG, 64>(nsb, a.q, a.s, a.b16, lane, x);
#pragma unroll 1
        for (int k = 0; k < groups; k++) {
            const int i = k * QG_WARPS + warp;
            if (i >= n) break;
            waiter.wait(&bar[k], 0u);
            qw_row_terms<TG, 64>(nsb, rg0 + i * a.stride_g, x, lane, terms + (size_t)i * 2 * nsb);
            if (TG != TU) qw_lane_load<TU, 64>(nsb, a.q, a.s, a.b16, lane, x);
            qw_row_terms<TU, 64>(nsb, ru0 + i * a.stride_u, x, lane, terms + ((size_t)i * 2 + 1) * nsb);
            if (TG != TU) qw_lane_load<TG, 64>(nsb, a.q, a.s, a.b16, lane, x);
        }
    };
    if (a.gate.type == 12) { if (a.up.type == 12) walk(KPair<12, 12>()); else walk(KPair<12, 14>()); }
    else { if (a.up.type == 12) walk(KPair<14, 12>()); else walk(KPair<14, 14>()); }
    __syncthreads();
    if (tid < n) {
        const float g = qw_terms_sum(terms + (size_t)tid * 2 * nsb, nsb), u = qw_terms_sum(terms + (size_t)tid * 2 * nsb + nsb, nsb);
        a.hbuf[i0 + tid] = __fmul_rn(__fdiv_rn(g, __fadd_rn(1.0f, brrr_expf_dev(-g))), u);
    }
}

// ---------------------------------------------------------------- down projection and combine (engine_qwen2.rs:432-441)
// A CTA owns per_cta outputs: their rows of every slot's matrix are contiguous, fetched before the wait (the routing is two kernels
// old).  Prologue: Q8_K of h (every CTA all of it: 24 KB from L2).  Then x += w[k] dot[slot of k], the exact experts in rank order.
struct QDownArgs {
    KMatDev down;
    const float *est;
    const int32_t *top;
    const float *wts;
    uint32_t seq;
    int ne, topk, d, ff, per_cta;
    const float *hbuf;
    float *x;
    DevState *state;
};

constexpr int QD_THREADS = QG_THREADS + 32;        // the last warp fetches the routing beside the others

template <int TYPE>
__device__ __forceinline__ void qw_down_rows(const QDownArgs &a, uint32_t rows, int rb, int nsb, int nun, int n, const int8_t *q, const float *s, const int32_t *b16, float *terms,
                                             int warp, int lane) {
    // unit = slot * nsb + superblock; a warp keeps eight units' activations and takes every (16 / passes)-th row
    const int passes = (nun + 7) / 8, step = QG_WARPS / passes, pass = warp % passes;
    if (warp >= passes * step) return;
    const int un = pass * 8 + (lane >> 2), c = min(un, nun - 1), slot = c / nsb;
    KAct x;
    kact_load<TYPE, KQ_SM_CHUNK>(q, b16, c, lane & 3, c & 1, x);
    const float ys = s[c];
    const uint32_t base = rows + slot * a.per_cta * rb;
#pragma unroll 1
    for (int r = warp / passes; r < n; r += step) {
        const float t = kq_term<TYPE>(nsb, base + r * rb, c - slot * nsb, x, ys, lane & 3, c & 1);
        if (!(lane & 3) && un < nun) terms[r * nun + un] = t;
    }
}

__global__ void __launch_bounds__(QD_THREADS, 2) qw_down_kernel(const __grid_constant__ QDownArgs a) {
    extern __shared__ __align__(16) unsigned char qsm[];
    __shared__ int slot_of[8];
    __shared__ float wts[8];
    __shared__ __align__(8) uint64_t bar;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int nsb = a.ff / 256, nun = a.topk * nsb, rb = (int)a.down.bpr(), r0 = blockIdx.x * a.per_cta, n = min(a.per_cta, a.d - r0);
    unsigned char *rows = qsm;                                         // [slot][row]
    int8_t *q = reinterpret_cast<int8_t *>(rows + (size_t)a.topk * a.per_cta * rb);
    float *s = reinterpret_cast<float *>(q + nun * 4 * KQ_SM_CHUNK);
    int32_t *b16 = reinterpret_cast<int32_t *>(s + ((nun + 3) & ~3));
    float *terms = reinterpret_cast<float *>(b16 + nun * 16);          // [row][slot][nsb]
    float *dots = terms + (size_t)a.per_cta * nun;                     // [slot][row]
    Waiter waiter(a.state ? &a.state->err : nullptr);
    int picked = 0;              // warp 0 (the copies) and the last (the routing): the expert of slot `lane`
    if (warp == 0 || warp == QG_WARPS) picked = a.est ? spec_pick(a.est, a.ne, a.topk, a.topk, a.state, lane) : a.top[min(lane, a.topk - 1)];
    if (warp == 0) {
        if (lane == 0) {
            mbar_init(&bar, 1);
            mbar_fence_init();
            mbar_expect_tx(&bar, (uint32_t)a.topk * n * rb);
        }
        __syncwarp();
        if (lane < a.topk) bulk_g2s(rows + (size_t)lane * a.per_cta * rb, a.down.p + ((size_t)picked * a.d + r0) * rb, (uint32_t)n * rb, &bar);
    }
    float xr = tid < n ? a.x[r0 + tid] : 0.0f;                         // written several kernels back
    pdl_wait_cta();      // h is complete
    pdl_trigger();
    if (warp == QG_WARPS) qw_routing(a.est != nullptr, picked, a.top, a.wts, a.topk, a.seq, a.state, slot_of, wts, lane);
    else {
        for (int sb = warp; sb < nun; sb += QG_WARPS) {
            float v[8];
            qw_load8(a.hbuf + (size_t)sb * 256 + lane * 8, v);
            warp_quant_q8k16<KQ_SM_CHUNK>(v, lane, sb, q, s, b16);
        }
        asm volatile("bar.sync 1, %0;" ::"r"(QG_THREADS) : "memory");
        waiter.wait(&bar, 0u);
        if (a.down.type == 12) qw_down_rows<12>(a, smem_u32(rows), rb, nsb, nun, n, q, s, b16, terms, warp, lane);
        else qw_down_rows<14>(a, smem_u32(rows), rb, nsb, nun, n, q, s, b16, terms, warp, lane);
        asm volatile("bar.sync 1, %0;" ::"r"(QG_THREADS) : "memory");
        for (int i = tid; i < n * a.topk; i += QG_THREADS) {
            const int slot = i / n, r = i - slot * n;
            dots[slot * n + r] = qw_terms_sum(terms + r * nun + slot * nsb, nsb);
        }
    }
    __syncthreads();
    if (tid < n) {
        float p[8];
#pragma unroll
        for (int k = 0; k < 8; k++) p[k] = k < a.topk ? __fmul_rn(wts[k], dots[slot_of[k] * n + tid]) : 0.0f;
#pragma unroll
        for (int k = 0; k < 8; k++) if (k < a.topk) xr = __fadd_rn(xr, p[k]);
        a.x[r0 + tid] = xr;
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

template <int PASSES>
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
    float *terms = reinterpret_cast<float *>(qsm + (size_t)depth * QG_WARPS * rb) + warp * 2 * nsb;      // the warp's own, two rows
    unsigned long long best = 0ull;
    auto walk = [&](auto types) {
        constexpr int T = decltype(types)::gate;
        QLane<PASSES> x;
        qw_lane_load<T, 64>(nsb, a.q, a.s, a.b16, lane, x);
        const uint32_t mine = smem_u32(qsm) + warp * rb;
#pragma unroll 1
        for (int t = 0; t < stages; t++) {
            const int slot = t % depth, i = t * QG_WARPS + warp;
            waiter.wait(&full[slot], (uint32_t)(t / depth) & 1u);
            float *tr = terms + (t & 1) * nsb;
            if (i < n) qw_row_terms<T, 64>(nsb, mine + slot * QG_WARPS * rb, x, lane, tr);
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
    };
    if (a.m.type == 12) walk(KPair<12, 12>());
    else walk(KPair<14, 14>());
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

// passes of eight superblocks per row (16 at most)
int qw_passes(int nsb) { return nsb <= 8 ? 1 : nsb <= 16 ? 2 : 0; }
size_t qw_act_bytes(int nsb) { return (size_t)nsb * 4 * KQ_SM_CHUNK + (size_t)((nsb + 3) & ~3) * 4 + (size_t)nsb * 64; }
bool qw_type_ok(const KMatDev &m) { return m.type == 12 || (m.type == 14 && m.planes); }
// An even share of 140 SMs, unless that takes more shared memory than two kernels can share.
int qw_rows_per_cta(int rows, size_t bytes_per_row) {
    const int share = (rows + 139) / 140, fit = (int)(QG_ROW_BYTES / bytes_per_row);
    return share < fit ? share : fit;
}
constexpr int QG_SMEM_MAX = 200 * 1024;

struct QwPlan { int per_cta, ctas; size_t smem; };
// a stack of `rows` rows, `stride` bytes apart in shared memory, against one activation of nsb superblocks
QwPlan qw_gemv_plan(int rows, size_t stride, int nsb, bool norm) {
    const int per = qw_rows_per_cta(rows, stride + nsb * 4);
    return {per, (rows + per - 1) / per, (size_t)per * (stride + nsb * 4) + qw_act_bytes(nsb) + (norm ? (size_t)nsb * 1024 : 0)};
}
QwPlan qw_down_plan(const KMatDev &down, int topk, int d, int ff) {
    const int nun = topk * (ff / 256);
    const size_t row = (size_t)topk * down.bpr() + nun * 4 + topk * 4;
    const int per = qw_rows_per_cta(d, row);
    return {per, (d + per - 1) / per, per * row + qw_act_bytes(nun)};
}
size_t qw_stack_stride(const KMatDev *mats, int n) {
    size_t stride = 0;
    for (int i = 0; i < n; i++) if (mats[i].bpr() > stride) stride = mats[i].bpr();
    return stride;
}

template <int PASSES, bool NORM>
cudaError_t qw_gemv_launch(const QGemvArgs &a, size_t smem, bool pdl, cudaStream_t st) {
    static unsigned long long configured = 0;      // one bit per device
    cudaError_t e = smem_optin(qw_gemv_kernel<PASSES, NORM>, QG_SMEM_MAX, configured);
    if (e != cudaSuccess) return e;
    return launch_k(qw_gemv_kernel<PASSES, NORM>, dim3((a.k.rows + a.k.per_cta - 1) / a.k.per_cta), dim3(QG_THREADS), smem, st, pdl, a);
}

cudaError_t qw_gemv(const KMatDev *mats, float *const *ys_out, int n, const float *x, const float *norm_w, float eps, DevState *state, bool pdl, cudaStream_t st) {
    QGemvArgs a{};
    a.k.n = n;
    for (int i = 0; i < n; i++) {
        a.k.m[i] = mats[i]; a.k.y[i] = ys_out[i]; a.k.rows += mats[i].rows;
        if (mats[i].cols != mats[0].cols || !qw_type_ok(mats[i])) return cudaErrorInvalidValue;
    }
    const int nsb = mats[0].cols / 256, passes = qw_passes(nsb);
    if (!passes) return cudaErrorInvalidValue;
    a.k.stride = (int)qw_stack_stride(mats, n);
    const QwPlan p = qw_gemv_plan(a.k.rows, a.k.stride, nsb, norm_w != nullptr);
    a.k.per_cta = p.per_cta;
    a.x = x; a.norm_w = norm_w; a.eps = eps; a.state = state;
    if (norm_w) return passes == 1 ? qw_gemv_launch<1, true>(a, p.smem, pdl, st) : qw_gemv_launch<2, true>(a, p.smem, pdl, st);
    return passes == 1 ? qw_gemv_launch<1, false>(a, p.smem, pdl, st) : qw_gemv_launch<2, false>(a, p.smem, pdl, st);
}

template <int PASSES>
cudaError_t qw_gate_up_launch(const QGateUpArgs &a, size_t smem, bool pdl, cudaStream_t st) {
    static unsigned long long configured = 0;      // one bit per device
    cudaError_t e = smem_optin(qw_gate_up_kernel<PASSES>, QG_SMEM_MAX, configured);
    if (e != cudaSuccess) return e;
    return launch_k(qw_gate_up_kernel<PASSES>, dim3((a.topk * a.ff + a.per_cta - 1) / a.per_cta), dim3(QG_THREADS), smem, st, pdl, a);
}
template <int PASSES>
cudaError_t qw_head_launch(const QHeadArgs &a, size_t smem, bool pdl, cudaStream_t st) {
    static unsigned long long configured = 0;      // one bit per device
    cudaError_t e = smem_optin(qw_head_kernel<PASSES>, 224 * 1024, configured);
    if (e != cudaSuccess) return e;
    return launch_k(qw_head_kernel<PASSES>, dim3((a.m.rows + a.per_cta - 1) / a.per_cta), dim3(QG_THREADS + 32), smem, st, pdl, a);
}

}  // namespace

// ---------------------------------------------------------------- launchers
cudaError_t launch_qw_embed(const uint8_t *embd, int d, DevState *state, float *x, bool pdl, cudaStream_t st) {
    return launch_k(qw_embed_kernel, dim3(d / 256), dim3(256), 0, st, pdl, embd, d, state, x);
}

cudaError_t launch_qw_norm(const float *x, const float *norm_w, float eps, int d, int8_t *q, float *s, int32_t *b16, float *x_copy, bool pdl, cudaStream_t st) {
    if (d > 256 * QG_WARPS) return cudaErrorInvalidValue;
    return launch_k(qw_norm_kernel, dim3(1), dim3(QG_THREADS), (size_t)d * 4, st, pdl, x, norm_w, eps, d, q, s, b16, x_copy);
}

cudaError_t launch_qw_qkv(const KMatDev *mats, float *const *ys_out, const float *x, const float *norm_w, float eps, DevState *state, bool pdl, cudaStream_t st) {
    return qw_gemv(mats, ys_out, 3, x, norm_w, eps, state, pdl, st);
}

cudaError_t launch_qw_oproj(const KMatDev &wo, const float *act, float *x, DevState *state, bool pdl, cudaStream_t st) {
    return qw_gemv(&wo, &x, 1, act, nullptr, 0.0f, state, pdl, st);
}

cudaError_t launch_qw_attn(const QwCache &c, const float *q, const float *k, const float *v, const float *q_norm, const float *k_norm, const float *rope, float eps, int nh,
                           int nkv, DevState *state, float *out, bool pdl, cudaStream_t st) {
    static unsigned long long configured = 0;      // one bit per device
    cudaError_t e = smem_optin(qw_attn_kernel, (int)QA_SMEM, configured);
    if (e != cudaSuccess) return e;
    QAttnArgs a{c.km, c.vm, q, k, v, q_norm, k_norm, rope, eps, c.k, c.v, nh, nkv, state, out};
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
    const int nsb = gate.cols / 256, passes = qw_passes(nsb);
    if (gate.cols != up.cols || !qw_type_ok(gate) || !qw_type_ok(up) || !passes || ne > 256 || topk > 8) return cudaErrorInvalidValue;
    QGateUpArgs a{gate, up, est, top, ne, topk, ff, 0, (int)gate.bpr(), (int)up.bpr(), q, s, b16, hbuf, state};
    const size_t row = (size_t)a.stride_g + a.stride_u + nsb * 8;
    a.per_cta = qw_rows_per_cta(topk * ff, row);
    if (a.per_cta > 256) return cudaErrorInvalidValue;
    // at least 112 KB: no room beside it for the router's CTAs (117 KB), whose chains then have an SM of their own - 5.4 us instead of 8.8
    const size_t smem = a.per_cta * row > 112 * 1024 ? a.per_cta * row : 112 * 1024;
    return passes == 1 ? qw_gate_up_launch<1>(a, smem, pdl, st) : qw_gate_up_launch<2>(a, smem, pdl, st);
}

cudaError_t launch_qw_down(const KMatDev &down, const float *est, const int32_t *top, const float *wts, uint32_t seq, int ne, int topk, int d, int ff, const float *hbuf,
                           float *x, DevState *state, bool pdl, cudaStream_t st) {
    if (!qw_type_ok(down) || ff % 256 || ff > 1024 || topk > 8 || ne > 256) return cudaErrorInvalidValue;
    const QwPlan p = qw_down_plan(down, topk, d, ff);
    QDownArgs a{down, est, top, wts, seq, ne, topk, d, ff, p.per_cta, hbuf, x, state};
    static unsigned long long configured = 0;      // one bit per device
    cudaError_t e = smem_optin(qw_down_kernel, QG_SMEM_MAX, configured);
    if (e != cudaSuccess) return e;
    return launch_k(qw_down_kernel, dim3(p.ctas), dim3(QD_THREADS), p.smem, st, pdl, a);
}

// The kernels that can be on the SMs while the exact router has not published are the down projection, whose CTAs poll for its words, and the
// q|k|v projection behind it, whose CTAs wait for down's (what comes after q|k|v is launched only once down has ended, and gate/up and the
// hint end by themselves).  If an SM with one of their CTAs still takes a router CTA, an SM that refuses one holds two; with fewer
// than two per SM in all, some SM always has room and the router ends.  Registers and threads allow it (half an SM at most for
// either: launch bounds, ffn_in_takes_half_an_sm); shared memory decides.  Where this does not hold - rows of 4096 values, say, where the router alone takes 133 KB - the down
// projection must not start before the router has ended (a graph edge instead of the poll's bounded second).  One decoding
// engine per device is assumed; the kernels of others can only run the bounded wait out.
QwRoom qw_router_room(const KMatDev &down, const KMatDev *next_qkv, int ne, int topk, int d, int ff) {
    constexpr size_t SM_SMEM = 228 * 1024, CTA_EXTRA = 3 * 1024;       // CTA_EXTRA: the system's 1 KB and the kernels' static variables
    constexpr int SMS = 148;
    const QwPlan dn = qw_down_plan(down, topk, d, ff);
    // behind the last layer: the one CTA of the output norm
    const QwPlan nx = next_qkv ? qw_gemv_plan(next_qkv[0].rows + next_qkv[1].rows + next_qkv[2].rows, qw_stack_stride(next_qkv, 3), d / 256, true) : QwPlan{1, 1, (size_t)d * 4};
    QwRoom r{dn.ctas, nx.ctas, dn.smem, nx.smem, ffn_in_smem(ne, d), false};
    const size_t waiting = dn.smem > nx.smem ? dn.smem : nx.smem;
    const int per_sm = waiting + r.router_smem + 2 * CTA_EXTRA <= SM_SMEM ? 2 : 1;
    r.ok = dn.ctas + nx.ctas < per_sm * SMS;
    return r;
}

cudaError_t launch_qw_head(const KMatDev &head, const int8_t *q, const float *s, const int32_t *b16, float *logits, DevState *state, bool pdl, cudaStream_t st) {
    const int nsb = head.cols / 256, passes = qw_passes(nsb);
    if (!qw_type_ok(head) || !passes) return cudaErrorInvalidValue;
    const size_t stage = QG_WARPS * head.bpr(), terms = (size_t)QG_WARPS * 2 * nsb * 4;
    const int depth = (int)((220 * 1024 - terms) / stage);
    QHeadArgs a{head, q, s, b16, logits, state, (head.rows + 147) / 148, depth < 8 ? depth : 8};
    a.per_cta = (a.per_cta + QG_WARPS - 1) / QG_WARPS * QG_WARPS;
    const size_t smem = a.depth * stage + terms;
    return passes == 1 ? qw_head_launch<1>(a, smem, pdl, st) : qw_head_launch<2>(a, smem, pdl, st);
}

void launch_q6k_planes(const uint8_t *src, size_t rows, int cols, uint8_t *dst, cudaStream_t st) {
    if (rows) q6k_planes_kernel<<<1184, 256, 0, st>>>(src, rows, cols / 256, dst);
}

}  // namespace brrr
