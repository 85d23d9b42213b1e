// FFN entry stage: RMSNorm of the residual stream, router GEMV and top-k softmax.
//
// The router logit of expert e is the *serial* f32 sum  acc = b[e]; acc += W[e][j] * xn[j]
// for j ascending, multiply and add rounded separately.  That chain cannot be split without
// changing bits, so one lane owns one expert and walks the whole row: 4 cycles of dependent
// FADD latency per element is the floor of this stage.  The lane is kept fed from a ring of
// shared-memory tiles; each tile is ONE bulk asynchronous copy, because the router matrix is
// re-laid at load time as [32-expert group][tile][32 experts][256 + 4 floats] (the 4-float row
// padding makes a 128-bit read per lane bank-conflict free).  Experts are split 32 per CTA; with
// several CTAs the last one to finish runs the top-k.
#include "brrr_kernels.h"
#include "brrr_block.cuh"
#include "brrr_tma.cuh"
#include "brrr_mxt.cuh"
#include "brrr_kq.cuh"

namespace brrr {

constexpr int RT_STAGES = 5;
constexpr int RT_THREADS = 256;

// ---------------------------------------------------------------- pack: W[ne][d] -> tiled layout
__global__ void router_pack_kernel(const float *__restrict__ W, int ne, int d, float *__restrict__ out) {
    const int ntiles = (d + RT_TJ - 1) / RT_TJ;
    const size_t total = (size_t)((ne + 31) / 32) * ntiles * RT_TILE_FLOATS;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x) {
        int jj = (int)(i % RT_STRIDE);
        size_t r = i / RT_STRIDE;
        int el = (int)(r % 32);
        size_t gt = r / 32;
        int t = (int)(gt % ntiles), g = (int)(gt / ntiles);
        int e = g * 32 + el, j = t * RT_TJ + jj;
        out[i] = (jj < RT_TJ && e < ne && j < d) ? W[(size_t)e * d + j] : 0.0f;
    }
}

void launch_router_pack(const float *W, int ne, int d, float *out, cudaStream_t st) {
    router_pack_kernel<<<148, 256, 0, st>>>(W, ne, d, out);
}

// acc += w[j] * x[j] for j = 0..len-1 (len % 64 == 0), strictly in order, product and sum rounded separately.  The operands of the next
// sixteen products are read while sixteen sums are formed, so that only the adds sit on the dependent path (4 cycles each).
// LEN: known at compile time, or 0 (len); known, the loop takes 5 cycles per element, else 7.
template <int LEN>
__device__ __forceinline__ float chain_span(const float *__restrict__ w, const float *__restrict__ x, int len, float acc) {
    if (LEN) len = LEN;
    float4 a[4], b[4];
#pragma unroll
    for (int k = 0; k < 4; k++) { a[k] = *reinterpret_cast<const float4 *>(w + 4 * k); b[k] = *reinterpret_cast<const float4 *>(x + 4 * k); }
#pragma unroll 4
    for (int j = 0; j < len; j += 16) {
        float p[16];
#pragma unroll
        for (int k = 0; k < 4; k++) {
            p[4 * k] = __fmul_rn(a[k].x, b[k].x); p[4 * k + 1] = __fmul_rn(a[k].y, b[k].y);
            p[4 * k + 2] = __fmul_rn(a[k].z, b[k].z); p[4 * k + 3] = __fmul_rn(a[k].w, b[k].w);
        }
        const int n = j + 16 < len ? j + 16 : 0;         // past the end: the first ones again, unused
#pragma unroll
        for (int k = 0; k < 4; k++) { a[k] = *reinterpret_cast<const float4 *>(w + n + 4 * k); b[k] = *reinterpret_cast<const float4 *>(x + n + 4 * k); }
#pragma unroll
        for (int k = 0; k < 16; k++) acc = __fadd_rn(acc, p[k]);
    }
    return acc;
}

struct RouterArgs {
    const float *x_in;       // residual stream (norm_w != null) or normalised vector
    const float *norm_w;
    float eps;
    int d;
    const float *Wt;         // tiled router matrix (router_pack_kernel)
    const float *b;
    int ne, topk;
    float *logits;
    int32_t *top;
    float *wts;
    unsigned int *counter;
    DevState *state;
    uint32_t *signal;        // nullable: sequence number of the published routing
    unsigned long long *pub;
    // qwen3moe: the norm is the 12-slice one, and the first CTA also leaves the Q8_K image of the
    // normalised token (quants, scales per 256, sums per 16) for the gate/up kernel
    int qwen_norm;
    int8_t *q8k_q;
    float *q8k_s;
    int32_t *q8k_b16;
    int epc, stages;         // experts per CTA, tiles in flight: 32 and 5; many experts: 16 and 6, a CTA that fits
                             // beside one waiting decode kernel of an SM but not beside gate/up (whose sixteen warps would slow the chain)
};

// The k largest logits, the lower index first among equals, which is the order the reference's strict-'>' insertion produces; then the
// softmax over them in rank order.  One warp: rounds of a maximum over order-preserving keys (lane l holds experts l * per ..., so among
// equals the lowest lane has the lowest index).  Lane r ends with the expert and weight of rank r, and publishes them if asked to: words
// tagged with the sequence number `seq`, each valid by itself, for a consumer that does not wait for this kernel to end (the
// combine of the speculative step).  Launches that publish are serialised on one stream, so the sequence word has a single writer.
template <int PER>
__device__ __forceinline__ void warp_topk_n(const RouterArgs &a, const float *lg, int lane, uint32_t seq) {
    uint32_t key[PER];
#pragma unroll
    for (int i = 0; i < PER; i++) key[i] = lane * PER + i < a.ne ? max(float_orderable(__fadd_rn(lg[lane * PER + i], 0.0f)), 1u) : 0u;      // (-0 and +0 are equals)
    float mine = 0.0f;                           // lane r: logit and expert of rank r
    int mine_e = 0;
#pragma unroll 1
    for (int r = 0; r < a.topk; r++) {
        uint32_t best = key[0];
#pragma unroll
        for (int i = 1; i < PER; i++) best = max(best, key[i]);
        const uint32_t top = __reduce_max_sync(0xffffffffu, best);
        const int owner = __ffs(__ballot_sync(0xffffffffu, best == top)) - 1;
        int at = 0;
#pragma unroll
        for (int i = PER - 1; i >= 0; i--) if (key[i] == top) at = i;
        const int e = min(__shfl_sync(0xffffffffu, lane * PER + at, owner), a.ne - 1);
        if (lane == owner) {
#pragma unroll
            for (int i = 0; i < PER; i++) if (i == at) key[i] = 0u;
        }
        if (lane == r) { mine = lg[e]; mine_e = e; }
    }
    const float first = __shfl_sync(0xffffffffu, mine, 0);
    const float ex = lane < a.topk ? brrr_expf_dev(__fsub_rn(mine, first)) : 0.0f;
    float wsum = 0.0f;
#pragma unroll 4
    for (int i = 0; i < a.topk; i++) wsum = __fadd_rn(wsum, __shfl_sync(0xffffffffu, ex, i));
    const float w = __fdiv_rn(ex, wsum);
    if (lane < a.topk) {
#ifdef BRRR_TEST_HOOKS
        const bool silent = a.state && (a.state->test_hooks & 2u);      // test hook: the consumer's bounded wait runs out
#else
        constexpr bool silent = false;
#endif
        if (a.signal && !silent) {
            __stcg(&a.pub[lane], ((unsigned long long)seq << 32) | (uint32_t)mine_e);
            __stcg(&a.pub[8 + lane], ((unsigned long long)seq << 32) | __float_as_uint(w));
        }
        a.wts[lane] = w;
        a.top[lane] = mine_e;
        if (a.signal && !silent && lane == 0) __stcg(a.signal, seq);
    }
}
__device__ __forceinline__ void warp_topk(const RouterArgs &a, const float *lg, int lane, uint32_t seq) {
    if (a.ne <= 32) warp_topk_n<1>(a, lg, lane, seq);
    else if (a.ne <= 128) warp_topk_n<4>(a, lg, lane, seq);
    else warp_topk_n<8>(a, lg, lane, seq);
}

__global__ void __launch_bounds__(RT_THREADS) ffn_in_kernel(RouterArgs a) {
    // blockIdx.y = token of a tile: inputs d apart, logits ne apart, routing 8 entries apart, one arrival counter each
    a.x_in += (size_t)blockIdx.y * a.d;
    a.logits += (size_t)blockIdx.y * a.ne;
    a.top += blockIdx.y * 8;
    a.wts += blockIdx.y * 8;
    a.counter += blockIdx.y;
    extern __shared__ __align__(128) unsigned char smraw[];
    const int stages = a.stages, epc = a.epc, tile_floats = epc * RT_STRIDE;
    float *tiles = reinterpret_cast<float *>(smraw);                                        // [stages][32][RT_STRIDE]
    float *xn = reinterpret_cast<float *>(smraw + (size_t)tile_floats * 4 * stages);   // d floats
    float *lg = xn + a.d;                                                                   // ne floats (top-k staging)
    float *wn = lg + ((a.ne + 3) & ~3);                                        // d floats: norm weights (16-byte aligned: float4 stores)
    uint64_t *bars = reinterpret_cast<uint64_t *>(wn + a.d);                   // [stages] tile landed
    uint64_t *empty = bars + stages;                                        // [stages] tile consumed
    __shared__ float inv_sh;
    __shared__ int last_sh;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, d = a.d;
    uint32_t *err = a.state ? &a.state->err : nullptr;
    Waiter waiter(err);
    const int e0 = blockIdx.x * epc;
    const int nloc = min(epc, a.ne - e0);
    const int ntiles = (d + RT_TJ - 1) / RT_TJ;
    const float *wsrc = a.Wt + (size_t)(e0 >> 5) * ntiles * RT_TILE_FLOATS + (e0 & 31) * RT_STRIDE;

    auto issue = [&](int t) {                                       // one thread
        int slot = t % stages;
        mbar_expect_tx(&bars[slot], (uint32_t)tile_floats * 4);
        bulk_g2s(tiles + (size_t)slot * tile_floats, wsrc + (size_t)t * RT_TILE_FLOATS, (uint32_t)tile_floats * 4, &bars[slot]);
    };
    BRRR_STAMP(a.state, 0);
    if (tid == 0) {
        for (int s = 0; s < stages; s++) { mbar_init(&bars[s], 1); mbar_init(&empty[s], 1); }
        mbar_fence_init();
    }
    __syncwarp();
    if (tid < min(stages, ntiles)) issue(tid);        // one lane per stage: the copies' address translations overlap
    if (a.norm_w) stage_vec4(a.norm_w, wn, d, tid, RT_THREADS);             // static: fetched before the wait
    const uint32_t seq = a.signal ? __ldcg(a.signal) + 1u : 0u;             // the launch before on this stream has ended
    const float bias_pre = (warp == 0 && lane < nloc && a.b) ? a.b[e0 + lane] : 0.0f;
    BRRR_STAMP(a.state, 1);
    pdl_wait_cta();      // residual stream complete
    BRRR_STAMP(a.state, 2);
    BRRR_GT_GO(a.state, 30);
    pdl_trigger();
    waiter.poison_if_failed();
    stage_vec4(a.x_in, xn, d, tid, RT_THREADS);
    __syncthreads();
    if (a.norm_w) {
        float inv;
        if (a.qwen_norm) {
            __shared__ float part[QW_NT];
            if (tid < QW_NT) {
                int lo, hi;
                qw_slice(tid, d, lo, hi);
                part[tid] = chain_squares(xn, lo, hi);
            }
            __syncthreads();
            float tot = 0.0f;
#pragma unroll
            for (int k = 0; k < QW_NT; k++) tot = __fadd_rn(tot, part[k]);
            inv = rms_inv(tot, d, a.eps);
        } else inv = block_rms_inv(xn, d, a.eps, &inv_sh);
        for (int i = tid; i < d; i += RT_THREADS) xn[i] = __fmul_rn(__fmul_rn(xn[i], inv), wn[i]);
        __syncthreads();
    }
    if (a.q8k_q && blockIdx.x == 0 && blockIdx.y == 0 && warp >= 2) {
        // warps 2..7 of the first CTA, beside the chain warp: Q8_K of the normalised token
        for (int sb = warp - 2; sb < d / 256; sb += RT_THREADS / 32 - 2) {
            float v[8];
#pragma unroll
            for (int i = 0; i < 8; i++) v[i] = xn[sb * 256 + lane * 8 + i];
            warp_quant_q8k16<64>(v, lane, sb, a.q8k_q, a.q8k_s, a.q8k_b16);
        }
    }

    BRRR_STAMP(a.state, 3);
    if (warp == 1 && lane == 0) {
        // refill thread: as soon as the chain warp releases a slot, the tile stages ahead goes in
        for (int t = stages; t < ntiles; t++) {
            waiter.wait(&empty[t % stages], (uint32_t)(t / stages - 1) & 1u);
            fence_proxy_async();
            issue(t);
        }
    }
    if (warp == 0) {
        float acc = bias_pre;
        int slot = 0;
        uint32_t parity = 0;
        for (int t = 0; t < ntiles; t++) {
            if (t < 12) BRRR_STAMP(a.state, 8 + t);
            const int j0 = t * RT_TJ, len = min(RT_TJ, d - j0);
            waiter.wait(&bars[slot], parity);
            const float *row = tiles + (size_t)slot * tile_floats + min(lane, epc - 1) * RT_STRIDE;
            const float *xr = xn + j0;
            acc = len == RT_TJ ? chain_span<RT_TJ>(row, xr, len, acc) : chain_span<0>(row, xr, len, acc);
            __syncwarp();                      // all lanes are done reading this slot
            if (lane == 0 && t + stages < ntiles) mbar_arrive(&empty[slot]);
            if (++slot == stages) { slot = 0; parity ^= 1u; }
        }
        if (lane < nloc) {
            if (gridDim.x == 1) lg[lane] = acc;
            a.logits[e0 + lane] = acc;
        }
        BRRR_STAMP(a.state, 4);
        if (gridDim.x == 1) {                  // single CTA: top-k straight from shared memory
            __syncwarp();
            warp_topk(a, lg, lane, seq);
        }
        BRRR_STAMP(a.state, 5);
        BRRR_GT_END(a.state, 31);
    }
    if (gridDim.x == 1) return;

    // several CTAs: the last one to arrive runs the top-k over all logits
    __threadfence();
    __syncthreads();
    if (tid == 0) {
        unsigned prev = atomicAdd(a.counter, 1u);
        last_sh = (prev == gridDim.x - 1);
    }
    __syncthreads();
    if (!last_sh) return;
    __threadfence();
    for (int e = tid; e < a.ne; e += RT_THREADS) lg[e] = __ldcg(a.logits + e);
    __syncthreads();
    if (warp == 0) warp_topk(a, lg, lane, seq);
    if (tid == 0) *a.counter = 0u;
}

// ---------------------------------------------------------------- router of token rows (normalised rows in, routing out)
// The serial sum of a (token, expert) pair cannot be split, but the pairs are independent: lane = expert of a 32-expert group, TPW
// tokens per warp, four warps.  Weight and activation tiles (256 elements of d) come through one ring of bulk copies; a lane's 16-byte
// weight read serves TPW tokens, the activations are broadcast reads.  Shared-memory reads are the bound: (4 + TPW) x 4 wavefronts
// per four elements.  With several groups the last CTA of a token block runs the top-k of its tokens.
constexpr int RR_WARPS = 4, RR_STAGES = 3;

// acc[k] += w[j] * x[k][j] for j = 0 .. len - 1 in order (len % 64 == 0; LEN: known at compile time, or 0)
template <int TPW, int LEN>
__device__ __forceinline__ void rows_span(const float *w, const float *x, int len, float (&acc)[TPW]) {
    constexpr int STEP = TPW == 4 ? 8 : 16;
    if (LEN) len = LEN;
    // STEP elements of the row and of every token are in registers while the STEP before them are added up (len % 64 == 0)
    float4 wv[STEP / 4], xv[TPW][STEP / 4];
#pragma unroll
    for (int q = 0; q < STEP / 4; q++) {
        wv[q] = *reinterpret_cast<const float4 *>(w + 4 * q);
#pragma unroll
        for (int k = 0; k < TPW; k++) xv[k][q] = *reinterpret_cast<const float4 *>(x + k * RT_TJ + 4 * q);
    }
#pragma unroll 2
    for (int j = 0; j < len; j += STEP) {
        float p[TPW][STEP];
#pragma unroll
        for (int k = 0; k < TPW; k++)
#pragma unroll
            for (int q = 0; q < STEP / 4; q++) {
                p[k][4 * q] = __fmul_rn(wv[q].x, xv[k][q].x); p[k][4 * q + 1] = __fmul_rn(wv[q].y, xv[k][q].y);
                p[k][4 * q + 2] = __fmul_rn(wv[q].z, xv[k][q].z); p[k][4 * q + 3] = __fmul_rn(wv[q].w, xv[k][q].w);
            }
        const int jn = j + STEP < len ? j + STEP : 0;         // past the end: the first step again, unused
#pragma unroll
        for (int q = 0; q < STEP / 4; q++) {
            wv[q] = *reinterpret_cast<const float4 *>(w + jn + 4 * q);
#pragma unroll
            for (int k = 0; k < TPW; k++) xv[k][q] = *reinterpret_cast<const float4 *>(x + k * RT_TJ + jn + 4 * q);
        }
#pragma unroll
        for (int i = 0; i < STEP; i++)
#pragma unroll
            for (int k = 0; k < TPW; k++) acc[k] = __fadd_rn(acc[k], p[k][i]);
    }
}

template <int TPW>
__global__ void __launch_bounds__(RR_WARPS * 32) router_rows_kernel(RouterArgs a, int ntok) {
    constexpr int TT = RR_WARPS * TPW;
    constexpr size_t STAGE = (size_t)(RT_TILE_FLOATS + TT * RT_TJ) * 4;
    extern __shared__ __align__(128) unsigned char smraw[];
    __shared__ __align__(8) uint64_t full[RR_STAGES];
    __shared__ int last_sh;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, d = a.d;
    const int e0 = blockIdx.x * 32, t0 = blockIdx.y * TT, nt = min(TT, ntok - t0);
    const int ntiles = (d + RT_TJ - 1) / RT_TJ;
    const float *wsrc = a.Wt + (size_t)blockIdx.x * ntiles * RT_TILE_FLOATS;
    Waiter waiter(a.state ? &a.state->err : nullptr);
    if (tid == 0) {
        for (int s = 0; s < RR_STAGES; s++) mbar_init(&full[s], 1);
        mbar_fence_init();
    }
    auto issue = [&](int t, bool weights, bool rows) {            // warp 0; the barrier counts both parts
        unsigned char *st = smraw + (size_t)(t % RR_STAGES) * STAGE;
        const uint32_t len = (uint32_t)min(RT_TJ, d - t * RT_TJ) * 4;
        if (weights && lane == 0) {
            mbar_expect_tx(&full[t % RR_STAGES], RT_TILE_FLOATS * 4 + nt * len);
            bulk_g2s(st, wsrc + (size_t)t * RT_TILE_FLOATS, RT_TILE_FLOATS * 4, &full[t % RR_STAGES]);
        }
        __syncwarp();
        if (rows && lane < nt) bulk_g2s(st + (size_t)RT_TILE_FLOATS * 4 + lane * RT_TJ * 4, a.x_in + (size_t)(t0 + lane) * d + t * RT_TJ, len, &full[t % RR_STAGES]);
    };
    __syncthreads();
    if (warp == 0)
        for (int t = 0; t < min(RR_STAGES, ntiles); t++) issue(t, true, false);        // weights do not depend on the kernel before
    pdl_wait();
    pdl_trigger();
    waiter.poison_if_failed();
    if (warp == 0)
        for (int t = 0; t < min(RR_STAGES, ntiles); t++) issue(t, false, true);
    float acc[TPW];
#pragma unroll
    for (int k = 0; k < TPW; k++) acc[k] = (a.b && e0 + lane < a.ne) ? a.b[e0 + lane] : 0.0f;
    int slot = 0;
    uint32_t parity = 0;
    for (int t = 0; t < ntiles; t++) {
        const unsigned char *st = smraw + (size_t)slot * STAGE;
        waiter.wait(&full[slot], parity);
        if (++slot == RR_STAGES) { slot = 0; parity ^= 1u; }
        const float *w = reinterpret_cast<const float *>(st) + lane * RT_STRIDE, *x = reinterpret_cast<const float *>(st) + RT_TILE_FLOATS + warp * TPW * RT_TJ;
        const int len = min(RT_TJ, d - t * RT_TJ);
        if (len == RT_TJ) rows_span<TPW, RT_TJ>(w, x, len, acc);
        else rows_span<TPW, 0>(w, x, len, acc);
        __syncthreads();                      // the stage is free
        if (warp == 0 && t + RR_STAGES < ntiles) { fence_proxy_async(); issue(t + RR_STAGES, true, true); }
    }
    float *lg = reinterpret_cast<float *>(smraw) + warp * 256;        // top-k staging, a warp's own
    const bool one = gridDim.x == 1;
#pragma unroll
    for (int k = 0; k < TPW; k++)
        if (warp * TPW + k < nt && e0 + lane < a.ne) a.logits[(size_t)(t0 + warp * TPW + k) * a.ne + e0 + lane] = acc[k];
    if (!one) {
        __threadfence();
        __syncthreads();
        if (tid == 0) last_sh = atomicAdd(a.counter + blockIdx.y, 1u) == gridDim.x - 1;
        __syncthreads();
        if (!last_sh) return;
        __threadfence();
        if (tid == 0) a.counter[blockIdx.y] = 0u;
    }
#pragma unroll
    for (int k = 0; k < TPW; k++) {
        const int t = warp * TPW + k;
        if (t >= nt) break;
        __syncwarp();
        if (one) { if (lane < a.ne) lg[lane] = acc[k]; }
        else for (int e = lane; e < a.ne; e += 32) lg[e] = __ldcg(a.logits + (size_t)(t0 + t) * a.ne + e);
        __syncwarp();
        RouterArgs b = a;
        b.top = a.top + (t0 + t) * 8;
        b.wts = a.wts + (t0 + t) * 8;
        warp_topk(b, lg, lane, 0u);
    }
}

template <int TPW>
static cudaError_t router_rows_launch(const RouterArgs &a, int ntok, bool pdl, cudaStream_t st) {
    constexpr int TT = RR_WARPS * TPW;
    constexpr size_t smem = (size_t)RR_STAGES * (RT_TILE_FLOATS + TT * RT_TJ) * 4;
    static unsigned long long configured = 0;      // one bit per device
    cudaError_t e = smem_optin(router_rows_kernel<TPW>, (int)smem, configured);
    if (e != cudaSuccess) return e;
    return launch_k(router_rows_kernel<TPW>, dim3((a.ne + 31) / 32, (ntok + TT - 1) / TT), dim3(RR_WARPS * 32), smem, st, pdl, a, ntok);
}

// (A check and no launch bound: a bound changes the code the compiler makes of the chain, and every router launch runs it.)
bool ffn_in_takes_half_an_sm() {
    cudaFuncAttributes at;
    return cudaFuncGetAttributes(&at, ffn_in_kernel) == cudaSuccess && at.numRegs * RT_THREADS <= 32768;
}
static int ffn_in_epc(int ne) { return ne > 32 ? 16 : 32; }
static int ffn_in_stages(int ne) { return ne > 32 ? 6 : RT_STAGES; }
size_t ffn_in_smem(int ne, int d) { return (size_t)ffn_in_epc(ne) * RT_STRIDE * 4 * ffn_in_stages(ne) + (size_t)d * 8 + (size_t)((ne + 3) & ~3) * 4 + ffn_in_stages(ne) * 16; }

size_t router_packed_floats(int ne, int d) { return (size_t)((ne + 31) / 32) * ((d + RT_TJ - 1) / RT_TJ) * RT_TILE_FLOATS; }

cudaError_t launch_ffn_in(const float *x_in, const float *norm_w, float eps, int d, const float *Wt, const float *b, int ne, int topk,
                          float *logits, int32_t *top, float *wts, unsigned int *counter, DevState *state, bool pdl, cudaStream_t st, int ntok,
                          uint32_t *signal, int qwen_norm, int8_t *q8k_q, float *q8k_s, int32_t *q8k_b16) {
    RouterArgs a{x_in, norm_w, eps, d, Wt, b, ne, topk, logits, top, wts, counter, state, signal, (signal && state) ? state->route_pub : nullptr,
                 qwen_norm, q8k_q, q8k_s, q8k_b16, ffn_in_epc(ne), ffn_in_stages(ne)};
    if (signal && !state) return cudaErrorInvalidValue;
    const size_t smem = ffn_in_smem(ne, d);
    static unsigned long long configured = 0;      // one bit per device
    {
        cudaError_t e = smem_optin(ffn_in_kernel, 200 * 1024, configured);
        if (e != cudaSuccess) return e;
    }
    return launch_k(ffn_in_kernel, dim3((ne + a.epc - 1) / a.epc, ntok), dim3(RT_THREADS), smem, st, pdl, a);
}

cudaError_t launch_router_rows(const float *xn, int d, const float *Wt, const float *b, int ne, int topk, int ntok, float *logits, int32_t *top, float *wts,
                               unsigned int *counter, DevState *state, bool pdl, cudaStream_t st) {
    if (d % 64 || ne > 256 || topk > 8 || ntok < 1) return cudaErrorInvalidValue;
    RouterArgs a{};
    a.x_in = xn; a.d = d; a.Wt = Wt; a.b = b; a.ne = ne; a.topk = topk; a.logits = logits; a.top = top; a.wts = wts; a.counter = counter; a.state = state;
    // a CTA per token (and sixteen experts) while each finds an SM of its own: its chain is alone there (16 against 18.5 us at 9 rows of 2880)
    if (ntok * ((ne + (ne > 32 ? 15 : 31)) / (ne > 32 ? 16 : 32)) <= 148) return launch_ffn_in(xn, nullptr, 0.0f, d, Wt, b, ne, topk, logits, top, wts, counter, state, pdl, st, ntok);
    // few tokens per warp are fast while every CTA finds an SM of its own (a CTA of four warps leaves its SM's schedulers half idle)
    const int groups = (ne + 31) / 32;
    if (groups * ((ntok + 3) / 4) <= 148) return router_rows_launch<1>(a, ntok, pdl, st);
    if (groups * ((ntok + 7) / 8) <= 148) return router_rows_launch<2>(a, ntok, pdl, st);
    return router_rows_launch<4>(a, ntok, pdl, st);
}

// ---------------------------------------------------------------- routing hint (speculation)
// A fast, order-free estimate of the router: one CTA per expert forms its logit with a parallel
// reduction (a few ulps away from the serial chain); consumers pick the k largest themselves
// (spec_pick).  The estimate only decides WHICH experts' gate/up weights start streaming while ffn_in_kernel walks
// the exact serial chains next to it; the exact top-k, its order and its weights still come from
// ffn_in_kernel, and down_combine_kernel refuses (spec_fail_step) any step whose exact expert set
// is not covered by the estimate, so results never depend on this kernel.
struct HintArgs {
    const float *x_in, *norm_w;
    float eps;
    int d;
    const float *Wt, *b;
    int ne, topk;
    float *est;              // [ne] estimated logits
    int8_t *xq_out;          // nullable: Q8 of the normalised vector, each CTA writes a share
    float *xs_out;
    DevState *state;
    uint8_t *dig_out;       // nullable: digits of the same vector (brrr_mxt.cuh)
};

constexpr int HINT_THREADS = 128;
constexpr int HINT_MAXG = 8;         // float4 groups per thread kept in registers (d <= 4096)

__global__ void __launch_bounds__(HINT_THREADS) router_hint_kernel(HintArgs a) {
    extern __shared__ __align__(16) float hsm[];      // d floats of x, then ne floats
    float *xf = hsm, *lg = hsm + a.d;
    __shared__ float inv_sh, red[HINT_THREADS / 32];
    const int tid = threadIdx.x, e = blockIdx.x, d = a.d, groups = d >> 2;
    const int ntiles = (d + RT_TJ - 1) / RT_TJ;
    // static operands first: this expert's row of the tiled matrix and the norm weights
    const float *wrow = a.Wt + ((size_t)(e >> 5) * ntiles * 32 + (e & 31)) * RT_STRIDE;
    float4 w[HINT_MAXG], nw[HINT_MAXG];
#pragma unroll
    for (int p = 0; p < HINT_MAXG; p++) {
        const int g = tid + p * HINT_THREADS;
        if (g < groups) {
            const int j = g * 4, t = j / RT_TJ, jj = j % RT_TJ;
            w[p] = *reinterpret_cast<const float4 *>(wrow + (size_t)t * RT_TILE_FLOATS + jj);
            nw[p] = a.norm_w ? reinterpret_cast<const float4 *>(a.norm_w)[g] : make_float4(1.f, 1.f, 1.f, 1.f);
        } else { w[p] = make_float4(0.f, 0.f, 0.f, 0.f); nw[p] = w[p]; }
    }
    const float bias = a.b ? a.b[e] : 0.0f;
    BRRR_GT_START(a.state, 235);
    pdl_wait_cta();
    BRRR_GT_GO(a.state, 224);
    pdl_trigger();
    stage_vec4(a.x_in, xf, d, tid, HINT_THREADS);
    __syncthreads();
    float inv = 1.0f;
    if (a.norm_w) inv = block_rms_inv(xf, d, a.eps, &inv_sh);
    float part = 0.0f;
#pragma unroll
    for (int p = 0; p < HINT_MAXG; p++) {
        const int g = tid + p * HINT_THREADS;
        if (g < groups) {
            float4 x = reinterpret_cast<const float4 *>(xf)[g];
            part += w[p].x * (x.x * inv * nw[p].x) + w[p].y * (x.y * inv * nw[p].y) + w[p].z * (x.z * inv * nw[p].z) + w[p].w * (x.w * inv * nw[p].w);
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) part += __shfl_xor_sync(0xffffffffu, part, o);
    if ((tid & 31) == 0) red[tid >> 5] = part;
    __syncthreads();
    if (tid == 0) {
        float s = bias;
        for (int i = 0; i < HINT_THREADS / 32; i++) s += red[i];
        a.est[e] = s;
    }
    // This CTA's share of the Q8 quantisation of the normalised vector (exact, block-local):
    // gate/up then stages 3 KB instead of normalising and quantising in every CTA.
    if (a.xq_out) {
        const int nb = d / 32, warp = tid >> 5, lane = tid & 31;
        for (int blk = e * (HINT_THREADS / 32) + warp; blk < nb; blk += gridDim.x * (HINT_THREADS / 32)) {
            float v = xf[blk * 32 + lane];
            if (a.norm_w) v = __fmul_rn(__fmul_rn(v, inv), a.norm_w[blk * 32 + lane]);
            const float amax = fmaxf(warp_max(fabsf(v)), 1e-12f);
            const float sc = __fdiv_rn(amax, 127.0f);
            const int qv = brrr_q8_round_inv(v, sc, brrr_q8_inv(amax));
            if (lane == 0) a.xs_out[blk] = sc;
            a.xq_out[blk * 32 + lane] = (int8_t)qv;
            if (a.dig_out) xt_emit_digits(qv, lane, blk, a.dig_out);
        }
    }
    BRRR_GT_END(a.state, 225);
}

cudaError_t launch_router_hint(const float *x_in, const float *norm_w, float eps, int d, const float *Wt, const float *b, int ne, int topk,
                               float *est, int8_t *xq_out, float *xs_out, DevState *state, bool pdl, cudaStream_t st, uint8_t *dig_out) {
    HintArgs a{x_in, norm_w, eps, d, Wt, b, ne, topk, est, xq_out, xs_out, state, dig_out};
    size_t smem = (size_t)(d + ne + 4) * sizeof(float);
    return launch_k(router_hint_kernel, dim3(ne), dim3(HINT_THREADS), smem, st, pdl, a);
}

}  // namespace brrr
