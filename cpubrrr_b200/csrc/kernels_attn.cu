// Decode attention for one token: RoPE of q and k, KV-cache append, GQA attention with an
// attention sink and an optional sliding window, and the Q8 quantisation of the output.
//
// One CTA per query head (head_dim = 64).  Fixed float order:
//   score(t): 16 chains (chain c covers dims c, c+16, c+32, c+48, fused), combined
//             ((a0+a1)+(a2+a3)) per lane then (l0+l1)+(l2+l3), times 1/sqrt(64)
//   mx = max(sink, scores); den = exp(sink-mx) + sum_t exp(s_t-mx), t ascending, serial
//   out[u] = (sum_t fma(v[t][u], p_t, .), t ascending, serial) * (1/den)
// The serial sums are one thread each (64 output dims + 1 denominator).
//
// The cache is laid out [kv head][position][64] so the window of one head is one contiguous
// range; K, then V run through one ring of tiles of 64 positions (32 for token rows) by bulk asynchronous copies, the first of them
// issued before the kernel waits on its predecessor (the cached positions are older than this
// token).  The current position's k and v never come from the cache: every head recomputes them.
//
// Nobody waits for a whole CTA inside the loops over the tiles: a warp leaves a tile through the tile's barrier and a warp of its own refills the
// ring.  A key's 16 chains belong to four neighbouring threads, four chains each in a 16-byte word.  The serial sums read sixteen keys ahead across
// tile borders.  20b shape, one token, full layer, from the dependency wait to the end: 4.1 us at 130 keys, 8.5 at 600, 20.5 at 1900 (before:
// 4.6, 11.5, 31.0).  Bound by the two serial sums, 8 to 10 cycles a key where the dependent multiply-add alone is 4.7, and by score passes of 8
// cycles a key; the copies come at 25 of the 67 bytes a cycle that one CTA can draw from L2.
#include "brrr_kernels.h"
#include "brrr_block.cuh"
#include "brrr_tma.cuh"
#include "brrr_tile.cuh"

#include <type_traits>

namespace brrr {

constexpr int HD = 64;
constexpr int AT_WORKERS = 256;
constexpr int AT_TILE_ONE = 64;                    // positions per tile: one token per launch (one CTA per SM streams its head's window)
constexpr int AT_TILE_ROWS = 32;                   // token rows: many (head, row) CTAs share an SM, so each holds less
__host__ __device__ constexpr int at_slots(int tile) { return tile == AT_TILE_ONE ? 8 : 4; }      // tiles in flight
__host__ __device__ constexpr int at_issuers(int tile) { return tile == AT_TILE_ONE ? 4 : 1; }    // warps that refill the ring, a tile each in turn (a bulk copy takes its thread 240 cycles)
__host__ __device__ constexpr int at_threads(int tile) { return AT_WORKERS + 32 * at_issuers(tile); }

struct AttnArgs {
    const float *qkv;
    float *kc, *vc;          // [nkv][MAXSEQ][64]
    const float *rope, *sinks;
    int nh, nkv;
    const DevState *state;
    int pos_val, window;
    int pos_off;             // added to the device-side position (token t of a prompt tile: t)
    float *ao;
    int8_t *aq;
    float *as;
    DevState *err_state;
    // token rows (grid.y = rows; nullptr: one token): row t attends at position row_pos[t] of sequence
    // row_seq[t] (caches seq_stride floats apart); its q | k | v are ldq floats after the previous row's,
    // its outputs nh * 64 values after it.  The cached positions may then have been written by the kernel
    // just before this one (earlier rows of the same sequence), so they are fetched after the dependency wait.
    const int *row_pos, *row_seq;
    size_t seq_stride;
    int ldq;
    uint8_t *img;            // token rows, nullable: half images of the outputs (brrr_tile.cuh)
};

// Q8 of 32-block b of a row's attention output, held one value per lane: int8 values, scale, half image
__device__ __forceinline__ void attn_quant(float o, int lane, int b, int8_t *aq, float *as, uint8_t *img) {
    const float amax = fmaxf(warp_max(fabsf(o)), 1e-12f), sc = __fdiv_rn(amax, 127.0f);
    const int qv = brrr_q8_round_inv(o, sc, brrr_q8_inv(amax));
    if (lane == 0) as[b] = sc;
    if (aq) aq[b * 32 + lane] = (int8_t)qv;
    if (img) ti_emit_block<TI_HALF>(qv, lane, b, img);
}


template <int AT_TILE>
__global__ void __launch_bounds__(at_threads(AT_TILE)) attn_decode_kernel(AttnArgs a) {
    constexpr size_t AT_TILE_BYTES = (size_t)AT_TILE * HD * sizeof(float);
    constexpr int SLOTS = at_slots(AT_TILE);
    extern __shared__ __align__(128) unsigned char smraw[];
    float *tiles = reinterpret_cast<float *>(smraw);                                    // [SLOTS][AT_TILE][64]
    float *sc = reinterpret_cast<float *>(smraw + AT_TILE_BYTES * SLOTS);                // [MAXSEQ]
    __shared__ __align__(8) uint64_t full[SLOTS], left_k[SLOTS], left_v[SLOTS];         // a tile has landed; its K, V readers have left it
    __shared__ __align__(16) float q[HD];
    __shared__ float kcur[HD], vcur[HD];
    __shared__ float red[AT_WORKERS / 32];
    __shared__ float den_sh;
    constexpr int PASS = AT_WORKERS / 4 / AT_TILE;      // K tiles that the workers read side by side
    const int h = blockIdx.x, tid = threadIdx.x;
    const int group = a.nh / a.nkv, kvh = h / group;
    uint32_t *err = a.err_state ? &a.err_state->err : nullptr;
    Waiter waiter(err);
    const bool rows = a.row_pos != nullptr;
    if (rows) {
        const int t = blockIdx.y;
        a.qkv += (size_t)t * a.ldq;
        a.kc += (size_t)a.row_seq[t] * a.seq_stride;
        a.vc += (size_t)a.row_seq[t] * a.seq_stride;
        a.ao += (size_t)t * a.nh * HD;
        if (a.aq) a.aq += (size_t)t * a.nh * HD;
        a.as += (size_t)t * a.nh * 2;
        if (a.img) a.img += (size_t)t * a.nh * ti_pair(TI_HALF);
    }

    // The position is an input of this step (written before the graph launch or by the previous
    // step's last kernel), never by the immediate predecessor, so it may be read before the wait.
    const int pos = rows ? a.row_pos[blockIdx.y] : (a.state ? (int)a.state->pos + a.pos_off : a.pos_val);
    const int start = a.window > 0 ? max(pos - (a.window - 1), 0) : 0;
    const int n = pos - start + 1;                  // keys including the current one
    const int ncached = n - 1;                      // keys that come from the cache
    const int ntiles = (ncached + AT_TILE - 1) / AT_TILE;
    const float *kbase = a.kc + ((size_t)kvh * BRRR_MAXSEQ + start) * HD;
    const float *vbase = a.vc + ((size_t)kvh * BRRR_MAXSEQ + start) * HD;

    auto issue = [&](int u) {                       // one thread: tile u of 2 ntiles, K then V
        const int slot = u % SLOTS, t = u < ntiles ? u : u - ntiles, cnt = min(AT_TILE, ncached - t * AT_TILE);
        mbar_expect_tx(&full[slot], (uint32_t)cnt * HD * 4);
        bulk_g2s(tiles + (size_t)slot * AT_TILE * HD, (u < ntiles ? kbase : vbase) + (size_t)t * AT_TILE * HD, (uint32_t)cnt * HD * 4, &full[slot]);
    };
    BRRR_STAMP(a.err_state, 160);
    BRRR_GT_START(a.err_state, 233);
    if (tid == 0) {
        for (int s = 0; s < SLOTS; s++) { mbar_init(&full[s], 1); mbar_init(&left_k[s], AT_WORKERS / 32 / PASS); mbar_init(&left_v[s], 2); }
        mbar_fence_init();
    }
    __syncwarp();
    // one lane per copy: their address translations overlap
    if (!rows && tid < min(SLOTS, 2 * ntiles)) issue(tid);
    // static / step-constant operands: the sink and this position's rotation
    const float sink = a.sinks[h];
    float rc = 0.0f, rs = 0.0f;
    if (tid < 64) { rc = a.rope[((size_t)pos * 32 + (tid & 31)) * 2]; rs = a.rope[((size_t)pos * 32 + (tid & 31)) * 2 + 1]; }
    BRRR_STAMP(a.err_state, 161);
    pdl_wait_cta();      // qkv projection done
    BRRR_STAMP(a.err_state, 162);
    BRRR_GT_GO(a.err_state, 190);
    pdl_trigger();
    waiter.poison_if_failed();
    if (rows && tid < min(SLOTS, 2 * ntiles)) issue(tid);

    // ---- RoPE (NeoX halves, table holds cos*mscale / sin*mscale) on q and k; v passes through
    if (tid < 64) {
        const float *src = tid < 32 ? a.qkv + h * HD : a.qkv + (a.nh + kvh) * HD;
        float *dst = tid < 32 ? q : kcur;
        int i = tid & 31;
        const float c = rc, s = rs;
        float x0 = src[i], x1 = src[32 + i];
        dst[i] = __fsub_rn(__fmul_rn(x0, c), __fmul_rn(x1, s));
        dst[32 + i] = __fadd_rn(__fmul_rn(x1, c), __fmul_rn(x0, s));
    } else if (tid < 128) {
        vcur[tid - 64] = a.qkv[(a.nh + a.nkv + kvh) * HD + (tid - 64)];
    }
    __syncthreads();
    // the first head of each KV group appends this position to the cache
    if (!rows && h % group == 0 && tid < 128) {        // (token rows: kv_append_rows_kernel has done it for every row)
        size_t o = ((size_t)kvh * BRRR_MAXSEQ + pos) * HD + (tid & 63);
        if (tid < 64) a.kc[o] = kcur[tid]; else a.vc[o] = vcur[tid - 64];
    }

    auto bar_workers = [&]() { asm volatile("bar.sync 1, %0;" ::"n"(AT_WORKERS) : "memory"); };
    if (tid >= AT_WORKERS) {
        // ---- ring: tile u + SLOTS takes the slot of tile u once its readers have left it
        if ((tid & 31) == 0) {
            for (int u = (tid - AT_WORKERS) >> 5; u + SLOTS < 2 * ntiles; u += at_issuers(AT_TILE)) {
                const int slot = u % SLOTS;
                // V tiles' uses of a slot are counted from its first one
                if (u < ntiles) waiter.wait(&left_k[slot], (uint32_t)(u / SLOTS) & 1u);
                else waiter.wait(&left_v[slot], (uint32_t)((u - ntiles) / SLOTS) & 1u);
                fence_proxy_async();
                issue(u + SLOTS);
            }
        }
        return;
    }
    const int lane = tid & 31, warp = tid >> 5;
    // ---- scores: four threads per key, thread j of them the chains 4 j .. 4 j + 3
    {
        const int j = tid & 3, key = (tid >> 2) % AT_TILE, odd = key & 1;
        float4 qv[4];
#pragma unroll
        for (int i = 0; i < 4; i++) qv[i] = *reinterpret_cast<const float4 *>(q + 16 * i + 4 * j);
        // U passes side by side, so that their loads and shuffles overlap
        auto pass = [&](auto U_, int t) {
            constexpr int U = decltype(U_)::value;
            float s[U][4];
            float4 f[U][4];
            int slot[U];
#pragma unroll
            for (int u = 0; u < U; u++) {
                slot[u] = (t + u * PASS) % SLOTS;
                waiter.wait(&full[slot[u]], (uint32_t)((t + u * PASS) / SLOTS) & 1u);
            }
#pragma unroll
            for (int u = 0; u < U; u++) {
                const float *kp = tiles + ((size_t)slot[u] * AT_TILE + key) * HD + 4 * j;
                // two neighbouring keys' words share banks: the odd key reads its quarters in the order 1, 0, 3, 2
#pragma unroll
                for (int i = 0; i < 4; i++) f[u][i] = *reinterpret_cast<const float4 *>(kp + 16 * (i ^ odd));
            }
#pragma unroll
            for (int u = 0; u < U; u++) {
#pragma unroll
                for (int e = 0; e < 4; e++) s[u][e] = 0.0f;
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    const float4 k = odd ? f[u][i ^ 1] : f[u][i];
                    s[u][0] = __fmaf_rn(k.x, qv[i].x, s[u][0]); s[u][1] = __fmaf_rn(k.y, qv[i].y, s[u][1]);
                    s[u][2] = __fmaf_rn(k.z, qv[i].z, s[u][2]); s[u][3] = __fmaf_rn(k.w, qv[i].w, s[u][3]);
                }
            }
            __syncwarp();
#pragma unroll
            for (int u = 0; u < U; u++) mbar_arrive_if(lane == 0 ? 1u : 0u, &left_k[slot[u]]);
            // chains c and c ^ 4, then c ^ 8, then c ^ 1, then c ^ 2.  The first two partners sit in other threads: an even thread keeps
            // chains 0 and 1 of its four and gives away 2 and 3, the odd one the other way round, and so on; every sum has two operands
            const bool b0 = j & 1, b1 = j & 2;
            float u0[U], u1[U], w[U];
#pragma unroll
            for (int u = 0; u < U; u++) {
                u0[u] = __fadd_rn(b0 ? s[u][2] : s[u][0], __shfl_xor_sync(0xffffffffu, b0 ? s[u][0] : s[u][2], 1));
                u1[u] = __fadd_rn(b0 ? s[u][3] : s[u][1], __shfl_xor_sync(0xffffffffu, b0 ? s[u][1] : s[u][3], 1));
            }
#pragma unroll
            for (int u = 0; u < U; u++) w[u] = __fadd_rn(b1 ? u1[u] : u0[u], __shfl_xor_sync(0xffffffffu, b1 ? u0[u] : u1[u], 2));      // chains of residue 2 b0 + b1
#pragma unroll
            for (int u = 0; u < U; u++) w[u] = __fadd_rn(w[u], __shfl_xor_sync(0xffffffffu, w[u], 2));
#pragma unroll
            for (int u = 0; u < U; u++) {
                w[u] = __fadd_rn(w[u], __shfl_xor_sync(0xffffffffu, w[u], 1));
                const int at = (t + u * PASS) * AT_TILE + key;
                if (j == 0 && at < ncached) sc[at] = __fmul_rn(w[u], 0.125f);
            }
        };
        int t = tid / (4 * AT_TILE);
#pragma unroll 1
        for (; t + PASS < ntiles; t += 2 * PASS) pass(std::integral_constant<int, 2>{}, t);
        if (t < ntiles) pass(std::integral_constant<int, 1>{}, t);
        // the current position, from this CTA's own rotated k
        if (tid < 16) {
            const int c = tid;
            float s = 0.0f;
            s = __fmaf_rn(kcur[c], q[c], s);
            s = __fmaf_rn(kcur[16 + c], q[16 + c], s);
            s = __fmaf_rn(kcur[32 + c], q[32 + c], s);
            s = __fmaf_rn(kcur[48 + c], q[48 + c], s);
            s = __fadd_rn(s, __shfl_xor_sync(0xffffu, s, 4));
            s = __fadd_rn(s, __shfl_xor_sync(0xffffu, s, 8));
            s = __fadd_rn(s, __shfl_xor_sync(0xffffu, s, 1));
            s = __fadd_rn(s, __shfl_xor_sync(0xffffu, s, 2));
            if (c == 0) sc[ncached] = __fmul_rn(s, 0.125f);
        }
    }
    bar_workers();

    BRRR_STAMP(a.err_state, 163);
    // ---- max (order-free), then exponentials in place
    float mx = sink;
    for (int t = tid; t < n; t += AT_WORKERS) mx = fmaxf(mx, sc[t]);
    mx = warp_max(mx);
    if (lane == 0) red[warp] = mx;
    bar_workers();
    mx = red[0];
#pragma unroll
    for (int w = 1; w < AT_WORKERS / 32; w++) mx = fmaxf(mx, red[w]);
    for (int t = tid; t < ((n + 3) & ~3); t += AT_WORKERS) sc[t] = t < n ? brrr_expf_dev(__fsub_rn(sc[t], mx)) : 0.0f;      // +0 past the end changes no sum
    bar_workers();

    BRRR_STAMP(a.err_state, 164);
    // ---- serial sums: thread u < 64 owns output dim u, thread 64 the denominator
    float acc = 0.0f;
    if (warp < 2) {
        // sixteen keys at a time, the next sixteen's values on the way, across tile borders (two sets of registers: reloading one set in place
        // exposed every load's latency; so did branches between a load and its use)
        constexpr int BLOCKS = AT_TILE / 16;
        const int nfull = ncached / AT_TILE;
        float v0[16], v1[16];
        float4 p0[4], p1[4];
        // (statements of their own, in program order: the compiler moves plain loads down to their uses)
        auto load = [&](float (&v)[16], float4 (&p)[4], const float *w, const float *o) {
            const uint32_t wa = smem_u32(w), oa = smem_u32(o);
#pragma unroll
            for (int i = 0; i < 4; i++) asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(p[i].x), "=f"(p[i].y), "=f"(p[i].z), "=f"(p[i].w) : "r"(oa + 16 * i));
#pragma unroll
            for (int i = 0; i < 16; i++) asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v[i]) : "r"(wa + i * HD * 4));
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
        int slot = ntiles % SLOTS;
        uint32_t par = (uint32_t)(ntiles / SLOTS) & 1u;
        const float *vt = tiles + (size_t)slot * AT_TILE * HD + tid, *pt = sc;
        if (ntiles) { waiter.wait(&full[slot], par); load(v0, p0, vt, pt); }
#pragma unroll 1
        for (int t = 0; t < nfull; t++) {
            const int here = slot;
            const float *vn = vt, *pn = pt;                    // the next tile; behind the last one: read again, not used
            if (t + 1 < ntiles) {
                if (++slot == SLOTS) { slot = 0; par ^= 1u; }
                waiter.wait(&full[slot], par);
                vn = tiles + (size_t)slot * AT_TILE * HD + tid; pn = pt + AT_TILE;
            }
#pragma unroll
            for (int b = 0; b < BLOCKS; b += 2) {
                load(v1, p1, vt + (b + 1) * 16 * HD, pt + (b + 1) * 16);
                add(v0, p0, 16);
                if (b + 2 < BLOCKS) load(v0, p0, vt + (b + 2) * 16 * HD, pt + (b + 2) * 16);
                else load(v0, p0, vn, pn);
                add(v1, p1, 16);
            }
            __syncwarp();
            mbar_arrive_if(lane == 0 ? 1u : 0u, &left_v[here]);      // the tile's values are used: its slot may take another
            vt = vn; pt = pn;
        }
        for (int k = nfull * AT_TILE; k < ncached; k += 32) {        // the last tile's keys
            load(v1, p1, vt + 16 * HD, pt + 16);
            add(v0, p0, ncached - k);
            add(v1, p1, ncached - k - 16);
            if (k + 32 < ncached) { vt += 32 * HD; pt += 32; load(v0, p0, vt, pt); }
        }
        acc = __fmaf_rn(vcur[tid], sc[ncached], acc);          // t = pos: this token's own v
    } else if (tid == 64) {
        float den = brrr_expf_dev(__fsub_rn(sink, mx));
        // sixteen probabilities at a time, the next sixteen on the way; the last four padded with +0
        const int quads = (n + 3) >> 2;
        const uint32_t pa = smem_u32(sc);
        float4 p0[4], p1[4];
        auto load = [&](float4 (&p)[4], int k) {              // (past the end: the first quad again, not used)
#pragma unroll
            for (int i = 0; i < 4; i++) asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(p[i].x), "=f"(p[i].y), "=f"(p[i].z), "=f"(p[i].w) : "r"(pa + (k + i < quads ? k + i : 0) * 16));
        };
        auto add = [&](const float4 (&p)[4], int left) {
#pragma unroll
            for (int i = 0; i < 4; i++)
                if (i < left) { den = __fadd_rn(den, p[i].x); den = __fadd_rn(den, p[i].y); den = __fadd_rn(den, p[i].z); den = __fadd_rn(den, p[i].w); }
        };
        load(p0, 0);
        int k = 0;
#pragma unroll 1
        for (; k + 8 <= quads; k += 8) {
            load(p1, k + 4);
            add(p0, 4);
            load(p0, k + 8);
            add(p1, 4);
        }
        load(p1, k + 4);
        add(p0, quads - k);
        add(p1, quads - k - 4);
        den_sh = den;
    }
    bar_workers();
    if (tid < 64) {
        float inv = __fdiv_rn(1.0f, den_sh);
        float o = __fmul_rn(acc, inv);
        a.ao[h * HD + tid] = o;
        // this head owns Q8 blocks 2h and 2h+1 of the attention output
        attn_quant(o, tid & 31, h * 2 + (tid >> 5), a.aq, a.as, a.img);
    }
    BRRR_STAMP(a.err_state, 165);
    BRRR_GT_END(a.err_state, 191);
}

// ---------------------------------------------------------------- prompt tiles: rows of one sequence share their keys
// attn_decode_kernel per (head, row) streams the row's whole window from L2 for every one of the 64 heads: a tile of
// R rows at position p costs 64 R p key reads.  Here one CTA serves one KV head and a block of consecutive rows of one
// sequence: 32 (query head, row) pairs = group x (32 / group) rows share every K and V tile it brings into shared
// memory.  Same operations in the same order per pair as attn_decode_kernel (the row's own key comes from the cache,
// where kv_append_rows_kernel wrote the same bits):
//   score(t)  one thread: the 16 four-term chains, then the pairwise combine of the shuffle butterfly (xor 4, 8, 1, 2)
//   pass 1    scores of every key -> workspace, the pair's maximum;  pass 2  p = exp(s - mx) into shared memory,
//             then, tile by tile in ascending key order, the serial denominator (one thread per pair) and the serial
//             p.V sums (one thread per (dim, 8 pairs)).  Keys outside a pair's range carry p = +0: x + 0 = x exactly
//             (no accumulator is ever -0: the sums start at +0 and round to nearest), so they need no branch.
// 32 pairs x 4096 keys of scores do not fit shared memory: they wait in a workspace (written and read by the same thread, 128 bytes per key and
// warp; mostly L2).  Formed twice instead, a 512-row tile at positions 1024 .. 1535 took 895 us, now 742.
constexpr int AR_THREADS = 256;
constexpr int AR_TILE = 128;
constexpr int AR_PAIRS = 32;
constexpr size_t AR_TILE_BYTES = (size_t)AR_TILE * HD * sizeof(float);
constexpr size_t AR_SMEM = 4 * AR_TILE_BYTES + (size_t)AR_TILE * AR_PAIRS * 4 + (size_t)AR_PAIRS * HD * 4;

struct AttnRowsArgs {
    const float *qkv;        // [rows][ldq]: q | k | v of every row, bias added, not rotated
    const float *kc, *vc;    // [sequence][nkv][MAXSEQ][64]
    const float *rope, *sinks;
    int nh, nkv, window, rows, ldq;
    const int *row_pos, *row_seq;
    size_t seq_stride;
    float *ao;
    int8_t *aq;
    float *as;
    uint8_t *img;            // nullable: half images of the outputs
    float *scores;           // workspace: [row block][kv head][MAXSEQ][32]
    DevState *err_state;
};

// one score: q in registers, the key's 64 floats at kp (shared memory, the same address in every lane)
__device__ __forceinline__ float ar_score(const float (&q)[HD], const float *kp) {
    float a[16];
#pragma unroll
    for (int c4 = 0; c4 < 4; c4++) {
        const float4 k0 = *reinterpret_cast<const float4 *>(kp + 4 * c4), k1 = *reinterpret_cast<const float4 *>(kp + 16 + 4 * c4);
        const float4 k2 = *reinterpret_cast<const float4 *>(kp + 32 + 4 * c4), k3 = *reinterpret_cast<const float4 *>(kp + 48 + 4 * c4);
        const float kk0[4] = {k0.x, k0.y, k0.z, k0.w}, kk1[4] = {k1.x, k1.y, k1.z, k1.w}, kk2[4] = {k2.x, k2.y, k2.z, k2.w}, kk3[4] = {k3.x, k3.y, k3.z, k3.w};
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const int c = 4 * c4 + i;
            float v = __fmaf_rn(kk0[i], q[c], 0.0f);
            v = __fmaf_rn(kk1[i], q[16 + c], v);
            v = __fmaf_rn(kk2[i], q[32 + c], v);
            a[c] = __fmaf_rn(kk3[i], q[48 + c], v);
        }
    }
    // butterfly xor 4, 8, 1, 2 of the 16-thread group, as one thread
    const float b0 = __fadd_rn(a[0], a[4]), b1 = __fadd_rn(a[1], a[5]), b2 = __fadd_rn(a[2], a[6]), b3 = __fadd_rn(a[3], a[7]);
    const float b8 = __fadd_rn(a[8], a[12]), b9 = __fadd_rn(a[9], a[13]), b10 = __fadd_rn(a[10], a[14]), b11 = __fadd_rn(a[11], a[15]);
    const float c0 = __fadd_rn(b0, b8), c1 = __fadd_rn(b1, b9), c2 = __fadd_rn(b2, b10), c3 = __fadd_rn(b3, b11);
    return __fmul_rn(__fadd_rn(__fadd_rn(c0, c1), __fadd_rn(c2, c3)), 0.125f);
}

__global__ void __launch_bounds__(AR_THREADS) attn_rows_kernel(AttnRowsArgs a) {
    extern __shared__ __align__(128) unsigned char smraw[];
    float *ktile = reinterpret_cast<float *>(smraw);                                    // [2][128][64]
    float *vtile = reinterpret_cast<float *>(smraw + 2 * AR_TILE_BYTES);                // [2][128][64]
    float *psm = reinterpret_cast<float *>(smraw + 4 * AR_TILE_BYTES);                  // [128 keys][32 pairs]
    float *qsm = psm + AR_TILE * AR_PAIRS;                                              // [32 pairs][64]
    __shared__ __align__(8) uint64_t kbar[2], vbar[2];
    __shared__ float red[AR_THREADS / 32][AR_PAIRS];
    __shared__ float mx_sm[AR_PAIRS], den_sm[AR_PAIRS];
    __shared__ int pos_sm[AR_PAIRS];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int group = a.nh / a.nkv, rb = AR_PAIRS / group;        // rows per CTA
    const int kvh = blockIdx.x, r0 = blockIdx.y * rb;
    const int nrows = min(rb, a.rows - r0);
    uint32_t *err = a.err_state ? &a.err_state->err : nullptr;
    Waiter waiter(err);
    if (tid == 0) {
        mbar_init(&kbar[0], 1); mbar_init(&kbar[1], 1); mbar_init(&vbar[0], 1); mbar_init(&vbar[1], 1);
        mbar_fence_init();
    }
    pdl_wait();          // q/k/v projection and the cache append of every row are done
    pdl_trigger();
    waiter.poison_if_failed();
    // ---- the pairs: pair = row-in-block * group + head-in-group
    const int pr = lane;                                           // this thread's pair in the score phases
    const int pr_row = pr / group, pr_h = kvh * group + pr % group;
    const bool pr_live = pr_row < nrows;
    if (tid < AR_PAIRS) pos_sm[tid] = (tid / group) < nrows ? a.row_pos[r0 + tid / group] : -1;
    // RoPE of q (NeoX halves), 1024 rotations over 256 threads
    for (int idx = tid; idx < AR_PAIRS * 32; idx += AR_THREADS) {
        const int p2 = idx >> 5, i = idx & 31, rr = p2 / group;
        if (rr < nrows) {
            const int pos = a.row_pos[r0 + rr];
            const float *src = a.qkv + (size_t)(r0 + rr) * a.ldq + (size_t)(kvh * group + p2 % group) * HD;
            const float c = a.rope[((size_t)pos * 32 + i) * 2], sn = a.rope[((size_t)pos * 32 + i) * 2 + 1];
            const float x0 = src[i], x1 = src[32 + i];
            qsm[p2 * HD + i] = __fsub_rn(__fmul_rn(x0, c), __fmul_rn(x1, sn));
            qsm[p2 * HD + 32 + i] = __fadd_rn(__fmul_rn(x1, c), __fmul_rn(x0, sn));
        } else { qsm[p2 * HD + i] = 0.0f; qsm[p2 * HD + 32 + i] = 0.0f; }
    }
    __syncthreads();
    float q[HD];
#pragma unroll
    for (int i = 0; i < HD; i++) q[i] = qsm[pr * HD + i];
    const int my_pos = pos_sm[pr];
    const int my_start = a.window > 0 ? max(my_pos - (a.window - 1), 0) : 0;
    // key range of the block: from the first row's window start to the last row's position
    const int pos_first = pos_sm[0], pos_last = pos_sm[(nrows - 1) * group];
    const int t_lo = a.window > 0 ? max(pos_first - (a.window - 1), 0) : 0;
    const int nkeys = pos_last - t_lo + 1, ntiles = (nkeys + AR_TILE - 1) / AR_TILE;
    const size_t seq_off = (size_t)a.row_seq[r0] * a.seq_stride;
    const float *kbase = a.kc + seq_off + ((size_t)kvh * BRRR_MAXSEQ + t_lo) * HD;
    const float *vbase = a.vc + seq_off + ((size_t)kvh * BRRR_MAXSEQ + t_lo) * HD;
    int k_issued = 0, v_issued = 0, k_used = 0, v_used = 0;       // tiles issued / consumed so far (buffer = count & 1, parity = count >> 1 & 1)
    auto issue_k = [&](int t) {       // thread 0
        const int buf = k_issued & 1, cnt = min(AR_TILE, nkeys - t * AR_TILE);
        mbar_expect_tx(&kbar[buf], (uint32_t)cnt * HD * 4);
        bulk_g2s(ktile + (size_t)buf * AR_TILE * HD, kbase + (size_t)t * AR_TILE * HD, (uint32_t)cnt * HD * 4, &kbar[buf]);
    };
    auto issue_v = [&](int t) {
        const int buf = v_issued & 1, cnt = min(AR_TILE, nkeys - t * AR_TILE);
        mbar_expect_tx(&vbar[buf], (uint32_t)cnt * HD * 4);
        bulk_g2s(vtile + (size_t)buf * AR_TILE * HD, vbase + (size_t)t * AR_TILE * HD, (uint32_t)cnt * HD * 4, &vbar[buf]);
    };

    float *my_scores = a.scores + ((size_t)blockIdx.y * a.nkv + kvh) * BRRR_MAXSEQ * AR_PAIRS + lane;
    // ---- pass 1: the maximum of every pair's scores
    float mx = -3.4028234663852886e38f;
    if (tid == 0) issue_k(0);
    k_issued++;
    for (int t = 0; t < ntiles; t++) {
        if (t + 1 < ntiles) { if (tid == 0) issue_k(t + 1); k_issued++; }        // the other buffer: free since the barrier that ended tile t - 1
        const int buf = k_used & 1;
        waiter.wait(&kbar[buf], (uint32_t)(k_used >> 1) & 1u);
        k_used++;
        const float *kt = ktile + (size_t)buf * AR_TILE * HD;
        const int cnt = min(AR_TILE, nkeys - t * AR_TILE), tb = t_lo + t * AR_TILE;
        for (int kk = warp; kk < cnt; kk += AR_THREADS / 32) {
            const float sc = ar_score(q, kt + kk * HD);
            const int key = tb + kk;
            my_scores[(size_t)(t * AR_TILE + kk) * AR_PAIRS] = sc;
            if (pr_live && key >= my_start && key <= my_pos) mx = fmaxf(mx, sc);
        }
        __syncthreads();              // everyone is done with this buffer
        if (tid == 0) fence_proxy_async();
    }
    red[warp][lane] = mx;
    __syncthreads();
    if (tid < AR_PAIRS) {
        float m = a.sinks[kvh * group + tid % group];
#pragma unroll
        for (int w = 0; w < AR_THREADS / 32; w++) m = fmaxf(m, red[w][tid]);
        mx_sm[tid] = m;
        den_sm[tid] = brrr_expf_dev(__fsub_rn(a.sinks[kvh * group + tid % group], m));      // the sink's term opens the denominator
    }
    __syncthreads();
    mx = mx_sm[pr];

    // ---- pass 2: probabilities tile by tile; denominator and p.V sums in ascending key order
    const int u = tid & 63, grp = tid >> 6;                        // this thread in the p.V phase: dim u of pairs grp * 8 .. + 7
    float acc[8];
#pragma unroll
    for (int j = 0; j < 8; j++) acc[j] = 0.0f;
    float den = tid < AR_PAIRS ? den_sm[tid] : 0.0f;
    if (tid == 0) issue_v(0);
    v_issued++;
    for (int t = 0; t < ntiles; t++) {
        if (t + 1 < ntiles) { if (tid == 0) issue_v(t + 1); v_issued++; }
        const int vb = v_used & 1;
        const int cnt = min(AR_TILE, nkeys - t * AR_TILE), tb = t_lo + t * AR_TILE;
        float sv[AR_TILE / 8];                // this thread's keys warp, warp + 8, ... of the tile
#pragma unroll
        for (int i = 0; i < AR_TILE / 8; i++) sv[i] = warp + 8 * i < cnt ? my_scores[(size_t)(t * AR_TILE + warp + 8 * i) * AR_PAIRS] : 0.0f;
#pragma unroll
        for (int i = 0; i < AR_TILE / 8; i++) {
            const int kk = warp + 8 * i, key = tb + kk;
            const bool valid = kk < cnt && pr_live && key >= my_start && key <= my_pos;
            if (kk < cnt) psm[kk * AR_PAIRS + pr] = valid ? brrr_expf_dev(__fsub_rn(sv[i], mx)) : 0.0f;
        }
        __syncthreads();
        if (tid < AR_PAIRS) {
#pragma unroll 8
            for (int kk = 0; kk < cnt; kk++) den = __fadd_rn(den, psm[kk * AR_PAIRS + tid]);
        }
        waiter.wait(&vbar[vb], (uint32_t)(v_used >> 1) & 1u);
        v_used++;
        const float *vt = vtile + (size_t)vb * AR_TILE * HD + u;
        const float *pt = psm + grp * 8;
#pragma unroll 4
        for (int kk = 0; kk < cnt; kk++) {
            const float v = vt[kk * HD];
            const float4 p0 = *reinterpret_cast<const float4 *>(pt + kk * AR_PAIRS), p1 = *reinterpret_cast<const float4 *>(pt + kk * AR_PAIRS + 4);
            acc[0] = __fmaf_rn(v, p0.x, acc[0]); acc[1] = __fmaf_rn(v, p0.y, acc[1]); acc[2] = __fmaf_rn(v, p0.z, acc[2]); acc[3] = __fmaf_rn(v, p0.w, acc[3]);
            acc[4] = __fmaf_rn(v, p1.x, acc[4]); acc[5] = __fmaf_rn(v, p1.y, acc[5]); acc[6] = __fmaf_rn(v, p1.z, acc[6]); acc[7] = __fmaf_rn(v, p1.w, acc[7]);
        }
        __syncthreads();              // the tile's buffers and the probabilities are free
        if (tid == 0) fence_proxy_async();
    }
    if (tid < AR_PAIRS) den_sm[tid] = den;
    __syncthreads();
    // ---- outputs: o = acc / den, and the Q8 image of every pair's two 32-blocks (a warp = one 32-block of a pair)
#pragma unroll
    for (int j = 0; j < 8; j++) {
        const int p2 = grp * 8 + j, rr = p2 / group, h = kvh * group + p2 % group;
        if (rr < nrows) {             // uniform over the warp
            const float inv = __fdiv_rn(1.0f, den_sm[p2]);
            const float o = __fmul_rn(acc[j], inv);
            const size_t row = (size_t)(r0 + rr);
            a.ao[row * a.nh * HD + h * HD + u] = o;
            attn_quant(o, lane, h * 2 + (u >> 5), a.aq ? a.aq + row * a.nh * HD : nullptr, a.as + row * a.nh * 2, a.img ? a.img + row * a.nh * ti_pair(TI_HALF) : nullptr);
        }
    }
}

static size_t attn_smem(int tile) { return (size_t)tile * HD * sizeof(float) * at_slots(tile) + (size_t)BRRR_MAXSEQ * 4; }

cudaError_t launch_attn_decode(const float *qkv, float *kc, float *vc, const float *rope, const float *sinks, int nh, int nkv,
                               const DevState *state, int pos_val, int window, float *ao, int8_t *aq, float *as,
                               DevState *err_state, bool pdl, cudaStream_t st, int pos_off, const int *row_pos, const int *row_seq, size_t seq_stride,
                               int ldq, int rows, uint8_t *aimg) {
    AttnArgs a{qkv, kc, vc, rope, sinks, nh, nkv, state, pos_val, window, pos_off, ao, aq, as, err_state, row_pos, row_seq, seq_stride, ldq, aimg};
    static unsigned long long configured = 0, configured_rows = 0;      // one bit per device
    if (row_pos) {
        cudaError_t e = smem_optin(attn_decode_kernel<AT_TILE_ROWS>, (int)attn_smem(AT_TILE_ROWS), configured_rows);
        if (e != cudaSuccess) return e;
        return launch_k(attn_decode_kernel<AT_TILE_ROWS>, dim3(nh, rows), dim3(at_threads(AT_TILE_ROWS)), attn_smem(AT_TILE_ROWS), st, pdl, a);
    }
    cudaError_t e = smem_optin(attn_decode_kernel<AT_TILE_ONE>, (int)attn_smem(AT_TILE_ONE), configured);
    if (e != cudaSuccess) return e;
    return launch_k(attn_decode_kernel<AT_TILE_ONE>, dim3(nh, 1), dim3(at_threads(AT_TILE_ONE)), attn_smem(AT_TILE_ONE), st, pdl, a);
}

// Attention for token rows of ONE sequence with ascending positions (a prompt tile): rows share the K / V tiles.
// Needs the rows' keys in the cache already (launch_kv_append_rows) and nh / nkv a power of two <= 32.
cudaError_t launch_attn_rows(const float *qkv, int ldq, const float *kc, const float *vc, size_t seq_stride, const float *rope, const float *sinks,
                             int nh, int nkv, int window, const int *row_pos, const int *row_seq, int rows, float *ao, int8_t *aq, float *as, uint8_t *aimg,
                             float *scores, DevState *err_state, bool pdl, cudaStream_t st) {
    const int group = nkv > 0 ? nh / nkv : 0;
    if (group < 1 || group > 32 || (group & (group - 1)) || nh % nkv || rows < 1) return cudaErrorInvalidValue;
    AttnRowsArgs a{qkv, kc, vc, rope, sinks, nh, nkv, window, rows, ldq, row_pos, row_seq, seq_stride, ao, aq, as, aimg, scores, err_state};
    static unsigned long long configured = 0;      // one bit per device
    cudaError_t e = smem_optin(attn_rows_kernel, (int)AR_SMEM, configured);
    if (e != cudaSuccess) return e;
    const int rb = AR_PAIRS / group;
    return launch_k(attn_rows_kernel, dim3(nkv, (rows + rb - 1) / rb), dim3(AR_THREADS), AR_SMEM, st, pdl, a);
}

}  // namespace brrr
