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
#include "brrr_tc.cuh"
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
//             (half of the warps) and, a tile behind and in ascending key order, the serial p.V sums (the other half: a thread for 8 dims of 2
//             pairs) and by the threads of the first dims the serial denominators.  Keys outside a pair's range carry p = +0: x + 0 = x exactly
//             (no accumulator is ever -0: the sums start at +0 and round to nearest), so they need no branch.
// 32 pairs x 4096 keys of scores do not fit shared memory: they wait in a workspace (128 bytes per key; mostly L2).
// What bounds it is shared memory: a key's row reaches a warp as 16 broadcast words of 16 bytes, 3 to 4 cycles each, for 80 arithmetic instructions
// (40 packed ones), and a key of the p.V sums costs every thread 40 bytes for 16 multiply-adds.  Two CTAs per SM fill each other's barriers.  512 rows of
// the 20b shape: window layer 78 to 87 us, full layer 122 / 280 / 442 us at positions 0 / 512 / 1024 (before, with tiles of 128 keys, one CTA per SM,
// scalar scores and every warp in the same phase: 140 to 146, 221 / 483 / 742).  Two pairs per thread and one CTA per SM took 85 to 95, 124 / 298 / 471.
constexpr int AR_THREADS = 256;
constexpr int AR_PAIRS = 32;
constexpr int AR_TILE = 64;
constexpr size_t AR_TILE_BYTES = (size_t)AR_TILE * HD * sizeof(float);
constexpr size_t AR_SMEM = 4 * AR_TILE_BYTES + 2 * (size_t)AR_TILE * AR_PAIRS * 4 + (size_t)AR_PAIRS * HD * 4;

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

// one score: q in registers, the key's 64 floats at kp (shared memory, the same address in every lane); two chains per instruction
__device__ __forceinline__ float ar_score(const f32x2 (&q)[HD / 2], const float *kp) {
    // butterfly xor 4, 8, 1, 2 of the 16-thread group, as one thread: chains i and 4 + i, 8 + i and 12 + i, then both, then across i
    f32x2 a[2], lo[2];
    const uint32_t ka = smem_u32(kp);
#pragma unroll
    for (int c4 = 0; c4 < 4; c4++) {
        f32x2 k[4][2];
#pragma unroll
        for (int m = 0; m < 4; m++) lds_pairs(ka + (16 * m + 4 * c4) * 4, k[m][0], k[m][1]);
#pragma unroll
        for (int i = 0; i < 2; i++) {
            f32x2 v = tl_fma2(k[0][i], q[2 * c4 + i], 0ull);
#pragma unroll
            for (int m = 1; m < 4; m++) v = tl_fma2(k[m][i], q[8 * m + 2 * c4 + i], v);
            if (c4 & 1) v = tl_add2(a[i], v);
            if (c4 == 1) lo[i] = v;
            else if (c4 == 3) lo[i] = tl_add2(lo[i], v);
            else a[i] = v;
        }
    }
    float c[4];
    tl_unpack2(lo[0], c[0], c[1]);
    tl_unpack2(lo[1], c[2], c[3]);
    return __fmul_rn(__fadd_rn(__fadd_rn(c[0], c[1]), __fadd_rn(c[2], c[3])), 0.125f);
}

__global__ void __launch_bounds__(AR_THREADS, 2) attn_rows_kernel(AttnRowsArgs a) {
    constexpr int HALF = AR_THREADS / 2;                           // pass 2: threads of the sums, and of the probabilities
    extern __shared__ __align__(128) unsigned char smraw[];
    float *ktile = reinterpret_cast<float *>(smraw);                                    // [2][AR_TILE][64]
    float *vtile = reinterpret_cast<float *>(smraw + 2 * AR_TILE_BYTES);                // [2][AR_TILE][64]
    float *psm = reinterpret_cast<float *>(smraw + 4 * AR_TILE_BYTES);                  // [2][AR_TILE keys][pairs]
    float *qsm = psm + 2 * AR_TILE * AR_PAIRS;                                             // [pairs][64]: q, then the outputs
    __shared__ __align__(8) uint64_t kbar[2], vbar[2];
    __shared__ float red[AR_THREADS / 32][AR_PAIRS];
    __shared__ float mx_sm[AR_PAIRS], den_sm[AR_PAIRS];
    __shared__ int pos_sm[AR_PAIRS];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int group = a.nh / a.nkv, lg = 31 - __clz(group), rb = AR_PAIRS >> lg;      // heads per KV head: a power of two; rows per CTA
    const int kvh = blockIdx.x, r0 = (gridDim.y - 1 - blockIdx.y) * rb;      // the last rows, whose ranges are the longest, first
    const int nrows = min(rb, a.rows - r0);
    uint32_t *err = a.err_state ? &a.err_state->err : nullptr;
    Waiter waiter(err);
    if (tid == 0) {
        for (int i = 0; i < 2; i++) { mbar_init(&kbar[i], 1); mbar_init(&vbar[i], 1); }
        mbar_fence_init();
    }
    pdl_wait();          // q/k/v projection and the cache append of every row are done
    pdl_trigger();
    waiter.poison_if_failed();
    // ---- the pairs: pair = row-in-block * group + head-in-group
    if (tid < AR_PAIRS) pos_sm[tid] = (tid >> lg) < nrows ? a.row_pos[r0 + (tid >> lg)] : -1;
    // RoPE of q (NeoX halves): a warp = a pair; every load before the first store (a store in between would order the loads behind it)
    {
        constexpr int N = AR_PAIRS / (AR_THREADS / 32);
        float x0[N], x1[N], rc[N], rs[N];
#pragma unroll
        for (int k = 0; k < N; k++) {
            const int p2 = warp + k * (AR_THREADS / 32), rr = p2 >> lg;
            x0[k] = x1[k] = rc[k] = rs[k] = 0.0f;
            if (rr < nrows) {
                const float *src = a.qkv + (size_t)(r0 + rr) * a.ldq + (size_t)(kvh * group + (p2 & (group - 1))) * HD, *rot = a.rope + ((size_t)a.row_pos[r0 + rr] * 32 + lane) * 2;
                x0[k] = src[lane]; x1[k] = src[32 + lane]; rc[k] = rot[0]; rs[k] = rot[1];
            }
        }
#pragma unroll
        for (int k = 0; k < N; k++) {
            float *o = qsm + (warp + k * (AR_THREADS / 32)) * HD + lane;
            o[0] = __fsub_rn(__fmul_rn(x0[k], rc[k]), __fmul_rn(x1[k], rs[k]));
            o[32] = __fadd_rn(__fmul_rn(x1[k], rc[k]), __fmul_rn(x0[k], rs[k]));
        }
    }
    __syncthreads();
    // key range of the block: from the first row's window start to the last row's position
    const int pos_first = pos_sm[0], pos_last = pos_sm[(nrows - 1) * group];
    const int t_lo = a.window > 0 ? max(pos_first - (a.window - 1), 0) : 0;
    const int nkeys = pos_last - t_lo + 1, ntiles = (nkeys + AR_TILE - 1) / AR_TILE;
    const size_t seq_off = (size_t)a.row_seq[r0] * a.seq_stride;
    // one thread: tile t of K or V into its buffer (t & 1)
    auto issue = [&](const float *cache, float *buf, uint64_t *bar, int t) {
        const uint32_t bytes = (uint32_t)min(AR_TILE, nkeys - t * AR_TILE) * HD * 4;
        mbar_expect_tx(&bar[t & 1], bytes);
        bulk_g2s(buf + (size_t)(t & 1) * AR_TILE * HD, cache + seq_off + ((size_t)kvh * BRRR_MAXSEQ + t_lo + (size_t)t * AR_TILE) * HD, bytes, &bar[t & 1]);
    };

    const int my_pos = pos_sm[lane];                               // this thread's pair in the score phases; -1: no such row, and no key
    const int my_start = a.window > 0 ? max(my_pos - (a.window - 1), 0) : 0;
    float mx = -3.4028234663852886e38f;
    float *my_scores = a.scores + ((size_t)blockIdx.y * a.nkv + kvh) * BRRR_MAXSEQ * AR_PAIRS + lane;
    {
        // ---- pass 1: the maximum of every pair's scores
        f32x2 q[HD / 2];
#pragma unroll
        for (int i = 0; i < HD / 2; i += 2) lds_pairs(smem_u32(qsm + lane * HD + 2 * i), q[i], q[i + 1]);
        if (tid == 0) { issue(a.kc, ktile, kbar, 0); issue(a.vc, vtile, vbar, 0); }
        for (int t = 0; t < ntiles; t++) {
            if (tid == 0 && t + 1 < ntiles) issue(a.kc, ktile, kbar, t + 1);      // the other buffer: free since the barrier that ended tile t - 1
            waiter.wait(&kbar[t & 1], (uint32_t)(t >> 1) & 1u);
            const float *kt = ktile + (size_t)(t & 1) * AR_TILE * HD;
            const int cnt = min(AR_TILE, nkeys - t * AR_TILE), tb = t_lo + t * AR_TILE;
            for (int kk = warp; kk < cnt; kk += AR_THREADS / 32) {
                const float sc = ar_score(q, kt + kk * HD);
                const int key = tb + kk;
                my_scores[(size_t)(t * AR_TILE + kk) * AR_PAIRS] = sc;
                if (key >= my_start && key <= my_pos) mx = fmaxf(mx, sc);
            }
            __syncthreads();              // everyone is done with this buffer
            if (tid == 0) fence_proxy_async();
        }
    }
    red[warp][lane] = mx;
    __syncthreads();
    if (tid < AR_PAIRS) {
        const float sink = a.sinks[kvh * group + (tid & (group - 1))];
        float m = sink;
#pragma unroll
        for (int w = 0; w < AR_THREADS / 32; w++) m = fmaxf(m, red[w][tid]);
        mx_sm[tid] = m;
        den_sm[tid] = brrr_expf_dev(__fsub_rn(sink, m));           // the sink's term opens the denominator
    }
    __syncthreads();
    mx = mx_sm[lane];

    // ---- pass 2: half of the warps make the probabilities of a tile while the other half forms the sums of the tile before, in ascending key order
    if (tid >= HALF) {
        constexpr int KEYS = AR_TILE / (HALF / 32);                // of a thread per tile: w, w + 4, ...
        const int w = warp - HALF / 32;
        float sv[KEYS], next[KEYS];                                // scores of this tile and of the next, on their way meanwhile
        auto fetch = [&](float (&o)[KEYS], int t) {
            const int cnt = min(AR_TILE, nkeys - t * AR_TILE);
            const float *src = my_scores + (size_t)(t * AR_TILE + w) * AR_PAIRS;
#pragma unroll
            for (int i = 0; i < KEYS; i++) o[i] = w + HALF / 32 * i < cnt ? src[HALF / 32 * i * AR_PAIRS] : 0.0f;
        };
        fetch(sv, 0);
#pragma unroll 1
        for (int t = 0; t <= ntiles; t++) {
            if (t < ntiles) {
                if (t + 1 < ntiles) fetch(next, t + 1);
                const int cnt = min(AR_TILE, nkeys - t * AR_TILE), tb = t_lo + t * AR_TILE;
                float *pb = psm + (size_t)(t & 1) * AR_TILE * AR_PAIRS + lane;
                // eight exponentials side by side (one after the other they take 190 cycles each)
                constexpr int SIDE = 8;
#pragma unroll
                for (int i0 = 0; i0 < KEYS; i0 += SIDE) {
                    float e[SIDE];
#pragma unroll
                    for (int i = 0; i < SIDE; i++) e[i] = __fsub_rn(sv[i0 + i], mx);
                    brrr_expf_n<SIDE>(e);
#pragma unroll
                    for (int i = 0; i < SIDE; i++) {
                        const int kk = w + HALF / 32 * (i0 + i), key = tb + kk;
                        if (kk < cnt) pb[kk * AR_PAIRS] = key >= my_start && key <= my_pos ? e[i] : 0.0f;
                    }
                }
#pragma unroll
                for (int i = 0; i < KEYS; i++) sv[i] = next[i];
            }
            __syncthreads();           // probabilities of tile t are there, the sums of tile t - 1 done
        }
        __syncthreads();               // outputs in shared memory
    } else {
        const int dq = tid & 7, pg = tid >> 3;                     // dims 4 dq .. + 3 and 32 + 4 dq .. + 3 of pairs 2 pg and 2 pg + 1
        float acc[2][8];
#pragma unroll
        for (int j = 0; j < 2; j++)
#pragma unroll
            for (int i = 0; i < 8; i++) acc[j][i] = 0.0f;
        float den = den_sm[2 * pg + (dq & 1)];                     // of one of the pairs (the threads past the first two repeat them)
        __syncthreads();
        for (int t = 0; t < ntiles; t++) {
            const int cnt = min(AR_TILE, nkeys - t * AR_TILE);
            if (tid == 0 && t + 1 < ntiles) { fence_proxy_async(); issue(a.vc, vtile, vbar, t + 1); }      // its buffer: the sums of tile t - 1 are done
            waiter.wait(&vbar[t & 1], (uint32_t)(t >> 1) & 1u);
            const float *vt = vtile + (size_t)(t & 1) * AR_TILE * HD + 4 * dq, *pt = psm + (size_t)(t & 1) * AR_TILE * AR_PAIRS + 2 * pg;
#pragma unroll 4
            for (int kk = 0; kk < cnt; kk++) {
                const float4 v = *reinterpret_cast<const float4 *>(vt + kk * HD), v2 = *reinterpret_cast<const float4 *>(vt + kk * HD + 32);
                const float2 w = *reinterpret_cast<const float2 *>(pt + kk * AR_PAIRS);
                const float p[2] = {w.x, w.y};
#pragma unroll
                for (int j = 0; j < 2; j++) {
                    acc[j][0] = __fmaf_rn(v.x, p[j], acc[j][0]); acc[j][1] = __fmaf_rn(v.y, p[j], acc[j][1]);
                    acc[j][2] = __fmaf_rn(v.z, p[j], acc[j][2]); acc[j][3] = __fmaf_rn(v.w, p[j], acc[j][3]);
                    acc[j][4] = __fmaf_rn(v2.x, p[j], acc[j][4]); acc[j][5] = __fmaf_rn(v2.y, p[j], acc[j][5]);
                    acc[j][6] = __fmaf_rn(v2.z, p[j], acc[j][6]); acc[j][7] = __fmaf_rn(v2.w, p[j], acc[j][7]);
                }
                den = __fadd_rn(den, (dq & 1) ? w.y : w.x);
            }
            __syncthreads();
        }
        // ---- outputs: o = acc / den through shared memory, then the Q8 image of every pair's two 32-blocks (a warp = one 32-block of a pair)
        const float inv1 = __fdiv_rn(1.0f, den);                   // lane dq of a group of eight holds pair dq & 1
#pragma unroll
        for (int j = 0; j < 2; j++) {
            const float inv = __shfl_sync(0xffffffffu, inv1, (lane & 24) + j);
            float *o = qsm + (2 * pg + j) * HD + 4 * dq;
            *reinterpret_cast<float4 *>(o) = make_float4(__fmul_rn(acc[j][0], inv), __fmul_rn(acc[j][1], inv), __fmul_rn(acc[j][2], inv), __fmul_rn(acc[j][3], inv));
            *reinterpret_cast<float4 *>(o + 32) = make_float4(__fmul_rn(acc[j][4], inv), __fmul_rn(acc[j][5], inv), __fmul_rn(acc[j][6], inv), __fmul_rn(acc[j][7], inv));
        }
        __syncthreads();               // outputs in shared memory
    }
    // (four at a time, side by side)
    constexpr int SIDE = 4, BLOCKS = 2 * AR_PAIRS / (AR_THREADS / 32);
#pragma unroll 1
    for (int k0 = warp * BLOCKS; k0 < (warp + 1) * BLOCKS; k0 += SIDE) {
        float o[SIDE], amax[SIDE];
#pragma unroll
        for (int k = 0; k < SIDE; k++) { o[k] = qsm[(k0 + k) * 32 + lane]; amax[k] = fabsf(o[k]); }
#pragma unroll
        for (int x = 16; x > 0; x >>= 1)
#pragma unroll
            for (int k = 0; k < SIDE; k++) amax[k] = fmaxf(amax[k], __shfl_xor_sync(0xffffffffu, amax[k], x));
#pragma unroll
        for (int k = 0; k < SIDE; k++) amax[k] = fmaxf(amax[k], 1e-12f);
        float sc[SIDE];
#pragma unroll
        for (int k = 0; k < SIDE; k++) sc[k] = __fdiv_rn(amax[k], 127.0f);
#pragma unroll
        for (int k = 0; k < SIDE; k++) {
            const int p2 = (k0 + k) >> 1, rr = p2 >> lg, b = (kvh * group + (p2 & (group - 1))) * 2 + ((k0 + k) & 1);
            if (rr >= nrows) break;             // uniform over the warp; the rows ascend
            const int qv = brrr_q8_round_inv(o[k], sc[k], brrr_q8_inv(amax[k]));
            const size_t row = (size_t)(r0 + rr);
            a.ao[row * a.nh * HD + b * 32 + lane] = o[k];
            if (lane == 0) a.as[row * a.nh * 2 + b] = sc[k];
            if (a.aq) a.aq[row * a.nh * HD + b * 32 + lane] = (int8_t)qv;
            if (a.img) ti_emit_block<TI_HALF>(qv, lane, b, a.img + row * a.nh * ti_pair(TI_HALF));
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
