// Matrices x token rows on the 5th-generation tensor cores (tcgen05.mma, accumulators in tensor memory): the
// MXFP4 experts and the Q8 projections of prompt tiles and batched decode.  One pass over the weights serves up to
// 512 token rows, as the reference's tile path does on the CPU for 16 (src/bin/engine_gpt2.rs:1005-1010, TILE = 16),
// and every output equals the per-token result bit for bit.
//
// Arithmetic.  A row's value is a set of float chains over the 32-blocks b, one step per block:
//   MXFP4: four lane chains,              acc_j    = fma(t_j(b), 2^(e_b-128) * xs[b], acc_j)
//   Q8:    2 block parities x four lanes, acc_{p,j} = fma(t_j(b), ws[b] * xs[b], acc_{p,j}),  p = b & 1
// with t_j(b) the exact integer dot of the lane's 8 weights with its 8 activation bytes.  The tensor core supplies
// t_j(b) as exact floats, so no thread converts an integer:
//   MXFP4  kind::f8f6f4, A = the raw e2m1 codes (4 bits in the low half of 16-byte containers), B = the two e4m3 planes
//          of the activation (brrr_tile.cuh).  One product per lane chain j and block pair: its K = 32 is the 16 codes of
//          lane j (8 of either block) twice - the descriptor's K stride is zero, so both 16-byte columns of operand A
//          are the same bytes - against plane 0 and plane 1.  |t| <= 12192: 14 bits, exact in the f32 accumulator.
//   Q8     kind::f16, A = the int8 weights as halves (re-laid at load), B = the activation bytes as halves; K = 16 is the
//          8 weights of lane j in either block.  |t| <= 129032: exact.
// Column n of product j is (token, block q): row n of B is zero outside block q, so one product gives both blocks' dots
// of 128 rows x NT tokens.  The worker threads (thread = matrix row and 8 tokens) read them from tensor memory
// (tcgen05.ld) and run the chains, two tokens per instruction (fma.rn.f32x2: two independent round-to-nearest operations).
//
// What bounds it: the workers' instruction stream.  The chains - per row, token and block four fused multiply-adds that nothing may
// reorder - take about 2.8 cycles per packed instruction (three 64-bit operands from the register file), 490 cycles per pair of
// 128 rows x 32 tokens and scheduler; with reads, scales and barriers a pair takes 900.  Beside it run the products (four of 50 to
// 60 cycles) and the copies.  Measured on 512 rows of the 20b shape (ncu, one launch): gate | up 595 us (671 with the products issued in a
// one-lane branch) and down 309 us (before, with int8 operands decoded by the workers and one conversion per dot: 2 x 835 and 835),
// q/k/v 161 and o-proj 142 us (integer units: 520 and 480).  At 8 tokens per CTA (64 rows, gate | up 138 us, three CTAs per SM) it is the workers too:
// of 900 to 1140 cycles a pair (with clock stamps) they multiply for 370 to 470, prepare scales for 100 to 160, read tensor memory for 110 and wait
// for products for 170 to 190, while the issuing warps wait for them to leave a buffer for three quarters of the time.
//
// Roles of a CTA (128 matrix rows x up to NT tokens).  Worker warps: NT / 8 groups of four.  Then two producer
// warps (asynchronous copies of the pairs' operands into a ring) and two issuing warps (four products per pair, even
// pairs into the one accumulator buffer, odd pairs into the other).  Barriers (all waits bounded): full[slot] the pair's
// operands have landed; empty[slot] the products have read them; dfull[buf] the pair's products are complete; dempty[buf]
// every live worker warp has read them; scbar the rows' scales of all pairs have landed.
#include <cuda.h>
#include <type_traits>
#include "brrr_kernels.h"
#include "brrr_block.cuh"
#include "brrr_tma.cuh"
#include "brrr_tc.cuh"
#include "brrr_mx.cuh"
#include "brrr_tile.cuh"
#include "brrr_tmap.h"

namespace brrr {

namespace {

constexpr int TL_ROWS = 128;             // rows per CTA = MMA M
constexpr int TL_MAXTOK = BRRR_TILE_MAX; // entries per expert and launch (one per token of the tile at most)

constexpr int QOP_UNIT = 16384 + 1024;    // bytes of a Q8 operand tile per block pair (launch_q8_operand_pack)

enum { TK_MX = 0, TK_GLU = 1, TK_Q8 = 2 };      // one MXFP4 matrix; gate | up with the SwiGLU and the Q8 of h; a Q8 matrix

template <int KIND>
__device__ __forceinline__ void tl_mma(uint32_t issue, uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc) {
    if (KIND == TK_Q8)
        asm volatile("{\n\t.reg .pred p, e;\n\tsetp.ne.b32 p, %4, 0;\n\tsetp.ne.b32 e, %5, 0;\n\t"
                     "@e tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%4, %4, %4, %4}, p;\n\t}" ::"r"(tmem_d), "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(0u), "r"(issue)
                     : "memory");
    else
        asm volatile("{\n\t.reg .pred p, e;\n\tsetp.ne.b32 p, %4, 0;\n\tsetp.ne.b32 e, %5, 0;\n\t"
                     "@e tcgen05.mma.cta_group::1.kind::f8f6f4 [%0], %1, %2, %3, {%4, %4, %4, %4}, p;\n\t}" ::"r"(tmem_d), "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(0u), "r"(issue)
                     : "memory");
}
// box of a 4-d tensor map at (0, 0, c2, c3) -> shared memory
__device__ __forceinline__ void tensor_g2s(uint32_t dst, const CUtensorMap *map, int c2, int c3, uint64_t *bar) {
    asm volatile("cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %2, %3, %4}], [%5];" ::"r"(dst), "l"(map),
                 "r"(0), "r"(c2), "r"(c3), "r"(smem_u32(bar))
                 : "memory");
}
// One launch serves blockIdx.y = task = (expert or the single matrix, chunk of its entries).  Each expert has a list of up
// to 512 entries; entry i multiplies the activation row i / src_div and writes output row i.
struct alignas(64) TileArgs {
    CUtensorMap ma, mb;      // MX, GLU: the 16-row units as tensors (mx_tensor_map; GLU: gate and up)
    const uint8_t *wa, *wb;  // MX, GLU: the same units (their exponents); Q8: operand tiles (launch_q8_operand_pack)
    int np;                  // block pairs per row
    int row0, nrows;         // rows [row0, row0 + nrows) of each expert's matrix (GLU: nrows of gate and of up)
    int rows_per_expert;     // matrix row of (expert e, row r) = e * rows_per_expert + r
    const int *cnt;          // [ne] entries per expert; nullptr: one matrix, entries 0 .. ntok - 1
    const int *list;         // [ne][TL_MAXTOK]
    int ne, ntok, src_div;
    const uint8_t *img;      // activation images [row][np * ti_pair]: planes (MX, GLU) or halves (Q8)
    const float *xs;         // block scales [row][2 np]
    const float *bias, *bias_b;  // nullable: [ne][rows_per_expert], added to every output (GLU: of gate and of up, required)
    float *y;                // MX, Q8: element [entry][row - row0], rows ldy apart
    int ldy, epi;            // Q8: Q8_EPI_*
    uint8_t *himg;           // GLU: plane images of h [entry][nrows / 64 * 256] and its scales [entry][nrows / 32]
    float *hs;
    DevState *state;
};

// A ring slot holds a pair's operands; the rows' scales stay in a region of their own for the whole kernel, so a worker waits for the
// products only.  Scales per row and pair: 2 e8m0 bytes, Q8: 2 floats.
template <int KIND> __host__ __device__ constexpr int tl_a_bytes() { return KIND == TK_Q8 ? 16384 : 8192; }       // four operands of 4 or 2 KB
template <int KIND> __host__ __device__ constexpr int tl_sc_bytes() { return KIND == TK_Q8 ? 1024 : 256; }        // per pair
template <int KIND, int NT> __host__ __device__ constexpr bool tl_scale_table() { return KIND != TK_Q8 && NT == 32; }      // e8m0 bytes expanded to floats once
template <int KIND, int NT> __host__ __device__ constexpr int tl_slot_bytes() { return tl_a_bytes<KIND>() + NT * 256; }
// Even: each issuing warp then has slots of its own.  (With an odd depth both use every slot, and a warp could take the other one's
// phase of full[] for its own: a parity wait returns as well while the phase before last is the last complete one.)
template <int KIND, int NT> __host__ __device__ constexpr int tl_depth() { return KIND == TK_Q8 || NT == 8 ? 4 : 6; }
template <int KIND, int NT>
size_t tl_smem(int np) {
    return (size_t)tl_depth<KIND, NT>() * tl_slot_bytes<KIND, NT>() + (size_t)np * tl_sc_bytes<KIND>() + (tl_scale_table<KIND, NT>() ? (size_t)np * 1024 : 0) +
           (size_t)np * 2 * NT * 4 + (KIND == TK_GLU ? NT * 128 * 4 : 0);
}

template <int KIND, int NT, bool FEW = false>
__global__ void __launch_bounds__(NT * 16 + 128, KIND == TK_Q8 || NT == 32 ? 1 : NT == 16 ? 2 : 3) tile_kernel(const __grid_constant__ TileArgs a) {
    constexpr int WORKERS = NT * 16, THREADS = WORKERS + 128;
    constexpr int TL_DEPTH = tl_depth<KIND, NT>(), SLOT = tl_slot_bytes<KIND, NT>(), A_BYTES = tl_a_bytes<KIND>(), B_OFF = A_BYTES, SC = tl_sc_bytes<KIND>();
    // operand A of product j at j * A_STEP; MX: core matrix (8 rows, chain j) at (row / 8) * 512 + j * 128, both K columns the same
    constexpr uint32_t A_STEP = KIND == TK_Q8 ? 4096 : 128, A_LBO = KIND == TK_Q8 ? 2048 : 0, A_SBO = KIND == TK_Q8 ? 128 : 512;
    constexpr int PAIR = ti_pair(KIND == TK_Q8 ? TI_HALF : TI_PLANES);
    constexpr uint32_t B_LBO = NT * 32, B_STEP = NT * 64;        // operand B of product j at j * B_STEP: [K column][group of eight tokens][block][8 rows x 16 bytes]
    constexpr uint32_t BUF_COLS = 8 * NT;                                             // accumulator columns of one pair
    constexpr uint32_t TMEM_COLS = 2 * BUF_COLS;
    static_assert(TL_DEPTH % 2 == 0, "each issuing warp has slots of its own");
    constexpr bool TABLE = tl_scale_table<KIND, NT>();
    constexpr int CH = KIND == TK_Q8 ? 8 : 4;                                         // chains per row and token
    extern __shared__ __align__(128) unsigned char tsm[];
    const int np = a.np;
    unsigned char *ring = tsm;
    unsigned char *sc_sm = tsm + TL_DEPTH * SLOT;                                     // [pair][SC]
    float2 *sc2_sm = reinterpret_cast<float2 *>(sc_sm + (size_t)np * SC);             // scale table: [pair][128 rows]
    float *xs_sm = reinterpret_cast<float *>(sc2_sm + (TABLE ? (size_t)np * 128 : 0)); // [pair][block of the pair][NT]
    float *glu_sm = xs_sm + (size_t)np * 2 * NT;                                      // GLU: [NT][128 rows]
    __shared__ float tbl[256];
    __shared__ __align__(8) uint64_t full[TL_DEPTH], empty[TL_DEPTH], dfull[2], dempty[2], scbar;
    __shared__ uint32_t tmem_base_sh;
    __shared__ int task_sh[3];               // expert, first entry, entries
    __shared__ int ent[NT];
    // gate | up: a warp index the compiler knows to be uniform (7 % of a 512-row tile of the 20b shape; the other kinds lose 3 to 8 % with it)
    const int tid = threadIdx.x, warp = KIND == TK_GLU ? __shfl_sync(0xffffffffu, tid >> 5, 0) : tid >> 5, lane = tid & 31;
    // ---- what needs nothing from the kernels before
    if (KIND != TK_Q8) mx_fill_scale_table(tbl, tid, THREADS);
    else {
        // zero rows of operand B (a plane image brings its zeros along); rows of absent tokens only reach columns nobody stores
        constexpr int Z = (SLOT - B_OFF) / 16;
        for (int i = tid; i < TL_DEPTH * Z; i += THREADS) *reinterpret_cast<uint4 *>(ring + (i / Z) * SLOT + B_OFF + (i % Z) * 16) = make_uint4(0, 0, 0, 0);
        fence_proxy_async();                 // these stores -> the tensor core's reads
    }
    pdl_wait();
    pdl_trigger();
    if (warp == 0) {
        // task -> (expert, chunk): experts in order, ceil(entries / NT) chunks each
        const int per = a.cnt ? (a.ne + 31) / 32 : 1, e0 = lane * per;
        int c[8], mine = 0;
#pragma unroll
        for (int i = 0; i < 8; i++) {
            c[i] = 0;
            if (i < per) c[i] = a.cnt ? (e0 + i < a.ne ? a.cnt[e0 + i] : 0) : (lane == 0 ? a.ntok : 0);
            mine += (c[i] + NT - 1) / NT;
        }
        int incl = mine;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) { const int v = __shfl_up_sync(0xffffffffu, incl, o); if (lane >= o) incl += v; }
        if (lane == 0) task_sh[2] = 0;
        __syncwarp();
        int t = (int)blockIdx.y - (incl - mine);
        if (t >= 0 && t < mine) {
#pragma unroll
            for (int i = 0; i < 8; i++) {
                const int n = (c[i] + NT - 1) / NT;
                if (t >= 0 && t < n) {
                    const int step = ((c[i] + n - 1) / n + 7) & ~7;         // equal chunks, whole groups of eight
                    task_sh[0] = e0 + i; task_sh[1] = t * step; task_sh[2] = min(step, c[i] - t * step);
                    t = -1;
                } else if (t >= 0) t -= n;
            }
        }
    }
    __syncthreads();
    const int e = task_sh[0], first = task_sh[1], n_ent = task_sh[2];
    if (n_ent <= 0) return;                  // nothing here (before anything is allocated)
    const int groups = (n_ent + 7) >> 3;     // live groups of eight tokens
    const int live_warps = 4 * groups;
    if (tid == WORKERS) {
        for (int i = 0; i < TL_DEPTH; i++) { mbar_init(&full[i], 65); mbar_init(&empty[i], 1); }
        mbar_init(&scbar, KIND == TK_Q8 ? 1 : 32);
        for (int i = 0; i < 2; i++) { mbar_init(&dfull[i], 1); mbar_init(&dempty[i], live_warps); }
        mbar_fence_init();
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_sh)), "r"(TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (tid < NT) ent[tid] = tid < n_ent ? (a.list ? a.list[e * TL_MAXTOK + first + tid] : first + tid) : 0;
    tl_fence_before();
    __syncthreads();
    tl_fence_after();
    const uint32_t tmem_base = KIND == TK_GLU ? __shfl_sync(0xffffffffu, tmem_base_sh, 0) : tmem_base_sh;
    TlWaiter wait{a.state ? &a.state->err : nullptr, a.state && *reinterpret_cast<volatile uint32_t *>(&a.state->err) != 0u};
    const int tile = blockIdx.x;
    // MX, GLU: a tile starts on a 16-row unit; a row window that does not starts in the middle of its first tile
    const int row0 = e * a.rows_per_expert + a.row0, unit0 = (row0 >> 4) + tile * (KIND == TK_GLU ? 4 : 8);
    const int shift = KIND == TK_MX ? row0 & 15 : 0;
    const int n_units = KIND == TK_GLU ? 8 : min(8, (shift + a.nrows - tile * TL_ROWS + 15) >> 4);

    if (warp < WORKERS / 32 + 2 && warp >= WORKERS / 32) {
        // ---------------- producers: two warps share the tokens' activations; lane 0 of the first also issues the weights' copies
        const bool weights = warp == WORKERS / 32;
        if (weights) {
            if (KIND == TK_Q8) {
                if (lane == 0) {
                    mbar_expect_tx(&scbar, (uint32_t)np * SC);
                    bulk_g2s(sc_sm, a.wa + (size_t)tile * np * QOP_UNIT + (size_t)np * A_BYTES, (uint32_t)np * SC, &scbar);
                }
            } else {
                for (int i = lane; i < n_units * 2 * np; i += 32) {      // exponents of every pair
                    const int p = i / (n_units * 2), k = i % (n_units * 2), u = k >> 1;
                    const uint8_t *unit = KIND == TK_GLU && u >= 4 ? a.wb + mx_unit_off(unit0 + u - 4, p, np) : a.wa + mx_unit_off(unit0 + u, p, np);
                    cp_async16(smem_u32(sc_sm) + p * SC + k * 16, unit + MX_UNIT_EXPS + (k & 1) * 16);
                }
                cp_async_arrive(&scbar);
            }
        }
        // activations: lane = (token of a group of eight, quarter of its 16-byte pieces): planes: (chain jj, plane r >> 1, block r & 1);
        // halves: (chain 2 i + (r >> 1), block r & 1)
        constexpr int NG = NT / 8, MINE = (NG + 1) / 2;        // groups of eight tokens, at most MINE of them per producer warp
        const uint8_t *src[MINE];
        bool live[MINE];
        const int r = lane & 3;
#pragma unroll
        for (int k = 0; k < MINE; k++) {
            const int g = weights ? k : MINE + k, t = g * 8 + (lane >> 2);
            live[k] = g < NG && t < n_ent;
            src[k] = a.img + (size_t)(ent[live[k] ? t : 0] / a.src_div) * np * PAIR + r * 16;
        }
        const uint32_t ring0 = smem_u32(ring);
        const uint32_t dst0 = ring0 + B_OFF + (weights ? 0 : MINE * 256) + (lane >> 2) * 16 + (r & 1) * 128 +
                              (KIND == TK_Q8 ? (r >> 1) * B_STEP + (r & 1) * B_LBO : (r >> 1) * B_LBO);
        const uint8_t *wsrc = a.wa + (size_t)tile * np * QOP_UNIT;
        int slot = 0;
        uint32_t par = 1;
        for (int p = 0; p < np; p++) {
            wait(&empty[slot], par);
            if (weights && lane == 0) {
                // MX: a tensor copy (GLU: two) widens each 8-byte word of a row and chain into the 16-byte container of a 4-bit operand;
                // the barrier counts the packed bytes, not the padding
                mbar_expect_tx(&full[slot], KIND == TK_Q8 ? A_BYTES : A_BYTES / 2);
                if (KIND == TK_Q8) bulk_g2s(ring + slot * SLOT, wsrc + (size_t)p * A_BYTES, A_BYTES, &full[slot]);
                else tensor_g2s(ring0 + slot * SLOT, &a.ma, unit0, p, &full[slot]);
                if (KIND == TK_GLU) tensor_g2s(ring0 + slot * SLOT + A_BYTES / 2, &a.mb, unit0, p, &full[slot]);
            }
            __syncwarp();
            const uint32_t dst = dst0 + slot * SLOT;
#pragma unroll
            for (int k = 0; k < MINE; k++) {
                if (live[k]) {
                    if (KIND == TK_Q8) {
#pragma unroll
                        for (int i = 0; i < 2; i++) cp_async16(dst + k * 256 + i * 2 * B_STEP, src[k] + i * 64);
                    } else {
#pragma unroll
                        for (int jj = 0; jj < 4; jj++) cp_async16(dst + k * 256 + jj * B_STEP, src[k] + jj * 64);
                    }
                }
                src[k] += PAIR;
            }
            cp_async_arrive(&full[slot]);
            if (++slot == TL_DEPTH) { slot = 0; par ^= 1u; }
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
    } else if (warp >= WORKERS / 32 + 2) {
        // ---------------- issuers: one for the even pairs (buffer 0), one for the odd (the whole warp walks the loop, one elected lane issues)
        // D = f32, both K-major; MX: A = e2m1 (5), B = e4m3 (0); Q8: A = B = f16 (0); N = 16 columns per group of eight tokens
        const uint32_t idesc = (1u << 4) | (KIND == TK_Q8 ? 0u : (5u << 7)) | ((uint32_t)(2 * groups) << 17) | ((TL_ROWS >> 4) << 24);
        const uint64_t da0 = tl_smem_desc(ring, A_LBO, A_SBO), db0 = tl_smem_desc(ring + B_OFF, B_LBO, 128);
        const int buf = warp - (WORKERS / 32 + 2);
        const uint32_t issue = elect_one() ? 1u : 0u;
        int slot = buf;
        uint32_t fpar = 0, dpar = 1;
        for (int p = buf; p < np; p += 2) {
            wait(&full[slot], fpar);
            fence_proxy_async();                   // the copies seen through full[] (generic proxy) -> the tensor core's reads
            wait(&dempty[buf], dpar);
            dpar ^= 1u;
            tl_fence_after();
            const uint64_t da = da0 + (uint64_t)(slot * (SLOT / 16)), db = db0 + (uint64_t)(slot * (SLOT / 16));
            const uint32_t d0 = tmem_base + buf * BUF_COLS;
#pragma unroll
            for (int j = 0; j < 4; j++) tl_mma<KIND>(issue, d0 + j * 2 * NT, da + j * (A_STEP / 16), db + j * (B_STEP / 16), idesc);
            tl_commit_if(issue, &dfull[buf]);
            tl_commit_if(p + TL_DEPTH < np ? issue : 0u, &empty[slot]);      // nobody waits for the last ones
            __syncwarp();
            if ((slot += 2) >= TL_DEPTH) { slot -= TL_DEPTH; fpar ^= 1u; }
        }
    } else if (warp < live_warps) {
        // ---------------- workers: thread = matrix row m, tokens 8 wg .. + 7
        const int wg = warp >> 2, m = tid & 127;
        const int t_base = wg * 8;
        {
            // block scales of this group's tokens, [pair][block][token] so that two neighbours are one operand; every load before the
            // first store (a store in between would order the loads behind it, each a round trip to L2)
            const int t = t_base + (m & 7), nb = np * 2;
            const float *src = a.xs + (size_t)(ent[t < n_ent ? t : 0] / a.src_div) * nb;
            float v[8];
#pragma unroll
            for (int k = 0; k < 8; k++) v[k] = (m >> 3) + 16 * k < nb ? src[(m >> 3) + 16 * k] : 0.0f;
#pragma unroll
            for (int k = 0; k < 8; k++) if ((m >> 3) + 16 * k < nb) xs_sm[((m >> 3) + 16 * k) * NT + t] = v[k];
            for (int b = (m >> 3) + 128; b < nb; b += 16) xs_sm[b * NT + t] = src[b];
        }
        wait(&scbar, 0u);
        if (TABLE) {
            // this group's share of the pairs; then every live group has the whole table
#pragma unroll 4
            for (int p = wg; p < np; p += groups) {
                const uint32_t e2 = *reinterpret_cast<const unsigned short *>(sc_sm + p * SC + m * 2);
                sc2_sm[p * 128 + m] = make_float2(tbl[e2 & 0xFFu], tbl[e2 >> 8]);
            }
        }
        asm volatile("bar.sync 1, %0;" ::"r"(live_warps * 32) : "memory");
        uint32_t sc_addr = TABLE ? smem_u32(sc2_sm + m) : smem_u32(sc_sm) + m * (KIND == TK_Q8 ? 8 : 2), xs_addr = smem_u32(xs_sm + t_base);
        const uint32_t lane_addr = tmem_base + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)(t_base * 2);
        f32x2 acc[CH][4];
#pragma unroll
        for (int c = 0; c < CH; c++)
#pragma unroll
            for (int i = 0; i < 4; i++) acc[c][i] = 0ull;
        uint32_t par = 0;                              // of dfull of the pair at hand
        auto pair_step = [&](int buf) {
            uint2 w;                                   // this row's scales of the pair's blocks
            if (KIND == TK_Q8 || TABLE) w = lds64(sc_addr);
            else {
                uint32_t e2;
                asm volatile("ld.shared.u16 %0, [%1];" : "=r"(e2) : "r"(sc_addr));
                w = make_uint2(__float_as_uint(tbl[e2 & 0xFFu]), __float_as_uint(tbl[e2 >> 8]));
            }
            sc_addr += TABLE ? 1024 : SC;
            const f32x2 ww[2] = {tl_pack2(w.x, w.x), tl_pack2(w.y, w.y)};
            const uint32_t addr = lane_addr + buf * BUF_COLS;
            auto scales = [&](int q, f32x2 (&o)[4]) {  // of the eight tokens in block q: row scale x activation scale
                lds_pairs(xs_addr + q * NT * 4, o[0], o[1]);
                lds_pairs(xs_addr + q * NT * 4 + 16, o[2], o[3]);
#pragma unroll
                for (int i = 0; i < 4; i++) o[i] = tl_mul2(ww[q], o[i]);
            };
            auto release = [&]() {                     // every column of the pair has been read
                tl_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&dempty[buf]);
            };
            if (KIND == TK_Q8) {                       // fewer registers beside 64 of chains: one block at a time
#pragma unroll
                for (int q = 0; q < 2; q++) {
                    f32x2 s2[4];
                    scales(q, s2);
                    if (q == 0) { wait(&dfull[buf], par); tl_fence_after(); }
#pragma unroll
                    for (int j = 0; j < 4; j += 2) {
                        f32x2 v[4], u[4];
                        tl_ld8x2(addr + j * 2 * NT + q * 8, addr + (j + 1) * 2 * NT + q * 8, v, u);
                        if (j == 2 && q == 1) release();
#pragma unroll
                        for (int i = 0; i < 4; i++) {
                            f32x2 &c0 = acc[(q * 4 + j) % CH][i], &c1 = acc[(q * 4 + j + 1) % CH][i];
                            c0 = tl_fma2(v[i], s2[i], c0);
                            c1 = tl_fma2(u[i], s2[i], c1);
                        }
                    }
                }
            } else {
                f32x2 s2[2][4];
                scales(0, s2[0]);
                scales(1, s2[1]);
                wait(&dfull[buf], par);
                tl_fence_after();
#pragma unroll
                for (int j = 0; j < 4; j += 2) {
                    f32x2 v[8], u[8];
                    tl_ld16x2(addr + j * 2 * NT, addr + (j + 1) * 2 * NT, v, u);
                    if (j == 2) release();
#pragma unroll
                    for (int q = 0; q < 2; q++)
#pragma unroll
                        for (int i = 0; i < 4; i++) {
                            acc[j][i] = tl_fma2(v[q * 4 + i], s2[q][i], acc[j][i]);
                            acc[j + 1][i] = tl_fma2(u[q * 4 + i], s2[q][i], acc[j + 1][i]);
                        }
                }
            }
            xs_addr += 2 * NT * 4;
        };
        // A CTA of eight tokens often has one or two (a short prompt or a small batch meets most experts with a row each): then only their
        // columns are read and their chains carried.
        auto few_step = [&](auto pairs, int buf) {
            constexpr int TP = decltype(pairs)::value;
            uint32_t e2;
            asm volatile("ld.shared.u16 %0, [%1];" : "=r"(e2) : "r"(sc_addr));
            const uint32_t w0 = __float_as_uint(tbl[e2 & 0xFFu]), w1 = __float_as_uint(tbl[e2 >> 8]);
            sc_addr += SC;
            f32x2 s2[2][TP], v[8][TP];
#pragma unroll
            for (int q = 0; q < 2; q++) {
                if (TP == 2) lds_pairs(xs_addr + q * NT * 4, s2[q][0], s2[q][TP - 1]);
                else {
                    const uint2 x = lds64(xs_addr + q * NT * 4);
                    s2[q][0] = tl_pack2(x.x, x.y);
                }
#pragma unroll
                for (int i = 0; i < TP; i++) s2[q][i] = tl_mul2(q ? tl_pack2(w1, w1) : tl_pack2(w0, w0), s2[q][i]);
            }
            xs_addr += 2 * NT * 4;
            wait(&dfull[buf], par);
            tl_fence_after();
            tl_ld_blocks(lane_addr + buf * BUF_COLS, 2 * NT, v);
            tl_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&dempty[buf]);
#pragma unroll
            for (int q = 0; q < 2; q++)
#pragma unroll
                for (int j = 0; j < 4; j++)
#pragma unroll
                    for (int i = 0; i < TP; i++) acc[j][i] = tl_fma2(v[2 * j + q][i], s2[q][i], acc[j][i]);
        };
        auto few = [&](auto pairs) {
#pragma unroll 1
            for (int p = 0; p < np; p += 2) {
                few_step(pairs, 0);
                if (p + 1 < np) few_step(pairs, 1);
                par ^= 1u;
            }
        };
        if (FEW && n_ent <= 2) few(std::integral_constant<int, 1>{});
        else if (FEW && n_ent <= 4) few(std::integral_constant<int, 2>{});
        else {
#pragma unroll 1
            for (int p = 0; p < np; p += 2) {
                pair_step(0);
                if (p + 1 < np) pair_step(1);
                par ^= 1u;
            }
        }
        // ---------------- outputs
        const int row_local = KIND == TK_GLU ? tile * 64 + (m & 63) : tile * TL_ROWS + m - shift;
        const bool row_live = row_local >= 0 && row_local < a.nrows;
        const float *bp = KIND == TK_GLU && m >= 64 ? a.bias_b : a.bias;
        const float bias = bp && row_live ? bp[(size_t)e * a.rows_per_expert + a.row0 + row_local] : 0.0f;
#pragma unroll
        for (int i = 0; i < 4; i++) {
            float c[CH][2], v[2];
#pragma unroll
            for (int k = 0; k < CH; k++) tl_unpack2(acc[k][i], c[k][0], c[k][1]);
#pragma unroll
            for (int u = 0; u < 2; u++) {
                if (KIND == TK_Q8)               // acc_even + acc_odd per lane, then (l0 + l1) + (l2 + l3)
                    v[u] = __fadd_rn(__fadd_rn(__fadd_rn(c[0][u], c[4 % CH][u]), __fadd_rn(c[1][u], c[5 % CH][u])),
                                     __fadd_rn(__fadd_rn(c[2][u], c[6 % CH][u]), __fadd_rn(c[3][u], c[7 % CH][u])));
                else v[u] = __fadd_rn(__fadd_rn(c[0][u], c[1][u]), __fadd_rn(c[2][u], c[3][u]));
                const int t = t_base + 2 * i + u;
                if (KIND == TK_GLU) glu_sm[t * 128 + m] = __fadd_rn(v[u], bias);
                else if (row_live && t < n_ent) {
                    float *yp = a.y + (size_t)ent[t] * a.ldy + row_local;
                    if (KIND == TK_Q8 && a.epi == Q8_EPI_RESID_BIAS) *yp = __fadd_rn(*yp, __fadd_rn(v[u], bias));        // x += dot + bias
                    else *yp = a.bias ? __fadd_rn(v[u], bias) : v[u];
                }
            }
        }
        if (KIND == TK_GLU) {
            // h = SwiGLU(gate, up) of 64 outputs x 8 tokens, its Q8 and plane image: warp = 32-block (warp & 1) of four tokens, side by side
            asm volatile("bar.sync %0, 128;" ::"r"(2 + wg) : "memory");
            const int blk = warp & 1, b = tile * 2 + blk, t0 = t_base + ((warp >> 1) & 1) * 4;
            float hv[4], amax[4];
#pragma unroll
            for (int k = 0; k < 4; k++) {
                hv[k] = swiglu_oai(glu_sm[(t0 + k) * 128 + blk * 32 + lane], glu_sm[(t0 + k) * 128 + 64 + blk * 32 + lane]);
                amax[k] = fabsf(hv[k]);
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1)
#pragma unroll
                for (int k = 0; k < 4; k++) amax[k] = fmaxf(amax[k], __shfl_xor_sync(0xffffffffu, amax[k], o));
#pragma unroll
            for (int k = 0; k < 4; k++) {
                if (t0 + k >= n_ent) break;
                const float am = fmaxf(amax[k], 1e-12f), sc = __fdiv_rn(am, 127.0f);
                const size_t row = (size_t)ent[t0 + k];
                if (lane == 0) a.hs[row * (a.nrows / 32) + b] = sc;
                ti_emit_block<TI_PLANES>(brrr_q8_round_inv(hv[k], sc, brrr_q8_inv(am)), lane, b, a.himg + row * (size_t)(a.nrows / 64) * PAIR);
            }
        }
    }
    tl_fence_before();
    __syncthreads();
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(TMEM_COLS) : "memory");
}

// ---------------------------------------------------------------- load-time re-layout of a Q8 matrix into operand units
// A 128-row tile is [block pair][16384 B] operands, then [block pair][1024 B] scales.  Operands of a pair: [chain j][block q]
// [row / 8][row % 8][8 halves] = operand A of the four products; scales: [128 rows][2] f32.  Rows past the end are zero.
__global__ void q8_operand_kernel(Q8Dev m, uint8_t *__restrict__ out, size_t total) {
    const int np = m.cols / 64;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x) {
        // one thread = 16 bytes: of a tile, np x 1024 pieces of operands, then np x 64 of scales
        const size_t tile = i / ((size_t)np * (QOP_UNIT / 16));
        const int k = (int)(i % ((size_t)np * (QOP_UNIT / 16))), row0 = (int)tile * TL_ROWS, op = np * 1024;
        const int pair = k < op ? k >> 10 : (k - op) >> 6, w = k < op ? k & 1023 : 1024 + ((k - op) & 63);
        uint4 v = make_uint4(0, 0, 0, 0);
        if (w < 1024) {
            const int j = w >> 8, q = (w >> 7) & 1, row = row0 + (w & 127);
            if (row < m.rows) {
                const int2 s = *reinterpret_cast<const int2 *>(m.data + q8_unit_off(row >> 4, pair, np) + (row & 15) * 64 + q * 32 + j * 8);
                __half h[8];
#pragma unroll
                for (int k = 0; k < 8; k++) h[k] = __int2half_rn((int)(int8_t)((k < 4 ? s.x : s.y) >> (8 * (k & 3))));
                v = *reinterpret_cast<const uint4 *>(h);
            }
        } else {
            const int row = row0 + (w - 1024) * 2;
            if (row < m.rows) {
                const float *s = reinterpret_cast<const float *>(m.data + q8_unit_off(row >> 4, pair, np) + Q8_UNIT_SCALES) + (row & 15) * 2;
                v = *reinterpret_cast<const uint4 *>(s);                 // rows row, row + 1 (storage is padded to 16 rows)
            }
        }
        *reinterpret_cast<uint4 *>(out + i * 16) = v;
    }
}

// int8 activations and their scales -> image (callers that hold a Q8 vector only)
template <int IMG>
__global__ void image_kernel(const int8_t *__restrict__ xq, int nblocks_row, int nblocks, uint8_t *__restrict__ img) {
    const int b = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (b >= nblocks) return;
    ti_emit_block<IMG>((int)xq[(size_t)b * 32 + lane], lane, b % nblocks_row, img + (size_t)(b / nblocks_row) * (nblocks_row / 2) * ti_pair(IMG));
}

// Per expert, the (token, slot) pairs routed to it, in ascending order: entry = token * topk + slot.  One CTA per
// expert, thread = token (a token routes to an expert at most once, so the order is the token order).
__global__ void __launch_bounds__(TL_MAXTOK) tile_route_kernel(const int32_t *__restrict__ top, int ntok, int topk, int *__restrict__ cnt, int *__restrict__ list) {
    __shared__ int warp_cnt[TL_MAXTOK / 32];
    const int e = blockIdx.x, t = threadIdx.x;
    pdl_wait();
    pdl_trigger();
    int slot = -1;
    if (t < ntok)
        for (int s = 0; s < topk; s++)
            if (top[t * 8 + s] == e) { slot = s; break; }
    const unsigned m = __ballot_sync(0xffffffffu, slot >= 0);
    if ((t & 31) == 0) warp_cnt[t >> 5] = __popc(m);
    __syncthreads();
    int before = __popc(m & ((1u << (t & 31)) - 1u));
    for (int w = 0; w < (t >> 5); w++) before += warp_cnt[w];
    if (slot >= 0) list[e * TL_MAXTOK + before] = t * topk + slot;
    if (t == TL_MAXTOK - 1) cnt[e] = before + (slot >= 0 ? 1 : 0);
}

// The 16-row units of an MXFP4 matrix as a tensor of 4-bit elements: [pair][unit][8 = (row half, lane chain)][128 = 8 rows x 16 codes], boxes of
// `units` units of one pair.  In shared memory 16 codes take 16 bytes (the upper 8 unused), the form tcgen05 reads 4-bit operands in.
cudaError_t mx_tensor_map(MxDev w, int units, CUtensorMap *map) {
    const tmap_encode_t encode = tmap_encode();
    if (!encode) return cudaErrorNotSupported;
    const cuuint64_t np = (cuuint64_t)w.blocks / 2;
    const cuuint64_t dims[4] = {128, 8, (cuuint64_t)w.rows / 16, np}, strides[3] = {64, np * MX_UNIT, MX_UNIT};
    const cuuint32_t box[4] = {128, 8, (cuuint32_t)units, 1}, ones[4] = {1, 1, 1, 1};
    const CUresult r = encode(map, CU_TENSOR_MAP_DATA_TYPE_16U4_ALIGN16B, 4, w.data, dims, strides, box, ones, CU_TENSOR_MAP_INTERLEAVE_NONE,
                              CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? cudaSuccess : cudaErrorInvalidValue;
}

// Tokens per CTA.  Experts: by the entries an expert has on average - few tokens keep more CTAs and copies in flight (up to 16 rows
// the launch is a stream of weights), many amortise the products' reads of operand A.  The lines lie where whole prompts of the 20b shape (4 of 32
// experts: an eighth of the rows each) cross, ms with 8 / 16 / 32 tokens per CTA: 64 rows 7.97 / 8.20 / 10.53, 72 rows 8.30 / 8.35 / 10.53,
// 80 rows 9.06 / 8.95 / 10.96, 128 rows 12.82 / 12.43 / 12.72, 136 rows 13.25 / 12.82 / 12.86, 144 rows 13.70 / 13.26 / 13.01.
// One matrix: a CTA per SM, so the fewest rounds of 148 CTAs, a round of 8, 16 or 32 tokens weighing 30, 33 and 47.  Its time follows the rows in it:
// 19, 21 and 23 to 35 us at 45 pairs, 24, 27 and 30 to 45 us at 64 pairs, 20, 21 and 25 to 32 us of the vocabulary's 11 rounds.  Over 8 to 512 rows
// of the 20b shape's three matrices the weights pick the fastest (12, 64 rows x 2880 outputs: 24 / 26 / 29 and 47 / 29 / 44 us; 33 rows x the
// vocabulary 526 us with 32 tokens, 664 with 16), or at most 8 % more where full rounds of 32 meet three of 16 (128 rows x 5120 outputs 64 against
// 59 us, 256 x 2880 87 against 80); weights of 18, 20 and 32, which these two would ask for, lose 26 % at 33 rows x the vocabulary.
template <int KIND>
cudaError_t tl_launch(TileArgs a, int tiles, int entries, int experts, bool pdl, cudaStream_t st) {
    const int avg = (entries + experts - 1) / experts, most = a.cnt ? a.ntok : entries;
    if (most < 1 || most > TL_MAXTOK) return cudaErrorInvalidValue;
    int nt = avg > 17 ? 32 : avg > 9 ? 16 : 8;
    if (!a.cnt) {
        auto cost = [&](int n, int round) { return ((tiles * ((entries + n - 1) / n) + 147) / 148) * round; };
        nt = 8;
        if (entries > 8 && cost(16, 33) < cost(nt, 30)) nt = 16;
        if (entries > 16 && cost(32, 47) < cost(nt, nt == 8 ? 30 : 33)) nt = 32;
    }
    static unsigned long long configured[3] = {0, 0, 0};      // one bit per device
    // at most one partly filled chunk per expert, and never more chunks than entries
    const int full_chunks = entries / nt, tasks = full_chunks + experts < entries ? full_chunks + experts : entries;
    const dim3 grid(tiles, tasks);
    cudaError_t ce;
    if (nt == 32) {
        if ((ce = smem_optin(tile_kernel<KIND, 32>, 220 * 1024, configured[0])) != cudaSuccess) return ce;
        return launch_k(tile_kernel<KIND, 32>, grid, dim3(32 * 16 + 128), tl_smem<KIND, 32>(a.np), st, pdl, a);
    }
    if (nt == 16) {
        if ((ce = smem_optin(tile_kernel<KIND, 16>, 220 * 1024, configured[1])) != cudaSuccess) return ce;
        return launch_k(tile_kernel<KIND, 16>, grid, dim3(16 * 16 + 128), tl_smem<KIND, 16>(a.np), st, pdl, a);
    }
    // up to three entries per expert on average: the variant that carries one or two pairs of tokens where that is all a CTA has (a kernel of its own:
    // the general loop loses 7 % beside the others).  gate | up and down of the 20b shape, us, without and with: 3 rows 36 + 29, 30 + 24; 9 rows
    // 73 + 50, 67 + 44; 16 rows 84 + 50, 76 + 49; 24 rows 93 + 57, 87 + 55; 30 rows 93 + 57, 94 + 59
    constexpr bool MX = KIND != TK_Q8;
    static unsigned long long configured_few = 0;
    if (MX && a.cnt && avg <= 3) {
        if ((ce = smem_optin(tile_kernel<KIND, 8, MX>, 220 * 1024, configured_few)) != cudaSuccess) return ce;
        return launch_k(tile_kernel<KIND, 8, MX>, grid, dim3(256), tl_smem<KIND, 8>(a.np), st, pdl, a);
    }
    if ((ce = smem_optin(tile_kernel<KIND, 8>, 220 * 1024, configured[2])) != cudaSuccess) return ce;
    return launch_k(tile_kernel<KIND, 8>, grid, dim3(256), tl_smem<KIND, 8>(a.np), st, pdl, a);
}

}  // namespace

size_t image_bytes(int rows, int cols, int kind) { return (size_t)rows * (cols / 64) * ti_pair(kind); }

void launch_image(const int8_t *xq, int rows, int cols, int kind, uint8_t *img, cudaStream_t st) {
    const int nb = cols / 32, n = rows * nb;
    if (n <= 0) return;
    if (kind == TI_HALF) image_kernel<TI_HALF><<<(n + 7) / 8, 256, 0, st>>>(xq, nb, n, img);
    else image_kernel<TI_PLANES><<<(n + 7) / 8, 256, 0, st>>>(xq, nb, n, img);
}

size_t q8_operand_bytes(int rows, int cols) { return (size_t)((rows + TL_ROWS - 1) / TL_ROWS) * (cols / 64) * QOP_UNIT; }

void launch_q8_operand_pack(Q8Dev m, uint8_t *out, cudaStream_t st) {
    const size_t total = q8_operand_bytes(m.rows, m.cols) / 16;
    if (total) q8_operand_kernel<<<148 * 8, 256, 0, st>>>(m, out, total);
}

cudaError_t launch_q8_tile(const uint8_t *op, int rows, int cols, const uint8_t *img, const float *xs, int ntok, const float *bias, float *y, int ldy,
                           int epi, DevState *state, bool pdl, cudaStream_t st) {
    if (ntok < 1 || ntok > BRRR_TILE_MAX || cols % 64 || cols < 64) return cudaErrorInvalidValue;
    TileArgs a{};
    a.wa = op; a.np = cols / 64; a.nrows = rows; a.ntok = ntok; a.src_div = 1; a.img = img; a.xs = xs; a.bias = bias; a.y = y; a.ldy = ldy; a.epi = epi;
    a.state = state;
    return tl_launch<TK_Q8>(a, (rows + TL_ROWS - 1) / TL_ROWS, ntok, 1, pdl, st);
}

cudaError_t launch_mx_tile(MxDev w, int row0, int nrows, const uint8_t *img, const float *xs, int ntok, float *y, int ldy, DevState *state, cudaStream_t st) {
    if ((w.blocks & 1) || w.blocks < 2) return cudaErrorInvalidValue;
    TileArgs a{};
    a.wa = w.data; a.np = w.blocks / 2; a.row0 = row0; a.nrows = nrows; a.ntok = ntok; a.src_div = 1; a.img = img; a.xs = xs; a.y = y; a.ldy = ldy;
    a.state = state;
    if (cudaError_t e = mx_tensor_map(w, 8, &a.ma)) return e;
    return tl_launch<TK_MX>(a, ((row0 & 15) + nrows + TL_ROWS - 1) / TL_ROWS, ntok, 1, false, st);
}

cudaError_t launch_mx_tile_glu(MxDev gate, MxDev up, int ne, int d, const int *cnt, const int *list, int ntok, int topk, const uint8_t *img, const float *xs,
                               const float *gate_b, const float *up_b, uint8_t *himg, float *hs, DevState *state, bool pdl, cudaStream_t st) {
    if ((gate.blocks & 1) || gate.blocks < 2 || d % 64 || ne > 256) return cudaErrorInvalidValue;
    TileArgs a{};
    a.wa = gate.data; a.wb = up.data; a.np = gate.blocks / 2; a.nrows = d; a.rows_per_expert = d; a.cnt = cnt; a.list = list; a.ne = ne; a.ntok = ntok;
    a.src_div = topk; a.img = img; a.xs = xs; a.bias = gate_b; a.bias_b = up_b; a.himg = himg; a.hs = hs; a.state = state;
    if (cudaError_t e = mx_tensor_map(gate, 4, &a.ma)) return e;
    if (cudaError_t e = mx_tensor_map(up, 4, &a.mb)) return e;
    return tl_launch<TK_GLU>(a, d / 64, ntok * topk, ne, pdl, st);
}

cudaError_t launch_mx_tile_down(MxDev down, int ne, int d, const int *cnt, const int *list, int ntok, int topk, const uint8_t *himg, const float *hs,
                                const float *bias, float *part, DevState *state, bool pdl, cudaStream_t st) {
    if ((down.blocks & 1) || down.blocks < 2 || ne > 256) return cudaErrorInvalidValue;
    TileArgs a{};
    a.wa = down.data; a.np = down.blocks / 2; a.nrows = d; a.rows_per_expert = d; a.cnt = cnt; a.list = list; a.ne = ne; a.ntok = ntok; a.src_div = 1;
    a.img = himg; a.xs = hs; a.bias = bias; a.y = part; a.ldy = d; a.state = state;
    if (cudaError_t e = mx_tensor_map(down, 8, &a.ma)) return e;
    return tl_launch<TK_MX>(a, (d + TL_ROWS - 1) / TL_ROWS, ntok * topk, ne, pdl, st);
}

cudaError_t launch_tile_route(const int32_t *top, int ntok, int topk, int ne, int *cnt, int *list, bool pdl, cudaStream_t st) {
    return launch_k(tile_route_kernel, dim3(ne), dim3(TL_MAXTOK), 0, st, pdl, top, ntok, topk, cnt, list);
}

}  // namespace brrr
