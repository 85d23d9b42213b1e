// K-quant matrices (Q4_K, Q6_K) against up to 512 token rows on the fifth-generation tensor cores, bit-identical to the
// one-token products (src/bin/engine_qwen2.rs:84-114, 164-200).
//
// A superblock's dot is an exact integer, so its order is free: D = A x B with A = 128 matrix rows (weights with their sub-block
// scale applied, exact halves), B = up to 32 token rows (the int8 quants as halves), f32 accumulators that hold integers below 2^24:
//   Q4_K  w = sc q <= 945.  Halves 0 and 1 of the superblock are two accumulators (each <= 15.4 M), a = D0 + D1 rounds as (float)int
//         does; the minima sum is a third product of K = 16 (mn against l, 64 mn against h of the image's 32-sums, <= 2.1 M).
//   Q6_K  sc = 16 sh + sl, so (q - 32) sh and (q - 32) sl are exact halves: two accumulators over the whole superblock
//         (<= 8.4 M and 15.6 M), a = fma(16, Dh, Dl).
// Then, per row and token, sum += (ys d) a - (ys dmin) mint in superblock order, every operation rounded as in q4k_row_dot.
//
// A CTA is persistent over (chunk of up to 32 tokens, 128 rows) tasks.  Warp roles: one lane brings raw superblocks of the 128 rows (TMA
// boxes) and the chunk's image (bulk copies: gathered with 16-byte copies per token and piece instead, they filled the load/store
// pipe and every wait and shared-memory read of the CTA with them: 2650 cycles per superblock); eight warps widen the weights - thread =
// row and half superblock - into tensor memory, where operand A is read from (128 rows x 256 halves would otherwise cross shared
// memory twice, 64 KB written and 64 KB read per superblock); one warp issues the products; eight warps - thread = row and 16 tokens -
// read the accumulators and carry the float chain.  Operand A and the accumulators are double-buffered.
#include "brrr_kernels.h"
#include "brrr_kqt.cuh"
#include "brrr_tc.cuh"
#include "brrr_tile.cuh"
#include "brrr_tmap.h"

namespace brrr {

namespace {

constexpr int KT_ROWS = 128;
constexpr int KT_RAW = 28672, KT_RAW_DEPTH = 4;                // raw superblocks of 128 rows (Q4_K 18432, Q6_K 28672 bytes)
constexpr int KT_B_DEPTH = 4;                                  // operand B blocks
constexpr int KT_WARPS = 18, KT_THREADS = KT_WARPS * 32;       // 8 epilogue, 8 widening, 1 issuing, 1 copies
constexpr uint32_t KT_COL_A = 192, KT_COL_MIN = 448;           // tensor memory columns: 2 x 3 x 32 accumulators, 2 halves x 2 x 64, 2 x 8
constexpr size_t KT_SMEM = (size_t)KT_RAW * KT_RAW_DEPTH + (size_t)KIMG_BLOCK * KT_B_DEPTH + 1024;

struct alignas(64) KqtArgs {
    KqtMat m[3];             // stacked matrices of equal width
    float *y[3];             // outputs [entry or position][ldy] (+ row of the matrix)
    int ldy[3];
    int tile_end[3];         // running number of 128-row tiles of one expert
    int tiles, nsb;
    const KqPlan *plan;      // nullptr: one matrix, rows 0 .. ntok - 1
    int ntok, resid, by_entry;      // by_entry: outputs go to the plan's entries, else to positions 32 chunk + i
    const uint8_t *img;
    const float *ys;
    DevState *state;
};

__device__ __forceinline__ void kt_box(uint32_t dst, const CUtensorMap *map, int x, int row, uint64_t *bar) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(dst), "l"(map), "r"(x), "r"(row),
                 "r"(smem_u32(bar))
                 : "memory");
}
// (issue: the elected lane's predicate, see tl_commit_if)
__device__ __forceinline__ void kt_mma(uint32_t issue, uint32_t d, uint32_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
    asm volatile("{\n\t.reg .pred p, e;\n\tsetp.ne.b32 p, %4, 0;\n\tsetp.ne.b32 e, %6, 0;\n\t"
                 "@e tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, {%5, %5, %5, %5}, p;\n\t}" ::"r"(d), "r"(a), "l"(b), "r"(idesc), "r"(accumulate), "r"(0u), "r"(issue)
                 : "memory");
}
__device__ __forceinline__ void kt_st16(uint32_t t, const uint32_t (&v)[16]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};" ::"r"(t), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]),
                 "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15])
                 : "memory");
}
__device__ __forceinline__ void kt_st8(uint32_t t, const uint32_t (&v)[8]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"r"(t), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]),
                 "r"(v[7])
                 : "memory");
}
__device__ __forceinline__ f32x2 kt_add2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
// Products that feed an addition are formed one by one: a packed multiply followed by a packed add came out fused (one rounding),
// whatever the rounding modifiers and -fmad=false say; the scalar forms round twice.
__device__ __forceinline__ f32x2 kt_mul2_apart(f32x2 a, f32x2 b) {
    float a0, a1, b0, b1;
    tl_unpack2(a, a0, a1);
    tl_unpack2(b, b0, b1);
    return tl_pack2(__float_as_uint(__fmul_rn(a0, b0)), __float_as_uint(__fmul_rn(a1, b1)));
}
__device__ __forceinline__ f32x2 kt_sub2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ uint32_t lds32(uint32_t addr) {
    uint32_t r;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(r) : "r"(addr));
    return r;
}
// halves: pairs in a 32-bit word
__device__ __forceinline__ uint32_t h2fma(uint32_t a, uint32_t b, uint32_t c) {
    uint32_t r;
    asm("fma.rn.f16x2 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(c));
    return r;
}
__device__ __forceinline__ uint32_t h2mul(uint32_t a, uint32_t b) {
    uint32_t r;
    asm("mul.rn.f16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    return r;
}
__device__ __forceinline__ uint32_t h2sub(uint32_t a, uint32_t b) {
    uint32_t r;
    asm("sub.rn.f16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    return r;
}
constexpr uint32_t H2_1024 = 0x64006400u, H2_1032 = 0x64086408u, H2_SIXTEENTH = 0x2C002C00u, H2_64 = 0x54005400u, H2_M1024 = 0xE400E400u, H2_M64 = 0xD400D400u,
                   H2_M1056 = 0xE420E420u;
// byte j of w (below 64) as a pair of equal halves 1024 + byte
__device__ __forceinline__ uint32_t h2_byte(uint32_t w, int j) { return __byte_perm(w, 0x64u, 0x4040u | (uint32_t)j | ((uint32_t)j << 8)); }

// one task: chunk of tokens, 128-row tile of the stack
struct KtTask { int chunk, e, n, mi, row; };      // row: of the expert's matrix mi

__global__ void __launch_bounds__(KT_THREADS, 1) kqt_kernel(const __grid_constant__ KqtArgs a) {
    extern __shared__ unsigned char ksm_[];
    unsigned char *raw = ksm_ + ((1024u - (smem_u32(ksm_) & 1023u)) & 1023u);          // swizzled copies want 1024-byte alignment
    unsigned char *bsm = raw + KT_RAW * KT_RAW_DEPTH;
    // rfull / rempty: raw slot; bfull: B slot; afull: a half's operand (two stages); half0[n & 3]: the first half of superblock n has been
    // read; done[n & 3]: all of it, its block of B, and the accumulators are complete; dempty: they have been read
    __shared__ __align__(8) uint64_t rfull[KT_RAW_DEPTH], rempty[KT_RAW_DEPTH], bfull[KT_B_DEPTH], afull[2][2], half0[4], done[4], dempty[2];
    __shared__ float2 drow[4][KT_ROWS];              // d, dmin of the rows; written once the accumulators of four superblocks before have been read
    __shared__ __align__(16) float ysr[8][KT_NT];    // activation scales, eight superblocks deep
    __shared__ short chunk_e[KT_MAXCHUNK], chunk_n[KT_MAXCHUNK];
    __shared__ uint32_t tmem_sh;
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31, nsb = a.nsb;
    if (tid == 0) {
        for (int i = 0; i < KT_RAW_DEPTH; i++) { mbar_init(&rfull[i], 1); mbar_init(&rempty[i], 8); }
        for (int i = 0; i < KT_B_DEPTH; i++) mbar_init(&bfull[i], 1);
        for (int i = 0; i < 4; i++) { mbar_init(&half0[i], 1); mbar_init(&done[i], 2); }
        for (int i = 0; i < 2; i++) { mbar_init(&afull[0][i], 4); mbar_init(&afull[1][i], 4); mbar_init(&dempty[i], 8); }
        mbar_fence_init();
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_sh)), "r"(512u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    int nchunk = (a.ntok + KT_NT - 1) / KT_NT;
    if (a.plan) {                // the chunks depend on the routing; a single matrix's weights do not
        pdl_wait();
        nchunk = min(a.plan->nchunk, KT_MAXCHUNK);
        for (int i = tid; i < nchunk; i += KT_THREADS) { chunk_e[i] = (short)a.plan->e[i]; chunk_n[i] = (short)a.plan->n[i]; }
    }
    tl_fence_before();
    __syncthreads();
    tl_fence_after();
    pdl_trigger();
    const uint32_t tmem = __shfl_sync(0xffffffffu, tmem_sh, 0);
    const int ntask = nchunk * a.tiles;
    TlWaiter wait{a.state ? &a.state->err : nullptr, a.state && *reinterpret_cast<volatile uint32_t *>(&a.state->err) != 0u};
    auto task = [&](int t) {
        KtTask k;
        k.chunk = t / a.tiles;
        const int tile = t - k.chunk * a.tiles;
        k.e = a.plan ? chunk_e[k.chunk] : 0;
        k.n = a.plan ? chunk_n[k.chunk] : min(KT_NT, a.ntok - k.chunk * KT_NT);
        k.mi = 0;
        while (tile >= a.tile_end[k.mi]) k.mi++;
        k.row = (tile - (k.mi ? a.tile_end[k.mi - 1] : 0)) * KT_ROWS;
        return k;
    };
    // parity with which superblock n - back released its stages
    auto released = [](int n, int back) { return (uint32_t)((n - back) >> 2) & 1u; };
    const uint32_t raw0 = smem_u32(raw), b0 = smem_u32(bsm);

    if (warp == 17) {
        // ---------------- copies: raw superblocks of the rows, the chunk's block of operand B, its scales
        if (lane == 0) {
            int n = 0;
            bool waited = a.plan != nullptr;
            for (int t = blockIdx.x; t < ntask; t += gridDim.x) {
                const KtTask k = task(t);
                const KqtMat &m = a.m[k.mi];
                const int row = k.e * (a.tile_end[k.mi] - (k.mi ? a.tile_end[k.mi - 1] : 0)) * KT_ROWS + k.row;
                const uint32_t bytes = (m.type == 12 ? 34u : 32u) * kq_cap(k.n) * 16;
                auto brings_b = [&](int sb, int nn) {
                    const int slot = nn % KT_B_DEPTH;
                    if (nn >= KT_B_DEPTH) wait(&done[(nn - KT_B_DEPTH) & 3], released(nn, KT_B_DEPTH));
                    const size_t blk = (size_t)k.chunk * nsb + sb;
                    mbar_expect_tx(&bfull[slot], bytes + KT_NT * 4);
                    bulk_g2s(bsm + slot * KIMG_BLOCK, a.img + blk * KIMG_BLOCK, bytes, &bfull[slot]);
                    bulk_g2s(&ysr[nn & 7][0], a.ys + blk * KT_NT, KT_NT * 4, &bfull[slot]);
                };
                const int first = n;
                int held = 0;                          // blocks of B not requested yet: the kernel before may still be writing the image
                for (int sb = 0; sb < nsb; sb++, n++) {
                    const int slot = n % KT_RAW_DEPTH;
                    if (!waited && n >= min(KT_RAW_DEPTH, nsb)) {
                        pdl_wait();
                        waited = true;
                        for (int h = 0; h < held; h++) brings_b(h, first + h);
                        held = 0;
                    }
                    if (n >= KT_RAW_DEPTH) wait(&rempty[slot], ((n / KT_RAW_DEPTH) & 1) ^ 1);
                    const uint32_t dst = raw0 + slot * KT_RAW;
                    if (m.type == 12) {
                        mbar_expect_tx(&rfull[slot], KT_ROWS * 144);
                        kt_box(dst, &m.map[0], sb * 144, row, &rfull[slot]);
                    } else {
                        mbar_expect_tx(&rfull[slot], KT_RAW);
                        kt_box(dst, &m.map[0], sb * 128, row, &rfull[slot]);
                        kt_box(dst + 16384, &m.map[1], nsb * 128 + sb * 64, row, &rfull[slot]);
                        kt_box(dst + 24576, &m.map[2], nsb * 192 + sb * 16, row, &rfull[slot]);
                        kt_box(dst + 26624, &m.map[2], nsb * 208 + (sb & ~7) * 2, row, &rfull[slot]);
                    }
                    if (waited) brings_b(sb, n);
                    else held++;
                }
                if (!waited) {                         // nsb <= KT_RAW_DEPTH
                    pdl_wait();
                    waited = true;
                    for (int h = 0; h < held; h++) brings_b(h, first + h);
                }
            }
        }
    } else if (warp == 16) {
        // ---------------- products (the whole warp walks the loop, an elected lane issues)
        const uint32_t issue = elect_one() ? 1u : 0u;
        int n = 0, ca = 0;
        for (int t = blockIdx.x; t < ntask; t += gridDim.x) {
            const KtTask k = task(t);
            const bool q4 = a.m[k.mi].type == 12;
            const int cap = kq_cap(k.n);
            const uint32_t idesc = (1u << 4) | ((uint32_t)(k.n > 16 ? 4 : 2) << 17) | ((KT_ROWS >> 4) << 24);      // f32 += f16 x f16, N = 16 or 32
            const uint64_t db0 = tl_smem_desc(bsm, cap * 16, cap == 8 ? 0 : 128);      // room for eight: both groups of eight columns read them
            for (int sb = 0; sb < nsb; sb++, n++) {
                const int slot = n % KT_B_DEPTH, buf = n & 1;
                wait(&bfull[slot], (n / KT_B_DEPTH) & 1);
                wait(&dempty[buf], ((n >> 1) & 1) ^ 1);
                const uint64_t db = db0 + (uint64_t)(slot * (KIMG_BLOCK / 16));
                const uint32_t d = tmem + buf * 96;
                if (q4) {
                    const int ab = ca & 1;
#pragma unroll
                    for (int g = 0; g < 2; g++) {
                        wait(&afull[g][ab], (ca >> 1) & 1);
                        tl_fence_after();
#pragma unroll
                        for (int s = 0; s < 8; s++) kt_mma(issue, d + g * 32, tmem + KT_COL_A + (g * 2 + ab) * 64 + s * 8, db + (g * 8 + s) * 2 * cap, idesc, s > 0);
                        if (g == 1) kt_mma(issue, d + 64, tmem + KT_COL_MIN + ab * 8, db + 32 * cap, idesc, 0);
                        tl_commit_if(issue, g == 0 ? &half0[n & 3] : &done[n & 3]);
                        if (g == 1) mbar_arrive_if(issue, &done[n & 3]);      // orders drow and ysr, seen through afull and bfull, before the readers
                        __syncwarp();
                    }
                    ca++;
                } else {
#pragma unroll
                    for (int g = 0; g < 2; g++) {
#pragma unroll
                        for (int dig = 0; dig < 2; dig++) wait(&afull[g][(ca + dig) & 1], ((ca + dig) >> 1) & 1);
                        tl_fence_after();
#pragma unroll
                        for (int dig = 0; dig < 2; dig++)
#pragma unroll
                            for (int s = 0; s < 8; s++)
                                kt_mma(issue, d + dig * 32, tmem + KT_COL_A + (g * 2 + ((ca + dig) & 1)) * 64 + s * 8, db + (g * 8 + s) * 2 * cap, idesc, g > 0 || s > 0);
                        tl_commit_if(issue, g == 0 ? &half0[n & 3] : &done[n & 3]);
                        if (g == 1) mbar_arrive_if(issue, &done[n & 3]);
                        __syncwarp();
                    }
                    ca += 2;
                }
            }
        }
    } else if (warp >= 8) {
        // ---------------- widening: thread = row m, half g of the superblock
        const int g = (warp - 8) >> 2, m = (warp & 3) * 32 + lane;
        const uint32_t arow = tmem + ((uint32_t)((warp & 3) * 32) << 16);
        uint64_t *const rel = g == 0 ? half0 : done;
        int n = 0, ca = 0;
        bool both = false;                             // the superblock before took both stages of this half (Q6_K)
        for (int t = blockIdx.x; t < ntask; t += gridDim.x) {
            const KtTask k = task(t);
            const bool q4 = a.m[k.mi].type == 12;
            for (int sb = 0; sb < nsb; sb++, n++) {
                const int slot = n % KT_RAW_DEPTH;
                const uint32_t src = raw0 + slot * KT_RAW;
                wait(&rfull[slot], (n / KT_RAW_DEPTH) & 1);
                if (q4) {
                    const uint4 h = lds128(src + m * 144);
                    uint32_t w[16];
#pragma unroll
                    for (int i = 0; i < 4; i++) {
                        const uint4 v = lds128(src + m * 144 + 16 + g * 64 + i * 16);
                        w[4 * i] = v.x; w[4 * i + 1] = v.y; w[4 * i + 2] = v.z; w[4 * i + 3] = v.w;
                    }
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&rempty[slot]);
                    const int ab = ca & 1;
                    const int back = both ? 1 : 2;
                    if (n >= back) wait(&rel[(n - back) & 3], released(n, back));
                    both = false;
                    ca++;
                    if (g == 0) drow[n & 3][m] = make_float2(half_bits_to_f32(h.x & 0xffffu), half_bits_to_f32(h.x >> 16));
                    tl_fence_after();
                    const uint32_t dst = arow + KT_COL_A + (g * 2 + ab) * 64;
                    // 6-bit scales of sub-blocks 4g .. 4g + 3
                    const uint32_t sc4 = g == 0 ? h.y & 0x3F3F3F3Fu : (h.w & 0x0F0F0F0Fu) | ((h.y >> 2) & 0x30303030u);
#pragma unroll
                    for (int c = 0; c < 2; c++) {      // 32-byte chunk: low nibbles = sub-block 2c, high nibbles = 2c + 1 of the half
                        const uint32_t sl = h2sub(h2_byte(sc4, 2 * c), H2_1024), sh = h2sub(h2_byte(sc4, 2 * c + 1), H2_1024);
                        const uint32_t sh16 = h2mul(sh, H2_SIXTEENTH), cl = h2mul(sl, H2_M1024), chh = h2mul(sh, H2_M64);
                        uint32_t lo[16], hi[16];
#pragma unroll
                        for (int i = 0; i < 8; i++) {
                            const uint32_t v = w[8 * c + i], v8 = v >> 8;
                            lo[2 * i] = h2fma((v & 0x000F000Fu) | H2_1024, sl, cl);              // (1024 + q) sc - 1024 sc
                            lo[2 * i + 1] = h2fma((v8 & 0x000F000Fu) | H2_1024, sl, cl);
                            hi[2 * i] = h2fma((v & 0x00F000F0u) | H2_1024, sh16, chh);           // (1024 + 16 q) sc / 16 - 64 sc
                            hi[2 * i + 1] = h2fma((v8 & 0x00F000F0u) | H2_1024, sh16, chh);
                        }
                        kt_st16(dst + c * 32, lo);
                        kt_st16(dst + c * 32 + 16, hi);
                    }
                    if (g == 1) {
                        const uint32_t mlo = h.z & 0x3F3F3F3Fu, mhi = ((h.w >> 4) & 0x0F0F0F0Fu) | ((h.z >> 2) & 0x30303030u);
                        uint32_t mn[8];
#pragma unroll
                        for (int i = 0; i < 4; i++) {
                            const uint32_t s = i < 2 ? mlo : mhi;
                            mn[i] = h2sub(__byte_perm(s, 0x64u, (i & 1) ? 0x4342u : 0x4140u), H2_1024);
                            mn[4 + i] = h2mul(mn[i], H2_64);
                        }
                        kt_st8(arow + KT_COL_MIN + ab * 8, mn);
                    }
                    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                    tl_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&afull[g][ab]);
                } else {
                    uint32_t qa[8], qb[8], qh[8];
#pragma unroll
                    for (int i = 0; i < 2; i++) {      // ql: 128-byte rows, 16-byte chunk c of row m at c ^ (m & 7); qh: 64-byte rows, c ^ (m >> 1 & 3)
                        const uint4 va = lds128(src + m * 128 + (((4 * g + i) ^ (m & 7)) << 4)), vb = lds128(src + m * 128 + (((4 * g + 2 + i) ^ (m & 7)) << 4));
                        const uint4 vh = lds128(src + 16384 + m * 64 + (((2 * g + i) ^ ((m >> 1) & 3)) << 4));
                        qa[4 * i] = va.x; qa[4 * i + 1] = va.y; qa[4 * i + 2] = va.z; qa[4 * i + 3] = va.w;
                        qb[4 * i] = vb.x; qb[4 * i + 1] = vb.y; qb[4 * i + 2] = vb.z; qb[4 * i + 3] = vb.w;
                        qh[4 * i] = vh.x; qh[4 * i + 1] = vh.y; qh[4 * i + 2] = vh.z; qh[4 * i + 3] = vh.w;
                    }
                    const uint2 scw = lds64(src + 24576 + m * 16 + g * 8);
                    const uint32_t dw = lds32(src + 26624 + m * 16 + (sb & 6) * 2);
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&rempty[slot]);
                    const int a0 = ca & 1, a1 = a0 ^ 1;
                    if (n >= 1) wait(&rel[(n - 1) & 3], released(n, 1));
                    both = true;
                    ca += 2;
                    if (g == 0) drow[n & 3][m] = make_float2(half_bits_to_f32((sb & 1) ? dw >> 16 : dw & 0xffffu), 0.0f);
                    tl_fence_after();
                    const uint32_t d0 = arow + KT_COL_A + (g * 2 + a0) * 64, d1 = arow + KT_COL_A + (g * 2 + a1) * 64;
#pragma unroll
                    for (int qd = 0; qd < 4; qd++) {   // values 32 qd .. + 31 of the half
                        uint32_t hi[16], lo[16];
#pragma unroll
                        for (int s = 0; s < 2; s++) {  // sixteen values share a scale
                            const uint32_t word = qd < 2 ? scw.x : scw.y;
                            const int byte = (qd & 1) * 2 + s;
                            const uint32_t fh = h2sub(h2_byte(((word ^ 0x80808080u) >> 4) & 0x0F0F0F0Fu, byte), H2_1032), fl = h2sub(h2_byte(word & 0x0F0F0F0Fu, byte), H2_1024);
                            const uint32_t ch = h2mul(fh, H2_M1056), cl = h2mul(fl, H2_M1056);
#pragma unroll
                            for (int i = 4 * s; i < 4 * s + 4; i++) {
                                const uint32_t src4 = (qd & 1) ? qb[i] : qa[i], hv = qh[i];
                                const uint32_t x = (qd & 2) ? src4 >> 4 : src4, y = qd == 0 ? hv << 4 : qd == 1 ? hv << 2 : qd == 2 ? hv : hv >> 2;
                                const uint32_t v0 = (x & 0x000F000Fu) | (y & 0x00300030u) | H2_1024;
                                const uint32_t v1 = ((x >> 8) & 0x000F000Fu) | ((y >> 8) & 0x00300030u) | H2_1024;
                                hi[2 * i] = h2fma(v0, fh, ch);                                   // (1024 + q) s - 1056 s
                                hi[2 * i + 1] = h2fma(v1, fh, ch);
                                lo[2 * i] = h2fma(v0, fl, cl);
                                lo[2 * i + 1] = h2fma(v1, fl, cl);
                            }
                        }
                        kt_st16(d0 + qd * 16, hi);
                        kt_st16(d1 + qd * 16, lo);
                    }
                    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                    tl_fence_before();
                    __syncwarp();
                    if (lane == 0) { mbar_arrive(&afull[g][a0]); mbar_arrive(&afull[g][a1]); }
                }
            }
        }
    } else {
        // ---------------- accumulators and the float chain: thread = row m, tokens 16 wg .. + 15
        if (!a.plan) pdl_wait();
        const int wg = warp >> 2, m = (warp & 3) * 32 + lane;
        const uint32_t lane_addr = tmem + ((uint32_t)((warp & 3) * 32) << 16) + wg * 16;
        int n = 0;
        for (int t = blockIdx.x; t < ntask; t += gridDim.x) {
            const KtTask k = task(t);
            const bool q4 = a.m[k.mi].type == 12, live = wg * 16 < k.n;
            const int ti = wg * 16 + (lane & 15);
            const int ent = ti < k.n ? (a.by_entry ? a.plan->ent[k.chunk * KT_NT + ti] : k.chunk * KT_NT + ti) : 0;
            f32x2 acc[8];
#pragma unroll
            for (int i = 0; i < 8; i++) acc[i] = 0ull;
            for (int sb = 0; sb < nsb; sb++, n++) {
                const int buf = n & 1;
                wait(&done[n & 3], (n >> 2) & 1);
                if (!live) {
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&dempty[buf]);
                    continue;
                }
                tl_fence_after();
                f32x2 p[8], q[8], r[8];
                tl_ld16x2(lane_addr + buf * 96, lane_addr + buf * 96 + 32, p, q);
                if (q4) tl_ld8x2(lane_addr + buf * 96 + 64, lane_addr + buf * 96 + 72, *reinterpret_cast<f32x2(*)[4]>(&r[0]), *reinterpret_cast<f32x2(*)[4]>(&r[4]));
                const float2 dd = drow[n & 3][m];
                f32x2 ys[8];
                const uint32_t ya = smem_u32(&ysr[n & 7][wg * 16]);
#pragma unroll
                for (int i = 0; i < 4; i++) lds_pairs(ya + i * 16, ys[2 * i], ys[2 * i + 1]);
                tl_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&dempty[buf]);
                const f32x2 d2 = tl_pack2(__float_as_uint(dd.x), __float_as_uint(dd.x)), m2 = tl_pack2(__float_as_uint(dd.y), __float_as_uint(dd.y));
                if (q4) {
#pragma unroll
                    for (int i = 0; i < 8; i++) {
                        const f32x2 pos = kt_mul2_apart(tl_mul2(ys[i], d2), kt_add2(p[i], q[i])), neg = kt_mul2_apart(tl_mul2(ys[i], m2), r[i]);
                        acc[i] = kt_add2(acc[i], kt_sub2(pos, neg));
                    }
                } else {
                    const f32x2 sixteen = tl_pack2(0x41800000u, 0x41800000u);
#pragma unroll
                    for (int i = 0; i < 8; i++) acc[i] = kt_add2(acc[i], kt_mul2_apart(tl_mul2(ys[i], d2), tl_fma2(sixteen, p[i], q[i])));
                }
            }
            if (!live) continue;
            float *y = a.y[k.mi] + k.row + m;
            const int ldy = a.ldy[k.mi];
            float v[16], old[16];
#pragma unroll
            for (int i = 0; i < 8; i++) tl_unpack2(acc[i], v[2 * i], v[2 * i + 1]);
            size_t off[16];
#pragma unroll
            for (int i = 0; i < 16; i++) off[i] = (size_t)__shfl_sync(0xffffffffu, ent, i) * ldy;
            if (a.resid) {
#pragma unroll
                for (int i = 0; i < 16; i++) old[i] = wg * 16 + i < k.n ? y[off[i]] : 0.0f;
#pragma unroll
                for (int i = 0; i < 16; i++) v[i] = __fadd_rn(old[i], v[i]);
            }
#pragma unroll
            for (int i = 0; i < 16; i++)
                if (wg * 16 + i < k.n) y[off[i]] = v[i];
        }
    }
    tl_fence_before();
    __syncthreads();
    if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
}

}  // namespace

cudaError_t qw_cache(float *kc, float *vc, int nkv, QwCache *out) {
    const tmap_encode_t encode = tmap_encode();
    if (!encode) return cudaErrorNotSupported;
    const cuuint64_t dims[2] = {128, (cuuint64_t)nkv * BRRR_MAXSEQ}, strides[1] = {512};
    const cuuint32_t box[2] = {32, 64}, ones[2] = {1, 1};
    for (int i = 0; i < 2; i++)
        if (encode(i ? &out->vm : &out->km, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, i ? vc : kc, dims, strides, box, ones, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                   CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
            return cudaErrorInvalidValue;
    out->k = kc; out->v = vc;
    return cudaSuccess;
}

cudaError_t kqt_matrix(const KMatDev &m, size_t rows_total, KqtMat *out) {
    const tmap_encode_t encode = tmap_encode();
    if (!encode) return cudaErrorNotSupported;
    if (m.rows % KT_ROWS || m.cols % 256 || (m.type != 12 && !(m.type == 14 && m.planes)) || rows_total % KT_ROWS) return cudaErrorInvalidValue;
    const cuuint64_t dims[2] = {(cuuint64_t)m.bpr(), (cuuint64_t)rows_total}, strides[1] = {(cuuint64_t)m.bpr()};
    const cuuint32_t ones[2] = {1, 1}, width4[1] = {144}, width6[3] = {128, 64, 16};
    const CUtensorMapSwizzle sw[3] = {CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_SWIZZLE_NONE};
    const int n = m.type == 12 ? 1 : 3;
    for (int i = 0; i < n; i++) {
        const cuuint32_t box[2] = {m.type == 12 ? width4[0] : width6[i], KT_ROWS};
        if (encode(&out->map[i], CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, (void *)m.p, dims, strides, box, ones, CU_TENSOR_MAP_INTERLEAVE_NONE,
                   m.type == 12 ? CU_TENSOR_MAP_SWIZZLE_NONE : sw[i], CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
            return cudaErrorInvalidValue;
    }
    out->type = m.type; out->rows = m.rows; out->cols = m.cols;
    return cudaSuccess;
}

// Tasks are known on the host up to the number of chunks an expert's tokens fall into: at most one partly filled per expert, and never
// more than entries.
int kqt_max_chunks(int entries, int ne) { return entries / KT_NT + ne < entries ? entries / KT_NT + ne : entries; }

cudaError_t launch_kqt(const KqtMat *const *mats, float *const *ys_out, const int *ldy, int nmat, int rows_per_expert, const KqPlan *plan, int ne, int ntok, int topk,
                       bool by_entry, const uint8_t *img, const float *ys, bool resid, DevState *state, bool pdl, cudaStream_t st) {
    const int chunks = plan ? kqt_max_chunks(ntok * topk, ne) : (ntok + KT_NT - 1) / KT_NT;
    if (nmat < 1 || nmat > 3 || ntok < 1 || ntok > BRRR_TILE_MAX || chunks > KT_MAXCHUNK || ne > 256) return cudaErrorInvalidValue;
    KqtArgs a{};
    int tiles = 0;
    for (int i = 0; i < nmat; i++) {
        const int rows = plan ? rows_per_expert : mats[i]->rows;
        if (mats[i]->cols != mats[0]->cols || rows % KT_ROWS) return cudaErrorInvalidValue;
        a.m[i] = *mats[i]; a.y[i] = ys_out[i]; a.ldy[i] = ldy[i];
        a.tile_end[i] = tiles += rows / KT_ROWS;
    }
    a.tiles = tiles; a.nsb = mats[0]->cols / 256; a.plan = plan; a.ntok = ntok; a.resid = resid; a.by_entry = plan && by_entry;
    a.img = img; a.ys = ys; a.state = state;
    static unsigned long long configured = 0;      // one bit per device
    cudaError_t e = smem_optin(kqt_kernel, (int)KT_SMEM, configured);
    if (e != cudaSuccess) return e;
    const int tasks = chunks * tiles;
    return launch_k(kqt_kernel, dim3(tasks < 148 ? tasks : 148), dim3(KT_THREADS), KT_SMEM, st, pdl, a);
}

}  // namespace brrr
