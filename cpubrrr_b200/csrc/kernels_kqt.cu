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
// A CTA is persistent over (expert, up to 32 of its tokens, 128 rows) tasks.  Warp roles: one lane brings raw superblocks of the 128
// rows (TMA boxes, 4 deep); eight warps widen them - thread = row and half superblock - into tensor memory, where operand A is read
// from (128 rows x 256 halves would otherwise cross shared memory twice: 64 KB written and 64 KB read per superblock, the bound of the
// layout with A in shared memory); two warps gather the tokens' images into operand B; one issues the products; eight warps - thread =
// row and 16 tokens - read the accumulators and carry the float chain.  Operand A and the accumulators are double-buffered.
#include "brrr_kernels.h"
#include "brrr_kqt.cuh"
#include "brrr_tc.cuh"
#include "brrr_tile.cuh"

namespace brrr {

namespace {

constexpr int KT_ROWS = 128, KT_NT = 32;
constexpr int KT_RAW = 28672, KT_RAW_DEPTH = 4;                // raw superblocks of 128 rows (Q4_K 18432, Q6_K 28672 bytes)
constexpr int KT_B = 34 * KT_NT * 16, KT_B_DEPTH = 4;          // operand B of a superblock: [16-byte chunk][token] (the last two: minima)
constexpr int KT_WARPS = 20, KT_THREADS = KT_WARPS * 32;       // 8 epilogue, 8 widening, 1 issuing, 1 raw copies, 2 images
constexpr int KT_MAXCHUNK = 512;                               // chunks of tokens: entries / 32 + experts at most
constexpr uint32_t KT_COL_A = 192, KT_COL_MIN = 448;           // tensor memory columns: 2 x 3 x 32 accumulators, 2 halves x 2 x 64, 2 x 8
constexpr size_t KT_SMEM = (size_t)KT_RAW * KT_RAW_DEPTH + (size_t)KT_B * KT_B_DEPTH + 1024;

struct alignas(64) KqtArgs {
    KqtMat m[3];             // stacked matrices of equal width
    float *y[3];             // outputs [entry][ldy] (+ row of the matrix)
    int ldy[3];
    int tile_end[3];         // running number of 128-row tiles of one expert
    int nmat, tiles, nsb;
    const int *cnt, *list;   // entries per expert, [ne][512] entry ids; cnt == nullptr: one matrix, entries 0 .. ntok - 1
    int ne, ntok, src_div, resid;
    const uint8_t *img;      // images [entry / src_div][nsb * 544]
    const float *ys;         // scales [entry / src_div][nsb]
    DevState *state;
};

__device__ __forceinline__ void kt_box(uint32_t dst, const CUtensorMap *map, int x, int row, uint64_t *bar) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(dst), "l"(map), "r"(x), "r"(row),
                 "r"(smem_u32(bar))
                 : "memory");
}
__device__ __forceinline__ void kt_mma(uint32_t d, uint32_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                 "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, {%5, %5, %5, %5}, p;\n\t}" ::"r"(d), "r"(a), "l"(b), "r"(idesc), "r"(accumulate), "r"(0u)
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
__device__ __forceinline__ uint4 lds128(uint32_t addr) {
    uint4 r;
    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w) : "r"(addr));
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

// one task: expert, first entry and number of entries of its chunk, 128-row tile of the stack
struct KtTask { int e, first, n, mi, row; };      // row: of the expert's matrix mi

__global__ void __launch_bounds__(KT_THREADS, 1) kqt_kernel(const __grid_constant__ KqtArgs a) {
    extern __shared__ unsigned char ksm_[];
    unsigned char *raw = ksm_ + ((1024u - (smem_u32(ksm_) & 1023u)) & 1023u);          // swizzled copies want 1024-byte alignment
    unsigned char *bsm = raw + KT_RAW * KT_RAW_DEPTH;
    __shared__ __align__(8) uint64_t rfull[KT_RAW_DEPTH], rempty[KT_RAW_DEPTH], bfull[KT_B_DEPTH], bempty[KT_B_DEPTH], afull[2][2], aempty[2][2], dfull[2], dempty[2];
    __shared__ float2 drow[4][KT_ROWS];              // d, dmin of the rows, four superblocks deep
    __shared__ __align__(16) float ysr[8][KT_NT];    // activation scales, eight superblocks deep
    __shared__ int chunk_e[KT_MAXCHUNK], chunk_fn[KT_MAXCHUNK], nchunk_sh;      // fn: first | entries << 16
    __shared__ uint32_t tmem_sh;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, nsb = a.nsb;
    if (tid == 0) {
        for (int i = 0; i < KT_RAW_DEPTH; i++) { mbar_init(&rfull[i], 1); mbar_init(&rempty[i], 8); }
        for (int i = 0; i < KT_B_DEPTH; i++) { mbar_init(&bfull[i], 64); mbar_init(&bempty[i], 1); }
        for (int i = 0; i < 2; i++) {
            mbar_init(&afull[0][i], 4); mbar_init(&afull[1][i], 4); mbar_init(&aempty[0][i], 1); mbar_init(&aempty[1][i], 1);
            mbar_init(&dfull[i], 2); mbar_init(&dempty[i], 8);
        }
        mbar_fence_init();
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_sh)), "r"(512u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (a.cnt) pdl_wait();       // the chunks depend on the routing; a single matrix's weights do not
    if (warp == 0) {
        // chunks: experts in order, ceil(entries / 32) each, of equal size in whole groups of sixteen
        const int per = a.cnt ? (a.ne + 31) / 32 : 1, e0 = lane * per;
        int c[8], mine = 0;
#pragma unroll
        for (int i = 0; i < 8; i++) {
            c[i] = 0;
            if (i < per) c[i] = a.cnt ? (e0 + i < a.ne ? a.cnt[e0 + i] : 0) : (lane == 0 ? a.ntok : 0);
            mine += (c[i] + KT_NT - 1) / KT_NT;
        }
        int incl = mine;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) { const int v = __shfl_up_sync(0xffffffffu, incl, o); if (lane >= o) incl += v; }
        int at = incl - mine;
#pragma unroll
        for (int i = 0; i < 8; i++) {
            const int n = (c[i] + KT_NT - 1) / KT_NT, step = n ? ((c[i] + n - 1) / n + 15) & ~15 : 0;
            for (int k = 0; k < n; k++, at++)
                if (at < KT_MAXCHUNK) { chunk_e[at] = e0 + i; chunk_fn[at] = (k * step) | (max(min(step, c[i] - k * step), 0) << 16); }
        }
        if (lane == 31) nchunk_sh = min(incl, KT_MAXCHUNK);
    }
    tl_fence_before();
    __syncthreads();
    tl_fence_after();
    pdl_trigger();
    const uint32_t tmem = tmem_sh;
    const int ntask = nchunk_sh * a.tiles;
    TlWaiter wait{a.state ? &a.state->err : nullptr, a.state && *reinterpret_cast<volatile uint32_t *>(&a.state->err) != 0u};
    auto task = [&](int t) {
        KtTask k;
        const int ch = t / a.tiles, tile = t % a.tiles;
        k.e = chunk_e[ch]; k.first = chunk_fn[ch] & 0xFFFF; k.n = chunk_fn[ch] >> 16;
        k.mi = 0;
        while (tile >= a.tile_end[k.mi]) k.mi++;
        k.row = (tile - (k.mi ? a.tile_end[k.mi - 1] : 0)) * KT_ROWS;
        return k;
    };
    const uint32_t raw0 = smem_u32(raw), b0 = smem_u32(bsm);

    if (warp == 17) {
        // ---------------- raw superblocks of the rows
        if (lane == 0) {
            int n = 0;
            for (int t = blockIdx.x; t < ntask; t += gridDim.x) {
                const KtTask k = task(t);
                const KqtMat &m = a.m[k.mi];
                const int row = k.e * (a.tile_end[k.mi] - (k.mi ? a.tile_end[k.mi - 1] : 0)) * KT_ROWS + k.row;
                for (int sb = 0; sb < nsb; sb++, n++) {
                    const int slot = n % KT_RAW_DEPTH;
                    wait(&rempty[slot], ((n / KT_RAW_DEPTH) & 1) ^ 1);
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
                }
            }
        }
    } else if (warp >= 18) {
        // ---------------- images of the tokens: lane = (token of a group of eight, 16-byte chunk of four); the two warps take alternate groups
        if (!a.cnt) pdl_wait();
        const int lw = warp - 18, tok8 = lane >> 2, c4 = lane & 3;
        int n = 0;
        for (int t = blockIdx.x; t < ntask; t += gridDim.x) {
            const KtTask k = task(t);
            const int quads = a.m[k.mi].type == 12 ? 9 : 8;
            const uint8_t *src[2];
            bool live[2];
#pragma unroll
            for (int g = 0; g < 2; g++) {
                const int i = (2 * g + lw) * 8 + tok8;
                live[g] = i < k.n;
                const int ent = live[g] ? (a.list ? a.list[k.e * BRRR_TILE_MAX + k.first + i] : k.first + i) : 0;
                src[g] = a.img + (size_t)(ent / a.src_div) * nsb * KIMG_SB + c4 * 16;
            }
            const float *ysrc = a.ys + (size_t)((lane < k.n ? (a.list ? a.list[k.e * BRRR_TILE_MAX + k.first + lane] : k.first + lane) : 0) / a.src_div) * nsb;
            for (int sb = 0; sb < nsb; sb++, n++) {
                const int slot = n % KT_B_DEPTH;
                wait(&bempty[slot], ((n / KT_B_DEPTH) & 1) ^ 1);
                const uint32_t dst = b0 + slot * KT_B + lw * 128 + tok8 * 16 + c4 * (KT_NT * 16);
#pragma unroll
                for (int g = 0; g < 2; g++) {
                    if (live[g]) {
#pragma unroll
                        for (int q = 0; q < 8; q++) cp_async16(dst + g * 256 + q * 4 * (KT_NT * 16), src[g] + q * 64);
                        if (quads == 9 && c4 < 2) cp_async16(dst + g * 256 + 32 * (KT_NT * 16), src[g] + 512);
                    }
                    src[g] += KIMG_SB;
                }
                if (lw == 0 && lane < k.n)
                    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(&ysr[n & 7][lane])), "l"(ysrc + sb) : "memory");
                cp_async_arrive(&bfull[slot]);
            }
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
    } else if (warp == 16) {
        // ---------------- products (the whole warp walks the loop, an elected lane issues)
        int n = 0, ca = 0;
        const uint64_t db0 = tl_smem_desc(bsm, KT_NT * 16, 128);
        for (int t = blockIdx.x; t < ntask; t += gridDim.x) {
            const KtTask k = task(t);
            const bool q4 = a.m[k.mi].type == 12;
            const uint32_t idesc = (1u << 4) | ((uint32_t)(2 * ((k.n + 15) >> 4)) << 17) | ((KT_ROWS >> 4) << 24);      // f32 += f16 x f16, N = 16 or 32
            for (int sb = 0; sb < nsb; sb++, n++) {
                const int slot = n % KT_B_DEPTH, buf = n & 1;
                wait(&bfull[slot], (n / KT_B_DEPTH) & 1);
                fence_proxy_async();                   // the copies seen through bfull[] (generic proxy) -> the tensor core's reads
                wait(&dempty[buf], ((n >> 1) & 1) ^ 1);
                const uint64_t db = db0 + (uint64_t)(slot * (KT_B / 16));
                const uint32_t d = tmem + buf * 96;
                if (q4) {
#pragma unroll
                    for (int g = 0; g < 2; g++) {
                        const int ab = ca & 1;
                        wait(&afull[g][ab], (ca >> 1) & 1);
                        tl_fence_after();
                        if (elect_one()) {
#pragma unroll
                            for (int s = 0; s < 8; s++)
                                kt_mma(d + g * 32, tmem + KT_COL_A + (g * 2 + ab) * 64 + s * 8, db + (g * 8 + s) * (2 * KT_NT), idesc, s > 0);
                            if (g == 1) kt_mma(d + 64, tmem + KT_COL_MIN + ab * 8, db + 16 * (2 * KT_NT), idesc, 0);
                            tl_commit(&aempty[g][ab]);
                        }
                        __syncwarp();
                    }
                    ca++;
                } else {
#pragma unroll
                    for (int g = 0; g < 2; g++)
#pragma unroll
                        for (int dig = 0; dig < 2; dig++) {
                            const int ab = (ca + dig) & 1;
                            wait(&afull[g][ab], ((ca + dig) >> 1) & 1);
                            tl_fence_after();
                            if (elect_one()) {
#pragma unroll
                                for (int s = 0; s < 8; s++)
                                    kt_mma(d + dig * 32, tmem + KT_COL_A + (g * 2 + ab) * 64 + s * 8, db + (g * 8 + s) * (2 * KT_NT), idesc, g > 0 || s > 0);
                                tl_commit(&aempty[g][ab]);
                            }
                            __syncwarp();
                        }
                    ca += 2;
                }
                if (elect_one()) {
                    tl_commit(&bempty[slot]);
                    tl_commit(&dfull[buf]);
                    mbar_arrive(&dfull[buf]);          // orders drow and ysr, seen through afull and bfull, before the readers
                }
                __syncwarp();
            }
        }
    } else if (warp >= 8) {
        // ---------------- widening: thread = row m, half g of the superblock
        const int g = (warp - 8) >> 2, m = (warp & 3) * 32 + lane;
        const uint32_t arow = tmem + ((uint32_t)((warp & 3) * 32) << 16);
        int n = 0, ca = 0;
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
                    if (g == 0) drow[n & 3][m] = make_float2(half_bits_to_f32(h.x & 0xffffu), half_bits_to_f32(h.x >> 16));
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&rempty[slot]);
                    const int ab = ca & 1;
                    wait(&aempty[g][ab], ((ca >> 1) & 1) ^ 1);
                    ca++;
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
                    if (g == 0) {
                        const uint32_t dw = lds32(src + 26624 + m * 16 + (sb & 6) * 2);
                        drow[n & 3][m] = make_float2(half_bits_to_f32((sb & 1) ? dw >> 16 : dw & 0xffffu), 0.0f);
                    }
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&rempty[slot]);
                    const int a0 = ca & 1, a1 = a0 ^ 1;
                    wait(&aempty[g][a0], ((ca >> 1) & 1) ^ 1);
                    wait(&aempty[g][a1], (((ca + 1) >> 1) & 1) ^ 1);
                    ca += 2;
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
        if (!a.cnt) pdl_wait();
        const int wg = warp >> 2, m = (warp & 3) * 32 + lane;
        const uint32_t lane_addr = tmem + ((uint32_t)((warp & 3) * 32) << 16) + wg * 16;
        int n = 0;
        for (int t = blockIdx.x; t < ntask; t += gridDim.x) {
            const KtTask k = task(t);
            const bool q4 = a.m[k.mi].type == 12, live = wg * 16 < k.n;
            const int ti = wg * 16 + (lane & 15);
            const int ent = ti < k.n ? (a.list ? a.list[k.e * BRRR_TILE_MAX + k.first + ti] : k.first + ti) : 0;
            f32x2 acc[8];
#pragma unroll
            for (int i = 0; i < 8; i++) acc[i] = 0ull;
            for (int sb = 0; sb < nsb; sb++, n++) {
                const int buf = n & 1;
                wait(&dfull[buf], (n >> 1) & 1);
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

cudaError_t kqt_matrix(const KMatDev &m, size_t rows_total, KqtMat *out) {
    typedef CUresult (*encode_t)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *, const cuuint64_t *, const cuuint32_t *,
                                 const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
    static encode_t encode = [] {
        void *f = nullptr;
        cudaDriverEntryPointQueryResult r;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &f, 12000, cudaEnableDefault, &r) != cudaSuccess || r != cudaDriverEntryPointSuccess) f = nullptr;
        return (encode_t)f;
    }();
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

cudaError_t launch_kqt(const KqtMat *const *mats, float *const *ys_out, const int *ldy, int nmat, int rows_per_expert, const int *cnt, const int *list, int ne, int ntok,
                       int topk, int src_div, const uint8_t *img, const float *ys, bool resid, DevState *state, bool pdl, cudaStream_t st) {
    const int entries = cnt ? ntok * topk : ntok;
    if (nmat < 1 || nmat > 3 || ntok < 1 || ntok > BRRR_TILE_MAX || entries / KT_NT + (cnt ? ne : 1) > KT_MAXCHUNK || (cnt && ne > 256)) return cudaErrorInvalidValue;
    KqtArgs a{};
    int tiles = 0;
    for (int i = 0; i < nmat; i++) {
        const int rows = cnt ? rows_per_expert : mats[i]->rows;
        if (mats[i]->cols != mats[0]->cols || rows % KT_ROWS) return cudaErrorInvalidValue;
        a.m[i] = *mats[i]; a.y[i] = ys_out[i]; a.ldy[i] = ldy[i];
        a.tile_end[i] = tiles += rows / KT_ROWS;
    }
    a.nmat = nmat; a.tiles = tiles; a.nsb = mats[0]->cols / 256; a.cnt = cnt; a.list = list; a.ne = ne; a.ntok = ntok; a.src_div = src_div; a.resid = resid;
    a.img = img; a.ys = ys; a.state = state;
    static unsigned long long configured = 0;      // one bit per device
    cudaError_t e = smem_optin(kqt_kernel, (int)KT_SMEM, configured);
    if (e != cudaSuccess) return e;
    // chunks of tokens: at most one partly filled per expert, and never more than entries
    const int chunks = cnt ? (entries / KT_NT + ne < entries ? entries / KT_NT + ne : entries) : (ntok + KT_NT - 1) / KT_NT;
    const int tasks = chunks * tiles;
    return launch_k(kqt_kernel, dim3(tasks < 148 ? tasks : 148), dim3(KT_THREADS), KT_SMEM, st, pdl, a);
}

}  // namespace brrr
