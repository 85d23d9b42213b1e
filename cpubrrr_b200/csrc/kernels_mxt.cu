// Single-token MXFP4 expert matvecs on the 5th-generation tensor cores in their native 4-bit format
// (tcgen05.mma kind::mxf4.block_scale): the e2m1 codes of the GGUF blocks are the tensor-core operand
// as they are, so the weight bytes go from HBM to shared memory by bulk copy and from there straight
// into the MMA, with no decode instructions at all.
//
// Arithmetic (bit-identical to the integer-unit kernels of kernels_mx.cu).  A row's value is four
// lane chains, chain j accumulating fma(float(t_j(b)), 2^(e_b-128) * xs[b], acc) over the 32-blocks
// b, where t_j(b) is the exact integer dot of the lane's 8 doubled e2m1 values with the lane's 8
// activation bytes.  The tensor core supplies t_j(b) 2^(e_b-128):
//   * an activation byte x in [-127, 127] is written as 64 a + 8 b + c with digits in [-4, 4], and half a
//     digit is an e2m1 value whose code is the digit itself: three digit planes give three exact partial sums;
//   * one MMA covers a block pair (K = 64): operand A = 128 weight rows x 64 codes, operand B = 24
//     columns (digit plane t, block of the pair q, lane j), each holding the plane's codes of the 8
//     positions of lane j in block q and zero elsewhere;
//   * the row's block scale is the block's own e8m0 byte (2^(e-127), true e2m1 values), the column's is 128, 16 or 2 for its plane
//     (ue8m0 134, 131, 128) in its own block and 2^-127 in the other, whose products are all zero: column t holds
//     64, 8 or 1 times its plane's partial sum, times 2^(e_b-128);
//   * every sum is an integer of at most 14 bits times 2^(e_b-128), exact in the f32 accumulator, and so are the two additions that
//     join the planes.  The product of that sum with xs[b] is the exact t_j 2^(e_b-128) xs[b] of the chain's definition whenever
//     2^(e_b-128) xs[b] neither underflows nor overflows: 1e-12 / 127 <= xs <= FLT_MAX / 127, so exponents XT_EXP_MIN .. XT_EXP_MAX qualify.
// Matrices with other exponents (launch_mx_exp_scan; MxtDev.wide) run the same kernels in their WIDE form: every product is formed with one constant
// row scale, column t then holds 64, 8 or 1 times its plane's partial sum, and the epilogue multiplies with the chain's own fl(2^(e_b-128) xs[b])
// from the exponent bytes, as the definition states it.  A step of two layers of the 20b shape, position 140: 86 us scaled, 98 us with every matrix
// wide, 116 us on the integer units.
// The eight epilogue warps read the accumulator columns of their rows from tensor memory
// (tcgen05.ld) and run the float chains, a thread for two chains of a row.
//
// Layout ("tile units").  A tile is 128 matrix rows; per two block pairs: the 4096-byte shared-memory image of operand A of either pair
// in the canonical K-major no-swizzle layout (16-byte chunk of (row m, block q) at q * 2048 + (m / 8) * 128 + (m % 8) * 16, the chunk
// being the 16 nibble bytes of the GGUF block), then the 512 bytes of the rows' e8m0 bytes of the four blocks in the order tensor
// memory wants block scales in (row m at (m % 32) * 16 + (m / 32) * 4 + block), so that one tcgen05.cp moves them there.  A tile is
// contiguous, so any run of these groups is one bulk copy.  Gate and up share tiles (rows 0-63 gate, 64-127 up, same 64 outputs),
// so the SwiGLU and the Q8 quantiser of h run in the same CTA.
//
// Operand B: the digits of an activation (brrr_mxt.cuh) are written once by the kernel that quantises it (the routing-estimate kernel
// for the token, the gate/up epilogue for h); every CTA spreads them over a zeroed image in its shared memory.
//
// Pipeline per CTA, in rounds of four block pairs: warp 8 issues the bulk copies into a ring of stages, an elected lane of warp 9 the scale copies
// and the MMAs of the even rounds into one accumulator region (96 columns), one of warp 10 those of the odd rounds into the other, warps 0-3 and 4-7
// read half a region each at once and carry two chains each.  Every wait is bounded.
//
// What bounds it: hand-overs and first instructions more than anything.  20b shape, position 100, gate/up from its dependency wait to its end 11.3 us
// (14.3 with the planes joined by multiply-adds and the scales multiplied in by the epilogue) for 35 MB, down 7.3 us (8.2) for 18 MB: 1.4 us until
// the experts are picked and the digits spread, 2.1 us until the first round is through, then 500-700 cycles a round (975), 220 of them arithmetic, but
// 1900 for the fifth, the first one whose copies were not under way from the beginning (down, whose copies start before h is there: 870).
// What did not help: announcing down's tiles to L2 from gate/up's last rounds (no change), the issuing loop unrolled by ring stage (1300 cycles
// for each of the first four rounds: instructions met for the first time), running indices in a one-lane branch (1091 against 1050 us a step).
#include "brrr_kernels.h"
#include "brrr_block.cuh"
#include "brrr_tma.cuh"
#include "brrr_tc.cuh"
#include "brrr_mx.cuh"
#include "brrr_mxt.cuh"

namespace brrr {

namespace {

constexpr int XT_CH = 4;                 // block pairs per ring stage = per round of the pipeline
constexpr int XT_REGION_COLS = XT_CH * XT_N;   // accumulator region = one round = 96 tensor-memory columns
constexpr int XT_REGIONS = 2;
constexpr int XT_STAGES = 4;               // two CTAs per SM at the 20b shape; a multiple of the regions: each issuer has stages of its own
static_assert(XT_STAGES % XT_REGIONS == 0, "stages per issuer");
constexpr uint32_t XT_TMEM_COLS = 256;   // 2 regions, their rows' scales, the columns' scales
constexpr int XT_SFA_COL = XT_REGIONS * XT_REGION_COLS;          // rows' block scales: four columns per two block pairs, a set per region
constexpr int XT_SFB_COL = XT_SFA_COL + XT_REGIONS * XT_CH * 2;  // columns' scales: constant
constexpr int XT_GROUP = 2 * MXT_PAIR + MXT_SCALES;              // bytes of two block pairs and their scales
constexpr int XT_STAGE = XT_CH / 2 * XT_GROUP;
__host__ __device__ constexpr uint32_t xt_run_bytes(int pairs) { return (uint32_t)(pairs * MXT_PAIR + (pairs + 1) / 2 * MXT_SCALES); }      // of a run that starts on a group
constexpr int XT_THREADS = 352;        // eight epilogue warps, producer, two issuers
constexpr int XT_PRODUCER = 8, XT_ISSUER = 9;
#ifdef BRRR_TEST_HOOKS
#define XT_T0() long long xt_t0_ = clock64()
#define XT_ACC(v) do { long long xt_t1_ = clock64(); (v) += xt_t1_ - xt_t0_; xt_t0_ = xt_t1_; } while (0)
#else
#define XT_T0() do { } while (0)
#define XT_ACC(v) do { } while (0)
#endif

// ---------------------------------------------------------------- pack: 16-row units -> tile units
struct PackArgs {
    MxDev a, b;              // b.data == nullptr: one matrix, 128 rows per tile; else rows 0-63 from a, 64-127 from b
    int rows_per_expert;     // logical rows of one expert in a (and b)
    int tiles_per_expert;
    MxtDev out;              // out.wide: exponent bytes as they are
};

__global__ void mxt_pack_kernel(PackArgs p, size_t total_words) {
    size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= total_words) return;
    // word index within the destination: [tile][two pairs][1024 words of operand A per pair | 128 words of exponents]
    const int np = p.out.np, tile_words = (int)(xt_run_bytes(np) / 4);
    const size_t tile = idx / tile_words;
    const int w = (int)(idx % tile_words), pair0 = w / (XT_GROUP / 4) * 2, r = w % (XT_GROUP / 4), here = min(2, np - pair0);
    const int e = (int)(tile / p.tiles_per_expert), t = (int)(tile % p.tiles_per_expert);
    // source unit of tile row m and pair, and the row within it; nullptr for rows past the end of the matrix
    auto locate = [&](int m, int pair, int &rl) -> const uint8_t * {
        const MxDev &mat = (p.b.data && m >= 64) ? p.b : p.a;
        const int r = p.b.data ? t * 64 + (m & 63) : t * 128 + m;
        if (r >= p.rows_per_expert) return nullptr;
        const int row = e * p.rows_per_expert + r;
        rl = row & 15;
        return mat.data + mx_unit_off(row >> 4, pair, np);
    };
    uint32_t v = 0;
    int rl = 0;
    if (r < here * 1024) {
        const int q = (r & 1023) >> 9, rem = r & 511, m = (rem >> 5) * 8 + ((rem >> 2) & 7), j = rem & 3;
        const uint8_t *u = locate(m, pair0 + (r >> 10), rl);
        if (u) v = *reinterpret_cast<const uint32_t *>(u + mx_word_off(rl, j) + q * 4);
    } else {
        const int s = r - here * 1024, m = (s & 3) * 32 + (s >> 2);
        for (int k = 0; k < 4; k++) {
            uint32_t ex = 0x7Fu;                      // rows and blocks past the end
            const uint8_t *u = (k >> 1) < here ? locate(m, pair0 + (k >> 1), rl) : nullptr;
            if (u) {
                ex = u[MX_UNIT_EXPS + rl * 2 + (k & 1)];
                if (!p.out.wide && ex < (uint32_t)XT_EXP_MIN) ex = 0x7Fu;      // all-zero blocks only (launch_mx_exp_scan): any finite scale gives the same sums
            }
            v |= ex << (8 * k);
        }
    }
    reinterpret_cast<uint32_t *>(p.out.data)[idx] = v;
}

// Block exponents of a tensor in GGUF form against the range of the scaled products: *bad != 0 when a block with a value other than zero
// lies below it, or any block above it.
__global__ void mx_exp_scan_kernel(const uint8_t *__restrict__ raw, size_t blocks, uint32_t *bad) {
    bool b = false;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < blocks; i += (size_t)gridDim.x * blockDim.x) {
        const uint8_t *p = raw + i * 17;
        if (p[0] > XT_EXP_MAX) b = true;
        else if (p[0] < XT_EXP_MIN)
            for (int k = 1; k <= 16; k++) b |= (p[k] & 0x77) != 0;
    }
    if (b) atomicOr(bad, 1u);
}

// ---------------------------------------------------------------- tensor-core plumbing
// block-scaled instruction descriptor: A = B = e2m1 (format 1), both K-major, N / 8 at bit 17,
// ue8m0 scales (bit 23), M / 16 at bit 24, K = 64; the rows' scale-factor id (bits 29-30) is 0 or 2: bytes 0, 1 or 2, 3 of their words
constexpr uint32_t XT_IDESC = (1u << 7) | (1u << 10) | ((uint32_t)(XT_N >> 3) << 17) | (1u << 23) | ((128u >> 4) << 24);

// (predicates: tl_commit_if)
__device__ __forceinline__ void xt_mma(uint32_t issue, uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc, uint32_t tmem_sfa, uint32_t tmem_sfb) {
    asm volatile(
        "{\n\t.reg .pred p, e;\n\tsetp.ne.b32 p, %4, 0;\n\tsetp.ne.b32 e, %7, 0;\n\t"
        "@e tcgen05.mma.cta_group::1.kind::mxf4.block_scale.block32 [%0], %1, %2, %3, [%5], [%6], p;\n\t}"
        ::"r"(tmem_d), "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(0u), "r"(tmem_sfa), "r"(tmem_sfb), "r"(issue)
        : "memory");
}
// 512 bytes of block scales -> four columns of tensor memory, the same 32 lanes for each of its quarters; in order with the products of the issuing thread
__device__ __forceinline__ void xt_cp_scales(uint32_t issue, uint32_t tmem, uint64_t desc) {
    asm volatile("{\n\t.reg .pred e;\n\tsetp.ne.b32 e, %2, 0;\n\t@e tcgen05.cp.cta_group::1.32x128b.warpx4 [%0], %1;\n\t}" ::"r"(tmem), "l"(desc), "r"(issue) : "memory");
}
__device__ __forceinline__ void xt_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void xt_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
// Half the accumulator columns of a region (two chains of four block pairs: runs of 12 columns, 24 apart) of this thread's row, as pairs.
// Loads, wait and packing are one statement, so nothing can use a register before the wait.
__device__ __forceinline__ void xt_ld48(uint32_t taddr, f32x2 (&v)[24]) {
    asm volatile("{\n\t.reg .b32 r<12>;\n\t.reg .b32 s<12>;\n\t.reg .b32 t<12>;\n\t.reg .b32 u<12>;\n\t"
                 "tcgen05.ld.sync.aligned.32x32b.x8.b32 {r0,r1,r2,r3,r4,r5,r6,r7}, [%24];\n\t"
                 "tcgen05.ld.sync.aligned.32x32b.x4.b32 {r8,r9,r10,r11}, [%25];\n\t"
                 "tcgen05.ld.sync.aligned.32x32b.x8.b32 {s0,s1,s2,s3,s4,s5,s6,s7}, [%26];\n\t"
                 "tcgen05.ld.sync.aligned.32x32b.x4.b32 {s8,s9,s10,s11}, [%27];\n\t"
                 "tcgen05.ld.sync.aligned.32x32b.x8.b32 {t0,t1,t2,t3,t4,t5,t6,t7}, [%28];\n\t"
                 "tcgen05.ld.sync.aligned.32x32b.x4.b32 {t8,t9,t10,t11}, [%29];\n\t"
                 "tcgen05.ld.sync.aligned.32x32b.x8.b32 {u0,u1,u2,u3,u4,u5,u6,u7}, [%30];\n\t"
                 "tcgen05.ld.sync.aligned.32x32b.x4.b32 {u8,u9,u10,u11}, [%31];\n\t"
                 "tcgen05.wait::ld.sync.aligned;\n\t"
                 "mov.b64 %0, {r0,r1};\n\tmov.b64 %1, {r2,r3};\n\tmov.b64 %2, {r4,r5};\n\tmov.b64 %3, {r6,r7};\n\tmov.b64 %4, {r8,r9};\n\tmov.b64 %5, {r10,r11};\n\t"
                 "mov.b64 %6, {s0,s1};\n\tmov.b64 %7, {s2,s3};\n\tmov.b64 %8, {s4,s5};\n\tmov.b64 %9, {s6,s7};\n\tmov.b64 %10, {s8,s9};\n\tmov.b64 %11, {s10,s11};\n\t"
                 "mov.b64 %12, {t0,t1};\n\tmov.b64 %13, {t2,t3};\n\tmov.b64 %14, {t4,t5};\n\tmov.b64 %15, {t6,t7};\n\tmov.b64 %16, {t8,t9};\n\tmov.b64 %17, {t10,t11};\n\t"
                 "mov.b64 %18, {u0,u1};\n\tmov.b64 %19, {u2,u3};\n\tmov.b64 %20, {u4,u5};\n\tmov.b64 %21, {u6,u7};\n\tmov.b64 %22, {u8,u9};\n\tmov.b64 %23, {u10,u11};\n\t"
                 "}"
                 : "=l"(v[0]),"=l"(v[1]),"=l"(v[2]),"=l"(v[3]),"=l"(v[4]),"=l"(v[5]),"=l"(v[6]),"=l"(v[7]),"=l"(v[8]),"=l"(v[9]),"=l"(v[10]),"=l"(v[11]),"=l"(v[12]),"=l"(v[13]),"=l"(v[14]),"=l"(v[15]),"=l"(v[16]),"=l"(v[17]),"=l"(v[18]),"=l"(v[19]),"=l"(v[20]),"=l"(v[21]),"=l"(v[22]),"=l"(v[23])
                 : "r"(taddr + 0), "r"(taddr + 8), "r"(taddr + 24), "r"(taddr + 32), "r"(taddr + 48), "r"(taddr + 56), "r"(taddr + 72), "r"(taddr + 80)
                 : "memory");
}
__device__ __forceinline__ void xt_bar_epi() { asm volatile("bar.sync 1, 256;" ::: "memory"); }       // both halves of the epilogue warps
__device__ __forceinline__ void xt_bar_half() { asm volatile("bar.sync 2, 128;" ::: "memory"); }      // the half that finishes the rows

// Waits of the pipeline loops.  The loops are executed by one warp per scheduler, so their code
// has to stay small enough for the instruction cache next to the scheduler: the common case (phase
// already complete) is one probe inline, everything else is out of line.  Bounded like Waiter::wait;
// returns false (after recording the error) when the wait ran out.
__device__ __noinline__ bool xt_wait_slow(uint64_t *bar, uint32_t parity, uint32_t *err, bool sleep) {
    if (err && *reinterpret_cast<volatile uint32_t *>(err) != 0u) return false;      // a wait has already failed: do not wait again
    const long long t0 = clock64();
    do {
        for (int i = 0; i < 64; i++) {
            if (sleep) __nanosleep(32);
            if (sleep ? mbar_test_wait(bar, parity) : mbar_try_wait(bar, parity)) return true;
        }
    } while (clock64() - t0 < WAIT_CYCLES);
    if (err) atomicCAS(err, (uint32_t)DEV_ERR_NONE, (uint32_t)DEV_ERR_COPY_TIMEOUT);
    return false;
}
__device__ __forceinline__ void xt_wait(uint64_t *bar, uint32_t parity, uint32_t *err, bool sleep = false) {
    if (!mbar_test_wait(bar, parity)) xt_wait_slow(bar, parity, err, sleep);
}

// The issuing warp's waits: suspended in hardware between probes (it waits most of the time, beside busy warps, and its wake-up is on the
// critical path), a bounded number of times - far above any copy or product; then the error word is set and it waits no more.
struct XtIssueWait {
    uint32_t *err;
    bool dead;
    __device__ __forceinline__ void operator()(uint64_t *bar, uint32_t parity) {
        if (dead || mbar_test_wait(bar, parity)) return;
        for (int i = 0; !mbar_try_wait_hint(bar, parity, 20000u);)
            if (++i == 1 << 17) {
                dead = true;
                if (err) atomicCAS(err, (uint32_t)DEV_ERR_NONE, (uint32_t)DEV_ERR_COPY_TIMEOUT);
                break;
            }
    }
};

// Digits of an activation that some other kernel quantised (stage-level entry points).
__global__ void xt_digits_kernel(const int8_t *__restrict__ xq, int nb, uint8_t *dig) {
    const int b = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (b >= nb) return;
    xt_emit_digits((int)xq[b * 32 + lane], lane, b, dig);
}

// ---------------------------------------------------------------- the two expert kernels
struct XtArgs {
    MxtDev w;                   // gate|up tiles, or down tiles
    const float *bias_a;        // gate bias, or down bias       [expert][d]
    const float *bias_b;        // up bias
    const int32_t *top;         // exact routing (used when est == nullptr)
    const float *wts;           // down: nullable, see launch_down_t
    const float *est;           // nullable: router estimate; slot s belongs to its s-th largest entry
    int ne, topk, d;
    const uint8_t *bdig;        // digits of the activation (brrr_mxt.cuh): gate/up [blocks][48]; down [slot][blocks][48]
    const float *xs;            // its block scales:                gate/up [blocks];   down [slot][blocks]
    int8_t *hq;                 // gate/up outputs: Q8 of h per slot, its scales, its digits
    float *hs;
    uint8_t *hdig;
    float *x;                   // down: residual stream, updated in place
    float *part;                // down: [topk][tiles * 128] row sums before bias
    uint32_t *counter;          // down: [tiles] arrival counters, zero between launches
    DevState *state;
    // expert parallelism (ep_on): w holds the experts [ep.e_lo, ep.e_lo + ep.e_cnt) only; CTAs of a slot
    // whose expert lives on another rank do nothing; down stores its row sums, each tagged with the step
    // number in one 64-bit word, into every rank's buffer ep.pairs ([layer][slot][d])
    int ep_on, layer;
    EpCtx ep;
};

struct XtShared {
    unsigned char *ring, *bimg;
    f32x2 *xsc;                 // block scales of the activation, each twice: the factor of two chains
    uint64_t *full, *empty, *dfull, *dempty;
};

// One block pair of one row: two chains' scaled lane dots of its two blocks from the three digit planes, then their fused multiply-adds,
// in block order.  Both chains share an instruction (two independent round-to-nearest operations).
// ex (wide matrices): the row's exponent bytes of the two blocks in the low half; else the products carry them.
template <bool WIDE>
__device__ __forceinline__ void xt_pair(const f32x2 *v, f32x2 xs0, f32x2 xs1, uint32_t ex, f32x2 &acc) {
    if (WIDE) {
        const uint32_t s0 = __float_as_uint(brrr_e8m0_scale(ex & 0xFFu)), s1 = __float_as_uint(brrr_e8m0_scale((ex >> 8) & 0xFFu));
        xs0 = tl_mul2(tl_pack2(s0, s0), xs0);
        xs1 = tl_mul2(tl_pack2(s1, s1), xs1);
    }
    acc = tl_fma2(tl_add2(tl_add2(v[0], v[2]), v[4]), xs0, acc);
    acc = tl_fma2(tl_add2(tl_add2(v[1], v[3]), v[5]), xs1, acc);
}

// WIDE: block exponents outside the range of the scaled products (top of this file)
template <bool DOWN, bool EP, bool WIDE>
__global__ void __launch_bounds__(XT_THREADS, 2) xt_expert_kernel(XtArgs a) {
    extern __shared__ __align__(128) unsigned char smraw[];
    // the warp index as the compiler can see it: the same in every lane, so the roles' loops keep their values in uniform registers
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    const int np = a.w.np, nb = np * 2;
    const int t = blockIdx.x, ei = blockIdx.y;
    const int nchunks = (np + XT_CH - 1) / XT_CH;
    XtShared sh;
    sh.ring = smraw;
    sh.bimg = smraw + XT_STAGE * XT_STAGES;
    sh.xsc = reinterpret_cast<f32x2 *>(sh.bimg + (size_t)np * XT_B_PAIR);
    sh.full = reinterpret_cast<uint64_t *>(sh.xsc + nchunks * 2 * XT_CH);      // (whole rounds: the last one reads past the blocks)
    sh.empty = sh.full + XT_STAGES;
    sh.dfull = sh.empty + XT_STAGES;
    sh.dempty = sh.dfull + XT_REGIONS;
    __shared__ uint32_t tmem_base_sh;
    __shared__ float half_s[128];
    __shared__ float gu_s[2][64];
    __shared__ int last_sh, expert_sh;
    uint32_t *err = a.state ? &a.state->err : nullptr;
    constexpr int SB = DOWN ? 128 : 96;          // clock stamps of timeline builds
    (void)SB;
    BRRR_STAMP(a.state, SB);
    BRRR_GT_START(a.state, DOWN ? 237 : 236);

    // ---- set-up that needs nothing from the kernels before
    if (tid == 0) {
        for (int s = 0; s < XT_STAGES; s++) { mbar_init(&sh.full[s], 1); mbar_init(&sh.empty[s], 1); }
        for (int r = 0; r < XT_REGIONS; r++) { mbar_init(&sh.dfull[r], 1); mbar_init(&sh.dempty[r], 8); }
        mbar_fence_init();
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_sh)), "r"(XT_TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    for (int i = tid; i < np * (XT_B_PAIR / 16); i += XT_THREADS) reinterpret_cast<uint4 *>(sh.bimg)[i] = make_uint4(0, 0, 0, 0);
    for (int i = nb + tid; i < nchunks * 2 * XT_CH; i += XT_THREADS) sh.xsc[i] = 0ull;
    xt_fence_before();
    __syncthreads();
    xt_fence_after();
    const uint32_t tmem_base = __shfl_sync(0xffffffffu, tmem_base_sh, 0);
    if (warp < 4) {
        // the columns' scales: lane n = column (plane (n % 12) / 4, block of the pair (n / 2) & 1), byte k = block k of the pair
        const uint32_t sc = lane < XT_N ? (134u - 3u * (uint32_t)((lane % 12) >> 2)) << (8 * ((lane >> 1) & 1)) : 0u;
        const uint32_t lanes = tmem_base + ((uint32_t)(warp * 32) << 16);
        asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1,%2,%2,%2};" ::"r"(lanes + XT_SFB_COL), "r"(sc), "r"(0u) : "memory");
        if (WIDE)      // 2 for every row and block: twice an e2m1 value is the doubled one
            for (int k = 0; k < XT_REGIONS * XT_CH * 2; k += 4)
                asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1,%1,%1,%1};" ::"r"(lanes + XT_SFA_COL + k), "r"(0x80808080u) : "memory");
        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
    }
    xt_fence_before();
    __syncthreads();                 // scales in place before the issuing thread can reach its first MMA, the image zeroed before the digits come
    xt_fence_after();
    // ---- routing of this slot (the ei-th largest entry of the estimate, or the exact routing), the
    // weight stream, the activation image (one bulk copy) and its block scales
    const size_t tile_bytes = xt_run_bytes(np), expert_bytes = tile_bytes * a.w.tiles_per_expert;
    auto is_local = [&](int e) { return !EP || (e >= a.ep.e_lo && e < a.ep.e_lo + a.ep.e_cnt); };
    auto tile_of = [&](int e) { return a.w.data + t * tile_bytes + (size_t)(EP ? e - a.ep.e_lo : e) * expert_bytes; };
    const uint32_t ep_epoch = EP ? *a.ep.epoch : 0u;          // the step in flight (written by the step's first kernel)
    // by the producer warp alone; the others read the expert behind the barrier in front of the rounds.  20b shape,
    // 73 + 128 tokens: 126.9 ms with every warp picking for itself, 125.9 so; 120b shape (128 experts): 652 tok/s, 707 so, 687 with a block-wide ranking.
    auto route_and_start = [&]() {
        if (warp != XT_PRODUCER) return;
        const int e = a.est ? __shfl_sync(0xffffffffu, spec_pick(a.est, a.ne, a.topk, ei + 1, a.state, lane), ei) : a.top[ei];
        if (is_local(e) && lane < min(XT_STAGES, nchunks)) {          // one lane per copy: the first stages of the weight stream
            const uint32_t bytes = xt_run_bytes(min(XT_CH, np - lane * XT_CH));
            mbar_expect_tx(&sh.full[lane], bytes);
            bulk_g2s_once(sh.ring + XT_STAGE * lane, tile_of(e) + (size_t)lane * XT_STAGE, bytes, &sh.full[lane]);
        }
        if (lane == 0) expert_sh = e;
    };
    // The down projection knows its expert before gate/up has finished (the routing is two kernels
    // old), and its CTAs have the footprint of a gate/up CTA: they become resident beside running
    // gate/up CTAs and start their weight stream there, before they wait for h.
    constexpr bool early = DOWN;
    if (early) route_and_start();
    BRRR_STAMP(a.state, SB + 1);
    pdl_wait_cta();
    BRRR_STAMP(a.state, SB + 2);
    BRRR_GT_GO(a.state, SB + 30);
    pdl_trigger();
    // the activation's block scales and digits: every load before the first store (each is a round trip to L2)
    float xs_mine = 0.0f;
    if (tid < nb) xs_mine = (DOWN ? a.xs + (size_t)ei * nb : a.xs)[tid];      // nb <= 128
    const uint4 *dig = reinterpret_cast<const uint4 *>(a.bdig + (DOWN ? (size_t)ei * nb * XT_DIG_BLOCK : 0));
    uint4 dw[2];
#pragma unroll
    for (int k = 0; k < 2; k++) dw[k] = tid + k * XT_THREADS < nb * 3 ? dig[tid + k * XT_THREADS] : make_uint4(0, 0, 0, 0);      // nb * 3 <= 384
    if (!early) route_and_start();
    if (tid < nb) sh.xsc[tid] = tl_pack2(__float_as_uint(xs_mine), __float_as_uint(xs_mine));
#pragma unroll
    for (int k = 0; k < 2; k++) if (tid + k * XT_THREADS < nb * 3) xt_spread_digits(dw[k], tid + k * XT_THREADS, sh.bimg);
    fence_proxy_async();                                         // these stores -> the tensor core's reads
    __syncthreads();
    const int e = expert_sh;
    const bool local = is_local(e);
    const unsigned char *src = tile_of(e);
    BRRR_STAMP(a.state, SB + 3);

    // Loop structure shared by the three roles: round r = ring stage r % stages = 4 block pairs =
    // accumulator region r % 2.  All indices advance incrementally.
    if (EP && !local) {
        // the slot's expert lives on another rank: nothing to compute here
    } else if (warp == XT_PRODUCER) {
        // ---- producer: refill a stage once its products are complete
        if (lane == 0) {
            int s = 0;
            uint32_t par = 0;                        // parity of the release being waited for
            for (int c = XT_STAGES; c < nchunks; c++) {
                const uint32_t bytes = xt_run_bytes(min(XT_CH, np - c * XT_CH));
                xt_wait(&sh.empty[s], par, err, true);
                mbar_expect_tx(&sh.full[s], bytes);
                bulk_g2s_once(sh.ring + XT_STAGE * s, src + (size_t)c * XT_STAGE, bytes, &sh.full[s]);
                if (++s == XT_STAGES) { s = 0; par ^= 1u; }
            }
        }
    } else if (warp >= XT_ISSUER) {
        // ---- MMA issue: one instruction per block pair, four per round into one accumulator region (the whole warp walks the loop, an
        // elected lane issues: in a one-lane branch every product costs 100 cycles of operand moves, 35 here)
        {
            XtIssueWait wait{err, err && *reinterpret_cast<volatile uint32_t *>(err) != 0u};
            const uint32_t sfb = tmem_base + XT_SFB_COL;
            const uint64_t dhi = ((uint64_t)((128u >> 4) & 0x3FFF) << 32) | ((uint64_t)1 << 46);     // descriptor bits common to A, B and the scales
            const uint64_t alo = dhi | ((uint64_t)((2048u >> 4) & 0x3FFF) << 16), blo = dhi | ((uint64_t)(((uint32_t)XT_B_PAIR / 2 >> 4) & 0x3FFF) << 16);
            const uint32_t b0 = smem_u32(sh.bimg) >> 4, r0 = smem_u32(sh.ring) >> 4;       // descriptor start-address fields (16-byte units)
            const uint32_t issue = elect_one() ? 1u : 0u;
            // Two issuers, one for the even rounds and region 0, one for the odd, so that a round's waits overlap the other's instructions.  Each has
            // stages, scale columns and barriers of its own.  73 + 128 tokens of the 20b shape: 128.4 ms with one issuer, 127.7 with two.
            const int reg = warp - XT_ISSUER;
            int s = reg, left = np - reg * XT_CH;
            uint32_t fpar = 0, epar = 1, baddr = b0 + reg * (XT_CH * XT_B_PAIR / 16);             // full-stage parity; region-free parity (first pass: free)
            // One body for every round and product: the instructions a CTA meets for the first time come from L2 or beyond and cost more
            // than the running indices (a body per stage: 1300 cycles for each of the first four rounds).
#pragma unroll 1
            for (int r = reg; r < nchunks; r += XT_REGIONS) {
                wait(&sh.full[s], fpar);
                wait(&sh.dempty[reg], epar);
                epar ^= 1u;
                xt_fence_after();
                const uint32_t sfa = tmem_base + XT_SFA_COL + reg * XT_CH * 2;
                uint32_t d0 = tmem_base + reg * XT_REGION_COLS, aaddr = r0 + s * (XT_STAGE / 16), baddr1 = baddr;
                const int cnt = min(left, XT_CH);
#pragma unroll 1
                for (int k = 0; k < cnt; k += 2) {
                    const uint32_t two = cnt - k > 1 ? issue : 0u;
                    if (!WIDE) xt_cp_scales(issue, sfa + k * 2, dhi | (aaddr + (cnt - k > 1 ? 2 : 1) * (MXT_PAIR / 16)));
                    xt_mma(issue, d0, alo | aaddr, blo | baddr1, XT_IDESC, sfa + k * 2, sfb);
                    xt_mma(two, d0 + XT_N, alo | (aaddr + MXT_PAIR / 16), blo | (baddr1 + XT_B_PAIR / 16), XT_IDESC | (2u << 29), sfa + k * 2, sfb);
                    d0 += 2 * XT_N; aaddr += XT_GROUP / 16; baddr1 += 2 * XT_B_PAIR / 16;
                }
                tl_commit_if(r + XT_STAGES < nchunks ? issue : 0u, &sh.empty[s]);      // nobody waits for the last ones
                tl_commit_if(issue, &sh.dfull[reg]);
                __syncwarp();
                baddr += XT_REGIONS * XT_CH * XT_B_PAIR / 16;
                left -= XT_REGIONS * XT_CH;
                if ((s += XT_REGIONS) >= XT_STAGES) { s -= XT_STAGES; fpar ^= 1u; }
            }
        }
    } else {
        // ---- epilogue: thread m of half h owns chains 2 h, 2 h + 1 of tile row m
        const int m = tid & 127, h = warp >> 2;
        const uint32_t lane_addr = tmem_base + ((uint32_t)((warp & 3) * 32) << 16) + h * (XT_N / 2);
        f32x2 acc = 0ull;
        const float bias_pre = DOWN ? 0.0f : ((m >> 6) ? a.bias_b : a.bias_a)[(size_t)e * a.d + t * 64 + (m & 63)];   // in flight during the stream
        int reg = 0, left = np;
        uint32_t dpar = 0, xaddr = smem_u32(sh.xsc);
        long long tw_d = 0, tw_ld = 0, tw_math = 0;
        (void)tw_d; (void)tw_ld; (void)tw_math;
#pragma unroll 1
        for (int r = 0; r < nchunks; r++) {
            XT_T0();
            f32x2 xs[2 * XT_CH], dv[XT_REGION_COLS / 4];
#pragma unroll
            for (int k = 0; k < 2 * XT_CH; k += 2) lds_pairs(xaddr + k * 8, xs[k], xs[k + 1]);
            uint32_t ex[XT_CH / 2] = {};
            if (WIDE) {              // this row's word of each group's exponents (the word may be read before the round is through: weights do not change)
#pragma unroll
                for (int k = 0; k < XT_CH / 2; k++)
                    if (2 * k < left) ex[k] = __ldg(reinterpret_cast<const uint32_t *>(src + (size_t)(r * (XT_CH / 2) + k) * XT_GROUP + min(2, left - 2 * k) * MXT_PAIR + (m & 31) * 16 + (m >> 5) * 4));
            }
            xt_wait(&sh.dfull[reg], dpar, err);
            XT_ACC(tw_d);
            xt_fence_after();
            xt_ld48(lane_addr + reg * XT_REGION_COLS, dv);
            XT_ACC(tw_ld);
            xt_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&sh.dempty[reg]);
#pragma unroll
            for (int k = 0; k < XT_CH; k++)
                if (k < left) xt_pair<WIDE>(dv + XT_N / 4 * k, xs[2 * k], xs[2 * k + 1], ex[k / 2] >> (16 * (k & 1)), acc);
            xaddr += 2 * XT_CH * 8;
            left -= XT_CH;
            if (++reg == XT_REGIONS) { reg = 0; dpar ^= 1u; }
            XT_ACC(tw_math);
            if (r < 12) BRRR_STAMP(a.state, SB + 4 + r);
        }
        BRRR_STAMP(a.state, SB + 16);
#ifdef BRRR_TEST_HOOKS
        if (a.state && tid == 0 && blockIdx.x == BRRR_STAMP_BX && blockIdx.y == 0) {
            long long *o = a.state->stamps + (DOWN ? 205 : 200);
            o[0] = tw_d; o[1] = tw_ld; o[2] = tw_math;
        }
#endif
        // row sum (a0 + a1) + (a2 + a3)
        float c0, c1;
        tl_unpack2(acc, c0, c1);
        float v = __fadd_rn(c0, c1);
        if (h) half_s[m] = v;
        xt_bar_epi();
        if (h) {
            // done
        } else if (!DOWN) {
            v = __fadd_rn(v, half_s[m]);
            gu_s[m >> 6][m & 63] = __fadd_rn(v, bias_pre);
            xt_bar_half();
            if (warp < 2) {
                // SwiGLU, Q8 of this 32-block of h, and the digits down reads
                const float h = swiglu_oai(gu_s[0][warp * 32 + lane], gu_s[1][warp * 32 + lane]);
                const float amax = fmaxf(warp_max(fabsf(h)), 1e-12f);
                const float sc = __fdiv_rn(amax, 127.0f);
                const int qv = brrr_q8_round_inv(h, sc, brrr_q8_inv(amax)), b = t * 2 + warp;
                if (lane == 0) a.hs[ei * nb + b] = sc;
                a.hq[(size_t)ei * a.d + b * 32 + lane] = (int8_t)qv;
                xt_emit_digits(qv, lane, b, a.hdig + (size_t)ei * nb * XT_DIG_BLOCK);
            }
        } else {
            v = __fadd_rn(v, half_s[m]);
            const int r = t * 128 + m, dpad = a.w.tiles_per_expert * 128;
            if (EP) {
                // the row sum, tagged with the step number, to every rank: one plain 64-bit store over
                // NVLink peer memory per rank; the consumer polls the word itself
                const size_t off = ((size_t)a.layer * a.topk + ei) * a.d + r;
                const unsigned long long word = ((unsigned long long)ep_epoch << 32) | __float_as_uint(v);
                if (r < a.d)
                    for (int p = 0; p < a.ep.world; p++) if (p != a.ep.rank) a.ep.pairs[p][off] = word;
                a.part[(size_t)ei * dpad + r] = v;          // this rank's own fold reads it after the kernel boundary
            } else a.part[(size_t)ei * dpad + r] = v;
            if (a.wts) {                     // exact routing known: fold here; else a fold kernel follows
                __threadfence();
                xt_bar_half();
                if (m == 0) last_sh = atomicAdd(&a.counter[t], 1u) == (uint32_t)(a.topk - 1);
                xt_bar_half();
            } else if (m == 0) last_sh = 0;
            if (a.wts && last_sh) {
                // the last of the top-k CTAs of these 128 rows folds them in slot order
                __threadfence();
                if (r < a.d) {
                    float s = a.x[r];
                    for (int k = 0; k < a.topk; k++)
                        s = __fadd_rn(s, __fmul_rn(a.wts[k], __fadd_rn(__ldcg(&a.part[(size_t)k * dpad + r]), a.bias_a[(size_t)a.top[k] * a.d + r])));
                    a.x[r] = s;
                }
                if (m == 0) a.counter[t] = 0;
            }
        }
    }
    BRRR_STAMP(a.state, SB + 17);
    BRRR_GT_END(a.state, SB + 31);
    xt_fence_before();
    __syncthreads();
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(XT_TMEM_COLS) : "memory");
}

// Fold of the down-projection partial sums once the exact routing is known:
//   x[r] += sum over k ascending of wts[k] * (part[slot of top[k]][r] + bias[top[k]][r])
// (multiply, then add, as the reference's combine).  With est != nullptr the partial sums were
// computed for the top-k of the estimate: exact experts missing from it flag the step.
struct FoldArgs {
    const int32_t *top;
    const float *wts, *est;
    int ne, topk, d, dpad;
    const float *part, *down_b;
    float *x;
    DevState *state;
};

__global__ void __launch_bounds__(128) xt_fold_kernel(FoldArgs a) {
    __shared__ int slot_of[8];
    const int tid = threadIdx.x;
    BRRR_GT_START(a.state, 238);
    pdl_wait();
    BRRR_GT_GO(a.state, 239);
    pdl_trigger();
    int found = -1;                          // slot of the exact routing's tid-th expert in the estimate
    if (a.est && tid < 32) {
        const int picked = spec_pick(a.est, a.ne, a.topk, a.topk, a.state, tid), want = a.top[min(tid, a.topk - 1)];
        for (int s = 0; s < a.topk; s++) if (__shfl_sync(0xffffffffu, picked, s) == want) found = s;
    }
    if (tid < a.topk) {
        int slot = tid;
        if (a.est) {
            slot = found;
            if (slot < 0) {                  // the estimate missed this expert: flag the step, keep going
                slot = 0;
                if (blockIdx.x == 0 && a.state) atomicMin(&a.state->spec_fail_step, a.state->n_out);
            }
        }
        slot_of[tid] = slot;
    }
    __syncthreads();
    const int r = blockIdx.x * 128 + tid;
    if (r < a.d) {
        float s = a.x[r];
        for (int k = 0; k < a.topk; k++)
            s = __fadd_rn(s, __fmul_rn(a.wts[k], __fadd_rn(a.part[(size_t)slot_of[k] * a.dpad + r], a.down_b[(size_t)a.top[k] * a.d + r])));
        a.x[r] = s;
    }
    BRRR_GT_END(a.state, 240);
}

// The same fold as one CTA that also prepares the next projection's activation.  Used by the
// speculative decode step, where the exact router runs on another stream beside gate/up and down:
// instead of a graph edge from the router (which would cost this kernel its programmatic launch),
// one lane per word polls, bounded, the routing words the router publishes, each tagged with the
// router's sequence number (this launch expects fold_seq + 1; the router does not depend on this
// kernel, so the wait cannot deadlock).  The partial sums, the
// residual and the routing estimate are fetched before that wait.  After the fold the whole
// residual is in shared memory, so the RMS norm (fixed 16-chain order) and the Q8 image that the
// next q/k/v projection (or the vocabulary head) needs are computed here once, rather than by every
// CTA of that projection.
struct FoldNormArgs {
    FoldArgs f;
    const float *norm_w;     // nullable: fold only
    float eps;
    int8_t *nq;              // Q8 of the normalised residual, element order
    float *ns;               // its block scales
    uint32_t *router_seq, *fold_seq;
    // expert parallelism: the row sums come from the ranks that own the estimate's experts, as 64-bit
    // words (step number << 32 | float bits) in this rank's buffer of the layer ([slot][d]); a word is
    // valid once it carries the step number *ep_epoch
    const unsigned long long *ep_pairs;
    const uint32_t *ep_epoch;
    int ep_lo, ep_cnt;       // this rank's experts: their slots' row sums are in f.part, as on a single GPU
};

constexpr int FN_THREADS = 1024;

template <int MAXS, bool EP>       // slots held in registers: top-k <= MAXS; EP: expert-parallel exchange
__global__ void __launch_bounds__(FN_THREADS) xt_fold_norm_kernel(FoldNormArgs a) {
    extern __shared__ __align__(16) float fsm[];          // d floats of the residual
    __shared__ int sel[8];
    __shared__ int slot_of[8];
    __shared__ float wts_sh[8];
    __shared__ float inv_sh;
    const int tid = threadIdx.x, d = a.f.d, dpad = a.f.dpad, topk = a.f.topk;
    float *xf = fsm;
    // ---- everything that kernels before down produced, before the dependency wait: norm weights,
    // the residual, the speculative expert set and those experts' biases
    float4 wreg[1];
    norm_prefetch<1>(a.norm_w, d, wreg, tid, FN_THREADS);
    BRRR_GT_START(a.f.state, 238);
    // thread g owns rows 4g .. 4g+3 (one 16-byte access per operand)
    const bool live = tid < (d >> 2);
    const float4 zero4 = make_float4(0.f, 0.f, 0.f, 0.f);
    float4 xr = live ? reinterpret_cast<const float4 *>(a.f.x)[tid] : zero4, pb[MAXS], ps[MAXS];
    if (a.f.est) {
        if (tid < 32) {
            const int picked = spec_pick(a.f.est, a.f.ne, topk, topk, a.f.state, tid);
            if (tid < topk) sel[tid] = picked;
        }
        __syncthreads();
#pragma unroll
        for (int s = 0; s < MAXS; s++) pb[s] = (live && s < topk) ? reinterpret_cast<const float4 *>(a.f.down_b + (size_t)sel[s] * d)[tid] : zero4;
    }
    const uint32_t want_seq = a.fold_seq ? __ldcg(a.fold_seq) + 1u : 0u;      // written by the previous launch of this kernel
    const uint32_t ep_epoch = EP ? *a.ep_epoch : 0u;                  // the step in flight (written by the step's first kernel)
#ifdef BRRR_FOLD_EARLY_TRIGGER
    pdl_trigger();       // the next projection may become resident and stream its weights while down still runs
#endif
    pdl_wait_cta();      // down's partial sums are complete
    BRRR_GT_GO(a.f.state, 239);
    BRRR_STAMP(a.f.state, 241);
#ifndef BRRR_FOLD_EARLY_TRIGGER
    pdl_trigger();
#endif
    // ---- slot s: partial sum of the s-th expert of the estimate
#pragma unroll
    for (int s = 0; s < MAXS; s++) {
        const bool mine = !EP || (sel[s < topk ? s : 0] >= a.ep_lo && sel[s < topk ? s : 0] < a.ep_lo + a.ep_cnt);
        ps[s] = (live && s < topk && mine) ? reinterpret_cast<const float4 *>(a.f.part + (size_t)s * dpad)[tid] : zero4;
    }
    if (EP && live) {
        // slots whose expert lives on another rank: every thread polls (bounded) the four tagged words
        // of its rows until all of them carry this step's number
        uint32_t *errp = a.f.state ? &a.f.state->err : nullptr;
        const long long t0 = clock64();
        bool ok = false;
        while (!ok) {
            ok = true;
#pragma unroll
            for (int s = 0; s < MAXS; s++) {
                if (s < topk && !(sel[s] >= a.ep_lo && sel[s] < a.ep_lo + a.ep_cnt)) {
                    // read at the L2, where the peers' stores to this GPU's memory land
                    const ulonglong2 *w = reinterpret_cast<const ulonglong2 *>(a.ep_pairs + (size_t)s * d) + 2 * tid;
                    const ulonglong2 lo = __ldcg(w), hi = __ldcg(w + 1);
                    ok = ok && (uint32_t)(lo.x >> 32) == ep_epoch && (uint32_t)(lo.y >> 32) == ep_epoch && (uint32_t)(hi.x >> 32) == ep_epoch &&
                         (uint32_t)(hi.y >> 32) == ep_epoch;
                    ps[s] = make_float4(__uint_as_float((uint32_t)lo.x), __uint_as_float((uint32_t)lo.y), __uint_as_float((uint32_t)hi.x),
                                        __uint_as_float((uint32_t)hi.y));
                }
            }
            if (!ok && (clock64() - t0 > EP_WAIT_CYCLES || (errp && *reinterpret_cast<volatile uint32_t *>(errp) != 0u))) {
                if (errp) atomicCAS(errp, (uint32_t)DEV_ERR_NONE, (uint32_t)DEV_ERR_PEER_TIMEOUT);
                break;
            }
        }
    }
    BRRR_STAMP(a.f.state, 242);
    // ---- the exact routing: the router publishes sequence-tagged words; one lane per word polls
    // (bounded) until its word carries this launch's sequence number
    if (tid < 32) {
        uint32_t payload = 0u;
        if (a.router_seq) {
            if (tid < 16 && (tid & 7) < topk) {
                const volatile unsigned long long *w = a.f.state->route_pub + tid;
                bool ok = false;
                const long long t0 = clock64();
                do {
                    for (int i = 0; i < 64 && !ok; i++) {
                        const unsigned long long v = *w;
                        ok = (uint32_t)(v >> 32) == want_seq;
                        payload = (uint32_t)v;
                    }
                    // give up at once when the error word is already set (an earlier wait of this step ran out)
                } while (!ok && clock64() - t0 < WAIT_CYCLES && *reinterpret_cast<volatile uint32_t *>(&a.f.state->err) == 0u);
                if (!ok) {
                    // the step is void from here: record where, so that the host can run it again without speculation
                    atomicCAS(&a.f.state->err, (uint32_t)DEV_ERR_NONE, (uint32_t)DEV_ERR_PEER_TIMEOUT);
                    atomicMin(&a.f.state->spec_fail_step, a.f.state->n_out);
                }
            }
        } else if (tid < 16 && (tid & 7) < topk) {
            payload = tid < 8 ? (uint32_t)__ldcg(a.f.top + tid) : __float_as_uint(__ldcg(a.f.wts + (tid - 8)));
        }
        __syncwarp();
        if (tid >= 8 && tid < 8 + topk) wts_sh[tid - 8] = __uint_as_float(payload);
        if (tid < topk) {
            const int want = (int)payload;
            int slot = tid;
            if (a.f.est) {
                slot = -1;
                for (int s = 0; s < topk; s++) if (sel[s] == want) slot = s;
                if (slot < 0) {                  // the estimate missed this expert: flag the step, keep going
                    slot = 0;
                    if (a.f.state) atomicMin(&a.f.state->spec_fail_step, a.f.state->n_out);
                }
            }
            slot_of[tid] = slot;
            if (!a.f.est) sel[tid] = want;
        }
    }
    BRRR_STAMP(a.f.state, 243);
    __syncthreads();
    BRRR_STAMP(a.f.state, 244);
    if (!a.f.est) {      // exact routing only: the biases could not be fetched ahead
#pragma unroll
        for (int s = 0; s < MAXS; s++) pb[s] = (live && s < topk) ? reinterpret_cast<const float4 *>(a.f.down_b + (size_t)sel[s] * d)[tid] : zero4;
    }
    if (live) {
        float4 acc = xr;
        for (int kk = 0; kk < topk; kk++) {
            const int sl = slot_of[kk];
            const float w = wts_sh[kk];
            float4 p = ps[0], bb = pb[0];
            switch (sl) {                    // uniform over the block: a branch, not a chain of selects
            case 1: p = ps[1]; bb = pb[1]; break;
            case 2: p = ps[2]; bb = pb[2]; break;
            case 3: p = ps[3]; bb = pb[3]; break;
            default:
                if (MAXS > 4) {
#pragma unroll
                    for (int q = 4; q < MAXS; q++) if (q == sl) { p = ps[q]; bb = pb[q]; }
                }
            }
            acc.x = __fadd_rn(acc.x, __fmul_rn(w, __fadd_rn(p.x, bb.x)));
            acc.y = __fadd_rn(acc.y, __fmul_rn(w, __fadd_rn(p.y, bb.y)));
            acc.z = __fadd_rn(acc.z, __fmul_rn(w, __fadd_rn(p.z, bb.z)));
            acc.w = __fadd_rn(acc.w, __fmul_rn(w, __fadd_rn(p.w, bb.w)));
        }
        reinterpret_cast<float4 *>(a.f.x)[tid] = acc;
        reinterpret_cast<float4 *>(xf)[tid] = acc;
    }
    BRRR_STAMP(a.f.state, 245);
    if (a.norm_w) {
        __syncthreads();
        BRRR_STAMP(a.f.state, 246);
        block_norm_quant_staged<NQ_NATURAL, 1>(a.norm_w, wreg, a.eps, d, xf, reinterpret_cast<int2 *>(a.nq), a.ns, &inv_sh, tid, FN_THREADS);
    }
    BRRR_STAMP(a.f.state, 247);
    if (tid == 0 && a.fold_seq) *a.fold_seq = want_seq;
    BRRR_GT_END(a.f.state, 240);
}

size_t xt_smem_bytes(int np) {
    return (size_t)XT_STAGES * XT_STAGE + (size_t)np * XT_B_PAIR + (size_t)(np + XT_CH - 1) / XT_CH * XT_CH * 2 * 8 + (size_t)(2 * XT_STAGES + 2 * XT_REGIONS) * 8;
}

}  // namespace

// ---------------------------------------------------------------- launchers
size_t mxt_bytes(int experts, int tiles_per_expert, int np) { return (size_t)experts * tiles_per_expert * xt_run_bytes(np); }

void launch_mxt_pack(MxDev a, MxDev b, int experts, int rows_per_expert, MxtDev out, cudaStream_t st) {
    PackArgs p{};
    p.a = a; p.b = b; p.rows_per_expert = rows_per_expert; p.tiles_per_expert = out.tiles_per_expert; p.out = out;
    const size_t words = mxt_bytes(experts, out.tiles_per_expert, out.np) / 4;
    if (!words) return;
    mxt_pack_kernel<<<(unsigned)((words + 255) / 256), 256, 0, st>>>(p, words);
}

void launch_xt_digits(const int8_t *xq, int nb, uint8_t *dig, cudaStream_t st) {
    if (nb > 0) xt_digits_kernel<<<(nb + 3) / 4, 128, 0, st>>>(xq, nb, dig);
}

void launch_mx_exp_scan(const uint8_t *raw, size_t blocks, uint32_t *bad, cudaStream_t st) {
    if (blocks) mx_exp_scan_kernel<<<148 * 8, 256, 0, st>>>(raw, blocks, bad);
}

// A down CTA has the footprint of a gate/up CTA: it fits beside a running one, sets up and starts its weight stream there, before gate/up has finished.
template <bool DOWN, bool EP, bool WIDE>
static cudaError_t xt_launch_form(const XtArgs &a, dim3 grid, bool pdl, cudaStream_t st) {
    static unsigned long long configured = 0;      // one bit per device
    const cudaError_t e = smem_optin(xt_expert_kernel<DOWN, EP, WIDE>, 200 * 1024, configured);
    if (e != cudaSuccess) return e;
    return launch_k(xt_expert_kernel<DOWN, EP, WIDE>, grid, dim3(XT_THREADS), xt_smem_bytes(a.w.np), st, pdl, a);
}
template <bool DOWN>
static cudaError_t xt_launch(const XtArgs &a, dim3 grid, bool pdl, cudaStream_t st) {
    if (a.w.wide) return a.ep_on ? xt_launch_form<DOWN, true, true>(a, grid, pdl, st) : xt_launch_form<DOWN, false, true>(a, grid, pdl, st);
    return a.ep_on ? xt_launch_form<DOWN, true, false>(a, grid, pdl, st) : xt_launch_form<DOWN, false, false>(a, grid, pdl, st);
}

cudaError_t launch_gate_up_t(MxtDev gu, const float *gate_b, const float *up_b, const int32_t *top, const float *est, int ne, int topk,
                             int d, const uint8_t *xdig, const float *xs, int8_t *hq, float *hs, uint8_t *hdig, DevState *state,
                             bool pdl, cudaStream_t st, const EpCtx *ep, int layer) {
    XtArgs a{};
    if (ep) { a.ep_on = 1; a.ep = *ep; a.layer = layer; }
    a.w = gu; a.bias_a = gate_b; a.bias_b = up_b; a.top = top; a.est = est; a.ne = ne; a.topk = topk; a.d = d;
    a.bdig = xdig; a.xs = xs; a.hq = hq; a.hs = hs; a.hdig = hdig; a.state = state;
    return xt_launch<false>(a, dim3(gu.tiles_per_expert, topk), pdl, st);
}

cudaError_t launch_down_t(MxtDev down, const float *down_b, const int32_t *top, const float *wts, const float *est, int ne, int topk,
                          int d, const uint8_t *hdig, const float *hs, float *x, float *part, uint32_t *counter, DevState *state,
                          bool pdl, cudaStream_t st, const EpCtx *ep, int layer) {
    XtArgs a{};
    if (ep) { a.ep_on = 1; a.ep = *ep; a.layer = layer; }
    a.w = down; a.bias_a = down_b; a.top = top; a.wts = wts; a.est = est; a.ne = ne; a.topk = topk; a.d = d;
    a.bdig = hdig; a.xs = hs; a.x = x; a.part = part; a.counter = counter; a.state = state;
    return xt_launch<true>(a, dim3(down.tiles_per_expert, topk), pdl, st);
}

cudaError_t launch_down_fold(const int32_t *top, const float *wts, const float *est, int ne, int topk, int d, const float *part,
                             const float *down_b, float *x, DevState *state, bool pdl, cudaStream_t st) {
    FoldArgs a{};
    a.top = top; a.wts = wts; a.est = est; a.ne = ne; a.topk = topk; a.d = d; a.dpad = (d + 127) / 128 * 128;
    a.part = part; a.down_b = down_b; a.x = x; a.state = state;
    return launch_k(xt_fold_kernel, dim3((d + 127) / 128), dim3(128), 0, st, pdl, a);
}

cudaError_t launch_fold_norm(const int32_t *top, const float *wts, const float *est, int ne, int topk, int d, const float *part,
                             const float *down_b, float *x, const float *next_norm_w, float eps, int8_t *nq, float *ns,
                             uint32_t *router_seq, uint32_t *fold_seq, DevState *state, bool pdl, cudaStream_t st, const EpCtx *ep, int layer) {
    if (d > 4 * FN_THREADS || d % 32 || topk > 8 || (router_seq && !state)) return cudaErrorInvalidValue;
    FoldNormArgs a{};

    a.f.top = top; a.f.wts = wts; a.f.est = est; a.f.ne = ne; a.f.topk = topk; a.f.d = d; a.f.dpad = (d + 127) / 128 * 128;
    a.f.part = part; a.f.down_b = down_b; a.f.x = x; a.f.state = state;
    a.norm_w = next_norm_w; a.eps = eps; a.nq = nq; a.ns = ns; a.router_seq = router_seq; a.fold_seq = fold_seq;
    if (ep) { a.ep_pairs = ep->pairs[ep->rank] + (size_t)layer * topk * d; a.ep_epoch = ep->epoch; a.ep_lo = ep->e_lo; a.ep_cnt = ep->e_cnt; }
    const size_t smem = (size_t)d * sizeof(float);
    if (ep) return topk <= 4 ? launch_k(xt_fold_norm_kernel<4, true>, dim3(1), dim3(FN_THREADS), smem, st, pdl, a)
                             : launch_k(xt_fold_norm_kernel<8, true>, dim3(1), dim3(FN_THREADS), smem, st, pdl, a);
    if (topk <= 4) return launch_k(xt_fold_norm_kernel<4, false>, dim3(1), dim3(FN_THREADS), smem, st, pdl, a);
    return launch_k(xt_fold_norm_kernel<8, false>, dim3(1), dim3(FN_THREADS), smem, st, pdl, a);
}

}  // namespace brrr
