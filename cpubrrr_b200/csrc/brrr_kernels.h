// Host-callable launchers of the decode kernels.  Every launcher only enqueues work on the given
// stream (capturable into a CUDA graph) and reports launch-configuration errors through
// cudaGetLastError at the call site.
#pragma once
#include "brrr_dev.cuh"

namespace brrr {

// ---- elementwise / small stages (kernels_small.cu)
void launch_quant_q8(const float *x, int n, int8_t *q, float *s, cudaStream_t st);
cudaError_t launch_rmsnorm_quant(const float *x, const float *w, float eps, int n, float *xn, int8_t *q, float *s, bool pdl, cudaStream_t st);
// ---- token rows (kernels_rows.cu): y[t][r] (+)= row r of m . activation t (+ bias) on the integer units
cudaError_t launch_q8_rows(Q8Dev m, const int8_t *xq, const float *xs, int ntok, const float *bias, float *y, int ldy, int epi, bool pdl, cudaStream_t st);
// residual rows x [rows][d]: part != nullptr: x[t] += sum over k of wts[8 t + k] * part[t * topk + k]; norm_w != nullptr: RMSNorm, Q8 per 32-block (scales s,
// int8 q nullable) and activation image img (nullable; image = TI_HALF or TI_PLANES, brrr_tile.cuh), normalised floats xn (nullable)
cudaError_t launch_rows_norm(float *x, int rows, int d, const float *part, const float *wts, int topk, const float *norm_w, float eps, float *xn, int8_t *q,
                             float *s, uint8_t *img, int image, bool pdl, cudaStream_t st);
// RoPE of every row's k and the cache append of k and v (row t: position row_pos[t] of sequence row_seq[t])
cudaError_t launch_kv_append_rows(const float *qkv, int ldq, int nh, int nkv, float *kc, float *vc, size_t seq_stride, const float *rope,
                                  const int *row_pos, const int *row_seq, int rows, bool pdl, cudaStream_t st);
void launch_embed(const uint16_t *embd, int d, const DevState *state, float *x, cudaStream_t st);
void launch_rows_argmax(const float *logits, int n_vocab, int rows, uint32_t *out, cudaStream_t st);   // out[t] = first index of the largest logit of row t
// ntok rows from token ids in device memory: x[t] = embedding of toks[t]
void launch_embed_tile(const uint16_t *embd, int d, const uint32_t *toks_dev, int ntok, float *x, cudaStream_t st);
void launch_swiglu_quant(const float *gu, int topk, int d, int8_t *hq, float *hs, cudaStream_t st);
void launch_finish_token(DevState *state, cudaStream_t st);
void launch_expf(const float *x, int n, float *y, cudaStream_t st);
// first_elem: index of the first generated element within the whole tensor (MXFP4 only; a multiple of 32)
void launch_synth(uint64_t seed, uint32_t layer, uint32_t kind, uint32_t type, uint64_t nelems, void *out, cudaStream_t st, uint64_t first_elem = 0);

// ---- K-quants of the qwen3moe path (kernels_kq.cu): weights stay in the GGUF byte layout
void launch_quant_q8k(const float *x, int n, int8_t *q, float *s, int32_t *bsum, cudaStream_t st);
void launch_q4k_matvec(const uint8_t *w, int rows, int cols, const int8_t *xq, const float *ys, const int32_t *bsum, float *y,
                       int32_t *dbg, cudaStream_t st);
void launch_q6k_matvec(const uint8_t *w, int rows, int cols, const int8_t *xq, const float *ys, float *y, int32_t *dbg, cudaStream_t st);

// ---- qwen3moe decode kernels (kernels_qwen.cu); KMatDev is declared in brrr_kq.cuh
struct KMatDev;
// Q8_K images of one token: quants, scales per 256, sums per 16.  kernels fetch rows known before their dependency wait ahead of it.
cudaError_t launch_qw_embed(const uint8_t *embd_q4k, int d, DevState *state, float *x, bool pdl, cudaStream_t st);
// norm and image of x in global memory; x_copy (nullable): x as well
cudaError_t launch_qw_norm(const float *x, const float *norm_w, float eps, int d, int8_t *q, float *s, int32_t *b16, float *x_copy, bool pdl, cudaStream_t st);
cudaError_t launch_qw_qkv(const KMatDev *mats, float *const *ys_out, const float *x, const float *norm_w, float eps, DevState *state, bool pdl, cudaStream_t st);
cudaError_t launch_qw_oproj(const KMatDev &wo, const float *act, float *x, DevState *state, bool pdl, cudaStream_t st);      // x += wo . Q8_K(act)
struct QwCache;
cudaError_t qw_cache(float *kc, float *vc, int nkv, QwCache *out);
cudaError_t launch_qw_attn(const QwCache &c, const float *q, const float *k, const float *v, const float *q_norm, const float *k_norm, const float *rope, float eps, int nh,
                           int nkv, DevState *state, float *out, bool pdl, cudaStream_t st);
cudaError_t launch_qw_hint(const float *x, const float *norm_w, float eps, int d, const float *Wt, int ne, float *est, int8_t *q, float *s, int32_t *b16, bool pdl,
                           cudaStream_t st);
// experts: est's topk largest, or top when est is null; hbuf: [slot][ff].  down: x += sum over k of w[k] dot of expert k, with the routing that the
// router publishes as the step's seq-th (est), or top and wts
cudaError_t launch_qw_gate_up(const KMatDev &gate, const KMatDev &up, const float *est, const int32_t *top, int ne, int topk, int ff, const int8_t *q, const float *s,
                              const int32_t *b16, float *hbuf, DevState *state, bool pdl, cudaStream_t st);
cudaError_t launch_qw_down(const KMatDev &down, const float *est, const int32_t *top, const float *wts, uint32_t seq, int ne, int topk, int d, int ff, const float *hbuf,
                           float *x, DevState *state, bool pdl, cudaStream_t st);
// Whether the exact router of a layer always finds room beside the CTAs that wait for its words: this layer's down projection and the next layer's
// q|k|v (next_qkv: three matrices; null behind the last layer).  Not ok: down has to be enqueued behind the router's end.
struct QwRoom {
    int down_ctas, next_ctas;
    size_t down_smem, next_smem, router_smem;
    bool ok;
};
QwRoom qw_router_room(const KMatDev &down, const KMatDev *next_qkv, int ne, int topk, int d, int ff);
cudaError_t launch_qw_head(const KMatDev &head, const int8_t *q, const float *s, const int32_t *b16, float *logits, DevState *state, bool pdl, cudaStream_t st);
// Q6_K rows from the GGUF layout (210-byte superblocks) into the aligned planes of KMatDev (planes = 1)
void launch_q6k_planes(const uint8_t *src, size_t rows, int cols, uint8_t *dst, cudaStream_t st);
// ---- qwen3moe token rows (kernels_qwrows.cu, kernels_kqt.cu): images and handles are described in brrr_kqt.cuh
struct KqtMat;
cudaError_t kqt_matrix(const KMatDev &m, size_t rows_total, KqtMat *out);      // rows_total: rows in memory (experts x rows)
struct KqPlan;
// y[i][..][row] (+)= matrix i (nmat of equal width, stacked) . token row.  plan == nullptr: rows 0 .. ntok - 1 of one matrix; else matrices of
// rows_per_expert rows per expert against the plan's chunks, outputs at the plan's entries (by_entry) or at positions 32 chunk + i
cudaError_t launch_kqt(const KqtMat *const *mats, float *const *ys_out, const int *ldy, int nmat, int rows_per_expert, const KqPlan *plan, int ne, int ntok, int topk,
                       bool by_entry, const uint8_t *img, const float *ys, bool resid, DevState *state, bool pdl, cudaStream_t st);
int kqt_max_chunks(int entries, int ne);
cudaError_t launch_qr_plan(const int32_t *top, int ntok, int topk, int ne, KqPlan *plan, bool pdl, cudaStream_t st);
cudaError_t launch_qr_gather(const KqPlan *plan, const uint8_t *img, const float *ys, int rows, int topk, int ne, int nsb, uint8_t *out, float *out_ys, bool pdl,
                             cudaStream_t st);
cudaError_t launch_qr_embed(const uint8_t *embd, int d, const uint32_t *toks, int rows, float *x, bool pdl, cudaStream_t st);
// part (nullable): x[t] += sum over k of wts[8 t + k] part[t topk + k]; w (nullable): norm and image (ys: scales per superblock), normalised floats xn (nullable)
cudaError_t launch_qr_norm(float *x, int rows, int d, const float *part, const float *wts, int topk, const float *w, float eps, float *xn, uint8_t *img, float *ys, bool pdl,
                           cudaStream_t st);
cudaError_t launch_qr_qknorm(float *q, const float *k, const float *v, const float *q_norm, const float *k_norm, const float *rope, float eps, int nh, int nkv, int pos0,
                             int rows, float *kc, float *vc, bool pdl, cudaStream_t st);
bool qr_attn_fits(int nh, int nkv);       // head groupings the row attention is written for
cudaError_t launch_qr_attn(const float *q, const float *kc, const float *vc, int nh, int nkv, int pos0, int rows, uint8_t *img, float *ys, bool pdl, cudaStream_t st);
cudaError_t launch_qr_glu(const KqPlan *plan, const float *g, const float *u, int entries, int ne, int ff, uint8_t *img, float *ys, bool pdl, cudaStream_t st);
void launch_qr_image(const float *x, int rows, int cols, uint8_t *img, float *ys, cudaStream_t st);
// router of normalised token rows: logits [ntok][ne], routing [ntok][8]; counter: one zeroed word per four tokens
cudaError_t launch_router_rows(const float *xn, int d, const float *Wt, const float *b, int ne, int topk, int ntok, float *logits, int32_t *top, float *wts,
                               unsigned int *counter, DevState *state, bool pdl, cudaStream_t st);
char *host_err_buf();   // thread-local text behind brrr_last_cuda_error (512 bytes)

// ---- Q8 matrices (kernels_q8.cu)
void launch_q8_pack(const uint16_t *w_bf16, int rows_src, int row0_dst, Q8Dev m, cudaStream_t st);
void launch_q8_export(Q8Dev m, int8_t *q, float *s, cudaStream_t st);
enum { Q8_EPI_PLAIN = 0, Q8_EPI_BIAS = 1, Q8_EPI_RESID_BIAS = 2, Q8_EPI_HEAD = 3 };
// Streaming GEMV.  x_f32 != nullptr: RMSNorm(x_f32, norm_w, eps) + Q8 quantisation in the prologue;
// otherwise the Q8 activation (xq, xs) is used.  pdl: launch with programmatic stream serialization.
cudaError_t launch_q8_stream(Q8Dev m, const float *x_f32, const float *norm_w, float eps, const int8_t *xq, const float *xs,
                             const float *bias, float *y, int epi, DevState *state, bool pdl, cudaStream_t st,
                             const float *pf_k = nullptr, const float *pf_v = nullptr, int pf_nkv = 0, int pf_window = 0);

// Direct-from-global GEMV for very large matrices (the vocabulary head); activation pre-quantised.
cudaError_t launch_q8_direct(Q8Dev m, const int8_t *xq, const float *xs, const float *bias, float *y, int epi, DevState *state, bool pdl, cudaStream_t st);
cudaError_t launch_q8_head(Q8Dev m, const int8_t *xq, const float *xs, float *y, DevState *state, bool pdl, cudaStream_t st);

// ---- MXFP4 matrices (kernels_mx.cu)
void launch_mx_pack(const uint8_t *raw, MxDev m, cudaStream_t st);
void launch_mx_gemv(MxDev m, int row0, int nrows, const int8_t *xq, const float *xs, float *y, int32_t *blockdots, cudaStream_t st);
// gate/up of the selected experts + clamped SwiGLU + Q8 of h.  Activation: x_f32 with norm_w
// (RMSNorm + quantise), x_f32 without norm_w (quantise only), or (xq, xs).  gu nullable.
cudaError_t launch_gate_up(MxDev gate, MxDev up, const float *gate_b, const float *up_b, const int32_t *top, int topk, int d,
                           const float *x_f32, const float *norm_w, float eps, const int8_t *xq, const float *xs,
                           int8_t *hq, float *hs, float *gu, DevState *state, bool pdl, cudaStream_t st,
                           const float *est = nullptr, int ne = 0, int e_lo = 0, int e_cnt = 1 << 30);
// e_lo, e_cnt: the matrices hold experts [e_lo, e_lo + e_cnt) only (biases stay indexed by the
// global expert id); CTAs of slots whose expert lives elsewhere return at once.
// est (nullable): slot s of hq/hs belongs to the s-th largest of the router estimate est[0..ne)
// rather than to top[s]; a step whose
// exact experts are not all among them is flagged in state->spec_fail_step.
cudaError_t launch_down_combine(MxDev down, const float *down_b, const int32_t *top, const float *wts, const float *est, int ne,
                                int topk, int d, const int8_t *hq, const float *hs, float *x, DevState *state, bool pdl, cudaStream_t st);

// ---- expert parallelism over NVLink peer memory (kernels_ep.cu)
constexpr int EP_MAX_WORLD = 8;
struct EpCtx {
    int rank, world, e_lo, e_cnt;          // experts [e_lo, e_lo + e_cnt) live on this rank
    uint32_t *epoch;                       // local: number of the step in flight
    float *xchg[EP_MAX_WORLD];             // every rank's exchange buffer [layer][slot][d]
    uint32_t *flags[EP_MAX_WORLD];         // every rank's slice flags [layer][slot][d / 16]
    uint32_t *done[EP_MAX_WORLD];          // every rank's completed-step counters [world]
    // speculative step: every rank's buffer of self-validating row sums [layer][slot][d], one 64-bit
    // word each = (step number << 32) | float bits, written with one store: no flag, no fence
    unsigned long long *pairs[EP_MAX_WORLD];
};
// ---- single-token expert matvecs on the tensor cores in native fp4 (kernels_mxt.cu)
// Tile units: [expert][tile of 128 rows][two block pairs][4096 B operand image per pair | 128 x 4 e8m0 bytes].
constexpr int MXT_PAIR = 4096, MXT_SCALES = 512;
// block exponents whose products with any activation scale, 1e-12 / 127 to FLT_MAX / 127, are exact (kernels_mxt.cu)
constexpr int XT_EXP_MIN = 49, XT_EXP_MAX = 134;
struct MxtDev {
    uint8_t *data;
    int tiles_per_expert, np;
    bool wide;               // a block exponent lies outside that range: scales in the epilogue
};
size_t mxt_bytes(int experts, int tiles_per_expert, int np);
// b.data == nullptr: tiles of 128 rows of a (rows past the end are zero); else rows 0-63 of a tile
// come from a and rows 64-127 from b (same 64 row indices)
void launch_mxt_pack(MxDev a, MxDev b, int experts, int rows_per_expert, MxtDev out, cudaStream_t st);
// *bad |= 1 when `blocks` GGUF blocks hold an exponent outside XT_EXP_MIN .. XT_EXP_MAX (zero blocks may lie below)
void launch_mx_exp_scan(const uint8_t *raw, size_t blocks, uint32_t *bad, cudaStream_t st);
// The activation enters as its digits (brrr_mxt.cuh; [blocks][48] bytes) and its block scales.
void launch_xt_digits(const int8_t *xq, int nb, uint8_t *dig, cudaStream_t st);
// same results, bit for bit, as launch_gate_up / launch_down_combine on the same Q8 activation;
// hdig: [topk][blocks][48] digits of h for launch_down_t
cudaError_t launch_gate_up_t(MxtDev gu, const float *gate_b, const float *up_b, const int32_t *top, const float *est, int ne, int topk,
                             int d, const uint8_t *xdig, const float *xs, int8_t *hq, float *hs, uint8_t *hdig, DevState *state,
                             bool pdl, cudaStream_t st, const EpCtx *ep = nullptr, int layer = 0);
// part: [topk][tiles_per_expert * 128] floats of scratch; counter: [tiles_per_expert] words, zero before the first launch.
// wts != nullptr (exact routing in top/wts, est == nullptr): the last CTA of a row tile folds it onto x.
// wts == nullptr: slot s is the s-th largest entry of est (or top[s]); only part[] is written and
// launch_down_fold finishes the step once the exact routing is there.
cudaError_t launch_down_fold(const int32_t *top, const float *wts, const float *est, int ne, int topk, int d, const float *part,
                             const float *down_b, float *x, DevState *state, bool pdl, cudaStream_t st);
// The fold for a step whose exact router runs on another stream: one CTA waits (bounded) until
// *router_seq == *fold_seq + 1, folds as launch_down_fold, then RMS-normalises the new residual with
// next_norm_w and writes its Q8 image (nq natural int8 order, ns block scales) for the projection
// that follows, and increments *fold_seq.  next_norm_w == nullptr: fold only.
cudaError_t launch_fold_norm(const int32_t *top, const float *wts, const float *est, int ne, int topk, int d, const float *part,
                             const float *down_b, float *x, const float *next_norm_w, float eps, int8_t *nq, float *ns,
                             uint32_t *router_seq, uint32_t *fold_seq, DevState *state, bool pdl, cudaStream_t st,
                             const EpCtx *ep = nullptr, int layer = 0);
cudaError_t launch_down_t(MxtDev down, const float *down_b, const int32_t *top, const float *wts, const float *est, int ne, int topk,
                          int d, const uint8_t *hdig, const float *hs, float *x, float *part, uint32_t *counter, DevState *state,
                          bool pdl, cudaStream_t st, const EpCtx *ep = nullptr, int layer = 0);

// ---- matrices x token rows on the tensor cores (kernels_tile.cu), t < ntok <= BRRR_TILE_MAX, every value bit-identical to the one-token kernels.
// Activations come as images (brrr_tile.cuh), image_bytes(rows, cols, kind) each, and block scales [row][cols / 32].
size_t image_bytes(int rows, int cols, int kind);      // plane images must be zero before their first use
void launch_image(const int8_t *xq, int rows, int cols, int kind, uint8_t *img, cudaStream_t st);      // kind = TI_HALF or TI_PLANES
// Q8 matrix re-laid as operand units (the weights as halves in operand order, 1.9 x the Q8 bytes)
size_t q8_operand_bytes(int rows, int cols);
void launch_q8_operand_pack(Q8Dev m, uint8_t *out, cudaStream_t st);
cudaError_t launch_q8_tile(const uint8_t *op, int rows, int cols, const uint8_t *img, const float *xs, int ntok, const float *bias, float *y, int ldy,
                           int epi, DevState *state, bool pdl, cudaStream_t st);
// y[t * ldy + i] = row (row0 + i) of w . activation t
cudaError_t launch_mx_tile(MxDev w, int row0, int nrows, const uint8_t *img, const float *xs, int ntok, float *y, int ldy, DevState *state, cudaStream_t st);
// per expert the (token, slot) entries routed to it: cnt[ne], list[ne][BRRR_TILE_MAX], entry = token * topk + slot
cudaError_t launch_tile_route(const int32_t *top, int ntok, int topk, int ne, int *cnt, int *list, bool pdl, cudaStream_t st);
// gate and up of every expert for its entries, SwiGLU, Q8 of h: plane images himg [entry] and scales hs [entry][d / 32]
cudaError_t launch_mx_tile_glu(MxDev gate, MxDev up, int ne, int d, const int *cnt, const int *list, int ntok, int topk, const uint8_t *img, const float *xs,
                               const float *gate_b, const float *up_b, uint8_t *himg, float *hs, DevState *state, bool pdl, cudaStream_t st);
// part[entry][d] = down row . h of the entry + bias
cudaError_t launch_mx_tile_down(MxDev down, int ne, int d, const int *cnt, const int *list, int ntok, int topk, const uint8_t *himg, const float *hs,
                                const float *bias, float *part, DevState *state, bool pdl, cudaStream_t st);

void launch_ep_begin(const EpCtx &c, DevState *state, cudaStream_t st);
// down-projection of the local experts, exchange of the 16-row slices, fold in slot order
cudaError_t launch_down_ep(MxDev down, const float *down_b, const int32_t *top, const float *wts, int topk, int d, int layer, const int8_t *hq,
                           const float *hs, float *x, DevState *state, const EpCtx &ep, bool pdl, cudaStream_t st);

// ---- router (kernels_router.cu)
// The router matrix is used in a tiled layout: [32-expert group][tile][32][RT_STRIDE] floats.
constexpr int RT_TJ = 256;                       // tile width (elements of d)
constexpr int RT_STRIDE = RT_TJ + 4;             // padded row stride in floats
constexpr int RT_TILE_FLOATS = 32 * RT_STRIDE;
size_t router_packed_floats(int ne, int d);
void launch_router_pack(const float *W, int ne, int d, float *out, cudaStream_t st);
// x_in is the residual stream when norm_w != nullptr (RMSNorm applied first) or an already
// normalised vector otherwise.
cudaError_t launch_ffn_in(const float *x_in, const float *norm_w, float eps, int d, const float *Wt, const float *b, int ne, int topk,
                          float *logits, int32_t *top, float *wts, unsigned int *counter, DevState *state, bool pdl, cudaStream_t st,
                          int ntok = 1, uint32_t *signal = nullptr, int qwen_norm = 0, int8_t *q8k_q = nullptr, float *q8k_s = nullptr,
                          int32_t *q8k_b16 = nullptr);
size_t ffn_in_smem(int ne, int d);        // dynamic shared memory of one of its CTAs
bool ffn_in_takes_half_an_sm();           // its registers, as built: no more than that
// ntok > 1: a tile of tokens in one launch (token t reads x_in + t * d, writes logits + t * ne, top + 8 t, wts + 8 t, uses counter + t)
// signal (nullable, ntok == 1): a device word the kernel increments after its routing is written, for a
// consumer that runs beside it instead of after it (launch_fold_norm)

// Order-free estimate of the router used only to start the gate/up weight stream early
// (speculative routing): est[ne] receives the estimated logits, xq_out/xs_out the Q8 image of the
// normalised vector (each CTA writes a share).
cudaError_t launch_router_hint(const float *x_in, const float *norm_w, float eps, int d, const float *Wt, const float *b, int ne, int topk,
                               float *est, int8_t *xq_out, float *xs_out, DevState *state, bool pdl, cudaStream_t st,
                               uint8_t *dig_out = nullptr);
// dig_out (nullable): also the digits of the quantised vector for the tensor-core expert kernels

// ---- attention (kernels_attn.cu)
// KV cache layout [n_head_kv][BRRR_MAXSEQ][64].  pos is read from state when state != nullptr,
// else pos_val.  window = 0 means full attention.
cudaError_t launch_attn_rows(const float *qkv, int ldq, const float *kc, const float *vc, size_t seq_stride, const float *rope, const float *sinks,
                             int nh, int nkv, int window, const int *row_pos, const int *row_seq, int rows, float *ao, int8_t *aq, float *as, uint8_t *aimg,
                             float *scores, DevState *err_state, bool pdl, cudaStream_t st);       // rows of one sequence share their K / V tiles (prompt tiles)
cudaError_t launch_attn_decode(const float *qkv, float *kc, float *vc, const float *rope, const float *sinks, int nh, int nkv,
                               const DevState *state, int pos_val, int window, float *ao, int8_t *aq, float *as,
                               DevState *err_state, bool pdl, cudaStream_t st, int pos_off = 0, const int *row_pos = nullptr,
                               const int *row_seq = nullptr, size_t seq_stride = 0, int ldq = 0, int rows = 1, uint8_t *aimg = nullptr);
// aimg (token rows; nullable): the half images of the quantised outputs (brrr_tile.cuh), nh * 128 bytes per row; aq may then be nullptr
// row_pos != nullptr: `rows` tokens in one launch (grid.y), see AttnArgs in kernels_attn.cu; the rows' k / v must be in the cache already
// pos_off is added to the position read from state (ignored with pos_val)

}  // namespace brrr
