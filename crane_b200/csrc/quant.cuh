// GGUF-quantised linear layers (Q4_K / Q6_K / Q8_0): GEMV on the quantised bytes for up to four rows (quant.cu),
// integer dots on the tensor cores for more (qgemm.cu), expansion of blocks to bf16.
#pragma once

#include "decode.cuh"

namespace cb {

// ggml_type values of the formats handled (crane-core/src/ops/linear.rs:55-78 `parse_ggml_dtype`)
enum QType : int { QT_NONE = 0, QT_Q8_0 = 8, QT_Q4_K = 12, QT_Q6_K = 14 };

// Device layout per 256 elements ("super-block"); Q4_K is ggml's own 144-byte block, the other two are repacked at load
// so every field is 16-byte aligned:
//   Q4_K : [f16 d][f16 dmin][12 B scales][128 B nibbles]                                  144 B (unchanged)
//   Q6_K : [128 B ql][64 B qh][16 x i8 scales][f16 d][14 B pad]                           224 B (ggml: 210 B)
//   Q8_0 : [256 x i8][8 x f16 d]                                                          272 B (ggml: 8 x 34 B)
__host__ __device__ inline int q_sb_bytes(int qt) { return qt == QT_Q4_K ? 144 : qt == QT_Q6_K ? 224 : qt == QT_Q8_0 ? 272 : 0; }
inline int q_src_block_bytes(int qt) { return qt == QT_Q4_K ? 144 : qt == QT_Q6_K ? 210 : qt == QT_Q8_0 ? 34 : 0; }
inline int q_src_block_elems(int qt) { return qt == QT_Q8_0 ? 32 : 256; }

// Host: repack `rows` rows of K elements from the ggml byte layout into the device layout (dst sized rows * K/256 * q_sb_bytes).
void q_repack_rows(int qt, const unsigned char* src, unsigned char* dst, size_t rows, int K);

// Further matrices of a GEMV launch (k and v of q's type beside q, which saves two launches a layer): n[i] rows of w[i], results one behind the other's.  n = 0: none.
struct QMore { const unsigned char* w[2] = {nullptr, nullptr}; int n[2] = {0, 0}; };

struct QGemvArgs {
    GemvArgs g;        // W is reinterpreted as the quantised bytes; g.x, g.ldx, and (nullable) g.norm_w with g.eps: the activation rows; epilogue fields as for the bf16 GEMV
    int qtype;
    int epi;           // GemvEpi
    QMore more;        // (GEMV_STORE only)
    int rpc[3];        // rows of each matrix per CTA (set by the launch)
    const unsigned char* xq;   // the rows quantised by xquant_launch (norm included), or nullptr: the kernel quantises them itself
};

// The activation block rule candle pairs with the weight type: XQ_Q8_K for Q4_K / Q6_K, XQ_Q8_0 for Q8_0 (see xq_block).
enum XQMode : int { XQ_Q8_0 = 0, XQ_Q8_K = 1 };
__host__ __device__ constexpr int xq_mode_for(int qt) { return qt == QT_Q8_0 ? XQ_Q8_0 : XQ_Q8_K; }

// Quantise B activation rows (f32, row stride ldx; RMS-normalised with norm_w first when non-null) for qgemv_launch.
size_t xquant_bytes(int B, int K);
int xquant_launch(cudaStream_t st, int B, const float* x, int ldx, int K, const float* norm_w, float eps, int mode, unsigned char* out, bool pdl);
// Does a launch of its own quantise the rows?  One row in front of Q8_0 weights is quantised by every CTA of the GEMV for itself, up to 32 super-blocks (two per
// warp); more rows, and the K-quants' blocks, whose largest value is looked for over the whole warp, are the shorter way apart.
// us a call of four steps, two layers, in the GEMV / apart: Q8_0 one token of width 1024 (4 - 12 super-blocks) 390 / 405, 2048 (8 - 24) 449 / 492, 4096 (16, 48) 679 / 712;
// two of 1024 (8 - 24) 482 / 485, of 2048 (16, 48) 583 / 544; four of 1024 (16 - 48) 608 / 560, of 2048 (32, 96) 706 / 642.  Q4_K_M one of 1024 443 / 432, of 2048 485 / 470, of
// 4096 (16, 48) 738 / 715; two of 2048 616 / 578; four of 2048 815 / 691.
constexpr bool xquant_apart(int B, int K, int qt) { return B > 1 || qt != QT_Q8_0 || K / 256 > 32; }

int qgemv_launch(cudaStream_t st, int B, const QGemvArgs& a, int num_sms, bool pdl);

// ---- many rows (qgemm.cu): the same codes as f16 integers, for the tensor cores ----
// From this many rows on: five are 4 + 1 through the GEMVs, six 4 + 2.  us per call of two layers, here / GEMVs, widths 1024, 2048, 4096:
//   Q4_K_M  5 rows 207 / 222, 230 / 257, 325 / 372
//   Q8_0    5 rows 213 / 210, 250 / 241, 377 / 356   6 213 / 217, 249 / 245, 374 / 366   7 214 / 277, 250 / 316, 375 / 476
constexpr int qrows_min(int qt) { return qt == QT_Q8_0 ? 7 : 5; }
// `rows` (a capacity) activation rows of up to K columns.  codes [rows, K] f16, elements of every group of four in the order 0, 2, 1, 3 (the order
// in which the weights' bytes unpack in pairs); dx [blocks][ldd] the blocks' scales (256 or 32 elements); bsum [rows, K / 16] f16, per super-block
// the eight 32-element sums mod 64 and their quotients by 64 (Q8_K codes only)
struct QRows { unsigned short* codes; float* dx; unsigned short* bsum; int ldd; };
size_t qrows_bytes(int rows, int K);
QRows qrows_at(unsigned char* buf, int rows, int K);
int xquant_rows_launch(cudaStream_t st, int M, const float* x, int ldx, int K, const float* norm_w, float eps, int mode, const QRows& out, bool pdl);
// y[m, n] = epi(sum_k W[n, k] x[m, k]); epi: GEMV_STORE, GEMV_RESID or GEMV_SILU_MUL (rows of W interleaved); x quantised for W's type
int qgemm_launch(cudaStream_t st, int qt, const unsigned char* w, const QRows& x, int M, int N, int K, int epi, float* y, int ldy, bool pdl);
// activation rows of a tile for such a linear (16, 32, 64 or 128)
int qgemm_rows(int qt, int M, int N, int K);
// several matrices of the same codes (GEMV_STORE): those whose CTAs fit the chip together share a launch.  *launches = how many there were
struct QMany { int qt; const unsigned char* w; int N; float* y; int ldy; };
int qgemm_many_launch(cudaStream_t st, const QMany* m, int n, const QRows& x, int M, int K, bool pdl, int* launches);
// rows x K quantised -> bf16 row-major
int q_dequant_bf16_launch(cudaStream_t st, int qt, const unsigned char* w, size_t rows, int K, bf16* out);
// gather + dequantise rows of a quantised embedding table to f32: ids[rows] (prefill) or, with ids == nullptr, state[r].token
int embed_rows_q_launch(cudaStream_t st, int qt, const unsigned char* table, int H, const uint32_t* ids, const SeqState* state, int rows,
                        float* x, bool pdl);

}  // namespace cb
