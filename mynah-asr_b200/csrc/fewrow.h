// A chain of few-row operations as one persistent kernel (fewrow.cu): the layer stack of a streaming step, or all
// positions of an AED decode.
#pragma once
#include <vector>

#include "common.cuh"
#include "gemm.h"
#include "qweight.h"

namespace mb {

enum { FR_GEMM = 0, FR_STREAM_ATTN = 1, FR_AED_SELF = 2, FR_AED_CROSS = 3 };
// the rows of a contraction (`rows` of FrOp)
enum { FR_ROWS_PLANES = 0,   // fp16 (hi, lo) planes [M, K] as they are
       FR_ROWS_LN = 1,       // LayerNorm(x; ln), x [M, K] f32
       FR_ROWS_LN2 = 2,      // y = LayerNorm(x; ln0), kept in x_copy; then LayerNorm(y; ln)
       FR_ROWS_LN_SILU = 3,  // SiLU(LayerNorm(x; ln))
       FR_ROWS_AED_NEXT = 4  // the turn to the next AED position: selection, embedding, LN2 of it
};
enum { FR_EPI_PLANES = 0,    // act(y + bias) as planes
       FR_EPI_RESID = 1,     // out = res + alpha (y + bias)
       FR_EPI_QKV = 2,       // columns below n_split: f32 out; the others: fp16 o_hi (first half) and o_lo (second half)
       FR_EPI_F32 = 3,       // out = y + bias
       FR_EPI_GLU_CONV = 4,  // streaming conv middle: GLU, depthwise taps over the cached rows, cache update; out f32
       FR_EPI_ARGMAX = 5     // per group of columns the first maximum of every row
};

struct alignas(16) FrOp {
    int type, rows, epi, act;
    int N, K, n_split, ldo;
    float alpha;
    int conv_k, ldq, ldrk;
    const uint8_t *w;                     // tiles (fr_retile)
    const float *bias;
    const float *x, *ln_w, *ln_b, *ln0_w, *ln0_b;
    float *x_copy;
    const __half *a_hi, *a_lo;            // planes of a contraction's rows; FR_AED_CROSS: (K | V) planes by (utterance, head)
    float *out;
    const float *res;
    __half *o_hi, *o_lo;
    const float *dw_w;                    // [d, conv_k]
    float *conv_cache;                    // [S][conv_k - 1][d]
    // attention: q [M, ldq] f32; streaming: chunk rows kn / vn, rings kc / vc, position keys rk; AED: f32 caches ck / cv
    const float *q;
    const __half *kn, *vn, *rk;
    __half *kc, *vc;
    const float *bias_u, *bias_v;
    float *ck, *cv;
};

struct FrArgs {
    const FrOp *ops;                      // device; these three are fr_launch's
    int n_ops;
    double inv_d;
    int M;                                // rows
    int tile_rows;                        // rows of a row tile (at most 16, whole streams)
    int mtiles, ngroups;                  // grid = mtiles x ngroups CTAs
    int terms;                            // 3: hi and lo planes of the activations; 1: hi only
    int d, H, dk;
    unsigned *bar;                        // [FR_BAR_WORDS]
    int *status;
    // streaming
    int S, Q, left, valid;
    const int *d_start;
    // AED
    int positions;                        // 0: the ops once; else positions 0 .. positions
    int V, B, eos, cap_stride, max_prompt, max_seq, max_len;
    int *st;                              // [cur | n_out | done | n_prompt | max_len | cap] x B, then n_done
    const int *prompts;
    int *tokens;
    const float *emb, *pos;
    float *cand_v;                        // [M][ngroups]
    int *cand_i;
    const int *enc_off, *enc_len;
    size_t v_off;
};

// Weights as the kernel reads them: units of eight rows, in every unit pairs of 32-element blocks of 544 bytes: the int8
// quants in fragment order, then the f16 block scales. Q8_0 blocks as they are; Q4_0 blocks with the nibbles widened
// (same values). glu: rows c and c + n / 2 (the two halves of a GLU) side by side, four of each in a unit.
bool fr_can_tile(const QWeight &w);
size_t fr_tile_bytes(int n, int k);
int fr_retile(const QWeight &w, uint8_t *dst, bool glu, cudaStream_t st);

static constexpr int FR_MAX_ROWS = 128;   // rows of an AED batch
static constexpr int FR_MAX_LAYERS = 48;  // encoder layers a chain has room for
static constexpr int FR_BAR_WORDS = 32 * (1 + FR_MAX_ROWS);   // the abort flag, then a counter per row tile, in a line each
bool fr_attn_fits(int dk);
int fr_grid(int M, int tile_rows, int *mtiles, int *ngroups);
size_t fr_table_bytes(size_t n_ops);
std::vector<uint8_t> fr_table(const std::vector<FrOp> &ops);              // what the kernel reads, to be copied to the device
int fr_launch(FrArgs a, const std::vector<FrOp> &ops, const void *table, cudaStream_t st);

}  // namespace mb
