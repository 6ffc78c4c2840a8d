// lin_split_tc.cuh -- launch interface of the f32-activation x bf16-weight contractions (lin_split_tc.cu).
#pragma once
#include "cwk_common.cuh"

// An f32 activation matrix as three bf16 planes [3][n][k] with x = plane 0 + plane 1 + plane 2: each plane is the
// bf16 rounding of what the planes before it leave over, so the three carry 24 bits and more -- the f32 value itself.
constexpr int CWK_PLANES = 3;

struct CwkSplitGemm {
    const uint16_t *A = nullptr;      // planes bf16 [planes][n][lda]
    int planes = CWK_PLANES;          // 3, or 1 for operands that are bf16 to begin with
    int64_t lda = 0;
    int n = 0;                        // tokens
    const uint16_t *W = nullptr;      // bf16 weights, row-major, ldw wide
    int64_t w_rows = 0, ldw = 0;      // the whole matrix (for bounds)
    int rows = 0;                     // output columns per head (or of the whole product)
    int k = 0;                        // contraction length per head
    int heads = 1;                    // > 1: head h reads A columns h*k.. and W rows h*w_head_rows + w_row_off ..
    int64_t w_head_rows = 0, w_row_off = 0;
    bool w_k_rows = false;            // W's rows are the contraction index (y = x . W) instead of the output index (y = W . x)
    const uint16_t *W2 = nullptr;     // a second matrix over the same A, its rows2 outputs behind the first's
    int rows2 = 0;
    int splits = 1;                   // f32 output: parts of the contraction, each its own partial sum
    enum Out { F32, BF16, PLANES } out = F32;
    void *Y = nullptr;                // F32: f32 [splits][n][ldy]; BF16: bf16 [n][ldy]; PLANES: bf16 [3][n][ldy]
    int64_t ldy = 0;
};

// Whether the tensor path takes these operands (shapes, alignment, tensor-map encoder).
bool cwk_split_gemm_ok(const CwkSplitGemm &g);
// How many parts of the contraction keep the SMs busy for an F32 output.
int cwk_split_gemm_splits(const cwk_ctx *ctx, int n, int rows, int rows2, int k);
int cwk_split_gemm(cwk_ctx *ctx, const CwkSplitGemm &g);
// x f32 [n][k] -> planes [3][n][k]
int cwk_split_planes(cwk_ctx *ctx, const float *x, int n, int k, uint16_t *planes);
// sum of `splits` partials [splits][n][cols] -> out f32 [n][cols] (PLANES = false) or planes [3][n][cols]
int cwk_sum_partials(cwk_ctx *ctx, const float *part, int splits, int n, int cols, float *out, uint16_t *planes);
