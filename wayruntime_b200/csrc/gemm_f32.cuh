// gemm_f32.cuh — F32 matrix product for many activation rows on the tensor cores (prompts of the dense F32 stack).
#pragma once

#include <cuda.h>

#include "wr_internal.cuh"

// An F32 matrix as two F16 ones: every row is scaled by a power of two that puts its largest magnitude into
// [2^14, 2^15), then hi = F16(x) and lo = F16(x - hi).  hi + lo is within 2^-24 of x (half a unit of F32's last place)
// as long as |x| is above 2^-16 of the row's largest, and within 2^-39 of that one below it.
//
// Weights: hi and lo each in wr_weight's block layout (gemm_bf16.cuh), lo behind hi.
struct wr_split_weight {
    char *blocks = nullptr;              // hi blocks, then lo blocks
    float *unscale = nullptr;            // [n]: 1 / (the row's power of two)
    uint32_t n = 0, k = 0;
};
size_t wr_split_weight_bytes(uint32_t n, uint32_t k);

// Rows of one split weight, from up to three F32 matrices [n_i][k] one below the other, or (pair) from gate and up
// rows eight by eight, so that a gate value and its up value lie eight columns apart.
struct wr_split_source {
    wr_split_weight to;
    const float *src[3];
    uint32_t n[3];
    uint32_t pair;
};
constexpr uint32_t kSplitSources = 4;
int wr_split_weights_launch(wr_cuda_ctx *ctx, const wr_split_source *list, uint32_t count);

// Activations: F16 rows [2 * pad][ld], hi of row r at r, lo at pad + r.
struct wr_split_rows_args {
    float *x;                            // [rows][x_stride]; gets the partial sums added when there are any
    uint32_t x_stride, k, rows;
    const float *parts;                  // [n_parts][rows][k] added to x in this order, or null
    uint32_t n_parts;
    const float *norm_w;                 // RMSNorm: x * norm_w is split, 1/rms goes to row_scale; or null
    float eps;
    __half *out;                         // null: only the sums are added
    uint32_t ld, pad;
    float *row_scale;                    // [rows]: what a product of the split row is multiplied by
};
int wr_split_rows_launch(wr_cuda_ctx *ctx, const wr_split_rows_args &a);

struct wr_f32_gemm_seg {
    float *out;                          // [m][ld], columns of this segment
    uint32_t n, ld;                      // n and ld multiples of 4
};
struct wr_f32_gemm_args {
    uint32_t m, pad;                     // rows; rows between hi and lo of the activations
    const float *row_scale;
    wr_f32_gemm_seg seg[3];              // the weight's rows in order
    uint32_t n_seg;
    uint32_t pair;                       // seg[0].out gets SiLU(gate) * up, n / 2 columns
    uint32_t k_parts;                    // > 1: seg[0].out is [k_parts][m][n], one sum per part of K
};
// How many parts K is cut into for a weight of n rows: a rule on the weight alone, so that a row's bits do not depend
// on how many rows the call has.
uint32_t wr_f32_gemm_k_parts(uint32_t n, uint32_t k);
int wr_f32_gemm_launch(wr_cuda_ctx *ctx, const CUtensorMap &x, const wr_split_weight &w, const wr_f32_gemm_args &a);
