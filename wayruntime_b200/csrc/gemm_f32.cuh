// gemm_f32.cuh — F32 matrix product for many activation rows on the tensor cores (prompts of the F32 stacks).
#pragma once

#include <cuda.h>

#include "gemm_bf16.cuh"
#include "wr_internal.cuh"

// An F32 row as four signed digits of base 256 per value: the row is scaled by a power of two that puts its largest magnitude
// into [2^30, 2^31) (of a few rows [2^29, 2^30), so that all digits lie within [-128, 127]) and rounded to integers.  A value is
// within 2^-31 of the row's largest value: all of its 24 bits are there down to 2^-7 of it, and the row as a vector is off by less
// than sqrt(k) 2^-31 of its length.
//
// Digits of 64 values take 256 bytes: 64 of each of two digits, and, elsewhere, 64 of each of the other two.
// Weights: digits 0 and 2 in wr_weight's 128-byte pieces (gemm_bf16.cuh), then digits 1 and 3 likewise, so that digits 0 and 1
// (2 and 3) of a tile's rows are one operand of twice the rows.
struct wr_split_weight {
    char *blocks = nullptr;
    int *exponent = nullptr;             // [n]: of the power of two that undoes the row's scale and the digits' unit; or one of the next two
    uint32_t n = 0, k = 0;
};
// A row with infinities, products with which are worked out from the F32 rows; a row with NaNs, products with which are NaN.  (No sum of
// two exponents comes near either, nor two of the first to the second.)
constexpr int kNotFinite = 1 << 20, kNotNumbers = 1 << 22;
size_t wr_split_weight_bytes(uint32_t n, uint32_t k);
// byte offset of digit `digit` of value i of a row
__host__ __device__ inline size_t wr_split_off(uint32_t n, uint32_t k, uint32_t row, uint32_t digit, uint32_t i)
{
    const uint32_t piece = (digit >> 1) * 4 + i % kWBlock / 16, kb = (digit & 1u) * wr_weight_blocks(k) + i / kWBlock;
    return wr_weight_row(n, row, kb) + ((piece ^ (row & 7u)) << 4) + i % 16;
}

// Rows of one split weight, from up to three F32 matrices [n_i][k] one below the other, or (pair) from gate and up
// rows eight by eight, so that a gate value and its up value lie eight columns apart.
struct wr_split_source {
    wr_split_weight to;
    const float *src[3];
    uint32_t n[3];
    uint32_t pair;
};
// The F32 row that a split weight's row comes from; null: a row of zeros
__host__ __device__ inline const float *wr_split_row(const wr_split_source &s, uint32_t row)
{
    uint32_t at = row, j = 0;
    if (s.pair) {
        at = row / 16 * 8 + row % 8;
        j = row / 8 & 1;
    } else {
        while (j < 2 && at >= s.n[j]) at -= s.n[j++];
    }
    return at < s.n[j] ? s.src[j] + (size_t)at * s.to.k : nullptr;
}
constexpr uint32_t kSplitSources = 4;
int wr_split_weights_launch(wr_cuda_ctx *ctx, const wr_split_source *list, uint32_t count);

// Activations: rows of digits, `ld` 16-bit places apart: digits 0 and 1 of row r at r, 2 and 3 at pad + r.
inline uint32_t wr_split_ld(uint32_t k) { return (k + kWBlock - 1) / kWBlock * kWBlock; }
struct wr_split_scale {
    float factor;                        // what a product of the row is multiplied by last (1 / rms)
    int exponent;                        // of the power of two that undoes the row's scale, or as for weights
};
struct wr_split_rows_args {
    float *x;                            // [rows][x_stride]; gets the partial sums added when there are any
    uint32_t x_stride, k, rows;
    const float *parts;                  // [n_parts][rows][k] added to x in this order, or null
    uint32_t n_parts;
    const float *norm_w;                 // RMSNorm: x * norm_w is split, 1/rms is the factor; or null
    float eps;
    __half *out;                         // null: only the sums are added
    uint32_t ld, pad;
    wr_split_scale *row_scale;           // [rows]
};
int wr_split_rows_launch(wr_cuda_ctx *ctx, const wr_split_rows_args &a);

struct wr_f32_gemm_seg {
    float *out;                          // [m][ld], columns of this segment
    uint32_t n, ld;                      // n and ld multiples of 4
};
struct wr_f32_gemm_args {
    wr_split_source source;              // the weight, and what it came from; pair: seg[0].out gets SiLU(gate) * up, n / 2 columns
    const float *x, *norm_w;             // what the rows were split from (as it still is), and its norm's weight or null
    uint32_t x_stride;
    uint32_t m, pad;                     // rows; rows between the first two digits of the activations and the others
    const wr_split_scale *row_scale;
    wr_f32_gemm_seg seg[3];              // the weight's rows in order
    uint32_t n_seg;
    uint32_t k_parts;                    // > 1: seg[0].out is [k_parts][m][n], one sum per part of K
};
// How many parts K is cut into for a weight of n rows: a rule on the weight alone, so that a row's bits do not depend
// on how many rows the call has.
uint32_t wr_f32_gemm_k_parts(uint32_t n, uint32_t k);
bool wr_f32_gemm_covers(uint32_t k, uint32_t k_parts);
// x: map of the split rows, wr_split_ld(k) places wide
int wr_f32_gemm_launch(wr_cuda_ctx *ctx, const CUtensorMap &x, const wr_f32_gemm_args &a);
