// The two tcgen05 GEMM kernels of the training step (step_gemm.cu) as the step (train_step.cu) calls them.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

// Weights are split into three bfloat16 matrices once per step and kept as shared-memory images: for every 128 output
// columns and every 64 k a block of three 16 KB planes (row n = 64 k = 128 bytes, 128-byte swizzle).
struct WeightSplitJob {
    const float *w;          // [rows, cols] row-major
    const float *gain;       // per-row factor (the gain of the layer norm in front), or null
    int rows, cols;
    int n_is_col;            // 1: image of W (n = column, k = row);  0: image of W^T (n = row, k = column)
    int n0, k0;              // where this matrix starts inside the image (several matrices share one image)
    int n_pad, k_pad;        // extents written, the matrix's own and zeros behind it (the image's end for the last matrix)
    int kb;                  // 64-k blocks of the image
    uint8_t *image;
};
int64_t agpt_weight_image_bytes(int n, int k);
int agpt_split_weights(const WeightSplitJob *jobs, int n_jobs, cudaStream_t st);

// Streams rows through one weight image: out[r, :] = f(A'[r, :] * W), A' = A, (A - mean) * rstd, or A * row scale.
enum RowPro { PRO_PLAIN = 0, PRO_NORM = 1, PRO_SCALE = 2 };
enum RowEpi { EPI_BIAS = 0, EPI_RELU = 1, EPI_MASKED = 2, EPI_ADD = 3, EPI_QKV = 4, EPI_NORM_BWD = 5 };
struct RowGemm {
    int64_t rows = 0;
    int N = 0, K = 0;                   // output columns, contraction (all segments)
    const float *a[3] = {nullptr, nullptr, nullptr};   // column segments of A, each [rows, seg_cols] with leading dimension lda
    int n_seg = 1, seg_cols = 0, lda = 0;
    const uint8_t *image = nullptr;
    int pro = PRO_PLAIN, epi = EPI_BIAS;
    // {mean, 1/std} per row (PRO_NORM, EPI_NORM_BWD) and the row scale: arrays of rows rounded up to 128, zeros behind the end
    const float2 *stats = nullptr;
    const float *row_scale = nullptr;   // PRO_SCALE
    const float *bias = nullptr;        // [N]
    float *out = nullptr;               // [rows, ldo] (all but EPI_QKV)
    int ldo = 0;
    uint32_t *mask_out = nullptr;       // EPI_RELU: bit 31 - c % 32 of word [r, c / 32] is set where the output is > 0
    const uint32_t *mask_in = nullptr;  // EPI_MASKED: such a mask; outputs whose bit is clear become 0
    const float *add = nullptr;         // EPI_ADD, EPI_NORM_BWD: [rows, ldo] added to the output; may be out itself
    float2 *stats_out = nullptr;        // EPI_ADD: {mean, 1/std} of the output rows (N <= 128), or null
    // EPI_QKV: three [rows, N / 3] outputs; q and k rotated by their row's position (cosv null: not rotated)
    void *qkv[3] = {nullptr, nullptr, nullptr};
    int kv_bf16 = 0, head_dim = 0;
    const int32_t *pos = nullptr;
    const float *cosv = nullptr, *sinv = nullptr;       // [positions, head_dim], pair-duplicated
    int n_pos = 0;                      // positions in use
    // EPI_NORM_BWD (N <= 128): the accumulators are the gradient of the normalised rows; out = layer-norm backward (+ add)
    const float *x = nullptr;           // [rows, N], what was normalised
};
int agpt_row_gemm(const RowGemm &g, cudaStream_t st);
bool agpt_row_gemm_rope_fits(int n_pos, int head_dim);

// Contracts over the rows: part[slice] = A'^T * B' for one slice of the rows (A' = A or the normalised A, B' = B or
// B * row scale), and the column sums of B'.
struct RowContract {
    int64_t rows = 0;
    int m = 0, n = 0;                   // columns of A, of B (all segments)
    const float *a = nullptr;
    int lda = 0;
    const float *b[3] = {nullptr, nullptr, nullptr};
    int n_seg = 1, seg_cols = 0, ldb = 0;
    const float2 *stats = nullptr;      // A' = normalised A
    const float *row_scale = nullptr;   // B' = B * scale
    int transposed = 0;                 // 1: partial tiles are stored [n][m]
    float *part = nullptr;              // [slices][m * n]
    float *col_part = nullptr;          // [slices][col_ld] column sums of B' (of A' when transposed), or null
    int col_ld = 0;
    int slices = 0;                     // agpt_row_contract_slices, or agpt_row_contract_shared_slices
};
int agpt_row_contract_units(int m, int n);
int agpt_row_contract_slices(int64_t rows, int m, int n);
int agpt_row_contract_shared_slices(int64_t rows, int units);      // units: those of all contractions of the launch
int64_t agpt_row_contract_most_slices_rows(int units);            // the last row count with a slice per row block
int agpt_row_contract(const RowContract &g, cudaStream_t st);
int agpt_row_contract_many(const RowContract *g, int n, cudaStream_t st);
