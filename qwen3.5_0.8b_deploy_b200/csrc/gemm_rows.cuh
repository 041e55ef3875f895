// Projections of a decode step over a few rows (gemm_rows.cu).
#pragma once

#include "common.cuh"

namespace b200 {

constexpr int kRowsGemmMax = 16;        // rows a launch takes (the figures: gemm_rows.cu)
enum { kRowsStore = 0, kRowsSwiglu, kRowsGeglu, kRowsArgmax, kRowsResidual, kRowsDeepStore };    // the last two: deep K, fp32 Y

// How X comes in: 16-bit rows; fp32 rows to normalise; fp32 rows to which normalised rows `add` are added first, the sums also going to x_out
// (row m from CTA m); fp32 rows to round; what rounding them to fp16 takes away, times kLoScale.
enum { kLoadAsIs = 0, kLoadNorm, kLoadAddNorm, kLoadF32, kLoadF32Lo };

struct RowsGemm {
    const void* x = nullptr;            // [M, K]
    int ldx = 0;
    const int* row_index = nullptr;     // row m of X is x + row_index[m] * ldx
    const void* w = nullptr;            // [N, K]; gated: gate and up rows in alternating groups of `group` rows
    int M = 0, N = 0, K = 0;
    const float* norm_w = nullptr;      // the normalised columns are multiplied by norm_base + norm_w, null: by one
    float norm_base = 0.f;
    float eps = 0.f;
    const float* add = nullptr;         // [M, K] fp32: X = x + norm(add), kept in x_out (another buffer than x)
    float* x_out = nullptr;
    float scale = 1.f, cap = 0.f;       // store: y = cap tanh(scale v / cap), no cap at 0
    bool accumulate = false;            // store, fp32: added to what is there
    void* y = nullptr;                  // store: [M, N]; gated: [M, N / 2]; residual: fp32 [M, N], added to
    int ldy = 0;
    int group = 0;
    unsigned long long* packed = nullptr;   // argmax words of M rows (see gemm_tc_argmax)
    int* error = nullptr;
    bool late = false;                  // let the next launch in only after this one's dependency wait
    int tiles = 0;                      // most column tiles of a CTA: filled in by the launcher
};

bool gemm_rows_takes(const RowsGemm& a, int epi);
int gemm_rows(cudaStream_t s, const RowsGemm& a, ElemType type, int epi, int load, ElemType out);

}  // namespace b200
