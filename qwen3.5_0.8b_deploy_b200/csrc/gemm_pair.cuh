// Prompt-sized products on pairs of CTAs with their element-wise successor in the epilogue (gemm_pair.cu).
#pragma once

#include "common.cuh"

namespace b200 {

// act[rows, ff] = f(gate) * up of X[rows, K] W[2 ff, K]^T; W holds the gate rows in front of the up rows (`split`) or groups of 32 gate and 32 up
// rows.  f: act_kind (B200ATTN_ACT_*); SiLU for fp16.
bool gemm_glu_takes(ElemType t, const void* x, const void* w, const void* act, int rows, int ff, int K);
int gemm_glu(cudaStream_t s, ElemType t, int act_kind, const void* x, const void* w, void* act, int rows, int ff, int K, bool split, int* error);

}  // namespace b200
