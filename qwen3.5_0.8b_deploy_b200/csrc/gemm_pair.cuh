// Prompt-sized products on pairs of CTAs with their element-wise successor in the epilogue (gemm_pair.cu).
#pragma once

#include "kernels.cuh"

namespace b200 {

// act[rows, ff] = f(gate) * up of X[rows, K] W[2 ff, K]^T; W holds the gate rows in front of the up rows (`split`) or groups of 32 gate and 32 up
// rows.  f: act_kind (B200ATTN_ACT_*); SiLU for fp16.
bool gemm_glu_takes(ElemType t, const void* x, const void* w, const void* act, int rows, int ff, int K);
int gemm_glu(cudaStream_t s, ElemType t, int act_kind, const void* x, const void* w, void* act, int rows, int ff, int K, bool split, int* error);

// Y[rows, out] = X[rows, in] W[out, in]^T, X and Y with row pitches.  fp32 results, or bf16 ones of bf16 operands; `takes`: where it is the faster route as well.
bool gemm_pair_takes(const void* x, int ldx, const void* w, const void* y, int ldy, ElemType in_type, ElemType out_type, int rows, int out, int in);
int gemm_pair(cudaStream_t s, const void* x, int ldx, const void* w, void* y, int ldy, ElemType in_type, ElemType out_type, int rows, int out, int in, int* error);

// The DeltaNet input projection of prompts with its convolution: X[rows, 1024] W[8224, 1024]^T, then for every token q, k, v (conv + SiLU, L2 norms,
// q / sqrt(128)) as fp16; z and the gates' inputs go to their columns of mixed [rows, 8224], and so do the unconvolved q, k, v of each sequence's last
// three rows (launch_la_conv_tail).  The sequences' rows follow one another without gaps.
struct LaConvArgs {
    const LaSeqMeta* seqs;
    int n_seqs;
    const float* conv_state;       // of the layer, conv_stride floats a slot
    size_t conv_stride;
    const float* conv_w;
    __half *q, *k, *v;
    float* mixed;
};
bool gemm_la_conv_takes(const void* x, const void* w, long long rows, int n_seqs);
int gemm_la_conv(cudaStream_t s, const __half* x, const __half* w, int rows, const LaConvArgs& la, int* error);

}  // namespace b200
