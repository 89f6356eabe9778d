// What the kernels behind b200_gemm_grouped share: their argument block and the epilogue of one element.
#pragma once
#include <cuda_bf16.h>

#include "b200_serve.h"
#include "common.cuh"

namespace b200 {

struct GG {
    const void* A; const void* W; void* C; const float* aux;
    const int* a_rows; const int* group_off;
    long long lda, ldw, ldc, ld_aux, sA, sW, sC, s_aux;
    int M, N, K, epi;
    float epi_param;
    const float* row_scale;
};

inline bool gg_is_glu(int epi) { return epi == B200_GG_GLU || epi == B200_GG_GLU_GELU || epi == B200_GG_GLU_CLAMP; }

// what becomes of one sum (gated units: v the gate's, v2 the up product's)
__device__ __forceinline__ float gg_value(const GG& g, long long row, int col, float v, float v2, long long aux_off) {
    if (g.row_scale) {   // the row of A was meant to be scaled: the products are linear in it
        const float f = g.row_scale[row];
        v *= f;
        v2 *= f;
    }
    if (g.epi == B200_GG_SIGMOID_MUL) v *= 1.f / (1.f + expf(-g.aux[aux_off + row * g.ld_aux + col]));
    else if (g.epi == B200_GG_GLU) v = v / (1.f + expf(-v)) * v2;
    else if (g.epi == B200_GG_GLU_GELU) v = gelu_tanh_f(v) * v2;
    else if (g.epi == B200_GG_GLU_CLAMP) v = glu_clamp_f(v, v2, g.epi_param);
    else if (g.epi == B200_GG_RELU2) { v = fmaxf(v, 0.f); v *= v; }
    else if (g.epi == B200_GG_BIAS_SOFTPLUS) {
        v += g.aux[aux_off + row * g.ld_aux + col];
        v = v > 20.f ? v : log1pf(expf(v));
    }
    return v;
}
template <typename TC>
__device__ __forceinline__ void gg_store(const GG& g, TC* C, long long row, int col, float v, float v2, long long aux_off) {
    C[row * g.ldc + col] = DT<TC>::from_f(gg_value(g, row, col, v, v2, aux_off));
}

// routed products on tcgen05 (gemm_grouped_tc.cu); -1: not built for this layout
template <typename TC>
int gg_launch_tc(const GG& g, int groups, cudaStream_t s);

}  // namespace b200
