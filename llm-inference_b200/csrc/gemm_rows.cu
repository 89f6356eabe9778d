// y[M, N] = x[M, K] W[N, K]^T for up to 16 token rows, fp16 or bfloat16 operands, fp32 sums: one CTA per 16 features (gated units: 16 gate rows and their 16 up
// rows), its eight warps (sixteen above K = 2048) share K in pieces of 32 and meet in shared memory.
//
// What bounds it is the weights' way from HBM and, at the sizes of a decode step (a few MB, 1 to 3 us), everything around it: launch, set-up, the first
// load's latency, the merge. So there is nothing to set up (no tensor maps, barriers, tensor memory or cluster): a lane's 16-byte loads are the fragments of
// mma.sync m16n8k16 as they come (a K index may stand anywhere as long as weights and tokens agree: a lane holds eight consecutive k of its row where the
// instruction thinks of two times two pairs), four pieces per warp are in flight ahead of the products, and the lines of a CTA's weights are prefetched
// to L2 while the launch before is still running (a prefetch reads nothing: what that launch writes is seen all the same).
// Measured at takes_rows (gemm_tcgen05.cu), where the lines to the tcgen05 kernels lie.
#include <cuda_bf16.h>

#include <type_traits>

#include "common.cuh"
#include "launch_count.h"

namespace b200 {

constexpr int kGrAhead = 4;

struct GrArgs {
    const void* x; const void* W; const __half* bias; void* y;
    int M, N, K, out_kind, act, unary;   // act (gated units): 0 silu, 1 gelu in its tanh form, 2 clamped
    float limit;
};

template <typename T>
__device__ __forceinline__ void gr_mma(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    if constexpr (std::is_same_v<T, __half>)
        asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
            : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
    else
        asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
            : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

template <typename T, int NT, bool GLU, int kGrWarps>   // NT: tiles of eight tokens
__global__ void __launch_bounds__(kGrWarps * 32, kGrWarps == 8 ? 2 : 1) gemm_rows_kernel(const GrArgs p) {
    constexpr int MT = GLU ? 2 : 1, kRow = 20;   // (a token's 16 features, padded: the fragments' stores touch 32 banks)
    __shared__ float part[kGrWarps][MT][NT * 8][kRow];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, gid = lane >> 2, tig = lane & 3, f0 = blockIdx.x * 16;
    const T* W = reinterpret_cast<const T*>(p.W);
    const int pieces = (p.K + 31) >> 5;
    {   // the CTA's lines, 16 rows' at a time
        const int lines = (p.K * 2 + 127) >> 7;
#pragma unroll
        for (int m = 0; m < MT; ++m) {
            const T* row = W + ((size_t)m * p.N + min(f0 + (int)threadIdx.x % 16, p.N - 1)) * p.K;
            for (int l = threadIdx.x / 16; l < lines; l += kGrWarps * 2) asm volatile("prefetch.global.L2 [%0];" ::"l"(row + l * 64));
        }
    }
    pdl_launch_dependents();
    pdl_wait();
    const T *wr[MT][2], *xr[NT];
#pragma unroll
    for (int m = 0; m < MT; ++m)
#pragma unroll
        for (int q = 0; q < 2; ++q) wr[m][q] = W + ((size_t)m * p.N + min(f0 + gid + 8 * q, p.N - 1)) * p.K;   // (features and tokens that are not there: the last ones again, never stored)
#pragma unroll
    for (int t = 0; t < NT; ++t) xr[t] = reinterpret_cast<const T*>(p.x) + (size_t)min(t * 8 + gid, p.M - 1) * p.K;
    float sum[MT][NT][4];
#pragma unroll
    for (int m = 0; m < MT; ++m)
#pragma unroll
        for (int t = 0; t < NT; ++t) sum[m][t][0] = sum[m][t][1] = sum[m][t][2] = sum[m][t][3] = 0.f;
    constexpr int A = kGrAhead / (MT * NT);
    uint4 a[2][A][MT][2], b[2][A][NT];
    auto load = [&](int i0, uint4 (&av)[A][MT][2], uint4 (&bv)[A][NT]) {
#pragma unroll
        for (int i = 0; i < A; ++i) {
            const int k = min((i0 + i * kGrWarps) * 32 + tig * 8, p.K - 8);   // (K % 8 == 0; behind K: dropped below)
#pragma unroll
            for (int m = 0; m < MT; ++m)
#pragma unroll
                for (int q = 0; q < 2; ++q) av[i][m][q] = __ldcg(reinterpret_cast<const uint4*>(wr[m][q] + k));
#pragma unroll
            for (int t = 0; t < NT; ++t) bv[i][t] = __ldcg(reinterpret_cast<const uint4*>(xr[t] + k));
        }
    };
    // (the tensor core cuts off where it adds: its chains are A pieces long, 128 or 64 numbers, and are added up in fp32)
    auto products = [&](int i0, uint4 (&av)[A][MT][2], uint4 (&bv)[A][NT]) {
        float acc[MT][NT][4] = {};
#pragma unroll
        for (int i = 0; i < A; ++i) {
            const int c = i0 + i * kGrWarps;
            if (c >= pieces) continue;
            if (c * 32 + 32 > p.K && c * 32 + tig * 8 >= p.K) {   // the ragged end
                const uint4 z = make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
                for (int m = 0; m < MT; ++m) av[i][m][0] = av[i][m][1] = z;
#pragma unroll
                for (int t = 0; t < NT; ++t) bv[i][t] = z;
            }
            __syncwarp();
#pragma unroll
            for (int m = 0; m < MT; ++m)
#pragma unroll
                for (int t = 0; t < NT; ++t) {
                    gr_mma<T>(acc[m][t], av[i][m][0].x, av[i][m][1].x, av[i][m][0].y, av[i][m][1].y, bv[i][t].x, bv[i][t].y);
                    gr_mma<T>(acc[m][t], av[i][m][0].z, av[i][m][1].z, av[i][m][0].w, av[i][m][1].w, bv[i][t].z, bv[i][t].w);
                }
        }
#pragma unroll
        for (int m = 0; m < MT; ++m)
#pragma unroll
            for (int t = 0; t < NT; ++t)
#pragma unroll
                for (int e = 0; e < 4; ++e) sum[m][t][e] += acc[m][t][e];
    };
    constexpr int kStep = A * kGrWarps;
    load(warp, a[0], b[0]);
    for (int i0 = warp; i0 < pieces; i0 += 2 * kStep) {
        if (i0 + kStep < pieces) load(i0 + kStep, a[1], b[1]);
        products(i0, a[0], b[0]);
        if (i0 + 2 * kStep < pieces) load(i0 + 2 * kStep, a[0], b[0]);
        if (i0 + kStep < pieces) products(i0 + kStep, a[1], b[1]);
    }
#pragma unroll
    for (int m = 0; m < MT; ++m)
#pragma unroll
        for (int t = 0; t < NT; ++t)
#pragma unroll
            for (int e = 0; e < 4; ++e) part[warp][m][t * 8 + tig * 2 + (e & 1)][gid + (e >> 1) * 8] = sum[m][t][e];
    __syncthreads();
    const int f = threadIdx.x % 16, n = f0 + f, tok = threadIdx.x / 16;
    if (tok >= p.M || n >= p.N || tok >= NT * 8) return;
    float v[MT];
#pragma unroll
    for (int m = 0; m < MT; ++m) {
        v[m] = part[0][m][tok][f];
#pragma unroll
        for (int w = 1; w < kGrWarps; ++w) v[m] += part[w][m][tok][f];
    }
    float r = v[0];
    if constexpr (GLU) r = p.act == 2 ? glu_clamp_f(v[0], v[1], p.limit) : (p.act ? gelu_tanh_f(v[0]) : v[0] / (1.f + expf(-v[0]))) * v[1];
    else {
        if (p.bias) r += __half2float(p.bias[n]);
        if (p.unary == 1) { r = fmaxf(r, 0.f); r *= r; }
    }
    const size_t at = (size_t)tok * p.N + n;
    if (p.out_kind == 0) reinterpret_cast<__half*>(p.y)[at] = __float2half_rn(r);
    else if (p.out_kind == 1) reinterpret_cast<__nv_bfloat16*>(p.y)[at] = __float2bfloat16_rn(r);
    else reinterpret_cast<float*>(p.y)[at] = r;
}

template <typename T, bool GLU>
static cudaError_t gr_launch(const GrArgs& p, cudaStream_t s) {
    const dim3 grid((unsigned)((p.N + 15) / 16));
    if (p.K > 2048) return p.M <= 8 ? launch_chained(gemm_rows_kernel<T, 1, GLU, 16>, grid, dim3(512), 0, s, p) : launch_chained(gemm_rows_kernel<T, 2, GLU, 16>, grid, dim3(512), 0, s, p);
    return p.M <= 8 ? launch_chained(gemm_rows_kernel<T, 1, GLU, 8>, grid, dim3(256), 0, s, p) : launch_chained(gemm_rows_kernel<T, 2, GLU, 8>, grid, dim3(256), 0, s, p);
}

// 1 <= M <= 16, K % 8 == 0, x and W on 16-byte boundaries; out_kind, act and unary as GemmParams in gemm_tcgen05.cu; gated units take bfloat16 operands (gemm_few_rows is asked for no others)
int gemm_rows(const void* x, const void* W, const void* bias, void* y, int M, int N, int K, bool bf16, int out_kind, bool glu, int act, int unary, float limit, cudaStream_t s) {
    const GrArgs p{x, W, reinterpret_cast<const __half*>(bias), y, M, N, K, out_kind, act, unary, limit};
    const cudaError_t e = bf16 ? (glu ? gr_launch<__nv_bfloat16, true>(p, s) : gr_launch<__nv_bfloat16, false>(p, s)) : gr_launch<__half, false>(p, s);
    count_launch();
    return (int)e;
}

}  // namespace b200
