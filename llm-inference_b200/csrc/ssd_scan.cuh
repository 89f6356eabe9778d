// What the two chunk forms of the state-space recurrence share (ssd_scan.cu: chunks in parallel; ssd_tc.cu: a CTA per head walks them).
#pragma once
#include "b200_serve.h"
#include "common.cuh"

namespace b200 {

struct SS {
    const float* u; long long ld_u; int x_off, b_off, c_off;
    const float* dt_raw; long long ld_dt; const float* dt_bias;
    const float* A; const float* D;
    float* state; float* out;
    const int* ent_row; const int* ent_len; const int* slot; const int* pos;
    int heads, groups, vdim, n_state;
    // chunk form: chunk c of entry e sits at place ent_row[e] / kSsdChunk + e + c
    float* chunk_state;   // [place, head, n_state, vdim]
    float* chunk_decay;   // [place, head]
    float* chunk_cb;      // [place, group, kSsdChunk, kSsdChunk]
    int col_blocks;
};

__device__ __forceinline__ float ssd_softplus(float v) { return v > 20.f ? v : log1pf(expf(v)); }

// row strides in floats: stride % 32 == 4 for operands whose rows run along the fragment's 8-wide index, 8 for those whose
// rows run along its 4-wide index (every fragment load then touches 32 different banks)
__host__ __device__ __forceinline__ int ssd_stride4(int n) { return ((n + 31) & ~31) + 4; }
__host__ __device__ __forceinline__ int ssd_stride8(int n) { return ((n + 31) & ~31) + 8; }

__device__ __forceinline__ float ssd_tf32(float v) {
    uint32_t r;
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(v));
    return __uint_as_float(r);
}
__device__ __forceinline__ void ssd_mma(float (&d)[4], const float (&a)[4], float b0, float b1) {
    asm("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(__float_as_uint(a[0])), "r"(__float_as_uint(a[1])), "r"(__float_as_uint(a[2])), "r"(__float_as_uint(a[3])),
          "r"(__float_as_uint(b0)), "r"(__float_as_uint(b1)));
}

// `rows` rows of `cols` columns from global (leading dimension ld) into shared memory, rows beyond `live` and columns beyond
// cols (up to cpad) zero. Rows that allow it travel by cp.async (nothing waits for a load here: ssd_landed() before the first
// read); the values are rounded to tf32 when a fragment picks them up.
__device__ __forceinline__ void ssd_stage(float* dst, int stride, const float* src, long long ld, int rows, int live, int cols, int cpad) {
    if ((cols & 3) == 0 && (ld & 3) == 0 && (reinterpret_cast<uintptr_t>(src) & 15u) == 0 && cpad == cols) {
        const int q = cols / 4;
        for (int i = threadIdx.x; i < rows * q; i += blockDim.x) {
            const int r = i / q, c = (i - r * q) * 4;
            const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst + r * stride + c);
            const float* g = src + (r < live ? (size_t)r * ld + c : 0);
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(g), "r"(r < live ? 16 : 0) : "memory");
        }
        return;
    }
    for (int i = threadIdx.x; i < rows * cpad; i += blockDim.x) {
        const int r = i / cpad, c = i - r * cpad;
        dst[r * stride + c] = (r < live && c < cols) ? src[(size_t)r * ld + c] : 0.f;
    }
}
__device__ __forceinline__ void ssd_landed() {
    __syncwarp();   // the lanes close their group of copies together
    asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory");
    __syncthreads();
}

// ssd_tc.cu: B200_OK when it took the call, -1 when the chunks of ssd_scan.cu shall (a.chunk_* and a.col_blocks are not set yet)
size_t ssd_scan_tc_bytes(int n_tokens, int n_entries, int heads, int groups, int vdim, int n_state);   // 0: not its shapes
int ssd_scan_tc(const SS& a, const b200_ssd_scan_args& p, cudaStream_t s);

}  // namespace b200
