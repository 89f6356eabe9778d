// What the two chunk forms of the state-space recurrence share (ssd_scan.cu: chunks of 64 tokens on mma.sync, and the walk; ssd_tc.cu: chunks of 128 on tcgen05).
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

__device__ __forceinline__ float ssd_tf32(float v) {
    uint32_t r;
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(v));
    return __uint_as_float(r);
}

// ssd_tc.cu: B200_OK when it took the call, -1 when the chunks of ssd_scan.cu shall (a.chunk_* and a.col_blocks are not set yet)
size_t ssd_scan_tc_bytes(int n_tokens, int n_entries, int heads, int groups, int vdim, int n_state);   // 0: not its shapes
int ssd_scan_tc(const SS& a, const b200_ssd_scan_args& p, cudaStream_t s);

}  // namespace b200
