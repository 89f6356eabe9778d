// The latent attention kernels of latent_attention.cu and latent_attention_tc.cu.
#pragma once
#include <cuda_runtime.h>

#include <algorithm>

#include "b200_serve.h"
#include "common.cuh"

namespace b200 {

// how many CTAs share a window of 128 / heads packed tokens there (its sequences are dealt out to them; a CTA without one leaves at once): a
// sequence per CTA where two rounds of the GPU allow it, two at least
inline int latent_tc_parts(int n_tokens, int longest_entry, int heads, int halves) {
    if (n_tokens == longest_entry) return 1;
    const int TQ = 128 / heads, windows = (n_tokens + TQ - 1) / TQ, most = std::min(TQ, n_tokens - longest_entry + 1);   // sequences that a window can hold
    return std::max(2, (int)std::min<long long>(most, 2ll * sm_count() / ((long long)windows * halves)));
}
// bfloat16 prompt portions on tcgen05 tiles; -1: not built for these sizes
int latent_attention_tc(const b200_latent_attention_args& a, int out_cols, cudaStream_t s);

}  // namespace b200
