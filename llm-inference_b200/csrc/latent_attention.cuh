// The latent attention kernels of latent_attention.cu and latent_attention_tc.cu.
#pragma once
#include <cuda_runtime.h>

#include "b200_serve.h"

namespace b200 {

// bfloat16 prompt portions on tcgen05 tiles; -1: not built for these sizes
int latent_attention_tc(const b200_latent_attention_args& a, int out_cols, cudaStream_t s);

}  // namespace b200
