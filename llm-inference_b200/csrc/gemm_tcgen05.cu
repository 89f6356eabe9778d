// tcgen05 / TMEM GEMM for fp16 linears with more than B200_GEMV_MAX_TOKENS rows:
//   prefill QKV / o / gate_up / down / LM-head (launchLinearGemm, src/kernels/linear.cu:39-104 ->
//   cublasWrapper::Gemm, cublas_utils.cc:32-71, call sites context_attention.cpp:99,166, ffn.cpp:72,88)
//   and the batched decode step (8 < B <= 256 sequences), where the weights are the tiles' rows.
//
//   D[128, BN] (fp32, TMEM) += A_tile[128, 64] * B_tile[BN, 64]^T      (both operands K-major fp16)
//
//   normal  : A = x [Nt, K] (tokens on the MMA M axis), B = W [N, K]    -> y[tok, n]   tensor-bound (gemm_tcgen05_kernel)
//   stream  : A = W [N, K] (weight rows on the M axis), B = x [Nt, K]   -> y[tok, n]   HBM-bound (gemm_stream_kernel, below):
//             every weight byte is read once, Nt <= 256 tokens ride along as the MMA N extent; the K range of a tile is shared by
//             a cluster, so that narrow projections still fill the GPU.
//   swapped : the same operands on the persistent gemm_tcgen05_kernel, for outputs so wide that every CTA has tiles of its own.
//
// Structure of gemm_tcgen05_kernel (one persistent CTA per SM, 192 threads):
//   warp 0    TMA producer: cp.async.bulk.tensor.2d (UTMALDG) of 128B-swizzled [rows x 64] boxes
//             into a STAGES-deep smem ring, completion on mbarriers (expect_tx);
//   warp 1    allocates TMEM, then one elected lane issues tcgen05.mma.cta_group::1.kind::f16
//             (UTCHMMA), 4 x (K=16) per stage; tcgen05.commit releases the smem stage and, at the end
//             of a tile, publishes the accumulator;
//   warps 2-5 epilogue: tcgen05.ld (LDTM) 32 lanes x 32 columns per instruction, convert, store;
//             two accumulator stages in TMEM so the epilogue of tile i overlaps the MMAs of i+1.
#include <cooperative_groups.h>

#include <algorithm>
#include <atomic>
#include <mutex>
#include <unordered_map>

#include "common.cuh"
#include "launch_count.h"
#include "tc_common.cuh"

namespace b200 {
namespace cg = cooperative_groups;

constexpr int kBM = 128;           // MMA M (rows of A per tile)
constexpr int kBK = 64;            // K per stage: 64 fp16 = one 128-byte swizzle row
constexpr int kGemmThreads = 192;  // producer, MMA, 4 epilogue warps

struct GemmParams {
    void* C;            // fp16 [tokens, ldc]
    const void* bias;   // fp16 [N_out] or nullptr
    const __half* residual;   // fp16 [tokens, ldc] or nullptr (plain fp16 outputs, tokens on the M axis): C = half(half(acc + bias) + residual)
    int rows_a;         // valid rows of the A operand (tokens in normal mode, N_out in stream mode)
    int rows_b;         // valid rows of the B operand
    int K;
    int ldc;            // = N_out
    int tokens;
    int m_tiles, n_tiles, k_blocks;
    int splits;         // stream mode: CTAs (one cluster) that share a tile's K range
    int accs;           // stream mode: chains that a CTA's share of K is formed in, one after another
    int in_bf16;        // operands are bfloat16 instead of fp16 (same tiles, other instruction descriptor)
    int out_kind;       // element type of C: 0 fp16 (rounding points of the reference sequence), 1 bfloat16, 2 fp32
    int wide_store;     // stream mode: C is 16-byte aligned
    int glu_act;        // GLU epilogue: 0 silu, 1 gelu in its tanh form, 2 clamped at glu_limit (out_kind 1 / 2 only)
    float glu_limit;
    int unary;          // plain epilogue: 0 none, 1 the square of relu on every output
};
__device__ __forceinline__ float gemm_unary(float v, int unary) {
    if (unary == 1) { v = fmaxf(v, 0.f); v *= v; }
    return v;
}

template <int BN>
struct GemmSmem {
    static constexpr int kStageBytes = (kBM + BN) * kBK * 2;
    static constexpr int kStages = (BN >= 256) ? 4 : (BN >= 128) ? 6 : (BN >= 64) ? 8 : 10;
    static constexpr int kBarrierBytes = (2 * kStages + 4) * 8 + 16;
    static constexpr int kTotal = kStages * kStageBytes + kBarrierBytes + 1024;  // + alignment slack
    static constexpr int kTmemCols = (2 * BN < 32) ? 32 : 2 * BN;                // two accumulator stages
};

// stores of the epilogue in the element type GemmParams::out_kind names (idx in elements)
__device__ __forceinline__ void store8(void* C, size_t idx, const float (&f)[8], int kind) {
    if (kind == 0) st16(reinterpret_cast<__half*>(C) + idx, Unpack<__half>::put(f));
    else if (kind == 1) {
        Pack16 v;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const __nv_bfloat162 h = __floats2bfloat162_rn(f[2 * i], f[2 * i + 1]);
            v.w[i] = *reinterpret_cast<const uint32_t*>(&h);
        }
        st16(reinterpret_cast<__nv_bfloat16*>(C) + idx, v);
    } else {
        float* d = reinterpret_cast<float*>(C) + idx;
        *reinterpret_cast<float4*>(d) = make_float4(f[0], f[1], f[2], f[3]);
        *reinterpret_cast<float4*>(d + 4) = make_float4(f[4], f[5], f[6], f[7]);
    }
}
__device__ __forceinline__ void store1(void* C, size_t idx, float f, int kind) {
    if (kind == 0) reinterpret_cast<__half*>(C)[idx] = __float2half_rn(f);
    else if (kind == 1) reinterpret_cast<__nv_bfloat16*>(C)[idx] = __float2bfloat16_rn(f);
    else reinterpret_cast<float*>(C)[idx] = f;
}

// GLU (normal mode, BN = 256): W = [2*inter, K] with gate rows first (act_kernel.cu:28-29). The B tile of
// feature tile nt is 128 gate rows (nt*128) followed by the matching 128 up rows (inter + nt*128), so the
// accumulator holds gate in columns [0,128) and up in [128,256) of the same 128 features, and the epilogue
// writes silu(gate)*up (launchAct, act_kernel.cu:57) straight to out [tokens, inter]: the [tokens, 2*inter]
// intermediate of ffn.cpp:72-80 is never stored.
// A thread's row of a gated tile, sixteen features at a time, the next sixteen on their way. KIND 0: fp16 with the rounding points of the unfused
// sequence (products, silu of the gate, their product), 1 silu, 2 gelu in its tanh form, 3 clamped. What bounds it is the instruction cache: with
// all units in one loop over 32 unrolled features a tile took 16 us, with one unit per loop 11, of which the divisions' branches were two thirds (tile_silu).
// The fp16 unit had kept them: 400 x 1024 -> gated 28672 80 us without, 134 with (and 199 on the pairs that choose_tile names), 8192 x 4096 -> gated 11008 923 and 1444.
template <int KIND>
__device__ __forceinline__ void store_glu_row(const GemmParams& p, uint32_t taddr, int row, int nt) {
    if (row - (int)(threadIdx.x & 31) >= p.tokens) return;   // (rows behind the tokens are zeros, which take the long way through the division: not here, and not below)
    uint32_t g[16], u[16];
    __syncwarp();   // (the loads and waits of tensor memory are warp-wide: lanes that left a branch or a wait one by one meet first, here and below)
    tmem_ld_32x16_async(taddr, g);
    tmem_ld_32x16_async(taddr + 128u, u);
#pragma unroll 1
    for (int c0 = 0; c0 < 128; c0 += 16) {
        float f[16];
        uint32_t gc[16], uc[16];
        __syncwarp();
        tmem_wait_ld<16>(g);
        tmem_wait_ld<16>(u);
#pragma unroll
        for (int e = 0; e < 16; ++e) { gc[e] = g[e]; uc[e] = u[e]; }
        if (c0 + 16 < 128) {
            tmem_ld_32x16_async(taddr + (uint32_t)(c0 + 16), g);
            tmem_ld_32x16_async(taddr + (uint32_t)(128 + c0 + 16), u);
        }
        const int col0 = nt * 128 + c0;
        if (row < p.tokens && col0 < p.rows_b) {
#pragma unroll
            for (int e = 0; e < 16; ++e) {
                float gv = __uint_as_float(gc[e]), uv = __uint_as_float(uc[e]);
                if (KIND == 0) {
                    gv = __half2float(__float2half_rn(gv));
                    uv = __half2float(__float2half_rn(uv));
                    f[e] = __half2float(__float2half_rn(tile_silu(gv))) * uv;
                } else if (KIND == 1) f[e] = tile_silu(gv) * uv;
                else if (KIND == 2) f[e] = tile_gelu_tanh(gv) * uv;
                else f[e] = tile_glu_clamp(gv, uv, p.glu_limit);
            }
            const size_t dst = (size_t)row * p.ldc + col0;
            store8(p.C, dst, *reinterpret_cast<const float(*)[8]>(f), p.out_kind);
            if (col0 + 16 <= p.rows_b) store8(p.C, dst + 8, *reinterpret_cast<const float(*)[8]>(f + 8), p.out_kind);
        }
    }
}

template <int BN, bool SWAP, bool GLU = false>
__global__ void __launch_bounds__(kGemmThreads, 1)
gemm_tcgen05_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
                    const GemmParams p) {
    using S = GemmSmem<BN>;
    constexpr int STAGES = S::kStages;
    constexpr uint32_t A_BYTES = kBM * kBK * 2, B_BYTES = BN * kBK * 2;
    extern __shared__ unsigned char smem_raw[];
    // 128B-swizzled tiles must start on a 1024-byte boundary
    unsigned char* tiles = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    uint64_t* full_bar = reinterpret_cast<uint64_t*>(tiles + (size_t)STAGES * S::kStageBytes);
    uint64_t* empty_bar = full_bar + STAGES;
    uint64_t* acc_full = empty_bar + STAGES;   // [2]
    uint64_t* acc_empty = acc_full + 2;        // [2]
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 2);

    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(&full_bar[s], 1);
            mbar_init(&empty_bar[s], 1);
        }
        for (int a = 0; a < 2; ++a) {
            mbar_init(&acc_full[a], 1);
            mbar_init(&acc_empty[a], 4);
        }
        mbar_fence_init();
        tma_prefetch_desc(&map_a);
        tma_prefetch_desc(&map_b);
    }
    if (warp == 1) tmem_alloc(tmem_slot, S::kTmemCols);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = __shfl_sync(0xffffffffu, *tmem_slot, 0);
    pdl_launch_dependents();
    pdl_wait();   // x (and, for PDL chains, the previous kernel's output) must be complete

    const int units = p.m_tiles * p.n_tiles;

    if (warp == 0) {
        // ================= TMA producer =================
        int stage = 0;
        uint32_t phase = 0;
        for (int u = blockIdx.x; u < units; u += gridDim.x) {
            const int mt = u % p.m_tiles, nt = u / p.m_tiles;
            for (int kb = 0; kb < p.k_blocks; ++kb) {
                mbar_wait(&empty_bar[stage], phase ^ 1);
                if (lane == 0) {
                    unsigned char* sa = tiles + (size_t)stage * S::kStageBytes;
                    mbar_expect_tx(&full_bar[stage], A_BYTES + B_BYTES);
                    tma_load_2d(sa, &map_a, kb * kBK, mt * kBM, &full_bar[stage]);
                    if (GLU) {   // map_b boxes are 128 rows: gate rows, then the up rows of the same features
                        tma_load_2d(sa + A_BYTES, &map_b, kb * kBK, nt * 128, &full_bar[stage]);
                        tma_load_2d(sa + A_BYTES + B_BYTES / 2, &map_b, kb * kBK, p.rows_b + nt * 128, &full_bar[stage]);
                    } else {
                        tma_load_2d(sa + A_BYTES, &map_b, kb * kBK, nt * BN, &full_bar[stage]);
                    }
                }
                __syncwarp();
                if (++stage == STAGES) { stage = 0; phase ^= 1; }
            }
        }
    } else if (warp == 1) {
        // ================= MMA issuer =================
        // bfloat16 operands: A format (bits [7,10)) and B format (bits [10,13)) = 1
        // (descriptors and addresses from values that are uniform over the warp, one elected lane: from lane 0's own registers the four products of a stage
        // took 560 clocks to issue, whatever their size. 512 x 8192 -> 2048 in tiles of 128 x 64: 41 -> 25 us, 128 x 128: 43 -> 31; 128 x 256, where the operands' way
        // into shared memory takes longer, 52 -> 50)
        const uint32_t idesc = make_idesc_f16(kBM, BN) | (p.in_bf16 ? ((1u << 7) | (1u << 10)) : 0u);
        const uint64_t a_desc = make_kmajor_sw128_desc(smem_u32(tiles)), b_desc = make_kmajor_sw128_desc(smem_u32(tiles) + A_BYTES);
        const bool leader = elect_one();
        int stage = 0;
        uint32_t phase = 0;
        int acc = 0;
        uint32_t acc_phase = 0;
        for (int u = blockIdx.x; u < units; u += gridDim.x) {
            mbar_wait(&acc_empty[acc], acc_phase ^ 1);   // epilogue has drained this accumulator
            tc_fence_after();
            const uint32_t d_tmem = tmem_base + (uint32_t)(acc * BN);
            for (int kb = 0; kb < p.k_blocks; ++kb) {
                mbar_wait(&full_bar[stage], phase);
                tc_fence_after();
                if (leader) {
                    const uint64_t da = a_desc + (uint64_t)(stage * (S::kStageBytes >> 4)), db = b_desc + (uint64_t)(stage * (S::kStageBytes >> 4));
#pragma unroll
                    for (int k = 0; k < kBK / kUmmaK; ++k)
                        umma_f16(d_tmem, da + (uint64_t)(2 * k), db + (uint64_t)(2 * k), idesc,
                                 (kb > 0 || k > 0) ? 1u : 0u);
                    umma_commit(&empty_bar[stage]);                 // smem stage reusable when the MMAs retire
                    if (kb == p.k_blocks - 1) umma_commit(&acc_full[acc]);  // accumulator complete
                }
                __syncwarp();
                if (++stage == STAGES) { stage = 0; phase ^= 1; }
            }
            acc ^= 1;
            if (acc == 0) acc_phase ^= 1;
        }
    } else {
        // ================= epilogue warps =================
        const int quarter = warp & 3;   // TMEM lanes [32*quarter, 32*quarter + 32) belong to this warp
        int acc = 0;
        uint32_t acc_phase = 0;
        void* const C = p.C;
        const int ok = p.out_kind;
        const __half* bias = reinterpret_cast<const __half*>(p.bias);
        for (int u = blockIdx.x; u < units; u += gridDim.x) {
            const int mt = u % p.m_tiles, nt = u / p.m_tiles;
            const int row = mt * kBM + quarter * 32 + lane;   // row of the A operand / of D
            const uint32_t taddr = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(acc * BN);
            // the residual's 32 columns of a pass are read a pass ahead, the first under the products: read where they are added, each piece was a round trip of its
            // own (512 x 4096 -> 4096 27.3 us with a residual against 18.0 without)
            Pack16 rr[4];
            const bool add = !GLU && !SWAP && p.residual != nullptr && row < p.tokens && (p.ldc & 7) == 0;
            auto load_residual = [&](int col0) {
                if (!add || col0 + 32 > p.rows_b) return;
#pragma unroll
                for (int q = 0; q < 4; ++q) rr[q] = ld16(p.residual + (size_t)row * p.ldc + col0 + q * 8);
            };
            load_residual(nt * BN);
            __syncwarp();
            mbar_wait(&acc_full[acc], acc_phase);
            tc_fence_after();
            if (GLU) {
                // rows_b = inter; gate in columns [0,128), up in [128,256)
                if (ok == 0) store_glu_row<0>(p, taddr, row, nt);
                else if (p.glu_act == 2) store_glu_row<3>(p, taddr, row, nt);
                else if (p.glu_act) store_glu_row<2>(p, taddr, row, nt);
                else store_glu_row<1>(p, taddr, row, nt);
            } else
#pragma unroll 1
            for (int c0 = 0; c0 < BN; c0 += 32) {
                uint32_t v[32];
                __syncwarp();   // as in store_glu_row
                tmem_ld_32x32(taddr + (uint32_t)c0, v);
                const int col0 = nt * BN + c0;   // first row of the B operand covered by this chunk
                if (SWAP) {
                    // row = output feature, col = token: lanes write consecutive features of one token
                    if (row < p.rows_a) {
                        const float bv = bias ? __half2float(bias[row]) : 0.f;
#pragma unroll
                        for (int j = 0; j < 32; ++j)
                            if (col0 + j < p.tokens) store1(C, (size_t)(col0 + j) * p.ldc + row, gemm_unary(__uint_as_float(v[j]) + bv, p.unary), ok);
                    }
                    continue;
                }
                // row = token, col = output feature: 32 consecutive features per thread
                if (row < p.tokens && col0 < p.rows_b) {
                    const size_t dst = (size_t)row * p.ldc + col0;
                    if (col0 + 32 <= p.rows_b && (p.ldc & 7) == 0) {
#pragma unroll
                        for (int q = 0; q < 4; ++q) {
                            float f[8];
#pragma unroll
                            for (int e = 0; e < 8; ++e) {
                                f[e] = __uint_as_float(v[q * 8 + e]);
                                if (bias) f[e] += __half2float(bias[col0 + q * 8 + e]);
                                f[e] = gemm_unary(f[e], p.unary);
                            }
                            if (p.residual) {
                                float b[8];
                                Unpack<__half>::get(rr[q], b);
#pragma unroll
                                for (int e = 0; e < 8; ++e) f[e] = __half2float(__float2half_rn(f[e])) + b[e];
                            }
                            store8(C, dst + q * 8, f, ok);
                        }
                        if (c0 + 32 < BN) load_residual(col0 + 32);
                    } else {
                        // unrolled with a predicate: a run-time index would move v[] to local memory (no L1 behind
                        // it with the 227 KB carve-out) for EVERY path of the epilogue
#pragma unroll
                        for (int j = 0; j < 32; ++j) {
                            if (col0 + j >= p.rows_b) continue;
                            float f = __uint_as_float(v[j]);
                            if (bias) f += __half2float(bias[col0 + j]);
                            if (p.residual) f = __half2float(__float2half_rn(f)) + __half2float(p.residual[dst + j]);
                            store1(C, dst + j, gemm_unary(f, p.unary), ok);
                        }
                    }
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&acc_empty[acc]);
            acc ^= 1;
            if (acc == 0) acc_phase ^= 1;
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem_base, S::kTmemCols);
    }
}

// Few token rows: the weights stream through the M axis, 128 rows of W per tile, and a cluster of `splits` CTAs shares a tile's K range.
// What bounds it is the weights' way from HBM, so what counts is how much of them is in flight and how few things follow: every CTA has
// up to 100 KB of its share under way before the first product, two CTAs fit an SM, and the partial sums meet in shared memory (rank
// order) instead of a workspace and a second launch.
// GLU: a tile is 64 gate rows and the 64 up rows of the same features (W = [2 * rows_a, K], rows_a = features).
// The tensor core cuts off when it adds to an accumulator, so a sum's error grows with the length of its chain (1.05e-9 of the result's norm per element
// of K: 2.1e-6 at 2048, 4.7e-7 at 512): for fp32 outputs a long share of K is formed in several chains, which are added in fp32.
// Measured, 8 rows, 2048 -> 4096, fp32 out: the persistent kernel with partial sums in global memory and a reduction launch 11.2 us, this 8.5 us.
template <int BN>
struct StreamSmem {
    static constexpr int kStageBytes = (kBM + BN) * kBK * 2;
    static constexpr int kStages = BN <= 32 ? 5 : BN <= 64 ? 4 : BN <= 128 ? 3 : 4;
    static constexpr int kPerSm = BN <= 128 ? 2 : 1, kAccs = 512 / kPerSm / BN;   // accumulators that fit a CTA's tensor memory
    // up to 64 rows a CTA's chains have an accumulator each; above, two take turns and eight warps add them up in registers, half a row each
    static constexpr bool kFold = kAccs == 2;
    static constexpr int kThreads = kFold ? 320 : 192;
    static constexpr int kTotal = kStages * kStageBytes + (2 * kStages + 4) * 8 + 16 + 1024;
    static_assert(BN * kBM * 4 <= kStages * kStageBytes, "the partial sums take the place of the stages");
};
constexpr int kStreamMaxSplits = 8;

template <int BN, bool GLU>
__global__ void __launch_bounds__(StreamSmem<BN>::kThreads, StreamSmem<BN>::kPerSm)
gemm_stream_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b, const GemmParams p) {
    using S = StreamSmem<BN>;
    constexpr int STAGES = S::kStages;
    constexpr bool FOLD = S::kFold;
    constexpr uint32_t A_BYTES = kBM * kBK * 2, B_BYTES = BN * kBK * 2;
    extern __shared__ unsigned char smem_raw[];
    unsigned char* tiles = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    uint64_t* full_bar = reinterpret_cast<uint64_t*>(tiles + (size_t)STAGES * S::kStageBytes);
    uint64_t* empty_bar = full_bar + STAGES;
    uint64_t *acc_full = empty_bar + STAGES, *acc_empty = acc_full + 2;   // [2] each; without FOLD only the first of acc_full
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 2);
    volatile int* dead = reinterpret_cast<volatile int*>(tmem_slot + 1);
    float* om = reinterpret_cast<float*>(tiles);   // [tokens][128]: this CTA's sums, once the stages have been used

    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    const int sp = blockIdx.x % p.splits, mt = blockIdx.x / p.splits;
    const int kb0 = (int)((long long)p.k_blocks * sp / p.splits), kb1 = (int)((long long)p.k_blocks * (sp + 1) / p.splits);
    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(&full_bar[s], 1);
            mbar_init(&empty_bar[s], 1);
        }
        for (int i = 0; i < 2; ++i) { mbar_init(&acc_full[i], 1); mbar_init(&acc_empty[i], 8); }
        *dead = 0;
        mbar_fence_init();
        tma_prefetch_desc(&map_a);
        tma_prefetch_desc(&map_b);
    }
    const uint32_t tmem_cols = (uint32_t)(FOLD ? min(p.accs, 2) : p.accs) * BN;
    if (warp == 1) tmem_alloc(tmem_slot, tmem_cols);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = __shfl_sync(0xffffffffu, *tmem_slot, 0);
    pdl_launch_dependents();
    pdl_wait();

    if (warp == 0) {
        int stage = 0;
        uint32_t phase = 0;
        for (int kb = kb0; kb < kb1; ++kb) {
            mbar_wait_or_leave(&empty_bar[stage], phase ^ 1, dead);
            if (lane == 0) {
                unsigned char* sa = tiles + (size_t)stage * S::kStageBytes;
                mbar_expect_tx(&full_bar[stage], A_BYTES + B_BYTES);
                if (GLU) {
                    tma_load_2d(sa, &map_a, kb * kBK, mt * 64, &full_bar[stage]);
                    tma_load_2d(sa + A_BYTES / 2, &map_a, kb * kBK, p.rows_a + mt * 64, &full_bar[stage]);
                } else
                    tma_load_2d(sa, &map_a, kb * kBK, mt * kBM, &full_bar[stage]);
                tma_load_2d(sa + A_BYTES, &map_b, kb * kBK, 0, &full_bar[stage]);
            }
            __syncwarp();
            if (++stage == STAGES) { stage = 0; phase ^= 1; }
        }
    } else if (warp == 1) {
        const uint32_t idesc = make_idesc_f16(kBM, BN) | (p.in_bf16 ? ((1u << 7) | (1u << 10)) : 0u);
        const uint64_t a_desc = make_kmajor_sw128_desc(smem_u32(tiles)), b_desc = make_kmajor_sw128_desc(smem_u32(tiles) + A_BYTES);
        const bool leader = elect_one();
        auto chain_end = [&](int i) { return p.accs == 1 ? kb1 : kb0 + (kb1 - kb0) * (i + 1) / p.accs; };
        int stage = 0, at = 0, end = chain_end(0);
        bool fresh = true;   // the first products of a chain
        uint32_t phase = 0;
        for (int kb = kb0; kb < kb1; ++kb) {
            const int slot = FOLD ? at & 1 : at;
            if (FOLD && fresh && at >= 2) mbar_wait_or_leave(&acc_empty[slot], (uint32_t)((at >> 1) - 1) & 1u, dead);
            mbar_wait_or_leave(&full_bar[stage], phase, dead);
            tc_fence_after();
            if (leader) {
                const uint64_t da = a_desc + (uint64_t)(stage * (S::kStageBytes >> 4)), db = b_desc + (uint64_t)(stage * (S::kStageBytes >> 4));
#pragma unroll
                for (int k = 0; k < kBK / kUmmaK; ++k)
                    umma_f16(tmem + (uint32_t)(slot * BN), da + (uint64_t)(2 * k), db + (uint64_t)(2 * k), idesc, (!fresh || k > 0) ? 1u : 0u);
                umma_commit(&empty_bar[stage]);
                if (FOLD ? kb + 1 == end : kb + 1 == kb1) umma_commit(&acc_full[FOLD ? slot : 0]);
            }
            __syncwarp();
            fresh = kb + 1 == end;
            if (fresh && kb + 1 < kb1) end = chain_end(++at);
            if (++stage == STAGES) { stage = 0; phase ^= 1; }
        }
    } else if constexpr (FOLD) {
        constexpr int COLS = BN / 2;
        const int quarter = warp & 3, first = (warp - 2) / 4 * COLS;
        const uint32_t taddr = tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)first;
        float sum[COLS];
#pragma unroll
        for (int j = 0; j < COLS; ++j) sum[j] = 0.f;
        for (int i = 0; i < p.accs; ++i) {
            mbar_wait_or_leave(&acc_full[i & 1], (uint32_t)(i >> 1) & 1u, dead);   // (the last: every load has landed and every product has read its stage)
            tc_fence_after();
#pragma unroll
            for (int c0 = 0; c0 < COLS; c0 += 16)
                if (first + c0 < p.tokens) {
                    uint32_t v[16];
                    tmem_ld_32x16_async(taddr + (uint32_t)((i & 1) * BN + c0), v);
                    tmem_wait_ld<16>(v);
#pragma unroll
                    for (int j = 0; j < 16; ++j) sum[c0 + j] += __uint_as_float(v[j]);
                }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&acc_empty[i & 1]);
        }
        const bool gone = *dead != 0;
#pragma unroll
        for (int j = 0; j < COLS; ++j)
            if (first + j < p.tokens) om[(first + j) * kBM + quarter * 32 + lane] = gone ? __int_as_float(0x7fffffff) : sum[j];
    } else {
        const int quarter = warp & 3;
        mbar_wait_or_leave(acc_full, 0, dead);   // every load has landed and every product has read its stage
        const bool gone = *dead != 0;
        tc_fence_after();
        const uint32_t taddr = tmem + ((uint32_t)(quarter * 32) << 16);
#pragma unroll 1
        for (int c0 = 0; c0 < BN && c0 < p.tokens; c0 += 32) {
            uint32_t v[32];
            tmem_ld_32x32(taddr + (uint32_t)c0, v);
#pragma unroll 1
            for (int i = 1; i < p.accs; ++i) {
                uint32_t w[32];
                tmem_ld_32x32(taddr + (uint32_t)(i * BN + c0), w);
#pragma unroll
                for (int j = 0; j < 32; ++j) v[j] = __float_as_uint(__uint_as_float(v[j]) + __uint_as_float(w[j]));
            }
#pragma unroll
            for (int j = 0; j < 32; ++j)
                if (c0 + j < p.tokens) om[(c0 + j) * kBM + quarter * 32 + lane] = gone ? __int_as_float(0x7fffffff) : __uint_as_float(v[j]);
        }
        tc_fence_before();
    }
    cg::cluster_group cluster = cg::this_cluster();
    if (p.splits > 1) cluster.sync();
    else __syncthreads();
    {
        constexpr int F = GLU ? 64 : kBM;                 // output features of the tile
        const int total = p.tokens * (F / 4), share = (total + p.splits - 1) / p.splits;
        const float* part[kStreamMaxSplits];
#pragma unroll
        for (int q = 0; q < kStreamMaxSplits; ++q) part[q] = q < p.splits ? cluster.map_shared_rank(om, q) : nullptr;
        auto sum4 = [&](int at) {
            float4 t[kStreamMaxSplits], acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int q = 0; q < kStreamMaxSplits; ++q)
                if (q < p.splits) t[q] = *reinterpret_cast<const float4*>(part[q] + at);
#pragma unroll
            for (int q = 0; q < kStreamMaxSplits; ++q)
                if (q < p.splits) {
                    if (q == 0) acc = t[0];
                    else { acc.x += t[q].x; acc.y += t[q].y; acc.z += t[q].z; acc.w += t[q].w; }
                }
            return acc;
        };
        const __half* bias = reinterpret_cast<const __half*>(p.bias);
        for (int i = sp * share + (int)threadIdx.x; i < min(total, (sp + 1) * share); i += S::kThreads) {
            const int tok = i / (F / 4), f0 = i % (F / 4) * 4, n = mt * F + f0;
            if (n >= p.rows_a) continue;
            const float4 s4 = sum4(tok * kBM + f0);
            float f[4] = {s4.x, s4.y, s4.z, s4.w};
            if (GLU) {
                const float4 u4 = sum4(tok * kBM + 64 + f0);
                const float u[4] = {u4.x, u4.y, u4.z, u4.w};
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    f[e] = p.glu_act == 2 ? glu_clamp_f(f[e], u[e], p.glu_limit) : (p.glu_act ? gelu_tanh_f(f[e]) : f[e] / (1.f + expf(-f[e]))) * u[e];
            } else {
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    if (bias && n + e < p.rows_a) f[e] += __half2float(bias[n + e]);
                    f[e] = gemm_unary(f[e], p.unary);
                }
            }
            const size_t dst = (size_t)tok * p.ldc + n;
            if (n + 4 <= p.rows_a && (p.ldc & 3) == 0 && p.wide_store) {
                if (p.out_kind == 2) *reinterpret_cast<float4*>(reinterpret_cast<float*>(p.C) + dst) = make_float4(f[0], f[1], f[2], f[3]);
                else {
                    uint2 v;
                    if (p.out_kind == 0) {
                        const __half2 a = __floats2half2_rn(f[0], f[1]), b = __floats2half2_rn(f[2], f[3]);
                        v = make_uint2(*reinterpret_cast<const uint32_t*>(&a), *reinterpret_cast<const uint32_t*>(&b));
                    } else {
                        const __nv_bfloat162 a = __floats2bfloat162_rn(f[0], f[1]), b = __floats2bfloat162_rn(f[2], f[3]);
                        v = make_uint2(*reinterpret_cast<const uint32_t*>(&a), *reinterpret_cast<const uint32_t*>(&b));
                    }
                    *reinterpret_cast<uint2*>(reinterpret_cast<__half*>(p.C) + dst) = v;
                }
            } else {
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    if (n + e < p.rows_a) store1(p.C, dst + e, f[e], p.out_kind);
            }
        }
    }
    if (p.splits > 1) cluster.sync();   // nobody leaves while its sums are read
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem, tmem_cols);
    }
}

// ------------------------------------------------------------------------------------------
// host side
// ------------------------------------------------------------------------------------------
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

// the driver entry point is resolved through the runtime, so the library has no link-time
// dependency on libcuda (it must load on the GPU-less build box)
static EncodeTiledFn encode_tiled_fn() {
    static EncodeTiledFn fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<EncodeTiledFn>(p);
    });
    return fn;
}

// 2-D map over a row-major fp16 matrix [rows, K]: box = [box_rows x 64], 128B swizzle, zero fill
// outside the tensor (ragged M / N / K tails need no special code in the kernel)
bool make_tma_map_2d(CUtensorMap* out, const void* ptr, long long rows, int K, int box_rows) {
    struct Key {
        const void* p; long long rows; int K, box;
        bool operator==(const Key& o) const { return p == o.p && rows == o.rows && K == o.K && box == o.box; }
    };
    struct Hash {
        size_t operator()(const Key& k) const {
            return std::hash<const void*>()(k.p) ^ (size_t)k.rows * 1000003u ^ (size_t)k.K * 7919u ^ (size_t)k.box;
        }
    };
    static std::unordered_map<Key, CUtensorMap, Hash> cache;
    static std::mutex mu;
    const Key key{ptr, rows, K, box_rows};
    // the thread's own look first (a map follows from its key alone): no lock and no search for what a program calls again and again
    struct Seen { Key key; CUtensorMap map; };
    static thread_local Seen seen[64];
    const size_t h = Hash()(key);
    Seen& mine = seen[(h ^ h >> 9 ^ h >> 17) & 63];
    if (mine.key.p && mine.key == key) { *out = mine.map; return true; }
    std::lock_guard<std::mutex> g(mu);
    auto it = cache.find(key);
    if (it != cache.end()) { *out = it->second; mine = Seen{key, it->second}; return true; }
    EncodeTiledFn enc = encode_tiled_fn();
    if (!enc) return false;
    const cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)rows};
    const cuuint64_t strides[1] = {(cuuint64_t)K * 2};
    const cuuint32_t box[2] = {(cuuint32_t)kBK, (cuuint32_t)box_rows};
    const cuuint32_t estr[2] = {1, 1};
    CUtensorMap m;
    const CUresult r = enc(&m, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<void*>(ptr), dims, strides, box, estr,
                           CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                           CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return false;
    if (cache.size() > 4096) cache.clear();
    cache.emplace(key, m);
    mine = Seen{key, m};
    *out = m;
    return true;
}

template <int BN, bool SWAP, bool GLU = false>
static int gemm_launch(const CUtensorMap& ma, const CUtensorMap& mb, const GemmParams& p, int grid, cudaStream_t s) {
    auto kern = gemm_tcgen05_kernel<BN, SWAP, GLU>;
    static unsigned long long attr_done = 0;   // per instantiation, one bit per device
    {
        cudaError_t e = ensure_max_dynamic_smem(reinterpret_cast<const void*>(kern), GemmSmem<BN>::kTotal, attr_done);
        if (e != cudaSuccess) return (int)e;
    }
    cudaError_t e = launch_k(kern, dim3(grid), dim3(kGemmThreads), (size_t)GemmSmem<BN>::kTotal, s, true, ma, mb, p);
    count_launch();
    return (int)e;
}

template <int BN, bool GLU>
static void stream_config(cudaLaunchConfig_t& cfg, cudaLaunchAttribute* at, int m_tiles, int splits, cudaStream_t s) {
    cfg = cudaLaunchConfig_t{};
    cfg.gridDim = dim3((unsigned)(m_tiles * splits));
    cfg.blockDim = dim3(StreamSmem<BN>::kThreads);
    cfg.dynamicSmemBytes = StreamSmem<BN>::kTotal;
    cfg.stream = s;
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = (unsigned)splits;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
}

// [n]: clusters of n CTAs that run at once, asked for once per device and kernel; nullptr: e says why. A cluster lives inside one GPC, so they are fewer than the
// SMs alone would hold. (The runtime counts one CTA per SM here, 148 74 45 33 26 22 15 15 clusters of 1 to 8, while kPerSm of them run: its answer is scaled.)
template <int BN, bool GLU>
static const int* stream_capacity(int dev, int sms, cudaError_t& e) {
    static std::atomic<const int*> known[kMaxDevices];
    const int* c = known[dev].load(std::memory_order_acquire);
    if (c) return c;
    auto kern = gemm_stream_kernel<BN, GLU>;
    prefer_max_smem_carveout(reinterpret_cast<const void*>(kern));
    e = cudaFuncSetAttribute(reinterpret_cast<const void*>(kern), cudaFuncAttributeMaxDynamicSharedMemorySize, StreamSmem<BN>::kTotal);
    if (e != cudaSuccess) return nullptr;
    int* t = new int[kStreamMaxSplits + 1]{};
    for (int n = 1; n <= kStreamMaxSplits; ++n) {
        cudaLaunchConfig_t cfg;
        cudaLaunchAttribute at[1];
        stream_config<BN, GLU>(cfg, at, sms, n, nullptr);
        if (cudaOccupancyMaxActiveClusters(&t[n], kern, &cfg) != cudaSuccess) { cudaGetLastError(); t[n] = 0; }
    }
    for (int n = kStreamMaxSplits; n > 0; --n) t[n] = t[1] > 0 ? t[n] * sms * StreamSmem<BN>::kPerSm / t[1] : 0;
    if (known[dev].compare_exchange_strong(c, t, std::memory_order_acq_rel)) return t;
    delete[] t;   // another thread was first
    return c;
}

// CTAs per tile: as many as run at once, each with two K blocks at least; more where their chains would be fewer than `shares`
template <int BN>
static int stream_splits(const int* capacity, int sms, int m_tiles, int k_blocks, int shares) {
    const int slots = sms * StreamSmem<BN>::kPerSm;
    int n = std::max(1, std::min({kStreamMaxSplits, slots / m_tiles, k_blocks / 2})), fit = n;
    // a second wave costs a whole pass (us, 2048 x 2048 at 256 rows in clusters of 8 / 6: 26.6 / 17.3, 6184 x 2048 at 32 rows of 6 / 5: 20.4 / 16.4), but leaving
    // more than a quarter of the places empty costs more (11008 x 4096 at 32 rows in clusters of 3 / 2: 28.7 / 36.1)
    while (fit > 1 && capacity[fit] < m_tiles) --fit;
    if (4 * fit * m_tiles >= 3 * slots || StreamSmem<BN>::kPerSm == 1) n = fit;
    return StreamSmem<BN>::kFold ? n : std::max(n, std::min(kStreamMaxSplits, (shares + StreamSmem<BN>::kAccs - 1) / StreamSmem<BN>::kAccs));
}

template <int BN, bool GLU>
static int stream_launch(const void* x, const void* W, GemmParams p, int M, int N, int K, int shares, int dev, int sms, cudaStream_t s) {
    cudaError_t e = cudaSuccess;
    const int* capacity = stream_capacity<BN, GLU>(dev, sms, e);
    if (!capacity) return (int)e;
    CUtensorMap ma, mb;
    if (!make_tma_map_2d(&ma, W, GLU ? 2ll * N : N, K, GLU ? 64 : kBM) || !make_tma_map_2d(&mb, x, M, K, BN)) return B200_EUNSUPPORTED;
    p.splits = stream_splits<BN>(capacity, sms, p.m_tiles, p.k_blocks, shares);
    const int share = p.k_blocks / p.splits;
    p.accs = 1;
    if (p.out_kind == 2) {
        if (StreamSmem<BN>::kFold) p.accs = std::max({1, share / 8, std::min(share, (shares + p.splits - 1) / p.splits)});
        else while (p.accs < StreamSmem<BN>::kAccs && p.accs * 4 < share) p.accs *= 2;
    }
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute at[2];
    stream_config<BN, GLU>(cfg, at, p.m_tiles, p.splits, s);
    if (pdl_enabled()) {
        at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        at[1].val.programmaticStreamSerializationAllowed = 1;
        cfg.numAttrs = 2;
    }
    e = cudaLaunchKernelEx(&cfg, gemm_stream_kernel<BN, GLU>, ma, mb, p);
    count_launch();
    return (int)e;
}

template <int BN>
static int swapped_launch(const void* x, const void* W, const GemmParams& p, int M, int N, int K, cudaStream_t s) {
    CUtensorMap ma, mb;
    if (!make_tma_map_2d(&ma, W, N, K, kBM) || !make_tma_map_2d(&mb, x, M, K, BN)) return B200_EUNSUPPORTED;
    return gemm_launch<BN, true>(ma, mb, p, std::min(p.m_tiles, sm_count()), s);
}

// the shares of K that fp32 outputs are formed in at least: what fills `sms` CTAs best when every share is a tile of its own (and what the kernel with partial
// sums in global memory formed them in: no sum is less exact than it was there)
static int least_shares(int m_tiles, int k_blocks, int sms) {
    int best = 1;
    long long best_cost = -1;
    for (int s = 1; s <= 16 && k_blocks / s >= 4; ++s) {
        const long long rounds = ((long long)m_tiles * s + sms - 1) / sms;
        const long long per = (k_blocks + s - 1) / s;
        const long long cost = rounds * (per + 2) + (s > 1 ? s : 0);
        if (best_cost < 0 || cost < best_cost) { best_cost = cost; best = s; }
    }
    return best;
}

int gemm_rows(const void* x, const void* W, const void* bias, void* y, int M, int N, int K, bool bf16, int out_kind, bool glu, int act, int unary, float limit, cudaStream_t s);

// Up to 16 rows against few weights, where set-up and latency count: no tensor maps, barriers or tensor memory (gemm_rows.cu). The lines lie where the time of
// gemm_stream_kernel is reached (rows / stream in a graph, weights from HBM, at 8 and at 16 rows unless it says otherwise).
//   K <= 2048: 13 M weights up to 8 rows (4096 x 2048 0.81, 6184 x 2048 0.96, 7000 x 2048 1.00; 12288 x 1024 1.09), 8.5 M up to 16 (4096 x 2048 0.89, 5504 x 2048 1.17),
//   17 M gated (2 x 4224 x 2048 0.86, 0.95; 2 x 8192 x 1024 0.95, 1.01; 2 x 5504 x 2048 1.17, 1.26); and 8192 features, whatever K: a CTA has too little to do for what it
//   sets up (16384 x 512 1.31, 1.13, gated 2 x 12288 x 512 1.00, 1.09).
//   Longer K, as long as every CTA has an SM: eight rows up to 12288 (2048 x 9216 0.94, 1024 x 12288 0.98, 1024 x 16384 1.10), more up to 6144 (2048 x 6144 0.95, 2048 x
//   7168 1.02, 2048 x 8192 1.07, 1024 x 16384 1.17 to 1.25); but 64 features or fewer, with few clusters to share K, at any K (64 x 16384 0.72, 0.85). Gated ones, two sums for a load of x, less far the fewer CTAs share the weights' way: 3072 (2 x 128 x 3072 0.96, 1.02), from
//   1024 features 4608 (2 x 1024 x 4608 0.94, 1.01; 2 x 256 x 4096 1.16, 1.28), from 2048 features 5504 (2 x 2048 x 5504 0.93, 0.97; 2 x 1408 x 5504 1.06, 1.09, 2 x 1920 x 6144 1.01, 1.07).
static bool takes_rows(int M, int N, int K, bool glu, int sms) {
    if (M > 16) return false;
    const long long weights = (long long)N * K * (glu ? 2 : 1);
    if (K <= 2048) return N <= 8192 && weights <= (glu ? 17000000 : M <= 8 ? 13000000 : 8500000);
    if (N > 16 * sms || weights > 24000000) return false;
    if (glu) return K <= (N >= 2048 ? 5504 : N >= 1024 ? 4608 : 3072);
    return N <= 64 || K <= (M <= 8 ? 12288 : 6144);
}

// M <= 256 token rows against W = [N, K] (GLU: M <= 128, W = [2 N, K], N % 64 == 0)
static int gemm_few_rows(const void* x, const void* W, GemmParams p, int M, int N, int K, bool glu, cudaStream_t s) {
    const int F = glu ? 64 : kBM, sms = sm_count();
    if (takes_rows(M, N, K, glu, sms)) return gemm_rows(x, W, p.bias, p.C, M, N, K, p.in_bf16 != 0, p.out_kind, glu, p.glu_act, p.unary, p.glu_limit, s);
    const int BN = M <= 32 ? 32 : M <= 64 ? 64 : M <= 128 ? 128 : 256;
    p.rows_a = N; p.rows_b = M;
    p.m_tiles = (N + F - 1) / F; p.n_tiles = 1;
    p.wide_store = (reinterpret_cast<uintptr_t>(p.C) & 15u) == 0;
    // Wide outputs: with a tile or more per CTA there is no K range to share, and the persistent kernel hides a tile's epilogue and set-up under the next
    // one's products. The lines lie where its time passes the stream kernel's (us, stream / persistent). More than 128 rows, where a CTA fills an SM, from
    // one CTA per tile on: 11008 x 4096 at 256 rows 57 / 53, 32000 x 1024 55 / 39, 128256 x 2048 222 / 137. 33 to 128 rows from 1.6 tiles per SM on
    // (25600 x 4096 at 64 rows 55 / 60, 32000 x 4096 67 / 62, 128256 x 2048 118 / 105) and where about one each is left (16384 x 1024 19 / 17). Fewer
    // only beyond the two tiles per SM that run at once and for short sums: 50304 x 1024 at 32 rows 36 / 32, 128256 x 2048 106 / 109.
    const bool wide = M > 128 ? 2 * p.m_tiles > sms : M > 32 ? 5 * p.m_tiles > 8 * sms || (5 * p.m_tiles > 4 * sms && p.m_tiles <= sms) : p.m_tiles > 2 * sms && p.k_blocks <= 16;
    // fp32 outputs are formed in least_shares shares of K at least (the persistent kernel knows one)
    const int shares = !glu && p.out_kind == 2 ? least_shares(p.m_tiles, p.k_blocks, sms) : 1;
    // three CTAs per tile whose clusters do not all run at once: 12288 x 4096 fp16 at 32 rows 38.9 us, 31.8 on the persistent kernel
    const int dev = current_device();
    bool late = false;
    if (!glu && shares == 1 && M <= 128 && 2 * sms / p.m_tiles == 3) {
        cudaError_t e = cudaSuccess;
        const int* c = BN == 32 ? stream_capacity<32, false>(dev, sms, e) : BN == 64 ? stream_capacity<64, false>(dev, sms, e) : stream_capacity<128, false>(dev, sms, e);
        late = c && c[3] < p.m_tiles;
    }
    if (!glu && (wide || late) && shares == 1) {
        switch (BN) {
            case 32: return swapped_launch<32>(x, W, p, M, N, K, s);
            case 64: return swapped_launch<64>(x, W, p, M, N, K, s);
            case 128: return swapped_launch<128>(x, W, p, M, N, K, s);
            default: return swapped_launch<256>(x, W, p, M, N, K, s);
        }
    }
    switch (BN) {
        case 32: return glu ? stream_launch<32, true>(x, W, p, M, N, K, shares, dev, sms, s) : stream_launch<32, false>(x, W, p, M, N, K, shares, dev, sms, s);
        case 64: return glu ? stream_launch<64, true>(x, W, p, M, N, K, shares, dev, sms, s) : stream_launch<64, false>(x, W, p, M, N, K, shares, dev, sms, s);
        case 128: return glu ? stream_launch<128, true>(x, W, p, M, N, K, shares, dev, sms, s) : stream_launch<128, false>(x, W, p, M, N, K, shares, dev, sms, s);
        default: return stream_launch<256, false>(x, W, p, M, N, K, shares, dev, sms, s);
    }
}

bool gemm_pairs_enabled();
int gemm2_tcgen05_ex(const void* x, const void* W, void* y, int M, int N, int K, int out_kind, bool glu, int glu_act, int unary, float glu_limit, int cols, cudaStream_t s);
int gemm2_tcgen05_f16(const void* x, const void* W, const void* bias, void* y, int M, int N, int K, bool glu, int cols, cudaStream_t s, const void* residual = nullptr);

// Which tile a product of many token rows takes: 128 rows on one CTA or 256 on a pair, by the columns of its accumulator. What a tile costs per 64-wide K step is its
// operands' way through L2 and shared memory, a round of tiles is paid in full however few there are, a tile's set-up and epilogue once, the outputs at 5 TB/s; so the
// width that just fills the chip's last round wins. The constants (us) are fitted to 105 plain and 28 gated shapes (200 to 2048 rows, 1000 to 12288 features, K 1024 to
// 11008, weights from HBM), each run with every tile: the tile that the rule names is 0.7 % slower than the best in the mean (gated: 0.2 %), and against the choice
// without pairs narrower than 256 columns 5 % (gated: 9 %) faster. us, that choice / now: 1522 x 8192 -> 2048 49.2 / 38.5 (192 columns), 1522 x 2048 -> 4096 28.9 / 23.3
// (192), 512 x 4096 -> 12288 48.1 / 41.8 (192), 512 x 11008 -> 4096 42.8 / 39.3 (128); 1024 x 1024 -> 1024 keeps 64 columns on one CTA (6.6; pairs 9.0). A pair has to be 3 %
// cheaper than one CTA's best: below that the fit does not tell them apart.
// Beyond what it was fitted to. A product of more than 100 GFLOP runs long enough for the power limit to set the clock, and a narrow tile moves more bytes per product: the pair of
// 256 columns stands there unless another tile is 8 % cheaper. us back to back for seconds at the clock that this leaves, the tile named without that / 256 columns: 4096 x 11008 ->
// 4096 355 (160) / 319, 4096 x 8192 -> 2048 128 (160) / 118, 6000 x 11008 -> 4096 502 (160) / 456, 6000 x 4096 -> 4096 179 (160) / 169, 2048 x 11008 -> 4096 162 (160) / 154, 8192 x 5504 -> 2048 168 (160) /
// 163, 4096 x 4096 -> 4096 117 (160) / 114, 4096 x 4096 -> 12288 307 (224) / 309, 8192 x 4096 -> 12288 622 (224) / 615, 8192 x 4096 -> gated 11008 1088 (224) / 1072, 3000 x 1024 -> 32000 192 (224) / 185; 256 either way:
// 8192 x 4096 -> 4096 210, 8192 x 11008 -> 4096 578, 4096 x 4096 -> gated 11008 535; kept: 2048 x 4096 -> 12288 159 (224) / 163. Shorter ones do not tell: 4096 x 5504 -> 2048 79.7 (160) / 79.3 for seconds, 72 / 77 one
// at a time. Above 2048 rows, outputs whose rows do not end on 64 columns: what is stored across the lines' borders is priced too (least where a pass has most columns of a
// row; one CTA stores a row per thread): 4096 x 1032 -> 1000 fp32 21.2 (128 columns on one CTA) / 15.3 (pairs of 256), weights from HBM.
struct Tile { int rows, cols; float step, round, once32, once16; };
struct TileChoice { int cols; bool pair; };
static constexpr Tile kPlainTiles[] = {{128, 64, 0.168f, 0.f, 4.16f, 3.43f}, {128, 128, 0.205f, 0.14f, 5.10f, 3.87f}, {128, 256, 0.334f, 0.24f, 7.01f, 4.82f},
                                       {256, 128, 0.177f, 0.f, 5.93f, 5.14f}, {256, 160, 0.190f, 0.f, 6.63f, 5.89f}, {256, 192, 0.230f, 0.f, 6.90f, 5.61f},
                                       {256, 224, 0.252f, 0.f, 7.68f, 6.69f}, {256, 256, 0.302f, 0.f, 7.86f, 6.27f}};
// gated: half of the columns are gates. us, pairs of 256 columns or one CTA / now: 512 x 2048 -> 2 x 5504 26.7 / 20.2 (160), 200 x 2048 -> 2 x 5504 19.1 / 14.8 (160), 2048 x 2048 -> 2 x 5504
// stays at 256 (62.8), 257 x 4096 -> 2 x 11008 on one CTA (64; pairs 96 and more)
static constexpr Tile kGatedTiles[] = {{128, 256, 0.349f, 1.06f, 4.23f, 4.23f}, {256, 128, 0.169f, 1.28f, 4.04f, 4.04f}, {256, 160, 0.170f, 1.76f, 5.04f, 5.04f},
                                       {256, 192, 0.204f, 1.50f, 5.47f, 5.47f}, {256, 224, 0.221f, 1.98f, 5.85f, 5.85f}, {256, 256, 0.258f, 1.88f, 6.06f, 6.06f}};
template <int COUNT>
static TileChoice choose_tile(const Tile (&tiles)[COUNT], int M, int N, int k_blocks, bool glu, bool f32, int sms, bool pairs_only = false) {
    TileChoice best{256, pairs_only};
    float least = -1.f, full = -1.f;   // full: the pair of 256 columns
    const float outputs = (float)M * N * 1e-6f;
    const bool pairs = pairs_only || gemm_pairs_enabled(), ragged = M > 2048 && N % 64 != 0;
    for (const Tile& t : tiles) {
        const bool pair = t.rows == 256;
        const int out_cols = glu ? t.cols / 2 : t.cols, at_once = pair ? sms / 2 : sms;
        if (pair ? !pairs || (N < 256 && !glu) : (pairs_only || (t.cols > N && t.cols > 64 && !glu))) continue;
        const long long n = ((long long)M + t.rows - 1) / t.rows * ((N + out_cols - 1) / out_cols), rounds = (n + at_once - 1) / at_once;
        float cost = (float)rounds * (k_blocks * t.step + t.round) + (f32 ? t.once32 : t.once16) + outputs * (f32 ? 4.f : 2.f) / 5.f;
        if (ragged) cost += outputs * (!pair ? 1.7f : t.cols < 256 ? 0.8f : 0.4f);
        if (pair && !pairs_only) cost *= 1.03f;
        if (least < 0.f || cost < least) { least = cost; best = {t.cols, pair}; }
        if (pair && t.cols == 256) full = cost;
    }
    const bool long_call = (glu ? 4.f : 2.f) * outputs * (float)k_blocks * kBK > 1e5f;   // MFLOP
    return long_call && full > 0.f && least > 0.92f * full ? TileChoice{256, true} : best;
}

// what the rule names, for tests: columns of the accumulator, negative on a pair of CTAs
int linear_tile(int M, int N, int K, bool gated, bool f32, int sms) {
    const int k_blocks = (K + kBK - 1) / kBK;
    const TileChoice t = gated ? choose_tile(kGatedTiles, M, N, k_blocks, true, f32, sms) : choose_tile(kPlainTiles, M, N, k_blocks, false, f32, sms);
    return t.pair ? -t.cols : t.cols;
}

// fewest token rows b200_linear sends to the tcgen05 weight-streaming GEMM instead of the GEMV (B200_GEMM_MIN_TOKENS
// overrides, for sweeps)
int gemm_min_tokens() {
    static int v = -1;
    if (v < 0) { const char* e = getenv("B200_GEMM_MIN_TOKENS"); v = e ? atoi(e) : 5; if (v < 1) v = 1; }
    return v;
}

// more than 256 token rows, plain: tokens on the M axis
static int gemm_many_rows(const void* x, const void* W, GemmParams p, int M, int N, int K, cudaStream_t s) {
    const int sms = sm_count();
    const TileChoice tile = choose_tile(kPlainTiles, M, N, p.k_blocks, false, p.out_kind == 2, sms);
    int BN = tile.cols;
    if (tile.pair) {
        const int rc = p.in_bf16 ? gemm2_tcgen05_ex(x, W, p.C, M, N, K, p.out_kind, false, 0, p.unary, 0.f, BN, s) : gemm2_tcgen05_f16(x, W, p.bias, p.C, M, N, K, false, BN, s, p.residual);
        if (rc != B200_EUNSUPPORTED) return rc;
        BN = 256;
    }
    if (N < 64) BN = 32;
    CUtensorMap ma, mb;
    p.rows_a = M; p.rows_b = N;
    p.m_tiles = (M + kBM - 1) / kBM; p.n_tiles = (N + BN - 1) / BN;
    if (!make_tma_map_2d(&ma, x, M, K, kBM) || !make_tma_map_2d(&mb, W, N, K, BN)) return B200_EUNSUPPORTED;
    const int grid = std::min(p.m_tiles * p.n_tiles, sms);
    switch (BN) {
        case 32: return gemm_launch<32, false>(ma, mb, p, grid, s);
        case 64: return gemm_launch<64, false>(ma, mb, p, grid, s);
        case 128: return gemm_launch<128, false>(ma, mb, p, grid, s);
        default: return gemm_launch<256, false>(ma, mb, p, grid, s);
    }
}

// 161 to 256 fp16 rows against a wide weight matrix (>= 60 column tiles of 256: most of the 74 cluster slots busy): one row tile of the two-CTA kernel beats a
// weight-streaming kernel's 2 waves of 128 x 256 tiles (measured, us: 22016 x 4096 at 192 / 256 rows: 60.9 / 61.4 vs 75.8 / 87.6; 12288 x 4096 at 256: 35.5 vs 44.0;
// narrow outputs keep streaming their weights: 4096 x 11008 at 256: 38.4 vs 65.5)
static bool one_row_of_pairs(int M, int N) { return M > 160 && M <= 256 && (N + 255) / 256 >= 60; }

// y[M, N] = x[M, K] * W[N, K]^T (+ bias), fp16 in / fp32 accumulate / fp16 out
int gemm_tcgen05_f16(const void* x, const void* W, const void* bias, void* y, int M, int N, int K, cudaStream_t s) {
    auto al = [](const void* q) { return (reinterpret_cast<uintptr_t>(q) & 15u) == 0; };
    if (M < 1 || N < 8 || K < 8 || (K & 7) || !al(x) || !al(W)) return B200_EUNSUPPORTED;
    static int disabled = -1;
    if (disabled < 0) { const char* e = getenv("B200_NO_TCGEN05"); disabled = (e && e[0] == '1') ? 1 : 0; }
    if (disabled) return B200_EUNSUPPORTED;
    GemmParams p{};
    p.C = y; p.bias = bias; p.K = K; p.ldc = N; p.tokens = M;
    p.k_blocks = (K + kBK - 1) / kBK;
    if (one_row_of_pairs(M, N)) {
        const int rc2 = gemm2_tcgen05_f16(x, W, bias, y, M, N, K, false, choose_tile(kPlainTiles, M, N, p.k_blocks, false, false, sm_count(), true).cols, s);
        if (rc2 != B200_EUNSUPPORTED) return rc2;
    }
    if (M <= 256) return gemm_few_rows(x, W, p, M, N, K, false, s);
    return gemm_many_rows(x, W, p, M, N, K, s);
}

// The linears of the model families of b200_serve.h: bfloat16 operands, bfloat16 or fp32 outputs, optionally with the GLU epilogue (glu 1 silu, 2 tanh-gelu:
// W = [2 N, K], gate rows then up rows, N % 128 == 0; glu 4: the clamped gated unit of common.cuh with its limit) or with the square of relu on every output
// (glu 3: not a GLU, W = [N, K]).
// Up to 256 token rows (gated units: 128) the weights stream through the M axis; above, tokens are the M axis, on one CTA or a pair.
int gemm_tcgen05_ex(const void* x, const void* W, void* y, int M, int N, int K, bool out_f32, int glu, cudaStream_t s, float glu_limit) {
    auto al = [](const void* q) { return (reinterpret_cast<uintptr_t>(q) & 15u) == 0; };
    if (M < 1 || N < 8 || K < 8 || (K & 7) || !al(x) || !al(W) || !al(y)) return B200_EUNSUPPORTED;
    const char* env = getenv("B200_NO_TCGEN05");
    if (env && env[0] == '1') return B200_EUNSUPPORTED;
    const int sms = sm_count();
    GemmParams p{};
    p.C = y; p.bias = nullptr; p.K = K; p.ldc = N; p.tokens = M;
    p.k_blocks = (K + kBK - 1) / kBK;
    p.in_bf16 = 1; p.out_kind = out_f32 ? 2 : 1; p.glu_act = glu == 2 ? 1 : glu == 4 ? 2 : 0; p.glu_limit = glu_limit;
    p.unary = glu == 3 ? 1 : 0;
    if (glu == 3) glu = 0;
    CUtensorMap ma, mb;
    if (glu) {
        if (N < 128 || (N & 127)) return B200_EUNSUPPORTED;
        // (96 rows of 28672 gated features: 110 us with the weights streaming in 1.5 waves, 107 with the tokens on the M axis; 72 rows 107 / 108)
        if (M <= 64 || (M <= 128 && N <= 128 * sms)) return gemm_few_rows(x, W, p, M, N, K, true, s);
        const TileChoice tile = choose_tile(kGatedTiles, M, N, p.k_blocks, true, out_f32, sms);
        if (tile.pair) return gemm2_tcgen05_ex(x, W, y, M, N, K, p.out_kind, true, p.glu_act, 0, glu_limit, tile.cols, s);
        p.rows_a = M; p.rows_b = N;
        p.m_tiles = (M + kBM - 1) / kBM; p.n_tiles = N / 128;
        if (!make_tma_map_2d(&ma, x, M, K, kBM) || !make_tma_map_2d(&mb, W, 2ll * N, K, 128)) return B200_EUNSUPPORTED;
        const int units = p.m_tiles * p.n_tiles;
        return gemm_launch<256, false, true>(ma, mb, p, units < sms ? units : sms, s);
    }
    return M <= 256 ? gemm_few_rows(x, W, p, M, N, K, false, s) : gemm_many_rows(x, W, p, M, N, K, s);
}
// out[M, inter] = silu(x W_gate^T) * (x W_up^T), W = [2*inter, K] (gate rows, then up rows): the gate_up GEMM of
// ffn.cpp:72 with launchAct (ffn.cpp:80) as its epilogue. Prefill shapes only (M > 256, inter % 128 == 0).
int gemm_tcgen05_f16_swiglu(const void* x, const void* W, void* out, int M, int inter, int K, cudaStream_t s) {
    auto al = [](const void* q) { return (reinterpret_cast<uintptr_t>(q) & 15u) == 0; };
    if (M <= 256 || inter < 128 || (inter & 127) || K < 8 || (K & 7) || !al(x) || !al(W) || !al(out)) return B200_EUNSUPPORTED;
    const char* e = getenv("B200_NO_TCGEN05");
    if (e && e[0] == '1') return B200_EUNSUPPORTED;
    const TileChoice tile = choose_tile(kGatedTiles, M, inter, (K + kBK - 1) / kBK, true, false, sm_count());
    if (tile.pair) {
        const int rc2 = gemm2_tcgen05_f16(x, W, nullptr, out, M, inter, K, true, tile.cols, s);
        if (rc2 != B200_EUNSUPPORTED) return rc2;
    }
    GemmParams p{};
    p.C = out; p.bias = nullptr; p.K = K; p.ldc = inter; p.tokens = M;
    p.k_blocks = (K + kBK - 1) / kBK;
    p.rows_a = M; p.rows_b = inter;
    p.m_tiles = (M + kBM - 1) / kBM; p.n_tiles = inter / 128;
    CUtensorMap ma, mb;
    if (!make_tma_map_2d(&ma, x, M, K, kBM) || !make_tma_map_2d(&mb, W, 2ll * inter, K, 128)) return B200_EUNSUPPORTED;
    const int units = p.m_tiles * p.n_tiles, sms = sm_count();
    return gemm_launch<256, false, true>(ma, mb, p, units < sms ? units : sms, s);
}

// y[M, N] = residual[M, N] + half(x W^T): launchLinearGemm followed by launchAddResidual (ffn.cpp:88 +
// context_decoder.cpp:134) in the epilogue; B200_EUNSUPPORTED below 512 rows, but for one row of pairs, and for narrow outputs
int gemm_tcgen05_f16_residual(const void* x, const void* W, const void* residual, void* y, int M, int N, int K, cudaStream_t s) {
    auto al = [](const void* q) { return (reinterpret_cast<uintptr_t>(q) & 15u) == 0; };
    if (!al(x) || !al(W) || !al(y) || !al(residual) || (N & 7)) return B200_EUNSUPPORTED;
    const char* e = getenv("B200_NO_TCGEN05");
    if (e && e[0] == '1') return B200_EUNSUPPORTED;
    if (N < 256 || K < 64 || (K & 7)) return B200_EUNSUPPORTED;
    if (one_row_of_pairs(M, N))
        return gemm2_tcgen05_f16(x, W, nullptr, y, M, N, K, false, choose_tile(kPlainTiles, M, N, (K + kBK - 1) / kBK, false, false, sm_count(), true).cols, s, residual);
    if (M < 512) return B200_EUNSUPPORTED;
    GemmParams p{};
    p.C = y; p.residual = reinterpret_cast<const __half*>(residual); p.K = K; p.ldc = N; p.tokens = M;
    p.k_blocks = (K + kBK - 1) / kBK;
    return gemm_many_rows(x, W, p, M, N, K, s);
}

}  // namespace b200
