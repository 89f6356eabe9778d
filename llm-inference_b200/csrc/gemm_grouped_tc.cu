// The routed products of b200_gemm_grouped (groups of gathered rows, bfloat16, W [N, K] per group) on tcgen05 / TMEM.
//
// What bounds it: the weights, read once (a group owns a few to a few hundred rows), so they lie on the M axis of the products, 128 rows
// (gated units: 64 gate rows and the 64 up rows of the same features) per CTA, and a group's rows ride along as the N extent, up to 128 or 192 of
// them, in an instruction just wide enough. Weights come by TMA; the rows, which lie anywhere, by cp.async into the same swizzled layout
// (warps 2-5, 16 bytes at a time, a few stages ahead). A stage takes the weights' 16 KB and what the block's rows need, so few rows get more stages. Two or three CTAs share an SM:
// a second round of few blocks, which read their weights again, cost half as much again as one round that holds all tiles (there the weights come at some 0.55 of the copy rate). The sums leave TMEM through shared memory,
// so that a token's features are stored side by side and the epilogue sees one element like the other kernels of this entry point.
//   grid: feature tiles x groups x blocks of rows; what lies behind a group's rows leaves at once
// Measured (before: the mma.sync tiles of gemm_grouped.cu): 512 rows, four of 16 experts each, 2048 -> gated 1024 -> 2048, with dispatch and
// combine: 247 -> 107 us, 106 -> 83 with the rows announced a stage earlier and the epilogue decided before its passes, 82 -> 71 with blocks of 192 rows.
// Tried and taken back: 256 rows and one CTA per SM with 192 KB of stages (58.6 against 48.8 us for 200 rows, 80.3 against 79.1 for 512).
#include <cuda_bf16.h>

#include <algorithm>
#include <type_traits>

#include "b200_serve.h"
#include "common.cuh"
#include "gemm_grouped.cuh"
#include "launch_count.h"
#include "tc_common.cuh"

namespace b200 {

constexpr int kGtM = 128, kGtK = 64, kGtThreads = 192;

template <int BN, int PER_SM>   // rows of a block at most, CTAs per SM
struct GtSmem {
    // The ring takes as many stages as the group's rows leave room for: the weights' 16 KB and 128 bytes per row (in sixteens) each
    // Blocks of 192 rows are for nearly two CTAs on every SM: more than 128 KB on their way to an SM are slower again (routed layers of 2048 -> 1024, 16 experts, four per row, us at up to 3 / 4 / 6 stages: 64
    // rows 42.7 / 41.9 / 43.1, 100 44.9 / 44.4 / 45.9; 200, 50 rows a group, 48.2 / 48.9 / 49.2). Where fewer CTAs share an SM more stages pay (1024 -> 1536, two per row, 33 rows 30.0 / 28.6 / 28.1)
    static constexpr int kMaxStages = BN > 128 ? 4 : 6, kTmemCols = BN > 128 ? 256 : BN;
    static constexpr int kRing = PER_SM == 3 ? 72 * 1024 : BN > 128 ? 108 * 1024 : 100 * 1024;
    static constexpr int kTotal = kRing + (2 * kMaxStages + 1) * 8 + 16 + 1024;
    static_assert(BN * kGtM * 4 <= kRing && kRing >= 2 * (kGtM + BN) * kGtK * 2, "the sums take the place of the stages; two stages at least");
    static_assert(kTotal + 1024 <= 228 * 1024 / PER_SM, "CTAs per SM");
};

template <int BN, int PER_SM, typename TC, bool GLU>
__global__ void __launch_bounds__(kGtThreads, PER_SM) gemm_grouped_tc_kernel(const __grid_constant__ CUtensorMap map_w, const GG g) {
    using S = GtSmem<BN, PER_SM>;
    using bf = __nv_bfloat16;
    constexpr uint32_t A_BYTES = kGtM * kGtK * 2;
    extern __shared__ unsigned char smem_raw[];
    unsigned char* tiles = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    uint64_t* full_bar = reinterpret_cast<uint64_t*>(tiles + S::kRing);
    uint64_t* empty_bar = full_bar + S::kMaxStages;
    uint64_t* acc_full = empty_bar + S::kMaxStages;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_full + 1);
    volatile int* dead = reinterpret_cast<volatile int*>(tmem_slot + 1);
    float* om = reinterpret_cast<float*>(tiles);   // [rows][128]: the sums, once the stages have been used

    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    pdl_wait();
    const int z = blockIdx.y, row0 = g.group_off[z] + (int)blockIdx.z * BN, rows = min(BN, g.group_off[z + 1] - row0);
    if (rows <= 0) return;
    const int stage_bytes = (int)A_BYTES + (rows + 15) / 16 * 16 * 128, stages = min(BN > 128 && rows > 48 ? 3 : S::kMaxStages, S::kRing / stage_bytes);
    if (threadIdx.x == 0) {
        for (int s = 0; s < stages; ++s) {
            mbar_init(&full_bar[s], 1 + 4);   // the weights, and the four warps that bring the rows
            mbar_init(&empty_bar[s], 1);
        }
        mbar_init(acc_full, 1);
        *dead = 0;
        mbar_fence_init();
        tma_prefetch_desc(&map_w);
    }
    if (warp == 1) tmem_alloc(tmem_slot, S::kTmemCols);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = __shfl_sync(0xffffffffu, *tmem_slot, 0);
    pdl_launch_dependents();
    const int k_blocks = (g.K + kGtK - 1) / kGtK;

    if (warp == 0) {
        const int wrow = z * (GLU ? 2 * g.N : g.N) + (int)blockIdx.x * (GLU ? 64 : kGtM);
        int s = 0;
        uint32_t par = 1u;
        for (int kb = 0; kb < k_blocks; ++kb) {
            mbar_wait_or_leave(&empty_bar[s], par, dead);
            if (lane == 0) {
                unsigned char* sa = tiles + (size_t)s * stage_bytes;
                mbar_expect_tx(&full_bar[s], A_BYTES);
                tma_load_2d(sa, &map_w, kb * kGtK, wrow, &full_bar[s]);
                tma_load_2d(sa + A_BYTES / 2, &map_w, kb * kGtK, GLU ? wrow + g.N : wrow + 64, &full_bar[s]);
            }
            __syncwarp();
            if (++s == stages) { s = 0; par ^= 1u; }
        }
    } else if (warp == 1) {
        const uint32_t idesc = make_idesc_f16(kGtM, 16) + ((uint32_t)((rows + 15) / 16 - 1) << 18) + ((1u << 7) | (1u << 10));   // N: rows rounded up to 16
        const bool leader = elect_one();
        const uint64_t a0 = make_kmajor_sw128_desc(smem_u32(tiles)), b0 = make_kmajor_sw128_desc(smem_u32(tiles + A_BYTES));
        int s = 0;
        uint32_t par = 0u;
        for (int kb = 0; kb < k_blocks; ++kb) {
            mbar_wait_or_leave(&full_bar[s], par, dead);
            tc_fence_after();
            if (leader) {
                const uint64_t off = (uint64_t)(s * (stage_bytes >> 4));
#pragma unroll
                for (int k = 0; k < kGtK / kUmmaK; ++k) umma_f16(tmem, a0 + off + (uint64_t)(2 * k), b0 + off + (uint64_t)(2 * k), idesc, (kb > 0 || k > 0) ? 1u : 0u);
                umma_commit(&empty_bar[s]);
                if (kb == k_blocks - 1) umma_commit(acc_full);
            }
            __syncwarp();
            if (++s == stages) { s = 0; par ^= 1u; }
        }
    } else {
        // ---- rows: a thread brings 16-byte piece c of rows r, r + 16, ...
        constexpr int NR = BN / 16;
        const int tid = threadIdx.x - 64, c = tid % 8, r0 = tid / 8;
        const bf* src[NR];
#pragma unroll
        for (int i = 0; i < NR; ++i) {
            const int r = r0 + i * 16;
            src[i] = nullptr;
            if (r < rows) src[i] = reinterpret_cast<const bf*>(g.A) + (size_t)(g.a_rows ? g.a_rows[row0 + r] : row0 + r) * g.lda + c * 8;
        }
        const uint32_t dst0 = smem_u32(tiles + A_BYTES) + (uint32_t)(r0 * 128 + ((c ^ (r0 & 7)) << 4));   // (rows 16 apart share r & 7)
        // stages of rows that are under way when one is announced: two fewer than there are (with all of them a stage was announced only after the products of
        // the one before)
        auto bring = [&](auto lag) {
            constexpr int LAG = decltype(lag)::value;
            int s = 0, told = 0;   // the stage that is filled, the one that is announced next
            uint32_t par = 1u;
            auto announce = [&]() {
                fence_proxy_async_smem();
                __syncwarp();
                if (lane == 0) mbar_arrive(&full_bar[told]);
                if (++told == stages) told = 0;
            };
            for (int kb = 0; kb < k_blocks; ++kb) {
                mbar_wait_or_leave(&empty_bar[s], par, dead);
                const bool in = kb * kGtK + c * 8 < g.K;
#pragma unroll
                for (int i = 0; i < NR; ++i) {
                    const bool ok = in && src[i] != nullptr;
                    asm volatile(   // (a sixteen without rows has no place in the stage)
                        "{\n"
                        ".reg .pred p;\n"
                        "setp.lt.s32 p, %3, %4;\n"
                        "@p cp.async.cg.shared.global [%0], [%1], 16, %2;\n"
                        "}\n" ::"r"(dst0 + (uint32_t)(s * stage_bytes + i * 16 * 128)),
                        "l"(ok ? src[i] + kb * kGtK : reinterpret_cast<const bf*>(g.A)), "r"(ok ? 16 : 0), "r"(i * 16), "r"(rows) : "memory");
                }
                __syncwarp();   // the lanes close their group of copies together
                asm volatile("cp.async.commit_group;" ::: "memory");
                if (kb >= LAG) {
                    asm volatile("cp.async.wait_group %0;" ::"n"(LAG) : "memory");
                    announce();
                }
                if (++s == stages) { s = 0; par ^= 1u; }
            }
            asm volatile("cp.async.wait_group 0;" ::: "memory");
            for (int kb = max(0, k_blocks - LAG); kb < k_blocks; ++kb) announce();
        };
        if (stages >= 5) bring(std::integral_constant<int, 3>{});
        else if (stages == 4) bring(std::integral_constant<int, 2>{});
        else if (stages == 3) bring(std::integral_constant<int, 1>{});
        else bring(std::integral_constant<int, 0>{});
        // ---- sums to shared memory
        const int quarter = warp & 3;
        mbar_wait_or_leave(acc_full, 0, dead);
        const bool gone = *dead != 0;
        if (gone) linger();   // a wait was given up: no late weights on the sums, or behind this CTA's end
        tc_fence_after();
        const uint32_t taddr = tmem + ((uint32_t)(quarter * 32) << 16);
#pragma unroll 1
        for (int c0 = 0; c0 < rows; c0 += 32) {
            uint32_t v[32];
            tmem_ld_32x32(taddr + (uint32_t)c0, v);
#pragma unroll
            for (int j = 0; j < 32; ++j)
                if (c0 + j < rows) om[(c0 + j) * kGtM + quarter * 32 + lane] = gone ? __int_as_float(0x7fffffff) : __uint_as_float(v[j]);
        }
        tc_fence_before();
    }
    __syncthreads();
    constexpr int F = GLU ? 64 : kGtM;
    const int n0 = blockIdx.x * F;
    TC* C = reinterpret_cast<TC*>(g.C);
    const bool wide = (g.ldc & 3) == 0 && (reinterpret_cast<uintptr_t>(g.C) & 15u) == 0;
    // four features of a row per thread and pass; what an element needs besides its sum is decided before the passes (asked for element by element it took as long
    // as the products: 20000 clocks for 128 rows)
    auto passes = [&](auto value) {
#pragma unroll 4
        for (int i = threadIdx.x; i < rows * (F / 4); i += kGtThreads) {
            const int r = i / (F / 4), f0 = i % (F / 4) * 4, n = n0 + f0;
            const long long row = row0 + r;
            const float4 a = *reinterpret_cast<const float4*>(om + r * kGtM + f0);
            float4 b = make_float4(0.f, 0.f, 0.f, 0.f);
            if (GLU) b = *reinterpret_cast<const float4*>(om + r * kGtM + 64 + f0);
            float v[4] = {a.x, a.y, a.z, a.w};
            const float u[4] = {b.x, b.y, b.z, b.w};
            value(row, n, v, u);
            if (wide && n + 4 <= g.N) {
                if constexpr (sizeof(TC) == 4) *reinterpret_cast<float4*>(C + row * g.ldc + n) = make_float4(v[0], v[1], v[2], v[3]);
                else {
                    const __nv_bfloat162 x = __floats2bfloat162_rn(v[0], v[1]), y = __floats2bfloat162_rn(v[2], v[3]);
                    *reinterpret_cast<uint2*>(C + row * g.ldc + n) = make_uint2(*reinterpret_cast<const uint32_t*>(&x), *reinterpret_cast<const uint32_t*>(&y));
                }
            } else {
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    if (n + e < g.N) C[row * g.ldc + n + e] = DT<TC>::from_f(v[e]);
            }
        }
    };
    if (GLU) {   // (the units of tile epilogues: without branches, see tile_silu)
        auto scaled = [&](long long row, float (&v)[4], const float (&u)[4], auto unit) {
            const float f = g.row_scale ? g.row_scale[row] : 1.f;   // the row of A was meant to be scaled: the products are linear in it
#pragma unroll
            for (int e = 0; e < 4; ++e) v[e] = g.row_scale ? unit(v[e] * f, u[e] * f) : unit(v[e], u[e]);
        };
        if (g.epi == B200_GG_GLU) passes([&](long long row, int, float (&v)[4], const float (&u)[4]) { scaled(row, v, u, [](float x, float y) { return tile_silu(x) * y; }); });
        else if (g.epi == B200_GG_GLU_GELU) passes([&](long long row, int, float (&v)[4], const float (&u)[4]) { scaled(row, v, u, [](float x, float y) { return tile_gelu_tanh(x) * y; }); });
        else passes([&](long long row, int, float (&v)[4], const float (&u)[4]) { scaled(row, v, u, [&](float x, float y) { return tile_glu_clamp(x, y, g.epi_param); }); });
    } else if (g.epi == B200_GG_NONE && !g.row_scale)
        passes([](long long, int, float (&)[4], const float (&)[4]) {});
    else
        passes([&](long long row, int n, float (&v)[4], const float (&)[4]) {
#pragma unroll
            for (int e = 0; e < 4; ++e)
                if (n + e < g.N) v[e] = gg_value(g, row, n + e, v[e], 0.f, 0);
        });
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem, S::kTmemCols);
    }
}

template <int BN, int PER_SM, typename TC, bool GLU>
static int launch_gt(const GG& g, int groups, cudaStream_t s) {
    CUtensorMap map;
    if (!make_tma_map_2d(&map, g.W, (long long)groups * (GLU ? 2 * g.N : g.N), g.K, 64)) return -1;
    auto kern = gemm_grouped_tc_kernel<BN, PER_SM, TC, GLU>;
    static unsigned long long done = 0;
    const cudaError_t e = ensure_max_dynamic_smem((const void*)kern, GtSmem<BN, PER_SM>::kTotal, done);
    if (e != cudaSuccess) return (int)e;
    const int F = GLU ? 64 : kGtM;
    const dim3 grid((g.N + F - 1) / F, groups, (g.M + BN - 1) / BN);
    if (grid.z > 65535) return -1;
    return (int)launch_k(kern, grid, dim3(kGtThreads), (size_t)GtSmem<BN, PER_SM>::kTotal, s, true, map, g);
}

template <typename TC>
int gg_launch_tc(const GG& g, int groups, cudaStream_t s) {
    const bool glu = gg_is_glu(g.epi);
    auto al16 = [](const void* q) { return (reinterpret_cast<uintptr_t>(q) & 15u) == 0; };
    // weights of all groups as one matrix without gaps, rows that 16-byte pieces can fetch
    if (!g.group_off || (g.K & 7) || (g.lda & 7) || g.ldw != g.K || g.sW != (long long)(glu ? 2 : 1) * g.N * g.K || !al16(g.A) || !al16(g.W) || (glu && g.N % 64) || groups > 65535) return -1;
    auto go = [&](auto bn, auto per_sm) {
        constexpr int BN = decltype(bn)::value, PER_SM = decltype(per_sm)::value;
        return glu ? launch_gt<BN, PER_SM, TC, true>(g, groups, s) : launch_gt<BN, PER_SM, TC, false>(g, groups, s);
    };
    using std::integral_constant;
    if (g.M <= 32) return go(integral_constant<int, 32>{}, integral_constant<int, 2>{});
    // One round of CTAs, as far as that goes without knowing the groups (us for a routed layer with dispatch and combination, 128 rows and two CTAs per SM / this; 16 experts, three or four per row): feature tiles for three CTAs per
    // SM, 2048 -> 1408, 50 rows 61.1 / 54.6, 129 65.8 / 55.4, 512 89.3 / 78.8; for nearly two, 2048 -> 1024, blocks of up to 192 rows so that few groups come twice, 400 rows 72.9 / 66.5, 512 82.2 / 70.7 (but 1024 -> 640, where
    // there is room for second blocks, 29.6 / 36.3)
    const long long tiles = (long long)groups * ((g.N + (glu ? 64 : kGtM) - 1) / (glu ? 64 : kGtM));
    const int sms = sm_count();
    if (tiles > 2 * sms && tiles <= 3 * sms) return go(integral_constant<int, 128>{}, integral_constant<int, 3>{});
    if (2 * tiles > 3 * sms && tiles <= 2 * sms) return go(integral_constant<int, 192>{}, integral_constant<int, 2>{});
    return go(integral_constant<int, 128>{}, integral_constant<int, 2>{});
}
template int gg_launch_tc<float>(const GG&, int, cudaStream_t);
template int gg_launch_tc<__nv_bfloat16>(const GG&, int, cudaStream_t);

}  // namespace b200
