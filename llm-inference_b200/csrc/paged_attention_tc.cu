// bfloat16 prompt portions of b200_paged_attention on tcgen05 / TMEM: 128 (token, query head) rows per tile, keys 64 at a time.
//
// What bounds it: the chain of a tile's key tiles. Per 128 x 64 scores of 128-wide heads the tensor pipe is active for 768 clocks (8 products of 64 columns at 32, 8 of 128
// columns at 64; issued one behind the other they take some 900), the special-function unit 512; but a key tile's way from its scores through softmax (1000 clocks from
// one product's end to the other's start) and weighted sum back to a free score buffer takes 3400. So two groups of softmax warps take the key tiles in turn, each with
// sums of its own, over four score buffers, and scores and weighted sums are issued by a warp each (one warp that issues both spends 1400 clocks per
// key tile on waits, products and commits): about 1150 clocks per key tile, 1620 with one group alone on an SM. Long contexts of few rows are shared out over a cluster.
//   rows        TQ tokens x the R query heads of one key head (TQ = 128 / R), so a key tile is read once for the whole group and a
//               causal edge wastes little. A CTA's window of TQ packed rows may hold the end of one sequence and the start of
//               the next: they are separate tiles, walked by neighbouring CTAs (gridDim.y is doubled, or for small batches made four times as large, when there is more than one entry; most of the others
//               find no tile and leave). Sequences that bring a single token are left to the cluster kernel of paged_decode.cu, launched behind this one.
//   warp 0      TMA: K and V tiles of 64 rows out of their page (one list lookup per tile), a ring as long as the score buffers
//   warp 1      tcgen05.mma: S = Q K^T (one group: the weighted sums too, the next tile's scores ahead of them)
//   softmax     four warps per group, a thread per row: scores are read from TMEM once, P_j goes back over its own scores and is the A operand of the second
//               product. O stays in TMEM: it is rescaled only when a row's maximum has grown by more than 2^8 since the last rescaling
//               (weights up to 256, sums in fp32). A row's largest weight is then any number instead of 1, so a weight rounded to
//               bfloat16 alone would cost more precision than against the running maximum (2.07e-3 of the result's norm, 2.03e-3
//               there): P_j is the sum of two bfloat16, hi + lo, in the 64 columns of its scores, and both are multiplied (1.61e-3, the
//               rounding of the outputs). At the end the groups' sums meet in registers.
//   last warp   two groups: O += P V
//   cluster     up to eight CTAs walk consecutive shares of a tile's key tiles; sums, references and denominators go through distributed shared
//               memory, each CTA adds and stores its part of the rows. Costs 3 us, so shares keep some eight key tiles.
// Two groups take an SM alone; one group leaves room for a second CTA, which hides what a CTA does before its first and after its last product (3.5 and 2 us):
// better only where many short tiles come in several rounds. Measured, launches of the same call one behind the other (with new inputs 0.5 to 6 more), 16 / 8 heads x 128, us, one group (two CTAs per SM, no
// sharing) / this: 2048 tokens 40.1 / 32.3, 1024 19.3 / 17.0, 64 tokens behind 4000 54 / 16, 256 behind 1000 and 4 single tokens 23.1 / 18.5, three portions up to 512 and 12 single tokens behind 4000, capped
// 119 / 107.
// Tried and taken back: query rows in TMEM and three score buffers (the buffers' round trip costs more than the shared memory saves: 17.5 against 16.8 for 1024 tokens), one warp
// for all products with three buffers (19.0), eight softmax warps per group, two threads per row (19.2: the pair has to meet at every tile), scores of 128 columns for both groups at
// once (17.1, 33.4 for 2048: the groups run in step and wait for each other).
// Rows of a page beyond the context, or ahead of what a window or a block mask leaves, may hold anything, so those V rows are cleared in the
// last and the first tile before they are multiplied by zero weights.
#include <cuda_bf16.h>

#include <algorithm>

#include "b200_serve.h"
#include "common.cuh"
#include "launch_count.h"
#include "paged_attention.cuh"
#include "tc_common.cuh"

namespace b200 {
enum { kTcPlain = 0, kTcCapped = 1, kTcBiased = 2, kTcSigmoid = 3 };
constexpr int kTcRows = 128, kTcKeys = 64;
constexpr int kTcBox = kTcKeys * 128;         // bytes of 64 rows x 64 columns
constexpr int kTcBiasFront = kTcKeys;          // distances in front of a head's staged table; behind it kTcRows + TQ: as far as a tile's last row sees where its first row sees the table's end
constexpr int kTcSorted = 192;                // windows that a CTA puts in order, at most (their keys take the place of the rows' slots and positions)
constexpr int kTcSplit = 8;                   // CTAs that share a tile's keys, at most
constexpr int kTcBiasFloats = 12288;          // at most this many staged bias numbers per CTA

// W groups of four softmax warps take the key tiles in turn, each with sums of its own: one group in each of two CTAs per SM, or two in the only one
template <int D, int DV, int W>
struct TcSmem {
    static constexpr int kRing = 2 * W;                        // score buffers, and stages of keys and of values
    static constexpr int kThreads = 64 + 128 * W + (W > 1 ? 32 : 0), kPvWarp = 2 + 4 * W;   // warps: TMA, products, softmax; two groups: scores and weighted sums have a warp each
    static constexpr int kQ = kTcRows * D * 2, kK = kTcKeys * D * 2, kV = kTcKeys * DV * 2;   // the query rows; a stage's bytes
    static constexpr int kOffK = kQ, kOffV = kOffK + kRing * kK, kOffBar = kOffV + kRing * kV, kOffSlot = kOffBar + 5 * kRing * 8;
    static constexpr int kOffMl = (kOffSlot + (2 * (kTcRows + 2) + 12) * 4 + 7) & ~7;   // (reference, sum) of every row and group
    static constexpr int kOffBias = kOffMl + (W > 1 || DV > 128 ? W * kTcRows * 8 : 0);   // (one group that shares no tile with other CTAs has no use for them)
    static constexpr int kOffSums = kRing * kTcKeys;           // tensor memory: score buffers, then the groups' sums
    static constexpr int kTmemCols = kOffSums + W * DV <= 256 ? 256 : 512, kPerSm = kTmemCols == 256 ? 2 : 1;
    static_assert(kOffSums + W * DV <= 512, "tensor memory");
    static_assert(kTcRows * DV * 4 <= kOffBar, "a CTA's sums take the operands' place");
    static_assert(kOffBias + kTcBiasFloats * 4 + 1024 <= 227 * 1024, "shared memory");
};

__device__ __forceinline__ float4 ld_cluster_v4(uint32_t addr) {
    float4 v;
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
    return v;
}
__device__ __forceinline__ float2 ld_cluster_v2(uint32_t addr) {
    float2 v;
    asm volatile("ld.shared::cluster.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(addr) : "memory");
    return v;
}

template <int D, int DV, int W, int FORM, bool SHARED>
__global__ void __launch_bounds__(TcSmem<D, DV, W>::kThreads, TcSmem<D, DV, W>::kPerSm)
paged_attn_tc_kernel(const __grid_constant__ CUtensorMap map_k, const __grid_constant__ CUtensorMap map_v, const PA a, int TQ, int parts, int skip_singles, int sorted, int split2) {   // split2: log2 of the CTAs that share a tile's keys
    using bf = __nv_bfloat16;
    using L = TcSmem<D, DV, W>;
    constexpr int NB = L::kRing, NT = L::kThreads;
    extern __shared__ __align__(1024) unsigned char tc_raw[];
    unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(tc_raw) + 1023) & ~(uintptr_t)1023);
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::kOffBar);
    uint64_t *k_full = bars, *v_full = bars + NB, *s_full = bars + 2 * NB, *p_full = bars + 3 * NB, *o_done = bars + 4 * NB;
    int* slots = reinterpret_cast<int*>(smem + L::kOffSlot);        // of the window's rows and one on either side
    int* poss = slots + kTcRows + 2;                                      // their positions
    uint32_t* masks = reinterpret_cast<uint32_t*>(poss + kTcRows + 2);    // [0..3] rows that begin a sequence, [4..7] those that begin a tile
    uint32_t* tmem_slot = masks + 8;
    volatile int* dead = reinterpret_cast<volatile int*>(masks + 9);
    float* bias_s = reinterpret_cast<float*>(smem + L::kOffBias);
    float2* ml = reinterpret_cast<float2*>(smem + L::kOffMl);

    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;   // (uniform as the compiler sees it)
    const int split = 1 << split2, rank = SHARED ? (int)blockIdx.x & (split - 1) : 0, ku = SHARED ? (int)blockIdx.x >> split2 : (int)blockIdx.x, g = ku / a.maps, mp = ku % a.maps, R = a.heads / a.kv_heads, q_units = a.heads * a.maps;
    // ---- TMEM and barriers, while the kernel before this one ends
    const bool early = parts != 2;   // every CTA has a tile, or all start at once
    if (warp == 1 && early) tmem_alloc(tmem_slot, L::kTmemCols);
    if (threadIdx.x == 0) {
#pragma unroll
        for (int b = 0; b < NB; ++b) { mbar_init(&k_full[b], 1); mbar_init(&v_full[b], 1); mbar_init(&s_full[b], 1); mbar_init(&p_full[b], 4); mbar_init(&o_done[b], 1); }
        mbar_fence_init();
        tma_prefetch_desc(&map_k);
        tma_prefetch_desc(&map_v);
        *dead = 0;
    }
    pdl_wait();

    // the windows that see the most keys come first: of one prompt the last rows, of several entries by what their first and last rows see
    const int yy = gridDim.y - 1 - blockIdx.y, part = yy % parts;
    int window = yy / parts;
    if (sorted) {
        const int n = (a.n_tokens + TQ - 1) / TQ;
        if ((int)threadIdx.x < n) {
            const int p0 = a.pos[threadIdx.x * TQ], p1 = a.pos[min(((int)threadIdx.x + 1) * TQ, a.n_tokens) - 1];
            slots[threadIdx.x] = max(p0 - pa_first_key(a, p0), p1 - pa_first_key(a, p1));
        }
        __syncthreads();
        if ((int)threadIdx.x < n) {
            const int mine = slots[threadIdx.x];
            int before = 0;
            for (int i = 0; i < n; ++i) before += slots[i] > mine || (slots[i] == mine && i < (int)threadIdx.x) ? 1 : 0;
            if (before == n - 1 - window) masks[10] = threadIdx.x;
        }
        __syncthreads();
        window = (int)masks[10];
        __syncthreads();
    }
    const int t0 = window * TQ, rows = min(TQ, a.n_tokens - t0);

    // ---- the window's tiles
    for (int i = (int)threadIdx.x - 64; i >= 0 && i < TQ + 2; i += NT - 64) {
        const int t = t0 - 1 + i;
        slots[i] = t >= 0 && t < a.n_tokens ? a.slot[t] : -1;
        poss[i] = t >= 0 && t < a.n_tokens ? a.pos[t] : 0;
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp < 4) {
        const int i = threadIdx.x;   // row of the window; slots[i + 1] is its own
        const bool in = i < rows, starts = in && (i == 0 || slots[i] != slots[i + 1]);
        const bool single = in && skip_singles && slots[i] != slots[i + 1] && slots[i + 2] != slots[i + 1];
        const uint32_t b = __ballot_sync(0xffffffffu, starts), tb = __ballot_sync(0xffffffffu, starts && !single);
        if (lane == 0) { masks[warp] = b; masks[4 + warp] = tb; }
    }
    if (parts > 1) {   // most windows hold one sequence: their second CTA leaves before it takes anything
        __syncthreads();
        int n_tiles = 0;
#pragma unroll
        for (int i = 4; i < 8; ++i) n_tiles += __popc(masks[i]);
        if (n_tiles <= part) {
            if (warp == 1 && early) tmem_dealloc(__shfl_sync(0xffffffffu, *tmem_slot, 0), L::kTmemCols);
            return;
        }
        if (warp == 1 && !early) tmem_alloc(tmem_slot, L::kTmemCols);
        tc_fence_before();
    }
    const int bias_pad = kTcBiasFront + kTcRows + TQ;
    int tn = 0;   // staged distances per head: those that a row of the window can have
    if (FORM == kTcBiased && a.dist_bias) {
        // per head: entry kTcBiasFront + distance; distances below 0 (masked keys) and beyond the table repeat its ends, so that no index needs a clamp
        for (int i = lane; i < rows; i += 32) tn = max(tn, poss[i + 1] + 1);
        tn = min(__reduce_max_sync(0xffffffffu, tn), a.dist_n);
        for (int x = 0; x < R; ++x) {
            const float* src = a.dist_bias + (size_t)(g * R + x) * a.dist_n;
#pragma unroll 4
            for (int i = threadIdx.x; i < tn + bias_pad; i += NT) bias_s[x * (tn + bias_pad) + i] = src[min(max(i - kTcBiasFront, 0), tn - 1)] * 1.4426950408889634f;
        }
    }
    __syncthreads();
    tc_fence_after();
    // the kernel for single tokens may move in (it waits for this one before it ends); TMEM has been allocated: a product kernel that moved in ahead of
    // that would wait for this one while holding it
    pdl_launch_dependents();
    const uint32_t tmem = __shfl_sync(0xffffffffu, *tmem_slot, 0), o_tmem = tmem + L::kOffSums;

    // the products of a tile, issued by one lane
    auto scores = [&](uint32_t b, bool leader) {
        constexpr uint32_t idesc_s = make_idesc_f16(kTcRows, kTcKeys) | (1u << 7) | (1u << 10);
        tc_fence_after();
        if (leader) {
            const uint64_t q_desc = make_kmajor_sw128_desc(smem_u32(smem)), kd = make_kmajor_sw128_desc(smem_u32(smem + L::kOffK)) + (uint64_t)(b * (L::kK >> 4));
            const uint32_t d = tmem + b * kTcKeys;
#pragma unroll
            for (int ks = 0; ks < D / kUmmaK; ++ks)
                umma_f16(d, q_desc + (uint64_t)((ks >> 2) * (kTcRows * 128 >> 4) + 2 * (ks & 3)), kd + (uint64_t)((ks >> 2) * (kTcBox >> 4) + 2 * (ks & 3)), idesc_s, ks > 0 ? 1u : 0u);
            umma_commit(&s_full[b]);
        }
        __syncwarp();
    };
    auto weighted = [&](int j, uint32_t b, bool leader) {
        constexpr uint32_t idesc_o = make_idesc_f16(kTcRows, DV) | (1u << 7) | (1u << 10) | (1u << 16);
        tc_fence_after();
        if (leader) {
            const uint64_t vd = make_mnmajor_sw128_desc(smem_u32(smem + L::kOffV), kTcBox, 1024u) + (uint64_t)(b * (L::kV >> 4));
            const uint32_t pa = tmem + b * kTcKeys, d = o_tmem + (uint32_t)(j % W * DV);
#pragma unroll
            for (int ks = 0; ks < 2 * kTcKeys / kUmmaK; ++ks)   // hi, then lo
                umma_f16_ts(d, pa + (uint32_t)(ks * 8), vd + (uint64_t)((ks & 3) * (2048 >> 4)), idesc_o, ks > 0 || j >= W ? 1u : 0u);
            umma_commit(&o_done[b]);
        }
        __syncwarp();
    };
    int it0 = 0, ordinal = 0;   // key tiles walked so far (stage and phase of every ring); tiles of the window seen so far
    for (int first = 0; first < rows;) {
        // the next tile: rows [first, end) of the window
        int w = first >> 5;
        uint32_t left = w < 4 ? masks[4 + w] & (0xffffffffu << (first & 31)) : 0u;
        while (left == 0u && ++w < 4) left = masks[4 + w];
        if (left == 0u || w >= 4) break;
        first = w * 32 + __ffs(left) - 1;
        int end = rows;
        {
            int v = (first + 1) >> 5;
            uint32_t nx = v < 4 ? masks[v] & (0xffffffffu << ((first + 1) & 31)) : 0u;
            while (nx == 0u && ++v < 4) nx = masks[v];
            if (nx != 0u && v < 4) end = min(end, v * 32 + __ffs(nx) - 1);
        }
        if (ordinal++ % parts != part) { first = end; continue; }
        const int tA = t0 + first, count = end - first;
        const int pA = poss[first + 1], pZ = poss[end];
        const int fA = pa_first_key(a, pA), n_all = (pZ - (fA & ~(kTcKeys - 1))) / kTcKeys + 1;
        // this CTA's share of the tile's keys: [key0, key0 + n_kt key tiles)
        const int j_lo = SHARED ? (n_all * rank) >> split2 : 0, n_kt = SHARED ? ((n_all * (rank + 1)) >> split2) - j_lo : n_all;
        const int key0 = (fA & ~(kTcKeys - 1)) + j_lo * kTcKeys;
        // ---- softmax warps: Q rows into the K-major swizzled operand (rows that this tile does not have: zeros), a thread's loads all in
        // flight together; K and V are on their way meanwhile
        if (warp >= 2 && warp < L::kPvWarp) {
            constexpr int CH = D / 8, kPass = 128 * W / CH, kBatch = kTcRows / kPass;   // 16-byte pieces per row; rows per pass of the threads
            const int tid = threadIdx.x - 64, c = tid % CH, by_r = (65536 + R - 1) / R;
            unsigned char* dst = smem + (c / 8) * (kTcRows * 128);
            const int r0 = tid / CH;
            {
                Pack16 v[kBatch];
                uint32_t flip = 0u;
#pragma unroll
                for (int i = 0; i < kBatch; ++i) {
                    const int r = r0 + i * kPass, tl = (r * by_r) >> 16, h = g * R + r - tl * R;   // r / R for r < 128
                    v[i] = Pack16{{0u, 0u, 0u, 0u}};
                    if (tl < count) {
                        v[i] = ld16(reinterpret_cast<const bf*>(a.q) + ((size_t)(tA + tl) * q_units + h * a.maps + mp) * D + c * 8);
                        flip |= pa_scale(a, h) < 0.f ? 1u << i : 0u;   // the softmax works with |scale|
                    }
                }
#pragma unroll
                for (int i = 0; i < kBatch; ++i) {
                    const int r = r0 + i * kPass;
                    if (flip >> i & 1u) {
#pragma unroll
                        for (int e = 0; e < 4; ++e) v[i].w[e] ^= 0x80008000u;
                    }
                    st16(dst + r * 128 + (((c & 7) ^ (r & 7)) << 4), v[i]);
                }
            }
            fence_proxy_async_smem();
        }
        const int* plist = a.pages + (size_t)slots[first + 1] * a.max_pages;
        __syncwarp();   // lanes without a row skipped its loads; the barrier is warp-wide
        if (warp >= 1 && warp < L::kPvWarp) asm volatile("bar.sync 1, %0;" ::"n"(32 + 128 * W) : "memory");
        tc_fence_after();

        if (SHARED && n_kt == 0) {   // fewer key tiles than CTAs
        } else if (warp == 0) {
            // K of tile j + 2 goes ahead of V of tile j, and a tile's place is looked up one tile before it is needed. A stage of keys is free when the scores
            // from it are there, a stage of values when their weighted sum is
            auto row_of = [&](int j) {
                const int k0 = key0 + min(j, n_kt - 1) * kTcKeys;
                return plist[k0 / a.page_rows] * a.page_rows + k0 % a.page_rows;
            };
            auto load = [&](uint64_t* full, uint64_t* freed, int j, int row, const CUtensorMap* map, int x, unsigned char* base, int boxes) {
                const int c = it0 + j, s = c % NB;
                mbar_wait_or_leave(&freed[s], ((uint32_t)(c / NB) & 1u) ^ 1u, dead);
                if (lane == 0) {
                    mbar_expect_tx(&full[s], boxes * kTcBox);
                    for (int b = 0; b < boxes; ++b) tma_load_2d(base + (s * boxes + b) * kTcBox, map, x + b * 64, row, &full[s]);
                }
                __syncwarp();
            };
            int row = row_of(0), row1 = row_of(1), row2 = row_of(2), row3;
            load(k_full, s_full, 0, row, &map_k, ku * D, smem + L::kOffK, D / 64);
            if (n_kt > 1) load(k_full, s_full, 1, row1, &map_k, ku * D, smem + L::kOffK, D / 64);
            for (int j = 0; j < n_kt; ++j, row = row1, row1 = row2, row2 = row3) {
                row3 = row_of(j + 3);
                if (NB > 2 && j + 2 < n_kt) load(k_full, s_full, j + 2, row2, &map_k, ku * D, smem + L::kOffK, D / 64);
                load(v_full, o_done, j, row, &map_v, g * DV, smem + L::kOffV, DV / 64);
                if (NB <= 2 && j + 2 < n_kt) load(k_full, s_full, j + 2, row2, &map_k, ku * D, smem + L::kOffK, D / 64);
            }
        } else if (warp == 1) {
            // everything that an instruction takes is uniform over the warp and mostly constant
            const int n = __shfl_sync(0xffffffffu, n_kt, 0), c0 = __shfl_sync(0xffffffffu, it0, 0);
            const bool leader = elect_one();
            uint32_t b = (uint32_t)(c0 % NB), bp = (uint32_t)(c0 / NB) & 1u;
            if (W > 1) {
                // scores of tile j as soon as its keys are there and the weights that lay in their place have been used
                for (int j = 0; j < n; ++j) {
                    mbar_wait_or_leave(&k_full[b], bp, dead);
                    mbar_wait_or_leave(&o_done[b], bp ^ 1u, dead);
                    scores(b, leader);
                    if (++b == NB) { b = 0; bp ^= 1u; }
                }
            } else {
                // the scores of tile j + 1 go ahead of the weighted sum of tile j; the weights that lay in their place are ahead of them in the tensor pipe
                mbar_wait_or_leave(&k_full[b], bp, dead);
                scores(b, leader);
                for (int j = 0; j < n; ++j) {
                    const uint32_t next = b + 1 == NB ? 0u : b + 1u;
                    if (j + 1 < n) {
                        mbar_wait_or_leave(&k_full[next], next == 0u ? bp ^ 1u : bp, dead);
                        scores(next, leader);
                    }
                    mbar_wait_or_leave(&v_full[b], bp, dead);
                    mbar_wait_or_leave(&p_full[b], bp, dead);
                    weighted(j, b, leader);
                    if (++b == NB) { b = 0; bp ^= 1u; }
                }
            }
        } else if (W > 1 && warp == L::kPvWarp) {
            const int n = __shfl_sync(0xffffffffu, n_kt, 0), c0 = __shfl_sync(0xffffffffu, it0, 0);
            uint32_t b = (uint32_t)(c0 % NB), bp = (uint32_t)(c0 / NB) & 1u;
            const bool leader = elect_one();
            for (int j = 0; j < n; ++j) {
                mbar_wait_or_leave(&v_full[b], bp, dead);
                mbar_wait_or_leave(&p_full[b], bp, dead);
                weighted(j, b, leader);
                if (++b == NB) { b = 0; bp ^= 1u; }
            }
        } else {
            // ================= softmax: a thread per row =================
            const int quarter = warp & 3, wg = (warp - 2) >> 2, r = quarter * 32 + lane, tl = r / R, hr = r % R, h = g * R + hr;
            const uint32_t my = (uint32_t)(quarter * 32) << 16;
            const bool mine = tl < count;
            const int p = mine ? poss[first + 1 + tl] : pZ, f = pa_first_key(a, p);   // rows without a token: like the last one
            const float sc = fabsf(pa_scale(a, h));
            constexpr float kLog2E = 1.4426950408889634f;
            // scores leave TMEM as q . k; plain: p = 2^(q . k * sl - m * sl), m the largest q . k; capped, biased: first x = the score times log2 e
            const float sl = fmaxf(sc * kLog2E, 1e-30f);   // never 0: a masked score is -inf
            const float over_cap = FORM == kTcCapped ? sc / a.softcap : 0.f, cap2 = a.softcap * kLog2E;
            const float hb2 = FORM == kTcSigmoid && a.head_bias ? a.head_bias[h] * kLog2E : 0.f;
            const float* brow = nullptr;
            float far_bias = 0.f;
            if (FORM == kTcBiased && a.dist_bias) {
                brow = bias_s + hr * (tn + bias_pad) + kTcBiasFront;
                far_bias = a.dist_bias[(size_t)h * a.dist_n + a.dist_n - 1] * kLog2E;
            }
            float m = -1e30f, l = 0.f;   // m: what the exponents are taken against (the scores of FORM plain unscaled)
            const float step = FORM == kTcPlain ? sl : 1.f;   // log2 units per unit of m
            // (this group's tiles: wg, wg + W, ...; place b of the rings, counted over all tiles of the CTA)
            int b = (it0 + wg) % NB, last_b = 0;
            uint32_t bp = (uint32_t)((it0 + wg) / NB) & 1u, last_bp = 0;
            for (int j = wg; j < n_kt; j += W) {
                const int k0 = key0 + j * kTcKeys;
                const uint32_t st = tmem + my + (uint32_t)(b * kTcKeys);
                mbar_wait_or_leave(&s_full[b], bp, dead);
                tc_fence_after();
                if (k0 + kTcKeys > pZ + 1 || k0 < fA) {
                    // V rows behind the context, and those ahead of the first key that any row sees: 0 * NaN must stay 0
                    mbar_wait_or_leave(&v_full[b], bp, dead);
                    for (int i = threadIdx.x - 64 - wg * 128; i < kTcKeys * (DV / 8); i += 128) {
                        const int vr = i / (DV / 8), c = i % (DV / 8);
                        if (k0 + vr >= fA && k0 + vr <= pZ) continue;
                        st_shared_v4(smem_u32(smem + L::kOffV + b * L::kV + (c / 8) * kTcBox) + (uint32_t)(vr * 128 + (c & 7) * 16), 0u, 0u, 0u, 0u);
                    }
                    fence_proxy_async_smem();
                    __syncwarp();
                }
                uint32_t sv[64];
                tmem_ld_32x32_async(st, sv);
                tmem_ld_32x32_async(st + 32u, sv + 32);
                tmem_wait_ld<64>(sv);
                auto S = [&](int e) { return __uint_as_float(sv[e]); };
                const bool whole = __all_sync(0xffffffffu, k0 + kTcKeys - 1 <= p && k0 >= f);
                if (FORM == kTcCapped) {
                    // cap * tanh(v / cap): the odd series up to x^7 while every |x| is below 0.2 (its next term is below 2^-24 of x there), else
                    // (t - 1) / (t + 1), t = e^(2x)
                    float big[2] = {0.f, 0.f};
#pragma unroll
                    for (int e = 0; e < 64; ++e) big[e & 1] = fmaxf(big[e & 1], fabsf(S(e)));
                    if (__all_sync(0xffffffffu, fmaxf(big[0], big[1]) * over_cap < 0.2f)) {
                        const uint64_t oc2 = pack2f(over_cap, over_cap), c2 = pack2f(cap2, cap2), one2 = pack2f(1.f, 1.f);
                        const uint64_t c7 = pack2f(-17.f / 315.f, -17.f / 315.f), c5 = pack2f(2.f / 15.f, 2.f / 15.f), c3 = pack2f(-1.f / 3.f, -1.f / 3.f);
#pragma unroll
                        for (int e = 0; e < 64; e += 2) {
                            const uint64_t x = mul2(pack2(sv[e], sv[e + 1]), oc2), x2 = mul2(x, x);
                            float y0, y1;
                            unpack2(mul2(mul2(c2, x), fma2(x2, fma2(x2, fma2(x2, c7, c5), c3), one2)), y0, y1);
                            sv[e] = __float_as_uint(y0);
                            sv[e + 1] = __float_as_uint(y1);
                        }
                    } else {
#pragma unroll
                        for (int e = 0; e < 64; ++e) {
                            const float t = ex2_approx(fminf(fmaxf(S(e) * over_cap * (2.f * kLog2E), -43.f), 43.f));
                            sv[e] = __float_as_uint(cap2 * __fdividef(t - 1.f, t + 1.f));
                        }
                    }
                } else if (FORM == kTcBiased) {
                    if (brow && !__all_sync(0xffffffffu, p - (k0 + kTcKeys - 1) >= a.dist_n - 1)) {
                        const int most = tn - 1 + kTcRows + TQ - kTcKeys;
                        const float* b = brow + max(min(p - k0, most), 0);
                        if (__all_sync(0xffffffffu, p - k0 <= most)) {
#pragma unroll
                            for (int e = 0; e < 64; ++e) sv[e] = __float_as_uint(fmaf(S(e), sl, b[-e]));
                        } else {
#pragma unroll
                            for (int e = 0; e < 64; ++e) sv[e] = __float_as_uint(fmaf(S(e), sl, brow[min(max(p - k0 - e, 0), tn - 1)]));
                        }
                    } else {
#pragma unroll
                        for (int e = 0; e < 64; ++e) sv[e] = __float_as_uint(fmaf(S(e), sl, far_bias));
                    }
                }
                if (!whole) {   // keys that the row does not see: -inf, a weight of 0 whatever comes
                    const int hi = p - k0, lo = f - k0;
#pragma unroll
                    for (int e = 0; e < 64; ++e) sv[e] = e <= hi ? sv[e] : 0xff800000u;
                    if (__any_sync(0xffffffffu, lo > 0)) {
#pragma unroll
                        for (int e = 0; e < 64; ++e) sv[e] = e >= lo ? sv[e] : 0xff800000u;
                    }
                }
                uint32_t pk[32], pl[32];
                if (FORM == kTcSigmoid) {   // weights that are not normalised over the keys
#pragma unroll
                    for (int e = 0; e < 64; e += 2)
                        split_bf16x2(__fdividef(1.f, 1.f + ex2_approx(-fmaf(S(e), sl, hb2))), __fdividef(1.f, 1.f + ex2_approx(-fmaf(S(e + 1), sl, hb2))), pk[e / 2], pl[e / 2]);
                } else {
                    float mx[4] = {-1e30f, -1e30f, -1e30f, -1e30f};
#pragma unroll
                    for (int e = 0; e < 64; ++e) mx[e & 3] = fmaxf(mx[e & 3], S(e));
                    const float top = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3]));
                    const bool grown = (top - m) * step > 8.f;
                    if (j >= W && __any_sync(0xffffffffu, grown)) {
                        mbar_wait_or_leave(&o_done[last_b], last_bp, dead);   // this group's tile before
                        tc_fence_after();
                        const float alpha = grown ? ex2_approx((m - top) * step) : 1.f;
#pragma unroll 1
                        for (int c = 0; c < DV; c += 32) {
                            uint32_t ov[32];
                            tmem_ld_32x32_async(o_tmem + my + (uint32_t)(wg * DV + c), ov);
                            tmem_wait_ld<32>(ov);
#pragma unroll
                            for (int e = 0; e < 32; ++e) ov[e] = __float_as_uint(__uint_as_float(ov[e]) * alpha);
                            tmem_st_32x32(o_tmem + my + (uint32_t)(wg * DV + c), ov);
                        }
                        l *= alpha;
                    }
                    if (grown) m = top;
                    const float ms = -m * step;
                    const uint64_t sl2 = pack2f(step, step), nm2 = pack2f(ms, ms);
                    uint64_t rs2[2] = {0ull, 0ull};
#pragma unroll
                    for (int e = 0; e < 64; e += 2) {
                        float a0, a1;
                        unpack2(FORM == kTcPlain ? fma2(pack2(sv[e], sv[e + 1]), sl2, nm2) : add2(pack2(sv[e], sv[e + 1]), nm2), a0, a1);
                        a0 = ex2_approx(a0);
                        a1 = ex2_approx(a1);
                        split_bf16x2(a0, a1, pk[e / 2], pl[e / 2]);
                        rs2[(e / 2) & 1] = add2(rs2[(e / 2) & 1], pack2f(a0, a1));
                    }
                    float r0, r1;
                    unpack2(add2(rs2[0], rs2[1]), r0, r1);
                    l += r0 + r1;
                }
                tmem_st_32x32(st, pk);
                tmem_st_32x32(st + 32u, pl);
                tmem_wait_st();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&p_full[b]);
                last_b = b; last_bp = bp;
                b += W;
                if (b >= NB) { b -= NB; bp ^= 1u; }
            }
            // the last W products (each on sums of its own)
#pragma unroll
            for (int w = 0; w < W; ++w)
                if (n_kt > w) {
                    const int c = it0 + n_kt - 1 - w;
                    mbar_wait_or_leave(&o_done[c % NB], (uint32_t)(c / NB) & 1u, dead);
                }
            tc_fence_after();
            // the groups' sums of a row against the larger of their references; each group stores its part of the columns
            float m2 = m * step, share[W];
            share[0] = 1.f;
            if (W > 1) {
                ml[wg * kTcRows + r] = make_float2(m2, l);
                asm volatile("bar.sync 2, %0;" ::"n"(128 * W) : "memory");
                const float2 other = ml[(wg ^ 1) * kTcRows + r];
                const bool both = n_kt > 1;   // otherwise the second group has seen no key, and its sums hold anything
                if (!both) {
                    if (wg == 1) { m2 = other.x; l = other.y; }
                    share[W - 1] = 0.f;
                } else if (FORM == kTcSigmoid) {
                    share[W - 1] = 1.f;
                } else {
                    const float M = fmaxf(m2, other.x), mine_f = ex2_approx(m2 - M), other_f = ex2_approx(other.x - M);
                    l = l * mine_f + other.y * other_f;
                    m2 = M;
                    share[0] = wg == 0 ? mine_f : other_f;
                    share[W - 1] = wg == 0 ? other_f : mine_f;
                }
            }
            constexpr int COLS = DV / W;
            auto sums = [&](int c, uint32_t (&ov)[32]) {   // columns [c, c + 32) of the row
                tmem_ld_32x32_async(o_tmem + my + (uint32_t)c, ov);
                if (W > 1 && n_kt > 1) {
                    uint32_t o2[32];
                    tmem_ld_32x32_async(o_tmem + my + (uint32_t)(DV + c), o2);
                    tmem_wait_ld<32>(ov);
                    tmem_wait_ld<32>(o2);
#pragma unroll
                    for (int e = 0; e < 32; ++e) ov[e] = __float_as_uint(fmaf(__uint_as_float(ov[e]), share[0], __uint_as_float(o2[e]) * share[W - 1]));
                } else
                    tmem_wait_ld<32>(ov);
            };
            if (SHARED) {
                // the row's sums to shared memory, for all CTAs of the tile: every product that reads the operands there is done
                const uint32_t at = smem_u32(smem) + (uint32_t)(r * DV * 4);
#pragma unroll 1
                for (int c = wg * COLS; c < (wg + 1) * COLS; c += 32) {
                    uint32_t ov[32];
                    sums(c, ov);
#pragma unroll
                    for (int q = 0; q < 8; ++q) st_shared_v4(at + (uint32_t)(((c / 4 + q) ^ (r & 7)) << 4), ov[4 * q], ov[4 * q + 1], ov[4 * q + 2], ov[4 * q + 3]);
                }
                if (W > 1) asm volatile("bar.sync 2, %0;" ::"n"(128 * W) : "memory");   // both groups have read each other's numbers
                if (wg == 0) ml[r] = make_float2(m2, *dead ? __int_as_float(0x7fffffff) : l);
            } else {
                const float sink_w = FORM == kTcSigmoid ? 0.f : a.sink ? 1.f : a.denom_bias, s2 = a.sink ? a.sink[h] * kLog2E : 0.f;
                const size_t dst = ((size_t)(tA + tl) * q_units + h * a.maps + mp) * DV;
                // division by the weights' sum, in which the sink counts
                float inv = 1.f;
                if (FORM != kTcSigmoid) {
                    const float M = sink_w > 0.f ? fmaxf(m2, s2) : m2, fo = ex2_approx(m2 - M);
                    inv = fo / (l * fo + (sink_w > 0.f ? sink_w * ex2_approx(s2 - M) : 0.f));
                }
                if (*dead) inv = __int_as_float(0x7fffffff);
#pragma unroll 1
                for (int c = wg * COLS; c < (wg + 1) * COLS; c += 32) {
                    uint32_t ov[32];
                    __syncwarp();
                    sums(c, ov);
                    if (!mine) continue;
                    if (a.out_f32) {
                        float4* d = reinterpret_cast<float4*>(reinterpret_cast<float*>(a.out) + dst + c);
#pragma unroll
                        for (int e = 0; e < 32; e += 4)
                            d[e / 4] = make_float4(__uint_as_float(ov[e]) * inv, __uint_as_float(ov[e + 1]) * inv, __uint_as_float(ov[e + 2]) * inv, __uint_as_float(ov[e + 3]) * inv);
                    } else {
#pragma unroll
                        for (int q = 0; q < 4; ++q) {
                            Pack16 w;
#pragma unroll
                            for (int e = 0; e < 4; ++e) w.w[e] = pa_pack(__uint_as_float(ov[q * 8 + 2 * e]) * inv, __uint_as_float(ov[q * 8 + 2 * e + 1]) * inv);
                            st16(reinterpret_cast<bf*>(a.out) + dst + c + q * 8, w);
                        }
                    }
                }
            }
            tc_fence_before();
        }
        if (SHARED) {
            __syncwarp();
            // 1 / split of the rows each: the shares are added in the order of their keys, the sink joins here
            cluster_sync_all();
            const int own = kTcRows >> split2, own0 = rank * own;
            // kBatch loads of 16 bytes on their way per thread: kBatch / split places of `split` shares each
            constexpr int kBatch = 8;
            static_assert(kBatch >= kTcSplit, "a place's shares together");
            const int by_r = (65536 + R - 1) / R;
            const int total = min(own * (DV / 4), max(0, count * R - own0) * (DV / 4)), places = kBatch >> split2;
            const float sink_w = FORM == kTcSigmoid ? 0.f : a.sink ? 1.f : a.denom_bias;
            for (int i0 = threadIdx.x; i0 < total; i0 += NT * places) {
                float4 o[kBatch];
                float2 w[kBatch];
#pragma unroll
                for (int e = 0; e < kBatch; ++e) {
                    const int x = e & (split - 1), i = i0 + (e >> split2) * NT, r = own0 + i / (DV / 4), c4 = i % (DV / 4);
                    w[e] = make_float2(-INFINITY, 0.f);
                    o[e] = make_float4(0.f, 0.f, 0.f, 0.f);
                    if (i < total && ((n_all * (x + 1)) >> split2) > ((n_all * x) >> split2)) {
                        w[e] = ld_cluster_v2(mapa_shared(smem_u32(ml + r), (uint32_t)x));
                        o[e] = ld_cluster_v4(mapa_shared(smem_u32(smem) + (uint32_t)(r * DV * 4 + ((c4 ^ (r & 7)) << 4)), (uint32_t)x));
                    }
                }
                float M = 0.f, sum = 0.f;
                float4 t = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
                for (int e = 0; e < kBatch; ++e) {
                    const int x = e & (split - 1), i = i0 + (e >> split2) * NT, r = own0 + i / (DV / 4), c4 = i % (DV / 4), tl = (r * by_r) >> 16, h = g * R + r - tl * R;
                    if (i >= total) continue;
                    // against the running largest reference
                    if (x == 0) { M = -INFINITY; sum = 0.f; t = make_float4(0.f, 0.f, 0.f, 0.f); }
                    if (w[e].x != -INFINITY) {
                        const float Mn = fmaxf(M, w[e].x), fo = FORM == kTcSigmoid ? 1.f : ex2_approx(M - Mn), fn = FORM == kTcSigmoid ? 1.f : ex2_approx(w[e].x - Mn);
                        M = Mn;
                        sum = fmaf(sum, fo, w[e].y * fn);
                        t.x = fmaf(t.x, fo, o[e].x * fn); t.y = fmaf(t.y, fo, o[e].y * fn); t.z = fmaf(t.z, fo, o[e].z * fn); t.w = fmaf(t.w, fo, o[e].w * fn);
                    }
                    if (x == split - 1) {
                        // (of weights that are not normalised the sum is 0, or NaN where a wait was given up)
                        float inv = 1.f + sum;
                        if (FORM != kTcSigmoid) {
                            const float s2 = a.sink ? a.sink[h] * 1.4426950408889634f : 0.f, top = sink_w > 0.f ? fmaxf(M, s2) : M, fo = ex2_approx(M - top);
                            inv = fo / (sum * fo + (sink_w > 0.f ? sink_w * ex2_approx(s2 - top) : 0.f));
                        }
                        const size_t dst = ((size_t)(tA + tl) * q_units + h * a.maps + mp) * DV + c4 * 4;
                        if (a.out_f32) *reinterpret_cast<float4*>(reinterpret_cast<float*>(a.out) + dst) = make_float4(t.x * inv, t.y * inv, t.z * inv, t.w * inv);
                        else *reinterpret_cast<uint2*>(reinterpret_cast<bf*>(a.out) + dst) = make_uint2(pa_pack(t.x * inv, t.y * inv), pa_pack(t.z * inv, t.w * inv));
                    }
                }
            }
            __syncwarp();
            fence_proxy_async_smem();   // TMA writes the next tile's keys where the sums lay
            cluster_sync_all();
        }
        it0 += n_kt;
        first = end;
        __syncthreads();   // the next tile's Q rows and products come after everybody is done with this one's
        tc_fence_after();
    }
    if (*dead) {   // a wait was given up: what is still under way must not land behind this CTA's end
        linger();
        __syncthreads();
    }
    if (warp == 1) tmem_dealloc(tmem, L::kTmemCols);
}

struct TcPlan {
    long long windows;
    int parts, sorted, split2, bias;   // split2: log2 of the CTAs that share a tile's keys; bias: staged numbers
    bool two_groups;   // else one, and two CTAs per SM
    bool chained;      // launched programmatically
};

template <int D, int DV, int W, int FORM, bool SHARED>
static int launch_tc(const PA& a, const TcPlan& p, cudaStream_t s) {
    using L = TcSmem<D, DV, W>;
    const int TQ = kTcRows / (a.heads / a.kv_heads), units = a.kv_heads * a.maps;
    static unsigned long long done = 0;
    cudaError_t e = ensure_max_dynamic_smem((const void*)paged_attn_tc_kernel<D, DV, W, FORM, SHARED>, L::kOffBias + kTcBiasFloats * 4 + 1024, done);
    if (e != cudaSuccess) return (int)e;
    CUtensorMap mk, mv;
    // the pool's height is not part of the call: any row that an int can name
    constexpr long long kAnyRow = (1ll << 31) - 1;
    if (!make_tma_map_2d(&mk, a.k_pool, kAnyRow, a.kv_heads * a.maps * D, kTcKeys) || !make_tma_map_2d(&mv, a.v_pool, kAnyRow, a.kv_heads * DV, kTcKeys)) return -1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)(units << p.split2), (unsigned)(p.windows * p.parts));
    cfg.blockDim = dim3(L::kThreads);
    cfg.dynamicSmemBytes = L::kOffBias + p.bias * 4 + 1024;
    cfg.stream = s;
    cudaLaunchAttribute at[2]{};
    cfg.attrs = at;
    if (SHARED) {
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = 1u << p.split2;
        at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
        cfg.numAttrs = 1;
    }
    if (p.chained && pdl_enabled()) {
        at[cfg.numAttrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        at[cfg.numAttrs++].val.programmaticStreamSerializationAllowed = 1;
    }
    e = cudaLaunchKernelEx(&cfg, paged_attn_tc_kernel<D, DV, W, FORM, SHARED>, mk, mv, a, TQ, p.parts, p.parts - 1, p.sorted, p.split2);
    return e != cudaSuccess ? (int)e : (int)cudaGetLastError();
}

template <int D, int DV, int FORM>
static int launch_tc_groups(const PA& a, const TcPlan& p, cudaStream_t s) {
    if constexpr (DV <= 128) {
        if (!p.two_groups) return launch_tc<D, DV, 1, FORM, false>(a, p, s);
        return p.split2 ? launch_tc<D, DV, 2, FORM, true>(a, p, s) : launch_tc<D, DV, 2, FORM, false>(a, p, s);
    } else
        return p.split2 ? launch_tc<D, DV, 1, FORM, true>(a, p, s) : launch_tc<D, DV, 1, FORM, false>(a, p, s);
}

template <int D, int DV>
static int launch_tc_for(const PA& a, const TcPlan& p, cudaStream_t s) {
    if (a.sigmoid) return launch_tc_groups<D, DV, kTcSigmoid>(a, p, s);
    if (a.softcap > 0.f) return launch_tc_groups<D, DV, kTcCapped>(a, p, s);
    if (a.dist_bias) return launch_tc_groups<D, DV, kTcBiased>(a, p, s);
    return launch_tc_groups<D, DV, kTcPlain>(a, p, s);
}

int paged_attention_tc(const PA& a, int longest_entry, int longest_seen, int longest_context, cudaStream_t s) {
    if (longest_entry < 0 || longest_entry > a.n_tokens) longest_entry = 0;   // a limit instead of the batch's own number: unknown
    const int R = a.heads / a.kv_heads;
    // a cap beside a sink or a bias keeps the row kernel, whose weights stay in 32 bits
    if (R > 8 || a.page_rows % kTcKeys || (a.softcap > 0.f && (a.dist_bias || a.sink)) || a.kv_heads * a.maps > 65535) return -1;
    // a short portion of one sequence, 64-wide heads, a distance bias: the fixed part of a CTA and a bias per score outweigh products half as long, and the
    // mma.sync tiles are faster (16 / 8 heads, us there / here: 40 tokens 11.2 / 13.3, 400 tokens 17.4 / 20.5, 100 behind 1000 31.7 / 35.8; but 700 tokens
    // 28.7 / 27.8, 2048 tokens 73 / 48). Where other sequences are beside it their single tokens decide
    if (a.dist_bias && a.dim == 64 && a.vdim == 64 && a.chunk == 0 && a.window == 0 && a.n_tokens == longest_entry && a.n_tokens <= 512 && longest_seen > 0 && longest_seen <= 1200) return -1;
    TcPlan p{};
    const int TQ = kTcRows / R, units = a.kv_heads * a.maps, sms = sm_count();
    const bool several = a.n_tokens != longest_entry;   // more than one entry, as far as the host knows
    p.windows = (a.n_tokens + TQ - 1) / TQ;
    p.parts = several ? 2 : 1;
    if (p.windows * 2 > 65535) return -1;
    if (a.dist_bias && !a.sigmoid && !(a.softcap > 0.f)) {
        if (a.dist_n > kTcBiasFloats) return -1;
        p.bias = R * (a.dist_n + kTcBiasFront + kTcRows + TQ);
        if (p.bias > kTcBiasFloats) return -1;
    }
    const long long tiles = p.windows * units;
    const int steps = longest_seen > 0 ? (longest_seen + kTcKeys - 1) / kTcKeys : 0;
    // tiles of several entries that come in more than one round: up to 32 key tiles each, two CTAs per SM that hide each other's start and end are faster (16 / 8 heads x 128, us, one group / two: three
    // portions of up to 680 20.7 / 25.7, of up to 512 behind 300 23.1 / 26.7, behind 1000 39.4 / 45.2), beyond that the shorter chain (behind 2000 63.7 / 65.9, behind 4000, capped, 119 / 107)
    // One entry: the shorter chain as long as it decides. Beyond one round the tiles of rank sms and sms + 1 share an SM: keys that they see together against a tenth more than the longest tile sees; beyond two rounds of
    // tiles two CTAs per SM, a cap, which lengthens the chain, aside (one group for short tiles beyond two rounds), and unless staged bias numbers leave room for one CTA only (us, one group / two, 16 / 8 heads x 128: 2048 tokens 37.1 / 32.0, 2400 42.6 / 45.3, 3000 53.1 / 61.8, capped
    // 2400 54.5 / 51.1, 4000 112 / 108; window of 1024, fp32 outputs, 1300 27.6 / 21.9, 1700 29.9 / 30.3, 2048 34.1 / 37.9, 4000 61.8 / 71.0; 32 / 16 heads, 600 behind 3000 64.2 / 78.8; 16 / 4, biased, 3000 95 / 76)
    // fp32 outputs keep two groups, whose chains of sums are half as long: 5.1e-6 of the result's norm for 2048 tokens behind a window of 1024, 5.5e-6 in one group (34.1 against 37.9 us).
    // (values of 256 columns: one group, whose sums take an SM alone all the same)
    auto fits_twice = [&](int bytes) { return bytes + p.bias * 4 + 1024 + 1024 <= 228 * 1024 / 2; };   // (what the driver keeps per CTA)
    const bool twice = a.dim == 64 ? fits_twice(TcSmem<64, 64, 1>::kOffBias) : fits_twice(TcSmem<128, 128, 1>::kOffBias);
    const double before = std::max(0, longest_context - a.n_tokens), shared_by = before + a.n_tokens * std::max(0.0, 1.0 - (double)sms / tiles);
    // (a portion of up to a block that begins inside one has its longest tiles at either end)
    const bool uneven = a.chunk > 0 ? before > 0 && a.n_tokens <= a.chunk : 2 * std::min<double>(shared_by, longest_seen) > 1.1 * longest_seen;
    const bool short_tiles = several && tiles > sms && steps <= 32, many_tiles = !several && !a.out_f32 && tiles > sms && steps > 0 && (a.softcap > 0.f ? tiles > 2 * sms && steps <= 32 : tiles > 2 * sms || uneven) && twice;
    p.two_groups = a.vdim > 128 || !(short_tiles || many_tiles);
    // shared key tiles: while the clusters fit beside each other (clusters of four and eight do not fill every group of SMs), leave room for single tokens if there may be some, and keep eight key tiles or more
    // per CTA (us at 1 / 2 / 4 / 8 CTAs: 100 tokens behind 3000 38.5 / 26.1 / 18.5 / 28.2, 300 40.5 / 27.6 / 36.6 / 45.0, 64 and 4 single ones behind 1000 19.0 / 16.6 / 14.5 / 17.6, behind 300 11.8 / 12.8 / 12.4 / 14.6,
    // 512 and 8 single ones behind 4000 57.0 / 61.5 / 77.5 / 115)
    const long long room = several ? 2 * sms / 3 : sms;
    while (p.two_groups && p.split2 < (tiles * 8 <= sms / 2 ? 3 : 2) && (tiles << (p.split2 + 1)) <= room && steps >= 12 && steps >= 8 << p.split2) ++p.split2;
    // CTAs that share a window's tiles: four where they all start at once (portions of 53, 45 and 33 tokens lie in one window and a bit: 16 heads x 128, capped, two / four 13.6 / 9.1 us)
    if (several && p.split2 == 0 && tiles * 4 <= sms) p.parts = 4;
    // several rounds: the longest tiles first (three portions of up to 512 behind 4000: 88.4 / 83.0 us)
    p.sorted = several && p.windows > 1 && p.windows <= kTcSorted && (tiles << p.split2) > sms && !short_tiles;
    // Tiles that start before the kernel ahead has ended sit down where room comes first: two to an SM where each should have one, or, in several rounds, out of their order (us behind a residual norm, programmatically / not,
    // 16 / 8 heads x 128: one group, 600 tokens 16.2 / 14.3, 1500, window of 1024, 34.3 / 28.4, three portions of 512 and 4 single tokens behind 300 24.3 / 23.5; sorted, behind 4000, capped, 112 / 110; but two groups, 100
    // tokens 7.0 / 7.7, 2048 31.5 / 32.7)
    p.chained = p.two_groups && !p.sorted;
    const int singles = a.n_tokens - longest_entry;   // at most; with several entries at least one
    const long long free = (p.two_groups ? 2 : 1) * std::max(0ll, (p.two_groups ? sms : 2 * sms) - (tiles << p.split2));   // CTAs of single tokens that fit beside the tiles'
    int rc = -1;
    if (a.dim == 128 && a.vdim == 128) rc = launch_tc_for<128, 128>(a, p, s);
    else if (a.dim == 64 && a.vdim == 64) rc = launch_tc_for<64, 64>(a, p, s);
    else if (a.dim == 128 && a.vdim == 256) rc = launch_tc_for<128, 256>(a, p, s);
    if (rc != 0) return rc;
    count_launch();
    if (several) return paged_decode(a, longest_seen, singles, free, s);   // the sequences that bring one token, on what the tiles leave free
    return 0;
}

}  // namespace b200
