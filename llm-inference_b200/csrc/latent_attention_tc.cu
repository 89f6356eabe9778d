// bfloat16 prompt portions of b200_latent_attention_ex on tcgen05 / TMEM: 128 (token, head) rows per tile, cached rows 64 at a time, 256 output
// columns per CTA (two CTAs form the 512 columns of a row, each with scores of its own: a whole row of sums would fill TMEM alone).
//
// What bounds it: per 128 x 64 scores over rows of 576 the tensor pipe is active for 2176 clocks (nine chunks of 64 dimensions, 1152, then the weighted
// sum over 256 columns, 1024; with what lies between products 2500), three times the softmax; so the next tile's scores run under the softmax of this one, and enough of the cached
// rows has to be on its way. Shared memory is what limits that: the query rows alone are 144 KB. Four of their chunks lie in TMEM as
// first operands instead, beside the sums (256 columns) and two score buffers, which leaves room for 144 KB of cached rows:
//   chunks of 64 dimensions that this CTA only scores with:  all of a row's at once (rows of 640: half of them), a ring of two such groups, given back after their products
//   the four chunks whose columns it also sums:              two groups, given back after the weighted sum; they are the operand of both products
//   warp 0      TMA: the query's chunks in fp32, through the places of the cached rows; then chunks of 64 rows x 64 dimensions out of their page
//   warp 1      tcgen05.mma: scores of a tile as soon as its rows are there and their buffer is free
//   warps 2-5   the query rows (rounded to bfloat16, as in the mma.sync kernel), then the softmax, a thread per row, as in paged_attention_tc.cu
//   warp 6      tcgen05.mma: the weighted sums. (One warp for both, and a barrier per chunk, spent 3550 clocks a tile on waits, products and commits; now 2970)
// The weights go back over their scores as the sum of two bfloat16; the sums are rescaled only when a row's maximum has grown by more than 2^8. A window of
// packed tokens that holds several sequences is walked tile by tile (latent_tc_parts CTAs share it).
// Measured, 2048 tokens, rows of 576, 16 heads, 512 columns out (floor 44 us): the mma.sync tiles of latent_attention.cu 856 us; launches of the same call one behind the other: one warp for all products
// 171, a second one 157, the query by TMA too 144 (with new inputs, whose query rows come from memory, 177 before and 158 now); 592 tokens behind 1024 62 / 57 / 53, 400 and 319 behind 900 with 3 single
// ones 73 / 67 / 65. A CTA's fixed part (its query rows, results 5000 clocks) is as much as five of its key tiles.
// Tried and taken back: the query's rows read by the four warps one row after the other, 16 bytes per thread (26000 clocks: three times the address and place arithmetic, on one warp per scheduler).
#include <cuda_bf16.h>

#include "b200_serve.h"
#include "common.cuh"
#include "latent_attention.cuh"
#include "launch_count.h"
#include "tc_common.cuh"

namespace b200 {

constexpr int kLtRows = 128, kLtKeys = 64, kLtThreads = 224, kLtChunk = kLtKeys * 128, kLtQChunk = kLtRows * 128, kLtV = 4;

template <int NCH>   // chunks of a cached row
struct LtSmem {
    static constexpr int kScoreOnly = NCH - kLtV, kInTmem = NCH >= 8 ? 4 : 0;   // chunks without sums; of these, how many of the query's lie in TMEM
    // what is only scored with comes kGroup chunks at a time, through a ring of kRing such groups
    static constexpr int kGroup = kScoreOnly == 6 ? 3 : kScoreOnly > 1 ? kScoreOnly : 1, kGroups = kScoreOnly / kGroup, kRing = kScoreOnly > 1 ? 2 : 4;
    static constexpr int kOffRing = (NCH - kInTmem) * kLtQChunk, kOffV = kOffRing + kRing * kGroup * kLtChunk, kOffBar = kOffV + 2 * kLtV * kLtChunk;
    // the query's chunks come in fp32 through the cached rows' places, kSlots at a time
    static constexpr int kSlot = 2 * kLtQChunk, kSlots = (kOffBar - kOffRing) / kSlot;
    static constexpr int kBars = 2 * kRing + 8 + 2 * kSlots, kOffSlot = kOffBar + kBars * 8, kTotal = kOffSlot + (kLtRows + 2 + 16) * 4 + 1024;
    static_assert(kTotal <= 227 * 1024, "one CTA per SM");
};

struct LtArgs {
    const float* qa; float* out; const int* pages; const int* slot; const int* pos; const float* sink;
    int max_pages, page_rows, n_tokens, heads, rank, window, TQ, parts;
    float scale;
};

template <int NCH>
__global__ void __launch_bounds__(kLtThreads, 1) latent_attn_tc_kernel(const __grid_constant__ CUtensorMap map, const __grid_constant__ CUtensorMap map_q, const LtArgs a) {
    using L = LtSmem<NCH>;
    constexpr int NS = L::kScoreOnly, QT = L::kInTmem;
    extern __shared__ __align__(1024) unsigned char lt_raw[];
    unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(lt_raw) + 1023) & ~(uintptr_t)1023);
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::kOffBar);
    constexpr int RING = L::kRing, GC = L::kGroup, GN = L::kGroups;
    uint64_t *r_full = bars, *r_empty = bars + RING, *v_full = bars + 2 * RING, *s_full = v_full + 2, *p_full = v_full + 4, *o_done = v_full + 6, *q_full = v_full + 8, *q_empty = q_full + L::kSlots;
    int* slots = reinterpret_cast<int*>(smem + L::kOffSlot);
    uint32_t* masks = reinterpret_cast<uint32_t*>(slots + kLtRows + 2);
    uint32_t* tmem_slot = masks + 8;
    volatile int* dead = reinterpret_cast<volatile int*>(masks + 9);

    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    const int half = blockIdx.x, H = a.heads, TQ = a.TQ;
    const int yy = gridDim.y - 1 - blockIdx.y, part = yy % a.parts, t0 = yy / a.parts * TQ, rows = min(TQ, a.n_tokens - t0);
    // the order in which a row's chunks are taken: those without sums first
    auto chunk_of = [&](int o) { return o >= NS ? half * kLtV + o - NS : o < half * kLtV ? o : o + kLtV; };

    pdl_wait();
    // ---- the window's tiles (paged_attention_tc.cu): rows that begin a sequence
    if (threadIdx.x < TQ) slots[threadIdx.x] = (int)threadIdx.x < rows ? a.slot[t0 + threadIdx.x] : -1;
    if (threadIdx.x == 0) *dead = 0;
    __syncthreads();
    if (warp < 4) {
        const int i = threadIdx.x;
        const uint32_t b = __ballot_sync(0xffffffffu, i < rows && (i == 0 || slots[i] != slots[i - 1]));
        if (lane == 0) masks[warp] = b;
    }
    __syncthreads();
    int n_tiles = 0;
#pragma unroll
    for (int i = 0; i < 4; ++i) n_tiles += __popc(masks[i]);
    if (n_tiles <= part) return;   // nothing here for this CTA (no barrier, no TMEM yet)
    if (warp == 1) tmem_alloc(tmem_slot, 512);
    if (threadIdx.x == 0) {
        for (int i = 0; i < RING; ++i) { mbar_init(&r_full[i], 1); mbar_init(&r_empty[i], 1); }
        for (int s = 0; s < 2; ++s) {
            mbar_init(&v_full[s], 1);
            mbar_init(&s_full[s], 1); mbar_init(&p_full[s], 4);
            mbar_init(&o_done[s], 1);
        }
        for (int i = 0; i < L::kSlots; ++i) { mbar_init(&q_full[i], 1); mbar_init(&q_empty[i], 4); }
        mbar_fence_init();
        tma_prefetch_desc(&map);
        tma_prefetch_desc(&map_q);
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    pdl_launch_dependents();   // (behind the allocation: a product kernel that moved in ahead of it would wait for this one while holding tensor memory)
    const uint32_t tmem = __shfl_sync(0xffffffffu, *tmem_slot, 0), o_tmem = tmem, s_tmem = tmem + 256, q_tmem = tmem + 256 + 2 * kLtKeys;

    int it0 = 0, q0 = 0, ordinal = 0;   // key tiles, query chunks, tiles of the window so far
    for (int first = 0; first < rows;) {
        int w = first >> 5;
        uint32_t left = w < 4 ? masks[w] & (0xffffffffu << (first & 31)) : 0u;
        while (left == 0u && ++w < 4) left = masks[w];
        if (left == 0u || w >= 4) break;
        first = w * 32 + __ffs(left) - 1;
        int end = rows;
        {
            int v = (first + 1) >> 5;
            uint32_t nx = v < 4 ? masks[v] & (0xffffffffu << ((first + 1) & 31)) : 0u;
            while (nx == 0u && ++v < 4) nx = masks[v];
            if (nx != 0u && v < 4) end = min(end, v * 32 + __ffs(nx) - 1);
        }
        if (ordinal++ % a.parts != part) { first = end; continue; }
        const int tA = t0 + first, count = end - first;
        const int pA = a.pos[tA], pZ = a.pos[tA + count - 1];
        const int key0 = (a.window > 0 ? max(0, pA - a.window + 1) : 0) & ~(kLtKeys - 1), n_kt = (pZ - key0) / kLtKeys + 1;
        const int* plist = a.pages + (size_t)slots[first] * a.max_pages;

        // ---- query rows: chunks [QT, NCH) to shared memory, chunks [0, QT) to TMEM, rounded to bfloat16 on the way. TMA brings them in fp32 into the places of the cached rows,
        // kSlots chunks under way (64 KB of loads per SM, requested by the four warps themselves, came at 16 bytes a clock, 18000 clocks in all)
        if (warp == 0) {
            for (int o = 0; o < NCH; ++o) {
                const int q = q0 + o, i = q % L::kSlots;
                mbar_wait_or_leave(&q_empty[i], ((uint32_t)(q / L::kSlots) & 1u) ^ 1u, dead);
                if (lane == 0) {
                    mbar_expect_tx(&q_full[i], L::kSlot);
#pragma unroll
                    for (int b = 0; b < 2; ++b) tma_load_2d(smem + L::kOffRing + i * L::kSlot + b * kLtQChunk, &map_q, chunk_of(o) * 128 + b * 64, tA * H, &q_full[i]);   // (in 16-bit columns)
                }
                __syncwarp();
            }
        } else if (warp >= 2 && warp < 6) {
            const int tid = threadIdx.x - 64, c = tid % 8, rb = tid / 8, quarter = warp & 3, mr = quarter * 32 + lane;
            const uint32_t flip = a.scale < 0.f ? 0x80008000u : 0u;   // the softmax works with |scale|
            auto ld4 = [&](uint32_t at) {
                float4 v;
                asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(at) : "memory");
                return v;
            };
            auto pack4 = [&](const float4& x, uint32_t* o) {
                const __nv_bfloat162 b0 = __floats2bfloat162_rn(x.x, x.y), b1 = __floats2bfloat162_rn(x.z, x.w);
                o[0] = *reinterpret_cast<const uint32_t*>(&b0) ^ flip;
                o[1] = *reinterpret_cast<const uint32_t*>(&b1) ^ flip;
            };
#pragma unroll 1
            for (int o = 0; o < NCH; ++o) {
                const int q = q0 + o, i = q % L::kSlots;
                const uint32_t src = smem_u32(smem + L::kOffRing + i * L::kSlot);
                mbar_wait_or_leave(&q_full[i], (uint32_t)(q / L::kSlots) & 1u, dead);
                if (o < QT) {   // a row per lane
                    uint32_t t[32];
#pragma unroll
                    for (int e = 0; e < 16; ++e) pack4(ld4(src + (uint32_t)((e >> 3) * kLtQChunk + mr * 128 + (((e & 7) ^ (mr & 7)) << 4))), t + 2 * e);
                    tmem_st_32x32(q_tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(o * 32), t);
                } else {        // columns 8 c .. 8 c + 7 of every 16th row (the halves of the lanes begin with different pieces: no bank conflicts)
                    const uint32_t dst = smem_u32(smem + (o - QT) * kLtQChunk), from = src + (uint32_t)((c >> 2) * kLtQChunk), swap = c >> 2;
                    uint32_t v[8][4];
#pragma unroll
                    for (int k = 0; k < 8; ++k) {
                        const int r = rb + k * 16;
                        const uint32_t piece = (uint32_t)((c & 3) * 2) + swap;
                        const float4 x = ld4(from + (uint32_t)(r * 128) + ((piece ^ (uint32_t)(r & 7)) << 4)), y = ld4(from + (uint32_t)(r * 128) + ((piece ^ 1u ^ (uint32_t)(r & 7)) << 4));
                        uint32_t px[2], py[2];
                        pack4(x, px);
                        pack4(y, py);
                        v[k][0] = swap ? py[0] : px[0]; v[k][1] = swap ? py[1] : px[1];
                        v[k][2] = swap ? px[0] : py[0]; v[k][3] = swap ? px[1] : py[1];
                    }
#pragma unroll
                    for (int k = 0; k < 8; ++k) {
                        const int r = rb + k * 16;
                        st_shared_v4(dst + (uint32_t)(r * 128 + ((c ^ (r & 7)) << 4)), v[k][0], v[k][1], v[k][2], v[k][3]);
                    }
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(&q_empty[i]);
            }
            tmem_wait_st();
            fence_proxy_async_smem();
            tc_fence_before();
        }
        if (warp == 0 || (warp >= 2 && warp < 6)) asm volatile("bar.sync 3, 160;" ::: "memory");   // the cached rows may come
        if (warp >= 1 && warp < 6) asm volatile("bar.sync 1, 160;" ::: "memory");
        tc_fence_after();

        if (warp == 0) {
            auto row_of = [&](int j) {
                const int k0 = key0 + min(j, n_kt - 1) * kLtKeys;
                return plist[k0 / a.page_rows] * a.page_rows + k0 % a.page_rows;
            };
            int row = row_of(0), next;
            for (int j = 0; j < n_kt; ++j, row = next) {
                const int it = it0 + j, s = it & 1;
                next = row_of(j + 1);
                for (int gi = 0; gi < GN; ++gi) {
                    const int q = it * GN + gi, i = q % RING;
                    mbar_wait_or_leave(&r_empty[i], ((uint32_t)(q / RING) & 1u) ^ 1u, dead);
                    if (lane == 0) {
                        mbar_expect_tx(&r_full[i], GC * kLtChunk);
#pragma unroll
                        for (int o = 0; o < GC; ++o) tma_load_2d(smem + L::kOffRing + (i * GC + o) * kLtChunk, &map, chunk_of(gi * GC + o) * 64, row, &r_full[i]);
                    }
                    __syncwarp();
                }
                mbar_wait_or_leave(&o_done[s], ((uint32_t)(it >> 1) & 1u) ^ 1u, dead);   // (the weighted sum is what last reads them)
                if (lane == 0) {
                    mbar_expect_tx(&v_full[s], kLtV * kLtChunk);
#pragma unroll
                    for (int c = 0; c < kLtV; ++c) tma_load_2d(smem + L::kOffV + (s * kLtV + c) * kLtChunk, &map, (half * kLtV + c) * 64, row, &v_full[s]);
                }
                __syncwarp();
            }
        } else if (warp == 1) {
            // scores of tile i as soon as its rows are there and the weights that lay in their place have been used
            constexpr uint32_t idesc_s = make_idesc_f16(kLtRows, kLtKeys) | (1u << 7) | (1u << 10);
            const uint64_t q_desc = make_kmajor_sw128_desc(smem_u32(smem)), r_desc = make_kmajor_sw128_desc(smem_u32(smem + L::kOffRing));
            const uint64_t vk_desc = make_kmajor_sw128_desc(smem_u32(smem + L::kOffV));
            const int n = __shfl_sync(0xffffffffu, n_kt, 0), c0 = __shfl_sync(0xffffffffu, it0, 0);
            const bool leader = elect_one();
            for (int i = c0; i < c0 + n; ++i) {
                const uint32_t s = (uint32_t)i & 1u, d = s_tmem + s * kLtKeys, ph = (uint32_t)(i >> 1) & 1u;
                mbar_wait_or_leave(&o_done[s], ph ^ 1u, dead);
#pragma unroll
                for (int gi = 0; gi < GN; ++gi) {
                    const uint32_t q = (uint32_t)(i * GN + gi), x = q % RING;
                    mbar_wait_or_leave(&r_full[x], (q / RING) & 1u, dead);
                    tc_fence_after();
                    if (leader) {
                        const uint64_t kd = r_desc + (uint64_t)(x * (GC * kLtChunk >> 4));
#pragma unroll
                        for (int oo = 0; oo < GC; ++oo) {
                            const int o = gi * GC + oo;
#pragma unroll
                            for (int k = 0; k < 4; ++k) {
                                if (o < QT) umma_f16_ts(d, q_tmem + (uint32_t)(o * 32 + k * 8), kd + (uint64_t)(oo * (kLtChunk >> 4) + 2 * k), idesc_s, o > 0 || k > 0 ? 1u : 0u);
                                else umma_f16(d, q_desc + (uint64_t)((o - QT) * (kLtQChunk >> 4) + 2 * k), kd + (uint64_t)(oo * (kLtChunk >> 4) + 2 * k), idesc_s, o > 0 || k > 0 ? 1u : 0u);
                            }
                        }
                        umma_commit(&r_empty[x]);
                    }
                    __syncwarp();
                }
                mbar_wait_or_leave(&v_full[s], ph, dead);
                tc_fence_after();
                if (leader) {
                    const uint64_t kd = vk_desc + (uint64_t)(s * (kLtV * kLtChunk >> 4));
#pragma unroll
                    for (int o = 0; o < kLtV; ++o)
#pragma unroll
                        for (int k = 0; k < 4; ++k)
                            umma_f16(d, q_desc + (uint64_t)((NS - QT + o) * (kLtQChunk >> 4) + 2 * k), kd + (uint64_t)(o * (kLtChunk >> 4) + 2 * k), idesc_s, NS > 0 || o > 0 || k > 0 ? 1u : 0u);
                    umma_commit(&s_full[s]);
                }
                __syncwarp();
            }
        } else if (warp == 6) {
            constexpr uint32_t idesc_o = make_idesc_f16(kLtRows, 256) | (1u << 7) | (1u << 10) | (1u << 16);
            const uint64_t vm_desc = make_mnmajor_sw128_desc(smem_u32(smem + L::kOffV), kLtChunk, 1024u);
            const int n = __shfl_sync(0xffffffffu, n_kt, 0), c0 = __shfl_sync(0xffffffffu, it0, 0);
            const bool leader = elect_one();
            for (int j = 0; j < n; ++j) {
                const uint32_t s = (uint32_t)(c0 + j) & 1u;
                mbar_wait_or_leave(&p_full[s], (uint32_t)((c0 + j) >> 1) & 1u, dead);
                tc_fence_after();
                if (leader) {
                    const uint64_t vd = vm_desc + (uint64_t)(s * (kLtV * kLtChunk >> 4));
#pragma unroll
                    for (int ks = 0; ks < 2 * kLtKeys / kUmmaK; ++ks)   // hi, then lo
                        umma_f16_ts(o_tmem, s_tmem + s * kLtKeys + (uint32_t)(ks * 8), vd + (uint64_t)((ks & 3) * (2048 >> 4)), idesc_o, j > 0 || ks > 0 ? 1u : 0u);
                    umma_commit(&o_done[s]);
                }
                __syncwarp();
            }
        } else {
            const int quarter = warp & 3, r = quarter * 32 + lane, by_h = (65536 + H - 1) / H, tl = (r * by_h) >> 16, h = r - tl * H;
            const uint32_t my = (uint32_t)(quarter * 32) << 16;
            const bool mine = tl < count;
            const int p = mine ? a.pos[tA + tl] : -1, f = mine && a.window > 0 ? max(0, p - a.window + 1) : 0;
            constexpr float kLog2E = 1.4426950408889634f;
            const float sl = fmaxf(fabsf(a.scale) * kLog2E, 1e-30f);   // never 0: a masked score is -inf
            float m = -1e30f, l = 0.f;
            for (int j = 0; j < n_kt; ++j) {
                const int it = it0 + j, s = it & 1, k0 = key0 + j * kLtKeys;
                const uint32_t st = s_tmem + my + (uint32_t)(s * kLtKeys);
                mbar_wait_or_leave(&s_full[s], (uint32_t)(it >> 1) & 1u, dead);
                tc_fence_after();
                if (k0 + kLtKeys > pZ + 1) {   // rows behind the context: 0 * NaN must stay 0 (their scores have been formed already)
                    const int valid = pZ + 1 - k0;
                    for (int i = threadIdx.x - 64; i < (kLtKeys - valid) * kLtV * 8; i += 128) {
                        const int vr = valid + i / (kLtV * 8), c = i % (kLtV * 8);
                        st_shared_v4(smem_u32(smem + L::kOffV + (s * kLtV + c / 8) * kLtChunk) + (uint32_t)(vr * 128 + (c & 7) * 16), 0u, 0u, 0u, 0u);
                    }
                    fence_proxy_async_smem();
                    __syncwarp();
                }
                uint32_t sv[64];
                tmem_ld_32x32_async(st, sv);
                tmem_ld_32x32_async(st + 32u, sv + 32);
                tmem_wait_ld<64>(sv);
                if (!__all_sync(0xffffffffu, k0 + kLtKeys - 1 <= p && k0 >= f)) {   // keys that the row does not see
                    const int hi = p - k0, lo = f - k0;
#pragma unroll
                    for (int e = 0; e < 64; ++e) sv[e] = e <= hi && e >= lo ? sv[e] : 0xff800000u;
                }
                float mx[4] = {-1e30f, -1e30f, -1e30f, -1e30f};
#pragma unroll
                for (int e = 0; e < 64; ++e) mx[e & 3] = fmaxf(mx[e & 3], __uint_as_float(sv[e]));
                const float top = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3]));
                const bool grown = (top - m) * sl > 8.f;
                if (j > 0 && __any_sync(0xffffffffu, grown)) {
                    mbar_wait_or_leave(&o_done[s ^ 1], (uint32_t)((it - 1) >> 1) & 1u, dead);
                    tc_fence_after();
                    const float alpha = grown ? ex2_approx((m - top) * sl) : 1.f;
#pragma unroll 1
                    for (int c = 0; c < 256; c += 32) {
                        uint32_t ov[32];
                        tmem_ld_32x32_async(o_tmem + my + (uint32_t)c, ov);
                        tmem_wait_ld<32>(ov);
#pragma unroll
                        for (int e = 0; e < 32; ++e) ov[e] = __float_as_uint(__uint_as_float(ov[e]) * alpha);
                        tmem_st_32x32(o_tmem + my + (uint32_t)c, ov);
                    }
                    l *= alpha;
                }
                if (grown) m = top;
                const float ms = -m * sl;
                const uint64_t sl2 = pack2f(sl, sl), nm2 = pack2f(ms, ms);
                uint64_t rs2[2] = {0ull, 0ull};
                uint32_t pk[32], pl[32];
#pragma unroll
                for (int e = 0; e < 64; e += 2) {
                    float a0, a1;
                    unpack2(fma2(pack2(sv[e], sv[e + 1]), sl2, nm2), a0, a1);
                    a0 = ex2_approx(a0);
                    a1 = ex2_approx(a1);
                    split_bf16x2(a0, a1, pk[e / 2], pl[e / 2]);
                    rs2[(e / 2) & 1] = add2(rs2[(e / 2) & 1], pack2f(a0, a1));
                }
                float r0, r1;
                unpack2(add2(rs2[0], rs2[1]), r0, r1);
                l += r0 + r1;
                tmem_st_32x32(st, pk);
                tmem_st_32x32(st + 32u, pl);
                tmem_wait_st();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&p_full[s]);
            }
            // ---- division by the weights' sum, in which the sink counts
            const int last = it0 + n_kt - 1;
            mbar_wait_or_leave(&o_done[last & 1], (uint32_t)(last >> 1) & 1u, dead);
            tc_fence_after();
            const float m2 = m * sl, s2 = a.sink ? a.sink[h] * kLog2E : 0.f, M = a.sink ? fmaxf(m2, s2) : m2, fo = ex2_approx(m2 - M);
            float inv = fo / (l * fo + (a.sink ? ex2_approx(s2 - M) : 0.f));
            if (*dead) inv = __int_as_float(0x7fffffff);
            // 32 rows x 32 columns per warp through the place of the query's first rows (every product that reads them is done), so that a store
            // instruction writes whole lines
            const uint32_t stg = smem_u32(smem) + (uint32_t)(warp - 2) * 4096u;
#pragma unroll 1
            for (int c = 0; c < 256; c += 32) {
                uint32_t ov[32];
                __syncwarp();
                tmem_ld_32x32_async(o_tmem + my + (uint32_t)c, ov);
                tmem_wait_ld<32>(ov);
#pragma unroll
                for (int q = 0; q < 8; ++q)
                    st_shared_v4(stg + (uint32_t)(lane * 128 + ((q ^ (lane & 7)) << 4)), __float_as_uint(__uint_as_float(ov[4 * q]) * inv), __float_as_uint(__uint_as_float(ov[4 * q + 1]) * inv),
                                 __float_as_uint(__uint_as_float(ov[4 * q + 2]) * inv), __float_as_uint(__uint_as_float(ov[4 * q + 3]) * inv));
                __syncwarp();
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const int lr = i * 4 + (lane >> 3), q = lane & 7, rr = quarter * 32 + lr, t = (rr * by_h) >> 16, hh = rr - t * H;
                    float4 o4;
                    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(o4.x), "=f"(o4.y), "=f"(o4.z), "=f"(o4.w) : "r"(stg + (uint32_t)(lr * 128 + ((q ^ (lr & 7)) << 4))) : "memory");
                    if (t < count) *reinterpret_cast<float4*>(a.out + ((size_t)(tA + t) * H + hh) * a.rank + half * 256 + c + q * 4) = o4;
                }
            }
            tc_fence_before();
        }
        it0 += n_kt;
        q0 += NCH;
        first = end;
        __syncthreads();   // the next tile's query rows and products come after everybody is done with this one's
        tc_fence_after();
    }
    if (*dead) {   // a wait was given up: what is still under way must not land behind this CTA's end
        linger();
        __syncthreads();
    }
    if (warp == 1) tmem_dealloc(tmem, 512);
}

template <int NCH>
static int launch_lt(const b200_latent_attention_args& a, int halves, cudaStream_t s) {
    CUtensorMap map, map_q;
    constexpr long long kAnyRow = (1ll << 31) - 1;   // the pool's height is not part of the call: any row that an int can name
    // (the query's fp32 as pairs of 16-bit columns)
    if (!make_tma_map_2d(&map, a.pool, kAnyRow, a.rank, kLtKeys) || !make_tma_map_2d(&map_q, a.qa, (long long)a.n_tokens * a.heads, 2 * a.rank, kLtRows)) return -1;
    static unsigned long long done = 0;
    const cudaError_t e = ensure_max_dynamic_smem((const void*)latent_attn_tc_kernel<NCH>, LtSmem<NCH>::kTotal, done);
    if (e != cudaSuccess) return (int)e;
    const int TQ = kLtRows / a.heads, parts = latent_tc_parts(a.n_tokens, a.longest_entry, a.heads, halves);
    const long long windows = (a.n_tokens + TQ - 1) / TQ;
    if (windows * parts > 65535) return -1;
    const LtArgs la{a.qa, a.out, a.pages, a.slot, a.pos, a.sink, a.max_pages, a.page_rows, a.n_tokens, a.heads, a.rank, a.window, TQ, parts, a.scale};
    const cudaError_t le = launch_chained(latent_attn_tc_kernel<NCH>, dim3((unsigned)halves, (unsigned)(windows * parts)), dim3(kLtThreads), (size_t)LtSmem<NCH>::kTotal, s, map, map_q, la);
    if (le != cudaSuccess) return (int)le;
    return (int)cudaGetLastError();
}

int latent_attention_tc(const b200_latent_attention_args& a, int out_cols, cudaStream_t s) {
    auto al16 = [](const void* q) { return (reinterpret_cast<uintptr_t>(q) & 15u) == 0; };
    if (a.heads > 64 || out_cols % 256 || out_cols > 512 || a.page_rows % kLtKeys || !al16(a.qa) || !al16(a.out) || !al16(a.pool)) return -1;
    const int halves = out_cols / 256;
    int rc = -1;
    if (halves == 2 && a.rank == 576) rc = launch_lt<9>(a, halves, s);
    else if (halves == 2 && a.rank == 512) rc = launch_lt<8>(a, halves, s);
    else if (halves == 2 && a.rank == 640) rc = launch_lt<10>(a, halves, s);
    else if (halves == 1 && a.rank == 320) rc = launch_lt<5>(a, halves, s);
    else if (halves == 1 && a.rank == 256) rc = launch_lt<4>(a, halves, s);
    if (rc == 0) count_launch();
    return rc;
}

}  // namespace b200
