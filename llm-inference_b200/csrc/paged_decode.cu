// Single tokens of b200_paged_attention in bfloat16 (decode batches): every (token, key head) is served by one cluster of CTAs that
// share the token's context, one launch, no workspace.
//
// What bounds it: the keys and values, read once (8 KB per 16 keys of 128 x 128), so the kernel has to keep enough of them on their way
// and spend few instructions per byte. A warp walks its own run of keys, 16 at a time, out of a ring of its own in shared memory that
// one lane fills three steps ahead by TMA (24 KB per warp, two CTAs of four warps per SM; keys are asked for again as soon as the scores are formed; heads of 64 / 64: four CTAs, by
// cp.async), and never waits for another warp:
//   S^T = K Q^T   mma.sync m16n8k16, keys on the M axis, the R <= 8 query heads of the key head on the N axis
//   softmax       fp32 in registers, a running (maximum, denominator) per warp; cap, bias, temperature and masks as in the row kernel
//   O^T = V^T P^T value dimensions on the M axis (ldmatrix.trans). The weights keep 24 bits: p = hi + mid + lo (three bfloat16, the
//                 difference exact at every step), three products with fp32 accumulation, so nothing is rounded to 16 bits on the way.
//                 movmatrix turns the weights' fragments. A step's products have sums of their own, added in fp32: left to the tensor core, which cuts off
//                 instead of rounding, fp32 outputs were off by 3.3e-7 over four shares of 1500 keys and 8.5e-7 over one; now 1.9e-7 whatever the shares, in the same time.
// Warps merge through shared memory, CTAs through distributed shared memory (rank order, so the sum does not depend on timing). The merge
// adds the sink.
// Measured (before: the group kernel of capped_attention.cu with a combine launch): one sequence of 500 tokens, 8 / 4 heads x 128: 20.5 -> 6.6 us;
// 32 sequences of up to 2048 tokens, 16 / 8 heads x 128 (190 MB), bias and sink: 384 -> 48 us. With the rows brought by cp.async (16 instructions and their addresses per lane and step) and a lookup of the bias for
// keys beyond its table those were 6.9 and 59 us, 8 sequences of up to 2048 17.6 / 14.2, 12 of up to 1500, capped, 24.0 / 17.1. Two stages per warp and three CTAs per SM: slower (8 of 2048 18.4:
// clusters are laid onto as few SMs as hold them).
#include <cooperative_groups.h>
#include <cuda_bf16.h>

#include <algorithm>

#include "b200_serve.h"
#include "common.cuh"
#include "launch_count.h"
#include "paged_attention.cuh"
#include "tc_common.cuh"

namespace b200 {
namespace cg = cooperative_groups;

constexpr int kPdWarps = 4, kPdStep = 16, kPdHeads = 8, kPdMaxCluster = 8;

template <int D, int VD>
struct PdRing {   // a step's keys, then its values: boxes of 16 rows x 64 columns, swizzled over 128 bytes as TMA does
    static constexpr int kStages = VD > 128 ? 2 : 3, kBox = kPdStep * 128;
    static constexpr int kK = D / 64 * kBox, kStep = kK + VD / 64 * kBox, kWarp = kStages * kStep;
    static constexpr int kBytes = kPdWarps * kWarp + 1024;
    static constexpr int kPerSm = D + VD <= 128 ? 4 : 2;
    // Heads of 64 / 64 leave room for four CTAs per SM. With more than two there, boxes by TMA come at less than half the rate of copies by cp.async (16 query / 8 key heads, us by
    // TMA / by cp.async: 22 sequences of up to 2000 keys 38 / 20.6, 40 53 / 34, 64 76 / 42, two shares each; at one share with 100 KB of shared memory, so that two fit, 40 take 46), so those keep cp.async
    static constexpr bool kTma = D + VD > 128;
};

__device__ __forceinline__ uint32_t pd_transpose(uint32_t v) {   // 8 x 8 tile of 16-bit numbers, a pair per thread
    uint32_t r;
    asm("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(r) : "r"(v));
    return r;
}

__device__ __forceinline__ void pd_ldsm_x4(uint32_t (&r)[4], uint32_t a) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a) : "memory");
}
__device__ __forceinline__ void pd_ldsm_x4_trans(uint32_t (&r)[4], uint32_t a) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a) : "memory");
}

// MIXED: a batch that also holds prompt portions, which other kernels take. Cluster z looks after the tokens z, z + gridDim.z, ... and serves
// those that are their sequence's only token in the batch.
template <int D, int VD, bool MIXED>
__global__ void __launch_bounds__(kPdWarps * 32, PdRing<D, VD>::kPerSm)
paged_decode_kernel(const __grid_constant__ CUtensorMap map_k, const __grid_constant__ CUtensorMap map_v, const PA a) {
    using bf = __nv_bfloat16;
    using L = PdRing<D, VD>;
    constexpr int KS = D / 16;        // k steps of the scores
    constexpr int MT = VD / 16;       // m tiles of the output
    constexpr int NS = L::kStages;
    extern __shared__ __align__(1024) unsigned char pd_raw[];
    unsigned char* pd_sm = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(pd_raw) + 1023) & ~(uintptr_t)1023);
    __shared__ uint64_t pd_bars[kPdWarps * 2 * NS];
    __shared__ int pd_dead;
    volatile int* dead = &pd_dead;
    const int warp = __shfl_sync(0xffffffffu, threadIdx.x / 32, 0), lane = threadIdx.x % 32, gid = lane >> 2, tig = lane & 3;
    uint64_t *k_full = pd_bars + warp * 2 * NS, *v_full = k_full + NS;   // of this warp's ring
    if (L::kTma) {
        if (lane == 0) {
#pragma unroll
            for (int i = 0; i < 2 * NS; ++i) mbar_init(&k_full[i], 1);
            mbar_fence_init();
            if (warp == 0) { *dead = 0; tma_prefetch_desc(&map_k); tma_prefetch_desc(&map_v); }
        }
        __syncthreads();
    }
    // A mixed batch's clusters run beside its tiles, whose kernel triggers behind its own pdl_wait(), in every thread: what came before both has ended and been written back when these start, and
    // they read nothing that the tiles write. One of their CTAs waits for the tiles before it ends (below). A wait here would put them behind the tiles, a fence in its place takes up
    // to 4 %, loads past the first-level cache up to 10 %.
    if (!MIXED) pdl_wait();
    pdl_launch_dependents();   // (what follows waits for this kernel, and so for the tiles)
    const int R = a.heads / a.kv_heads, splits = gridDim.x;
    float* om = reinterpret_cast<float*>(pd_sm);                                 // once the rings have been used: [warps][R][VD], then this CTA's share in the first [R][VD]
    __shared__ float ms[kPdWarps * kPdHeads], ls[kPdWarps * kPdHeads];   // [warps][R], then [R]
    const int ku = blockIdx.y, g = ku / a.maps, mp = ku % a.maps;
    const int q_units = a.heads * a.maps;
    const uint32_t ring = smem_u32(pd_sm) + (uint32_t)(warp * L::kWarp);
    // where this lane's rows of the matrix loads lie in a stage: keys row lane & 15, piece lane >> 4; values (transposed) row (lane & 7) + 8 (lane >> 4), piece
    // (lane >> 3) & 1; two pieces per 16 columns, swizzled by the row
    uint32_t k_at[4], v_at[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        k_at[i] = ring + (uint32_t)((lane & 15) * 128 + (((2 * i + (lane >> 4)) ^ (lane & 7)) << 4));
        v_at[i] = ring + (uint32_t)(L::kK + ((lane & 7) + (lane >> 4) * 8) * 128 + (((2 * i + ((lane >> 3) & 1)) ^ (lane & 7)) << 4));
    }
    uint32_t stage = 0, parity = 0;   // of the step that is worked on
    // by cp.async: this lane brings 16 bytes of rows lane / 8, lane / 8 + 4, ... of a step
    auto copy_rows = [&](uint32_t to, const void* pool, size_t row, size_t row_width, int column) {
        const int c = lane & 7;
        const bf* from = reinterpret_cast<const bf*>(pool) + row * row_width + column + c * 8;
#pragma unroll
        for (int i = 0; i < kPdStep / 4; ++i) {
            const int r = 4 * i + (lane >> 3);
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(to + (uint32_t)(r * 128 + ((c ^ (r & 7)) << 4))), "l"(from + r * row_width) : "memory");
        }
    };
    auto close_group = [&]() {
        __syncwarp();   // the lanes close their group of copies together
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    // this thread's two heads (columns of S^T and O^T)
    float sc[2], hb[2];
    const float over_cap = a.softcap > 0.f ? 1.f / a.softcap : 0.f;
    const float* bias[2];
    float far[2];
#pragma unroll
    for (int x = 0; x < 2; ++x) {
        const int h = min(g * R + 2 * tig + x, a.heads - 1);
        sc[x] = pa_scale(a, h);
        hb[x] = (a.sigmoid && a.head_bias) ? a.head_bias[h] : 0.f;
        bias[x] = a.dist_bias ? a.dist_bias + (size_t)h * a.dist_n : nullptr;
        far[x] = a.dist_bias ? bias[x][a.dist_n - 1] : 0.f;
    }
    for (int base = blockIdx.z; base < a.n_tokens; base += 32 * gridDim.z) {
        uint32_t todo = 1u;
        if (MIXED) {
            const long long c = base + (long long)lane * gridDim.z;
            const bool in = c < a.n_tokens;
            const int sl = in ? a.slot[c] : -1;
            todo = __ballot_sync(0xffffffffu, in && (c == 0 || a.slot[c - 1] != sl) && (c + 1 >= a.n_tokens || a.slot[c + 1] != sl));
        }
        for (; todo; todo &= todo - 1) {
            const int t = MIXED ? base + (__ffs(todo) - 1) * (int)gridDim.z : base;
            uint32_t qf[KS][2];               // query head gid (heads beyond the group: zeros)
#pragma unroll
            for (int ks = 0; ks < KS; ++ks) {
                const bf* q = reinterpret_cast<const bf*>(a.q) + ((size_t)t * q_units + (g * R + min(gid, R - 1)) * a.maps + mp) * D + ks * 16 + tig * 2;
                qf[ks][0] = gid < R ? *reinterpret_cast<const uint32_t*>(q) : 0u;
                qf[ks][1] = gid < R ? *reinterpret_cast<const uint32_t*>(q + 8) : 0u;
            }
            const int p = a.pos[t];
            const int* plist = a.pages + (size_t)a.slot[t] * a.max_pages;
            float m[2], l[2] = {0.f, 0.f}, o[MT][4];
            m[0] = m[1] = a.sigmoid ? 0.f : -INFINITY;
#pragma unroll
            for (int j = 0; j < MT; ++j) o[j][0] = o[j][1] = o[j][2] = o[j][3] = 0.f;

            // this warp's run of 16-key steps; a step lies inside one page (page_rows is a multiple of 16)
            const int j_lo = pa_first_key(a, p), first = j_lo & ~(kPdStep - 1), steps = (p - first) / kPdStep + 1;
            const int per = (steps + splits * kPdWarps - 1) / (splits * kPdWarps), w = blockIdx.x * kPdWarps + warp;
            const int s0 = w * per, s1 = min(steps, s0 + per);
            int j0 = first + s0 * kPdStep;
            int page_at = j0 / a.page_rows, off = j0 - page_at * a.page_rows;    // of the step that is fetched next
            int page = s0 < s1 ? plist[page_at] : 0;
            int row = 0;   // pool row of the step whose keys were asked for last
            auto fetch_k = [&](uint32_t st) {   // the keys of the next step into stage st (rows that the token does not see may hold anything)
                row = page * a.page_rows + off;
                if (!L::kTma) {
                    copy_rows(ring + st * L::kStep, a.k_pool, row, (size_t)a.kv_heads * a.maps * D, ku * D);
                } else if (lane == 0) {
                    mbar_expect_tx(&k_full[st], L::kK);
#pragma unroll
                    for (int c = 0; c < D / 64; ++c) tma_load_2d(pd_sm + warp * L::kWarp + st * L::kStep + c * L::kBox, &map_k, ku * D + c * 64, row, &k_full[st]);
                }
                __syncwarp();
            };
            auto fetch_v = [&](uint32_t st, int s) {   // and its values; the page of the step after is looked up
                if (!L::kTma) {
                    copy_rows(ring + st * L::kStep + L::kK, a.v_pool, row, (size_t)a.kv_heads * VD, g * VD);
                } else if (lane == 0) {
                    mbar_expect_tx(&v_full[st], L::kStep - L::kK);
#pragma unroll
                    for (int c = 0; c < VD / 64; ++c) tma_load_2d(pd_sm + warp * L::kWarp + st * L::kStep + L::kK + c * L::kBox, &map_v, g * VD + c * 64, row, &v_full[st]);
                }
                __syncwarp();
                off += kPdStep;
                if (off == a.page_rows) { off = 0; ++page_at; if (s + 1 < s1) page = plist[page_at]; }
            };
            {
                uint32_t st = stage;
#pragma unroll
                for (int i = 0; i < NS; ++i) {
                    if (s0 + i < s1) fetch_k(st);
                    if (!L::kTma) close_group();
                    if (s0 + i < s1) fetch_v(st, s0 + i);
                    if (!L::kTma) close_group();
                    st = st + 1 == NS ? 0 : st + 1;
                }
            }
            auto arrived = [&](uint64_t* bar) {   // by cp.async: a group of keys and one of values per step, the rest of the ring behind them
                if (L::kTma) mbar_wait_or_leave(bar, parity, dead);
                else {
                    asm volatile("cp.async.wait_group %0;" ::"n"(2 * NS - 1) : "memory");
                    __syncwarp();   // for every lane
                }
            };
            for (int s = s0; s < s1; ++s, j0 += kPdStep) {
                const bool whole = j0 >= j_lo && j0 + kPdStep - 1 <= p;
                const uint32_t at = stage * L::kStep;
                float bv[4] = {0.f, 0.f, 0.f, 0.f};
                if (a.dist_bias) {   // requested before the scores are formed; beyond the table the last number stands for all
                    if (p - (j0 + kPdStep - 1) >= a.dist_n - 1) {
#pragma unroll
                        for (int e = 0; e < 4; ++e) bv[e] = far[e & 1];
                    } else {
#pragma unroll
                        for (int e = 0; e < 4; ++e) bv[e] = bias[e & 1][min(max(p - (j0 + gid + (e >> 1) * 8), 0), a.dist_n - 1)];
                    }
                }
                arrived(&k_full[stage]);
                float st[4] = {0.f, 0.f, 0.f, 0.f}, su[4] = {0.f, 0.f, 0.f, 0.f};   // two chains of products
#pragma unroll
                for (int ks = 0; ks < KS; ks += 2) {
                    uint32_t k0[4], k1[4];
                    pd_ldsm_x4(k0, k_at[ks & 3] + at + (uint32_t)((ks >> 2) * L::kBox));
                    pd_ldsm_x4(k1, k_at[(ks + 1) & 3] + at + (uint32_t)((ks >> 2) * L::kBox));
                    pa_mma(st, k0, qf[ks]);
                    pa_mma(su, k1, qf[ks + 1]);
                }
#pragma unroll
                for (int e = 0; e < 4; ++e) st[e] = (st[e] + su[e]) * sc[e & 1];
                __syncwarp();   // every lane has read the keys: their place may be filled again
                if (s + NS < s1) fetch_k(stage);
                if (!L::kTma) close_group();
                bool seen[4] = {true, true, true, true};   // key j0 + gid (+ 8), head 2 tig (+ 1)
                if (!whole) {
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const int j = j0 + gid + (e >> 1) * 8;
                        seen[e] = j >= j_lo && j <= p;
                        if (!seen[e]) st[e] = 0.f;   // (of a key that may be anything)
                    }
                }
                if (a.softcap > 0.f) {
                    // cap * tanh(v / cap): the odd series up to x^7 while every |x| is below 0.2 (its next term is below 2^-24 of x there)
                    float x[4], big = 0.f;
#pragma unroll
                    for (int e = 0; e < 4; ++e) { x[e] = st[e] * over_cap; big = fmaxf(big, fabsf(x[e])); }
                    if (__all_sync(0xffffffffu, big < 0.2f)) {
#pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            const float x2 = x[e] * x[e];
                            st[e] = a.softcap * x[e] * fmaf(x2, fmaf(x2, fmaf(x2, -17.f / 315.f, 2.f / 15.f), -1.f / 3.f), 1.f);
                        }
                    } else {
#pragma unroll
                        for (int e = 0; e < 4; ++e) st[e] = a.softcap * tanhf(x[e]);
                    }
                }
                float pr[4];
#pragma unroll
                for (int e = 0; e < 4; ++e) pr[e] = seen[e] ? st[e] + bv[e] : -INFINITY;
                if (a.sigmoid) {
#pragma unroll
                    for (int e = 0; e < 4; ++e) pr[e] = pr[e] == -INFINITY ? 0.f : 1.f / (1.f + expf(-(pr[e] + hb[e & 1])));
                } else {
                    // the exponents' reference moves only when a score has passed it by 8 ln 2 (weights up to 256; the division at the end makes
                    // them exact again): seldom after the first step, and no reduction over the keys until then
                    const float top[2] = {fmaxf(pr[0], pr[2]), fmaxf(pr[1], pr[3])};
                    if (__any_sync(0xffffffffu, top[0] > m[0] + 5.545f || top[1] > m[1] + 5.545f)) {
                        float alpha[2];
#pragma unroll
                        for (int x = 0; x < 2; ++x) {
                            float mx = fmaxf(top[x], __shfl_xor_sync(0xffffffffu, top[x], 4));
                            mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 8));
                            mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 16));
                            const float mn = fmaxf(m[x], mx);
                            alpha[x] = m[x] == mn ? 1.f : expf(m[x] - mn);
                            m[x] = mn;
                            l[x] *= alpha[x];
                        }
#pragma unroll
                        for (int j = 0; j < MT; ++j) { o[j][0] *= alpha[0]; o[j][1] *= alpha[1]; o[j][2] *= alpha[0]; o[j][3] *= alpha[1]; }
                    }
#pragma unroll
                    for (int e = 0; e < 4; ++e) pr[e] = pr[e] == -INFINITY ? 0.f : expf(pr[e] - m[e & 1]);
                    l[0] += pr[0] + pr[2];
                    l[1] += pr[1] + pr[3];
                }
                uint32_t b[3][2];   // hi, mid, lo: p = hi + mid + lo to 24 bits
#pragma unroll
                for (int q = 0; q < 3; ++q)
#pragma unroll
                    for (int hf = 0; hf < 2; ++hf) {
                        const __nv_bfloat162 h2 = __floats2bfloat162_rn(pr[2 * hf], pr[2 * hf + 1]);
                        const float2 f = __bfloat1622float2(h2);
                        pr[2 * hf] -= f.x;
                        pr[2 * hf + 1] -= f.y;
                        b[q][hf] = pd_transpose(*reinterpret_cast<const uint32_t*>(&h2));
                    }
                arrived(&v_full[stage]);
                if (!whole) {   // values of keys that the token does not see: 0 * NaN must stay 0
                    for (int i = lane; i < kPdStep * (VD / 8); i += 32) {
                        const int r = i / (VD / 8), c = i % (VD / 8);
                        if (j0 + r < j_lo || j0 + r > p) st_shared_v4(ring + at + (uint32_t)(L::kK + (c / 8) * L::kBox + r * 128 + (c & 7) * 16), 0u, 0u, 0u, 0u);
                    }
                    if (L::kTma) fence_proxy_async_smem();
                    __syncwarp();
                }
#pragma unroll
                for (int j = 0; j < MT; j += 4) {   // four tiles of 16 dimensions at a time: consecutive products feed different sums
                    uint32_t af[4][4];
                    float t4[4][4] = {};   // the step's own sums: the tensor core cuts its sums off, so a chain of many steps there would lose by its length
#pragma unroll
                    for (int e = 0; e < 4; ++e) pd_ldsm_x4_trans(af[e], v_at[e] + at + (uint32_t)((j >> 2) * L::kBox));
#pragma unroll
                    for (int q = 2; q >= 0; --q)
#pragma unroll
                        for (int e = 0; e < 4; ++e) pa_mma(t4[e], af[e], b[q]);
#pragma unroll
                    for (int e = 0; e < 4; ++e)
#pragma unroll
                        for (int x = 0; x < 4; ++x) o[j + e][x] += t4[e][x];
                }
                __syncwarp();   // and the values
                if (s + NS < s1) fetch_v(stage, s + NS);
                if (!L::kTma) close_group();
                if (++stage == NS) { stage = 0; parity ^= 1u; }
            }
            if (!L::kTma) asm volatile("cp.async.wait_group 0;" ::: "memory");
            const bool gave_up = L::kTma && *dead != 0;
            if (gave_up) linger();   // nothing may land behind this CTA's end, or on the sums
            __syncthreads();    // the rings' place is taken by the sums
#pragma unroll
            for (int x = 0; x < 2; ++x) {
                l[x] += __shfl_xor_sync(0xffffffffu, l[x], 4);
                l[x] += __shfl_xor_sync(0xffffffffu, l[x], 8);
                l[x] += __shfl_xor_sync(0xffffffffu, l[x], 16);
                const int h = 2 * tig + x;
                if (h < R) {
                    if (gid == 0) { ms[warp * R + h] = gave_up ? 0.f : m[x]; ls[warp * R + h] = gave_up ? __int_as_float(0x7fffffff) : l[x]; }   // (NaN at a finite reference: every merge takes it in)
                    float* dst = om + (size_t)(warp * R + h) * VD + gid;
#pragma unroll
                    for (int j = 0; j < MT; ++j) {
                        dst[j * 16] = o[j][x];
                        dst[j * 16 + 8] = o[j][2 + x];
                    }
                }
            }
            __syncthreads();
            // the CTA's share: every output is added by one thread, which alone reads and writes its places
            for (int i = threadIdx.x; i < R * VD; i += blockDim.x) {
                const int h = i / VD;
                float M = ms[h];
#pragma unroll
                for (int v = 1; v < kPdWarps; ++v) M = fmaxf(M, ms[v * R + h]);
                float acc = 0.f;
#pragma unroll
                for (int v = 0; v < kPdWarps; ++v) {
                    const float mv = ms[v * R + h];
                    if (mv != -INFINITY) acc += om[(size_t)(v * R + h) * VD + i % VD] * expf(mv - M);
                }
                om[i] = acc;
            }
            __syncthreads();
            float cm = 0.f, cl = 0.f;
            if (threadIdx.x < R) {
                cm = ms[threadIdx.x];
                for (int v = 1; v < kPdWarps; ++v) cm = fmaxf(cm, ms[v * R + threadIdx.x]);
                for (int v = 0; v < kPdWarps; ++v) {
                    const float mv = ms[v * R + threadIdx.x];
                    if (mv != -INFINITY) cl += ls[v * R + threadIdx.x] * expf(mv - cm);
                }
            }
            __syncthreads();
            if (threadIdx.x < R) { ms[threadIdx.x] = cm; ls[threadIdx.x] = cl; }
            cg::cluster_group cluster = cg::this_cluster();
            cluster.sync();
            const int total = R * VD, share = (total + splits - 1) / splits;
            for (int i = blockIdx.x * share + threadIdx.x; i < min(total, ((int)blockIdx.x + 1) * share); i += blockDim.x) {
                const int h = i / VD, qh = g * R + h;
                // the sink joins here: a score without key and value
                float M = a.sigmoid ? 0.f : a.sink ? a.sink[qh] : a.denom_bias > 0.f ? 0.f : -INFINITY;
                const float sink_at = M, sink_l = a.sigmoid || a.sink ? 1.f : a.denom_bias;
                float mr[kPdMaxCluster];
#pragma unroll
                for (int r = 0; r < kPdMaxCluster; ++r)
                    if (r < splits) { mr[r] = cluster.map_shared_rank(ms, r)[h]; M = fmaxf(M, mr[r]); }
                float L = sink_at == -INFINITY ? 0.f : sink_l * expf(sink_at - M), acc = 0.f;
#pragma unroll
                for (int r = 0; r < kPdMaxCluster; ++r)
                    if (r < splits && mr[r] != -INFINITY) {
                        const float f = expf(mr[r] - M);
                        L += cluster.map_shared_rank(ls, r)[h] * f;
                        acc += cluster.map_shared_rank(om, r)[i] * f;
                    }
                pa_store<bf>(a, ((size_t)t * q_units + (size_t)qh * a.maps + mp) * VD + i % VD, acc / L);
            }
            if (L::kTma) fence_proxy_async_smem();   // TMA writes where the sums lay
            cluster.sync();   // nobody leaves (or starts its next token) while its shared memory is read
        }
        if (!MIXED) break;
    }
    // the prompt portions' kernel runs beside this one: done only when both are. One CTA to wait is enough: clusters without a token, which are most of them,
    // make room for those behind them (us with all of them waiting / with one, 8 / 4 heads x 128 and blocks of 1024: two portions
    // of up to 66 behind up to 3319 and 6 single tokens 20.4 / 12.3; 16 / 8: three of up to 40 alone 8.5 / 8.1, one of 512 behind 4000 and 8 single tokens 75 / 56)
    if (MIXED && blockIdx.x == 0 && blockIdx.y == 0 && blockIdx.z == 0) pdl_wait();
}

template <int D, int VD, bool MIXED>
static int launch_paged_decode(const PA& a, int splits, int rows, cudaStream_t s) {
    constexpr int smem = PdRing<D, VD>::kBytes;
    static_assert(kPdWarps * kPdHeads * VD * 4 <= smem, "the warps' sums take the rings' place");
    CUtensorMap mk{}, mv{};
    constexpr long long kAnyRow = (1ll << 31) - 1;   // the pool's height is not part of the call: any row that an int can name
    if (PdRing<D, VD>::kTma && (!make_tma_map_2d(&mk, a.k_pool, kAnyRow, a.kv_heads * a.maps * D, kPdStep) || !make_tma_map_2d(&mv, a.v_pool, kAnyRow, a.kv_heads * VD, kPdStep))) return -1;
    static unsigned long long done = 0;
    cudaError_t e = ensure_max_dynamic_smem((const void*)paged_decode_kernel<D, VD, MIXED>, smem, done);
    if (e != cudaSuccess) return (int)e;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)splits, (unsigned)(a.kv_heads * a.maps), (unsigned)rows);
    cfg.blockDim = dim3(kPdWarps * 32);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = (unsigned)splits;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    if (pdl_enabled()) {
        at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        at[1].val.programmaticStreamSerializationAllowed = 1;
        cfg.numAttrs = 2;
    }
    e = cudaLaunchKernelEx(&cfg, paged_decode_kernel<D, VD, MIXED>, mk, mv, a);
    if (e != cudaSuccess) return (int)e;
    count_launch();
    return (int)cudaGetLastError();
}

template <bool MIXED>
static int paged_decode_for(const PA& a, int splits, int rows, cudaStream_t s) {
    if (a.dim == 128 && a.vdim == 128) return launch_paged_decode<128, 128, MIXED>(a, splits, rows, s);
    if (a.dim == 64 && a.vdim == 64) return launch_paged_decode<64, 64, MIXED>(a, splits, rows, s);
    if (a.dim == 128 && a.vdim == 256) return launch_paged_decode<128, 256, MIXED>(a, splits, rows, s);
    if (a.dim == 64 && a.vdim == 128) return launch_paged_decode<64, 128, MIXED>(a, splits, rows, s);
    return -1;
}

int paged_decode(const PA& a, int longest_seen, int singles, long long room, cudaStream_t s) {
    const bool mixed = singles > 0;
    if (a.heads / a.kv_heads > kPdHeads || a.page_rows % kPdStep || a.kv_heads * a.maps > 65535) return -1;
    // how many tokens of a mixed batch are single ones is only known on the device: sixteen rows of clusters share them
    const int rows = mixed ? std::min(singles, 16) : a.n_tokens;
    if (rows > 65535) return -1;
    // as many shares as the two CTAs per SM that fit hold at once, as long as every warp of a cluster keeps a step of its own (16 / 8 heads x 128, us at 1 / 2 / 4 / 8
    // shares: 32 sequences of up to 2048 tokens 42.5 / 44.5 / 52.7 / 78.0, 16 such 35.0 / 24.4 / 28.2 / 40.9, 12 of up to 1500 27.4 / 17.1 / 20.4 / 25.4, 8 of up to 2048
    // 34.4 / 20.0 / 14.3 / 19.8, 4 such 34.3 / 19.8 / 13.5 / 10.8)
    const long long pairs = (long long)rows * a.kv_heads * a.maps;
    const int sms = sm_count();
    int splits = 1;
    if (mixed) {
        // on what the portions' CTAs leave free (`room` CTAs) if eight single tokens can sit there beside each other, else behind them (us at 2 / 4 / 8 shares: 8 single tokens and a portion of 512 behind
        // 4000 56.7 / 60.4 / 70.4, 4 and 64 35.9 / 23.8 / 23.9, 12 and three of 512, which fill the GPU, capped, 105 / 106 / 119, 1 and three 90.3 / 83.3 / 83.1, 3 and three behind 2200, biased, 64.1 / 62.2 / 63.7)
        const long long likely = (long long)std::min(singles, 8) * a.kv_heads * a.maps;
        // (values of 256 columns, 16 / 8 heads, us at 2 / 4: 8 single tokens and three of 512 behind 300 31.8 / 36.0, behind 1800 69.8 / 73.0, 12 and two of 500 behind 1500, two maps, 87.0 / 96.1)
        if (room < likely) room = (a.vdim > 128 ? 2 : 4) * likely;
        splits = 2;
        while (splits < (likely <= 8 ? kPdMaxCluster : 4) && likely * splits * 2 <= room) splits *= 2;
        while (splits > 1 && longest_seen > 0 && splits / 2 * kPdWarps * kPdStep >= longest_seen) splits /= 2;
    } else {
        // heads of 64 / 64, four CTAs per SM: three CTAs for every two SMs (us at 1 / 2 / 4 / 8 shares: 8 sequences of up to 2000 keys 25.3 / 15.1 / 11.7 / 10.6, 12 25.3 / 16.6 / 13.7 / 17.6,
        // 19 28.1 / 19.8 / 20.7 / 25.3, 28 28.5 / 21.5 / 24.3 / 33.4, 40 38.3 / 34.3 / 35.8 / 46.5, 64 43.2 / 42.0 / 49.1 / 69.4; all of 2000: 40 40.7 / 47.1 / 43.2 / 52.2)
        const bool narrow = a.dim == 64 && a.vdim == 64;
        auto room_for_twice = [&] { return narrow ? 2 * pairs * splits < 3ll * sms : pairs * splits <= sms; };
        while (splits < kPdMaxCluster && room_for_twice() && (longest_seen <= 0 || splits * kPdWarps * kPdStep < longest_seen)) splits *= 2;
        // just beyond one CTA per SM one share leaves nearly half of the places empty: long contexts in three, a round and a half (16 heads x 128, up to 2000 keys, us at 1 / 2 / 3 shares: 38 sequences and
        // 4 key heads 37.9 / 29.2 / 33.2, 19 and 8 37.6 / 34.1 / 32.7, 22 37.2 / 35.7 / 34.0, 10 and 16 36.5 / 31.5 / 30.4; all of 2000 39.8 / 47.1 / 40.9, 39.0 / 43.9 / 39.1, 40.4 / 48.6 / 41.2, 38.4 / 44.6 / 38.8;
        // 23 and 8 36.6 / 35.7 / 34.4, all of 2000 39.5 / 49.3 / 42.5; all of 1200 26.4 / 28.5 / 26.3 at 19, 27.0 / 32.8 / 29.6 at 22)
        if (!narrow && splits == 1 && pairs > sms && 4 * pairs <= 5 * sms && longest_seen > 1000) splits = 3;
    }
    return mixed ? paged_decode_for<true>(a, splits, rows, s) : paged_decode_for<false>(a, splits, rows, s);
}

}  // namespace b200
