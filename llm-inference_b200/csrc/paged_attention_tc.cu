// bfloat16 prompt portions of b200_paged_attention on tcgen05 / TMEM: 128 (token, query head) rows per tile, keys 64 at a time.
//
// What bounds it: per 128 x 64 scores of 128-wide heads the tensor pipe needs 512 clocks and more (the scores are 64 columns wide, so their
// operands count) and the special-function unit 512 for the exponentials; one tile alone is a chain of both, so two CTAs share an
// SM (96 KB of shared memory and 256 TMEM columns each) and fill each other's gaps. A step of 64 keys takes about 1200 clocks with two
// CTAs on an SM; the longest row tile of a prompt and what comes before its first and after its last step decide.
// Measured (before: the mma.sync tiles of paged_attention_tile.cuh), 16 / 8 heads x 128, 2048 tokens: 114 -> 36 us (32 with
// weights rounded to bfloat16 alone). Tried and taken back: 128 keys
// per tile with one score buffer (52 us: products and softmax take turns), two threads per row (43 us), the keys of a tile shared by a
// cluster of two (41 us: the fixed part of a CTA counts more than the chain).
//   rows        TQ tokens x the R query heads of one key head (TQ = 128 / R), so a key tile is read once for the whole group and a
//               causal edge wastes little. A CTA's window of TQ packed rows may hold the end of one sequence and the start of
//               the next: they are separate tiles, walked by neighbouring CTAs (gridDim.y is doubled when there is more than one entry).
//               Sequences that bring a single token are left to the cluster kernel of paged_decode.cu.
//   warp 0      TMA: K and V tiles of 64 rows out of their page (one list lookup per tile), two stages each
//   warp 1      tcgen05.mma: S_{j+1} = Q K^T is issued before O += P_j V_j, so the tensor pipe works under the softmax
//   warps 2-5   softmax, a thread per row: scores are read from TMEM once, P_j goes back over its own scores and is the A operand of the second
//               product. O stays in TMEM: it is rescaled only when a row's maximum has grown by more than 2^8 since the last rescaling
//               (weights up to 256, sums in fp32). A row's largest weight is then any number instead of 1, so a weight rounded to
//               bfloat16 alone would cost more precision than against the running maximum (2.07e-3 of the result's norm, 2.03e-3
//               there): P_j is the sum of two bfloat16, hi + lo, in the 64 columns of its scores, and both are multiplied (1.61e-3, the
//               rounding of the outputs).
// Rows of a page beyond the context, or ahead of what a window or a block mask leaves, may hold anything, so those V rows are cleared in the
// last and the first tile before they are multiplied by zero weights.
#include <cuda_bf16.h>

#include "b200_serve.h"
#include "common.cuh"
#include "launch_count.h"
#include "paged_attention.cuh"
#include "tc_common.cuh"

namespace b200 {
enum { kTcPlain = 0, kTcCapped = 1, kTcBiased = 2, kTcSigmoid = 3 };
constexpr int kTcRows = 128, kTcKeys = 64, kTcThreads = 192;
constexpr int kTcBox = kTcKeys * 128;         // bytes of 64 rows x 64 columns
constexpr int kTcBiasFront = kTcKeys, kTcBiasPad = kTcBiasFront + 2 * kTcRows;   // distances in front of, and around, a head's staged table
constexpr int kTcBiasFloats = 12288;          // at most this many staged bias numbers per CTA (from about 3500 on one CTA per SM)

template <int D, int DV>
struct TcSmem {
    static constexpr int kQ = kTcRows * D * 2, kK = kTcKeys * D * 2, kV = kTcKeys * DV * 2;
    static constexpr int kOffK = kQ, kOffV = kOffK + 2 * kK, kOffBar = kOffV + 2 * kV, kOffSlot = kOffBar + 16 * 8;
    static constexpr int kOffBias = kOffSlot + (kTcRows + 2 + 16) * 4;
    static constexpr int kTmemCols = 2 * kTcKeys + DV <= 256 ? 256 : 512;
};

template <int D, int DV, int FORM>
__global__ void __launch_bounds__(kTcThreads, TcSmem<D, DV>::kTmemCols == 256 ? 2 : 1)
paged_attn_tc_kernel(const __grid_constant__ CUtensorMap map_k, const __grid_constant__ CUtensorMap map_v, const PA a, int TQ, int parts, int skip_singles) {
    using bf = __nv_bfloat16;
    using L = TcSmem<D, DV>;
    extern __shared__ __align__(1024) unsigned char tc_raw[];
    unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(tc_raw) + 1023) & ~(uintptr_t)1023);
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::kOffBar);
    uint64_t *k_full = bars, *k_empty = bars + 2, *v_full = bars + 4, *v_empty = bars + 6, *s_full = bars + 8, *p_full = bars + 10, *o_done = bars + 12;
    int* slots = reinterpret_cast<int*>(smem + L::kOffSlot);        // of the window's rows and one on either side
    uint32_t* masks = reinterpret_cast<uint32_t*>(slots + kTcRows + 2);   // [0..3] rows that begin a sequence, [4..7] those that begin a tile
    uint32_t* tmem_slot = masks + 8;
    volatile int* dead = reinterpret_cast<volatile int*>(masks + 9);
    float* bias_s = reinterpret_cast<float*>(smem + L::kOffBias);

    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;   // (uniform as the compiler sees it)
    const int ku = blockIdx.x, g = ku / a.maps, mp = ku % a.maps, R = a.heads / a.kv_heads, q_units = a.heads * a.maps;
    // the last rows of a prompt see the most keys: those windows come first
    const int yy = gridDim.y - 1 - blockIdx.y, part = yy % parts, t0 = yy / parts * TQ, rows = min(TQ, a.n_tokens - t0);

    // ---- TMEM, barriers, and the window's tiles
    if (warp == 1) tmem_alloc(tmem_slot, L::kTmemCols);
    if (threadIdx.x == 0) {
#pragma unroll
        for (int s = 0; s < 2; ++s) {
            mbar_init(&k_full[s], 1); mbar_init(&k_empty[s], 1);
            mbar_init(&v_full[s], 1); mbar_init(&v_empty[s], 1);
            mbar_init(&s_full[s], 1); mbar_init(&p_full[s], 4);
            mbar_init(&o_done[s], 1);
        }
        mbar_fence_init();
        tma_prefetch_desc(&map_k);
        tma_prefetch_desc(&map_v);
        *dead = 0;
    }
    for (int i = (int)threadIdx.x - 64; i >= 0 && i < TQ + 2; i += kTcThreads - 64) {
        const int t = t0 - 1 + i;
        slots[i] = t >= 0 && t < a.n_tokens ? a.slot[t] : -1;
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    // the kernel for single tokens may move in (it waits for this one before it ends); TMEM has been allocated: a product kernel that moved in ahead of
    // that would wait for this one while holding it
    pdl_launch_dependents();
    if (warp < 4) {
        const int i = threadIdx.x;   // row of the window; slots[i + 1] is its own
        const bool in = i < rows, starts = in && (i == 0 || slots[i] != slots[i + 1]);
        const bool single = in && skip_singles && slots[i] != slots[i + 1] && slots[i + 2] != slots[i + 1];
        const uint32_t b = __ballot_sync(0xffffffffu, starts), tb = __ballot_sync(0xffffffffu, starts && !single);
        if (lane == 0) { masks[warp] = b; masks[4 + warp] = tb; }
    }
    int tn = 0;   // staged distances per head: those that a row of the window can have
    if (FORM == kTcBiased && a.dist_bias) {
        // per head: entry kTcBiasFront + distance; distances below 0 (masked keys) and beyond the table repeat its ends, so that no index needs a clamp
        for (int i = lane; i < rows; i += 32) tn = max(tn, a.pos[t0 + i] + 1);
        tn = min(__reduce_max_sync(0xffffffffu, tn), a.dist_n);
        for (int x = 0; x < R; ++x) {
            const float* src = a.dist_bias + (size_t)(g * R + x) * a.dist_n;
#pragma unroll 4
            for (int i = threadIdx.x; i < tn + kTcBiasPad; i += kTcThreads) bias_s[x * (tn + kTcBiasPad) + i] = src[min(max(i - kTcBiasFront, 0), tn - 1)] * 1.4426950408889634f;
        }
    }
    __syncthreads();
    const uint32_t tmem = __shfl_sync(0xffffffffu, *tmem_slot, 0), o_tmem = tmem + 2 * kTcKeys;

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
        // ---- warps 2-5: Q rows into the K-major swizzled operand (rows that this tile does not have: zeros), a thread's loads all in
        // flight together; K and V are on their way meanwhile
        if (warp >= 2) {
            constexpr int CH = D / 8, kPass = 128 / CH, kBatch = kTcRows / kPass;   // 16-byte pieces per row; rows per pass of the 128 threads
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
        const int pA = a.pos[tA], pZ = a.pos[tA + count - 1];
        const int fA = pa_first_key(a, pA), key0 = fA & ~(kTcKeys - 1), n_kt = (pZ - key0) / kTcKeys + 1;
        const int* plist = a.pages + (size_t)slots[first + 1] * a.max_pages;
        __syncwarp();   // lanes without a row skipped its loads; the barrier is warp-wide
        if (warp >= 1) asm volatile("bar.sync 1, 160;" ::: "memory");

        if (warp == 0) {
            // K of tile j + 1 goes ahead of V of tile j (which may have to wait for an older product), and a tile's place is looked up one tile
            // before it is needed
            auto row_of = [&](int j) {
                const int k0 = key0 + min(j, n_kt - 1) * kTcKeys;
                return plist[k0 / a.page_rows] * a.page_rows + k0 % a.page_rows;
            };
            auto load = [&](uint64_t* full, uint64_t* empty, int j, int row, const CUtensorMap* map, int x, unsigned char* base, int bytes, int boxes) {
                const int it = it0 + j, s = it & 1;
                mbar_wait_or_leave(&empty[s], ((uint32_t)(it >> 1) & 1u) ^ 1u, dead);
                if (lane == 0) {
                    mbar_expect_tx(&full[s], bytes);
                    for (int c = 0; c < boxes; ++c) tma_load_2d(base + s * bytes + c * kTcBox, map, x + c * 64, row, &full[s]);
                }
                __syncwarp();
            };
            int row = row_of(0), row1 = row_of(1), row2;
            load(k_full, k_empty, 0, row, &map_k, ku * D, smem + L::kOffK, L::kK, D / 64);
            for (int j = 0; j < n_kt; ++j, row = row1, row1 = row2) {
                row2 = row_of(j + 2);
                if (j + 1 < n_kt) load(k_full, k_empty, j + 1, row1, &map_k, ku * D, smem + L::kOffK, L::kK, D / 64);
                load(v_full, v_empty, j, row, &map_v, g * DV, smem + L::kOffV, L::kV, DV / 64);
            }
        } else if (warp == 1) {
            constexpr uint32_t kBf16 = (1u << 7) | (1u << 10);
            constexpr uint32_t idesc_s = make_idesc_f16(kTcRows, kTcKeys) | kBf16, idesc_o = make_idesc_f16(kTcRows, DV) | kBf16 | (1u << 16);
            // everything that an instruction takes is uniform over the warp and mostly constant: one lane issues twelve of them per tile, and the
            // softmax waits for the last
            const uint64_t q_desc = make_kmajor_sw128_desc(smem_u32(smem)), k_desc = make_kmajor_sw128_desc(smem_u32(smem + L::kOffK));
            const uint64_t v_desc = make_mnmajor_sw128_desc(smem_u32(smem + L::kOffV), kTcBox, 1024u);
            const int n = __shfl_sync(0xffffffffu, n_kt, 0);
            int it = __shfl_sync(0xffffffffu, it0, 0);
            const bool leader = elect_one();
            auto issue_s = [&](int i) {   // tile i (counted over all tiles of this CTA)
                const uint32_t s = (uint32_t)i & 1u;
                mbar_wait_or_leave(&k_full[s], (uint32_t)(i >> 1) & 1u, dead);
                tc_fence_after();
                if (leader) {
                    const uint64_t kd = k_desc + (uint64_t)(s * (L::kK >> 4));
                    const uint32_t d = tmem + s * kTcKeys;
#pragma unroll
                    for (int ks = 0; ks < D / kUmmaK; ++ks)
                        umma_f16(d, q_desc + (uint64_t)((ks >> 2) * (kTcRows * 128 >> 4) + 2 * (ks & 3)), kd + (uint64_t)((ks >> 2) * (kTcBox >> 4) + 2 * (ks & 3)), idesc_s, ks > 0 ? 1u : 0u);
                    umma_commit(&s_full[s]);
                    umma_commit(&k_empty[s]);
                }
                __syncwarp();
            };
            issue_s(it);
            for (int j = 0; j < n; ++j, ++it) {
                // (the score buffer of the next tile last held this one's predecessor's weights, whose product is ahead of it in the tensor pipe)
                if (j + 1 < n) issue_s(it + 1);
                const uint32_t s = (uint32_t)it & 1u, ph = (uint32_t)(it >> 1) & 1u;
                mbar_wait_or_leave(&v_full[s], ph, dead);
                mbar_wait_or_leave(&p_full[s], ph, dead);
                tc_fence_after();
                if (leader) {
                    const uint64_t vd = v_desc + (uint64_t)(s * (L::kV >> 4));
                    const uint32_t pa = tmem + s * kTcKeys;
#pragma unroll
                    for (int ks = 0; ks < 2 * kTcKeys / kUmmaK; ++ks)   // hi, then lo
                        umma_f16_ts(o_tmem, pa + (uint32_t)(ks * 8), vd + (uint64_t)((ks & 3) * (2048 >> 4)), idesc_o, ks > 0 || j > 0 ? 1u : 0u);
                    umma_commit(&v_empty[s]);
                    umma_commit(&o_done[s]);
                }
                __syncwarp();
            }
        } else {
            // ================= softmax: a thread per row =================
            const int quarter = warp & 3, r = quarter * 32 + lane, tl = r / R, hr = r % R, h = g * R + hr;
            const uint32_t my = (uint32_t)(quarter * 32) << 16;
            const bool mine = tl < count;
            const int p = mine ? a.pos[tA + tl] : -1, f = mine ? pa_first_key(a, p) : 0;
            const float sc = fabsf(pa_scale(a, h));
            constexpr float kLog2E = 1.4426950408889634f;
            // scores leave TMEM as q . k; plain: p = 2^(q . k * sl - m * sl), m the largest q . k; capped, biased: first x = the score times log2 e
            const float sl = fmaxf(sc * kLog2E, 1e-30f);   // never 0: a masked score is -inf
            const float over_cap = FORM == kTcCapped ? sc / a.softcap : 0.f, cap2 = a.softcap * kLog2E;
            const float hb2 = FORM == kTcSigmoid && a.head_bias ? a.head_bias[h] * kLog2E : 0.f;
            const float* brow = nullptr;
            float far_bias = 0.f;
            if (FORM == kTcBiased && a.dist_bias) {
                brow = bias_s + hr * (tn + kTcBiasPad) + kTcBiasFront;
                far_bias = a.dist_bias[(size_t)h * a.dist_n + a.dist_n - 1] * kLog2E;
            }
            float m = -1e30f, l = 0.f;   // m: what the exponents are taken against (the scores of FORM plain unscaled)
            const float step = FORM == kTcPlain ? sl : 1.f;   // log2 units per unit of m
            for (int j = 0; j < n_kt; ++j) {
                const int it = it0 + j, s = it & 1, k0 = key0 + j * kTcKeys;
                const uint32_t ph = (uint32_t)(it >> 1) & 1u, st = tmem + my + (uint32_t)(s * kTcKeys);
                mbar_wait_or_leave(&s_full[s], ph, dead);
                tc_fence_after();
                if (k0 + kTcKeys > pZ + 1 || k0 < fA) {
                    // V rows behind the context, and those ahead of the first key that any row sees: 0 * NaN must stay 0. (After the wait above: these scores follow the product two tiles before in
                    // the tensor pipe, so the stage has seen its last but one load and its barrier can be waited on by parity.)
                    mbar_wait_or_leave(&v_full[s], ph, dead);
                    for (int i = threadIdx.x - 64; i < kTcKeys * (DV / 8); i += 128) {
                        const int vr = i / (DV / 8), c = i % (DV / 8);
                        if (k0 + vr >= fA && k0 + vr <= pZ) continue;
                        st_shared_v4(smem_u32(smem + L::kOffV + s * L::kV + (c / 8) * kTcBox) + (uint32_t)(vr * 128 + (c & 7) * 16), 0u, 0u, 0u, 0u);
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
                    if (brow && !__all_sync(0xffffffffu, p < 0 || p - (k0 + kTcKeys - 1) >= a.dist_n - 1)) {
                        const int most = tn - 1 + 2 * kTcRows - kTcKeys;
                        const float* b = brow + max(min(p - k0, most), 0);   // rows without a token: any place of the table
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
                    if (j > 0 && __any_sync(0xffffffffu, grown)) {
                        mbar_wait_or_leave(&o_done[s ^ 1], (uint32_t)((it - 1) >> 1) & 1u, dead);
                        tc_fence_after();
                        const float alpha = grown ? ex2_approx((m - top) * step) : 1.f;
#pragma unroll 1
                        for (int c = 0; c < DV; c += 32) {
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
                if (lane == 0) mbar_arrive(&p_full[s]);
            }
            // (a wait by parity must be neither two phases behind nor ahead: a barrier per stage, whose last but one product these scores imply)
            const int last = it0 + n_kt - 1;
            mbar_wait_or_leave(&o_done[last & 1], (uint32_t)(last >> 1) & 1u, dead);
            tc_fence_after();
            const float m2 = m * step, sink_w = FORM == kTcSigmoid ? 0.f : a.sink ? 1.f : a.denom_bias, s2 = a.sink ? a.sink[h] * kLog2E : 0.f;
            const size_t dst = ((size_t)(tA + tl) * q_units + h * a.maps + mp) * DV;
            // division by the weights' sum, in which the sink counts
            float inv = 1.f;
            if (FORM != kTcSigmoid) {
                const float M = sink_w > 0.f ? fmaxf(m2, s2) : m2, fo = ex2_approx(m2 - M);
                inv = fo / (l * fo + (sink_w > 0.f ? sink_w * ex2_approx(s2 - M) : 0.f));
            }
            if (*dead) inv = __int_as_float(0x7fffffff);
#pragma unroll 1
            for (int c = 0; c < DV; c += 32) {
                uint32_t ov[32];
                __syncwarp();
                tmem_ld_32x32_async(o_tmem + my + (uint32_t)c, ov);
                tmem_wait_ld<32>(ov);
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
            tc_fence_before();
        }
        it0 += n_kt;
        first = end;
        __syncthreads();   // the next tile's Q rows and products come after everybody is done with this one's
        tc_fence_after();
    }
    if (warp == 1) tmem_dealloc(tmem, L::kTmemCols);
}

template <int D, int DV, int FORM>
static int launch_tc(const PA& a, int longest_entry, cudaStream_t s) {
    using L = TcSmem<D, DV>;
    const int R = a.heads / a.kv_heads, TQ = kTcRows / R;
    int bias = 0;
    if (FORM == kTcBiased && a.dist_bias) {
        if (a.dist_n > kTcBiasFloats) return -1;
        bias = R * (a.dist_n + kTcBiasPad);
    }
    if (bias > kTcBiasFloats) return -1;
    const int smem = L::kOffBias + bias * 4 + 1024;
    const bool several = a.n_tokens != longest_entry;   // more than one entry, as far as the host knows
    const long long windows = (a.n_tokens + TQ - 1) / TQ;
    if (windows * 2 > 65535) return -1;
    static unsigned long long done = 0;
    const cudaError_t e = ensure_max_dynamic_smem((const void*)paged_attn_tc_kernel<D, DV, FORM>, L::kOffBias + kTcBiasFloats * 4 + 1024, done);
    if (e != cudaSuccess) return (int)e;
    CUtensorMap mk, mv;
    // the pool's height is not part of the call: any row that an int can name
    constexpr long long kAnyRow = (1ll << 31) - 1;
    if (!make_tma_map_2d(&mk, a.k_pool, kAnyRow, a.kv_heads * a.maps * D, kTcKeys) || !make_tma_map_2d(&mv, a.v_pool, kAnyRow, a.kv_heads * DV, kTcKeys)) return -1;
    const int parts = several ? 2 : 1;
    paged_attn_tc_kernel<D, DV, FORM><<<dim3((unsigned)(a.kv_heads * a.maps), (unsigned)(windows * parts)), kTcThreads, smem, s>>>(mk, mv, a, TQ, parts, several ? 1 : 0);
    return (int)cudaGetLastError();
}

template <int D, int DV>
static int launch_tc_for(const PA& a, int longest_entry, cudaStream_t s) {
    if (a.sigmoid) return launch_tc<D, DV, kTcSigmoid>(a, longest_entry, s);
    if (a.softcap > 0.f) return launch_tc<D, DV, kTcCapped>(a, longest_entry, s);
    if (a.dist_bias) return launch_tc<D, DV, kTcBiased>(a, longest_entry, s);
    return launch_tc<D, DV, kTcPlain>(a, longest_entry, s);
}

int paged_attention_tc(const PA& a, int longest_entry, int longest_seen, cudaStream_t s) {
    const int R = a.heads / a.kv_heads;
    // a cap beside a sink or a bias keeps the row kernel, whose weights stay in 32 bits
    if (R > 8 || a.page_rows % kTcKeys || (a.softcap > 0.f && (a.dist_bias || a.sink)) || a.kv_heads * a.maps > 65535) return -1;
    // a short portion of one sequence, 64-wide heads, a distance bias: the fixed part of a CTA and a bias per score outweigh products half as long, and the
    // mma.sync tiles are faster (16 / 8 heads, us there / here: 40 tokens 11.2 / 13.3, 400 tokens 17.4 / 20.5, 100 behind 1000 31.7 / 35.8; but 700 tokens
    // 28.7 / 27.8, 2048 tokens 73 / 48). Where other sequences are beside it their single tokens decide
    if (a.dist_bias && a.dim == 64 && a.vdim == 64 && a.chunk == 0 && a.window == 0 && a.n_tokens == longest_entry && a.n_tokens <= 512 && longest_seen > 0 && longest_seen <= 1200) return -1;
    int rc = -1;
    if (a.dim == 128 && a.vdim == 128) rc = launch_tc_for<128, 128>(a, longest_entry, s);
    else if (a.dim == 64 && a.vdim == 64) rc = launch_tc_for<64, 64>(a, longest_entry, s);
    else if (a.dim == 128 && a.vdim == 256) rc = launch_tc_for<128, 256>(a, longest_entry, s);
    if (rc != 0) return rc;
    count_launch();
    if (a.n_tokens != longest_entry) return paged_decode(a, longest_seen, a.n_tokens - (longest_entry > 0 ? longest_entry : 0), 0, s);   // the sequences that bring one token
    return 0;
}

}  // namespace b200
