// Latent attention: the cache holds ONE normed low-rank row c_j per token and layer (no per-head keys or values).
// With k_j = W_uk c_j and v_j = W_uv c_j the key up-projection is folded into the query (qa = W_uk,h^T q_h) and the
// value up-projection is applied after the weighted sum, so attention runs on the cached rows themselves:
//   s_j = scale <qa_h, c_j>,  out_h = sum_j p_j c_j,  p = softmax over {s_j} and one sink logit per head that has no
//   row and no value (it only enlarges the denominator).
// Rows live in a page pool [n_pages, page_rows, rank] addressed through per-sequence page lists (page_pool.h), the
// same lists for every layer. Scores, softmax and the weighted sum are fp32 whatever the cache dtype.
// Designs that rotate one key part shared by all heads append it to the cached row ([latent | rotated part],
// latent_store_rot_kernel) and the head's rotated query part to the absorbed query: the score is still one dot product over
// the row, and of the weighted sum the caller uses the latent columns. A sliding window (window > 0: position p sees rows
// p - window < j <= p) bounds the walk from below; without a sink (NULL) the softmax is plain.
//
// Kernels:
//   latent_store_kernel        RMS norm (eps inside the root) of the down-projected row, times weight -> its page slot
//   latent_attn_kernel         one CTA per (token, head): the warps walk the visible rows round-robin, each row read
//                              coalesced by one warp; per-warp online softmax, merged with the sink at the end
//   latent_attn_tile_kernel    bf16 tensor-core form (mma.sync): one CTA per 32 (token, head) rows; half tiles of 32 cached
//                              rows arrive in two shared-memory buffers by cp.async and are the operand of both the
//                              scores and the weighted sum (prompt portions and decoded tokens alike; the default for
//                              bf16 caches); decode batches split long contexts over several CTAs
//   latent_attn_combine_kernel merges the shares of a split launch and the sink
#include <cooperative_groups.h>

#include <algorithm>

#include "b200_serve.h"
#include "common.cuh"
#include "latent_attention.cuh"
#include "launch_count.h"
#include "rotary.cuh"
#include "tc_common.cuh"

namespace b200 {
namespace cg = cooperative_groups;

constexpr int kMaxRankPerLane = 20;   // rank <= 640 (a latent of 512 with a rotated part of 64 or 128)

template <typename T>
__global__ void __launch_bounds__(128) latent_store_kernel(const float* __restrict__ raw, long long ld_raw,
                                                           const float* __restrict__ w, float eps, T* __restrict__ pool,
                                                           const int* __restrict__ pages, int max_pages, int page_rows,
                                                           const int* __restrict__ slot, const int* __restrict__ pos,
                                                           int rank) {
    __shared__ float red[4];
    const int t = blockIdx.x;
    const float* src = raw + (size_t)t * ld_raw;
    float q = 0.f;
    for (int i = threadIdx.x; i < rank; i += blockDim.x) q += src[i] * src[i];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) q += __shfl_xor_sync(0xffffffffu, q, o);
    if (threadIdx.x % 32 == 0) red[threadIdx.x / 32] = q;
    __syncthreads();
    const float tot = red[0] + red[1] + red[2] + red[3];
    const float r = 1.0f / sqrtf(tot / (float)rank + eps);
    const int p = pos[t];
    const size_t row = (size_t)pages[(size_t)slot[t] * max_pages + p / page_rows] * page_rows + p % page_rows;
    T* dst = pool + row * rank;
    for (int i = threadIdx.x; i < rank; i += blockDim.x) dst[i] = DT<T>::from_f(src[i] * r * w[i]);
}

// 1 / sqrt(mean(src[0:n]^2) + eps) over a CTA of 128 threads
__device__ __forceinline__ float row_rinv(const float* src, int n, float eps, float* red) {
    float q = 0.f;
    for (int i = threadIdx.x; i < n; i += blockDim.x) q += src[i] * src[i];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) q += __shfl_xor_sync(0xffffffffu, q, o);
    if (threadIdx.x % 32 == 0) red[threadIdx.x / 32] = q;
    __syncthreads();
    const float tot = red[0] + red[1] + red[2] + red[3];
    return 1.0f / sqrtf(tot / (float)n + eps);
}

// row = [norm(raw[0:rank]) * w | rot(raw[rank:rank+extra])]
template <typename T>
__device__ __forceinline__ void store_rot_row(const float* raw, long long ld_raw, const float* w, float eps, T* pool, const int* pages,
                                              int max_pages, int page_rows, const int* slot, const int* pos, int rank, int extra,
                                              const float* cs, const float* sn, int layout, float* red) {
    const int t = blockIdx.x;
    const float* src = raw + (size_t)t * ld_raw;
    const float r = row_rinv(src, rank, eps, red);
    const int p = pos[t];
    const size_t row = (size_t)pages[(size_t)slot[t] * max_pages + p / page_rows] * page_rows + p % page_rows;
    T* dst = pool + row * (rank + extra);
    for (int i = threadIdx.x; i < rank; i += blockDim.x) dst[i] = DT<T>::from_f(src[i] * r * w[i]);
    const int nf = extra / 2;
    for (int i = threadIdx.x; i < extra; i += blockDim.x)
        dst[rank + i] = DT<T>::from_f(rotary_component(src + rank, i, 2 * nf, layout, cs + (size_t)t * nf, sn + (size_t)t * nf));
}

template <typename T>
__global__ void __launch_bounds__(128) latent_store_rot_kernel(const float* __restrict__ raw, long long ld_raw, const float* __restrict__ w,
                                                               float eps, T* __restrict__ pool, const int* __restrict__ pages, int max_pages,
                                                               int page_rows, const int* __restrict__ slot, const int* __restrict__ pos, int rank,
                                                               int extra, const float* __restrict__ cs, const float* __restrict__ sn, int layout) {
    __shared__ float red[4];
    store_rot_row<T>(raw, ld_raw, w, eps, pool, pages, max_pages, page_rows, slot, pos, rank, extra, cs, sn, layout, red);
}

// blockIdx.y 0: the normed query row as GEMM operand; 1: the cache row
template <typename T>
__global__ void __launch_bounds__(128) latent_norms_kernel(const b200_latent_norms_args a) {
    __shared__ float red[4];
    if (blockIdx.y == 0) {
        const float* src = a.raw + (size_t)blockIdx.x * a.ld_raw + a.q_off;
        const float r = row_rinv(src, a.q_rank, a.eps, red);
        T* dst = reinterpret_cast<T*>(a.q_out) + (size_t)blockIdx.x * a.q_rank;
        for (int i = threadIdx.x; i < a.q_rank; i += blockDim.x) dst[i] = DT<T>::from_f(src[i] * r * a.q_norm[i]);
    } else
        store_rot_row<T>(a.raw + a.kv_off, a.ld_raw, a.kv_norm, a.eps, reinterpret_cast<T*>(a.pool), a.pages, a.max_pages, a.page_rows, a.slot,
                         a.pos, a.rank, a.extra, a.cos, a.sin, a.rot_layout, red);
}

template <typename T>
__global__ void __launch_bounds__(128) latent_attn_kernel(const float* __restrict__ qa, float* __restrict__ out,
                                                          const T* __restrict__ pool, const int* __restrict__ pages,
                                                          int max_pages, int page_rows, const int* __restrict__ slot,
                                                          const int* __restrict__ pos, const float* __restrict__ sink,
                                                          float scale, int heads, int rank, int window) {
    extern __shared__ float sm[];          // q[rank] | o[4][rank] | m[4] | l[4]
    float* q = sm;
    float* so = sm + rank;
    float* sml = so + 4 * rank;
    const int t = blockIdx.x, h = blockIdx.y;
    const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
    const float* qsrc = qa + ((size_t)t * heads + h) * rank;
    for (int i = threadIdx.x; i < rank; i += blockDim.x) q[i] = qsrc[i];
    __syncthreads();
    float qr[kMaxRankPerLane], o[kMaxRankPerLane];
#pragma unroll
    for (int i = 0; i < kMaxRankPerLane; ++i) {
        const int r = i * 32 + lane;
        qr[i] = r < rank ? q[r] : 0.f;
        o[i] = 0.f;
    }
    const int n_keys = pos[t] + 1;
    const int* list = pages + (size_t)slot[t] * max_pages;
    float m = -INFINITY, l = 0.f;
    const int j_lo = window > 0 ? max(0, n_keys - window) : 0;
    for (int j = j_lo + warp; j < n_keys; j += 4) {
        const T* c = pool + ((size_t)list[j / page_rows] * page_rows + j % page_rows) * rank;
        float cr[kMaxRankPerLane];
        float d = 0.f;
#pragma unroll
        for (int i = 0; i < kMaxRankPerLane; ++i) {
            const int r = i * 32 + lane;
            cr[i] = (i * 32 < rank && r < rank) ? DT<T>::to_f(c[r]) : 0.f;
            d = fmaf(qr[i], cr[i], d);
        }
#pragma unroll
        for (int s = 16; s > 0; s >>= 1) d += __shfl_xor_sync(0xffffffffu, d, s);
        const float sc = d * scale;
        const float mn = fmaxf(m, sc);
        const float alpha = expf(m - mn), p = expf(sc - mn);
        l = l * alpha + p;
#pragma unroll
        for (int i = 0; i < kMaxRankPerLane; ++i) o[i] = o[i] * alpha + p * cr[i];
        m = mn;
    }
#pragma unroll
    for (int i = 0; i < kMaxRankPerLane; ++i) {
        const int r = i * 32 + lane;
        if (r < rank) so[warp * rank + r] = o[i];
    }
    if (lane == 0) { sml[warp] = m; sml[4 + warp] = l; }
    __syncthreads();
    const float sk = sink ? sink[h] : -INFINITY;   // no sink: nothing joins the denominator
    float M = sk;
#pragma unroll
    for (int w = 0; w < 4; ++w) M = fmaxf(M, sml[w]);
    float f[4], den = expf(sk - M);
#pragma unroll
    for (int w = 0; w < 4; ++w) {
        f[w] = expf(sml[w] - M);     // a warp without rows: exp(-inf) = 0
        den += sml[4 + w] * f[w];
    }
    const float inv = 1.0f / den;
    float* dst = out + ((size_t)t * heads + h) * rank;
    for (int r = threadIdx.x; r < rank; r += blockDim.x)
        dst[r] = (so[r] * f[0] + so[rank + r] * f[1] + so[2 * rank + r] * f[2] + so[3 * rank + r] * f[3]) * inv;
}


// ---- bf16 tensor-core form ---------------------------------------------------------------------------------------
// One CTA = 32 rows of (token, head) pairs: TQ consecutive tokens of the packed batch x HG heads (all heads share the
// cached rows, so a row tile staged once serves HG heads). 8 warps. Per half tile of 32 cached rows (two buffers: the
// next half arrives by cp.async while this one is used):
//   S = Q C^T   : warp w computes the 8 keys [8 (w & 3), +8) for all 32 rows over its half of the padded rank; the two
//                 partial scores go to smem and are added in the softmax
//   softmax     : warp w owns rows [4w, 4w+4): mask, running max / sum (fp32), P as bf16 to smem, rescale factors
//   O += P C    : warp w owns output columns [64w', ...) of all 32 rows; the SAME smem tile is the B operand, read
//                 transposed with ldmatrix.trans
// The sink enters as the initial state (m = sink, l = 1, O = 0): a virtual row with a zero value.
// Tokens of different sequences inside one CTA (entry borders, decode batches) are walked segment by segment.
constexpr int kTileRows = 32, kTileKeys = 64, kHalfKeys = 32, kTileWarps = 8, kMaxSplits = 16;

__device__ __forceinline__ void ldsm_x4(uint32_t (&r)[4], const void* p) {
    const uint32_t a = (uint32_t)__cvta_generic_to_shared(p);
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a));
}
__device__ __forceinline__ void ldsm_x2_trans(uint32_t (&r)[2], const void* p) {
    const uint32_t a = (uint32_t)__cvta_generic_to_shared(p);
    asm volatile("ldmatrix.sync.aligned.m8n8.x2.trans.shared.b16 {%0,%1}, [%2];" : "=r"(r[0]), "=r"(r[1]) : "r"(a));
}
__device__ __forceinline__ void mma_bf16_16816(float (&d)[4], const uint32_t (&a)[4], const uint32_t (&b)[2]) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

template <int NT>   // n8 column tiles of the output per warp: padded rank <= 64 * NT
__global__ void __launch_bounds__(256, NT <= 8 ? 2 : 1) latent_attn_tile_kernel(const float* __restrict__ qa, float* __restrict__ out,
                                                               const __nv_bfloat16* __restrict__ pool, const int* __restrict__ pages,
                                                               int max_pages, int page_rows, const int* __restrict__ slot,
                                                               const int* __restrict__ pos, const float* __restrict__ sink, float scale,
                                                               int n_tokens, int heads, int rank, int HG, int TQ, int splits,
                                                               float* __restrict__ part, int window, int out_cols, int single) {
    // out_cols: the weighted sum is formed for the first out_cols columns of a row only (a caller that uses the latent part
    // of [latent | rotated part] rows). single: one half-tile buffer instead of two (rows wider than 512: two CTAs still
    // share an SM, and the other CTA's arithmetic covers this one's load)
    // splits > 1 (blockIdx.z): this CTA walks one share of the key tiles and leaves (m, l, unnormalised O) per row in
    // `part` [token, head, split, 2 + rank]; latent_attn_combine_kernel merges the shares and the sink
    using bf = __nv_bfloat16;
    extern __shared__ __align__(16) unsigned char smraw[];
    const int rpad = (rank + 15) & ~15, RS = rpad + 8;           // smem row stride in elements (16-byte multiple)
    bf* Qs = reinterpret_cast<bf*>(smraw);                        // [32][RS]
    bf* Ks = Qs + kTileRows * RS;                                 // [2][32][RS]: half tiles, one being filled while the other is used
    float* Ss = reinterpret_cast<float*>(Ks + (single ? kHalfKeys : kTileKeys) * RS);    // [2][32][36]: partial scores of the two halves of the rank
    bf* Ps = reinterpret_cast<bf*>(Ss);                           // [32][72]: a row's probabilities overwrite its own scores
    float* alpha_s = Ss + 2 * kTileRows * 36;                     // [32]
    float* linv_s = alpha_s + kTileRows;                          // [32]
    int* row_pos = reinterpret_cast<int*>(linv_s + kTileRows);    // [32]: position of the row's token, -1 = inactive

    const int warp = threadIdx.x / 32, lane = threadIdx.x % 32, gid = lane / 4, tig = lane % 4;
    const int t0 = blockIdx.x * TQ, h0 = blockIdx.y * HG;
    const int ntok = min(TQ, n_tokens - t0);
    const int n8 = ((out_cols + 15) & ~15) / 8;                   // n8 tiles of the output
    const int ntw = (n8 + kTileWarps - 1) / kTileWarps;           // per warp (<= NT)
    const int tile0 = warp * ntw;

    for (int first = 0; first < ntok;) {
        const int sl = slot[t0 + first];
        int cnt = 1;
        while (first + cnt < ntok && slot[t0 + first + cnt] == sl) ++cnt;
        const int all_keys = pos[t0 + first + cnt - 1] + 1;
        // the first row of the segment sees the oldest key: whole tiles from there (a half tile stays inside its page)
        const int seg_lo = window > 0 ? max(0, pos[t0 + first] - window + 1) / kTileKeys * kTileKeys : 0;
        const int per = ((all_keys - seg_lo + kTileKeys - 1) / kTileKeys + splits - 1) / splits * kTileKeys;   // keys per share
        const int key_lo = seg_lo + blockIdx.z * per, n_keys = min(all_keys, key_lo + per);
        const int* list = pages + (size_t)sl * max_pages;
        __syncthreads();   // the previous segment's readers are done with the shared state
        if (threadIdx.x < kTileRows) {
            const int r = threadIdx.x, tl = r / HG, h = h0 + r % HG;
            row_pos[r] = (tl >= first && tl < first + cnt && tl < TQ && h < heads) ? pos[t0 + tl] : -1;
        }
        for (int i = threadIdx.x; i < kTileRows * rpad; i += blockDim.x) {
            const int r = i / rpad, c = i - r * rpad;
            const int tl = r / HG, h = h0 + r % HG;
            const bool on = tl >= first && tl < first + cnt && tl < TQ && h < heads && c < rank;
            Qs[r * RS + c] = __float2bfloat16_rn(on ? qa[((size_t)(t0 + tl) * heads + h) * rank + c] : 0.f);
        }
        // running state of the rows this warp owns in the softmax phase (uniform over the lanes)
        float m_run[4], l_run[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int r = warp * 4 + i, h = h0 + r % HG;
            const bool own_sink = splits == 1 && sink != nullptr;           // shares: the sink joins in the combine
            m_run[i] = !own_sink ? -1e30f : (h < heads ? sink[h] : 0.f);
            l_run[i] = own_sink ? 1.f : 0.f;
        }
        float o[2][NT][4];
#pragma unroll
        for (int a = 0; a < 2; ++a)
#pragma unroll
            for (int b = 0; b < NT; ++b)
#pragma unroll
                for (int c = 0; c < 4; ++c) o[a][b][c] = 0.f;

        // half tiles of 32 cached rows, double-buffered: the rows of half i + 1 arrive (cp.async, 16 bytes each, zero-filled
        // beyond the context and in the padding columns) while half i is scored, normalised and accumulated
        const bool vec = (rank & 7) == 0;
        const int chunks = rpad / 8;
        auto load_half = [&](int k0, bf* dstbuf) {
            if (vec) {
                const bool one_page = page_rows % kHalfKeys == 0;   // a half tile never straddles two pages
                const size_t page_base = one_page ? (size_t)list[k0 / page_rows] * page_rows + k0 % page_rows : 0;
                for (int i = threadIdx.x; i < kHalfKeys * chunks; i += blockDim.x) {
                    const int kr = i / chunks, ch = i - kr * chunks;
                    const int j = k0 + kr;
                    const bool ok = j < n_keys && ch * 8 < rank;
                    const size_t row = !ok ? 0 : one_page ? page_base + kr : (size_t)list[j / page_rows] * page_rows + j % page_rows;
                    const bf* src = ok ? pool + row * rank + ch * 8 : pool;
                    const uint32_t dst = (uint32_t)__cvta_generic_to_shared(dstbuf + kr * RS + ch * 8);
                    const int bytes = ok ? 16 : 0;
                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
                }
            } else {
                for (int i = threadIdx.x; i < kHalfKeys * rpad; i += blockDim.x) {
                    const int kr = i / rpad, c = i - kr * rpad;
                    const int j = k0 + kr;
                    bf v = __float2bfloat16_rn(0.f);
                    if (j < n_keys && c < rank) v = pool[((size_t)list[j / page_rows] * page_rows + j % page_rows) * rank + c];
                    dstbuf[kr * RS + c] = v;
                }
            }
            __syncwarp();   // the lanes close their group of copies together
            asm volatile("cp.async.commit_group;" ::: "memory");
        };
        // the rank is split between the warp groups 0-3 and 4-7 in the score phase (k steps of 16)
        const int ksplit = (rpad / 32) * 16;
        const int kbeg = warp < 4 ? 0 : ksplit, kend = warp < 4 ? ksplit : rpad;
        if (!single && key_lo < n_keys) load_half(key_lo, Ks);
        int buf = 0;
        for (int k0 = key_lo; k0 < n_keys; k0 += kHalfKeys, buf ^= single ? 0 : 1) {
            bf* Kb = Ks + buf * kHalfKeys * RS;
            if (single) {
                __syncthreads();   // the buffer, Ss and Ps are no longer read
                load_half(k0, Ks);
            }
            asm volatile("cp.async.wait_group 0;" ::: "memory");
            __syncthreads();   // half k0 has landed for everybody; the other buffer, Ss and Ps are no longer read
            if (!single && k0 + kHalfKeys < n_keys) load_half(k0 + kHalfKeys, Ks + (buf ^ 1) * kHalfKeys * RS);
            {   // ---- partial scores: keys [8 (warp & 3), +8), rank columns [kbeg, kend)
                float s[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
                const bf* krow = Kb + ((warp & 3) * 8 + gid) * RS + tig * 2;
                const bf* q0 = Qs + ((lane & 7) + ((lane >> 3) & 1) * 8) * RS + (lane >> 4) * 8;
                const bf* q1 = q0 + 16 * RS;
                for (int ks = kbeg; ks < kend; ks += 16) {
                    uint32_t a0[4], a1[4], b[2];
                    ldsm_x4(a0, q0 + ks);
                    ldsm_x4(a1, q1 + ks);
                    b[0] = *reinterpret_cast<const uint32_t*>(krow + ks);
                    b[1] = *reinterpret_cast<const uint32_t*>(krow + ks + 8);
                    mma_bf16_16816(s[0], a0, b);
                    mma_bf16_16816(s[1], a1, b);
                }
                float* base = Ss + (warp >> 2) * kTileRows * 36;
#pragma unroll
                for (int mt = 0; mt < 2; ++mt) {
                    float* d0 = base + (mt * 16 + gid) * 36 + (warp & 3) * 8 + tig * 2;
                    d0[0] = s[mt][0]; d0[1] = s[mt][1];
                    d0[8 * 36] = s[mt][2]; d0[8 * 36 + 1] = s[mt][3];
                }
            }
            __syncthreads();
#pragma unroll
            for (int i = 0; i < 4; ++i) {   // ---- softmax of rows [4 warp, 4 warp + 4): one key per lane
                const int r = warp * 4 + i, rp = row_pos[r];
                const int ka = k0 + lane;
                const bool seen = ka <= rp && (window <= 0 || ka > rp - window);
                const float sa = seen ? (Ss[r * 36 + lane] + Ss[(kTileRows + r) * 36 + lane]) * scale : -INFINITY;
                float mx = sa;
#pragma unroll
                for (int d = 16; d > 0; d >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, d));
                const float mn = fmaxf(m_run[i], mx);           // finite: m starts at the sink (or at -1e30 in a share)
                const float pa = seen ? expf(sa - mn) : 0.f;
                float sum = pa;
#pragma unroll
                for (int d = 16; d > 0; d >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, d);
                const float al = expf(m_run[i] - mn);
                l_run[i] = l_run[i] * al + sum;
                m_run[i] = mn;
                Ps[r * 72 + lane] = __float2bfloat16_rn(pa);    // after every lane has read its scores (the shuffles above)
                if (lane == 0) alpha_s[r] = al;
            }
            __syncthreads();
            {   // ---- O = O * alpha + P C for this warp's output columns
#pragma unroll
                for (int mt = 0; mt < 2; ++mt) {
                    const float a0 = alpha_s[mt * 16 + gid], a1 = alpha_s[mt * 16 + gid + 8];
#pragma unroll
                    for (int nt = 0; nt < NT; ++nt) { o[mt][nt][0] *= a0; o[mt][nt][1] *= a0; o[mt][nt][2] *= a1; o[mt][nt][3] *= a1; }
                }
#pragma unroll
                for (int kk = 0; kk < kHalfKeys; kk += 16) {
                    uint32_t p0[4], p1[4];
                    ldsm_x4(p0, Ps + ((lane & 7) + ((lane >> 3) & 1) * 8) * 72 + kk + (lane >> 4) * 8);
                    ldsm_x4(p1, Ps + (16 + (lane & 7) + ((lane >> 3) & 1) * 8) * 72 + kk + (lane >> 4) * 8);
#pragma unroll
                    for (int nt = 0; nt < NT; ++nt) {
                        const int tile = tile0 + nt;
                        if (nt < ntw && tile < n8) {
                            uint32_t b[2];
                            ldsm_x2_trans(b, Kb + (kk + (lane & 15)) * RS + tile * 8);
                            mma_bf16_16816(o[0][nt], p0, b);
                            mma_bf16_16816(o[1][nt], p1, b);
                        }
                    }
                }
            }
        }
        if (lane == 0) {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int r = warp * 4 + i;
                linv_s[r] = splits > 1 ? 1.0f : 1.0f / l_run[i];
                if (splits > 1 && row_pos[r] >= 0) {
                    float* pr = part + (((size_t)(t0 + r / HG) * heads + h0 + r % HG) * splits + blockIdx.z) * (rank + 2);
                    pr[0] = m_run[i];
                    pr[1] = l_run[i];
                }
            }
        }
        __syncthreads();
#pragma unroll
        for (int mt = 0; mt < 2; ++mt)
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                const int r = mt * 16 + gid + half * 8;
                if (row_pos[r] < 0) continue;
                const int tl = r / HG, h = h0 + r % HG;
                float* dst = splits > 1 ? part + (((size_t)(t0 + tl) * heads + h) * splits + blockIdx.z) * (rank + 2) + 2
                                        : out + ((size_t)(t0 + tl) * heads + h) * rank;
                const float inv = linv_s[r];
#pragma unroll
                for (int nt = 0; nt < NT; ++nt) {
                    const int tile = tile0 + nt;
                    if (nt < ntw && tile < n8) {
                        const int c = tile * 8 + tig * 2;
                        if (c < out_cols) dst[c] = o[mt][nt][half * 2] * inv;
                        if (c + 1 < out_cols) dst[c + 1] = o[mt][nt][half * 2 + 1] * inv;
                    }
                }
            }
        first += cnt;
    }
}

// merges the shares of a split launch: grid (token, head)
__global__ void __launch_bounds__(128) latent_attn_combine_kernel(const float* __restrict__ part, float* __restrict__ out,
                                                                  const float* __restrict__ sink, int heads, int rank, int splits, int out_cols) {
    const int t = blockIdx.x, h = blockIdx.y;
    const float* p = part + ((size_t)t * heads + h) * splits * (rank + 2);
    const float sk = sink ? sink[h] : -INFINITY;
    float M = sk;
    for (int z = 0; z < splits; ++z) M = fmaxf(M, p[(size_t)z * (rank + 2)]);
    float den = expf(sk - M);
    for (int z = 0; z < splits; ++z) den += p[(size_t)z * (rank + 2) + 1] * expf(p[(size_t)z * (rank + 2)] - M);
    const float inv = 1.0f / den;
    for (int c = threadIdx.x; c < out_cols; c += blockDim.x) {
        float acc = 0.f;
        for (int z = 0; z < splits; ++z) acc += p[(size_t)z * (rank + 2) + 2 + c] * expf(p[(size_t)z * (rank + 2)] - M);
        out[((size_t)t * heads + h) * rank + c] = acc * inv;
    }
}

// ---- bf16, single tokens (decode batches) ------------------------------------------------------------------------------
// A cluster of CTAs shares one token's cached rows; a CTA holds up to 16 heads of it, the M rows of one mma tile. What bounds it is
// the way to the rows (a few MB per launch) and the length of the chain behind them, so the rows are requested before anything else,
// two half tiles of 32 at once, two CTAs fit an SM, and the shares meet in distributed shared memory (rank order) in the same launch.
// A half tile comes by TMA, a box per lane of one warp, its place in the pool looked up a step before (by cp.async, twelve copies and their addresses
// per lane behind that lookup, a step of 32 rows took 2.6 us); pages that are no multiple of a half tile keep cp.async.
//   scores   warp w: keys [16 (w & 1), +16) x 16 heads over a quarter (w >> 1) of the row; the four partial sums meet in shared memory
//   softmax  warp w: heads 2w, 2w + 1, a key per lane; the weights leave as the sum of two bfloat16: rounded to one, they lose the more the fewer
//            shares there are (a share's largest is 1, which is exact): 1.84e-3 of the result's norm for 32 sequences in 512 shares, 1.86e-3 in 256; 1.54e-3 now, the queries' rounding
//   values   warp w: an eighth of the output columns, the rows read transposed by ldmatrix
// The sink joins in the merge. Measured, 8 sequences of up to 1024 rows of 576, 16 heads, 512 columns out: the tile kernel with its
// combine launch 53.3 us, by cp.async 16.2, this 14.6 us (weights of one bfloat16: 14.0); 32 sequences of up to 2048 rows 34 / 26, one of 2048 19.1 / 16.1.
constexpr int kLdMaxCluster = 16;

__device__ __forceinline__ void ldsm_x4_at(uint32_t (&r)[4], uint32_t a) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a) : "memory");
}
__device__ __forceinline__ void ldsm_x4_trans_at(uint32_t (&r)[4], uint32_t a) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a));
}

// n8 column tiles of the output per warp: out_cols <= 64 * NT. TMA: a half tile lies in one page, and comes as boxes of 32 rows x 64 columns, swizzled over 128 bytes
template <int NT, bool TMA>
__global__ void __launch_bounds__(256, 2) latent_decode_kernel(const __grid_constant__ CUtensorMap map, const float* __restrict__ qa, float* __restrict__ out, const __nv_bfloat16* __restrict__ pool,
                                                               const int* __restrict__ pages, int max_pages, int page_rows, const int* __restrict__ slot,
                                                               const int* __restrict__ pos, const float* __restrict__ sink, float scale, int heads, int rank,
                                                               int window, int out_cols) {
    using bf = __nv_bfloat16;
    extern __shared__ __align__(1024) unsigned char smraw0[];
    unsigned char* smraw = TMA ? reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smraw0) + 1023) & ~(uintptr_t)1023) : smraw0;
    __shared__ uint64_t full[2];
    __shared__ int dead_s;
    volatile int* dead = &dead_s;
    if (TMA && threadIdx.x == 0) {
        mbar_init(&full[0], 1);
        mbar_init(&full[1], 1);
        *dead = 0;
        mbar_fence_init();
        tma_prefetch_desc(&map);
    }
    pdl_wait();
    pdl_launch_dependents();
    const int rpad = (rank + 15) & ~15, RS = rpad + 8, splits = gridDim.x;
    bf* Ks = reinterpret_cast<bf*>(smraw);                     // [2][32][RS]
    const int boxes = (rank + 63) / 64, stage = boxes * kHalfKeys * 128;   // TMA: bytes of a half tile
    bf* Qs = TMA ? reinterpret_cast<bf*>(smraw + 2 * stage) : Ks + 2 * kHalfKeys * RS;   // [16][RS]
    float* Ss = reinterpret_cast<float*>(Qs + 16 * RS);        // [4][16][36]: partial scores [head][key]
    bf* Ps = reinterpret_cast<bf*>(Ss + 4 * 16 * 36);          // [16][40]: the weights, rounded
    bf* Pl = reinterpret_cast<bf*>(Ss);                        // [16][72]: what that left, over a row's own scores
    float* al_s = reinterpret_cast<float*>(Ps + 16 * 40);      // [16]
    float* ms = al_s + 16;                                     // [16]
    float* ls = ms + 16;                                       // [16]
    float* om = reinterpret_cast<float*>(smraw);               // [16][out_cols]: this CTA's share, once the rows have been used
    const int t = blockIdx.z, h0 = blockIdx.y * 16, warp = __shfl_sync(0xffffffffu, threadIdx.x / 32, 0), lane = threadIdx.x % 32, gid = lane / 4, tig = lane % 4;
    const int n = min(16, heads - h0), chunks = rpad / 8;
    // the query rows are requested first, ahead of the chain position -> page -> rows; a warp brings two heads
    constexpr int kQv = (32 * kMaxRankPerLane / 4 + 31) / 32;
    float4 qv[2][kQv];
#pragma unroll
    for (int x = 0; x < 2; ++x)
#pragma unroll
        for (int i = 0; i < kQv; ++i) {
            const int r = 2 * warp + x, c = (i * 32 + lane) * 4;   // rank % 8 == 0: four floats lie inside a head's row or behind it
            qv[x][i] = r < n && c < rank ? *reinterpret_cast<const float4*>(qa + ((size_t)t * heads + h0 + r) * rank + c) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
    const int p = pos[t];
    const int* list = pages + (size_t)slot[t] * max_pages;
    const int lo = window > 0 ? max(0, p - window + 1) : 0, first = lo & ~(kHalfKeys - 1);
    const int halves = (p - first) / kHalfKeys + 1, per = (halves + splits - 1) / splits;
    const int b0 = blockIdx.x * per, b1 = min(halves, b0 + per);
    const bool one_page = page_rows % kHalfKeys == 0;
    // a warp brings four whole rows, its lanes the 16-byte pieces of a row (one place in the pool per row, no division per piece)
    auto load_half = [&](int b) {
        const int k0 = first + b * kHalfKeys;
        const size_t base = one_page ? (size_t)list[k0 / page_rows] * page_rows + k0 % page_rows : 0;
        const uint32_t dst0 = (uint32_t)__cvta_generic_to_shared(Ks + ((b - b0) & 1) * kHalfKeys * RS);
#pragma unroll
        for (int i = 0; i < kHalfKeys / 8; ++i) {
            const int kr = i * 8 + warp, j = k0 + kr;
            const bool in = j <= p && j >= lo;
            const size_t row = !in ? 0 : one_page ? base + kr : (size_t)list[j / page_rows] * page_rows + j % page_rows;
            const bf* src = pool + row * rank;
            const uint32_t dst = dst0 + (uint32_t)(kr * RS) * 2u;
            for (int ch = lane; ch < chunks; ch += 32) {
                const bool ok = in && ch * 8 < rank;
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst + (uint32_t)ch * 16u), "l"(ok ? src + ch * 8 : pool), "r"(ok ? 16 : 0) : "memory");
            }
        }
    };
    auto close_group = [&]() {
        __syncwarp();   // the lanes close their group of copies together
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    auto row_of = [&](int b) { return list[(first + b * kHalfKeys) / page_rows] * page_rows + (first + b * kHalfKeys) % page_rows; };
    auto fetch = [&](int b, int row) {   // one warp, a box per lane
        uint64_t* bar = &full[(b - b0) & 1];
        if (lane == 0) mbar_expect_tx(bar, stage);
        __syncwarp();
        if (lane < boxes) tma_load_2d(smraw + ((b - b0) & 1) * stage + lane * (kHalfKeys * 128), &map, lane * 64, row, bar);
        __syncwarp();
    };
    if (TMA) {
        if (warp == 0) {
            const int r0 = b0 < b1 ? row_of(b0) : 0, r1 = b0 + 1 < b1 ? row_of(b0 + 1) : 0;
            if (b0 < b1) fetch(b0, r0);
            if (b0 + 1 < b1) fetch(b0 + 1, r1);
        }
    } else {
        if (b0 < b1) load_half(b0);
        close_group();
        if (b0 + 1 < b1) load_half(b0 + 1);
        close_group();
    }
#pragma unroll
    for (int x = 0; x < 2; ++x)
#pragma unroll
        for (int i = 0; i < kQv; ++i) {
            const int c = (i * 32 + lane) * 4;
            if (c < rpad) {
                const __nv_bfloat162 u = __floats2bfloat162_rn(qv[x][i].x, qv[x][i].y), v = __floats2bfloat162_rn(qv[x][i].z, qv[x][i].w);
                *reinterpret_cast<uint2*>(Qs + (2 * warp + x) * RS + c) = make_uint2(*reinterpret_cast<const uint32_t*>(&u), *reinterpret_cast<const uint32_t*>(&v));
            }
        }
    float m_run[2] = {-INFINITY, -INFINITY}, l_run[2] = {0.f, 0.f}, o[NT][4];
#pragma unroll
    for (int i = 0; i < NT; ++i) o[i][0] = o[i][1] = o[i][2] = o[i][3] = 0.f;
    const int steps = rpad / 16, kq = warp >> 1, ks0 = steps * kq / 4, ks1 = steps * (kq + 1) / 4;
    const int n8 = out_cols / 8, ntw = ((n8 + kTileWarps - 1) / kTileWarps + 1) & ~1, tile0 = warp * ntw;   // pairs of column tiles
    // where this lane's rows of the matrix loads lie: keys, columns 16 ks .. (row, then which of the two pieces), and values, a pair of column tiles
    const int k_row = (warp & 1) * 16 + (lane & 15), piece_hi = lane >> 4;
    auto k_at = [&](int b, int ks) -> uint32_t {
        if (TMA) return smem_u32(smraw) + (uint32_t)(((b - b0) & 1) * stage + (ks >> 2) * (kHalfKeys * 128) + k_row * 128 + ((((ks & 3) * 2 + piece_hi) ^ (k_row & 7)) << 4));
        return smem_u32(Ks + (((b - b0) & 1) * kHalfKeys + k_row) * RS + piece_hi * 8 + ks * 16);
    };
    auto v_at = [&](int b, int kk, int tile) -> uint32_t {
        const int r = kk + (lane & 15), piece = tile + piece_hi;
        if (TMA) return smem_u32(smraw) + (uint32_t)(((b - b0) & 1) * stage + (piece >> 3) * (kHalfKeys * 128) + r * 128 + (((piece & 7) ^ (r & 7)) << 4));
        return smem_u32(Ks + (((b - b0) & 1) * kHalfKeys + r) * RS + piece * 8);
    };
    if (TMA) __syncthreads();   // the barriers, and the query rows
    for (int b = b0; b < b1; ++b) {
        const int k0 = first + b * kHalfKeys;
        int next_row = 0;
        if (TMA) {
            if (warp == 0 && b + 2 < b1) next_row = row_of(b + 2);   // its place is looked up a step ahead
            mbar_wait_or_leave(&full[(b - b0) & 1], (uint32_t)((b - b0) >> 1) & 1u, dead);
            if (k0 < lo || k0 + kHalfKeys - 1 > p) {   // rows that the token does not see may hold anything: 0 * NaN must stay 0
                for (int kr = warp; kr < kHalfKeys; kr += kTileWarps)
                    if (k0 + kr < lo || k0 + kr > p)
                        for (int x = lane; x < boxes * 8; x += 32) *reinterpret_cast<uint4*>(smraw + ((b - b0) & 1) * stage + (x >> 3) * (kHalfKeys * 128) + kr * 128 + (x & 7) * 16) = make_uint4(0u, 0u, 0u, 0u);
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                __syncthreads();
            }
        } else {
            asm volatile("cp.async.wait_group 1;" ::: "memory");
            __syncthreads();   // half b has landed for everybody (and, the first time, the query rows)
        }
        {
            float s[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
            const bf* qb = Qs + ((lane & 7) + (lane >> 4) * 8) * RS + ((lane >> 3) & 1) * 8;
#pragma unroll 3
            for (int ks = ks0; ks < ks1; ++ks) {
                uint32_t a[4], q[4];
                ldsm_x4_at(a, k_at(b, ks));
                ldsm_x4(q, qb + ks * 16);
                const uint32_t q0[2] = {q[0], q[1]}, q1[2] = {q[2], q[3]};
                mma_bf16_16816(s[0], a, q0);
                mma_bf16_16816(s[1], a, q1);
            }
#pragma unroll
            for (int x = 0; x < 2; ++x)
#pragma unroll
                for (int e = 0; e < 4; ++e) Ss[(kq * 16 + x * 8 + tig * 2 + (e & 1)) * 36 + (warp & 1) * 16 + gid + (e >> 1) * 8] = s[x][e];
        }
        __syncthreads();
        const int j = k0 + lane;
        const bool seen = j <= p && j >= lo;
#pragma unroll
        for (int x = 0; x < 2; ++x) {
            const int r = 2 * warp + x;
            const float* sr = Ss + r * 36 + lane;
            const float v = seen ? ((sr[0] + sr[16 * 36]) + (sr[32 * 36] + sr[48 * 36])) * scale : -INFINITY;
            float mx = v;
#pragma unroll
            for (int d = 16; d > 0; d >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, d));
            const float mn = fmaxf(m_run[x], mx);
            const float pv = seen ? expf(v - mn) : 0.f, al = m_run[x] == mn ? 1.f : expf(m_run[x] - mn);
            float sum = pv;
#pragma unroll
            for (int d = 16; d > 0; d >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, d);
            l_run[x] = l_run[x] * al + sum;
            m_run[x] = mn;
            const bf hi = __float2bfloat16_rn(pv);
            Ps[r * 40 + lane] = hi;
            Pl[r * 72 + lane] = __float2bfloat16_rn(pv - __bfloat162float(hi));   // after every lane has read its scores (the shuffles above)
            if (lane == 0) al_s[r] = al;
        }
        __syncthreads();
        {
            const float a0 = al_s[gid], a1 = al_s[gid + 8];
#pragma unroll
            for (int i = 0; i < NT; ++i) { o[i][0] *= a0; o[i][1] *= a0; o[i][2] *= a1; o[i][3] *= a1; }
#pragma unroll
            for (int kk = 0; kk < kHalfKeys; kk += 16) {
                uint32_t a[4], al[4];
                ldsm_x4(a, Ps + (lane & 15) * 40 + kk + (lane >> 4) * 8);
                ldsm_x4(al, Pl + (lane & 15) * 72 + kk + (lane >> 4) * 8);
#pragma unroll
                for (int i = 0; i < NT; i += 2) {
                    if (i < ntw && tile0 + i < n8) {   // n8 is even: a pair of column tiles is inside or outside together
                        uint32_t v[4];
                        ldsm_x4_trans_at(v, v_at(b, kk, tile0 + i));
                        const uint32_t v0[2] = {v[0], v[1]}, v1[2] = {v[2], v[3]};
                        mma_bf16_16816(o[i], al, v0);
                        mma_bf16_16816(o[i + 1], al, v1);
                        mma_bf16_16816(o[i], a, v0);
                        mma_bf16_16816(o[i + 1], a, v1);
                    }
                }
            }
        }
        __syncthreads();   // nobody reads half b any more
        if (TMA) {
            if (warp == 0 && b + 2 < b1) fetch(b + 2, next_row);
        } else {
            if (b + 2 < b1) load_half(b + 2);
            close_group();
        }
    }
    if (!TMA) asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    if (TMA && *dead) {   // a wait was given up: nothing may land on the sums, or behind this CTA's end
        linger();
        __syncthreads();
        l_run[0] = l_run[1] = __int_as_float(0x7fffffff);
    }
#pragma unroll
    for (int i = 0; i < NT; ++i) {
        const int c = (tile0 + i) * 8 + tig * 2;
        if (i < ntw && c < out_cols) {
            *reinterpret_cast<float2*>(om + gid * out_cols + c) = make_float2(o[i][0], o[i][1]);
            *reinterpret_cast<float2*>(om + (gid + 8) * out_cols + c) = make_float2(o[i][2], o[i][3]);
        }
    }
    if (lane == 0) {
#pragma unroll
        for (int x = 0; x < 2; ++x) { ms[2 * warp + x] = m_run[x]; ls[2 * warp + x] = l_run[x]; }
    }
    cg::cluster_group cluster = cg::this_cluster();
    cluster.sync();
    float* fs = Ss;   // [16 heads][16 shares]: what a share counts with
    {
        const int r = threadIdx.x / kLdMaxCluster, q = threadIdx.x % kLdMaxCluster;
        const bool on = q < splits && r < n;
        const float sk = sink && r < n ? sink[h0 + r] : -INFINITY;
        const float mq = on ? cluster.map_shared_rank(ms, q)[r] : -INFINITY, lq = on ? cluster.map_shared_rank(ls, q)[r] : 0.f;
        float M = fmaxf(sk, mq);
#pragma unroll
        for (int d = kLdMaxCluster / 2; d > 0; d >>= 1) M = fmaxf(M, __shfl_xor_sync(0xffffffffu, M, d));
        const float f = mq == -INFINITY ? 0.f : expf(mq - M);
        float den = lq * f;
#pragma unroll
        for (int d = kLdMaxCluster / 2; d > 0; d >>= 1) den += __shfl_xor_sync(0xffffffffu, den, d);
        if (sk != -INFINITY) den += expf(sk - M);
        fs[threadIdx.x] = f / den;
    }
    __syncthreads();
    const int total = n * (out_cols / 4), share = (total + splits - 1) / splits;
    for (int i = blockIdx.x * share + threadIdx.x; i < min(total, ((int)blockIdx.x + 1) * share); i += 256) {
        const int r = i / (out_cols / 4), c = (i - r * (out_cols / 4)) * 4;
        float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 8
        for (int q = 0; q < splits; ++q) {
            const float4 v = *reinterpret_cast<const float4*>(cluster.map_shared_rank(om, q) + r * out_cols + c);
            const float f = fs[r * kLdMaxCluster + q];
            acc.x = fmaf(v.x, f, acc.x); acc.y = fmaf(v.y, f, acc.y); acc.z = fmaf(v.z, f, acc.z); acc.w = fmaf(v.w, f, acc.w);
        }
        *reinterpret_cast<float4*>(out + ((size_t)t * heads + h0 + r) * rank + c) = acc;
    }
    cluster.sync();   // nobody leaves while its share is read
}

template <int NT, bool TMA>
static int launch_latent_decode(const b200_latent_attention_args& a, int out_cols, int splits, cudaStream_t s) {
    const int rpad = (a.rank + 15) & ~15, RS = rpad + 8;
    const size_t rows = TMA ? 1024 + (size_t)2 * ((a.rank + 63) / 64) * kHalfKeys * 128 : (size_t)2 * kHalfKeys * RS * 2, smem = rows + (size_t)16 * RS * 2 + 4 * 16 * 36 * 4 + 16 * 40 * 2 + 3 * 16 * 4;
    static unsigned long long done = 0, wide = 0;
    cudaError_t e = ensure_max_dynamic_smem((const void*)latent_decode_kernel<NT, TMA>, 114 * 1024, done);
    if (e == cudaSuccess && splits > 8) {
        const int dev = current_device();
        if (!(wide & (1ull << dev))) {
            e = cudaFuncSetAttribute((const void*)latent_decode_kernel<NT, TMA>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
            if (e == cudaSuccess) wide |= 1ull << dev;
        }
    }
    if (e != cudaSuccess) return (int)e;
    CUtensorMap map{};
    constexpr long long kAnyRow = (1ll << 31) - 1;   // the pool's height is not part of the call: any row that an int can name
    if (TMA && !make_tma_map_2d(&map, a.pool, kAnyRow, a.rank, kHalfKeys)) return launch_latent_decode<NT, false>(a, out_cols, splits, s);
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)splits, (unsigned)((a.heads + 15) / 16), (unsigned)a.n_tokens);
    cfg.blockDim = dim3(256);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = (unsigned)splits;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = pdl_enabled() ? 2 : 1;
    e = cudaLaunchKernelEx(&cfg, latent_decode_kernel<NT, TMA>, map, a.qa, a.out, (const __nv_bfloat16*)a.pool, a.pages, a.max_pages, a.page_rows, a.slot, a.pos,
                           a.sink, a.scale, a.heads, a.rank, a.window, out_cols);
    if (e != cudaSuccess) return (int)e;
    count_launch();
    return (int)cudaGetLastError();
}

// -1: not built for these sizes
static int latent_decode(const b200_latent_attention_args& a, int out_cols, int longest_seen, cudaStream_t s) {
    auto al16 = [](const void* q) { return (reinterpret_cast<uintptr_t>(q) & 15u) == 0; };
    if ((a.rank & 7) || (out_cols & 15) || a.n_tokens > 65535 || !al16(a.qa) || !al16(a.out) || !al16(a.pool)) return -1;
    // as many shares as two CTAs per SM hold at once (clusters of sixteen: one), as long as every CTA keeps a half tile of its own (us at 4 / 8 / 16 shares, 16 heads, rows of 576: 32 sequences of up to 2048
    // 49.1 / 33.8 / 51.1, of up to 700 21.5 / 17.4 / 33.5, 24 of up to 1000 26.3 / 20.0 / 27.9, 16 such 26.3 / 18.9 / 23.3, 8 of up to 1024 28.6 / 19.0 / 16.6, measured with
    // rows by cp.async and weights of one bfloat16; by TMA, in two, this rule's choices take 26.5, 15.2, 16.8, 15.4 and 14.1)
    const long long ctas = (long long)a.n_tokens * ((a.heads + 15) / 16);
    const long long sms = sm_count();
    int splits = 1;
    while (splits < kLdMaxCluster && ctas * splits * 2 <= (splits < 8 ? 2 * sms : sms) && (longest_seen <= 0 ? splits < 8 : splits * kHalfKeys < longest_seen)) splits *= 2;
    const int nt = ((out_cols / 8 + kTileWarps - 1) / kTileWarps + 1) & ~1;
    const bool tma = a.page_rows % kHalfKeys == 0;   // a half tile never straddles two pages
    if (nt <= 2) return tma ? launch_latent_decode<2, true>(a, out_cols, splits, s) : launch_latent_decode<2, false>(a, out_cols, splits, s);
    if (nt <= 4) return tma ? launch_latent_decode<4, true>(a, out_cols, splits, s) : launch_latent_decode<4, false>(a, out_cols, splits, s);
    if (nt <= 8) return tma ? launch_latent_decode<8, true>(a, out_cols, splits, s) : launch_latent_decode<8, false>(a, out_cols, splits, s);
    if (nt <= 10) return tma ? launch_latent_decode<10, true>(a, out_cols, splits, s) : launch_latent_decode<10, false>(a, out_cols, splits, s);
    return -1;
}

static bool tile_attention_enabled() {
    static int v = -1;
    if (v < 0) {
        const char* e = getenv("B200_LATENT_ATTN_SIMT");   // 1: the per-(token, head) kernel for bfloat16 caches too
        v = (e && e[0] == '1') ? 0 : 1;
    }
    return v == 1;
}

// Batches with prompt portions: rows of whole 64-dimension chunks with 256 or 512 columns of output go to the tcgen05 tiles (2048 tokens, 16 heads, rows
// of 576: 180 us there, 856 us on the mma.sync tiles), unless a few rows sit behind long contexts, which only the mma.sync tiles share out. A tcgen05
// CTA takes about 1.8 us per 64 cached rows of a sequence and walks those of its window that fall to it; an mma.sync CTA, two to an SM, takes 7 times
// as long at 512 columns and 5 times at 256, over its share and once per sequence of its rows. Measured, rows of 576, 16 heads, tcgen05 / shared out:
// 2 or 16 tokens behind 8000 rows 255 / 122 us, 64 tokens 254 / 212, 200 tokens behind 4000 147 / 407, 64 behind 1000 51 / 77; 12 single tokens and a
// portion of 16 over 4000 137 / 144, 64 and 256 over 1000 119 / 338; rows of 320 (256 columns), 16 behind a window of 1024 49 / 42, 200 48 / 58.
static bool shares_are_shorter(const b200_latent_attention_args& a, int out_cols, int tokens_per_tile, int splits, int longest_context) {
    if (a.heads > 64) return false;   // not built for the tcgen05 tiles
    const int tiles = (longest_context + kTileKeys - 1) / kTileKeys, share = (tiles + splits - 1) / splits, halves = out_cols > 256 ? 2 : 1;
    const int others = std::max(0, a.n_tokens - a.longest_entry);   // tokens of the other entries
    const int parts = latent_tc_parts(a.n_tokens, a.longest_entry, a.heads, halves), held = std::min(128 / a.heads, others + 1);
    const int walked = others == 0 ? 1 : (held + parts - 1) / parts, walked_here = std::min(tokens_per_tile, others + 1);
    return (halves == 2 ? 7 : 5) * share * walked_here < tiles * walked;
}

}  // namespace b200

using namespace b200;

extern "C" int b200_latent_store(const float* raw, long long ld_raw, const float* w, float eps, void* pool, const int* pages,
                                 int max_pages, int page_rows, const int* slot, const int* pos, int n_tokens, int rank,
                                 int dtype, void* stream) {
    if (!raw || !w || !pool || !pages || !slot || !pos || n_tokens < 0 || rank < 1 || page_rows < 1) return B200_EINVAL;
    if (n_tokens == 0) return B200_OK;
    cudaStream_t s = (cudaStream_t)stream;
    if (dtype == B200_BF16)
        latent_store_kernel<__nv_bfloat16><<<n_tokens, 128, 0, s>>>(raw, ld_raw, w, eps, (__nv_bfloat16*)pool, pages, max_pages,
                                                                   page_rows, slot, pos, rank);
    else if (dtype == B200_F32)
        latent_store_kernel<float><<<n_tokens, 128, 0, s>>>(raw, ld_raw, w, eps, (float*)pool, pages, max_pages, page_rows, slot,
                                                           pos, rank);
    else
        return B200_EINVAL;
    count_launch();
    return (int)cudaGetLastError();
}

extern "C" size_t b200_latent_attention_workspace_bytes(int n_tokens, int heads, int rank) {
    return (size_t)n_tokens * heads * kMaxSplits * (rank + 2) * sizeof(float);
}

extern "C" int b200_latent_store_rot(const float* raw, long long ld_raw, const float* w, float eps, void* pool, const int* pages,
                                     int max_pages, int page_rows, const int* slot, const int* pos, int n_tokens, int rank, int extra,
                                     const float* cos, const float* sin, int rot_layout, int dtype, void* stream) {
    if (!raw || !w || !pool || !pages || !slot || !pos || n_tokens < 0 || rank < 1 || extra < 0 || page_rows < 1) return B200_EINVAL;
    if (extra > 0 && (!cos || !sin || (rot_layout != B200_ROPE_HALF && rot_layout != B200_ROPE_INTERLEAVED))) return B200_EINVAL;
    if (n_tokens == 0) return B200_OK;
    cudaStream_t s = (cudaStream_t)stream;
    if (dtype == B200_BF16)
        latent_store_rot_kernel<__nv_bfloat16><<<n_tokens, 128, 0, s>>>(raw, ld_raw, w, eps, (__nv_bfloat16*)pool, pages, max_pages, page_rows,
                                                                       slot, pos, rank, extra, cos, sin, rot_layout);
    else if (dtype == B200_F32)
        latent_store_rot_kernel<float><<<n_tokens, 128, 0, s>>>(raw, ld_raw, w, eps, (float*)pool, pages, max_pages, page_rows, slot, pos, rank,
                                                               extra, cos, sin, rot_layout);
    else
        return B200_EINVAL;
    count_launch();
    return (int)cudaGetLastError();
}

extern "C" int b200_latent_norms(const b200_latent_norms_args* a, void* stream) {
    if (!a || !a->raw || !a->q_norm || !a->q_out || a->q_rank < 1 || a->n_tokens < 0 || a->q_off < 0) return B200_EINVAL;
    if (a->pool && (!a->kv_norm || !a->pages || !a->slot || !a->pos || a->rank < 1 || a->extra < 0 || a->page_rows < 1 || a->kv_off < 0)) return B200_EINVAL;
    if (a->pool && a->extra > 0 && (!a->cos || !a->sin || (a->rot_layout != B200_ROPE_HALF && a->rot_layout != B200_ROPE_INTERLEAVED))) return B200_EINVAL;
    if (a->n_tokens == 0) return B200_OK;
    const dim3 grid(a->n_tokens, a->pool ? 2 : 1);
    if (a->dtype == B200_BF16) latent_norms_kernel<__nv_bfloat16><<<grid, 128, 0, (cudaStream_t)stream>>>(*a);
    else if (a->dtype == B200_F32) latent_norms_kernel<float><<<grid, 128, 0, (cudaStream_t)stream>>>(*a);
    else return B200_EINVAL;
    count_launch();
    return (int)cudaGetLastError();
}

extern "C" int b200_latent_attention(const float* qa, float* out, const void* pool, const int* pages, int max_pages,
                                     int page_rows, const int* slot, const int* pos, const float* sink, float scale,
                                     int n_tokens, int heads, int rank, int dtype, int longest_entry, int longest_context,
                                     void* workspace, size_t workspace_bytes, void* stream) {
    if (!sink) return B200_EINVAL;
    b200_latent_attention_args a{qa, out, pool, pages, max_pages, page_rows, slot, pos, sink, scale, n_tokens, heads, rank, 0, dtype,
                                 longest_entry, longest_context, workspace, workspace_bytes, 0};
    return b200_latent_attention_ex(&a, stream);
}

extern "C" int b200_latent_attention_ex(const b200_latent_attention_args* ap, void* stream) {
    if (!ap) return B200_EINVAL;
    const float* qa = ap->qa; float* out = ap->out; const void* pool = ap->pool; const int* pages = ap->pages;
    const int max_pages = ap->max_pages, page_rows = ap->page_rows; const int* slot = ap->slot; const int* pos = ap->pos;
    const float* sink = ap->sink; const float scale = ap->scale;
    const int n_tokens = ap->n_tokens, heads = ap->heads, rank = ap->rank, window = ap->window, dtype = ap->dtype, longest_entry = ap->longest_entry;
    const int longest_context = window > 0 && ap->longest_context > 0 ? std::min(ap->longest_context, window + kTileKeys) : ap->longest_context;
    void* workspace = ap->workspace; const size_t workspace_bytes = ap->workspace_bytes;
    const int out_cols = ap->out_cols > 0 && ap->out_cols < rank ? ap->out_cols : rank;
    if (!qa || !out || !pool || !pages || !slot || !pos || n_tokens < 0 || heads < 1 || rank < 1 || window < 0) return B200_EINVAL;
    if (rank > 32 * kMaxRankPerLane || heads > 65535) return B200_EUNSUPPORTED;
    if (n_tokens == 0) return B200_OK;
    cudaStream_t s = (cudaStream_t)stream;
    const size_t smem = ((size_t)5 * rank + 8) * sizeof(float);
    dim3 grid(n_tokens, heads);
    // single tokens: a cluster per token whatever the batch (the tile kernel spends half of its 32 rows on nothing there)
    if (dtype == B200_BF16 && tile_attention_enabled() && longest_entry == 1) {
        const int rc = latent_decode(*ap, out_cols, longest_context, s);
        if (rc >= 0) return rc;
    }
    if (dtype == B200_BF16 && tile_attention_enabled()) {
        // tensor-core form: 32 rows of (token, head) per CTA
        // every entry a single token (a decode batch): one token per CTA, its heads the only rows
        const int HG = heads < kTileRows ? heads : kTileRows, TQ = longest_entry == 1 ? 1 : kTileRows / HG;
        const int rpad = (rank + 15) & ~15, RS = rpad + 8;
        const int single = rpad > 512;   // with one half-tile buffer two CTAs of such rows still fit an SM
        const size_t tsm = (size_t)(kTileRows + (single ? kHalfKeys : kTileKeys)) * RS * 2 + 2 * kTileRows * 36 * 4 + 3 * kTileRows * 4;
        const int ntw = ((((out_cols + 15) & ~15) / 8) + kTileWarps - 1) / kTileWarps;
        dim3 tg((n_tokens + TQ - 1) / TQ, (heads + HG - 1) / HG);
        // few CTAs over long contexts (decoding): shares of the key tiles on blockIdx.z, merged by the combine kernel
        int splits = 1;
        if (longest_context > 0 && workspace) {
            const int tiles = (longest_context + kTileKeys - 1) / kTileKeys;
            const int want = (2 * sm_count()) / (int)(tg.x * tg.y);
            splits = std::max(1, std::min({want, tiles / 2, kMaxSplits}));
            if (workspace_bytes < (size_t)n_tokens * heads * splits * (rank + 2) * sizeof(float)) splits = 1;
        }
        if (longest_entry != 1 && !(splits > 1 && shares_are_shorter(*ap, out_cols, TQ, splits, longest_context))) {
            const int rc = latent_attention_tc(*ap, out_cols, s);
            if (rc >= 0) return rc;
        }
        tg.z = splits;
        float* part = reinterpret_cast<float*>(workspace);
        // every instantiation has the same function type, so the lambda is ONE function: a mask per kernel, not one static
        auto go = [&](auto kern, int which) -> int {
            static unsigned long long done[5] = {0, 0, 0, 0, 0};
            if (tsm > 48 * 1024 && ensure_max_dynamic_smem((const void*)kern, 200 * 1024, done[which]) != cudaSuccess) return B200_EUNSUPPORTED;
            kern<<<tg, 256, tsm, s>>>(qa, out, (const __nv_bfloat16*)pool, pages, max_pages, page_rows, slot, pos, sink, scale, n_tokens,
                                      heads, rank, HG, TQ, splits, part, window, out_cols, single);
            count_launch();
            if (splits > 1) {
                latent_attn_combine_kernel<<<dim3(n_tokens, heads), 128, 0, s>>>(part, out, sink, heads, rank, splits, out_cols);
                count_launch();
            }
            return (int)cudaGetLastError();
        };
        if (ntw <= 1) return go(latent_attn_tile_kernel<1>, 0);
        if (ntw <= 2) return go(latent_attn_tile_kernel<2>, 1);
        if (ntw <= 4) return go(latent_attn_tile_kernel<4>, 2);
        if (ntw <= 8) return go(latent_attn_tile_kernel<8>, 3);
        return go(latent_attn_tile_kernel<10>, 4);
    }
    if (dtype == B200_BF16)
        latent_attn_kernel<__nv_bfloat16><<<grid, 128, smem, s>>>(qa, out, (const __nv_bfloat16*)pool, pages, max_pages, page_rows,
                                                                 slot, pos, sink, scale, heads, rank, window);
    else if (dtype == B200_F32)
        latent_attn_kernel<float><<<grid, 128, smem, s>>>(qa, out, (const float*)pool, pages, max_pages, page_rows, slot, pos,
                                                         sink, scale, heads, rank, window);
    else
        return B200_EINVAL;
    count_launch();
    return (int)cudaGetLastError();
}
