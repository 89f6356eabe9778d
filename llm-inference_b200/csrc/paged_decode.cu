// Single tokens of b200_paged_attention in bfloat16 (decode batches): every (token, key head) is served by one cluster of CTAs that
// share the token's context, one launch, no workspace.
//
// What bounds it: the keys and values, read once (8 KB per 16 keys of 128 x 128), so the kernel has to keep enough of them on their way
// and spend few instructions per byte. A warp walks its own run of keys, 16 at a time, out of a ring of its own in shared memory that
// cp.async fills three steps deep (24 KB per warp, two CTAs of four warps per SM), and never waits for another warp:
//   S^T = K Q^T   mma.sync m16n8k16, keys on the M axis, the R <= 8 query heads of the key head on the N axis
//   softmax       fp32 in registers, a running (maximum, denominator) per warp; cap, bias, temperature and masks as in the row kernel
//   O^T = V^T P^T value dimensions on the M axis (ldmatrix.trans). The weights keep 24 bits: p = hi + mid + lo (three bfloat16, the
//                 difference exact at every step), three products with fp32 accumulation, so nothing is rounded to 16 bits on the way.
//                 movmatrix turns the weights' fragments.
// Warps merge through shared memory, CTAs through distributed shared memory (rank order, so the sum does not depend on timing). The merge
// adds the sink.
// Measured (before: the group kernel of capped_attention.cu with a combine launch): one sequence of 500 tokens, 8 / 4 heads x 128: 20.5 -> 7.1 us;
// 32 sequences of up to 2048 tokens, 16 / 8 heads x 128 (190 MB), bias and sink: 384 -> 59 us (69 us with a step's keys and values in
// registers, requested one step ahead); 128 such sequences without bias run at 5.0 TB/s.
#include <cooperative_groups.h>
#include <cuda_bf16.h>

#include <algorithm>

#include "b200_serve.h"
#include "common.cuh"
#include "launch_count.h"
#include "paged_attention.cuh"

namespace b200 {
namespace cg = cooperative_groups;

constexpr int kPdWarps = 4, kPdStep = 16, kPdHeads = 8, kPdMaxCluster = 8;

template <int D, int VD>
struct PdRing {   // row strides in elements (16 bytes of padding: conflict-free ldmatrix), a step's keys, then its values
    static constexpr int kRS = D + 8, kRSV = VD + 8, kStages = VD > 128 ? 2 : 3;
    static constexpr int kStep = kPdStep * (kRS + kRSV), kWarp = kStages * kStep;   // elements
    static constexpr int kBytes = kPdWarps * kWarp * 2;
};

__device__ __forceinline__ uint32_t pd_transpose(uint32_t v) {   // 8 x 8 tile of 16-bit numbers, a pair per thread
    uint32_t r;
    asm("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(r) : "r"(v));
    return r;
}

// MIXED: a batch that also holds prompt portions, which other kernels take. Cluster z looks after the tokens z, z + gridDim.z, ... and serves
// those that are their sequence's only token in the batch.
template <int D, int VD, bool MIXED>
__global__ void __launch_bounds__(kPdWarps * 32, 2) paged_decode_kernel(const PA a) {
    using bf = __nv_bfloat16;
    using L = PdRing<D, VD>;
    constexpr int KS = D / 16;        // k steps of the scores
    constexpr int MT = VD / 16;       // m tiles of the output
    extern __shared__ __align__(16) float pd_sm[];
    if (!MIXED) {
        pdl_wait();
        pdl_launch_dependents();
    }
    const int R = a.heads / a.kv_heads, splits = gridDim.x;
    float* om = pd_sm;                                 // once the rings have been used: [warps][R][VD], then this CTA's share in the first [R][VD]
    __shared__ float ms[kPdWarps * kPdHeads], ls[kPdWarps * kPdHeads];   // [warps][R], then [R]
    const int ku = blockIdx.y, g = ku / a.maps, mp = ku % a.maps;
    const int warp = threadIdx.x / 32, lane = threadIdx.x % 32, gid = lane >> 2, tig = lane & 3;
    const int k_units = a.kv_heads * a.maps, q_units = a.heads * a.maps;
    const bf* K = reinterpret_cast<const bf*>(a.k_pool) + (size_t)ku * D;
    const bf* V = reinterpret_cast<const bf*>(a.v_pool) + (size_t)g * VD;
    bf* ring = reinterpret_cast<bf*>(pd_sm) + warp * L::kWarp;
    const size_t k_row = (size_t)k_units * D, v_row = (size_t)a.kv_heads * VD;

    // this thread's two heads (columns of S^T and O^T)
    float sc[2], hb[2];
    const float over_cap = a.softcap > 0.f ? 1.f / a.softcap : 0.f;
    const float* bias[2];
#pragma unroll
    for (int x = 0; x < 2; ++x) {
        const int h = min(g * R + 2 * tig + x, a.heads - 1);
        sc[x] = pa_scale(a, h);
        hb[x] = (a.sigmoid && a.head_bias) ? a.head_bias[h] : 0.f;
        bias[x] = a.dist_bias ? a.dist_bias + (size_t)h * a.dist_n : nullptr;
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
            auto fetch = [&](int s) {   // step s into its stage; keys that the token does not see arrive as zeros (their rows may hold anything)
                bf* dst = ring + (s - s0) % L::kStages * L::kStep;
                const size_t row0 = (size_t)page * a.page_rows + off;
                const int j = first + s * kPdStep;
#pragma unroll
                for (int i = 0; i < kPdStep * (D / 8) / 32; ++i) {
                    const int at = i * 32 + lane, r = at / (D / 8), c = at % (D / 8) * 8;
                    const uint32_t to = (uint32_t)__cvta_generic_to_shared(dst + r * L::kRS + c);
                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(to), "l"(K + (row0 + r) * k_row + c), "r"(j + r >= j_lo && j + r <= p ? 16 : 0) : "memory");
                }
                dst += kPdStep * L::kRS;
#pragma unroll
                for (int i = 0; i < kPdStep * (VD / 8) / 32; ++i) {
                    const int at = i * 32 + lane, r = at / (VD / 8), c = at % (VD / 8) * 8;
                    const uint32_t to = (uint32_t)__cvta_generic_to_shared(dst + r * L::kRSV + c);
                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(to), "l"(V + (row0 + r) * v_row + c), "r"(j + r >= j_lo && j + r <= p ? 16 : 0) : "memory");
                }
                off += kPdStep;   // the page of the step after is looked up now
                if (off == a.page_rows) { off = 0; ++page_at; if (s + 1 < s1) page = plist[page_at]; }
            };
            auto close_group = [&]() {
                __syncwarp();   // the lanes close their group of copies together
                asm volatile("cp.async.commit_group;" ::: "memory");
            };
#pragma unroll
            for (int i = 0; i < L::kStages - 1; ++i) {
                if (s0 + i < s1) fetch(s0 + i);
                close_group();
            }
            for (int s = s0; s < s1; ++s, j0 += kPdStep) {
                const bool whole = j0 >= j_lo && j0 + kPdStep - 1 <= p;
                if (s + L::kStages - 1 < s1) fetch(s + L::kStages - 1);
                close_group();
                asm volatile("cp.async.wait_group %0;" ::"n"(L::kStages - 1) : "memory");
                __syncwarp();   // step s has landed for every lane
                const bf* Ks = ring + (s - s0) % L::kStages * L::kStep;
                const bf* Vs = Ks + kPdStep * L::kRS;
                float bv[4] = {0.f, 0.f, 0.f, 0.f};
                if (a.dist_bias) {   // requested before the scores are formed
#pragma unroll
                    for (int e = 0; e < 4; ++e) bv[e] = bias[e & 1][min(max(p - (j0 + gid + (e >> 1) * 8), 0), a.dist_n - 1)];
                }
                float st[4] = {0.f, 0.f, 0.f, 0.f}, su[4] = {0.f, 0.f, 0.f, 0.f};   // two chains of products
#pragma unroll
                for (int ks = 0; ks < KS; ks += 2) {
                    uint32_t k0[4], k1[4];
                    pa_ldsm_x4(k0, Ks + (lane & 15) * L::kRS + (lane >> 4) * 8 + ks * 16);
                    pa_ldsm_x4(k1, Ks + (lane & 15) * L::kRS + (lane >> 4) * 8 + ks * 16 + 16);
                    pa_mma(st, k0, qf[ks]);
                    pa_mma(su, k1, qf[ks + 1]);
                }
#pragma unroll
                for (int e = 0; e < 4; ++e) st[e] = (st[e] + su[e]) * sc[e & 1];
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
                for (int e = 0; e < 4; ++e) {   // key j0 + gid (+ 8), head 2 tig (+ 1)
                    const int j = j0 + gid + (e >> 1) * 8;
                    pr[e] = whole || (j >= j_lo && j <= p) ? st[e] + bv[e] : -INFINITY;
                }
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
#pragma unroll
                for (int j = 0; j < MT; j += 4) {   // four tiles of 16 dimensions at a time: consecutive products feed different sums
                    uint32_t af[4][4];
#pragma unroll
                    for (int e = 0; e < 4; ++e) pa_ldsm_x4_trans(af[e], Vs + ((lane & 7) + (lane >> 4) * 8) * L::kRSV + (j + e) * 16 + ((lane >> 3) & 1) * 8);
#pragma unroll
                    for (int q = 2; q >= 0; --q)
#pragma unroll
                        for (int e = 0; e < 4; ++e) pa_mma(o[j + e], af[e], b[q]);
                }
                __syncwarp();   // the stage may be filled again
            }
            asm volatile("cp.async.wait_group 0;" ::: "memory");
            __syncthreads();    // the rings' place is taken by the sums
#pragma unroll
            for (int x = 0; x < 2; ++x) {
                l[x] += __shfl_xor_sync(0xffffffffu, l[x], 4);
                l[x] += __shfl_xor_sync(0xffffffffu, l[x], 8);
                l[x] += __shfl_xor_sync(0xffffffffu, l[x], 16);
                const int h = 2 * tig + x;
                if (h < R) {
                    if (gid == 0) { ms[warp * R + h] = m[x]; ls[warp * R + h] = l[x]; }
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
            cluster.sync();   // nobody leaves (or starts its next token) while its shared memory is read
        }
        if (!MIXED) break;
    }
    if (MIXED) pdl_wait();   // the prompt portions' kernel runs beside this one: done only when both are
}

template <int D, int VD, bool MIXED>
static int launch_paged_decode(const PA& a, int splits, int rows, cudaStream_t s) {
    constexpr int smem = PdRing<D, VD>::kBytes;
    static_assert(kPdWarps * kPdHeads * VD * 4 <= smem, "the warps' sums take the rings' place");
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
    e = cudaLaunchKernelEx(&cfg, paged_decode_kernel<D, VD, MIXED>, a);
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

int paged_decode(const PA& a, int longest_seen, bool mixed, cudaStream_t s) {
    if (a.heads / a.kv_heads > kPdHeads || a.page_rows % kPdStep || a.kv_heads * a.maps > 65535) return -1;
    // how many tokens of a mixed batch are single ones is only known on the device: sixteen rows of clusters share them
    const int rows = mixed ? std::min(a.n_tokens, 16) : a.n_tokens;
    if (rows > 65535) return -1;
    // three CTAs for every two SMs, as long as every warp of a cluster keeps a step of its own (32 sequences of up to 2048 tokens, 16 / 8
    // heads: 256 / 512 / 1024 CTAs 49 / 51 / 63 us; 8 of up to 1024: 256 / 512 CTAs 14.5 / 20.6 us)
    const long long pairs = (long long)rows * a.kv_heads * a.maps;
    const int most = mixed ? 4 : kPdMaxCluster;
    int splits = 1;
    while (splits < most && (mixed || 2 * pairs * splits < 3ll * sm_count()) && (longest_seen <= 0 || splits * kPdWarps * kPdStep < longest_seen)) splits *= 2;
    return mixed ? paged_decode_for<true>(a, splits, rows, s) : paged_decode_for<false>(a, splits, rows, s);
}

}  // namespace b200
