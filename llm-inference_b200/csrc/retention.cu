// Retention (linear attention with a fixed decay per head and a carried state, no softmax) and the unit-RMS output gate (which
// can carry a weight and a sigmoid instead of the silu).
// Everything here is fp32: the rotated q and k, the state, the decays and the sums.
//
//   retention_walk_kernel   one CTA per (entry, head, group of value columns): a thread owns one column of the state
//                           S[:, c] in registers and walks the entry's tokens in order, S <- decay S + k_t v_t[c],
//                           out[t, c] = <S[:, c], q_t>. Columns are independent, so no thread waits on another inside a
//                           token; q_t and k_t are rotated and staged in shared memory eight tokens at a time.
//                           Decode batches and short portions take this path.
//   chunk form (entries of 128 tokens and more): the same recurrence regrouped over chunks of 64 tokens, three launches:
//     retention_chunk_state_kernel   U_c = sum_j decay^(L-1-j) k_j v_j^T of every chunk, chunks in parallel;
//     retention_chunk_scan_kernel    S at the start of every chunk, S_(c+1) = decay^L S_c + U_c, element-wise, and the
//                                    state the entry leaves behind;
//     retention_chunk_out_kernel     out_i = decay^(i+1) S_c^T q_i + sum_(j<=i) decay^(i-j) (q_i . k_j) v_j, chunks in parallel.
//   The same sums in another order: results agree with the walk to fp32 rounding.
#include <math.h>
#include <stdlib.h>

#include "b200_serve.h"
#include "common.cuh"
#include "launch_count.h"
#include "rotary.cuh"
#include "tc_common.cuh"

namespace b200 {

struct RT {
    const float* proj; long long ld_proj; int q_off, k_off, v_off;
    const float* cos; const float* sin; int rot_dims, rot_layout;
    const float* decay; float k_scale;
    float* state; float* out;
    const int* ent_row; const int* ent_len; const int* slot; const int* pos;
    int heads, dim, vdim;
};

constexpr int kWalkTokens = 8;   // tokens whose q / k are staged per synchronisation

template <int DIM>
__global__ void __launch_bounds__(128) retention_walk_kernel(const RT a) {
    pdl_wait();
    pdl_launch_dependents();
    extern __shared__ float sm[];
    const int dim = a.dim;
    float* raw = sm;                              // [2][dim] un-rotated q, k of the token being staged
    float* rq = sm + 2 * dim;                     // [kWalkTokens][dim]
    float* rk = rq + kWalkTokens * dim;           // [kWalkTokens][dim]
    const int e = blockIdx.x, h = blockIdx.y, c = blockIdx.z * blockDim.x + threadIdx.x;
    const int row0 = a.ent_row[e], n = a.ent_len[e], b = a.slot[row0], p0 = a.pos[row0];
    const bool live = c < a.vdim;
    const float decay = a.decay[h];
    float S[DIM];
    float* sp = a.state + (((size_t)b * a.heads + h) * dim) * a.vdim + c;
#pragma unroll
    for (int d = 0; d < DIM; ++d) S[d] = (live && d < dim && p0 > 0) ? sp[(size_t)d * a.vdim] : 0.f;
    const int nf = a.rot_dims / 2;
    for (int t0 = 0; t0 < n; t0 += kWalkTokens) {
        const int nt = min(kWalkTokens, n - t0);
        for (int k = 0; k < nt; ++k) {
            const size_t r = (size_t)(row0 + t0 + k);
            __syncthreads();   // raw (and, for k = 0, rq / rk of the previous group) are free
            for (int i = threadIdx.x; i < 2 * dim; i += blockDim.x)
                raw[i] = a.proj[r * a.ld_proj + (i < dim ? a.q_off + h * dim + i : a.k_off + h * dim + (i - dim))];
            __syncthreads();
            for (int i = threadIdx.x; i < 2 * dim; i += blockDim.x) {
                const bool is_k = i >= dim;
                const int d = is_k ? i - dim : i;
                const float v = rotary_component(raw + (is_k ? dim : 0), d, a.rot_dims, a.rot_layout, a.cos + r * nf, a.sin + r * nf);
                if (is_k) rk[k * dim + d] = v * a.k_scale;
                else rq[k * dim + d] = v;
            }
        }
        __syncthreads();
        if (live) {
            for (int k = 0; k < nt; ++k) {
                const size_t r = (size_t)(row0 + t0 + k);
                const float v = a.proj[r * a.ld_proj + a.v_off + h * a.vdim + c];
                float acc = 0.f;
#pragma unroll
                for (int d = 0; d < DIM; ++d)
                    if (d < dim) {
                        S[d] = fmaf(decay, S[d], rk[k * dim + d] * v);
                        acc = fmaf(S[d], rq[k * dim + d], acc);
                    }
                a.out[r * ((size_t)a.heads * a.vdim) + h * a.vdim + c] = acc;
            }
        }
    }
    if (live) {
#pragma unroll
        for (int d = 0; d < DIM; ++d)
            if (d < dim) sp[(size_t)d * a.vdim] = S[d];
    }
}


// ---------------------------------------------------------------------------------------------------------------
// chunk form
// ---------------------------------------------------------------------------------------------------------------
constexpr int kChunk = 64, kColsPerThread = 2, kChunkCols = 64 * kColsPerThread;   // a thread owns columns c, c + 64

struct RC {
    RT a;
    float* chunk_state;   // [chunk slot, head, dim, vdim]; slot of chunk c of entry e = ent_row[e] / kChunk + e + c
    int col_blocks;       // blocks of kChunkCols value columns; blockIdx.x = entry * col_blocks + column block
};

__host__ __device__ __forceinline__ int chunk_row_stride(int dim) { return ((dim + 3) & ~3) + 4; }   // floats; rows stay 16-byte aligned

// rotated q (or k * k_scale * weight[j]) of a chunk into shared memory: TRANS false: [token][rs], the padding columns zero; true: [component][kChunkT].
// A warp takes two tokens at a time and four components per lane of each, all their loads at once (and none behind a condition: such a load waits for the one
// before it, which is what a chunk's 64 tokens spent most of their time on).
constexpr int kChunkT = kChunk + 4;
template <bool TRANS>
__device__ __forceinline__ void stage_rotated_wide(const RT& a, float* dst, int col_off, int h, int row0, int len, float mul, const float* rowmul) {
    const int dim = a.dim, nf = a.rot_dims / 2, rs = chunk_row_stride(dim), lane = threadIdx.x & 31, warps = blockDim.x / 32;
    const bool halves = a.rot_layout == B200_ROPE_HALF;
    const float *cosines = nf > 0 ? a.cos : a.decay, *sines = nf > 0 ? a.sin : a.decay;   // (without rotation something that can be read)
    for (int d0 = lane; d0 < dim; d0 += 128) {
        int lo[4], hi[4], f[4];
        bool rot[4], first[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {   // the pair of component d and its place in it
            const int d = min(d0 + 32 * k, dim - 1);
            rot[k] = d < a.rot_dims;
            first[k] = halves ? d < nf : (d & 1) == 0;
            f[k] = !rot[k] ? 0 : halves ? (d < nf ? d : d - nf) : d / 2;
            lo[k] = !rot[k] ? d : halves ? f[k] : 2 * f[k];
            hi[k] = !rot[k] ? d : halves ? f[k] + nf : 2 * f[k] + 1;
        }
#pragma unroll 1
        for (int j0 = threadIdx.x / 32; j0 < len; j0 += 2 * warps) {
            float u[2][4], v[2][4], cs[2][4], sn[2][4];
#pragma unroll
            for (int t = 0; t < 2; ++t) {
                const size_t r = (size_t)(row0 + min(j0 + t * warps, len - 1));
                const float *vals = a.proj + r * a.ld_proj + col_off + h * dim, *c = cosines + r * nf, *s = sines + r * nf;
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    u[t][k] = vals[lo[k]];
                    v[t][k] = vals[hi[k]];
                    cs[t][k] = __ldg(c + f[k]);
                    sn[t][k] = __ldg(s + f[k]);
                }
            }
#pragma unroll
            for (int t = 0; t < 2; ++t) {
                const int j = j0 + t * warps;
                const float w = rowmul ? rowmul[min(j, len - 1)] : 1.f;
                float* to = dst + (TRANS ? d0 * kChunkT + j : j * rs + d0);
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    float x = first[k] ? u[t][k] * cs[t][k] - v[t][k] * sn[t][k] : v[t][k] * cs[t][k] + u[t][k] * sn[t][k];
                    if (!rot[k]) x = u[t][k];
                    if (j < len && d0 + 32 * k < dim) to[TRANS ? 32 * k * kChunkT : 32 * k] = x * mul * w;
                }
            }
        }
    }
    if (!TRANS)
        for (int i = threadIdx.x; i < len * (rs - dim); i += blockDim.x) dst[i / (rs - dim) * rs + dim + i % (rs - dim)] = 0.f;
}

// the same for up to 32 components, where most lanes of the above would have none: a thread per number, four at a time (and the state kernel with value rows four
// at a time, in 64 registers instead of 92, so that four CTAs share an SM: 2048 tokens, 16 heads of 4 x 4 60 -> 39 us, of 16 x 32 69 -> 46)
template <bool TRANS>
__device__ __forceinline__ void stage_rotated_narrow(const RT& a, float* dst, int col_off, int h, int row0, int len, float mul, const float* rowmul) {
    const int dim = a.dim, nf = a.rot_dims / 2, rs = chunk_row_stride(dim), step = blockDim.x;
    const bool halves = a.rot_layout == B200_ROPE_HALF;
    const float *cosines = nf > 0 ? a.cos : a.decay, *sines = nf > 0 ? a.sin : a.decay;
#pragma unroll 1
    for (int i0 = threadIdx.x; i0 < len * dim; i0 += 4 * step) {
        float u[4], v[4], cs[4], sn[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int i = min(i0 + k * step, len * dim - 1), j = i / dim, d = i - j * dim;
            const bool rot = d < a.rot_dims;
            const int f = !rot ? 0 : halves ? (d < nf ? d : d - nf) : d / 2;
            const size_t r = (size_t)(row0 + j);
            const float* vals = a.proj + r * a.ld_proj + col_off + h * dim;
            u[k] = vals[!rot ? d : halves ? f : 2 * f];
            v[k] = vals[!rot ? d : halves ? f + nf : 2 * f + 1];
            cs[k] = __ldg(cosines + r * nf + f);
            sn[k] = __ldg(sines + r * nf + f);
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int i = i0 + k * step, j = i / dim, d = i - j * dim;
            float x = (halves ? d < nf : (d & 1) == 0) ? u[k] * cs[k] - v[k] * sn[k] : v[k] * cs[k] + u[k] * sn[k];
            if (d >= a.rot_dims) x = u[k];
            if (i < len * dim) dst[TRANS ? d * kChunkT + j : j * rs + d] = x * mul * (rowmul ? rowmul[j] : 1.f);
        }
    }
    if (!TRANS)
        for (int i = threadIdx.x; i < len * (rs - dim); i += blockDim.x) dst[i / (rs - dim) * rs + dim + i % (rs - dim)] = 0.f;
}
template <bool TRANS, bool NARROW>
__device__ __forceinline__ void stage_rotated(const RT& a, float* dst, int col_off, int h, int row0, int len, float mul, const float* rowmul) {
    if constexpr (NARROW) stage_rotated_narrow<TRANS>(a, dst, col_off, h, row0, len, mul, rowmul);
    else stage_rotated_wide<TRANS>(a, dst, col_off, h, row0, len, mul, rowmul);
}

// What bounds these kernels is fp32 arithmetic (two columns and NACC rows of the state per thread: NACC packed products of two per 16-byte read of Kw), once the
// loads come in groups. 4 entries of 312 to 512 tokens, 4 heads of 128 x 256: 68 us with a load per token and column, one behind the other, 34 now.
template <int NACC, bool FULL>   // accumulators per thread (a multiple of 4): dim <= 4 * NACC, FULL: equal
__global__ void __launch_bounds__(256, NACC == 8 ? 4 : 1) retention_chunk_state_kernel(const RC rc) {
    pdl_wait();
    pdl_launch_dependents();
    extern __shared__ __align__(16) float sm[];
    const RT& a = rc.a;
    const int e = blockIdx.x / rc.col_blocks, cb = blockIdx.x % rc.col_blocks;
    const int c_in = blockIdx.y, h = blockIdx.z;
    const int row_e = a.ent_row[e], n = a.ent_len[e];
    if (c_in * kChunk >= n) return;
    const int row0 = row_e + c_in * kChunk, len = min(kChunk, n - c_in * kChunk), dim = a.dim, rs = chunk_row_stride(dim);
    float* Kw = sm;                  // [kChunk][rs], row j weighted by decay^(len-1-j)
    float* pw = sm + kChunk * rs;    // [kChunk]
    const float decay = a.decay[h];
    for (int j = threadIdx.x; j < len; j += blockDim.x) pw[j] = powf(decay, (float)(len - 1 - j));
    __syncthreads();
    stage_rotated<false, NACC == 8>(a, Kw, a.k_off, h, row0, len, a.k_scale, pw);
    __syncthreads();
    // thread: kColsPerThread value columns, NACC consecutive rows of the state (read from shared memory four at a time)
    const int c = cb * kChunkCols + (threadIdx.x & 63), d0 = (threadIdx.x >> 6) * NACC, dpad = (dim + 3) & ~3;
    uint64_t acc[kColsPerThread][NACC / 2];
#pragma unroll
    for (int q = 0; q < kColsPerThread; ++q)
#pragma unroll
        for (int k = 0; k < NACC / 2; ++k) acc[q][k] = 0ull;
    if (c < a.vdim && d0 < dim) {
        const float* vcol = a.proj + (size_t)row0 * a.ld_proj + a.v_off + h * a.vdim + c;
        constexpr int J = NACC == 8 ? 4 : 8;
        int off[kColsPerThread];
#pragma unroll
        for (int q = 0; q < kColsPerThread; ++q) off[q] = c + 64 * q < a.vdim ? 64 * q : 0;
        auto load = [&](int j0, float (&v)[J][kColsPerThread]) {
#pragma unroll
            for (int x = 0; x < J; ++x)
#pragma unroll
                for (int q = 0; q < kColsPerThread; ++q) v[x][q] = vcol[(size_t)min(j0 + x, len - 1) * a.ld_proj + off[q]];
        };
        auto product = [&](int j, const float (&v)[kColsPerThread]) {
            uint64_t v2[kColsPerThread];
#pragma unroll
            for (int q = 0; q < kColsPerThread; ++q) v2[q] = pack2f(v[q], v[q]);
            const float* kr = Kw + j * rs + d0;
#pragma unroll
            for (int k = 0; k < NACC; k += 4)
                if (FULL || d0 + k < dpad) {
                    const ulonglong2 k4 = *reinterpret_cast<const ulonglong2*>(kr + k);
#pragma unroll
                    for (int q = 0; q < kColsPerThread; ++q) {
                        acc[q][k / 2] = fma2(k4.x, v2[q], acc[q][k / 2]);
                        acc[q][k / 2 + 1] = fma2(k4.y, v2[q], acc[q][k / 2 + 1]);
                    }
                }
        };
        float v[J][kColsPerThread], next[J][kColsPerThread];
        load(0, next);
        int j0 = 0;
        for (; j0 + J <= len; j0 += J) {
#pragma unroll
            for (int x = 0; x < J; ++x)
#pragma unroll
                for (int q = 0; q < kColsPerThread; ++q) v[x][q] = next[x][q];
            load(j0 + J, next);
#pragma unroll
            for (int x = 0; x < J; ++x) product(j0 + x, v[x]);
        }
#pragma unroll
        for (int x = 0; x < J; ++x)
            if (j0 + x < len) product(j0 + x, next[x]);
        float* U = rc.chunk_state + (((size_t)(row_e / kChunk + e + c_in) * a.heads + h) * dim) * a.vdim + c;
#pragma unroll
        for (int q = 0; q < kColsPerThread; ++q)
            if (c + 64 * q < a.vdim)
#pragma unroll
                for (int k = 0; k < NACC; k += 2) {
                    float lo, hi;
                    unpack2(acc[q][k / 2], lo, hi);
                    if (d0 + k < dim) U[(size_t)(d0 + k) * a.vdim + 64 * q] = lo;
                    if (d0 + k + 1 < dim) U[(size_t)(d0 + k + 1) * a.vdim + 64 * q] = hi;
                }
    }
}

// element-wise over (dim, vdim), VEC consecutive elements per thread: walks the entry's chunks, leaves S at each chunk's start in place of its U
__device__ __forceinline__ float retention_next(float S, float d, float u) { return fmaf(d, S, u); }
__device__ __forceinline__ float4 retention_next(float4 S, float d, float4 u) { return make_float4(fmaf(d, S.x, u.x), fmaf(d, S.y, u.y), fmaf(d, S.z, u.z), fmaf(d, S.w, u.w)); }
template <typename V>
__global__ void __launch_bounds__(256) retention_chunk_scan_kernel(const RC rc) {
    pdl_wait();
    pdl_launch_dependents();
    const RT& a = rc.a;
    const int e = blockIdx.x, h = blockIdx.y, i = blockIdx.z * blockDim.x + threadIdx.x;
    const int per = a.dim * a.vdim / (int)(sizeof(V) / 4);
    if (i >= per) return;
    const int row_e = a.ent_row[e], n = a.ent_len[e], b = a.slot[row_e], p0 = a.pos[row_e];
    const float decay = a.decay[h];
    V* sp = reinterpret_cast<V*>(a.state) + ((size_t)b * a.heads + h) * per + i;
    V S{};
    if (p0 > 0) S = *sp;
    const int chunks = (n + kChunk - 1) / kChunk;
    const float full = powf(decay, (float)kChunk), tail = powf(decay, (float)(n - (chunks - 1) * kChunk));
    V* U = reinterpret_cast<V*>(rc.chunk_state) + ((size_t)(row_e / kChunk + e) * a.heads + h) * per + i;
    const size_t step = (size_t)a.heads * per;
    for (int c0 = 0; c0 < chunks; c0 += 8) {   // eight loads in flight, then the dependent chain
        V u[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) u[k] = __ldcg(U + (size_t)min(c0 + k, chunks - 1) * step);   // (behind a condition each would wait for the one before)
#pragma unroll
        for (int k = 0; k < 8; ++k)
            if (c0 + k < chunks) {
                U[(size_t)(c0 + k) * step] = S;
                S = retention_next(S, c0 + k + 1 < chunks ? full : tail, u[k]);
            }
    }
    *sp = S;
}

// Thread: columns c, c + 64; sixteen consecutive rows, two per packed product (q and A lie transposed: a 16-byte read is four rows of one j or component).
template <bool NARROW>
__global__ void __launch_bounds__(256, 2) retention_chunk_out_kernel(const RC rc) {
    pdl_wait();
    pdl_launch_dependents();
    extern __shared__ __align__(16) float sm[];
    const RT& a = rc.a;
    const int e = blockIdx.x / rc.col_blocks, cb = blockIdx.x % rc.col_blocks;
    const int c_in = blockIdx.y, h = blockIdx.z;
    const int row_e = a.ent_row[e], n = a.ent_len[e];
    if (c_in * kChunk >= n) return;
    const int row0 = row_e + c_in * kChunk, len = min(kChunk, n - c_in * kChunk), dim = a.dim;
    float* Qt = sm;                               // [dim][kChunkT]
    float* Kt = Qt + dim * kChunkT;               // [dim][kChunkT]
    float* At = Kt + dim * kChunkT;               // [j][kChunkT]: row i of A at At[j][i]
    float* pw = At + kChunk * kChunkT;            // [kChunk + 1]: decay^k
    const float decay = a.decay[h];
    for (int k = threadIdx.x; k <= kChunk; k += blockDim.x) pw[k] = powf(decay, (float)k);
    if (len < kChunk)   // rows and columns behind the entry: the tiles below read them
        for (int i = threadIdx.x; i < 2 * dim * (kChunk - len); i += blockDim.x) Qt[i / (kChunk - len) * kChunkT + len + i % (kChunk - len)] = 0.f;
    stage_rotated<true, NARROW>(a, Qt, a.q_off, h, row0, len, 1.f, nullptr);
    stage_rotated<true, NARROW>(a, Kt, a.k_off, h, row0, len, a.k_scale, nullptr);
    __syncthreads();
    {   // q . k in tiles of four rows and four columns
        const int ti = threadIdx.x >> 4, tj = threadIdx.x & 15;
        uint64_t t[4][2];   // [column][row pair]
#pragma unroll
        for (int y = 0; y < 4; ++y) t[y][0] = t[y][1] = 0ull;
        if (tj <= ti)
#pragma unroll 4
            for (int d = 0; d < dim; ++d) {
                const ulonglong2 q4 = *reinterpret_cast<const ulonglong2*>(Qt + d * kChunkT + ti * 4);
                const float4 k4 = *reinterpret_cast<const float4*>(Kt + d * kChunkT + tj * 4);
                const float kk[4] = {k4.x, k4.y, k4.z, k4.w};
#pragma unroll
                for (int y = 0; y < 4; ++y) {
                    const uint64_t k2 = pack2f(kk[y], kk[y]);
                    t[y][0] = fma2(q4.x, k2, t[y][0]);
                    t[y][1] = fma2(q4.y, k2, t[y][1]);
                }
            }
#pragma unroll
        for (int y = 0; y < 4; ++y) {
            float f[4];
            unpack2(t[y][0], f[0], f[1]);
            unpack2(t[y][1], f[2], f[3]);
            const int jj = tj * 4 + y;
#pragma unroll
            for (int x = 0; x < 4; ++x) {
                const int i = ti * 4 + x;
                f[x] = jj <= i && i < len ? f[x] * pw[i - jj] : 0.f;
            }
            *reinterpret_cast<float4*>(At + jj * kChunkT + ti * 4) = make_float4(f[0], f[1], f[2], f[3]);
        }
    }
    __syncthreads();
    const int c = cb * kChunkCols + (threadIdx.x & 63), r0 = (threadIdx.x >> 6) * 16;
    if (c >= a.vdim || r0 >= len) return;
    constexpr int CP = kColsPerThread, J = 8;
    uint64_t acc[CP][8], cross[CP][8];
#pragma unroll
    for (int q = 0; q < CP; ++q)
#pragma unroll
        for (int k = 0; k < 8; ++k) acc[q][k] = cross[q][k] = 0ull;
    int off[CP];
#pragma unroll
    for (int q = 0; q < CP; ++q) off[q] = c + 64 * q < a.vdim ? 64 * q : 0;
    // `rows` rows of `src` (leading dimension ld), eight at a time ahead of the eight in use, times the sixteen of m
    auto products = [&](const float* src, long long ld, int rows, const float* m, uint64_t (&to)[CP][8]) {
        float v[J][CP], next[J][CP];
        auto load = [&](int at, float (&x)[J][CP]) {
#pragma unroll
            for (int y = 0; y < J; ++y)
#pragma unroll
                for (int q = 0; q < CP; ++q) x[y][q] = src[(size_t)min(at + y, rows - 1) * ld + off[q]];
        };
        auto product = [&](int at, const float (&x)[CP]) {
            uint64_t v2[CP];
#pragma unroll
            for (int q = 0; q < CP; ++q) v2[q] = pack2f(x[q], x[q]);
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const ulonglong2 m4 = *reinterpret_cast<const ulonglong2*>(m + at * kChunkT + r0 + 4 * k);
#pragma unroll
                for (int q = 0; q < CP; ++q) {
                    to[q][2 * k] = fma2(m4.x, v2[q], to[q][2 * k]);
                    to[q][2 * k + 1] = fma2(m4.y, v2[q], to[q][2 * k + 1]);
                }
            }
        };
        load(0, next);
        int at = 0;
        for (; at + J <= rows; at += J) {
#pragma unroll
            for (int y = 0; y < J; ++y)
#pragma unroll
                for (int q = 0; q < CP; ++q) v[y][q] = next[y][q];
            load(at + J, next);
#pragma unroll
            for (int y = 0; y < J; ++y) product(at + y, v[y]);
        }
#pragma unroll
        for (int y = 0; y < J; ++y)
            if (at + y < rows) product(at + y, next[y]);
    };
    products(a.proj + (size_t)row0 * a.ld_proj + a.v_off + h * a.vdim + c, a.ld_proj, min(len, r0 + 16), At, acc);
    products(rc.chunk_state + (((size_t)(row_e / kChunk + e + c_in) * a.heads + h) * dim) * a.vdim + c, a.vdim, dim, Qt, cross);
#pragma unroll
    for (int q = 0; q < CP; ++q)
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            float x[2], y[2];
            unpack2(cross[q][k], x[0], x[1]);
            unpack2(acc[q][k], y[0], y[1]);
#pragma unroll
            for (int z = 0; z < 2; ++z) {
                const int i = r0 + 2 * k + z;
                if (i < len && c + 64 * q < a.vdim) a.out[(size_t)(row0 + i) * ((size_t)a.heads * a.vdim) + h * a.vdim + c + 64 * q] = fmaf(pw[i + 1], x[z], y[z]);
            }
        }
}

// one warp per (token, head); w [heads, vdim] may be NULL; the gate is silu(z) or (SIG) sigmoid(z)
template <typename T, bool SIG>
__global__ void unit_rms_gate_kernel(const float* __restrict__ o, const float* __restrict__ gate, long long ld_gate, const float* __restrict__ w,
                                     T* __restrict__ out, int units, int heads, int vdim, float eps) {
    pdl_wait();
    pdl_launch_dependents();
    const int u = blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32, lane = threadIdx.x % 32;
    if (u >= units) return;
    const int t = u / heads, h = u % heads;
    const float* src = o + (size_t)u * vdim;
    float ss = 0.f;
    for (int i = lane; i < vdim; i += 32) ss += src[i] * src[i];
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, d);
    const float rinv = 1.0f / sqrtf(ss / (float)vdim + eps);
    const float* g = gate + (size_t)t * ld_gate + (size_t)h * vdim;
    for (int i = lane; i < vdim; i += 32) {
        const float z = g[i];
        const float v = w ? src[i] * rinv * w[(size_t)h * vdim + i] : src[i] * rinv;
        out[(size_t)u * vdim + i] = DT<T>::from_f(v * ((SIG ? 1.f : z) / (1.f + expf(-z))));
    }
}

// the same for heads in whole groups of four columns, at most 4 * 32 * PER of them: loads in flight together, the head in registers
template <typename T, bool SIG, int PER>
__global__ void __launch_bounds__(128) unit_rms_gate_reg_kernel(const float* __restrict__ o, const float* __restrict__ gate, long long ld_gate,
                                                                const float* __restrict__ w, T* __restrict__ out, int units, int heads, int vdim,
                                                                float eps) {
    pdl_wait();
    pdl_launch_dependents();
    const int u = blockIdx.x * 4 + threadIdx.x / 32, lane = threadIdx.x % 32, quads = vdim / 4;
    if (u >= units) return;
    const int t = u / heads, h = u % heads;
    const float4* src = reinterpret_cast<const float4*>(o + (size_t)u * vdim);
    const float4* g = reinterpret_cast<const float4*>(gate + (size_t)t * ld_gate + (size_t)h * vdim);
    const float4* wp = reinterpret_cast<const float4*>(w + (size_t)h * vdim);
    float4 v[PER], z[PER], wv[PER];
    float ss = 0.f;
#pragma unroll
    for (int k = 0; k < PER; ++k) {
        const int c = lane + 32 * k;
        v[k] = z[k] = make_float4(0.f, 0.f, 0.f, 0.f);
        wv[k] = make_float4(1.f, 1.f, 1.f, 1.f);
        if (c < quads) {
            v[k] = src[c];
            z[k] = g[c];
            if (w) wv[k] = wp[c];
        }
        ss += v[k].x * v[k].x + v[k].y * v[k].y + v[k].z * v[k].z + v[k].w * v[k].w;
    }
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, d);
    const float rinv = 1.0f / sqrtf(ss / (float)vdim + eps);
    T* dst = out + (size_t)u * vdim;
#pragma unroll
    for (int k = 0; k < PER; ++k) {
        const int c = lane + 32 * k;
        if (c >= quads) continue;
        const float f[4] = {v[k].x * rinv * wv[k].x * ((SIG ? 1.f : z[k].x) / (1.f + expf(-z[k].x))), v[k].y * rinv * wv[k].y * ((SIG ? 1.f : z[k].y) / (1.f + expf(-z[k].y))),
                            v[k].z * rinv * wv[k].z * ((SIG ? 1.f : z[k].z) / (1.f + expf(-z[k].z))), v[k].w * rinv * wv[k].w * ((SIG ? 1.f : z[k].w) / (1.f + expf(-z[k].w)))};
        if constexpr (sizeof(T) == 4) reinterpret_cast<float4*>(dst)[c] = make_float4(f[0], f[1], f[2], f[3]);
        else {
            const __nv_bfloat162 lo = __floats2bfloat162_rn(f[0], f[1]), hi = __floats2bfloat162_rn(f[2], f[3]);
            reinterpret_cast<uint2*>(dst)[c] = make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
        }
    }
}

template <typename T, bool SIG>
static void launch_unit_rms(const float* o, const float* gate, long long ld_gate, const float* w, T* out, int units, int heads, int vdim, float eps,
                            cudaStream_t s) {
    auto al16 = [](const void* q) { return (reinterpret_cast<uintptr_t>(q) & 15u) == 0; };
    const unsigned grid = (unsigned)((units + 3) / 4);
    if (vdim % 4 == 0 && vdim <= 512 && ld_gate % 4 == 0 && al16(o) && al16(gate) && al16(w) && al16(out)) {
        if (vdim <= 128) launch_chained(unit_rms_gate_reg_kernel<T, SIG, 1>, grid, 128, 0, s, o, gate, ld_gate, w, out, units, heads, vdim, eps);
        else if (vdim <= 256) launch_chained(unit_rms_gate_reg_kernel<T, SIG, 2>, grid, 128, 0, s, o, gate, ld_gate, w, out, units, heads, vdim, eps);
        else launch_chained(unit_rms_gate_reg_kernel<T, SIG, 4>, grid, 128, 0, s, o, gate, ld_gate, w, out, units, heads, vdim, eps);
    } else
        launch_chained(unit_rms_gate_kernel<T, SIG>, grid, 128, 0, s, o, gate, ld_gate, w, out, units, heads, vdim, eps);
}

}  // namespace b200

using namespace b200;

extern "C" size_t b200_retention_workspace_bytes(int n_tokens, int n_entries, int heads, int dim, int vdim) {
    if (n_tokens < 2 * kChunk || n_entries < 1 || heads < 1 || dim < 1 || vdim < 1) return 0;
    return (size_t)(n_tokens / kChunk + n_entries + 1) * heads * dim * vdim * sizeof(float);
}

extern "C" int b200_retention(const b200_retention_args* p, void* stream) {
    if (!p || !p->proj || !p->decay || !p->state || !p->out || !p->ent_row || !p->ent_len || !p->slot || !p->pos || p->n_entries < 0 ||
        p->heads < 1 || p->dim < 1 || p->vdim < 1)
        return B200_EINVAL;
    if (p->rot_dims < 0 || (p->rot_dims & 1) || p->rot_dims > p->dim || (p->rot_dims && (!p->cos || !p->sin))) return B200_EINVAL;
    if (p->rot_layout != B200_ROPE_HALF && p->rot_layout != B200_ROPE_INTERLEAVED) return B200_EINVAL;
    if (p->dim > 256) return B200_EUNSUPPORTED;
    if (p->n_entries == 0) return B200_OK;
    RT a{p->proj, p->ld_proj, p->q_off, p->k_off, p->v_off, p->cos, p->sin, p->rot_dims, p->rot_layout, p->decay, p->k_scale,
         p->state, p->out, p->ent_row, p->ent_len, p->slot, p->pos, p->heads, p->dim, p->vdim};
    cudaStream_t s = (cudaStream_t)stream;
    const char* env = getenv("B200_RETENTION_WALK");   // 1: every entry on the token-by-token kernel (debugging aid)
    const size_t need = b200_retention_workspace_bytes(p->n_tokens, p->n_entries, p->heads, p->dim, p->vdim);
    if (p->longest_entry >= 2 * kChunk && need > 0 && p->workspace && p->workspace_bytes >= need && !(env && env[0] == '1')) {
        RC rc{a, reinterpret_cast<float*>(p->workspace), 1};
        const int col_blocks = (p->vdim + kChunkCols - 1) / kChunkCols, chunks = (p->longest_entry + kChunk - 1) / kChunk;
        if (chunks > 65535 || p->heads > 65535) return B200_EUNSUPPORTED;
        const dim3 grid(p->n_entries * col_blocks, chunks, p->heads);
        const int rs = chunk_row_stride(p->dim);
        const size_t smem1 = ((size_t)kChunk * rs + kChunk) * sizeof(float);
        const size_t smem3 = ((size_t)2 * p->dim * kChunkT + kChunk * kChunkT + kChunk + 4) * sizeof(float);
        static unsigned long long done1[8] = {}, done3[2] = {};
        // the attribute is set once per kernel: to the most any supported dim (256) needs
        constexpr int kMax1 = (kChunk * 260 + kChunk) * 4, kMax3 = (2 * 256 * kChunkT + kChunk * kChunkT + kChunk + 4) * 4;
        auto out = p->dim <= 32 ? retention_chunk_out_kernel<true> : retention_chunk_out_kernel<false>;
        cudaError_t e = ensure_max_dynamic_smem((const void*)out, kMax3, done3[p->dim <= 32]);
        if (e != cudaSuccess) return (int)e;
        rc.col_blocks = col_blocks;
        auto state = [&](auto kernel, unsigned long long& done) {
            ensure_max_dynamic_smem((const void*)kernel, kMax1, done);
            launch_chained(kernel, grid, 256, smem1, s, rc);
        };
        if (p->dim < 32) state(retention_chunk_state_kernel<8, false>, done1[0]);
        else if (p->dim == 32) state(retention_chunk_state_kernel<8, true>, done1[1]);
        else if (p->dim < 64) state(retention_chunk_state_kernel<16, false>, done1[2]);
        else if (p->dim == 64) state(retention_chunk_state_kernel<16, true>, done1[3]);
        else if (p->dim < 128) state(retention_chunk_state_kernel<32, false>, done1[4]);
        else if (p->dim == 128) state(retention_chunk_state_kernel<32, true>, done1[5]);
        else if (p->dim < 256) state(retention_chunk_state_kernel<64, false>, done1[6]);
        else state(retention_chunk_state_kernel<64, true>, done1[7]);
        const int per = p->dim * p->vdim;
        if (per % 4 == 0 && ((reinterpret_cast<uintptr_t>(p->state) | reinterpret_cast<uintptr_t>(p->workspace)) & 15u) == 0)
            launch_chained(retention_chunk_scan_kernel<float4>, dim3(p->n_entries, p->heads, (per / 4 + 255) / 256), 256, 0, s, rc);
        else
            launch_chained(retention_chunk_scan_kernel<float>, dim3(p->n_entries, p->heads, (per + 255) / 256), 256, 0, s, rc);
        launch_chained(out, grid, 256, smem3, s, rc);
        count_launch(3);
        return (int)cudaGetLastError();
    }
    const int threads = p->vdim <= 32 ? 32 : p->vdim <= 64 ? 64 : 128;
    const dim3 grid(p->n_entries, p->heads, (p->vdim + threads - 1) / threads);
    if (grid.y > 65535 || grid.z > 65535) return B200_EUNSUPPORTED;
    const size_t smem = (size_t)(2 + 2 * kWalkTokens) * p->dim * sizeof(float);
    if (p->dim <= 32) launch_chained(retention_walk_kernel<32>, grid, threads, smem, s, a);
    else if (p->dim <= 64) launch_chained(retention_walk_kernel<64>, grid, threads, smem, s, a);
    else if (p->dim <= 128) launch_chained(retention_walk_kernel<128>, grid, threads, smem, s, a);
    else launch_chained(retention_walk_kernel<256>, grid, threads, smem, s, a);
    count_launch();
    return (int)cudaGetLastError();
}

extern "C" int b200_unit_rms_gate(const float* o, const float* gate, long long ld_gate, void* out, int n_tokens, int heads, int vdim,
                                  float eps, int out_dtype, void* stream) {
    return b200_head_rms_gate(o, gate, ld_gate, nullptr, 0, out, n_tokens, heads, vdim, eps, out_dtype, stream);
}

extern "C" int b200_head_rms_gate(const float* o, const float* gate, long long ld_gate, const float* w, int sigmoid_gate, void* out, int n_tokens,
                                  int heads, int vdim, float eps, int out_dtype, void* stream) {
    if (!o || !gate || !out || n_tokens < 0 || heads < 1 || vdim < 1) return B200_EINVAL;
    if (out_dtype != B200_BF16 && out_dtype != B200_F32) return B200_EINVAL;
    if (n_tokens == 0) return B200_OK;
    const int units = n_tokens * heads;
    cudaStream_t s = (cudaStream_t)stream;
    using bf = __nv_bfloat16;
    if (out_dtype == B200_BF16) {
        if (sigmoid_gate) launch_unit_rms<bf, true>(o, gate, ld_gate, w, (bf*)out, units, heads, vdim, eps, s);
        else launch_unit_rms<bf, false>(o, gate, ld_gate, w, (bf*)out, units, heads, vdim, eps, s);
    } else {
        if (sigmoid_gate) launch_unit_rms<float, true>(o, gate, ld_gate, w, (float*)out, units, heads, vdim, eps, s);
        else launch_unit_rms<float, false>(o, gate, ld_gate, w, (float*)out, units, heads, vdim, eps, s);
    }
    count_launch();
    return (int)cudaGetLastError();
}
