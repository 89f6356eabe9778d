// The chunk form of the state-space recurrence (ssd_scan.cu has the mathematics) on tcgen05 / TMEM: chunks of 128 tokens, 64 value columns of a head at
// a time ("a unit"), four launches:
//   ssd_tc_prep_kernel   what all heads of a group share, once: C, B and B^T rounded and laid out for shared memory; and every head's sums of A dt
//   ssd_tc_state_kernel  U = B^T (exp(cum_end - cum_j) dt_j x_j) of every chunk; a CTA keeps B^T of a chunk and takes several units
//   ssd_tc_carry_kernel  S at the start of every chunk and behind the entry, in fp32; what the products read is rounded here, once
//   ssd_tc_out_kernel    y = exp(cum_i) C S + [(C_i . B_j) exp(cum_i - cum_j), j <= i] (dt_j x_j) + D x; a CTA forms C . B, keeps
//                        it and C, and takes several units
// Operands are tf32 (rounded to nearest, once each) with fp32 sums; cum is summed in double and its differences are formed from two floats each, so
// neighbours behind a large sum still decay by exactly their own.
// What bounded the 64-token chunks on mma.sync: every head loaded and rounded the B and C that its group shares, fragments were rounded each time they were
// picked up, and states crossed memory for every 64 tokens. Here a unit's inputs are its x, its state and its sums; the next units' are under way
// meanwhile. (One CTA per head that walks its chunks with the state in TMEM was built too: 110 us, everything of a chunk waits for something of the chunk before.)
// The 64 columns of a unit lie in operands and TMEM as row r = (p % 4) * 16 + p / 4: 16-byte pieces of x go to shared memory without bank conflicts.
// The state and out kernels, a CTA on each SM that they use, start what follows by ending, not ahead of it: launched earlier, the CTAs of the carry (of the next call's
// prep) sat down on the SMs that happened to be free, and where 128 of 148 were busy they worked there in a heap. 2 entries, 2048 tokens, 64 heads, 128: 74.4 -> 68.5 us; 1, 2048, 16
// heads, 64: 44.7 -> 28.9 (37.3 in chunks of 64); 1, 2048, 33 heads, 128: 59.6 -> 39.6.
// A product dt x that is not finite is multiplied as zero and its column is NaN from its token on: the zeros above the diagonal would carry it to
// earlier tokens.
// Measured in a graph, us, chunks of 64 on mma.sync against these (entries, tokens, heads, n_state; 64 value columns): 2, 2048, 64, 128: 149 / 68.5 (floor 11; under ncu 9, 19,
// 22 and 39 of 90: the latency of loads, DRAM a quarter and L2 a fifth to two fifths busy, the tensor pipe an eighth); 1, 2048, 33, 128: 86 / 40; 1, 128, 8, 128: 25.7 / 18.7; 2, 2048, 64, 64: 92 / 67; 4, 1500, 64, 64: 74 / 54. Error against 64 bits 3.2e-4 of the outputs'
// norm, 2.9e-4 of the states', in either.
#include <limits.h>

#include <algorithm>

#include "launch_count.h"
#include "ssd_scan.cuh"
#include "tc_common.cuh"

namespace b200 {

constexpr int kStChunk = 128, kStCols = 64, kStSums = 5 * kStChunk * 4, kStImg = kStChunk * 128 * 4, kStUnit = kStCols * 128 * 4;   // bytes

struct SsTc {
    SS s;
    float* c_img;    // [place, group]: C, four blocks of 32 columns, 128-byte rows (tokens) with the 128-byte swizzle
    float* bt_img;   // [place, group]: B^T, four blocks of 32 tokens, 128-byte rows (n)
    float* b_img;    // [place, group]: B, as C
    float* sums;     // [place, head]: see st_sums
    float* states;   // [place, unit]: U, then S at the chunk's start, four blocks of 32 n, 128-byte rows r
    int blocks;      // CTAs per (chunk, entry), as many for each group
};

// D[tmem] (+)= A B on tf32 operands, K = 8: A from shared memory, or from TMEM (a row per lane, one operand per column)
__device__ __forceinline__ void umma_tf32(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        "setp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, p;\n"
        "}\n" ::"r"(d_tmem),
        "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
        : "memory");
}
__device__ __forceinline__ void umma_tf32_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        "setp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::1.kind::tf32 [%0], [%1], %2, %3, p;\n"
        "}\n" ::"r"(d_tmem),
        "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate)
        : "memory");
}
// (no "memory": loads may move past it, which a chain of stores otherwise forbids; barriers and fences are volatile and keep their place)
__device__ __forceinline__ void st_shared_f32(uint32_t addr, float v) { asm volatile("st.shared.f32 [%0], %1;" ::"r"(addr), "f"(v)); }
// two numbers rounded to tf32 operands; what is finite stays finite. (Veltkamp's splitting, three packed instructions for both, made NaN of what lies above 2^114
// and saved nothing: 2 entries, 2048 tokens, 64 heads 74.4 us with it and 74.2 with the conversions, in a graph.)
__device__ __forceinline__ uint64_t st_tf32x2(uint64_t x) {
    float a, b;
    unpack2(x, a, b);
    return pack2f(ssd_tf32(a), ssd_tf32(b));
}
__device__ __forceinline__ void tmem_ld_32x4_async(uint32_t taddr, uint32_t* v) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]) : "r"(taddr) : "memory");
}
__device__ __forceinline__ void tmem_st_32x16(uint32_t taddr, const uint32_t* v) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};" ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]),
                 "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15])
                 : "memory");
}
__device__ __forceinline__ size_t st_place(int row_e, int e, int c) { return (size_t)(row_e / kStChunk + e + c); }
// the 16 bytes (piece of eight) of a swizzled 128-byte row
__device__ __forceinline__ uint32_t st_piece(int row, int piece) { return (uint32_t)(row * 128 + ((piece ^ (row & 7)) << 4)); }

// A chunk and head per warp, four tokens per lane: -hi and -lo of cum log2(e) (cum the running sum of A dt, in double, hi + lo in float), dt, exp(cum), and
// exp(cum_end - cum), the last zero behind the entry
__device__ void st_sums(const SS& a, int h, int row0, int len, float* sm) {
    const int lane = threadIdx.x & 31;
    const float bias = a.dt_bias[h];
    float raw[4], dt[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) raw[k] = __ldcg(a.dt_raw + (size_t)(row0 + min(4 * lane + k, len - 1)) * a.ld_dt + h);
    const double A = (double)a.A[h] * 1.4426950408889634;
    double v[4], run = 0.0;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        dt[k] = 4 * lane + k < len ? ssd_softplus(raw[k] + bias) : 0.f;
        run += A * dt[k];
        v[k] = run;
    }
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const double up = __shfl_up_sync(0xffffffffu, run, o);
        if (lane >= o) run += up;
    }
    const double end = __shfl_sync(0xffffffffu, run, 31);
    double before = __shfl_up_sync(0xffffffffu, run, 1);
    if (lane == 0) before = 0.0;
    float out[5][4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const double cum = before + v[k];
        const float hi = (float)cum;
        out[0][k] = -hi;
        out[1][k] = fabsf(hi) < __int_as_float(0x7f800000) ? -(float)(cum - (double)hi) : 0.f;
        out[2][k] = dt[k];
        out[3][k] = exp2f(hi);
        out[4][k] = 4 * lane + k < len ? exp2f((float)(end - cum)) : 0.f;
    }
#pragma unroll
    for (int q = 0; q < 5; ++q) *reinterpret_cast<float4*>(sm + q * kStChunk + 4 * lane) = make_float4(out[q][0], out[q][1], out[q][2], out[q][3]);
}

// 16 tokens of a chunk per CTA for what a group shares; and, in CTAs of their own, the sums of four heads
__global__ void __launch_bounds__(128) ssd_tc_prep_kernel(const SsTc t) {
    pdl_wait();
    pdl_launch_dependents();
    const SS& a = t.s;
    const int per_entry = 8 * a.groups + (a.heads + 3) / 4, e = blockIdx.x / per_entry, job = blockIdx.x % per_entry, chunk = blockIdx.y;
    const int row_e = a.ent_row[e], len = min(kStChunk, a.ent_len[e] - chunk * kStChunk);
    if (len <= 0) return;
    if (job >= 8 * a.groups) {
        const int h = (job - 8 * a.groups) * 4 + (int)threadIdx.x / 32;
        if (h < a.heads) st_sums(a, h, row_e + chunk * kStChunk, len, t.sums + (st_place(row_e, e, chunk) * a.heads + h) * (kStSums / 4));
        return;
    }
    const int m0 = (job & 7) * 16, g = job >> 3, N = a.n_state, n = threadIdx.x;
    const size_t place = st_place(row_e, e, chunk) * a.groups + g;
    // thread n: column n of 16 tokens; tokens that are not there are zeros, and so are columns behind n_state
    const float* row = a.u + (size_t)(row_e + chunk * kStChunk) * a.ld_u + g * N + min(n, N - 1);
    float c[16], b[16];
#pragma unroll
    for (int k = 0; k < 16; ++k) {
        const size_t at = (size_t)min(m0 + k, len - 1) * a.ld_u;
        c[k] = __ldcg(row + a.c_off + at);
        b[k] = __ldcg(row + a.b_off + at);
    }
#pragma unroll
    for (int k = 0; k < 16; ++k) {
        const bool in = n < N && m0 + k < len;
        c[k] = in ? ssd_tf32(c[k]) : 0.f;
        b[k] = in ? ssd_tf32(b[k]) : 0.f;
    }
    unsigned char* bt = reinterpret_cast<unsigned char*>(t.bt_img) + place * kStImg + (m0 >> 5) * 16384;
#pragma unroll
    for (int q = 0; q < 4; ++q) *reinterpret_cast<float4*>(bt + st_piece(n, ((m0 & 31) >> 2) + q)) = make_float4(b[4 * q], b[4 * q + 1], b[4 * q + 2], b[4 * q + 3]);
    unsigned char *ci = reinterpret_cast<unsigned char*>(t.c_img) + place * kStImg + (n >> 5) * 16384 + (n & 3) * 4, *bi = reinterpret_cast<unsigned char*>(t.b_img) + place * kStImg + (n >> 5) * 16384 + (n & 3) * 4;
#pragma unroll
    for (int k = 0; k < 16; ++k) {
        *reinterpret_cast<float*>(ci + st_piece(m0 + k, (n & 31) >> 2)) = c[k];
        *reinterpret_cast<float*>(bi + st_piece(m0 + k, (n & 31) >> 2)) = b[k];
    }
}

// ---- half of the x of a unit: 32 tokens x 32 columns per warp, four tokens x 128 bytes per load
struct StX {
    float4 v[8];
    // row0, len: the chunk's. Tokens behind it are its last one again (their weights are zero), columns behind vdim the unit's first ones (never stored): a
    // load behind a condition would wait for the one before it.
    __device__ __forceinline__ void load(const SS& a, int row0, int len, int quarter, int half, int head, int p0, int lane) {
        const int t = quarter * 32 + (lane >> 3), c = half * 32 + (lane & 7) * 4;
        const float* src = a.u + (size_t)row0 * a.ld_u + a.x_off + (size_t)head * a.vdim + p0 + (p0 + c < a.vdim ? c : 0);
#pragma unroll
        for (int k = 0; k < 8; ++k) v[k] = __ldcg(reinterpret_cast<const float4*>(src + (size_t)min(t + 4 * k, len - 1) * a.ld_u));
    }
    // times the tokens' weights, rounded, transposed into the operand; returns whether every product of the warp was finite
    template <bool TWO>
    __device__ __forceinline__ bool store(uint32_t dst, int quarter, int half, int lane, const float* w0, const float* w1) {
        const int t = lane >> 3, l7 = lane & 7;
        const uint32_t base = dst + (uint32_t)(quarter * 8192 + half * 1024 + l7 * 128 + t * 4);
        uint64_t odd[2] = {0ull, 0ull};
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const int j = quarter * 32 + k * 4 + t;
            const float w = TWO ? w0[j] * w1[j] : w0[j];
            const uint64_t w2 = pack2f(w, w), lo = st_tf32x2(mul2(pack2f(v[k].x, v[k].y), w2)), hi = st_tf32x2(mul2(pack2f(v[k].z, v[k].w), w2));
            odd[0] = fma2(lo, 0ull, odd[0]);
            odd[1] = fma2(hi, 0ull, odd[1]);
            float r0, r1, r2, r3;
            unpack2(lo, r0, r1);
            unpack2(hi, r2, r3);
            const uint32_t at = base + (uint32_t)((k ^ l7) << 4);
            st_shared_f32(at, r0);
            st_shared_f32(at + 2048u, r1);
            st_shared_f32(at + 4096u, r2);
            st_shared_f32(at + 6144u, r3);
        }
        float o0, o1;
        unpack2(add2(odd[0], odd[1]), o0, o1);
        return !__any_sync(0xffffffffu, o0 + o1 != 0.f);   // a NaN: something was not finite
    }
};

struct StWork {   // a CTA's units
    int e, chunk, g, first, step, count, row0, len, per_group, col_blocks;
    size_t place;
    __device__ __forceinline__ StWork(const SsTc& t) {
        const SS& a = t.s;
        e = blockIdx.x / t.blocks;
        const int b = blockIdx.x % t.blocks;
        col_blocks = a.col_blocks;
        per_group = a.heads / a.groups * col_blocks;
        const int per = t.blocks / a.groups;   // blocks per group
        g = b / per;
        first = b % per;   // neighbours take neighbouring units at the same time: x then leaves DRAM in runs of 256 bytes times the blocks
        step = per;
        count = (per_group - first + per - 1) / per;
        chunk = blockIdx.y;
        const int row_e = a.ent_row[e];
        len = min(kStChunk, a.ent_len[e] - chunk * kStChunk);
        row0 = row_e + chunk * kStChunk;
        place = st_place(row_e, e, chunk);
    }
    __device__ __forceinline__ int unit(int u) const { return g * per_group + first + u * step; }   // of all units
    __device__ __forceinline__ int head(int u) const { return col_blocks == 1 ? unit(u) : unit(u) / col_blocks; }
    __device__ __forceinline__ int p0(int u) const { return col_blocks == 1 ? 0 : unit(u) % col_blocks * kStCols; }
};

// ---- U of every chunk. Warps 0-7: x; 8-11: U out of TMEM; 12: products; 13: copies
constexpr int kSuOffX = kStImg, kSuOffSums = kSuOffX + 2 * kStUnit, kSuOffBar = kSuOffSums + 2 * kStSums, kSuSmem = kSuOffBar + 16 * 8 + 16 + 1024;
__global__ void __launch_bounds__(448, 1) ssd_tc_state_kernel(const SsTc t) {
    pdl_wait();
    extern __shared__ __align__(1024) unsigned char st_raw[];
    unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(st_raw) + 1023) & ~(uintptr_t)1023);
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + kSuOffBar);
    uint64_t *sum_full = bars, *sum_empty = bars + 2, *x_full = bars + 4, *x_empty = bars + 6, *d_full = bars + 8, *d_empty = bars + 10, *b_full = bars + 12;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 13);
    volatile int* dead = reinterpret_cast<volatile int*>(tmem_slot + 1);
    uint64_t* drained = bars + 14;
    volatile int* asked = reinterpret_cast<volatile int*>(bars + 15);   // sums requested so far
    const SS& a = t.s;
    const StWork w(t);
    if (w.len <= 0 || w.count <= 0) return;
    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31, quarter = warp & 3;
    if (warp == 12) tmem_alloc(tmem_slot, 128);
    if (threadIdx.x == 0) {
        *dead = *asked = 0;
        mbar_init(drained, 1);
        for (int i = 0; i < 2; ++i) {
            mbar_init(&sum_full[i], 1); mbar_init(&sum_empty[i], 8);
            mbar_init(&x_full[i], 8); mbar_init(&x_empty[i], 1);
            mbar_init(&d_full[i], 1); mbar_init(&d_empty[i], 4);
        }
        mbar_init(b_full, 1);
        mbar_fence_init();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = __shfl_sync(0xffffffffu, *tmem_slot, 0);
    const float* sums = reinterpret_cast<const float*>(smem + kSuOffSums);
    if (warp < 8) {
        const int half = warp >> 2;
        StX x[2];   // of this unit and of the next
        auto load = [&](int u, StX& v) {
            if (u < w.count) v.load(a, w.row0, w.len, quarter, half, w.head(u), w.p0(u), lane);
        };
        auto put = [&](int u, StX& v) {
            const int b = u & 1;
            const uint32_t ph = (uint32_t)(u >> 1) & 1u;
            const float* sm = sums + b * (kStSums / 4);
            mbar_wait_or_leave(&sum_full[b], ph, dead);
            mbar_wait_or_leave(&x_empty[b], ph ^ 1u, dead);
            v.store<true>(smem_u32(smem + kSuOffX + b * kStUnit), quarter, half, lane, sm + 2 * kStChunk, sm + 4 * kStChunk);
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) {
                mbar_arrive(&x_full[b]);
                mbar_arrive(&sum_empty[b]);
            }
        };
        load(0, x[0]);
        load(1, x[1]);
        __syncwarp();
#pragma unroll 1
        for (int u = 0; u < w.count; u += 2) {
            put(u, x[0]);
            load(u + 2, x[0]);
            if (u + 1 < w.count) {
                put(u + 1, x[1]);
                load(u + 3, x[1]);
            }
            __syncwarp();
        }
    } else if (warp < 12) {
#pragma unroll 1
        for (int u = 0; u < w.count; ++u) {
            const int b = u & 1;
            unsigned char* dst = reinterpret_cast<unsigned char*>(t.states) + (w.place * ((size_t)a.heads * a.col_blocks) + w.unit(u)) * kStUnit + quarter * 8192 + (lane & 3) * 4;
            mbar_wait_or_leave(&d_full[b], (uint32_t)(u >> 1) & 1u, dead);
            tc_fence_after();
            const bool lost = *dead != 0;
#pragma unroll 1
            for (int half = 0; half < 2; ++half) {
                uint32_t v[32];
                tmem_ld_32x32_async(tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(b * 64 + half * 32), v);
                tmem_wait_ld<32>(v);
                if (half) {
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&d_empty[b]);
                }
#pragma unroll
                for (int k = 0; k < 32; ++k)
                    *reinterpret_cast<uint32_t*>(dst + half * 4096 + st_piece(k, lane >> 2)) = lost ? 0x7fffffffu : v[k];
            }
        }
    } else if (warp == 12) {
        constexpr uint32_t idesc = make_idesc_f16(128, kStCols) | (2u << 7) | (2u << 10);   // tf32 operands
        const uint64_t b_desc = make_kmajor_sw128_desc(smem_u32(smem)), x_desc = make_kmajor_sw128_desc(smem_u32(smem + kSuOffX));
        const int n = __shfl_sync(0xffffffffu, w.count, 0);
        const bool leader = elect_one();
        mbar_wait_or_leave(b_full, 0u, dead);
#pragma unroll 1
        for (int u = 0; u < n; ++u) {
            const uint32_t b = (uint32_t)u & 1u, ph = (uint32_t)(u >> 1) & 1u;
            mbar_wait_or_leave(&d_empty[b], ph ^ 1u, dead);
            mbar_wait_or_leave(&x_full[b], ph, dead);
            tc_fence_after();
            if (leader) {
#pragma unroll
                for (int k = 0; k < 16; ++k)
                    umma_tf32(tmem + b * 64u, b_desc + (uint64_t)((k >> 2) * (16384 >> 4) + 2 * (k & 3)), x_desc + (uint64_t)(b * (kStUnit >> 4) + (k >> 2) * (8192 >> 4) + 2 * (k & 3)), idesc, k > 0 ? 1u : 0u);
                umma_commit(&x_empty[b]);
                umma_commit(&d_full[b]);
            }
            __syncwarp();
        }
    } else {
        if (lane == 0) {
            mbar_expect_tx(b_full, kStImg);
            bulk_g2s(smem, reinterpret_cast<const unsigned char*>(t.bt_img) + (w.place * a.groups + w.g) * kStImg, kStImg, b_full);
        }
        __syncwarp();
#pragma unroll 1
        for (int u = 0; u < w.count; ++u) {
            const int b = u & 1;
            mbar_wait_or_leave(&sum_empty[b], ((uint32_t)(u >> 1) & 1u) ^ 1u, dead);
            if (__any_sync(0xffffffffu, *dead)) break;
            if (lane == 0) {
                *asked = u + 1;
                mbar_expect_tx(&sum_full[b], kStSums);
                bulk_g2s(smem + kSuOffSums + b * kStSums, t.sums + (w.place * a.heads + w.head(u)) * (kStSums / 4), kStSums, &sum_full[b]);
            }
            __syncwarp();
        }
    }
    __syncthreads();
    if (*dead) {   // what is under way lands first
        if (warp == 13) {
            mbar_wait_limited(b_full, 0u);
            for (int u = max(0, *asked - 2); u < *asked; ++u) mbar_wait_limited(&sum_full[u & 1], (uint32_t)(u >> 1) & 1u);
        } else if (warp == 12) {
            if (elect_one()) umma_commit(drained);
            mbar_wait_limited(drained, 0u);
        }
        __syncthreads();
    }
    tc_fence_after();
    if (warp == 12) tmem_dealloc(tmem, 128);
}

// ---- four n x four value columns of a unit per thread: U of the entry's chunks to S at their starts (rounded), and the state behind the entry
__global__ void __launch_bounds__(128) ssd_tc_carry_kernel(const SsTc t) {
    pdl_wait();
    pdl_launch_dependents();
    const SS& a = t.s;
    const int e = blockIdx.y, unit = blockIdx.x / 4, i = (blockIdx.x & 3) * 128 + threadIdx.x;   // of 512 threads: n in steps of 4, then p
    const int q = i >> 1 & 15, n4 = (i & 1) + (i >> 5) * 2, h = unit / a.col_blocks, p = unit % a.col_blocks * kStCols + q * 4, N = a.n_state, P = a.vdim;
    const int row_e = a.ent_row[e], n_tok = a.ent_len[e], chunks = (n_tok + kStChunk - 1) / kStChunk;
    if (chunks <= 0) return;
    const size_t units = (size_t)a.heads * a.col_blocks, first = st_place(row_e, e, 0);
    float* st = a.state + (((size_t)a.slot[row_e] * a.heads + h) * N + n4 * 4) * P + p;
    const bool in = p < P;
    uint64_t S[4][2];   // [p][n pair]
#pragma unroll
    for (int c = 0; c < 4; ++c) S[c][0] = S[c][1] = 0ull;
    if (a.pos[row_e] > 0 && in) {
        float4 v[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) v[k] = n4 * 4 + k < N ? *reinterpret_cast<const float4*>(st + (size_t)k * P) : make_float4(0.f, 0.f, 0.f, 0.f);
        S[0][0] = pack2f(v[0].x, v[1].x); S[0][1] = pack2f(v[2].x, v[3].x);
        S[1][0] = pack2f(v[0].y, v[1].y); S[1][1] = pack2f(v[2].y, v[3].y);
        S[2][0] = pack2f(v[0].z, v[1].z); S[2][1] = pack2f(v[2].z, v[3].z);
        S[3][0] = pack2f(v[0].w, v[1].w); S[3][1] = pack2f(v[2].w, v[3].w);
    }
    // rows r = c * 16 + q of the unit's block of 32 n
    unsigned char* U = reinterpret_cast<unsigned char*>(t.states) + (first * units + unit) * kStUnit + (n4 >> 3) * 8192 + st_piece(q, n4 & 7);
    const float* dec = t.sums + (first * a.heads + h) * (kStSums / 4) + 4 * kStChunk - 1;   // exp(cum_end)
    constexpr int F = 4;
    for (int c0 = 0; c0 < chunks; c0 += F) {   // F chunks' loads in flight, then the dependent chain
        ulonglong2 u[F][4];
        float d[F];
#pragma unroll
        for (int k = 0; k < F; ++k) {   // (behind the last chunk: the last one again, without a condition, see StX)
            const size_t ck = (size_t)min(c0 + k, chunks - 1);
            d[k] = __ldcg(dec + ck * a.heads * (kStSums / 4));
#pragma unroll
            for (int c = 0; c < 4; ++c) u[k][c] = __ldcg(reinterpret_cast<const ulonglong2*>(U + ck * units * kStUnit + c * 2048));
        }
#pragma unroll
        for (int k = 0; k < F; ++k)
            if (c0 + k < chunks) {
                const uint64_t d2 = pack2f(d[k], d[k]);
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    ulonglong2 o;
                    o.x = st_tf32x2(S[c][0]);
                    o.y = st_tf32x2(S[c][1]);
                    *reinterpret_cast<ulonglong2*>(U + (size_t)(c0 + k) * units * kStUnit + c * 2048) = o;
                    S[c][0] = fma2(d2, S[c][0], u[k][c].x);
                    S[c][1] = fma2(d2, S[c][1], u[k][c].y);
                }
            }
    }
    if (!in) return;
    float v[4][4];
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        unpack2(S[c][0], v[0][c], v[1][c]);
        unpack2(S[c][1], v[2][c], v[3][c]);
    }
#pragma unroll
    for (int k = 0; k < 4; ++k)
        if (n4 * 4 + k < N) *reinterpret_cast<float4*>(st + (size_t)k * P) = make_float4(v[k][0], v[k][1], v[k][2], v[k][3]);
}

// ---- the outputs. Warps 0-7: C . B with its decays, every other block of 32 tokens each; 8-15: x, half of the columns each; 16-23: outputs, half of the columns
// each; 24: products; 25: copies. (Half of the warps with twice the work each took a quarter longer: what they do is a chain of short waits.)
static_assert(kStImg == 2 * kStUnit, "B takes the place of two states");
constexpr int kSoOffS = kStImg, kSoOffX = kSoOffS + 2 * kStUnit, kSoOffStage = kSoOffX + 2 * kStUnit, kSoOffSums = kSoOffStage + 8 * 2048, kSoOffBad = kSoOffSums + 4 * kStSums,
              kSoBad = (4 * kStCols + 8) * 4, kSoOffBar = kSoOffBad + 2 * kSoBad, kSoSmem = kSoOffBar + 32 * 8 + 16 + 1024;
static_assert(kSoSmem <= 227 * 1024 && kSoOffBar % 8 == 0, "one CTA per SM");
constexpr uint32_t kSoCB = 0, kSoM = 128, kSoD = 256;   // TMEM columns; D: two buffers of C S and M x
__global__ void __launch_bounds__(26 * 32, 1) ssd_tc_out_kernel(const SsTc t) {
    pdl_wait();
    extern __shared__ __align__(1024) unsigned char st_raw[];
    unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(st_raw) + 1023) & ~(uintptr_t)1023);
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + kSoOffBar);
    uint64_t *sum_full = bars, *sum_empty = bars + 4, *m_full = bars + 8, *m_empty = bars + 12, *x_full = bars + 16, *x_empty = bars + 18, *s_full = bars + 20, *s_empty = bars + 22,
             *d_full = bars + 24, *d_empty = bars + 26, *c_full = bars + 28, *cb_full = bars + 29;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 30);
    volatile int* dead = reinterpret_cast<volatile int*>(tmem_slot + 1);
    uint64_t* drained = bars + 31;
    volatile int* asked = reinterpret_cast<volatile int*>(bars + 32);   // sums, states requested so far
    const SS& a = t.s;
    const StWork w(t);
    if (w.len <= 0 || w.count <= 0) return;
    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31, quarter = warp & 3;
    if (warp == 24) tmem_alloc(tmem_slot, 512);
    if (threadIdx.x == 0) {
        *dead = asked[0] = asked[1] = 0;
        mbar_init(drained, 1);
        for (int i = 0; i < 4; ++i) {
            mbar_init(&sum_full[i], 1); mbar_init(&sum_empty[i], 24);
            mbar_init(&m_full[i], 4 - i); mbar_init(&m_empty[i], 1);
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(&x_full[i], 8); mbar_init(&x_empty[i], 9);   // the products, and the outputs' look at what was not finite
            mbar_init(&s_full[i], 1); mbar_init(&s_empty[i], 1);
            mbar_init(&d_full[i], 1); mbar_init(&d_empty[i], 8);
        }
        mbar_init(c_full, 1);
        mbar_init(cb_full, 1);
        mbar_fence_init();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = __shfl_sync(0xffffffffu, *tmem_slot, 0), my = (uint32_t)(quarter * 32) << 16;
    const float* sums = reinterpret_cast<const float*>(smem + kSoOffSums);
    if (warp < 8) {   // ---- lane i
        const int odd = warp >> 2, i = quarter * 32 + lane;
        {
            uint32_t v[32];
#pragma unroll
            for (int k = 0; k < 32; ++k) v[k] = 0u;
#pragma unroll 1
            for (int b = quarter + 1; b < 4 && !odd; ++b) tmem_st_32x32(tmem + kSoM + my + (uint32_t)(b * 32), v);   // above the diagonal the operand stays zero
        }
        tmem_wait_st();
        mbar_wait_or_leave(cb_full, 0u, dead);
        tc_fence_after();
#pragma unroll 1
        for (int u = 0; u < w.count; ++u) {
            const float* sm = sums + (u & 3) * (kStSums / 4);
            mbar_wait_or_leave(&sum_full[u & 3], (uint32_t)(u >> 2) & 1u, dead);
            const uint64_t hi2 = pack2f(-sm[i], -sm[i]), lo2 = pack2f(-sm[kStChunk + i], -sm[kStChunk + i]);
#pragma unroll 1
            for (int b = odd; b <= quarter; b += 2) {
                bool waited = false;
#pragma unroll 1
                for (int k0 = 0; k0 < 32; k0 += 16) {
                    uint32_t v[16], cb[16];
                    tmem_ld_32x16_async(tmem + kSoCB + my + (uint32_t)(b * 32 + k0), cb);
#pragma unroll
                    for (int k = 0; k < 16; k += 4) {
                        const float4 nh = *reinterpret_cast<const float4*>(sm + b * 32 + k0 + k), nl = *reinterpret_cast<const float4*>(sm + kStChunk + b * 32 + k0 + k);
                        float x0, x1, x2, x3;
                        unpack2(add2(add2(hi2, pack2f(nh.x, nh.y)), add2(lo2, pack2f(nl.x, nl.y))), x0, x1);
                        unpack2(add2(add2(hi2, pack2f(nh.z, nh.w)), add2(lo2, pack2f(nl.z, nl.w))), x2, x3);
                        v[k] = __float_as_uint(ex2_approx(x0));
                        v[k + 1] = __float_as_uint(ex2_approx(x1));
                        v[k + 2] = __float_as_uint(ex2_approx(x2));
                        v[k + 3] = __float_as_uint(ex2_approx(x3));
                    }
                    tmem_wait_ld<16>(cb);
#pragma unroll
                    for (int k = 0; k < 16; k += 2) {
                        float r0, r1;
                        unpack2(st_tf32x2(mul2(pack2(v[k], v[k + 1]), pack2(cb[k], cb[k + 1]))), r0, r1);
                        v[k] = __float_as_uint(r0);
                        v[k + 1] = __float_as_uint(r1);
                    }
                    if (b == quarter) {
#pragma unroll
                        for (int k = 0; k < 16; ++k) v[k] = k0 + k <= lane ? v[k] : 0u;
                    }
                    if (!waited) {
                        mbar_wait_or_leave(&m_empty[b], (uint32_t)(u & 1) ^ 1u, dead);
                        tc_fence_after();
                        waited = true;
                    }
                    tmem_st_32x16(tmem + kSoM + my + (uint32_t)(b * 32 + k0), v);
                }
                tmem_wait_st();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&m_full[b]);
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(&sum_empty[u & 3]);
        }
    } else if (warp < 16) {
        const int half = (warp >> 2) & 1;
        StX x;
        x.load(a, w.row0, w.len, quarter, half, w.head(0), w.p0(0), lane);
        __syncwarp();
#pragma unroll 1
        for (int u = 0; u < w.count; ++u) {
            const int b = u & 1;
            const uint32_t dst = smem_u32(smem + kSoOffX + b * kStUnit);
            mbar_wait_or_leave(&sum_full[u & 3], (uint32_t)(u >> 2) & 1u, dead);
            mbar_wait_or_leave(&x_empty[b], ((uint32_t)(u >> 1) & 1u) ^ 1u, dead);
            const bool fine = x.store<false>(dst, quarter, half, lane, sums + (u & 3) * (kStSums / 4) + 2 * kStChunk, nullptr);
            unsigned* bad = reinterpret_cast<unsigned*>(smem + kSoOffBad + b * kSoBad);
            if (!fine) {   // rare: back out of shared memory, token `lane`, one of the warp's rows at a time
                __syncwarp();
#pragma unroll 1
                for (int q = 0; q < 32; ++q) {
                    const int r = (q >> 3) * 16 + half * 8 + (q & 7);
                    const uint32_t at = dst + (uint32_t)(quarter * 8192 + (lane & 3) * 4) + st_piece(r, lane >> 2);
                    float v;
                    asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(at) : "memory");
                    const bool off = !(fabsf(v) < __int_as_float(0x7f800000));
                    const unsigned m = __ballot_sync(0xffffffffu, off);
                    if (off) st_shared_f32(at, 0.f);
                    if (lane == 0) bad[quarter * kStCols + r] = m;
                }
            }
            if (lane == 0) bad[4 * kStCols + half * 4 + quarter] = fine ? 0u : 1u;
            if (u + 1 < w.count) x.load(a, w.row0, w.len, quarter, half, w.head(u + 1), w.p0(u + 1), lane);
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) {
                mbar_arrive(&x_full[b]);
                mbar_arrive(&sum_empty[u & 3]);
            }
        }
    } else if (warp < 24) {   // ---- lane i; stores: eight rows of 64 bytes per instruction
        const int half = (warp >> 2) & 1, m = lane & 3, r0 = quarter * 32 + (lane >> 2), left = w.len - r0;
        const long long ld_o = (long long)a.heads * a.vdim;
        const uint32_t stg = smem_u32(smem + kSoOffStage) + (uint32_t)((warp - 16) * 2048);
        auto stage_at = [&](int row, int piece) { return stg + (uint32_t)(row * 64 + ((piece ^ (row >> 1 & 3)) << 4)); };
        float4 x[8];   // [part][rows]
        auto load = [&](int u) {
            const float* xs = a.u + (size_t)w.row0 * a.ld_u + a.x_off + (size_t)w.head(u) * a.vdim;
            const int p = w.p0(u) + half * 32 + m * 4, c0 = p < a.vdim ? p : 0, c1 = p + 16 < a.vdim ? p + 16 : 0;
#pragma unroll
            for (int k = 0; k < 4; ++k) {   // (without a condition, see StX)
                const float* row = xs + (size_t)min(r0 + 8 * k, w.len - 1) * a.ld_u;
                x[k] = __ldcg(reinterpret_cast<const float4*>(row + c0));
                x[4 + k] = __ldcg(reinterpret_cast<const float4*>(row + c1));
            }
        };
        load(0);
        float Dn = __ldg(a.D + w.head(0));
        __syncwarp();
#pragma unroll 1
        for (int u = 0; u < w.count; ++u) {
            const int b = u & 1;
            const float Dh = Dn;
            if (u + 1 < w.count) Dn = __ldg(a.D + w.head(u + 1));
            mbar_wait_or_leave(&d_full[b], (uint32_t)(u >> 1) & 1u, dead);
            tc_fence_after();
            float ei = sums[(u & 3) * (kStSums / 4) + 3 * kStChunk + quarter * 32 + lane];
            if (*dead) ei = __int_as_float(0x7fffffff);
            const uint64_t ei2 = pack2f(ei, ei);
            const unsigned* bad = reinterpret_cast<const unsigned*>(smem + kSoOffBad + b * kSoBad);
            const unsigned* off = bad + 4 * kStCols + half * 4;
            const bool any_bad = (off[0] | off[1] | off[2] | off[3]) != 0u;
            float* dst = a.out + (size_t)(w.row0 + r0) * ld_o + (size_t)w.head(u) * a.vdim;
#pragma unroll
            for (int part = 0; part < 2; ++part) {   // four pieces of four columns
                uint32_t d1[16], d2[16];
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    tmem_ld_32x4_async(tmem + kSoD + my + (uint32_t)(b * 128 + c * 16 + half * 8 + part * 4), d1 + c * 4);
                    tmem_ld_32x4_async(tmem + kSoD + my + (uint32_t)(b * 128 + 64 + c * 16 + half * 8 + part * 4), d2 + c * 4);
                }
                tmem_wait_ld<16>(d1);
                tmem_wait_ld<16>(d2);
#pragma unroll
                for (int k = 0; k < 16; k += 2) {
                    float y0, y1;
                    unpack2(fma2(ei2, pack2(d1[k], d1[k + 1]), pack2(d2[k], d2[k + 1])), y0, y1);
                    d2[k] = __float_as_uint(y0);
                    d2[k + 1] = __float_as_uint(y1);
                }
                if (any_bad) {   // what was not finite reaches its own and later tokens
#pragma unroll 1
                    for (int q = 0; q <= quarter; ++q) {
                        const unsigned seen = !off[q] ? 0u : q < quarter ? 0xffffffffu : 0xffffffffu >> (31 - lane);
#pragma unroll
                        for (int k = 0; k < 16; ++k) d2[k] = bad[q * kStCols + (k >> 2) * 16 + half * 8 + part * 4 + (k & 3)] & seen ? 0x7fffffffu : d2[k];
                    }
                }
                __syncwarp();   // the part before has been read out of the stage
#pragma unroll
                for (int k = 0; k < 4; ++k) st_shared_v4(stage_at(lane, k), d2[k], d2[4 + k], d2[8 + k], d2[12 + k]);
                if (part) tc_fence_before();
                __syncwarp();
                if (part && lane == 0) {
                    mbar_arrive(&d_empty[b]);
                    mbar_arrive(&x_empty[b]);
                    mbar_arrive(&sum_empty[u & 3]);
                }
                const int p = w.p0(u) + half * 32 + part * 16 + m * 4;
                float4 s[4];
#pragma unroll
                for (int k = 0; k < 4; ++k)
                    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(s[k].x), "=f"(s[k].y), "=f"(s[k].z), "=f"(s[k].w) : "r"(stage_at(k * 8 + (lane >> 2), m)));
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const float4 v = x[part * 4 + k];
                    if (p < a.vdim && 8 * k < left) *reinterpret_cast<float4*>(dst + 8ll * k * ld_o + p) = make_float4(fmaf(Dh, v.x, s[k].x), fmaf(Dh, v.y, s[k].y), fmaf(Dh, v.z, s[k].z), fmaf(Dh, v.w, s[k].w));
                }
            }
            if (u + 1 < w.count) load(u + 1);
            __syncwarp();
        }
    } else if (warp == 24) {
        constexpr uint32_t idesc = make_idesc_f16(128, kStCols) | (2u << 7) | (2u << 10);   // tf32 operands
        const uint64_t c_desc = make_kmajor_sw128_desc(smem_u32(smem)), x_desc = make_kmajor_sw128_desc(smem_u32(smem + kSoOffX)), s_desc = make_kmajor_sw128_desc(smem_u32(smem + kSoOffS));
        const int n = __shfl_sync(0xffffffffu, w.count, 0), nk = __shfl_sync(0xffffffffu, (a.n_state + 7) / 8, 0);
        const bool leader = elect_one();
        mbar_wait_or_leave(c_full, 0u, dead);
        tc_fence_after();
        if (leader) {   // C . B; B lies where the states go
            constexpr uint32_t idesc_cb = make_idesc_f16(128, 128) | (2u << 7) | (2u << 10);
#pragma unroll 1
            for (int k = 0; k < nk; ++k) {
                const uint64_t o = (uint64_t)((k >> 2) * (16384 >> 4) + 2 * (k & 3));
                umma_tf32(tmem + kSoCB, c_desc + o, s_desc + o, idesc_cb, k > 0 ? 1u : 0u);
            }
            umma_commit(cb_full);
        }
        __syncwarp();
#pragma unroll 1
        for (int u = 0; u < n; ++u) {
            const uint32_t b = (uint32_t)u & 1u, ph = (uint32_t)(u >> 1) & 1u, d = tmem + kSoD + b * 128u;
            const uint64_t xd = x_desc + (uint64_t)(b * (kStUnit >> 4)), sd = s_desc + (uint64_t)(b * (kStUnit >> 4));
            mbar_wait_or_leave(&d_empty[b], ph ^ 1u, dead);
            mbar_wait_or_leave(&s_full[b], ph, dead);
            tc_fence_after();
            if (leader) {
#pragma unroll 1
                for (int k = 0; k < nk; ++k)
                    umma_tf32(d, c_desc + (uint64_t)((k >> 2) * (16384 >> 4) + 2 * (k & 3)), sd + (uint64_t)((k >> 2) * (8192 >> 4) + 2 * (k & 3)), idesc, k > 0 ? 1u : 0u);
                umma_commit(&s_empty[b]);
            }
            __syncwarp();
            mbar_wait_or_leave(&x_full[b], ph, dead);
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                mbar_wait_or_leave(&m_full[q], (uint32_t)u & 1u, dead);
                tc_fence_after();
                if (leader) {
#pragma unroll
                    for (int k = 0; k < 4; ++k)
                        umma_tf32_ts(d + 64u, tmem + kSoM + (uint32_t)(q * 32 + k * 8), xd + (uint64_t)(q * (8192 >> 4) + 2 * k), idesc, q > 0 || k > 0 ? 1u : 0u);
                    umma_commit(&m_empty[q]);
                }
                __syncwarp();
            }
            if (leader) {
                umma_commit(&x_empty[b]);
                umma_commit(&d_full[b]);
            }
            __syncwarp();
        }
    } else {
        if (lane == 0) {
            mbar_expect_tx(c_full, 2 * kStImg);
            bulk_g2s(smem, reinterpret_cast<const unsigned char*>(t.c_img) + (w.place * a.groups + w.g) * kStImg, kStImg, c_full);
            bulk_g2s(smem + kSoOffS, reinterpret_cast<const unsigned char*>(t.b_img) + (w.place * a.groups + w.g) * kStImg, kStImg, c_full);
        }
        __syncwarp();
#pragma unroll 1
        for (int u = 0; u < w.count; ++u) {
            const int b = u & 1;
            mbar_wait_or_leave(&sum_empty[u & 3], ((uint32_t)(u >> 2) & 1u) ^ 1u, dead);
            if (__any_sync(0xffffffffu, *dead)) break;
            if (lane == 0) {
                asked[0] = u + 1;
                mbar_expect_tx(&sum_full[u & 3], kStSums);
                bulk_g2s(smem + kSoOffSums + (u & 3) * kStSums, t.sums + (w.place * a.heads + w.head(u)) * (kStSums / 4), kStSums, &sum_full[u & 3]);
            }
            __syncwarp();
            if (u == 0) mbar_wait_or_leave(cb_full, 0u, dead);   // B has been read
            mbar_wait_or_leave(&s_empty[b], ((uint32_t)(u >> 1) & 1u) ^ 1u, dead);
            if (__any_sync(0xffffffffu, *dead)) break;
            if (lane == 0) {
                asked[1] = u + 1;
                mbar_expect_tx(&s_full[b], kStUnit);
                bulk_g2s(smem + kSoOffS + b * kStUnit, reinterpret_cast<const unsigned char*>(t.states) + (w.place * ((size_t)a.heads * a.col_blocks) + w.unit(u)) * kStUnit, kStUnit, &s_full[b]);
            }
            __syncwarp();
        }
    }
    __syncthreads();
    if (*dead) {   // what is under way lands first
        if (warp == 25) {
            mbar_wait_limited(c_full, 0u);
            for (int u = max(0, asked[0] - 4); u < asked[0]; ++u) mbar_wait_limited(&sum_full[u & 3], (uint32_t)(u >> 2) & 1u);
            for (int u = max(0, asked[1] - 2); u < asked[1]; ++u) mbar_wait_limited(&s_full[u & 1], (uint32_t)(u >> 1) & 1u);
        } else if (warp == 24) {
            if (elect_one()) umma_commit(drained);
            mbar_wait_limited(drained, 0u);
        }
        __syncthreads();
    }
    tc_fence_after();
    if (warp == 24) tmem_dealloc(tmem, 512);
}

size_t ssd_scan_tc_bytes(int n_tokens, int n_entries, int heads, int groups, int vdim, int n_state) {
    if (n_state > 128 || n_state <= 32 || vdim % 4) return 0;
    const size_t places = (size_t)n_tokens / kStChunk + (size_t)n_entries + 1, units = (size_t)heads * ((vdim + kStCols - 1) / kStCols);
    return places * ((size_t)groups * 3 * kStImg + (size_t)heads * kStSums + units * kStUnit) + 256;
}

// units per CTA: the rounds of CTAs, one per SM, times what a CTA takes, three units' time for what its units share (state and out: 8 us before the first
// unit, 2 to 4 us each)
int ssd_tc_units(int n_tokens, int n_entries, int longest_entry, int heads, int groups, int vdim, int sms) {
    const long long places = (long long)n_tokens / kStChunk + n_entries + 1, chunks = (longest_entry + kStChunk - 1) / kStChunk;
    const long long some_chunks = std::min<long long>(chunks * n_entries, places - 1), per_group = (long long)heads * ((vdim + kStCols - 1) / kStCols) / groups;
    long long per = 1, best = LLONG_MAX;
    for (long long u = 1; u <= std::min<long long>(per_group, 64); ++u) {
        const long long cost = (some_chunks * groups * ((per_group + u - 1) / u) + sms - 1) / sms * (u + 3);
        if (cost < best) { best = cost; per = u; }
    }
    return (int)per;
}

int ssd_scan_tc(const SS& s, const b200_ssd_scan_args& p, cudaStream_t stream) {
    auto al16 = [](const void* q) { return (reinterpret_cast<uintptr_t>(q) & 15u) == 0; };
    // n_state: the products' rows are padded to 128. us here / in chunks of 64, 2 entries, 2048 tokens, 64 heads: 16 states 66 / 61, 32 states 66 / 69, 64 states 69 / 92; 8 entries of 150
    // tokens, 8 heads of 128 columns: 27 / 22, 28 / 24, 28 / 28
    if (p.n_state > 128 || p.n_state <= 32 || p.vdim % 4 || p.ld_u % 4 || p.x_off % 4 || !al16(p.u) || !al16(p.out) || !al16(p.state) || !p.workspace) return -1;
    const long long places = (long long)p.n_tokens / kStChunk + p.n_entries + 1, col_blocks = (p.vdim + kStCols - 1) / kStCols, all_units = p.heads * col_blocks;
    const long long chunks = (p.longest_entry + kStChunk - 1) / kStChunk, per_group = all_units / p.groups;
    const size_t pad = (256 - (reinterpret_cast<uintptr_t>(p.workspace) & 255u)) & 255u;
    const size_t need = ssd_scan_tc_bytes(p.n_tokens, p.n_entries, p.heads, p.groups, p.vdim, p.n_state);
    const long long jobs = p.n_entries * (8ll * p.groups + (p.heads + 3) / 4);
    if (p.workspace_bytes < need || chunks > 65535 || p.n_entries > 65535 || jobs > 0x7fffffffll) return -1;
    SsTc t{};
    t.s = s;
    t.s.col_blocks = (int)col_blocks;
    const long long per = ssd_tc_units(p.n_tokens, p.n_entries, p.longest_entry, p.heads, p.groups, p.vdim, sm_count());
    const long long blocks = (long long)p.groups * ((per_group + per - 1) / per);
    t.blocks = (int)blocks;
    if (blocks * p.n_entries > 0x7fffffffll || all_units * 4 > 0x7fffffffll) return -1;
    float* at = reinterpret_cast<float*>(reinterpret_cast<unsigned char*>(p.workspace) + pad);
    auto take = [&](size_t bytes) { float* r = at; at += bytes / 4; return r; };
    t.states = take((size_t)places * all_units * kStUnit);
    t.c_img = take((size_t)places * p.groups * kStImg);
    t.bt_img = take((size_t)places * p.groups * kStImg);
    t.b_img = take((size_t)places * p.groups * kStImg);
    t.sums = take((size_t)places * p.heads * kStSums);
    static unsigned long long d1 = 0, d2 = 0;
    cudaError_t e = ensure_max_dynamic_smem((const void*)ssd_tc_state_kernel, kSuSmem, d1);
    if (e == cudaSuccess) e = ensure_max_dynamic_smem((const void*)ssd_tc_out_kernel, kSoSmem, d2);
    const dim3 grid((unsigned)(blocks * p.n_entries), (unsigned)chunks);
    if (e == cudaSuccess) e = launch_chained(ssd_tc_prep_kernel, dim3((unsigned)jobs, (unsigned)chunks), dim3(128), 0, stream, t);
    if (e == cudaSuccess) e = launch_chained(ssd_tc_state_kernel, grid, dim3(448), kSuSmem, stream, t);
    if (e == cudaSuccess) e = launch_chained(ssd_tc_carry_kernel, dim3((unsigned)(all_units * 4), p.n_entries), dim3(128), 0, stream, t);
    if (e == cudaSuccess) e = launch_chained(ssd_tc_out_kernel, grid, dim3(26 * 32), kSoSmem, stream, t);
    if (e != cudaSuccess) return (int)e;
    count_launch(4);
    return B200_OK;
}

}  // namespace b200
