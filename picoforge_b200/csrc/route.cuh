// Device functions shared by the routing kernels: libm-exact expf / sigmoid and the
// warp-per-token softmax + top-k (picoforge src/qwen4_moe.c:209-247).
#pragma once
#include <cuda_runtime.h>
#include <math_constants.h>
#include <stdint.h>

#include "cuda_shim.h"

namespace qw4 {

// ------------------------------------------------------------------------------------
// expf with glibc's bits.
//
// The reference computes softmax and sigmoid with libm expf (picoforge src/qwen4_moe.c:228,
// src/qwen4_cpu_internal.h:103-106).  glibc's expf is the table-driven double-precision
// algorithm published in ARM's optimized routines (N = 32 table, cubic polynomial); on x86-64
// machines with FMA its products and sums are fused.  Restating it with explicit fma() gives
// the same binary32 result as glibc 2.39 for every input <= 0 (1 120 927 745 values checked
// on the CPU), which is the whole domain used here: z - max <= 0 and -|x|.
// ------------------------------------------------------------------------------------
// In global (not constant) memory: lanes index it with different k, which the constant cache
// would serialise; the 256 bytes stay in L1.
static __device__ const unsigned long long c_exp2_table[32] = {
    0x3ff0000000000000ull, 0x3fefd9b0d3158574ull, 0x3fefb5586cf9890full, 0x3fef9301d0125b51ull,
    0x3fef72b83c7d517bull, 0x3fef54873168b9aaull, 0x3fef387a6e756238ull, 0x3fef1e9df51fdee1ull,
    0x3fef06fe0a31b715ull, 0x3feef1a7373aa9cbull, 0x3feedea64c123422ull, 0x3feece086061892dull,
    0x3feebfdad5362a27ull, 0x3feeb42b569d4f82ull, 0x3feeab07dd485429ull, 0x3feea47eb03a5585ull,
    0x3feea09e667f3bcdull, 0x3fee9f75e8ec5f74ull, 0x3feea11473eb0187ull, 0x3feea589994cce13ull,
    0x3feeace5422aa0dbull, 0x3feeb737b0cdc5e5ull, 0x3feec49182a3f090ull, 0x3feed503b23e255dull,
    0x3feee89f995ad3adull, 0x3feeff76f2fb5e47ull, 0x3fef199bdd85529cull, 0x3fef3720dcef9069ull,
    0x3fef5818dcfba487ull, 0x3fef7c97337b9b5full, 0x3fefa4afa2a490daull, 0x3fefd0765b6e4540ull,
};
// `table` may point at a copy of c_exp2_table in shared memory.
__device__ __forceinline__ float expf_libm_table(float x, const unsigned long long *table) {          // x <= 0 (or +0)
    if (x < -0x1.9fe368p6f) return 0.0f;
    const double inv_ln2_n = 0x1.71547652b82fep+0 * 32.0, shift = 0x1.8p+52;
    const double c0 = 0x1.c6af84b912394p-5 / 32 / 32 / 32, c1 = 0x1.ebfce50fac4f3p-3 / 32 / 32, c2 = 0x1.62e42ff0c52d6p-1 / 32;
    const double xd = (double)x;
    double kd = fma(inv_ln2_n, xd, shift);
    const unsigned long long ki = (unsigned long long)__double_as_longlong(kd);
    kd = __dsub_rn(kd, shift);
    const double r = fma(inv_ln2_n, xd, -kd);
    unsigned long long t = table[ki & 31u];
    t += ki << 47;
    const double s = __longlong_as_double((long long)t);
    const double z = fma(c0, r, c1), r2 = __dmul_rn(r, r);
    double y = fma(c2, r, 1.0);
    y = fma(z, r2, y);
    return __double2float_rn(__dmul_rn(y, s));
}
__device__ __forceinline__ float expf_libm(float x) { return expf_libm_table(x, c_exp2_table); }
__device__ __forceinline__ float sigmoid_libm(float x) {      // src/qwen4_cpu_internal.h:103-106
    if (x >= 0.0f) return __fdiv_rn(1.0f, __fadd_rn(1.0f, expf_libm(-x)));
    const float z = expf_libm(x);
    return __fdiv_rn(z, __fadd_rn(1.0f, z));
}
__device__ __forceinline__ bool finite_f32(float v) { return (__float_as_uint(v) & 0x7f800000u) != 0x7f800000u; }

// Top-k of up to 32 * PL ordered keys held in registers, one warp: lane L holds the keys of elements
// L, L + 32, ... (0: absent).  Sequential selection (k dependent warp reductions) costs a lone warp
// several hundred cycles per round, so the work is arranged in parallel steps instead:
//   1. every lane's maximum, and the k-th largest of those 32 maxima: at least k elements reach it;
//   2. the elements that reach it (typically a dozen or two) are compacted into `cand` (shared memory);
//   3. every candidate counts the candidates that beat it (larger key, or equal key and lower element):
//      that count is its place, and places below k are written out.
// Returns false when more than 64 elements qualify (heavy ties): the caller then selects sequentially.
// cand: 128 words.  ids_out[place] = element, keys_out[place] = key (either may alias nothing else).
template <int PL>
__device__ __forceinline__ uint32_t topk_bound(const uint32_t (&key)[PL], uint32_t lane, uint32_t k) {
    uint32_t m = 0;
#pragma unroll
    for (int i = 0; i < PL; i++) m = max(m, key[i]);
    uint32_t ahead = 0;                                                     // lanes whose maximum beats this lane's
#pragma unroll 8                                                              // all 32 at once: 1% slower in the decode kernel, whose code is fetched cold
    for (int j = 0; j < 32; j++) {
        const uint32_t v = __shfl_sync(0xffffffffu, m, j);
        ahead += (v > m || (v == m && (uint32_t)j < lane)) ? 1u : 0u;
    }
    const uint32_t holder = __ballot_sync(0xffffffffu, ahead == min(k, 32u) - 1u);
    return max(__shfl_sync(0xffffffffu, m, __ffs(holder) - 1), 1u);
}
template <int PL>
__device__ __forceinline__ uint32_t topk_collect(const uint32_t (&key)[PL], uint32_t lane, uint32_t bound, uint32_t *cand) {
    uint32_t count = 0;
    const uint32_t below = (1u << lane) - 1u;
#pragma unroll
    for (int i = 0; i < PL; i++) {
        const bool in = key[i] >= bound;
        const uint32_t votes = __ballot_sync(0xffffffffu, in);
        const uint32_t at = count + __popc(votes & below);
        if (in && at < 64) { cand[at] = key[i]; cand[64 + at] = lane + 32u * i; }
        count += __popc(votes);
    }
    __syncwarp();
    return count;
}
// `count` <= 64 candidates: (k0, e0) of lane and (k1, e1) of lane + 32 are this lane's, key 0 beyond the last
__device__ __forceinline__ void topk_place(const uint32_t *cand, uint32_t count, uint32_t lane, uint32_t k, uint32_t *ids_out, uint32_t *keys_out) {
    const uint32_t k0 = lane < count ? cand[lane] : 0u, e0 = cand[64 + lane];
    const uint32_t k1 = lane + 32 < count ? cand[lane + 32] : 0u, e1 = cand[96 + lane];
    uint32_t place0 = 0, place1 = 0;
#pragma unroll 4
    for (uint32_t j = 0; j < count; j++) {
        const uint32_t kj = cand[j], ej = cand[64 + j];
        place0 += (kj > k0 || (kj == k0 && ej < e0)) ? 1u : 0u;
        place1 += (kj > k1 || (kj == k1 && ej < e1)) ? 1u : 0u;
    }
    if (lane < count && place0 < k) { ids_out[place0] = e0; if (keys_out) keys_out[place0] = k0; }
    if (lane + 32 < count && place1 < k) { ids_out[place1] = e1; if (keys_out) keys_out[place1] = k1; }
    __syncwarp();
}
template <int PL>
__device__ __forceinline__ bool warp_topk(const uint32_t (&key)[PL], uint32_t lane, uint32_t k, uint32_t *cand, uint32_t *ids_out,
                                          uint32_t *keys_out) {
    const uint32_t count = topk_collect<PL>(key, lane, topk_bound<PL>(key, lane, k), cand);
    if (count > 64) return false;
    topk_place(cand, count, lane, k, ids_out, keys_out);
    return true;
}
// The sequential form: every lane keeps its best three (key, element) pairs, so a selection step is one
// warp maximum and a ballot, and a lane rescans its registers only when it has won three times.
template <int PL>
__device__ __forceinline__ void topk_scan(const uint32_t (&key)[PL], uint32_t lane, uint32_t &b1, uint32_t &e1, uint32_t &b2, uint32_t &e2,
                                          uint32_t &b3, uint32_t &e3) {
    b1 = 0; e1 = 0xffffffffu; b2 = 0; e2 = 0xffffffffu; b3 = 0; e3 = 0xffffffffu;
#pragma unroll
    for (int i = 0; i < PL; i++) {                                         // ascending element: the lowest wins among equals
        const uint32_t k = key[i], e = lane + 32u * i;
        if (k > b1) { b3 = b2; e3 = e2; b2 = b1; e2 = e1; b1 = k; e1 = e; }
        else if (k > b2) { b3 = b2; e3 = e2; b2 = k; e2 = e; }
        else if (k > b3) { b3 = k; e3 = e; }
    }
}
template <int PL>
__device__ __forceinline__ void topk_clear(uint32_t (&key)[PL], uint32_t index) {
#pragma unroll
    for (int i = 0; i < PL; i++) if ((uint32_t)i == index) key[i] = 0;
}
template <int PL>
__device__ __noinline__ void warp_topk_sequential(uint32_t (&key)[PL], uint32_t lane, uint32_t k, uint32_t *ids_out, uint32_t *keys_out) {
    uint32_t b1, e1, b2, e2, b3, e3, spare = 2;
    topk_scan<PL>(key, lane, b1, e1, b2, e2, b3, e3);
#pragma unroll 1
    for (uint32_t slot = 0; slot < k; slot++) {
        const uint32_t top = __reduce_max_sync(0xffffffffu, b1);
        const uint32_t e_win = __reduce_min_sync(0xffffffffu, b1 == top ? e1 : 0xffffffffu);
        if (lane == 0) { ids_out[slot] = e_win; if (keys_out) keys_out[slot] = top; }
        if ((e_win & 31u) == lane) {
            topk_clear<PL>(key, e_win >> 5);
            if (spare) { b1 = b2; e1 = e2; b2 = b3; e2 = e3; spare--; }
            else { topk_scan<PL>(key, lane, b1, e1, b2, e2, b3, e3); spare = 2; }
        }
    }
    __syncwarp();
}

// Softmax, top-k and renormalisation of the rows row0 .. row0 + rows - 1 (at most 16) of a batch by one CTA of NW warps, for
// experts <= 512 and k <= 32; src/qwen4_moe.c:209-247 with its order of operations: ties go to the lower id, and with `exact`
// the exp-sum runs serially over e = 0..E-1 (the reference's bits); otherwise it is a tree sum.
//
// The serial sum (512 dependent additions, 2.1 k cycles) is the one part that cannot be cut, so all else is laid around it: the exps are
// spread over the CTA's warps (every warp finds its row's maximum for itself), the sums of the CTA's rows run in the lanes of
// one warp, and while they run the other warps pick the candidates for the top-k by exp value.  The division by the sum is
// monotone but may make equal what was not, so everything within 2^-20 of the bound is a candidate, and only the candidates
// (a dozen or two) are divided and ranked, by quotient and id.  Rows with very small k-th values or more than 64
// candidates are divided in full and selected one by one.
//
// load(row, e) gives a logit; emit(row, slot, id, weight) takes a result (rows with a nonfinite logit emit nothing: the row is
// recorded in the status words and its bit is set in the result, which is CTA-uniform).  probs: the softmax itself, or nullptr.
constexpr uint32_t RT_PITCH = 516;                              // floats per row of exps: the pad keeps the summing lanes' reads apart
struct __align__(16) RouteShared {
    unsigned long long table[32];
    float sum[16];
    uint32_t count[16], bad;
    uint32_t cand[16][128], ids[16][32], keys[16][32];
};
// ((p[0] + p[1]) + p[2]) + ... of n floats in shared memory (16-byte aligned, 512 of them readable).  The next 32 values are on their way while
// 32 are added: the statements are volatile so that the reads stay where they stand, between the additions (left to itself the compiler
// gathers them and a read's latency shows in every turn: 6.2 cycles per value instead of 4.25).
__device__ __forceinline__ float serial_sum(const float *p, uint32_t n) {
    const uint32_t base = (uint32_t)__cvta_generic_to_shared(p);
    float4 v[2][8];
    auto read = [&](float4 &to, uint32_t i) {
        asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(to.x), "=f"(to.y), "=f"(to.z), "=f"(to.w) : "r"(base + i * 4u));
    };
    float sum = 0.0f;
    auto add = [&](float t) { asm volatile("add.rn.f32 %0, %0, %1;" : "+f"(sum) : "f"(t)); };
#pragma unroll
    for (int j = 0; j < 8; j++) read(v[0][j], 4 * j);
    uint32_t e = 0;
#pragma unroll 1
    for (; e + 64 <= n; e += 64) {
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const uint32_t next = min(e + 32u * h + 32u, 480u);
#pragma unroll
            for (int j = 0; j < 8; j++) {
                add(v[h][j].x); read(v[h ^ 1][j], next + 4 * j);
                add(v[h][j].y); add(v[h][j].z); add(v[h][j].w);
            }
        }
    }
    for (; e < n; e++) add(p[e]);
    return sum;
}
template <int NW, typename Load, typename Emit>
__device__ __forceinline__ uint32_t route_rows(uint32_t row0, uint32_t rows, uint32_t E, uint32_t k, int norm, bool exact, float *es, RouteShared &s,
                                               uint32_t *status, float *probs, Load load, Emit emit) {
    constexpr int PL = 16;
    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31u;
    if (tid < 32) s.table[tid] = c_exp2_table[tid];
    if (tid == 0) s.bad = 0;
    const uint32_t per_row = NW / rows, r = warp / per_row, sub = warp % per_row;          // warps on one row (rows <= NW)
    float m = -CUDART_INF_F, z[PL];
    bool bad = false;
    if (r < rows) {
#pragma unroll
        for (int i = 0; i < PL; i++) { const uint32_t e = lane + 32u * i; z[i] = e < E ? load(row0 + r, e) : -CUDART_INF_F; }
#pragma unroll
        for (int i = 0; i < PL; i++) { bad |= lane + 32u * i < E && !finite_f32(z[i]); m = fmaxf(m, z[i]); }
        for (int o = 16; o; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
        bad = __any_sync(0xffffffffu, bad);
    }
    __syncthreads();
    if (bad && lane == 0 && sub == 0) { atomicOr(status, QW4SH_ERR_NONFINITE); atomicMin(status + 1, row0 + r); atomicOr(&s.bad, 1u << r); }
    if (r < rows)
#pragma unroll 1
        for (uint32_t i = sub; i < PL; i += per_row) {
            const uint32_t e = lane + 32u * i;
            float zi = z[0];                                     // register i: sixteen selects, where a second read of the logit is a round trip to L2
#pragma unroll
            for (int j = 1; j < PL; j++) zi = i == (uint32_t)j ? z[j] : zi;
            es[r * RT_PITCH + e] = e < E && !bad ? expf_libm_table(__fsub_rn(zi, m), s.table) : 0.0f;
        }
    __syncthreads();
    const uint32_t bad_rows = s.bad;
    if (warp == 0) {
        if (exact) {
            if (lane < rows) s.sum[lane] = serial_sum(es + lane * RT_PITCH, E);
        } else {
            for (uint32_t q = 0; q < rows; q++) {
                float sum = 0.0f;
#pragma unroll 4
                for (uint32_t e = lane; e < 512; e += 32) sum += es[q * RT_PITCH + e];
                for (int o = 16; o; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
                if (lane == 0) s.sum[q] = sum;
            }
        }
    } else {
        for (uint32_t q = warp - 1; q < rows; q += NW - 1) {
            uint32_t key[PL];                                   // bits of the exp (>= 0: ordered as integers) + 1, 0: absent
#pragma unroll
            for (int i = 0; i < PL; i++) { const uint32_t e = lane + 32u * i; key[i] = e < E ? __float_as_uint(es[q * RT_PITCH + e]) + 1u : 0u; }
            const float bound = __uint_as_float(topk_bound<PL>(key, lane, k) - 1u);
            const uint32_t count = bound > 1e-30f ? topk_collect<PL>(key, lane, __float_as_uint(bound * 0x1.ffffep-1f) + 1u, s.cand[q]) : 65u;
            if (lane == 0) s.count[q] = count;
        }
    }
    __syncthreads();
    if (probs)
        for (uint32_t q = 0; q < rows; q++)
            if (!((bad_rows >> q) & 1u)) for (uint32_t e = tid; e < E; e += NW * 32) probs[(uint64_t)(row0 + q) * E + e] = __fdiv_rn(es[q * RT_PITCH + e], s.sum[q]);
    if (warp < rows && !((bad_rows >> warp) & 1u)) {
        const uint32_t w = warp;
        const uint32_t count = s.count[w];
        const float sum = s.sum[w];
        uint32_t *cand = s.cand[w];
        if (count <= 64) {
            for (uint32_t j = lane; j < count; j += 32) cand[j] = __float_as_uint(__fdiv_rn(__uint_as_float(cand[j] - 1u), sum)) + 1u;
            __syncwarp();
            topk_place(cand, count, lane, k, s.ids[w], s.keys[w]);
        } else {
            uint32_t key[PL];
#pragma unroll
            for (int i = 0; i < PL; i++) { const uint32_t e = lane + 32u * i; key[i] = e < E ? __float_as_uint(__fdiv_rn(es[w * RT_PITCH + e], sum)) + 1u : 0u; }
            warp_topk_sequential<PL>(key, lane, k, s.ids[w], s.keys[w]);
        }
        const float mine = lane < k ? __uint_as_float(s.keys[w][lane] - 1u) : 0.0f;
        float selected = 0.0f;
#pragma unroll 4
        for (uint32_t slot = 0; slot < k; slot++) selected = __fadd_rn(selected, __shfl_sync(0xffffffffu, mine, slot));        // slot order
        if (lane < k) emit(row0 + w, lane, s.ids[w][lane], norm ? __fdiv_rn(mine, selected) : mine);
    }
    return bad_rows;
}

}  // namespace qw4
