// Expert products of every batch beyond the one-kernel decode path, on the 5th-generation tensor cores (sm_100a):
// packed weights -> exact integers in TMEM -> tcgen05.mma against fp16 hi + lo activations -> FP32 scales.
//
// A GGUF block weight is d * (sc * q) - dmin * m with small integers sc, q, m (Q4_K: sc * q <= 945; Q2_K: <= 45;
// IQ2_XXS: (2 s + 1) * magnitude <= 1333, sign folded in, no minimum), so A = sc * q and the minima m are EXACT in fp16,
// and an activation is carried as fp16 hi + lo after a power-of-two scale that puts the row's largest value into
// [512, 1024): hi + lo is then within half a unit in the last place of the FP32 value over 34 bits of range.  fp16
// super-scales (and the rows' powers of two) are applied in FP32 when a block's accumulators are read back.
//
// What bounds it, measured on a B200 (tcgen05.mma, M 128, K 16, one issuing thread, 256 in a row): with A in shared memory an
// instruction costs 39 cycles at N 16 and 48 at N 64 (the 4 KB of A have to be read); with A in TMEM 9.6 at N 16, 16.5 at
// N 32, 32 at N 64: the full rate at any N.  (An issue loop behind `lane == 0` costs 58 cycles an instruction whatever
// else, and cost the previous form of this kernel 144: the loop must be warp-uniform around elect.sync.)  Hence:
//   - weights sit on M, and the dequantising thread of weight row r writes its row straight into TMEM lane r
//     (tcgen05.st): no operand tile in shared memory, no swizzle, one thread owns one row's scales;
//   - tokens sit on N, 16 or 32 to a group: hi and lo are two MMAs into ONE accumulator, so the read-back is N wide;
//   - per 128 x 256 weights the dequantiser needs about 1500 warp instructions (380 cycles on four schedulers), the MMAs 326
//     (N 16) or 561 (N 32) cycles, HBM 804 (Q4_K), 469 (Q2_K), 369 (IQ2_XXS) cycles at 6.45 TB/s over 148 SMs: the three sides are
//     near each other, and all of them run at the same time.
//
// Work item: one group (<= 32 token rows of one expert) x two 128-row tiles that share the activations: gate rows and the
// same up rows (mode 0: SwiGLU stays in the CTA), or two neighbouring row tiles (mode 1, down).  Sharing halves the
// activation traffic from L2, and the two tiles take turns on the tensor pipe, so one is read back while the other is
// multiplied.  CTAs are persistent and walk the item list with a stride.
//
// Measured, routed experts of 1024 tokens: Q4_K (Zipf) gate/up 484 -> 151 us, down 275 -> 97; Q2_K gate/up 579 -> 188 us.  A
// step (128 columns of both tiles) takes about 1500 cycles where its MMAs take 528 and its dequantising 560: the rest is the
// hand-over between the two (barrier answers behind the shared-memory and TMEM traffic, 100 to 200 cycles each way, and two A
// slots per tile are all that TMEM holds beside the accumulators).
//
// Warps (21; 25 for IQ2_XXS, whose dequantiser takes three sets of four):
//   0-7         dequantise: each set of four takes (step, tile) pairs in turn (TMEM lane = weight row), 128 columns at a time into two A slots per tile
//   next 8      read tile 0 / 1 back (tcgen05.ld), scale, accumulate; SwiGLU + split of the activation, or the store
//   next 1      TMA of the packed rows;  next 2: tcgen05.mma issue, one warp per tile;  last 2: activation rows (cp.async gathers of hi and lo)
//
// A unit is the span of columns between two read-backs: 256 (mode 0: a block, one row scale per token) or 128 (mode 1: the
// activation of a token has one power of two per 128 columns, because those come out of different CTAs).  The minima of a
// unit are one more K = 16 MMA (hi and lo) against sums over 16 (mode 0) or 8 (mode 1) columns of the activation.
//
// Every mbarrier wait is bounded (about a second); a role that gives up records QW4SH_ERR_STATE, all roles leave their
// loops, copies in flight are waited for and TMEM is freed on every path.
#pragma once
#include <cuda.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "cuda_shim.h"
#include "formats.cuh"

namespace qw4 {

// Formats of the kernel: the GGUF types, and the wide form of everything else (see experts_tc.cu).
constexpr uint32_t T_WIDE = 117;

constexpr uint32_t XROWS = 128;                              // weight rows per tile
constexpr uint32_t XTOK = 32;                                // most token rows per group
constexpr uint32_t XSLOTS = 2;                               // A slots of one step per tile
// TMEM columns: A [2 slots][2 tiles][64], minima [2][2 tiles][8], Q [2 buffers][2 tiles][32], M [2 tiles][32]
constexpr uint32_t XT_A = 0, XT_AM = 256, XT_Q = 320, XT_M = 448, XT_COLS = 512;

struct XGroup { uint32_t expert, first, count, pad; };

// Per-format geometry: columns per TMA stage, bytes per tile and stage, stages, activation slots of a step, 64-column chunks per
// step (the wide form's hi and lo halves of one chunk fill a slot), sets of four dequantising warps, bytes for look-up tables and
// for the fp16 scales that the resident image keeps apart from the codes.
template <uint32_t F> struct XFmt;
template <> struct XFmt<T_Q4_K>    { static constexpr uint32_t COLS = 256, TILE = 128 * 144, STAGES = 3, BSLOTS = 4, CPS = 2, SETS = 2, TABLES = 0, SIDE = 0, SIDE_BLOCK = 0; static constexpr bool MIN = true; };
template <> struct XFmt<T_Q2_K>    { static constexpr uint32_t COLS = 256, TILE = 128 * 80, STAGES = 4, BSLOTS = 4, CPS = 2, SETS = 2, TABLES = 0, SIDE = 32768, SIDE_BLOCK = 4; static constexpr bool MIN = true; };
template <> struct XFmt<T_IQ2_XXS> { static constexpr uint32_t COLS = 512, TILE = 128 * 128, STAGES = 2, BSLOTS = 4, CPS = 2, SETS = 3, TABLES = 49152, SIDE = 16384, SIDE_BLOCK = 2; static constexpr bool MIN = false; };
template <> struct XFmt<T_WIDE>    { static constexpr uint32_t COLS = 64, TILE = 128 * 256, STAGES = 2, BSLOTS = 8, CPS = 1, SETS = 2, TABLES = 0, SIDE = 0, SIDE_BLOCK = 0; static constexpr bool MIN = false; };
// warps of a launch of format F: dequantise, read back, TMA, MMA (2), activations (2)
template <uint32_t F> struct XRole {
    static constexpr int EPI = 4 * XFmt<F>::SETS, TMA = EPI + 8, MMA = TMA + 1, ACT = MMA + 2, WARPS = ACT + 2, THREADS = 32 * WARPS;
};

constexpr uint32_t XPITCH = 136;                             // floats per token of the hand-over tile: column c at c + c / 16, no bank conflicts either way
constexpr uint32_t XB_ONE = XTOK * 128;                      // 4096: hi (or lo) rows of one activation slot, 128-byte swizzle
constexpr uint32_t XS_ONE = 2 * XTOK * 16;                   // 1024: hi (or lo) column sums of one unit
// shared-memory map
constexpr uint32_t XM_BARS = 0, XM_TMEM = 512, XM_DSC = 1024 /* [2][4][128] words */, XM_SUMS = XM_DSC + 4096 /* [4][2] x XS_ONE */,
                   XM_BSC = XM_SUMS + 4 * 2 * XS_ONE /* [8][32] floats: unit scales of mode 1 */, XM_SHARE = XM_BSC + 1024 /* [8 warps][32] */, XM_HAND = XM_SHARE + 1024,
                   XM_B = (XM_HAND + XTOK * XPITCH * 4 + 1023) & ~1023u;
template <uint32_t F> __host__ __device__ constexpr uint32_t xm_tables() { return XM_B + XFmt<F>::BSLOTS * XFmt<F>::CPS * 2 * XB_ONE; }
template <uint32_t F> __host__ __device__ constexpr uint32_t xm_side() { return xm_tables<F>() + XFmt<F>::TABLES; }
template <uint32_t F> __host__ __device__ constexpr uint32_t xm_weights() { return xm_side<F>() + XFmt<F>::SIDE; }
template <uint32_t F> __host__ __device__ constexpr uint32_t xm_total() { return xm_weights<F>() + XFmt<F>::STAGES * 2 * XFmt<F>::TILE; }
static_assert(xm_total<T_Q4_K>() <= 232448 && xm_total<T_Q2_K>() <= 232448 && xm_total<T_IQ2_XXS>() <= 232448 && xm_total<T_WIDE>() <= 232448, "shared memory");
static_assert(xm_weights<T_Q4_K>() % 1024 == 0 && xm_weights<T_IQ2_XXS>() % 1024 == 0, "swizzled stages need 1024-byte alignment");

struct XMaps { CUtensorMap m[2][2]; };                       // [gate or down, up][section]

struct XArgs {
    DevTensor w0, w1;                                        // gate and up, or down twice
    const float *row_scale0, *row_scale1;                    // wide form: power of two of a weight row
    uint32_t units;                                          // units per item: logical K / 256 (mode 0), / 128 (mode 1)
    uint32_t tiles;                                          // items per group
    uint32_t k_div;                                          // input row = pair / k_div
    const XGroup *groups;
    const uint32_t *n_groups;
    const uint32_t *row_to_pair;                             // nullptr: pair = row (shared expert)
    const __half *in_hi, *in_lo;                             // [rows][K], column order of xperm
    const __half *sum_hi, *sum_lo;                           // [rows][units * 16]
    const float *in_scale;                                   // mode 0: [rows]; mode 1: [rows][units]; what a value is to be multiplied by
    uint32_t in_pitch;                                       // K
    __half *out_hi, *out_lo, *osum_hi, *osum_lo;             // mode 0: the activation as the down product wants it
    float *out_scale;                                        // mode 0: [pairs][n_out / 128]
    float *out;                                              // mode 1: [pairs][n_out]
    uint32_t *status;
    unsigned long long *debug;                               // optional [32]: cycles CTA 0's roles spent in their waits
};

// Column order inside a group of eight (an involution up to the pairing): what byte extraction from a word yields.
__host__ __device__ __forceinline__ uint32_t xperm(uint32_t j) { return (j & ~7u) | ((0x75643120u >> (4 * (j & 7u))) & 7u); }

// ---- PTX helpers ------------------------------------------------------------------------------
__device__ __forceinline__ uint32_t xs_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void xbar_init(uint32_t bar, uint32_t count) { asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory"); }
__device__ __forceinline__ void xbar_arrive(uint32_t bar) { asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory"); }
__device__ __forceinline__ void xbar_arrive_n(uint32_t bar, uint32_t n) { asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(n) : "memory"); }
__device__ __forceinline__ void xbar_expect(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool xbar_try(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}" : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    return ok != 0;
}
__device__ __forceinline__ bool xbar_test(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile("{\n .reg .pred p;\n mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}" : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    return ok != 0;
}
// Bounded wait; `dead` (shared memory) is set by whoever gives up, and ends every other wait.
__device__ __noinline__ bool xbar_wait_slow(uint32_t bar, uint32_t parity, volatile uint32_t *dead, uint32_t *status) {
    const long long start = clock64();
    while (!xbar_try(bar, parity)) {
        if (*dead) return false;
        if (clock64() - start > (1ll << 31)) { *dead = 1; atomicOr(status, QW4SH_ERR_STATE); return false; }
    }
    return true;
}
__device__ __forceinline__ bool xbar_wait(uint32_t bar, uint32_t parity, volatile uint32_t *dead, uint32_t *status) {
    return xbar_try(bar, parity) || xbar_wait_slow(bar, parity, dead, status);
}
__device__ __forceinline__ uint32_t xelect() {
    uint32_t r;
    asm volatile("{\n .reg .pred p;\n elect.sync _|p, 0xffffffff;\n selp.u32 %0, 1, 0, p;\n}" : "=r"(r));
    return r;
}
__device__ __forceinline__ void xtma_2d(uint32_t dst, const CUtensorMap *map, uint32_t x, uint32_t y, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
                 ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(bar) : "memory");
}
__device__ __forceinline__ void xtma_3d(uint32_t dst, const CUtensorMap *map, uint32_t x, uint32_t y, uint32_t z, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
                 ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(z), "r"(bar) : "memory");
}
__device__ __forceinline__ void xbulk(uint32_t dst, const void *src, uint32_t bytes, uint32_t bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst), "l"(src), "r"(bytes), "r"(bar) : "memory");
}
__device__ __forceinline__ void xcp16(uint32_t dst, const void *src, uint32_t src_bytes) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(src_bytes) : "memory");
}
__device__ __forceinline__ void xtc_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void xtc_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void xtc_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
// D (TMEM) += A (TMEM) x B (shared memory)
__device__ __forceinline__ void xmma(uint32_t d, uint32_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
    asm volatile("{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n}"
                 ::"r"(d), "r"(a), "l"(b), "r"(idesc), "r"(accumulate) : "memory");
}
#define X8(v, o) "r"(v[o]), "r"(v[o + 1]), "r"(v[o + 2]), "r"(v[o + 3]), "r"(v[o + 4]), "r"(v[o + 5]), "r"(v[o + 6]), "r"(v[o + 7])
#define X8O(v, o) "=r"(v[o]), "=r"(v[o + 1]), "=r"(v[o + 2]), "=r"(v[o + 3]), "=r"(v[o + 4]), "=r"(v[o + 5]), "=r"(v[o + 6]), "=r"(v[o + 7])
__device__ __forceinline__ void xst32(uint32_t taddr, const uint32_t (&v)[32]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
                 "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};"
                 ::"r"(taddr), X8(v, 0), X8(v, 8), X8(v, 16), X8(v, 24) : "memory");
}
__device__ __forceinline__ void xst8(uint32_t taddr, const uint32_t (&v)[8]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(taddr), X8(v, 0) : "memory");
}
__device__ __forceinline__ void xst_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
// Sixteen accumulator columns of Q and of M (or of Q alone); load and wait in one statement, so that no use can slip between.
__device__ __forceinline__ void xld_qm(uint32_t q_addr, uint32_t m_addr, uint32_t (&q)[16], uint32_t (&m)[16]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%32];\n"
                 "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%33];\n"
                 "tcgen05.wait::ld.sync.aligned;"
                 : X8O(q, 0), X8O(q, 8), X8O(m, 0), X8O(m, 8) : "r"(q_addr), "r"(m_addr) : "memory");
}
__device__ __forceinline__ void xld_q(uint32_t q_addr, uint32_t (&q)[16]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];\n"
                 "tcgen05.wait::ld.sync.aligned;"
                 : X8O(q, 0), X8O(q, 8) : "r"(q_addr) : "memory");
}
// Shared-memory matrix descriptors (version 1), K-major: rows of 128 bytes with the 128-byte swizzle, eight-row groups 1024 bytes
// apart; and two 16-byte core-matrix columns 512 bytes apart, no swizzle (the column sums).
__device__ __forceinline__ uint64_t xdesc_sw128(uint32_t a) {
    return (uint64_t)((a >> 4) & 0x3fffu) | ((uint64_t)1 << 16) | ((uint64_t)(1024 >> 4) << 32) | (1ull << 46) | (2ull << 61);
}
__device__ __forceinline__ uint64_t xdesc_sums(uint32_t a) {
    return (uint64_t)((a >> 4) & 0x3fffu) | ((uint64_t)((XTOK * 16) >> 4) << 16) | ((uint64_t)(128 >> 4) << 32) | (1ull << 46);
}
__device__ __forceinline__ uint4 xlds128(uint32_t a) {
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a));
    return v;
}
__device__ __forceinline__ uint32_t xlds32(uint32_t a) {
    uint32_t v;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(a));
    return v;
}
__device__ __forceinline__ uint32_t xlds16(uint32_t a) {
    uint32_t v;
    asm volatile("{\n .reg .u16 h;\n ld.shared.u16 h, [%1];\n cvt.u32.u16 %0, h;\n}" : "=r"(v) : "r"(a));
    return v;
}
__device__ __forceinline__ __half2 xh2(uint32_t v) { return *reinterpret_cast<const __half2 *>(&v); }
__device__ __forceinline__ uint32_t xu32(__half2 v) { return *reinterpret_cast<const uint32_t *>(&v); }
__device__ __forceinline__ float xhalf_bits(uint32_t v) { return __half2float(__ushort_as_half((unsigned short)(v & 0xffffu))); }
// bytes i and j of `v` (each < 256) as two exact halves
__device__ __forceinline__ __half2 xbytes2(uint32_t v, uint32_t i, uint32_t j) {
    return __hsub2(xh2(__byte_perm(v, 0x64646464u, 0x4040u | i | (j << 8))), xh2(0x64006400u));
}

// ---- dequantisers: the thread's weight row, one step (two chunks of 64 columns) at a time ---------------------------------------
// load(): packed words and scales of step `sp` of the stage, once per step; chunk(h): 32 words of two halves, the step's columns
// 64 h .. 64 h + 63 (wide form: hi, then lo, of 64 columns); minima(): the unit's 16 slots, on its first step; word(): what the
// read-back multiplies by, {d, dmin} or a float.
template <uint32_t F> struct XDeq;

// Codes masked out in place ARE halves, subnormal ones: a code at bit b of its half is code * 2^(b - 24), and times s * 2^(10 - b) it
// becomes s * code * 2^-14, exactly; the 2^14 goes to the FP32 scale of the read-back.  One logic operation and one multiply
// per two weights (both pipes take two cycles a warp instruction); masking a bias in as well compiles to two logic operations,
// and the logic pipe is the busiest one.
constexpr float XUP = 16384.0f;
__device__ __forceinline__ uint32_t xfold(uint32_t bits, __half2 mul) { return xu32(__hmul2(xh2(bits), mul)); }
__device__ __forceinline__ void xwords(uint32_t (&w)[8], uint4 a, uint4 b) {
    w[0] = a.x; w[1] = a.y; w[2] = a.z; w[3] = a.w; w[4] = b.x; w[5] = b.y; w[6] = b.z; w[7] = b.w;
}

template <> struct XDeq<T_Q4_K> {
    uint32_t sc, mlo, mhi, dd, w[2][8];
    __device__ __forceinline__ void load(uint32_t tile, uint32_t row, const uint8_t *, uint32_t, uint32_t, uint32_t sp, uint32_t) {
        const uint32_t base = tile + row * 144u, at = base + 16 + sp * 64;
        const uint4 h = xlds128(base), qa = xlds128(at), qb = xlds128(at + 16), qc = xlds128(at + 32), qd = xlds128(at + 48);
        dd = h.x;
        sc = sp ? (h.w & 0x0f0f0f0fu) | ((h.y >> 2) & 0x30303030u) : h.y & 0x3f3f3f3fu;
        mlo = h.z & 0x3f3f3f3fu; mhi = ((h.w >> 4) & 0x0f0f0f0fu) | ((h.z >> 2) & 0x30303030u);
        xwords(w[0], qa, qb); xwords(w[1], qc, qd);
    }
    __device__ __forceinline__ void chunk(uint32_t h, uint32_t (&v)[32]) {
        const __half2 m0 = __hmul2(xbytes2(sc, 2 * h, 2 * h), __float2half2_rn(1024.0f)), m1 = __hmul2(xbytes2(sc, 2 * h + 1, 2 * h + 1), __float2half2_rn(64.0f));
#pragma unroll
        for (int j = 0; j < 8; j++) {
            const uint32_t q = w[h][j], r = q >> 8;
            v[2 * j] = xfold(q & 0x000f000fu, m0); v[2 * j + 1] = xfold(r & 0x000f000fu, m0);
            v[16 + 2 * j] = xfold(q & 0x00f000f0u, m1); v[17 + 2 * j] = xfold(r & 0x00f000f0u, m1);
        }
    }
    // mode 0: 16 slots of 16 columns, mode 1 (half block sp): 16 slots of 8 columns; a minimum covers 32 columns
    template <int MODE> __device__ __forceinline__ void minima(uint32_t sp, uint32_t (&v)[8]) {
        const uint32_t half = sp ? mhi : mlo;
#pragma unroll
        for (uint32_t j = 0; j < 8; j++) {
            const uint32_t sub = MODE == 0 ? j : j >> 1, m = MODE == 0 ? (j < 4 ? mlo : mhi) : half;
            v[j] = xu32(xbytes2(m, sub & 3u, sub & 3u));
        }
    }
    __device__ __forceinline__ uint32_t word() const { return dd; }
};

// Q2_K stage: [128][64] code bytes with the 64-byte swizzle, then [128][16] scale bytes; {d, dmin} of all the item's blocks beside the stages
template <> struct XDeq<T_Q2_K> {
    uint32_t q[4], sh[2], dd, w[8];
    __device__ __forceinline__ void load(uint32_t tile, uint32_t row, const uint8_t *, uint32_t side, uint32_t b, uint32_t sp, uint32_t) {
        const uint32_t base = tile + row * 64u, swz = ((row >> 1) & 3u) << 4;
        const uint4 s = xlds128(tile + 8192u + row * 16u), qa = xlds128(base + ((sp * 32u) ^ swz)), qb = xlds128(base + ((sp * 32u + 16u) ^ swz));
        q[0] = s.x; q[1] = s.y; q[2] = s.z; q[3] = s.w;
        sh[0] = sp ? s.z : s.x; sh[1] = sp ? s.w : s.y;
        dd = xlds32(side + b * 4u);
        xwords(w, qa, qb);
    }
    __device__ __forceinline__ void chunk(uint32_t h, uint32_t (&v)[32]) {
        const uint32_t word = sh[h] & 0x0f0f0f0fu;
#pragma unroll
        for (int r = 0; r < 2; r++) {                        // runs of 32 columns: bit pair 2 h + r of the bytes, in place
            const __half2 up = __float2half2_rn((h ? 64.0f : 1024.0f) * (r ? 0.25f : 1.0f));
            const __half2 ma = __hmul2(xbytes2(word, 2 * r, 2 * r), up), mb = __hmul2(xbytes2(word, 2 * r + 1, 2 * r + 1), up);
            const uint32_t mask = (h ? 0x00300030u : 0x00030003u) << (2 * r);
#pragma unroll
            for (int j = 0; j < 8; j++) {
                v[16 * r + 2 * j] = xfold(w[j] & mask, j < 4 ? ma : mb);
                v[16 * r + 2 * j + 1] = xfold((w[j] >> 8) & mask, j < 4 ? ma : mb);
            }
        }
    }
    template <int MODE> __device__ __forceinline__ void minima(uint32_t, uint32_t (&v)[8]) {
#pragma unroll
        for (uint32_t j = 0; j < 8; j++) {                   // a minimum covers 16 columns
            if (MODE == 0) v[j] = xu32(xbytes2((q[j >> 1] >> 4) & 0x0f0f0f0fu, (j & 1u) * 2u, (j & 1u) * 2u + 1u));
            else v[j] = xu32(xbytes2((sh[j >> 2] >> 4) & 0x0f0f0f0fu, j & 3u, j & 3u));
        }
    }
    __device__ __forceinline__ uint32_t word() const { return dd; }
};

// IQ2_XXS stage: [128][128] payload bytes (two blocks) with the 128-byte swizzle on top of the image's own group swizzle.
// Tables in shared memory, copies side by side so that no lanes meet in a bank: 256 codebook vectors of eight halves (eight
// copies of 16 bytes, read 128 bits wide), 128 sign words (32 copies; bits 15 - r and 31 - r are the signs of word r).
template <> struct XDeq<T_IQ2_XXS> {
    uint32_t grid, sign, dd;
    uint4 g[2];
    __device__ __forceinline__ void load(uint32_t tile, uint32_t row, const uint8_t *tables, uint32_t side, uint32_t b, uint32_t sp, uint32_t lane) {
        const uint32_t base = tile + row * 128u, swz = ((((row & 3u) << 1) ^ (row & 7u)) << 4);
        g[0] = xlds128(base + ((sp * 32u) ^ swz)); g[1] = xlds128(base + ((sp * 32u + 16u) ^ swz));       // two groups of 32 columns each
        grid = xs_u32(tables) + (lane & 7u) * 16u; sign = xs_u32(tables) + 32768u + lane * 4u;
        dd = xlds16(side + (2 * b + (sp >> 1)) * 2u);
    }
    __device__ __forceinline__ void chunk(uint32_t h, uint32_t (&v)[32]) {
#pragma unroll
        for (int r = 0; r < 2; r++) {
            const uint32_t index = r ? g[h].z : g[h].x, bits = r ? g[h].w : g[h].y;
            const __half2 s = __hsub2(xh2(((bits >> 27) | 1u) * 0x10001u + 0x64006400u), xh2(0x64006400u));       // 2 * scale + 1
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const uint4 m = xlds128(grid + (k == 0 ? (index << 7) & 0x7f80u : k == 1 ? (index >> 1) & 0x7f80u : k == 2 ? (index >> 9) & 0x7f80u : (index >> 17) & 0x7f80u));
                const uint32_t w = xlds32(sign + ((k == 0 ? bits << 7 : bits >> (7 * k - 7)) & 0x3f80u));
                const uint32_t mm[4] = {m.x, m.y, m.z, m.w};
#pragma unroll
                for (int q = 0; q < 4; q++) v[16 * r + 4 * k + q] = xu32(__hmul2(xh2(mm[q] ^ ((w << q) & 0x80008000u)), s));
            }
        }
    }
    template <int MODE> __device__ __forceinline__ void minima(uint32_t, uint32_t (&)[8]) {}
    __device__ __forceinline__ uint32_t word() const { return dd; }
};

// Wide form: fp16 hi and lo images of the weights (row scaled by a power of two), [128][128 bytes] each with the 128-byte swizzle.
template <> struct XDeq<T_WIDE> {
    uint32_t base, swz, scale;
    __device__ __forceinline__ void load(uint32_t tile, uint32_t row, const uint8_t *, uint32_t row_scale, uint32_t, uint32_t, uint32_t) {
        base = tile + row * 128u; swz = (row & 7u) << 4; scale = row_scale;
    }
    __device__ __forceinline__ void chunk(uint32_t h, uint32_t (&v)[32]) {
#pragma unroll
        for (uint32_t i = 0; i < 8; i++) {
            const uint4 q = xlds128(base + h * 16384u + ((i * 16u) ^ swz));
            v[4 * i] = q.x; v[4 * i + 1] = q.y; v[4 * i + 2] = q.z; v[4 * i + 3] = q.w;
        }
    }
    template <int MODE> __device__ __forceinline__ void minima(uint32_t, uint32_t (&)[8]) {}
    __device__ __forceinline__ uint32_t word() const { return scale; }
};

// The power of two that puts `m` (>= 0, finite) into [512, 1024), and its inverse.
__device__ __forceinline__ void xscale_of(float m, float &up, float &down) {
    const int e = (int)(__float_as_uint(m) >> 23);
    const int biased = m > 0.0f ? min(max(263 - e, 1), 253) : 127;
    up = __uint_as_float((uint32_t)biased << 23); down = __uint_as_float((uint32_t)(254 - biased) << 23);
}
// Eight scaled values -> four words of hi and of lo in the kernel's column order.
__device__ __forceinline__ void xsplit8(const float (&v)[8], uint32_t (&hi)[4], uint32_t (&lo)[4]) {
#pragma unroll
    for (int q = 0; q < 4; q++) {
        const float a = v[(q >> 1) * 4 + (q & 1)], b = v[(q >> 1) * 4 + (q & 1) + 2];
        const __half2 h = __floats2half2_rn(a, b);
        const float2 f = __half22float2(h);
        hi[q] = xu32(h); lo[q] = xu32(__floats2half2_rn(a - f.x, b - f.y));
    }
}

// Wait with the time spent added to a role-local counter when CTA 0 is being profiled.
#define XWAIT(counter, bar, parity) ([&]() { if (!prof) return xbar_wait(bar, parity, dead, a.status); \
    const long long t0_ = clock64(); const bool ok_ = xbar_wait(bar, parity, dead, a.status); counter += clock64() - t0_; return ok_; }())

template <uint32_t F, int MODE>
__device__ __forceinline__ void expert_tc_body(const XMaps &maps, const XArgs &a, uint8_t *smem) {
    using Fm = XFmt<F>;
    using R = XRole<F>;
    constexpr uint32_t UNIT = MODE == 0 ? 256 : 128, CPS = Fm::CPS, SPU = UNIT / (64 * CPS), STCH = Fm::COLS / 64;   // steps per unit, chunks per stage
    constexpr uint32_t BSTEP = CPS * 2 * XB_ONE, NB = Fm::BSLOTS, NBLOG = NB == 8 ? 3 : 2;
    constexpr uint32_t STEP = MODE == 0 ? 128 : 256;                        // weight rows per item
    const uint32_t sbase = xs_u32(smem);
    const uint32_t w_full = sbase + XM_BARS, w_empty = w_full + 8 * Fm::STAGES, full = w_empty + 8 * Fm::STAGES /* [step][tile] */,
                   done = full + 8 * 2 * NB, d_empty = done + 8 * NB /* [buffer][tile] */;
    static_assert(8 * (2 * Fm::STAGES + 3 * NB + 4) <= 512, "barrier block");
    volatile uint32_t *dead = reinterpret_cast<volatile uint32_t *>(smem + XM_TMEM + 8);
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    // items whose apart-lying scales are held: more than the stages reach ahead (a stage holds at least one block of a row)
    const uint32_t ring_mask = (a.w0.k_storage >> 8) <= 8 ? 3u : 1u;
    const bool prof = a.debug && blockIdx.x == 0;
    long long w0 = 0, w1 = 0, w2 = 0;
    const long long t_begin = prof ? clock64() : 0;

    if (tid == 0) {
        for (uint32_t i = 0; i < Fm::STAGES; i++) { xbar_init(w_full + 8 * i, 1); xbar_init(w_empty + 8 * i, 8 * (STCH / CPS)); }
        // a step of a tile is ready when its four dequantising warps and the two activation warps say so: one wait for its products
        for (uint32_t i = 0; i < 2 * NB; i++) xbar_init(full + 8 * i, 6);
        for (uint32_t i = 0; i < NB; i++) xbar_init(done + 8 * i, 2);
        for (uint32_t i = 0; i < 4; i++) xbar_init(d_empty + 8 * i, 4);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        *dead = 0;
    }
    if (F == T_IQ2_XXS) {
        uint8_t *tables = smem + xm_tables<F>();
        for (uint32_t i = tid; i < 256 * 8; i += R::THREADS) {
            const uint32_t levels = c_iq2_levels[i >> 3];
            uint32_t v[4];
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const int c = (q >> 1) * 4 + (q & 1);
                v[q] = xu32(__halves2half2(__ushort2half_rn((unsigned short)iq2_magnitude((levels >> (2 * c)) & 3u)),
                                           __ushort2half_rn((unsigned short)iq2_magnitude((levels >> (2 * c + 4)) & 3u))));
            }
            *reinterpret_cast<uint4 *>(tables + i * 16u) = make_uint4(v[0], v[1], v[2], v[3]);
        }
        for (uint32_t i = tid; i < 128 * 32; i += R::THREADS) {
            const uint32_t s = iq2_signs8(i >> 5);
            uint32_t w = 0;
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const int c = (q >> 1) * 4 + (q & 1);
                w |= ((s >> c) & 1u) << (15 - q) | ((s >> (c + 2)) & 1u) << (31 - q);
            }
            *reinterpret_cast<uint32_t *>(tables + 32768u + i * 4u) = w;
        }
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(sbase + XM_TMEM), "r"(XT_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    xtc_before();
    __syncthreads();
    xtc_after();
    // The down product is launched while gate/up still runs: its CTAs move in as those leave, and fetch and dequantise weights (the groups are
    // older than both) until the activation rows, which alone wait for gate/up's end, hold them up.
    if (MODE == 0) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    constexpr uint32_t tmem = 0;                                            // all 512 columns are this CTA's
    const uint32_t n_items = *a.n_groups * a.tiles;

    if (warp == R::TMA) {
        // ---------------- packed rows ----------------
        const uint32_t steps = (a.units * UNIT + Fm::COLS - 1) / Fm::COLS, el = xelect();
        const uint32_t nb = a.w0.k_storage >> 8, side = 128 * nb * Fm::SIDE_BLOCK;    // bytes of a tile's scales that lie apart from the codes
        uint32_t st = 0, ph = 0, issued = 0, ring = 0;
        bool ok = true;
        for (uint32_t it = blockIdx.x; it < n_items && ok; it += gridDim.x) {
            const uint32_t expert = a.groups[it / a.tiles].expert, row0 = (it % a.tiles) * STEP;
            for (uint32_t s = 0; s < steps; s++) {
                if (!(ok = XWAIT(w0, w_empty + 8 * st, ph ^ 1u))) break;
                const uint32_t bar = w_full + 8 * st;
                if (el) {
                    xbar_expect(bar, 2 * Fm::TILE + (Fm::SIDE && s == 0 ? 2 * side : 0));
#pragma unroll
                    for (uint32_t m = 0; m < 2; m++) {
                        const uint32_t dst = sbase + xm_weights<F>() + (st * 2 + m) * Fm::TILE, y = row0 + (MODE == 1 ? m * 128u : 0u);
                        const CUtensorMap *mp = maps.m[MODE == 0 ? m : 0];
                        if (F == T_Q4_K) xtma_2d(dst, mp, s * 144u, expert * a.w0.n_out + y, bar);
                        else if (F == T_Q2_K) { xtma_3d(dst, mp, s * 64u, y, expert, bar); xtma_3d(dst + 8192u, mp + 1, s * 16u, y, expert, bar); }
                        else if (F == T_IQ2_XXS) xtma_3d(dst, mp, s * 128u, y, expert, bar);
                        else { xtma_2d(dst, mp, s * 64u, expert * a.w0.n_out + y, bar); xtma_2d(dst + 16384u, mp + 1, s * 64u, expert * a.w0.n_out + y, bar); }
                        if (Fm::SIDE && s == 0) {                              // with the item's first stage, for all of its units
                            const DevTensor &w = m == 0 || MODE == 1 ? a.w0 : a.w1;
                            xbulk(sbase + xm_side<F>() + (ring * 2 + m) * side,
                                  w.data + (uint64_t)expert * w.expert_bytes + ((uint64_t)w.n_out * (F == T_Q2_K ? 80u : 64u) + (uint64_t)y * Fm::SIDE_BLOCK) * nb, side, bar);
                        }
                    }
                }
                __syncwarp();
                issued++;
                if (++st == Fm::STAGES) { st = 0; ph ^= 1u; }
            }
            ring = (ring + 1) & ring_mask;
        }
        // leave only when the copies issued last have landed (a bounded wait of its own: `dead` does not end it)
        __shared__ uint32_t never;
        if (lane == 0) never = 0;
        __syncwarp();
        for (uint32_t i = 0; i < Fm::STAGES && i < issued; i++) {
            if (st == 0) { st = Fm::STAGES; ph ^= 1u; }
            st--;
            xbar_wait(w_full + 8 * st, ph, &never, a.status);
        }
    } else if (warp >= R::ACT) {
        // ---------------- activation rows: hi by one warp, lo by the other ----------------
        // eight lanes take the 128 bytes of a row, so an instruction touches four lines of the cache and not thirty-two
        const uint32_t part = warp - R::ACT, piece = lane & 7u, sub = lane >> 3;
        if (MODE == 1) asm volatile("griddepcontrol.wait;" ::: "memory");
        constexpr uint32_t LAG = 2;                                           // steps between a copy's issue and its hand-over
        uint32_t n = 0, un = 0;
        bool ok = true;
        auto hand_over = [&](uint32_t step) {                                 // this thread's copies of the step have landed
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane < 2) xbar_arrive(full + 8 * ((step & (NB - 1)) * 2 + lane));
        };
        const __half *in = (part ? a.in_lo : a.in_hi) + piece * 8, *sums = part ? a.sum_lo : a.sum_hi;
        for (uint32_t it = blockIdx.x; it < n_items && ok; it += gridDim.x) {
            const XGroup grp = a.groups[it / a.tiles];
            uint32_t src_row = 0;
            if (lane < grp.count) src_row = (a.row_to_pair ? a.row_to_pair[grp.first + lane] : grp.first + lane) / a.k_div;
            const __half *src[8];                                             // rows sub, sub + 4, ...
#pragma unroll
            for (uint32_t i = 0; i < 8; i++) src[i] = in + (uint64_t)__shfl_sync(0xffffffffu, src_row, sub + 4 * i) * a.in_pitch;
            const uint32_t rounds = grp.count > 16 ? 8u : 4u, rows = rounds * 4;
            const __half *ssrc = sums + (uint64_t)src_row * a.units * 16u;
            const uint32_t dst_row = sbase + XM_B + part * XB_ONE + sub * 128u;
            for (uint32_t u = 0; u < a.units && ok; u++, un++) {
#pragma unroll 1
                for (uint32_t c = 0; c < SPU; c++, n++) {
                    if (n >= NB && !(ok = XWAIT(w0, done + 8 * (n & (NB - 1)), ((n >> NBLOG) - 1) & 1u))) break;
                    const uint32_t dst = dst_row + (n & (NB - 1)) * BSTEP, col = u * UNIT + c * CPS * 64;
#pragma unroll
                    for (uint32_t i = 0; i < 8; i++)
                        if (i < rounds) {                                     // rows beyond the group read as zero; row & 7 = sub + 4 (i & 1)
                            const uint32_t bytes = sub + 4 * i < grp.count ? 16u : 0u, to = dst + i * 512u + ((piece ^ (sub + 4 * (i & 1u))) << 4);
                            xcp16(to, src[i] + col, bytes);
                            if (CPS == 2) xcp16(to + 2 * XB_ONE, src[i] + col + 64, bytes);
                        }
                    if (c == 0 && lane < rows) {
                        const uint32_t bytes = lane < grp.count ? 16u : 0u;
                        if (Fm::MIN) {                                         // the unit's sixteen column sums
                            const uint32_t sd = sbase + XM_SUMS + ((un & 3u) * 2 + part) * XS_ONE + lane * 16u;
                            xcp16(sd, ssrc + u * 16u, bytes); xcp16(sd + XTOK * 16u, ssrc + u * 16u + 8, bytes);
                        }
                        if (MODE == 1 && part == 0)
                            asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(sbase + XM_BSC + ((un & 7u) * XTOK + lane) * 4u),
                                         "l"(a.in_scale + (uint64_t)src_row * a.units + u), "r"(bytes >> 2) : "memory");
                    }
                    asm volatile("cp.async.commit_group;" ::: "memory");
                    if (n >= LAG) {
                        asm volatile("cp.async.wait_group %0;" ::"n"(LAG) : "memory");
                        hand_over(n - LAG);
                    }
                }
            }
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
        for (uint32_t i = n > LAG ? n - LAG : 0; i < n; i++) hand_over(i);
    } else if (warp >= R::MMA) {
        // ---------------- tcgen05.mma issue: one warp a tile, so that one's waits and commits lie under the other's products ----------------
        // The whole warp walks this loop and every value an instruction names is warp-uniform for the compiler too (waits
        // end in a vote, counts come out of a reduction, TMEM starts at column 0 because all of it is ours, no calls):
        // otherwise each operand of each MMA is moved to a uniform register first, which costs 58 cycles an instruction.
        const uint32_t el = xelect();
        const uint64_t b_desc = xdesc_sw128(sbase + XM_B), s_desc = xdesc_sums(sbase + XM_SUMS);
        auto wait = [&](uint32_t bar, uint32_t parity, long long &spent) -> bool {
            bool done = __all_sync(0xffffffffu, xbar_try(bar, parity));
            if (done) return true;
            const long long start = clock64();
            bool give_up = false;
            while (!done && !give_up) {
                done = __all_sync(0xffffffffu, xbar_try(bar, parity));
                if (!done && clock64() - start > (1ll << 31)) { *dead = 1; atomicOr(a.status, QW4SH_ERR_STATE); }
                give_up = __any_sync(0xffffffffu, !done && *dead);
            }
            spent += clock64() - start;
            return done;
        };
        const uint32_t items = __reduce_max_sync(0xffffffffu, n_items), units = a.units;
        const uint32_t m = warp - R::MMA;
        uint32_t n = 0, un = 0;
        bool ok = true, ready = false;
        for (uint32_t it = blockIdx.x; it < items && ok; it += gridDim.x) {
            const uint32_t tok = __any_sync(0xffffffffu, a.groups[it / a.tiles].count > 16) ? 32u : 16u;
            const uint32_t idesc = (1u << 4) | ((tok >> 3) << 17) | ((XROWS >> 4) << 24);   // D F32, A and B F16, K-major
            for (uint32_t u = 0; u < units && ok; u++, un++) {
                const uint32_t ub = un & 1u;
#pragma unroll 1
                for (uint32_t c = 0; c < SPU; c++, n++) {
                    if (!ready && !(ok = wait(full + 8 * ((n & (NB - 1)) * 2 + m), (n >> NBLOG) & 1u, w0))) break;
                    xtc_after();
                    // asked before the products are issued, used after them: a barrier's answer takes a hundred cycles and more behind
                    // the dequantisers' shared-memory and TMEM traffic
                    const bool next = xbar_test(full + 8 * (((n + 1) & (NB - 1)) * 2 + m), ((n + 1) >> NBLOG) & 1u);
                    const bool drained = c != SPU - 1 || un == 0 || xbar_test(d_empty + 8 * ((ub ^ 1u) * 2 + m), ((un - 1) >> 1) & 1u);
                    const uint64_t bd = b_desc + (n & (NB - 1)) * (BSTEP >> 4);
                    const uint32_t at = XT_A + (n & 1u) * 128 + m * 64, q = XT_Q + ub * 64 + m * 32;
                    if (el) {
#pragma unroll
                        for (uint32_t h = 0; h < 2; h++)                                  // 64 columns; wide form: hi, then lo, of the same ones
#pragma unroll
                            for (uint32_t j = 0; j < 4; j++) {
                                const uint64_t b = bd + (F == T_WIDE ? 0u : h * ((2 * XB_ONE) >> 4)) + j * 2;
                                xmma(q, at + h * 32 + j * 8, b, idesc, (c | h | j) ? 1u : 0u);
                                if (F != T_WIDE || h == 0) xmma(q, at + h * 32 + j * 8, b + (XB_ONE >> 4), idesc, 1u);
                            }
                    }
                    if (c == SPU - 1) {
                        // M has one buffer: the previous unit's has to be read; that also frees the Q buffer of the next unit
                        __syncwarp();
                        if (!__all_sync(0xffffffffu, drained) && !(ok = wait(d_empty + 8 * ((ub ^ 1u) * 2 + m), ((un - 1) >> 1) & 1u, w2))) break;
                        xtc_after();
                        if (Fm::MIN && el) {
                            const uint64_t sd = s_desc + (un & 3u) * ((2 * XS_ONE) >> 4);
                            xmma(XT_M + m * 32, XT_AM + ub * 16 + m * 8, sd, idesc, 0u);
                            xmma(XT_M + m * 32, XT_AM + ub * 16 + m * 8, sd + (XS_ONE >> 4), idesc, 1u);
                        }
                    }
                    if (el) xtc_commit(done + 8 * (n & (NB - 1)));
                    ready = __all_sync(0xffffffffu, next);
                }
            }
        }
    } else if (warp < R::EPI) {
        // ---------------- dequantise: packed bytes -> exact halves in TMEM ----------------
        // the sets of four warps take turns at the (step, tile) pairs
        const uint32_t set = warp >> 2, row = (warp & 3u) * 32 + lane, quad = ((warp & 3u) * 32) << 16, nb = a.w0.k_storage >> 8;
        constexpr uint32_t STPS = STCH / CPS;                                 // steps per stage
        const uint32_t steps = a.units * SPU, stages = (steps + STPS - 1) / STPS, spare = stages * STPS - steps;
        uint32_t *dsc = reinterpret_cast<uint32_t *>(smem + XM_DSC) + row;
        const uint32_t side = 128 * nb * Fm::SIDE_BLOCK;
        uint32_t n0 = 0, k0 = 0, u0 = 0, ring = 0, l = set;                   // steps, stages, units before this item; this set's next pair of it
        bool ok = true;
        XDeq<F> q;
        for (uint32_t it = blockIdx.x; it < n_items && ok; it += gridDim.x) {
            uint32_t row_scale[2] = {0, 0};                                   // wide form: the rows' powers of two
            if (F == T_WIDE) {
                const uint64_t at = (uint64_t)a.groups[it / a.tiles].expert * a.w0.n_out + (it % a.tiles) * STEP + row;
                row_scale[0] = __float_as_uint(__ldg(a.row_scale0 + at)); row_scale[1] = __float_as_uint(__ldg(a.row_scale1 + at + (MODE == 1 ? 128 : 0)));
            }
            for (; l < 2 * steps; l += Fm::SETS) {
                const uint32_t m = l & 1u, step = l >> 1, n = n0 + step, ks = step / STPS, sp = step % STPS, k = k0 + ks, st = k % Fm::STAGES;
                const uint32_t beside = F == T_WIDE ? row_scale[m] : sbase + xm_side<F>() + (ring * 2 + m) * side + row * nb * Fm::SIDE_BLOCK;
                if (!(ok = XWAIT(w0, w_full + 8 * st, (k / Fm::STAGES) & 1u))) break;
                const bool free = n < 2 || xbar_test(done + 8 * ((n - 2) & (NB - 1)), ((n - 2) >> NBLOG) & 1u);      // asked early, used after the first chunk
                q.load(sbase + xm_weights<F>() + (st * 2 + m) * Fm::TILE, row, smem + xm_tables<F>(), beside, ks, sp, lane);
                const uint32_t at = quad + XT_A + (n & 1u) * 128 + m * 64, un = u0 + step / SPU;
                uint32_t v[32];
                q.chunk(0, v);
                if (!free && !(ok = XWAIT(w1, done + 8 * ((n - 2) & (NB - 1)), ((n - 2) >> NBLOG) & 1u))) break;
                xtc_after();
                xst32(at, v);
                q.chunk(1, v);
                xst32(at + 32, v);
                if (step % SPU == 0) {
                    if (Fm::MIN) {
                        uint32_t mn[8];
                        q.template minima<MODE>(sp, mn);
                        xst8(quad + XT_AM + (un & 1u) * 16 + m * 8, mn);
                    }
                    dsc[(m * 4 + (un & 3u)) * 128] = q.word();
                }
                xst_wait();
                xtc_before();
                __syncwarp();
                if (lane == 0) {
                    xbar_arrive(full + 8 * ((n & (NB - 1)) * 2 + m));
                    // four arrivals a warp-row and stage: one for each of its pairs, the item's last for the columns never multiplied
                    xbar_arrive_n(w_empty + 8 * st, step == steps - 1 ? 1 + spare : 1);
                }
            }
            l -= 2 * steps; n0 += steps; k0 += stages; u0 += a.units; ring = (ring + 1) & ring_mask;
        }
    } else {
        // ---------------- read-back: TMEM -> scales -> SwiGLU + split / store ----------------
        const uint32_t m = (warp - R::EPI) >> 2, row = (warp & 3u) * 32 + lane, quad = ((warp & 3u) * 32) << 16, et = tid - R::EPI * 32;
        const uint32_t *dsc = reinterpret_cast<const uint32_t *>(smem + XM_DSC) + m * 512 + row;
        float *hand = reinterpret_cast<float *>(smem + XM_HAND);
        uint32_t *share = reinterpret_cast<uint32_t *>(smem + XM_SHARE) + (warp - R::EPI) * 32;      // this warp's broadcast words
        uint32_t un = 0;
        bool ok = true;                                                       // once false: no more waits, but every CTA-internal barrier below is still met
        for (uint32_t it = blockIdx.x; it < n_items; it += gridDim.x) {
            const XGroup grp = a.groups[it / a.tiles];
            const uint32_t tile = it % a.tiles;
            float acc[XTOK];
#pragma unroll
            for (uint32_t n = 0; n < XTOK; n++) acc[n] = 0.0f;
            for (uint32_t u = 0; u < a.units; u++, un++) {
                const uint32_t last = (un + 1) * SPU - 1;                    // the unit's last step
                if (ok) ok = XWAIT(w0, done + 8 * (last & (NB - 1)), (last >> NBLOG) & 1u);
                if (!ok) continue;
                xtc_after();
                const uint32_t word = dsc[(un & 3u) * 128];
                float d, dmin = 0.0f;
                if (F == T_WIDE) d = __uint_as_float(word);
                else if (F == T_IQ2_XXS) d = xhalf_bits(word) * 0.125f;
                else { d = xhalf_bits(word) * XUP; dmin = -xhalf_bits(word >> 16); }
                const float4 *bsc = reinterpret_cast<const float4 *>(smem + XM_BSC + (un & 7u) * (XTOK * 4));
                const uint32_t qa = tmem + quad + XT_Q + (un & 1u) * 64 + m * 32, ma = tmem + quad + XT_M + m * 32;
#pragma unroll
                for (uint32_t h = 0; h < XTOK / 16; h++) {
                    if (16 * h < grp.count) {
                        uint32_t qv[16], mv[16];
                        if (Fm::MIN) xld_qm(qa + 16 * h, ma + 16 * h, qv, mv);
                        else xld_q(qa + 16 * h, qv);
#pragma unroll
                        for (int n4 = 0; n4 < 16; n4 += 4) {
                            float4 sc = make_float4(1.0f, 1.0f, 1.0f, 1.0f);
                            if (MODE == 1) sc = bsc[4 * h + n4 / 4];
                            const float s4[4] = {sc.x, sc.y, sc.z, sc.w};
#pragma unroll
                            for (int i = 0; i < 4; i++) {
                                float &to = acc[16 * h + n4 + i];
                                if (MODE == 0) {
                                    to = fmaf(d, __uint_as_float(qv[n4 + i]), to);
                                    if (Fm::MIN) to = fmaf(dmin, __uint_as_float(mv[n4 + i]), to);
                                } else {
                                    float t = d * __uint_as_float(qv[n4 + i]);
                                    if (Fm::MIN) t = fmaf(dmin, __uint_as_float(mv[n4 + i]), t);
                                    to = fmaf(s4[i], t, to);
                                }
                            }
                        }
                    }
                }
                xtc_before();
                __syncwarp();
                if (lane == 0) xbar_arrive(d_empty + 8 * ((un & 1u) * 2 + m));
            }
            const uint32_t my_pair = lane < grp.count ? (a.row_to_pair ? a.row_to_pair[grp.first + lane] : grp.first + lane) : 0;
            if (MODE == 0) {
                share[lane] = __float_as_uint(lane < grp.count ? __ldg(a.in_scale + my_pair / a.k_div) : 0.0f);
                float *mine = hand + row + (row >> 4);
                asm volatile("bar.sync 1, 256;" ::: "memory");                // the hand-over tile's previous content has been taken
                // the gate's warps take the lower half of the tokens, the up's the upper: each hands over what the other needs
                const uint32_t half = (grp.count + 7u) / 8u * 4u;
#pragma unroll
                for (uint32_t n = 0; n < XTOK; n++) if (n < grp.count && (n < half) == (m == 1)) mine[n * XPITCH] = acc[n];
                asm volatile("bar.sync 1, 256;" ::: "memory");
#pragma unroll
                for (uint32_t n4 = 0; n4 < XTOK; n4 += 4) {
                    if (n4 >= grp.count) break;
                    if ((n4 < half) != (m == 0)) continue;
                    const float4 s4 = *reinterpret_cast<const float4 *>(share + n4);
                    const float sv[4] = {s4.x, s4.y, s4.z, s4.w};
#pragma unroll
                    for (uint32_t i = 0; i < 4; i++) {
                        const uint32_t n = n4 + i;
                        if (n < grp.count) {
                            const float own = acc[n] * sv[i], other = mine[n * XPITCH] * sv[i];
                            const float g = m == 0 ? own : other, up = m == 0 ? other : own;
                            const float e = __expf(-fabsf(g));
                            mine[n * XPITCH] = g * __fdividef(g >= 0.0f ? 1.0f : e, 1.0f + e) * up;
                        }
                    }
                }
                asm volatile("bar.sync 1, 256;" ::: "memory");
                // eight threads a token, sixteen columns each: the tile's power of two, hi and lo, sums of eight columns
                const uint32_t n = et >> 3, seg = et & 7u;
                const bool live = n < grp.count;
                const uint32_t pair = live ? (a.row_to_pair ? a.row_to_pair[grp.first + n] : grp.first + n) : 0;
                float v[2][8], top = 0.0f;
#pragma unroll
                for (int i = 0; i < 16; i++) { v[i >> 3][i & 7] = live ? hand[n * XPITCH + seg * 17 + i] : 0.0f; top = fmaxf(top, fabsf(v[i >> 3][i & 7])); }
                bool bad = false;
#pragma unroll
                for (int i = 0; i < 16; i++) bad |= (__float_as_uint(v[i >> 3][i & 7]) & 0x7f800000u) == 0x7f800000u;
                for (int o = 1; o < 8; o <<= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, o));
                float up, down;
                xscale_of(top, up, down);
                if (live && ok) {
                    if (bad) atomicOr(a.status, QW4SH_ERR_NONFINITE);
                    const uint64_t at = (uint64_t)pair * a.w0.n_out + tile * 128 + seg * 16;
                    float s8[2];
#pragma unroll
                    for (int h = 0; h < 2; h++) {
                        uint32_t hi[4], lo[4];
                        s8[h] = 0.0f;
#pragma unroll
                        for (int i = 0; i < 8; i++) { v[h][i] *= up; s8[h] += v[h][i]; }
                        xsplit8(v[h], hi, lo);
                        *reinterpret_cast<uint4 *>(a.out_hi + at + 8 * h) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
                        *reinterpret_cast<uint4 *>(a.out_lo + at + 8 * h) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
                    }
                    const __half2 sh = __floats2half2_rn(s8[0], s8[1]);
                    const float2 f = __half22float2(sh);
                    const uint64_t sat = (uint64_t)pair * (a.w0.n_out >> 3) + tile * 16 + seg * 2;
                    *reinterpret_cast<__half2 *>(a.osum_hi + sat) = sh;
                    *reinterpret_cast<__half2 *>(a.osum_lo + sat) = __floats2half2_rn(s8[0] - f.x, s8[1] - f.y);
                    if (seg == 0) a.out_scale[(uint64_t)pair * (a.w0.n_out >> 7) + tile] = down;
                }
            } else {
                share[lane] = my_pair;
                __syncwarp();
                float *to = a.out + tile * 256 + m * 128 + row;
                bool bad = false;
                if (ok)
#pragma unroll
                    for (uint32_t n4 = 0; n4 < XTOK; n4 += 4) {
                        if (n4 >= grp.count) break;
                        const uint4 p4 = *reinterpret_cast<const uint4 *>(share + n4);
                        const uint32_t pv[4] = {p4.x, p4.y, p4.z, p4.w};
#pragma unroll
                        for (uint32_t i = 0; i < 4; i++)
                            if (n4 + i < grp.count) {
                                bad |= (__float_as_uint(acc[n4 + i]) & 0x7f800000u) == 0x7f800000u;
                                to[(uint64_t)pv[i] * a.w0.n_out] = acc[n4 + i];
                            }
                    }
                __syncwarp();                                                 // the list is read before the next item's is written
                if (bad) atomicOr(a.status, QW4SH_ERR_NONFINITE);
            }
        }
    }
    if (prof && lane == 0 && (warp == 0 || warp == R::EPI || warp == R::TMA || warp == R::MMA || warp == R::ACT)) {
        const uint32_t role = warp == 0 ? 1 : warp == R::EPI ? 0 : warp == R::TMA ? 2 : warp == R::MMA ? 3 : 4;
        a.debug[role * 4] = (unsigned long long)w0; a.debug[role * 4 + 1] = (unsigned long long)w1;
        a.debug[role * 4 + 2] = (unsigned long long)w2; a.debug[role * 4 + 3] = (unsigned long long)(clock64() - t_begin);
    }
    // ---------------- teardown: TMEM is freed on every path ----------------
    xtc_before();
    __syncthreads();
    if (warp == 0) {
        xtc_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(XT_COLS) : "memory");
    }
}

}  // namespace qw4
