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
//   - per 128 x 256 weights the dequantiser needs about 1700 warp instructions, the MMAs 326 (N 16) or 561 (N 32) cycles, HBM 804 (Q4_K),
//     469 (Q2_K), 369 (IQ2_XXS) cycles at 6.45 TB/s over 148 SMs, all of them at the same time.
//
// Work item: one group (<= 32 token rows of one expert) x two 128-row tiles that share the activations: gate rows and the
// same up rows (mode 0: SwiGLU stays in the CTA), or two neighbouring row tiles (mode 1, down).  Sharing halves the
// activation traffic from L2, and the two tiles take turns on the tensor pipe, so one is read back while the other is
// multiplied.  CTAs are persistent and walk the item list with a stride.
//
// What a step (128 columns of both tiles) waits for is hand-overs, not a rate: its MMAs hold the tensor pipe for 528 cycles (N 32), and an
// mbarrier's answer takes a hundred cycles even when it is positive and nothing else runs (a named barrier's 24), so every question on a role's
// path counts, and so does every load from global memory.  Hence:
//   - each tile has barriers of its own from the dequantiser to the read-back: with one between them the tiles ran in step, and the pipe stood
//     still while both asked (1400 cycles a step, 1050 without);
//   - the dequantiser asks for a stage once, unrolls its steps, and has the next step's words on their way before it hands one over;
//   - copies of activations report to the step's barrier themselves (cp.async.mbarrier.arrive), groups are asked for one item ahead, and pairs and
//     scales of an item lie in shared memory when the read-back needs them;
//   - the read-back gives accumulators back when it has read them, two sums to an instruction (fma.rn.f32x2).
// Routed experts of 1024 tokens, us, before and after these: Q4_K (Zipf) gate/up 152 and 133, down 96 and 92; Q2_K 188 and 158, 115 and 106;
// 777 tokens of the IQ2_XXS checkpoint layer 328 and 291, 158 (Q2_K, 640 columns) and 141.  Measured without gain: twelve or sixteen
// dequantising warps (the read-back is then later by as much), sixteen read-back warps (64 registers a thread: down 127), gathering the
// activations by TMA (tile::gather4: 85 cycles each, 2750 a step).
//
// Warps (21):
//   0-7         dequantise, four a tile (TMEM lane = weight row), 128 columns at a time into two A slots per tile
//   next 8      read back (tcgen05.ld), scale, accumulate; SwiGLU + split of the activation, or the store
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
#include <type_traits>

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
// step (the wide form's hi and lo halves of one chunk fill a slot), bytes for look-up tables and
// for the fp16 scales that the resident image keeps apart from the codes.
template <uint32_t F> struct XFmt;
template <> struct XFmt<T_Q4_K>    { static constexpr uint32_t COLS = 256, TILE = 128 * 144, STAGES = 3, BSLOTS = 4, CPS = 2, TABLES = 0, SIDE = 0, SIDE_BLOCK = 0; static constexpr bool MIN = true; };
template <> struct XFmt<T_Q2_K>    { static constexpr uint32_t COLS = 256, TILE = 128 * 80, STAGES = 4, BSLOTS = 4, CPS = 2, TABLES = 0, SIDE = 32768, SIDE_BLOCK = 4; static constexpr bool MIN = true; };
template <> struct XFmt<T_IQ2_XXS> { static constexpr uint32_t COLS = 512, TILE = 128 * 128, STAGES = 2, BSLOTS = 4, CPS = 2, TABLES = 49152, SIDE = 16384, SIDE_BLOCK = 2; static constexpr bool MIN = false; };
template <> struct XFmt<T_WIDE>    { static constexpr uint32_t COLS = 64, TILE = 128 * 256, STAGES = 2, BSLOTS = 8, CPS = 1, TABLES = 0, SIDE = 0, SIDE_BLOCK = 0; static constexpr bool MIN = false; };
// warps of a launch of format F: dequantise, read back, TMA, MMA (2), activations (2)
template <uint32_t F> struct XRole {
    static constexpr int EPI = 8, TMA = EPI + 8, MMA = TMA + 1, ACT = MMA + 2, WARPS = ACT + 2, THREADS = 32 * WARPS;
};

constexpr uint32_t XPITCH = 136;                             // floats per token of the hand-over tile: column c at c + c / 16, no bank conflicts either way
constexpr uint32_t XB_ONE = XTOK * 128;                      // 4096: hi (or lo) rows of one activation slot, 128-byte swizzle
constexpr uint32_t XS_ONE = 2 * XTOK * 16;                   // 1024: hi (or lo) column sums of one unit
// shared-memory map
constexpr uint32_t XM_BARS = 0, XM_TMEM = 512, XM_GROUP = 512 + 64 /* [8] group records */, XM_DSC = 1024 /* [2][4][128] words */, XM_SUMS = XM_DSC + 4096 /* [4][2] x XS_ONE */,
                   XM_BSC = XM_SUMS + 4 * 2 * XS_ONE /* [8][32] floats: unit scales of mode 1 */, XM_PAIR = XM_BSC + 1024 /* [8 items][32]: pairs */,
                   XM_ROW = XM_PAIR + 1024 /* [8 items][32]: row scales of mode 0 */, XM_HAND = XM_ROW + 1024,
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
// by one lane of a converged warp, as one predicated instruction
__device__ __forceinline__ void xbar_arrive_if(uint32_t bar, bool mine) {
    asm volatile("{\n .reg .pred p;\n setp.ne.b32 p, %1, 0;\n @p mbarrier.arrive.shared::cta.b64 _, [%0];\n}" ::"r"(bar), "r"((uint32_t)mine) : "memory");
}
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
// Bounded wait; `dead` (shared memory) is set by whoever gives up, and ends every other wait.  `spent` counts the cycles of waits that were not
// over at once.  SLEEP: nanoseconds between two questions, for the roles that wait most of their time and have slack; their questions
// would take issue slots from the dequantising warps.
template <uint32_t SLEEP = 0>
__device__ __forceinline__ bool xbar_wait(uint32_t bar, uint32_t parity, volatile uint32_t *dead, uint32_t *status, uint32_t &spent) {
    if (xbar_try(bar, parity)) return true;
    const uint32_t start = clock();
    uint32_t now = start;
    while (!xbar_try(bar, parity)) {
        if (SLEEP) __nanosleep(SLEEP);
        now = clock();
        if (*dead) return false;
        if (now - start > (1u << 31)) { *dead = 1; atomicOr(status, QW4SH_ERR_STATE); return false; }
    }
    spent += clock() - start;
    return true;
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
__device__ __forceinline__ void xcp4(uint32_t dst, const void *src, uint32_t src_bytes) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(src_bytes) : "memory");
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
__device__ __forceinline__ void xst16(uint32_t taddr, const uint32_t (&v)[16]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
                 ::"r"(taddr), X8(v, 0), X8(v, 8) : "memory");
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
// Two floats to an instruction, each rounded like a scalar one.
__device__ __forceinline__ unsigned long long xpair_bits(uint32_t a, uint32_t b) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "r"(a), "r"(b));
    return r;
}
__device__ __forceinline__ unsigned long long xpair(float a, float b) { return xpair_bits(__float_as_uint(a), __float_as_uint(b)); }
__device__ __forceinline__ unsigned long long xfma2(unsigned long long a, unsigned long long b, unsigned long long c) {
    unsigned long long r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ unsigned long long xmul2(unsigned long long a, unsigned long long b) {
    unsigned long long r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
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
// load<SP>(): packed words of step SP of the stage (scales of the whole block with step 0); part<SP, P>(): sixteen words of two halves, the
// step's columns 32 P .. 32 P + 31 (wide form: hi, then lo, of 64 columns); minima<SP>(): the unit's 16 slots, on its first step;
// word(): what the read-back multiplies by, {d, dmin} or a float.
template <uint32_t F> struct XDeq;

// Codes masked out in place ARE halves, subnormal ones: a code at bit b of its half is code * 2^(b - 24), and times s * 2^(10 - b) it
// becomes s * code * 2^-14, exactly; the 2^14 goes to the FP32 scale of the read-back.  One logic operation with an immediate (one
// cycle a warp instruction; with three registers two) and one multiply (two cycles) per two weights.
// 2^-14 makes every operand that is not zero a normal half.  With 2^-20 the multipliers come out of one fused multiply-add instead of a
// subtraction and a product, but the operands (all of Q2_K's, many of Q4_K's) are subnormal: as exact, yet the tensor core then adds the
// same products with other last bits (1e-7 of the result on Q2_K, 1.6e-8 on Q4_K; with 2^-14 the same bits whatever else the kernel
// does).  RMS error of y against 64 bits, 2^-14 and 2^-20: Q2_K 1.5435e-6 and 1.5425e-6 (1024 tokens), 1.9594e-6 and 1.9586e-6 (7), Q4_K
// 1.6450e-6 and 1.6452e-6 (64), 2.0619e-6 and 2.0622e-6 (333, rows with outliers); time the same within its spread.
constexpr float XUP = 16384.0f;
__device__ __forceinline__ uint32_t xfold(uint32_t bits, __half2 mul) { return xu32(__hmul2(xh2(bits), mul)); }
// byte i of `v` (at most 63) times `up` (a power of two), in both halves
__device__ __forceinline__ __half2 xscaled(uint32_t v, uint32_t i, float up) { return __hmul2(xbytes2(v, i, i), __float2half2_rn(up)); }

template <> struct XDeq<T_Q4_K> {
    uint4 h;
    uint32_t w[16];
    template <int SP> __device__ __forceinline__ void load(uint32_t tile, uint32_t row, const uint8_t *, uint32_t, uint32_t, uint32_t) {
        const uint32_t base = tile + row * 144u;
        if (SP == 0) h = xlds128(base);
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const uint4 q = xlds128(base + 16 + SP * 64 + 16 * i);
            w[4 * i] = q.x; w[4 * i + 1] = q.y; w[4 * i + 2] = q.z; w[4 * i + 3] = q.w;
        }
    }
    template <int SP, int P> __device__ __forceinline__ void part(uint32_t (&v)[16]) {
        constexpr uint32_t mask = P & 1 ? 0x00f000f0u : 0x000f000fu;         // low nibbles are columns 0-31 of 64, high ones 32-63
        const uint32_t sc = SP ? (h.w & 0x0f0f0f0fu) | ((h.y >> 2) & 0x30303030u) : h.y & 0x3f3f3f3fu;
        const __half2 mul = xscaled(sc, P, P & 1 ? 64.0f : 1024.0f);
#pragma unroll
        for (int j = 0; j < 8; j++) {
            const uint32_t q = w[8 * (P >> 1) + j];
            v[2 * j] = xfold(q & mask, mul);
            v[2 * j + 1] = xfold((q >> 8) & mask, mul);
        }
    }
    // mode 0: 16 slots of 16 columns, mode 1 (half block SP): 16 slots of 8 columns; a minimum covers 32 columns
    template <int MODE, int SP> __device__ __forceinline__ void minima(uint32_t (&v)[8]) {
        const uint32_t lo = h.z & 0x3f3f3f3fu, hi = ((h.w >> 4) & 0x0f0f0f0fu) | ((h.z >> 2) & 0x30303030u), half = SP ? hi : lo;
#pragma unroll
        for (uint32_t j = 0; j < 8; j++) {
            const uint32_t sub = MODE == 0 ? j : j >> 1, m = MODE == 0 ? (j < 4 ? lo : hi) : half;
            v[j] = xu32(xbytes2(m, sub & 3u, sub & 3u));
        }
    }
    __device__ __forceinline__ uint32_t word() const { return h.x; }
};

// Q2_K stage: [128][64] code bytes with the 64-byte swizzle, then [128][16] scale bytes; {d, dmin} of all the item's blocks beside the stages
template <> struct XDeq<T_Q2_K> {
    uint32_t q[4], dd, w[8];
    template <int SP> __device__ __forceinline__ void load(uint32_t tile, uint32_t row, const uint8_t *, uint32_t side, uint32_t b, uint32_t) {
        const uint32_t base = tile + row * 64u, swz = ((row >> 1) & 3u) << 4;
        if (SP == 0) {
            const uint4 s = xlds128(tile + 8192u + row * 16u);
            q[0] = s.x; q[1] = s.y; q[2] = s.z; q[3] = s.w;
            dd = xlds32(side + b * 4u);
        }
#pragma unroll
        for (int i = 0; i < 2; i++) {
            const uint4 c = xlds128(base + ((SP * 32u + 16u * i) ^ swz));
            w[4 * i] = c.x; w[4 * i + 1] = c.y; w[4 * i + 2] = c.z; w[4 * i + 3] = c.w;
        }
    }
    template <int SP, int P> __device__ __forceinline__ void part(uint32_t (&v)[16]) {
        constexpr uint32_t r = P & 1, mask = 0x00030003u << (2 * P);         // bit pair P of the bytes, in place
        constexpr float up = P == 0 ? 1024.0f : P == 1 ? 256.0f : P == 2 ? 64.0f : 16.0f;
        const uint32_t word = q[2 * SP + (P >> 1)] & 0x0f0f0f0fu;
        const __half2 ma = xscaled(word, 2 * r, up), mb = xscaled(word, 2 * r + 1, up);
#pragma unroll
        for (int j = 0; j < 8; j++) {
            v[2 * j] = xfold(w[j] & mask, j < 4 ? ma : mb);
            v[2 * j + 1] = xfold((w[j] >> 8) & mask, j < 4 ? ma : mb);
        }
    }
    template <int MODE, int SP> __device__ __forceinline__ void minima(uint32_t (&v)[8]) {
#pragma unroll
        for (uint32_t j = 0; j < 8; j++) {                   // a minimum covers 16 columns
            if (MODE == 0) v[j] = xu32(xbytes2((q[j >> 1] >> 4) & 0x0f0f0f0fu, (j & 1u) * 2u, (j & 1u) * 2u + 1u));
            else v[j] = xu32(xbytes2((q[2 * SP + (j >> 2)] >> 4) & 0x0f0f0f0fu, j & 3u, j & 3u));
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
    template <int SP> __device__ __forceinline__ void load(uint32_t tile, uint32_t row, const uint8_t *tables, uint32_t side, uint32_t b, uint32_t lane) {
        const uint32_t base = tile + row * 128u, swz = ((((row & 3u) << 1) ^ (row & 7u)) << 4);
        g[0] = xlds128(base + ((SP * 32u) ^ swz)); g[1] = xlds128(base + ((SP * 32u + 16u) ^ swz));       // two groups of 32 columns each
        grid = xs_u32(tables) + (lane & 7u) * 16u; sign = xs_u32(tables) + 32768u + lane * 4u;
        dd = xlds16(side + (2 * b + (SP >> 1)) * 2u);
    }
    template <int SP, int P> __device__ __forceinline__ void part(uint32_t (&v)[16]) {
        const uint32_t index = P & 1 ? g[P >> 1].z : g[P >> 1].x, bits = P & 1 ? g[P >> 1].w : g[P >> 1].y;
        const __half2 s = __hsub2(xh2(((bits >> 27) | 1u) * 0x10001u + 0x64006400u), xh2(0x64006400u));           // 2 * scale + 1
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const uint4 m = xlds128(grid + (k == 0 ? (index << 7) & 0x7f80u : k == 1 ? (index >> 1) & 0x7f80u : k == 2 ? (index >> 9) & 0x7f80u : (index >> 17) & 0x7f80u));
            const uint32_t w = xlds32(sign + ((k == 0 ? bits << 7 : bits >> (7 * k - 7)) & 0x3f80u));
            const uint32_t mm[4] = {m.x, m.y, m.z, m.w};
#pragma unroll
            for (int q = 0; q < 4; q++) v[4 * k + q] = xu32(__hmul2(xh2(mm[q] ^ ((w << q) & 0x80008000u)), s));
        }
    }
    template <int MODE, int SP> __device__ __forceinline__ void minima(uint32_t (&)[8]) {}
    __device__ __forceinline__ uint32_t word() const { return dd; }
};

// Wide form: fp16 hi and lo images of the weights (row scaled by a power of two), [128][128 bytes] each with the 128-byte swizzle.
template <> struct XDeq<T_WIDE> {
    uint32_t base, swz, scale;
    template <int SP> __device__ __forceinline__ void load(uint32_t tile, uint32_t row, const uint8_t *, uint32_t row_scale, uint32_t, uint32_t) {
        base = tile + row * 128u; swz = (row & 7u) << 4; scale = row_scale;
    }
    template <int SP, int P> __device__ __forceinline__ void part(uint32_t (&v)[16]) {
#pragma unroll
        for (uint32_t i = 0; i < 4; i++) {
            const uint4 q = xlds128(base + (P >> 1) * 16384u + (((4 * (P & 1) + i) * 16u) ^ swz));
            v[4 * i] = q.x; v[4 * i + 1] = q.y; v[4 * i + 2] = q.z; v[4 * i + 3] = q.w;
        }
    }
    template <int MODE, int SP> __device__ __forceinline__ void minima(uint32_t (&)[8]) {}
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

template <uint32_t F, int MODE>
__device__ __forceinline__ void expert_tc_body(const XMaps &maps, const XArgs &a, uint8_t *smem) {
    using Fm = XFmt<F>;
    using R = XRole<F>;
    constexpr uint32_t UNIT = MODE == 0 ? 256 : 128, CPS = Fm::CPS, SPU = UNIT / (64 * CPS), STCH = Fm::COLS / 64;   // steps per unit, chunks per stage
    constexpr uint32_t BSTEP = CPS * 2 * XB_ONE, NB = Fm::BSLOTS, NBLOG = NB == 8 ? 3 : 2;
    constexpr uint32_t STEP = MODE == 0 ? 128 : 256;                        // weight rows per item
    const uint32_t sbase = xs_u32(smem);
    const uint32_t w_full = sbase + XM_BARS, w_empty = w_full + 8 * Fm::STAGES, full = w_empty + 8 * Fm::STAGES /* [step][tile] */,
                   done = full + 8 * 2 * NB /* [step][tile] */, q_empty = done + 8 * 2 * NB /* [buffer][tile] */, m_empty = q_empty + 8 * 4 /* [tile] */;
    static_assert(8 * (2 * Fm::STAGES + 4 * NB + 6) <= 512, "barrier block");
    volatile uint32_t *dead = reinterpret_cast<volatile uint32_t *>(smem + XM_TMEM + 8);
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    // items whose apart-lying scales are held: four where the rows are short enough, else two (rows of 9 to 16 blocks); four are more than the
    // stages reach ahead, two are not where an item is one or two stages of four (see the TMA warp)
    const uint32_t ring_mask = (a.w0.k_storage >> 8) <= 8 ? 3u : 1u;
    const bool prof = a.debug && blockIdx.x == 0;
    uint32_t w0 = 0, w1 = 0, w2 = 0;                                        // cycles spent in this role's waits
    const long long t_begin = prof ? clock64() : 0;

    if (tid == 0) {
        for (uint32_t i = 0; i < Fm::STAGES; i++) { xbar_init(w_full + 8 * i, 1); xbar_init(w_empty + 8 * i, 8); }
        // a step of a tile is ready when its four dequantising warps and the copies of every lane of the two activation warps say so: one wait
        // for its products
        for (uint32_t i = 0; i < 2 * NB; i++) xbar_init(full + 8 * i, 4 + 64);
        for (uint32_t i = 0; i < 2 * NB; i++) xbar_init(done + 8 * i, 1);
        for (uint32_t i = 0; i < 4; i++) xbar_init(q_empty + 8 * i, MODE == 0 ? 8 : 4);
        for (uint32_t i = 0; i < 2; i++) xbar_init(m_empty + 8 * i, MODE == 0 ? 8 : 4);
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
    constexpr uint32_t tmem = 0;                                            // all 512 columns are this CTA's, so no address below adds it
    const uint32_t n_items = *a.n_groups * a.tiles;

    if (warp == R::TMA) {
        // ---------------- packed rows ----------------
        const uint32_t steps = (a.units * UNIT + Fm::COLS - 1) / Fm::COLS, el = xelect();
        const uint32_t nb = a.w0.k_storage >> 8, side = 128 * nb * Fm::SIDE_BLOCK;    // bytes of a tile's scales that lie apart from the codes
        uint32_t st = 0, ph = 0, issued = 0, ring = 0;
        bool ok = true;
        uint32_t next_expert = blockIdx.x < n_items ? a.groups[blockIdx.x / a.tiles].expert : 0u;      // asked for an item ahead
        for (uint32_t it = blockIdx.x; it < n_items && ok; it += gridDim.x) {
            const uint32_t expert = next_expert, row0 = (it % a.tiles) * STEP;
            if (it + gridDim.x < n_items) next_expert = a.groups[(it + gridDim.x) / a.tiles].expert;
            // Where two items' scales are held and an item is so few stages that the stages alone would reach a third one (down with few logical
            // columns of long stored rows), these scales wait until the item before the last has been dequantised.  Its last stage is its slot's
            // latest use.  (Gate/up stores what it multiplies: nine stages where two are held.  Asking there as well cost a layer of seven tokens 0.4%.)
            if (MODE == 1 && Fm::SIDE && ring_mask == 1 && steps + 1 < Fm::STAGES && issued >= 2 * steps) {
                const uint32_t last = issued - steps - 1;
                if (!(ok = xbar_wait<200>(w_empty + 8 * (last % Fm::STAGES), (last / Fm::STAGES) & 1u, dead, a.status, w0))) break;
            }
            for (uint32_t s = 0; s < steps; s++) {
                if (!(ok = xbar_wait<200>(w_empty + 8 * st, ph ^ 1u, dead, a.status, w0))) break;
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
            xbar_wait(w_full + 8 * st, ph, &never, a.status, w1);
        }
    } else if (warp >= R::ACT) {
        // ---------------- activation rows: hi by one warp, lo by the other ----------------
        // eight lanes take the 128 bytes of a row, so an instruction touches four lines of the cache and not thirty-two
        const uint32_t part = warp - R::ACT, piece = lane & 7u, sub = lane >> 3;
        if (MODE == 1) asm volatile("griddepcontrol.wait;" ::: "memory");
        uint32_t n = 0, un = 0;
        bool ok = true;
        const __half *in = (part ? a.in_lo : a.in_hi) + piece * 8, *sums = part ? a.sum_lo : a.sum_hi;
        // an item's group and rows are asked for while the one before is being copied
        auto pair_of = [&](const XGroup &g) { return lane < g.count ? (a.row_to_pair ? a.row_to_pair[g.first + lane] : g.first + lane) : 0u; };
        XGroup next = {};
        uint32_t next_pair = 0, item = 0;
        if (blockIdx.x < n_items) { next = a.groups[blockIdx.x / a.tiles]; next_pair = pair_of(next); }
        for (uint32_t it = blockIdx.x; it < n_items && ok; it += gridDim.x, item++) {
            const XGroup grp = next;
            const uint32_t src_row = next_pair / a.k_div;
            if (it + gridDim.x < n_items) next = a.groups[(it + gridDim.x) / a.tiles];
            const __half *src[8];                                             // rows sub, sub + 4, ...
#pragma unroll
            for (uint32_t i = 0; i < 8; i++) src[i] = in + (uint64_t)__shfl_sync(0xffffffffu, src_row, sub + 4 * i) * a.in_pitch;
            const uint32_t rounds = grp.count > 16 ? 8u : 4u, rows = rounds * 4;
            const __half *ssrc = sums + (uint64_t)src_row * a.units * 16u;
            const uint32_t dst_row = sbase + XM_B + part * XB_ONE + sub * 128u;
            for (uint32_t u = 0; u < a.units && ok; u++, un++) {
#pragma unroll 1
                for (uint32_t c = 0; c < SPU; c++, n++) {
                    if (!(ok = xbar_wait<64>(done + 16 * (n & (NB - 1)), ((n - NB) >> NBLOG) & 1u, dead, a.status, w0) &&
                               xbar_wait<64>(done + 16 * (n & (NB - 1)) + 8, ((n - NB) >> NBLOG) & 1u, dead, a.status, w0))) break;
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
                        if (u == 0) {                                          // for the read-back, which must not wait for global memory between items
                            const uint32_t at = (item & 7u) * XTOK + lane;
                            if (part == 0 && a.row_to_pair) xcp4(sbase + XM_PAIR + at * 4, a.row_to_pair + grp.first + lane, bytes >> 2);
                            if (part == 0 && lane == 0) xcp16(sbase + XM_GROUP + (item & 7u) * 16, a.groups + it / a.tiles, 16);
                            if (part == 1 && MODE == 0) xcp4(sbase + XM_ROW + at * 4, a.in_scale + src_row, bytes >> 2);
                        }
                        if (MODE == 1 && part == 0)
                            xcp4(sbase + XM_BSC + ((un & 7u) * XTOK + lane) * 4u, a.in_scale + (uint64_t)src_row * a.units + u, bytes >> 2);
                    }
                    // the copies hand the step over themselves when they land (the MMA warps order them before the tensor core's reads)
#pragma unroll
                    for (uint32_t m = 0; m < 2; m++)
                        asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(full + 8 * ((n & (NB - 1)) * 2 + m)) : "memory");
                    if (u == 0 && c == 0) next_pair = pair_of(next);
                }
            }
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
    } else if (warp >= R::MMA) {
        // ---------------- tcgen05.mma issue: one warp a tile, so that one's waits and commits lie under the other's products ----------------
        // The whole warp walks this loop and every value an instruction names is warp-uniform for the compiler too (waits
        // end in a vote, counts come out of a reduction, TMEM starts at column 0 because all of it is ours, no calls):
        // otherwise each operand of each MMA is moved to a uniform register first, which costs 58 cycles an instruction.
        const uint32_t el = xelect();
        const uint64_t b_desc = xdesc_sw128(sbase + XM_B), s_desc = xdesc_sums(sbase + XM_SUMS);
        auto wait = [&](uint32_t bar, uint32_t parity, uint32_t &spent) -> bool {
            bool done = __all_sync(0xffffffffu, xbar_try(bar, parity));
            if (done) return true;
            const uint32_t start = clock();
            bool give_up = false;
            while (!done && !give_up) {
                done = __all_sync(0xffffffffu, xbar_try(bar, parity));
                if (!done && (uint32_t)clock() - start > (1u << 31)) { *dead = 1; atomicOr(a.status, QW4SH_ERR_STATE); }
                give_up = __any_sync(0xffffffffu, !done && *dead);
            }
            spent += clock() - start;
            return done;
        };
        const uint32_t items = __reduce_max_sync(0xffffffffu, n_items), units = a.units;
        const uint32_t m = warp - R::MMA;
        uint32_t n = 0, un = 0;
        bool ok = true;
        uint32_t next_count = blockIdx.x < items ? a.groups[blockIdx.x / a.tiles].count : 0u;          // asked for an item ahead
        for (uint32_t it = blockIdx.x; it < items && ok; it += gridDim.x) {
            const uint32_t tok = __any_sync(0xffffffffu, next_count > 16) ? 32u : 16u;
            if (it + gridDim.x < items) next_count = a.groups[(it + gridDim.x) / a.tiles].count;
            const uint32_t idesc = (1u << 4) | ((tok >> 3) << 17) | ((XROWS >> 4) << 24);   // D F32, A and B F16, K-major
            for (uint32_t u = 0; u < units && ok; u++, un++) {
                const uint32_t ub = un & 1u, q_bar = q_empty + 8 * (ub * 2 + m), q_ph = ((un - 2) >> 1) & 1u;
#pragma unroll 1
                for (uint32_t c = 0; c < SPU; c++, n++) {
                    const uint32_t slot = n & (NB - 1), ph = (n >> NBLOG) & 1u;
                    if (!(ok = wait(full + 8 * (slot * 2 + m), ph, w0))) break;
                    if (c == 0 && !(ok = wait(q_bar, q_ph, w2))) break;                          // the unit before last has been read
                    xtc_after();
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                    const uint64_t bd = b_desc + slot * (BSTEP >> 4);
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
                    if (Fm::MIN && c == SPU - 1) {
                        // M has one buffer: the previous unit's has to be read
                        __syncwarp();
                        if (!(ok = wait(m_empty + 8 * m, (un - 1) & 1u, w2))) break;
                        xtc_after();
                        if (el) {
                            const uint64_t sd = s_desc + (un & 3u) * ((2 * XS_ONE) >> 4);
                            xmma(XT_M + m * 32, XT_AM + ub * 16 + m * 8, sd, idesc, 0u);
                            xmma(XT_M + m * 32, XT_AM + ub * 16 + m * 8, sd + (XS_ONE >> 4), idesc, 1u);
                        }
                    }
                    if (el) xtc_commit(done + 8 * (slot * 2 + m));
                }
            }
        }
    } else if (warp < R::EPI) {
        // ---------------- dequantise: packed bytes -> exact halves in TMEM ----------------
        // Four warps a tile.  A step goes to TMEM in four parts; the next step's packed words are fetched before the stores are waited for.  All of
        // a stage's steps are unrolled, so that what remains beside the weights is counters: the issue slots bound the kernel.
        const uint32_t m = warp >> 2, row = (warp & 3u) * 32 + lane, quad = ((warp & 3u) * 32) << 16, nb = a.w0.k_storage >> 8;
        constexpr uint32_t STPS = STCH / CPS;                                 // steps per stage
        const uint32_t steps = a.units * SPU, stages = (steps + STPS - 1) / STPS, side = 128 * nb * Fm::SIDE_BLOCK;
        const uint32_t mine = n_items > blockIdx.x ? (n_items - 1 - blockIdx.x) / gridDim.x + 1 : 0, total = mine * stages;
        uint32_t *dsc = reinterpret_cast<uint32_t *>(smem + XM_DSC) + m * 512 + row;
        const uint32_t side_row = sbase + xm_side<F>() + m * side + row * nb * Fm::SIDE_BLOCK, tiles0 = sbase + xm_weights<F>() + m * Fm::TILE;
        const uint32_t a_at = quad + XT_A + m * 64, am_at = quad + XT_AM + m * 8, full_m = full + 8 * m;
        uint32_t st = 0, ph = 0, ks = 0, ring = 0, it = blockIdx.x;           // stage, its phase, its place in the item, the item
        uint32_t n = 0, un = 0xffffffffu, beside = 0;                         // steps before, units begun before
        bool ok = true;
        XDeq<F> q;
        auto new_item = [&]() {                                               // wide form: the row's power of two
            if (F == T_WIDE) {
                const uint64_t at = (uint64_t)a.groups[it / a.tiles].expert * a.w0.n_out + (it % a.tiles) * STEP + row;
                beside = __float_as_uint(__ldg((m ? a.row_scale1 : a.row_scale0) + at + (MODE == 1 ? m * 128u : 0u)));
            } else beside = side_row + ring * 2 * side;
        };
        if (total) {
            new_item();
            if ((ok = xbar_wait(w_full, 0, dead, a.status, w0))) q.template load<0>(tiles0, row, smem + xm_tables<F>(), beside, 0, lane);
        }
        for (uint32_t k = 0; k < total && ok; k++) {
            const uint32_t left = steps - ks * STPS, emptied = w_empty + 8 * st, tile = tiles0 + st * 2 * Fm::TILE, ks_now = ks;
            if (++st == Fm::STAGES) { st = 0; ph ^= 1u; }
            if (++ks == stages) { ks = 0; ring = (ring + 1) & ring_mask; it += gridDim.x; }
            const bool more = k + 1 < total;
            const bool full_too = more && __all_sync(0xffffffffu, xbar_test(w_full + 8 * st, ph));
            auto step = [&](auto SPC) {
                constexpr int SP = decltype(SPC)::value;
                if (SP > 0 && (SP >= left || !ok)) return;
                // asked early, used after the first part; before there were two steps, the barrier's phase before its first
                const uint32_t freed = done + 8 * (((n - 2) & (NB - 1)) * 2 + m), freed_ph = ((n - 2) >> NBLOG) & 1u;
                const bool free = xbar_test(freed, freed_ph);
                const uint32_t at = a_at + (n & 1u) * 128;
                const bool first = STPS % SPU == 0 ? SP % SPU == 0 : n % SPU == 0;
                uint32_t v[16];
                q.template part<SP, 0>(v);
                if (!free && !(ok = xbar_wait(freed, freed_ph, dead, a.status, w1))) return;
                xtc_after();
                xst16(at, v);
                q.template part<SP, 1>(v); xst16(at + 16, v);
                q.template part<SP, 2>(v); xst16(at + 32, v);
                if (first) {
                    un++;
                    if (Fm::MIN) {
                        uint32_t mn[8];
                        q.template minima<MODE, SP>(mn);
                        xst8(am_at + (un & 1u) * 16, mn);
                    }
                    dsc[(un & 3u) * 128] = q.word();
                }
                q.template part<SP, 3>(v); xst16(at + 48, v);
                constexpr int NEXT = SP + 1 < (int)STPS ? SP + 1 : 0;
                if (NEXT && NEXT < left) q.template load<NEXT>(tile, row, smem + xm_tables<F>(), beside, ks_now, lane);
                else if (full_too) {
                    if (ks == 0) new_item();
                    q.template load<0>(tiles0 + st * 2 * Fm::TILE, row, smem + xm_tables<F>(), beside, ks, lane);
                }
                xst_wait();
                xtc_before();
                __syncwarp();
                xbar_arrive_if(full_m + 8 * (n & (NB - 1)) * 2, lane == 0);
                if (!NEXT || NEXT >= left) xbar_arrive_if(emptied, lane == 0);
                n++;
            };
            step(std::integral_constant<int, 0>());
            if constexpr (STPS > 1) step(std::integral_constant<int, 1>());
            if constexpr (STPS > 2) { step(std::integral_constant<int, 2>()); step(std::integral_constant<int, 3>()); }
            if (more && !full_too && ok) {
                if (ks == 0) new_item();
                if ((ok = xbar_wait(w_full + 8 * st, ph, dead, a.status, w0))) q.template load<0>(tiles0 + st * 2 * Fm::TILE, row, smem + xm_tables<F>(), beside, ks, lane);
            }
        }
    } else {
        // ---------------- read-back: TMEM -> scales -> SwiGLU + split / store ----------------
        // Mode 0: four warps take the lower half of the group's tokens, four the upper, each of both tiles, so that gate and up of a token meet in a
        // thread.  Mode 1: four warps a tile, all tokens (one wait a unit).  A unit's accumulators are given back as soon as they are in
        // registers, before the last arithmetic on them: the next unit's products wait for M, which has one buffer.
        typedef unsigned long long u64;
        constexpr uint32_t MINE = MODE == 0 ? XTOK / 2 : XTOK, TILES = MODE == 0 ? 2 : 1;         // most tokens of a warp, tiles of a warp
        const uint32_t part = (warp - R::EPI) >> 2, row = (warp & 3u) * 32 + lane, quad = ((warp & 3u) * 32) << 16, pt = tid - (R::EPI + 4 * part) * 32;
        const uint32_t *dsc = reinterpret_cast<const uint32_t *>(smem + XM_DSC) + row;
        float *hand = reinterpret_cast<float *>(smem + XM_HAND) + part * (XTOK / 2) * XPITCH;
        uint32_t un = 0, item = 0;
        bool ok = true;                                                       // once false: no more waits, but every CTA-internal barrier below is still met
        for (uint32_t it = blockIdx.x; it < n_items; it += gridDim.x, item++) {
            const uint32_t tile = it % a.tiles;
            const XGroup *grp = reinterpret_cast<const XGroup *>(smem + XM_GROUP) + (item & 7u);       // there with the item's first step
            uint32_t first = 0, mine = 0;                                     // this warp's tokens of the group
            u64 acc2[TILES][MINE / 2];                                        // [tile][tokens], two to an instruction
#pragma unroll
            for (uint32_t m = 0; m < TILES; m++)
#pragma unroll
                for (uint32_t n = 0; n < MINE / 2; n++) acc2[m][n] = 0;
            for (uint32_t u = 0; u < a.units; u++, un++) {
                const uint32_t last = (un + 1) * SPU - 1;                    // the unit's last step
#pragma unroll
                for (uint32_t t = 0; t < TILES; t++) {
                    const uint32_t m = MODE == 0 ? t : part;
                    if (ok) ok = xbar_wait<32>(done + 8 * ((last & (NB - 1)) * 2 + m), (last >> NBLOG) & 1u, dead, a.status, w0);
                    if (!ok) continue;
                    xtc_after();
                    if (t == 0 && u == 0) {
                        const uint32_t count = grp->count, half = (count + 7u) / 8u * 4u;
                        if (MODE == 1) mine = count;
                        else { first = part ? half : 0; mine = part ? (count > half ? count - half : 0) : min(count, half); }
                    }
                    const uint32_t word = dsc[(m * 4 + (un & 3u)) * 128];
                    float d, dmin = 0.0f;
                    if (F == T_WIDE) d = __uint_as_float(word);
                    else if (F == T_IQ2_XXS) d = xhalf_bits(word) * 0.125f;
                    else { d = xhalf_bits(word) * XUP; dmin = -xhalf_bits(word >> 16); }
                    const u64 d2 = xpair(d, d), dmin2 = xpair(dmin, dmin);
                    const ulonglong2 *bsc = reinterpret_cast<const ulonglong2 *>(smem + XM_BSC + (un & 7u) * (XTOK * 4));
                    const uint32_t qa = quad + XT_Q + (un & 1u) * 64 + m * 32 + first, ma = quad + XT_M + m * 32 + first;
#pragma unroll
                    for (uint32_t h = 0; h < MINE; h += 16) {
                        if (h == 0 || h < mine) {
                            uint32_t qv[16], mv[16];
                            if (Fm::MIN) xld_qm(qa + h, ma + h, qv, mv);
                            else xld_q(qa + h, qv);
                            if (h + 16 >= MINE || h + 16 >= mine) {
                                xtc_before();
                                __syncwarp();
                                if (Fm::MIN) xbar_arrive_if(m_empty + 8 * m, lane == 0);
                                xbar_arrive_if(q_empty + 8 * ((un & 1u) * 2 + m), lane == 0);
                            }
#pragma unroll
                            for (uint32_t n4 = 0; n4 < 16; n4 += 4) {
                                if (h + n4 < mine) {
                                    ulonglong2 sc = make_ulonglong2(0, 0);
                                    if (MODE == 1) sc = bsc[(h + n4) / 4];
#pragma unroll
                                    for (uint32_t i = 0; i < 4; i += 2) {
                                        u64 &to = acc2[t][(h + n4 + i) / 2];
                                        const u64 qq = xpair_bits(qv[n4 + i], qv[n4 + i + 1]), mm = Fm::MIN ? xpair_bits(mv[n4 + i], mv[n4 + i + 1]) : 0;
                                        if (MODE == 0) {
                                            to = xfma2(d2, qq, to);
                                            if (Fm::MIN) to = xfma2(dmin2, mm, to);
                                        } else {
                                            u64 v = xmul2(d2, qq);
                                            if (Fm::MIN) v = xfma2(dmin2, mm, v);
                                            to = xfma2(i ? sc.y : sc.x, v, to);
                                        }
                                    }
                                }
                            }
                        }
                    }
                }
            }
            const uint32_t *pairs = reinterpret_cast<const uint32_t *>(smem + XM_PAIR) + (item & 7u) * XTOK + first;
            const uint32_t pair0 = a.row_to_pair || !mine ? 0u : grp->first + first;      // the shared expert's rows are in token order
            auto sum_of = [&](uint32_t t, uint32_t n) { return __uint_as_float((uint32_t)(acc2[t][n / 2] >> (32 * (n & 1u)))); };
            if constexpr (MODE == 0) {
                const float *row_scale = reinterpret_cast<const float *>(smem + XM_ROW) + (item & 7u) * XTOK + first;
                asm volatile("bar.sync %0, 128;" ::"r"(1 + part) : "memory");  // the hand-over tile's previous content has been taken
#pragma unroll
                for (uint32_t n4 = 0; n4 < MINE; n4 += 4) {
                    if (n4 >= mine) break;
                    const float4 s4 = *reinterpret_cast<const float4 *>(row_scale + n4);
                    const float sv[4] = {s4.x, s4.y, s4.z, s4.w};
#pragma unroll
                    for (uint32_t i = 0; i < 4; i++) {                        // values beyond the group's last token are written and not read
                        const float g = sum_of(0, n4 + i) * sv[i], up = sum_of(1, n4 + i) * sv[i];
                        const float e = __expf(-fabsf(g));
                        hand[(n4 + i) * XPITCH + row + (row >> 4)] = g * __fdividef(g >= 0.0f ? 1.0f : e, 1.0f + e) * up;
                    }
                }
                asm volatile("bar.sync %0, 128;" ::"r"(1 + part) : "memory");
                // eight threads a token, sixteen columns each: the tile's power of two, hi and lo, sums of eight columns
                const uint32_t n = pt >> 3, seg = pt & 7u;
                const bool live = n < mine;
                const uint32_t pair = live ? (a.row_to_pair ? pairs[n] : pair0 + n) : 0;
                float v[2][8], top = 0.0f;
#pragma unroll
                for (int i = 0; i < 16; i++) { v[i >> 3][i & 7] = live ? hand[n * XPITCH + seg * 17 + i] : 0.0f; top = fmaxf(top, fabsf(v[i >> 3][i & 7])); }
                for (int o = 1; o < 8; o <<= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, o));
                float up, down;
                xscale_of(top, up, down);
                if (live && ok) {
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
                    // finite values are at most 1024 here, so a sum that is not finite has a term that is not, and the other way round
                    if (((__float_as_uint(s8[0]) & 0x7f800000u) == 0x7f800000u) | ((__float_as_uint(s8[1]) & 0x7f800000u) == 0x7f800000u)) atomicOr(a.status, QW4SH_ERR_NONFINITE);
                    const __half2 sh = __floats2half2_rn(s8[0], s8[1]);
                    const float2 f = __half22float2(sh);
                    const uint64_t sat = (uint64_t)pair * (a.w0.n_out >> 3) + tile * 16 + seg * 2;
                    *reinterpret_cast<__half2 *>(a.osum_hi + sat) = sh;
                    *reinterpret_cast<__half2 *>(a.osum_lo + sat) = __floats2half2_rn(s8[0] - f.x, s8[1] - f.y);
                    if (seg == 0) a.out_scale[(uint64_t)pair * (a.w0.n_out >> 7) + tile] = down;
                }
            } else if (ok) {
                float *to = a.out + tile * 256 + part * 128 + row;
                float bad = 0.0f;                                             // becomes NaN where a value is not finite
#pragma unroll
                for (uint32_t n4 = 0; n4 < MINE; n4 += 4) {
                    if (n4 >= mine) break;
                    const uint4 p4 = a.row_to_pair ? *reinterpret_cast<const uint4 *>(pairs + n4) : make_uint4(pair0 + n4, pair0 + n4 + 1, pair0 + n4 + 2, pair0 + n4 + 3);
                    const uint32_t pv[4] = {p4.x, p4.y, p4.z, p4.w};
#pragma unroll
                    for (uint32_t i = 0; i < 4; i++)
                        if (n4 + i < mine) {
                            const float v = sum_of(0, n4 + i);
                            bad = fmaf(v, 0.0f, bad);
                            to[(uint64_t)pv[i] * a.w0.n_out] = v;
                        }
                }
                if (bad != 0.0f) atomicOr(a.status, QW4SH_ERR_NONFINITE);
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
