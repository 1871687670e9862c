// The whole MoE layer for a decode step of up to four tokens as ONE persistent kernel (sm_100a).
//
// One CTA per SM, all resident at once; picoforge src/qwen4_moe.c:334-382 is the CPU statement of
// the sequence.  The CTAs have two roles.
//
// CHAIN CTAs (the first NC) own the reference's router arithmetic: every logit is one chain of K
// separately rounded multiply-adds in ascending k (src/qwen4_packed.c:164-173), 32 router rows
// per CTA, one warp per token, lane = row, the rows streamed through a swizzled cp.async ring by
// the CTA's other warps.  A chain is 2048 dependent adds, about 9 k cycles whatever else happens,
// so it is kept OFF the critical path: when all chains are done, chain CTA t routes token t
// (libm-exact softmax, serial exp-sum, top-k, renormalisation: src/qwen4_moe.c:209-247) and
// publishes ids and weights.
//
// STREAMING CTAs (all others) do not wait for that.  They compute tree-summed logits of their 3-4
// router rows at once (phase A), exchange them through the first grid-wide barrier, take the
// top-k SET of every token from those logits (a speculation: the tree sums differ from the chains
// in the last bits, which matters only for a near-tie at the k-th place) and stream the gate/up
// rows of the experts in that set (phase B).  At the second barrier they also wait for the chain
// CTAs' routes and compare: if a token's exact expert set differs from the speculated one, phase B
// runs again with the exact ids, so ids and weights are always the reference's bits.  Phase C
// (down projection, weighted combine, sigmoid-gated shared expert) uses the exact weights.
//
//   A  x -> shared memory, int8 digit pairs of x, tree-summed logits of rows sc, sc + NS, ...
//   B  work unit = 8 gate rows + the same 8 up rows of one expert (gate in MMA rows 0-7, up in
//      8-15); a unit is cut into slices of 512 columns dealt to the CTA's warps, each warp fetching
//      slices into its own ring (Q4_K: one 3-D tensor-map request per matrix; IQ2_XXS: one bulk copy
//      of a block of its expanded image) and feeding int8 tensor-core MMAs with the codes.
//      Units come in granules of four (32 activation columns): the warp that sums a granule's
//      slices applies SwiGLU and writes the activation as int8 digit pairs with ONE SCALE PER
//      32-COLUMN CHUNK, so that no row maximum has to cross the grid and phase C starts with a
//      bulk copy of ready-made digits.
//   C  streaming CTA sc owns 16 columns of y: its warps split the sources (shared expert +
//      distinct routed experts), each runs the 16 x K down tile on the tensor cores against the
//      digits of the pair's activation, scales by the route weight (or the sigmoid gate), and the
//      partial sums are added in warp order: y is deterministic.  The digits and the first tiles are
//      fetched under the comparison of the routes; a repair drops them.
//
// The kernel is launched as a normal grid of one CTA per SM with programmatic stream
// serialisation: the next layer's launch may begin while this one drains, and everything that
// touches memory another launch writes comes after griddepcontrol.wait.  All CTAs are resident
// together because each needs more than half of an SM's shared memory and the grid is the SM
// count; every wait (mbarrier, counter) is bounded: after about a second the kernel records
// QW4SH_ERR_STATE and leaves.
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include <stdio.h>
#include <string.h>

#include "cuda_shim.h"
#include "formats.cuh"
#include "iq2n.cuh"
#include "route.cuh"

namespace qw4 {

constexpr int FW = 12;                          // warps per CTA (with sixteen a Q4_K token took 2% longer, four IQ2_XXS tokens the same)
constexpr int FT = FW * 32;
constexpr int FTOK = 4;                         // tokens per launch
constexpr int FMAXK = 16;                       // top-k limit
constexpr int FMAXE = 512;                      // experts limit
constexpr int FMAXSRC = FTOK * FMAXK + 1;       // shared expert + distinct routed experts
constexpr int FRMAX = 4;                        // router rows per streaming CTA
constexpr int FNS = 2;                          // ring stages per warp, gate/up phase (three stages fit and were measured: no faster)
constexpr int FNC = 2;                          // ring stages per warp, down phase
constexpr uint32_t FSTAGE = 4608;               // bytes per ring stage: sixteen rows x 512 columns (4608 of Q4_K, 3392 of the expanded IQ2_XXS image)
constexpr uint32_t FSMEM = 226 * 1024;          // most dynamic shared memory of a launch: an SM's 227 KB less a kilobyte for static variables
constexpr uint32_t FZP = FMAXE + 4;             // pitch of a logit row in shared memory (floats)
constexpr int CROWS = 32;                       // router rows per chain CTA (lane = row).  64 rows (two chain warps per token, nine
                                                // chain CTAs) evened out the streaming CTAs' shares but ran the chains at 42 k cycles
                                                // instead of 25 k, and the step at 44.4 us instead of 42.0
constexpr int CCH = 512;                        // columns per chunk: a bulk copy of 2 KB per row
constexpr int CSTG = 2;                         // chunks in flight in a chain CTA: 128 KB, half of K = 2048, before the first addition
constexpr uint32_t CPITCH = CCH * 4 + 16;       // bytes per row of a chunk: the pad keeps the lanes' 128-bit reads apart
// words of the sync array
enum : uint32_t { S_FAST = 0, S_CHAIN = 1, S_ROUTED = 2, S_ACT0 = 3, S_ACT1 = 4, S_EXITS = 5, S_ROUTE_FAIL = 6, S_CLOCKS = 8, S_REPAIRS = 48, S_MARKS = 256 };

struct FusedArgs {
    DevTensor w[8];                             // router, gate, up, down, sgate, sup, sdown, srouter
    const float *x;
    float *y;
    uint32_t tokens, hidden, experts, top_k, inter, shared_inter;
    int norm, router_mode;                      // 0 exact, 1 fast, 2 exact with a wrong speculation forced (test aid)
    float *logits, *shared_logit;               // [T, E], [T]: the logits the routes were made from
    float *logits_fast;                         // [T, fast_pitch]: tree sums, the shared router's at column E
    uint32_t fast_pitch;
    uint32_t *ids;                              // [T, k]
    float *weights;                             // [T, k]
    uint8_t *aq;                                // [T*k + T][2][ap] activation digits (pairs, then the shared expert's rows)
    float2 *asc;                                // [T*k + T][imax / 32] per chunk: scale, sum of the chunk's represented values
    uint32_t *ids_out;
    float *weights_out;
    uint32_t *sync;                             // counters (S_*), then the phase clocks of the first streaming CTA
    uint32_t *status;
    uint32_t partial_slices;                    // capacity of the partial-sum buffer (slices per CTA)
    uint32_t chain_ctas;                        // NC
    uint32_t clear;                             // see make_fplan
    long long t0;                               // (device side) this CTA's clock at its start
    HcAdd hc;                                   // hyper-connection add applied where y is written (residual nullptr: none)
    uint32_t *status_mirror;                    // pinned host words [4] that receive the status words at the end, or nullptr
};

// One distinct source of phase C / one expert of phase B.
struct Src {
    uint16_t expert; uint8_t mask, shared;
    uint32_t slots;                             // slot of token t in byte t
    __device__ __forceinline__ uint32_t slot(uint32_t t) const { return (slots >> (8 * t)) & 0xffu; }
};

// Shared-memory plan of a streaming CTA (byte offsets), the same on host and device.  `clear`: phase C keeps clear of the digit image of x, so that
// its first copies may be under way while it is still open whether phase B has to run again.  `region` is
// reused by the three phases; the digit image of x lives at its start through phases A and B.
struct FPlan {
    uint32_t bars, ids, wts, idx, wtx, misc, tokmask, slotmap, src, region, total;
    uint32_t kp;                                // pitch of one digit row of x
    uint32_t xq, xsum;                          // phases A and B (inside region)
    uint32_t xf, xf_pitch, rows, row_pitch;     // phase A
    uint32_t zs, ring, partial;                 // phase B
    uint32_t aq, ap, asc, tiles, cpartial;      // phase C
};
__host__ __device__ inline FPlan make_fplan(uint32_t hidden, uint32_t inter_max, uint32_t rows_c, uint32_t partial_slices, bool clear) {
    FPlan p;
    uint32_t at = 0;
    p.bars = at; at += 512;
    p.ids = at; at += FTOK * FMAXK * 4;
    p.wts = at; at += FTOK * FMAXK * 4;
    p.idx = at; at += FTOK * FMAXK * 4;         // the exact routes as published
    p.wtx = at; at += FTOK * FMAXK * 4;
    p.misc = at; at += 1024;                    // floats [0..3] x maxima then scales, [4..7] shared logits; words from +64; +512: digitiser constants of x
    p.tokmask = at; at += FMAXE;
    p.slotmap = at; at += FMAXE * 4;
    p.src = at; at += ((FMAXSRC * 8 + 127) & ~127u);
    p.region = at;
    p.kp = hidden + 32;
    uint32_t head = 0;
    p.xq = head; head += 8 * p.kp;
    p.xsum = head; head += FTOK * (hidden / 32) * 8;
    head = (head + 127) & ~127u;
    // phase A
    uint32_t a = head;
    p.xf_pitch = hidden * 4 + 16;
    p.xf = a; a += FTOK * p.xf_pitch;
    p.row_pitch = hidden * 4 + 16;
    p.rows = a; a += FRMAX * p.row_pitch + 8 * 16 * 4;      // + the partial sums of the fast logits
    // phase B: the logit keys are dead before the first copy lands in the ring
    uint32_t b = head;
    p.zs = b;
    p.ring = b; b += FW * FNS * FSTAGE;
    if (b < head + FTOK * FZP * 4) b = head + FTOK * FZP * 4;
    p.partial = b; b += partial_slices * 256;
    // phase C
    uint32_t c = clear ? head : 0;
    p.ap = inter_max + 32;
    p.aq = c; c += rows_c * 2 * p.ap;
    c = (c + 127) & ~127u;
    p.asc = c; c += rows_c * (inter_max / 32) * 8;
    c = (c + 127) & ~127u;
    p.tiles = c; c += FW * FNC * FSTAGE;
    p.cpartial = c; c += FW * 32 * 8;
    uint32_t m = a > b ? a : b;
    m = m > c ? m : c;
    p.total = p.region + m;
    return p;
}
// Shared-memory plan of a chain CTA.
struct CPlan { uint32_t bars, misc, xf, xf_pitch, ring, route, total; };
__host__ __device__ inline CPlan make_cplan(uint32_t hidden) {
    CPlan p;
    uint32_t at = 0;
    p.bars = at; at += 512;
    p.misc = at; at += 512;
    p.xf_pitch = hidden * 4 + 16;
    p.xf = at; at += FTOK * p.xf_pitch;
    at = (at + 127) & ~127u;
    p.ring = at; p.route = at;                  // the routing starts when the chains are done
    const uint32_t ring = CSTG * CROWS * CPITCH, route = (uint32_t)sizeof(RouteShared) + RT_PITCH * 4;
    at += ring > route ? ring : route;
    p.total = at;
    return p;
}

// ---- small PTX helpers --------------------------------------------------------------------
__device__ __forceinline__ uint32_t fs_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void fbar_init(uint64_t *bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(fs_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void fbar_expect(uint64_t *bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(fs_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void fbar_arrive(uint64_t *bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(fs_u32(bar)) : "memory");
}
__device__ __forceinline__ bool fbar_try(uint64_t *bar, uint32_t parity) {
    uint32_t ok;
    asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
                 : "=r"(ok) : "r"(fs_u32(bar)), "r"(parity) : "memory");
    return ok != 0;
}
// Bounded wait (about a second); false with the error bit set when it runs out.
__device__ __forceinline__ bool fbar_wait(uint64_t *bar, uint32_t parity, uint32_t *status) {
    if (fbar_try(bar, parity)) return true;
    const long long start = clock64();
    while (!fbar_try(bar, parity)) {
        if (clock64() - start > (1ll << 31)) { atomicOr(status, QW4SH_ERR_STATE); return false; }
    }
    return true;
}
__device__ __forceinline__ void fbulk(void *dst_smem, const void *src, uint32_t bytes, uint64_t *bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(fs_u32(dst_smem)), "l"(src), "r"(bytes), "r"(fs_u32(bar)) : "memory");
}
// Rows [y, y + 8) of expert z, 32-bit words [x, x + box) of each, through a 3-D tensor map {words per row, rows per
// expert, experts}: one request for the eight row pieces of a unit slice, which lie a row apart in memory.
__device__ __forceinline__ void ftma_rows(void *dst_smem, const CUtensorMap *map, uint32_t x, uint32_t y, uint32_t z, uint64_t *bar) {
    asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
                 ::"r"(fs_u32(dst_smem)), "l"(map), "r"(x), "r"(y), "r"(z), "r"(fs_u32(bar)) : "memory");
}
__device__ __forceinline__ void fprefetch_l2(const void *src, uint32_t bytes) {
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void fproxy_fence() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ uint32_t fld_acquire(const uint32_t *p) {
    uint32_t v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void fred_release(uint32_t *p) {
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(p) : "memory");
}
__device__ __forceinline__ void fmma_zero(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
                 : "=r"(c[0]), "=r"(c[1]), "=r"(c[2]), "=r"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "r"(0));
}

// Shared-memory loads by 32-bit shared address, volatile: they read memory that bulk copies rewrite between uses
// and must stay behind the mbarrier wait that precedes them in program order.
__device__ __forceinline__ uint2 lds_ring2(uint32_t a) {
    uint2 v;
    asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(a));
    return v;
}
__device__ __forceinline__ uint32_t lds_ring_u16(uint32_t a) {
    uint32_t v;
    asm volatile("ld.shared.u16 %0, [%1];" : "=r"(v) : "r"(a));
    return v;
}
// Thread 0 waits until *counter >= expected (bounded); the verdict reaches every thread.
// False (CTA-uniform) when the wait ran out.
__device__ __forceinline__ bool wait_counter(const uint32_t *counter, uint32_t expected, uint32_t *status) {
    int ok = 1;
    if (threadIdx.x == 0) {
        const long long start = clock64();
        while (fld_acquire(counter) < expected) {
            if (clock64() - start > (1ll << 31)) { atomicOr(status, QW4SH_ERR_STATE); ok = 0; break; }
        }
    }
    return __syncthreads_and(ok) != 0;
}
// All threads' earlier global writes are ordered before one release increment (the barrier puts them before it, and a release is cumulative).
__device__ __forceinline__ void arrive_counter(uint32_t *counter) {
    __syncthreads();
    if (threadIdx.x == 0) fred_release(counter);
}

// ---- half blocks (128 columns) on the tensor cores ----------------------------------------------
// MMA k-slots are permuted so that lane (g, t) owns the eight consecutive columns 8t..8t+7 of
// every 32-column chunk, for MMA rows g and g + 8 and for activation column g (token g >> 1,
// digit g & 1).  f0 += row g . x[token t], f1 += row g+8 . x[token t].
//
// Halves (phase B): the activation has one scale per row, so the sums stay integers over a half
// block and the results are in units of the token's digit scale; xsum holds the token's digit
// sums (Q4_K's min term).
// HalvesS (phase C): one scale per 32-column chunk; `asc` points at the token row's (scale, chunk
// sum) pairs and the results are plain values.
template <uint32_t TYPE> struct Halves;
template <uint32_t TYPE> struct HalvesS;

__device__ __forceinline__ void q4k_scales(const uint4 h0, uint32_t hb, uint32_t &sc, uint32_t &mn) {
    if (hb == 0) { sc = h0.y & 0x3f3f3f3fu; mn = h0.z & 0x3f3f3f3fu; }
    else { sc = (h0.w & 0x0f0f0f0fu) | ((h0.y >> 2) & 0x30303030u); mn = ((h0.w >> 4) & 0x0f0f0f0fu) | ((h0.z >> 2) & 0x30303030u); }
}

// Q4_K: r0 / r1 point at the first 144-byte block of the two rows; `halves` half blocks follow.
template <> struct Halves<T_Q4_K> {
    static __device__ __forceinline__ void run(const uint8_t *r0, const uint8_t *r1, uint32_t halves, uint32_t t, const uint8_t *xq, const int2 *xsum,
                                            float &f0, float &f1) {
#pragma unroll 1
        for (uint32_t h = 0; h < halves; h++, xq += 128, xsum += 4) {
            const uint8_t *b0 = r0 + (h >> 1) * 144u, *b1 = r1 + (h >> 1) * 144u;
            const uint32_t hb = h & 1u;
            const uint4 h0 = *reinterpret_cast<const uint4 *>(b0), h1 = *reinterpret_cast<const uint4 *>(b1);
            uint32_t sc0, mn0, sc1, mn1;
            q4k_scales(h0, hb, sc0, mn0);
            q4k_scales(h1, hb, sc1, mn1);
            int qacc[4] = {0, 0, 0, 0}, macc[4] = {0, 0, 0, 0};
#pragma unroll
            for (int cc = 0; cc < 2; cc++) {                             // 64 columns: low and high nibbles of 32 bytes
                const uint2 q0 = *reinterpret_cast<const uint2 *>(b0 + 16 + (hb * 2 + cc) * 32 + 8 * t);
                const uint2 q1 = *reinterpret_cast<const uint2 *>(b1 + 16 + (hb * 2 + cc) * 32 + 8 * t);
#pragma unroll
                for (int nib = 0; nib < 2; nib++) {
                    const int j = cc * 2 + nib;
                    const uint2 bq = *reinterpret_cast<const uint2 *>(xq + j * 32);
                    int c[4];
                    fmma_zero(c, (q0.x >> (4 * nib)) & 0x0f0f0f0fu, (q1.x >> (4 * nib)) & 0x0f0f0f0fu,
                              (q0.y >> (4 * nib)) & 0x0f0f0f0fu, (q1.y >> (4 * nib)) & 0x0f0f0f0fu, bq.x, bq.y);
                    const int s0 = (int)((sc0 >> (8 * j)) & 0xffu), s1 = (int)((sc1 >> (8 * j)) & 0xffu);
                    const int m0 = (int)((mn0 >> (8 * j)) & 0xffu), m1 = (int)((mn1 >> (8 * j)) & 0xffu);
                    const int2 sx = xsum[j];
                    qacc[0] += c[0] * s0; qacc[1] += c[1] * s0; qacc[2] += c[2] * s1; qacc[3] += c[3] * s1;
                    macc[0] += sx.x * m0; macc[1] += sx.y * m0; macc[2] += sx.x * m1; macc[3] += sx.y * m1;
                }
            }
            const float lo = 1.0f / 254.0f;
            const float d0 = __half2float(__ushort_as_half((uint16_t)(h0.x & 0xffffu))), n0 = __half2float(__ushort_as_half((uint16_t)(h0.x >> 16)));
            const float d1 = __half2float(__ushort_as_half((uint16_t)(h1.x & 0xffffu))), n1 = __half2float(__ushort_as_half((uint16_t)(h1.x >> 16)));
            f0 += d0 * fmaf((float)qacc[1], lo, (float)qacc[0]) - n0 * fmaf((float)macc[1], lo, (float)macc[0]);
            f1 += d1 * fmaf((float)qacc[3], lo, (float)qacc[2]) - n1 * fmaf((float)macc[3], lo, (float)macc[2]);
        }
    }
};
template <> struct HalvesS<T_Q4_K> {
    static __device__ __forceinline__ void run(const uint8_t *r0, const uint8_t *r1, uint32_t halves, uint32_t t, const uint8_t *aq, const float2 *asc,
                                            float &f0, float &f1) {
#pragma unroll 1
        for (uint32_t h = 0; h < halves; h++, aq += 128, asc += 4) {
            const uint8_t *b0 = r0 + (h >> 1) * 144u, *b1 = r1 + (h >> 1) * 144u;
            const uint32_t hb = h & 1u;
            const uint4 h0 = *reinterpret_cast<const uint4 *>(b0), h1 = *reinterpret_cast<const uint4 *>(b1);
            uint32_t sc0, mn0, sc1, mn1;
            q4k_scales(h0, hb, sc0, mn0);
            q4k_scales(h1, hb, sc1, mn1);
            float qf0 = 0.0f, qf1 = 0.0f, mf0 = 0.0f, mf1 = 0.0f;
            const float lo = 1.0f / 254.0f;
#pragma unroll
            for (int cc = 0; cc < 2; cc++) {
                const uint2 q0 = *reinterpret_cast<const uint2 *>(b0 + 16 + (hb * 2 + cc) * 32 + 8 * t);
                const uint2 q1 = *reinterpret_cast<const uint2 *>(b1 + 16 + (hb * 2 + cc) * 32 + 8 * t);
#pragma unroll
                for (int nib = 0; nib < 2; nib++) {
                    const int j = cc * 2 + nib;
                    const uint2 bq = *reinterpret_cast<const uint2 *>(aq + j * 32);
                    int c[4];
                    fmma_zero(c, (q0.x >> (4 * nib)) & 0x0f0f0f0fu, (q1.x >> (4 * nib)) & 0x0f0f0f0fu,
                              (q0.y >> (4 * nib)) & 0x0f0f0f0fu, (q1.y >> (4 * nib)) & 0x0f0f0f0fu, bq.x, bq.y);
                    const float2 a = asc[j];
                    const float s0 = (float)((sc0 >> (8 * j)) & 0xffu), s1 = (float)((sc1 >> (8 * j)) & 0xffu);
                    const float m0 = (float)((mn0 >> (8 * j)) & 0xffu), m1 = (float)((mn1 >> (8 * j)) & 0xffu);
                    qf0 = fmaf(s0 * a.x, fmaf((float)c[1], lo, (float)c[0]), qf0);
                    qf1 = fmaf(s1 * a.x, fmaf((float)c[3], lo, (float)c[2]), qf1);
                    mf0 = fmaf(m0, a.y, mf0); mf1 = fmaf(m1, a.y, mf1);
                }
            }
            const float d0 = __half2float(__ushort_as_half((uint16_t)(h0.x & 0xffffu))), n0 = __half2float(__ushort_as_half((uint16_t)(h0.x >> 16)));
            const float d1 = __half2float(__ushort_as_half((uint16_t)(h1.x & 0xffffu))), n1 = __half2float(__ushort_as_half((uint16_t)(h1.x >> 16)));
            f0 += d0 * qf0 - n0 * mf0;
            f1 += d1 * qf1 - n1 * mf1;
        }
    }
};

__device__ __forceinline__ uint32_t lds_ring1(uint32_t a) {
    uint32_t v;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(a));
    return v;
}

template <> struct Halves<T_IQ2N> {
    static __device__ __forceinline__ void run(const uint8_t *block, uint32_t g, uint32_t t, const uint8_t *xq, float &f0, float &f1) {
        const uint32_t base = fs_u32(block), lv = base + 32u * g + 8u * t, sg = base + IQ2N_SIGNS + 16u * g + 4u * t, sc = base + IQ2N_SCALES + 16u * g,
                       dd = base + IQ2N_D + 4u * g;
        uint32_t xs = fs_u32(xq);
#pragma unroll 1
        for (uint32_t h = 0; h < 4; h++, xs += 128) {
            const uint2 l0 = lds_ring2(lv + 512u * h), l1 = lds_ring2(lv + 512u * h + 256u);
            const uint32_t g0 = lds_ring1(sg + 256u * h), g1 = lds_ring1(sg + 256u * h + 128u);
            const uint32_t s0 = lds_ring1(sc + 4u * h), s1 = lds_ring1(sc + 4u * h + 128u);
            const uint32_t dh0 = lds_ring_u16(dd + (h >> 1) * 2u), dh1 = lds_ring_u16(dd + (h >> 1) * 2u + 32u);
            const uint32_t c0[4] = {iq2n_select<0>(l0, g0), iq2n_select<1>(l0, g0), iq2n_select<2>(l0, g0), iq2n_select<3>(l0, g0)};
            const uint32_t c1[4] = {iq2n_select<0>(l1, g1), iq2n_select<1>(l1, g1), iq2n_select<2>(l1, g1), iq2n_select<3>(l1, g1)};
            int iacc[4] = {0, 0, 0, 0};
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const uint2 bq = lds_ring2(xs + j * 32);
                int c[4];
                fmma_zero(c, __byte_perm(IQ2N_LO, IQ2N_HI, c0[j]), __byte_perm(IQ2N_LO, IQ2N_HI, c1[j]),
                          __byte_perm(IQ2N_LO, IQ2N_HI, c0[j] >> 16), __byte_perm(IQ2N_LO, IQ2N_HI, c1[j] >> 16), bq.x, bq.y);
                const int k0 = (int)((s0 >> (8 * j)) & 0xffu), k1 = (int)((s1 >> (8 * j)) & 0xffu);               // 2 * scale + 1
                iacc[0] += c[0] * k0; iacc[1] += c[1] * k0; iacc[2] += c[2] * k1; iacc[3] += c[3] * k1;
            }
            const float lo = 1.0f / 254.0f;
            const float d0 = __half2float(__ushort_as_half((uint16_t)dh0)) * 0.125f, d1 = __half2float(__ushort_as_half((uint16_t)dh1)) * 0.125f;
            f0 += d0 * fmaf((float)iacc[1], lo, (float)iacc[0]);
            f1 += d1 * fmaf((float)iacc[3], lo, (float)iacc[2]);
        }
    }
};
template <> struct HalvesS<T_IQ2N> {
    static __device__ __forceinline__ void run(const uint8_t *block, uint32_t g, uint32_t t, const uint8_t *aq, const float2 *asc, float &f0, float &f1) {
        const uint32_t base = fs_u32(block), lv = base + 32u * g + 8u * t, sg = base + IQ2N_SIGNS + 16u * g + 4u * t, sc = base + IQ2N_SCALES + 16u * g,
                       dd = base + IQ2N_D + 4u * g;
        uint32_t xs = fs_u32(aq), ss = fs_u32(asc);
#pragma unroll 1
        for (uint32_t h = 0; h < 4; h++, xs += 128, ss += 32) {
            const uint2 l0 = lds_ring2(lv + 512u * h), l1 = lds_ring2(lv + 512u * h + 256u);
            const uint32_t g0 = lds_ring1(sg + 256u * h), g1 = lds_ring1(sg + 256u * h + 128u);
            const uint32_t s0 = lds_ring1(sc + 4u * h), s1 = lds_ring1(sc + 4u * h + 128u);
            const uint32_t dh0 = lds_ring_u16(dd + (h >> 1) * 2u), dh1 = lds_ring_u16(dd + (h >> 1) * 2u + 32u);
            const uint32_t c0[4] = {iq2n_select<0>(l0, g0), iq2n_select<1>(l0, g0), iq2n_select<2>(l0, g0), iq2n_select<3>(l0, g0)};
            const uint32_t c1[4] = {iq2n_select<0>(l1, g1), iq2n_select<1>(l1, g1), iq2n_select<2>(l1, g1), iq2n_select<3>(l1, g1)};
            float fa0 = 0.0f, fa1 = 0.0f;
            const float lo = 1.0f / 254.0f;
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const uint2 bq = lds_ring2(xs + j * 32), as = lds_ring2(ss + j * 8);
                int c[4];
                fmma_zero(c, __byte_perm(IQ2N_LO, IQ2N_HI, c0[j]), __byte_perm(IQ2N_LO, IQ2N_HI, c1[j]),
                          __byte_perm(IQ2N_LO, IQ2N_HI, c0[j] >> 16), __byte_perm(IQ2N_LO, IQ2N_HI, c1[j] >> 16), bq.x, bq.y);
                const float k0 = (float)((s0 >> (8 * j)) & 0xffu), k1 = (float)((s1 >> (8 * j)) & 0xffu);       // 2 * scale + 1
                const float a = __uint_as_float(as.x);
                fa0 = fmaf(k0 * a, fmaf((float)c[1], lo, (float)c[0]), fa0);
                fa1 = fmaf(k1 * a, fmaf((float)c[3], lo, (float)c[2]), fa1);
            }
            const float d0 = __half2float(__ushort_as_half((uint16_t)dh0)) * 0.125f, d1 = __half2float(__ushort_as_half((uint16_t)dh1)) * 0.125f;
            f0 = fmaf(d0, fa0, f0);
            f1 = fmaf(d1, fa1, f1);
        }
    }
};

// One thread per 128-column half of a row, from the resident IQ2_XXS image into the expanded one.
// which < 0: [expert][tile of 16 rows][block] (down; one block where a tile is 512 columns deep).  which = 0 / 1 (gate / up):
// unit slices, [expert][unit of 8 rows][block], the gate's rows in block rows 0-7, the up's in 8-15.
__device__ __forceinline__ uint8_t *iq2n_block(uint8_t *image, uint32_t n_out, uint32_t nb5, uint32_t expert, uint32_t row, uint32_t block, int which, uint32_t &r) {
    const uint32_t rows_log = which < 0 ? 4 : 3;
    r = which < 0 ? row & 15u : (row & 7u) + 8u * (uint32_t)which;
    return image + (((uint64_t)expert * (n_out >> rows_log) + (row >> rows_log)) * nb5 + block) * IQ2N_BLOCK;
}
__global__ void __launch_bounds__(256) iq2_expand_kernel(DevTensor t, uint8_t *__restrict__ out, int which) {
    const uint32_t nb = t.k_storage >> 8, halves = t.k_storage >> 7;
    const uint64_t rows = (uint64_t)t.n_out * t.n_experts, total = rows * halves;
    const uint64_t i = (uint64_t)blockIdx.x * 256 + threadIdx.x;
    if (i >= total) return;
    const uint64_t grow = i / halves;                                          // expert * n_out + row
    const uint32_t q = (uint32_t)(i % halves), expert = (uint32_t)(grow / t.n_out), row = (uint32_t)(grow % t.n_out);
    const uint8_t *mat = t.data + (uint64_t)expert * t.expert_bytes;
    uint32_t r;
    uint8_t *block = iq2n_block(out, t.n_out, t.k_storage >> 9, expert, row, q >> 2, which, r);
    const uint32_t h = q & 3u, blk = q >> 1;                                    // half of the 512-column block; 256-column source block
    uint32_t levels[4][2] = {}, signs[4] = {}, scales = 0;                      // by slot = lane t of the consumer: columns 8 t .. 8 t + 7
#pragma unroll
    for (uint32_t j = 0; j < 4; j++) {
        const uint8_t *group = mat + ((uint64_t)row * nb * 8u + ((blk * 8u + (q & 1u) * 4u + j) ^ iq2_swizzle(row, nb))) * 8u;
        const uint32_t bits = load_u32(group + 4), codes = load_u32(group);
#pragma unroll
        for (uint32_t slot = 0; slot < 4; slot++) {
            const uint32_t lv = c_iq2_levels[(codes >> (8 * slot)) & 0xffu], sg = iq2_signs8((bits >> (7 * slot)) & 127u);
#pragma unroll
            for (uint32_t c = 0; c < 8; c++) {
                levels[slot][j >> 1] |= ((lv >> (2 * c)) & 3u) << (4 * c + 2 * (j & 1u));
                signs[slot] |= ((sg >> c) & 1u) << (4 * c + j);
            }
        }
        scales |= (2u * (bits >> 28) + 1u) << (8 * j);
    }
#pragma unroll
    for (uint32_t slot = 0; slot < 4; slot++) {
        *reinterpret_cast<uint2 *>(block + 512u * h + 32u * r + 8u * slot) = make_uint2(levels[slot][0], levels[slot][1]);
        *reinterpret_cast<uint32_t *>(block + IQ2N_SIGNS + 256u * h + 16u * r + 4u * slot) = signs[slot];
    }
    *reinterpret_cast<uint32_t *>(block + IQ2N_SCALES + 16u * r + 4u * h) = scales;
    if (!(q & 1u)) {
        const uint64_t blocks = (uint64_t)t.n_out * nb;
        *reinterpret_cast<uint16_t *>(block + IQ2N_D + 4u * r + h) = (uint16_t)load_u16(mat + blocks * 64u + ((uint64_t)row * nb + blk) * 2u);      // h is 0 or 2
    }
}

// Probe: rows [row0, row0 + rows) of one expert decoded FROM THE EXPANDED IMAGE into floats [rows, k], with the
// arithmetic of the reference's decoder (src/qwen4_packed.c:102-120: d * (2 s + 1) * 0.125 * magnitude, signed), so
// that the image can be compared bit for bit with a CPU decode of the GGUF bytes.  which as above.
__global__ void __launch_bounds__(256) iq2n_decode_rows_kernel(const uint8_t *__restrict__ image, uint32_t k, uint32_t n_out, uint32_t expert,
                                                               uint32_t row0, uint32_t rows, int which, float *__restrict__ out) {
    const uint64_t i = (uint64_t)blockIdx.x * 256 + threadIdx.x;
    if (i >= (uint64_t)rows * k) return;
    const uint32_t row = row0 + (uint32_t)(i / k), col = (uint32_t)(i % k);
    uint32_t r;
    const uint8_t *block = iq2n_block(const_cast<uint8_t *>(image), n_out, k >> 9, expert, row, col >> 9, which, r);
    const uint32_t c = col & 511u, h = c >> 7, j = (c >> 5) & 3u, t = (c >> 3) & 3u, n = c & 7u;
    const uint32_t word = *reinterpret_cast<const uint32_t *>(block + 512u * h + 32u * r + 8u * t + 4u * (j >> 1));
    const uint32_t sign = (*reinterpret_cast<const uint32_t *>(block + IQ2N_SIGNS + 256u * h + 16u * r + 4u * t) >> (4 * n + j)) & 1u;
    const uint32_t code = ((word >> (4 * n + 2 * (j & 1u))) & 3u) | sign << 2;
    const uint32_t twice_plus_one = block[IQ2N_SCALES + 16u * r + 4u * h + j];
    const float d = half_bits_to_float(*reinterpret_cast<const uint16_t *>(block + IQ2N_D + 4u * r + (h >> 1) * 2u));
    const float scale = __fmul_rn(__fmul_rn(d, (float)twice_plus_one), 0.125f);
    const float value = __fmul_rn(scale, (float)iq2_magnitude(code & 3u));
    out[i] = (code & 4u) ? -value : value;
}

// Geometry of one format inside the rings.
template <uint32_t TYPE> struct FGeo;
template <> struct FGeo<T_Q4_K> { static constexpr uint32_t SLICE_BLOCKS = 2, SLICE_BYTES = 16 * 288; };      // sixteen rows x 512 columns
template <> struct FGeo<T_IQ2N> { static constexpr uint32_t SLICE_BLOCKS = 2, SLICE_BYTES = IQ2N_BLOCK; };

// Copies of slice `s` of a gate/up unit (8 gate rows + 8 up rows from row `row0` of expert `expert`) into `stage`:
// row r at r * slice bytes.  The eight row pieces of a
// matrix are ONE tensor-map request (issuing a request costs the warp about a hundred cycles whatever its size).
template <uint32_t TYPE>
__device__ __forceinline__ void issue_unit_slice(const CUtensorMap *gate_map, const CUtensorMap *up_map, const uint8_t *gate_mat,
                                              const uint8_t *up_mat, uint32_t expert, uint32_t n_out, uint32_t nb, uint32_t row0, uint32_t s,
                                              uint8_t *stage, uint64_t *bar, uint32_t lane) {
    constexpr uint32_t bytes = FGeo<TYPE>::SLICE_BYTES;
    if (TYPE == T_IQ2N) {
        // the expanded image keeps a unit slice (gate rows, then up rows) as one span: gate_mat is the image's base
        if (lane == 0) {
            fbar_expect(bar, bytes);
            fbulk(stage, gate_mat + (((uint64_t)expert * (n_out >> 3) + (row0 >> 3)) * (nb >> 1) + s) * bytes, bytes, bar);
        }
        return;
    }
    if (lane == 0) fbar_expect(bar, bytes);
    __syncwarp();
    if (lane < 2) ftma_rows(stage + lane * (bytes / 2), lane ? up_map : gate_map, s * (bytes / 64), row0, expert, bar);
}
template <uint32_t TYPE>
__device__ __forceinline__ void consume_unit_slice(const uint8_t *stage, uint32_t nb, uint32_t s, const uint8_t *xq_lane,
                                                   const int2 *xsum_tok, uint32_t g, uint32_t t, float &f0, float &f1) {
    constexpr uint32_t SB = FGeo<TYPE>::SLICE_BLOCKS;
    if constexpr (TYPE == T_IQ2N) Halves<TYPE>::run(stage, g, t, xq_lane + s * SB * 256u, f0, f1);
    else {
        constexpr uint32_t pitch = FGeo<TYPE>::SLICE_BYTES / 16;
        Halves<TYPE>::run(stage + g * pitch, stage + (8 + g) * pitch, SB * 2, t, xq_lane + s * SB * 256u, xsum_tok + s * SB * 8u, f0, f1);
    }
}

// Down tile: 16 rows x K (K <= 512), fetched whole.
template <uint32_t TYPE>
__device__ __forceinline__ void issue_down_tile(const uint8_t *mat, uint32_t n_out, uint32_t nb, uint32_t row0, uint8_t *stage, uint64_t *bar,
                                             uint32_t lane) {
    const uint32_t bytes = (nb >> 1) * FGeo<TYPE>::SLICE_BYTES;
    if (lane == 0) {
        fbar_expect(bar, bytes);
        fbulk(stage, mat + (row0 >> 4) * bytes, bytes, bar);
    }
}
template <uint32_t TYPE>
__device__ __forceinline__ void consume_down_tile(const uint8_t *stage, uint32_t nb, const uint8_t *aq_lane,
                                                  const float2 *asc_tok, uint32_t g, uint32_t t, float &f0, float &f1) {
    if constexpr (TYPE == T_IQ2N) HalvesS<TYPE>::run(stage, g, t, aq_lane, asc_tok, f0, f1);              // nb = 2
    else {
        const uint32_t row_bytes = nb * 144u;
        HalvesS<TYPE>::run(stage + g * row_bytes, stage + (8 + g) * row_bytes, nb * 2, t, aq_lane, asc_tok, f0, f1);
    }
}

// Two int8 digits per value: v ~ dx * (q1 + q2 / 254), |v| <= 127 dx.  Rounding by the
// 1.5 * 2^23 trick (no conversion instructions): the integer sits in the low mantissa bits, so
// the low byte of the rounded float's bit pattern IS the int8 digit.  c = (dx, 1 / dx, 254 / dx).
__device__ __forceinline__ void digit_pair(float v, const float4 c, uint32_t &ra, uint32_t &rb) {
    const float magic = 12582912.0f;
    const float r1 = fmaf(v, c.y, magic);
    const float q1 = r1 - magic;
    // second digit clamped to [-127, 127] in the float domain, before the rounding add
    const float r2 = fmaxf(-127.0f, fminf(127.0f, fmaf(-q1, c.x, v) * c.z)) + magic;
    ra = __float_as_uint(r1); rb = __float_as_uint(r2);
}
// Four values at once, packed; `s` accumulates both digit sums: the first in its low half, the
// second in its high half (each below 2^15 in magnitude for a 32-column chunk).
__device__ __forceinline__ void digits4(const float4 v, const float4 c, uint32_t &hi, uint32_t &lo, int &s) {
    const float vv[4] = {v.x, v.y, v.z, v.w};
    uint32_t ra[4], rb[4];
#pragma unroll
    for (int j = 0; j < 4; j++) digit_pair(vv[j], c, ra[j], rb[j]);
    hi = __byte_perm(__byte_perm(ra[0], ra[1], 0x0040), __byte_perm(ra[2], ra[3], 0x0040), 0x5410);
    lo = __byte_perm(__byte_perm(rb[0], rb[1], 0x0040), __byte_perm(rb[2], rb[3], 0x0040), 0x5410);
    s += __dp4a((int)hi, 0x01010101, 0) + (__dp4a((int)lo, 0x01010101, 0) << 16);
}

// Rows of `k` floats (k % 256 == 0) in shared memory with known maxima -> digit images, digit
// sums per 32-column chunk and scales.  A warp takes one 256-column segment of one row at a time:
// two float4 per lane, eight consecutive lanes cover one chunk.  `amax` holds the maxima on entry
// and the scales (max / 127, or 0 for an unusable row) on return; `consts` is scratch, one float4
// per row.  CTA-wide.
__device__ __forceinline__ void digitise_rows(const float *src, uint32_t src_pitch, uint32_t rows, uint32_t k, float *amax, uint8_t *dq,
                                           uint32_t dq_pitch, int2 *sums, uint32_t sums_pitch, float4 *consts) {
#pragma unroll 1
    for (uint32_t r = threadIdx.x; r < rows; r += FT) {
        const float m = amax[r];
        const bool usable = finite_f32(m) && m > 0.0f;
        const float inv = usable ? __fdividef(127.0f, m) : 0.0f;
        consts[r] = make_float4(usable ? m * (1.0f / 127.0f) : 0.0f, inv, 2.0f * inv * 127.0f, 0.0f);
    }
    __syncthreads();
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u, segs = k >> 8, units = rows * segs;
#pragma unroll 1
    for (uint32_t u = warp; u < units; u += FW) {
        const uint32_t r = u / segs, seg = u - r * segs;
        const float4 *from = reinterpret_cast<const float4 *>(src + (uint64_t)r * src_pitch) + seg * 64u + lane;
        const float4 v0 = *from, v1 = *(from + 32);
        const float4 c = consts[r];
        uint32_t hi0, lo0, hi1, lo1;
        int s0 = 0, s1 = 0;
        digits4(v0, c, hi0, lo0, s0);
        digits4(v1, c, hi1, lo1, s1);
        uint8_t *out = dq + (2 * r) * dq_pitch + seg * 256u + lane * 4u;
        *reinterpret_cast<uint32_t *>(out) = hi0; *reinterpret_cast<uint32_t *>(out + 128) = hi1;
        *reinterpret_cast<uint32_t *>(out + dq_pitch) = lo0; *reinterpret_cast<uint32_t *>(out + dq_pitch + 128) = lo1;
        for (int o = 1; o < 8; o <<= 1) { s0 += __shfl_xor_sync(0xffffffffu, s0, o); s1 += __shfl_xor_sync(0xffffffffu, s1, o); }
        if ((lane & 7u) == 0) {
            const int a0 = (int)(short)(s0 & 0xffff), a1 = (int)(short)(s1 & 0xffff);
            int2 *to = sums + r * sums_pitch + seg * 8u + (lane >> 3);
            to[0] = make_int2(a0, (s0 - a0) >> 16);
            to[4] = make_int2(a1, (s1 - a1) >> 16);
        }
    }
    __syncthreads();
#pragma unroll 1
    for (uint32_t r = threadIdx.x; r < rows; r += FT) amax[r] = consts[r].x;
    __syncthreads();
}

__device__ __forceinline__ float fast_sigmoid(float v) {
    const float e = __expf(-fabsf(v));
    return v >= 0.0f ? __fdividef(1.0f, 1.0f + e) : __fdividef(e, 1.0f + e);
}

// The k largest of one row of logits by VALUE (ties to the lower id), one warp.  The row is read straight from global memory into ordered integer
// keys: through a bulk copy into shared memory the same round trip took 1.8 k cycles instead of 0.7 (90.4 against 93.4 us for four Q4_K layers of one
// token).  cand: 256 words of scratch.  `extra`: choose k + 1 and put the last one in slot k - 1 (a
// deliberately wrong set, for the test of the repair path).  Returns false on a nonfinite logit.
__device__ __forceinline__ bool speculate_row(const float *logits, uint32_t *cand, uint32_t E, uint32_t k, bool extra, uint32_t *ids_s, uint32_t lane) {
    constexpr int PL = FMAXE / 32;
    uint32_t key[PL];
    bool bad = false;
#pragma unroll
    for (int i = 0; i < PL; i++) {
        const uint32_t e = lane + 32u * i;
        const uint32_t u = e < E ? __float_as_uint(__ldcg(logits + e)) : 0u;
        bad |= e < E && (u & 0x7f800000u) == 0x7f800000u;
        key[i] = e < E ? ((u & 0x80000000u) ? ~u : (u | 0x80000000u)) : 0u;      // monotone in the value, never 0
    }
    if (__any_sync(0xffffffffu, bad)) return false;
    const uint32_t want = extra && k < E ? k + 1 : k;
    uint32_t *out = extra ? cand + 128 : ids_s;
    if (!warp_topk<PL>(key, lane, want, cand, out, nullptr)) warp_topk_sequential<PL>(key, lane, want, out, nullptr);
    if (extra) {                                                                // the wrong set: the (k + 1)-th takes the k-th's place
        if (lane < k) ids_s[lane] = out[lane == k - 1 && want > k ? k : lane];
        __syncwarp();
    }
    return true;
}

// CLOCK: SM clock of the first streaming CTA at a phase boundary.  MARK: cycles since its own start, for every CTA
// (words S_MARKS + 4 * cta + i of the sync array), by kernels of their own (MARKS) that are launched on request: stored at every launch the
// marks cost 0.7 us in four Q4_K layers of one token (83.8 against 83.1) and 1.9 in four IQ2_XXS layers of four (140.9 against 139.0), and a
// switch among the arguments costs as much without storing any (88.0 against 87.4, 143.1 against 142.2).
#define CLOCK(i) do { if (clocked) clocks[i] = clock64(); } while (0)
#define MARK_CYCLES(i, cycles) do { if (MARKS && threadIdx.x == 0) a.sync[S_MARKS + 4 * blockIdx.x + (i)] = (uint32_t)(cycles); } while (0)
#define MARK(i) MARK_CYCLES(i, clock64() - a.t0)

// ---- chain CTA -----------------------------------------------------------------------------------
// Exact logits of router rows [32 c, 32 c + 32) (row E is the shared expert's router) for every
// token, then, in CTA t < T, the routing of token t.
//
// A chain is H dependent additions of four cycles (8.2 k cycles at H = 2048), and everything else of it is kept under them: the
// rows come by bulk copies of 512 columns, two chunks at once, and a lane reads the operands of
// the next sixteen columns while the products of the current ones are added.  (Before: 64-column chunks through a
// 16-stage cp.async ring, with a barrier wait and exposed read latency per chunk: 20 k cycles with resident
// rows, 35 k when the rows came from HBM.)
template <bool MARKS>
__device__ __forceinline__ void chain_cta(FusedArgs &a, uint8_t *smem) {
    const uint32_t T = a.tokens, H = a.hidden, E = a.experts, k = a.top_k;
    const CPlan p = make_cplan(H);
    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31u, cta = blockIdx.x;
    uint64_t *full = reinterpret_cast<uint64_t *>(smem + p.bars);              // [CSTG]
    uint64_t *empty = full + CSTG;                                             // [CSTG]
    uint64_t *xbar = empty + CSTG;
    const bool exact = a.router_mode != 1;
    if (tid < CSTG) { fbar_init(&full[tid], 1); fbar_init(&empty[tid], T); }
    if (tid == CSTG) fbar_init(xbar, 1);
    if (tid <= CSTG) asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    __syncthreads();
    const uint32_t r0 = cta * CROWS;
    const uint32_t nr = exact && r0 <= E ? min((uint32_t)CROWS, E + 1 - r0) : 0;
    const uint32_t chunks = (H + CCH - 1) / CCH;
    uint8_t *ring = smem + p.ring;
    bool alive = true;
    auto issue = [&](uint32_t c) {                                             // by warp T: lane = row
        const uint32_t st = c % CSTG, bytes = min((uint32_t)CCH, H - c * CCH) * 4u, gr = r0 + lane;
        if (lane == 0) fbar_expect(&full[st], bytes * nr);
        __syncwarp();
        if (lane < nr)
            fbulk(ring + (st * CROWS + lane) * CPITCH, (gr < E ? a.w[0].data + (uint64_t)gr * a.w[0].row_bytes : a.w[7].data) + (uint64_t)c * CCH * 4, bytes, &full[st]);
    };
    asm volatile("griddepcontrol.wait;" ::: "memory");
    if (tid == 0) a.t0 = clock64();                                            // read back by thread 0 only
    if (nr && warp == T) {
        // not before the previous launch has drained: its last phase is bound by memory, and the chains have slack (ahead of the
        // wait, four tokens took 40.9 us a layer instead of 40.0)
        for (uint32_t c = 0; c < CSTG && c < chunks; c++) issue(c);
        for (uint32_t c = CSTG; c < chunks && alive; c++) {
            const long long start = clock64();
            while (alive && !fbar_try(&empty[c % CSTG], (c / CSTG - 1u) & 1u)) {
                __nanosleep(100);                                              // the chain warps share the schedulers: poll gently
                if (clock64() - start > (1ll << 31)) { atomicOr(a.status, QW4SH_ERR_STATE); alive = false; }
            }
            alive = __all_sync(0xffffffffu, alive);
            if (!alive) break;
            fproxy_fence();
            issue(c);
        }
    }
    if (nr && warp < T) {
        // chain warp: token = warp, lane = row.  Multiplies and adds are separately rounded.
        uint8_t *xf = smem + p.xf;
        if (tid == 0) {
            fbar_expect(xbar, T * H * 4u);
            for (uint32_t q = 0; q < T; q++) fbulk(xf + q * p.xf_pitch, a.x + (uint64_t)q * H, H * 4u, xbar);
        }
        alive = fbar_wait(xbar, 0, a.status);
        MARK(2);
        long long waited = 0;
        float sum = 0.0f;
#pragma unroll 1
        for (uint32_t c = 0; c < chunks; c++) {
            const uint32_t st = c % CSTG;
            const long long w0 = clock64();
            if (alive) alive = fbar_wait(&full[st], (c / CSTG) & 1u, a.status);
            alive = __all_sync(0xffffffffu, alive);
            waited += clock64() - w0;
            if (!alive) break;
            const ulonglong2 *w = reinterpret_cast<const ulonglong2 *>(ring + (st * CROWS + lane) * CPITCH);
            const ulonglong2 *v = reinterpret_cast<const ulonglong2 *>(xf + warp * p.xf_pitch) + c * (CCH / 4);
            const uint32_t quads = min((uint32_t)CCH, H - c * CCH) / 4;       // a multiple of four
            ulonglong2 wa[4], va[4];
#pragma unroll
            for (int j = 0; j < 4; j++) { wa[j] = w[j]; va[j] = v[j]; }
            // a lone warp issues every other cycle: the products go two at a time (mul.rn.f32x2 rounds each half
            // like a scalar multiply), which leaves two loads + 2 packed multiplies + 4 adds per four columns, just
            // under the adds' own latency
#pragma unroll 2
            for (uint32_t q = 0; q < quads; q += 4) {
                ulonglong2 wb[4], vb[4];
                const uint32_t next = q + 4 < quads ? q + 4 : q;
#pragma unroll
                for (int j = 0; j < 4; j++) { wb[j] = w[next + j]; vb[j] = v[next + j]; }
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    unsigned long long p01, p23;
                    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(p01) : "l"(wa[j].x), "l"(va[j].x));
                    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(p23) : "l"(wa[j].y), "l"(va[j].y));
                    sum = __fadd_rn(sum, __uint_as_float((uint32_t)p01)); sum = __fadd_rn(sum, __uint_as_float((uint32_t)(p01 >> 32)));
                    sum = __fadd_rn(sum, __uint_as_float((uint32_t)p23)); sum = __fadd_rn(sum, __uint_as_float((uint32_t)(p23 >> 32)));
                }
#pragma unroll
                for (int j = 0; j < 4; j++) { wa[j] = wb[j]; va[j] = vb[j]; }
            }
            __syncwarp();
            if (lane == 0) fbar_arrive(&empty[st]);
        }
        if (alive && lane < nr) {
            const uint32_t r = r0 + lane;
            if (!finite_f32(sum)) { atomicOr(a.status, QW4SH_ERR_NONFINITE); atomicMin(a.status + 1, warp); }
            if (r < E) a.logits[(uint64_t)warp * E + r] = sum; else a.shared_logit[warp] = sum;
        }
        MARK_CYCLES(3, waited);
    }
    MARK(0);
    if (exact) arrive_counter(a.sync + S_CHAIN);          // also for a CTA without rows: the count is NC
    if (cta >= T) return;
    // ---- routing of token `cta` ----
    const uint32_t waited = exact ? S_CHAIN : S_FAST;
    const uint32_t expected = exact ? a.chain_ctas : gridDim.x - a.chain_ctas;
    bool ok = wait_counter(a.sync + waited, expected, a.status);
    if (ok) {
        const float *from = exact ? a.logits + (uint64_t)cta * E : a.logits_fast + (uint64_t)cta * a.fast_pitch;
        if (!exact) {
            for (uint32_t e = tid; e < E; e += FT) a.logits[(uint64_t)cta * E + e] = __ldcg(from + e);
            if (tid == 0) a.shared_logit[cta] = __ldcg(from + E);
        }
        RouteShared &rs = *reinterpret_cast<RouteShared *>(smem + p.route);
        ok = route_rows<FW>(cta, 1, E, k, a.norm, exact, reinterpret_cast<float *>(smem + p.route + sizeof(RouteShared)), rs, a.status, nullptr,
                            [&](uint32_t, uint32_t e) { return __ldcg(from + e); },
                            [&](uint32_t t, uint32_t slot, uint32_t id, float w) {
                                a.ids[t * k + slot] = id; a.weights[t * k + slot] = w;
                                if (a.ids_out) a.ids_out[t * k + slot] = id;
                                if (a.weights_out) a.weights_out[t * k + slot] = w;
                            }) == 0;
    }
    if (!ok && tid == 0) atomicOr(a.sync + S_ROUTE_FAIL, 1u);
    arrive_counter(a.sync + S_ROUTED);
    MARK(1);
}

// ---- the kernel ---------------------------------------------------------------------------------
template <uint32_t RT, uint32_t ST, bool MARKS>
__global__ void __launch_bounds__(FT, 1) fused_decode_kernel(const __grid_constant__ FusedArgs args, const __grid_constant__ CUtensorMap map_g,
                                                             const __grid_constant__ CUtensorMap map_u, const __grid_constant__ CUtensorMap map_sg,
                                                             const __grid_constant__ CUtensorMap map_su) {
    extern __shared__ __align__(128) uint8_t smem[];
    // The arguments span several cache lines of the constant bank, and a first touch of each line
    // costs a miss that every SM takes at the same moment.  All lines are fetched at once here,
    // into shared memory, and read from there afterwards.
    __shared__ FusedArgs a;
    for (uint32_t i = threadIdx.x; i < sizeof(FusedArgs) / 4; i += FT)
        reinterpret_cast<uint32_t *>(&a)[i] = reinterpret_cast<const uint32_t *>(&args)[i];
    __syncthreads();
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const uint32_t NC = a.chain_ctas;
    const uint32_t tid = threadIdx.x;
    __shared__ uint32_t leaving_last;
    auto leave = [&]() {
        // the CTA that leaves last clears the counters for the next launch
        __syncthreads();
        if (tid == 0) {
            if (a.status_mirror) __threadfence_system(); else __threadfence();      // results in host memory are out before the exit count
            leaving_last = atomicAdd(a.sync + S_EXITS, 1u) == gridDim.x - 1 ? 1u : 0u;
        }
        __syncthreads();
        if (leaving_last && tid < 8) { a.sync[tid] = 0; __threadfence(); }
        // every CTA's error bits and results are in before its exit count: the last one hands the words to the host, which polls the first
        if (leaving_last && tid == 0 && a.status_mirror) {
            const volatile uint32_t *from = a.status;
            volatile uint32_t *to = a.status_mirror;
            const uint32_t bits = from[0];
            to[1] = from[1]; to[2] = from[2]; to[3] = from[3];
            __threadfence_system();
            to[0] = bits;
        }
    };
    if (blockIdx.x < NC) { chain_cta<MARKS>(a, smem); leave(); return; }

    const uint32_t T = a.tokens, H = a.hidden, E = a.experts, k = a.top_k, I = a.inter, IS = a.shared_inter;
    const uint32_t pairs = T * k, rows_c = pairs + T, imax = I > IS ? I : IS;
    const FPlan p = make_fplan(H, imax, rows_c, a.partial_slices, a.clear != 0);
    const uint32_t warp = tid >> 5, lane = tid & 31u, g = lane >> 2, t = lane & 3u;
    const uint32_t sc = blockIdx.x - NC, NS = gridDim.x - NC;
    uint64_t *ringbar = reinterpret_cast<uint64_t *>(smem + p.bars);           // [FW][FNS], four single ones, then [FW][FNC]
    uint64_t *rowbar = ringbar + FW * FNS;
    uint64_t *tilebar = ringbar + FW * FNS + 4 + (threadIdx.x >> 5) * FNC;     // this warp's barriers of the down phase
    static_assert((FW * FNS + 4 + FW * FNC) * 8 <= 512, "the barrier block is 512 bytes");
    uint64_t *lutbar = rowbar + 1;
    uint64_t *xbar = lutbar + 1;                                               // x rows (phase A)
    uint64_t *abar = xbar + 1;                                                 // activation digits (phase C)
    uint32_t *ids_s = reinterpret_cast<uint32_t *>(smem + p.ids);              // the ids phase B works with
    float *wts_s = reinterpret_cast<float *>(smem + p.wts);                    // exact weights in the order of ids_s
    uint32_t *ids_x = reinterpret_cast<uint32_t *>(smem + p.idx);              // the exact routes as published
    float *wts_x = reinterpret_cast<float *>(smem + p.wtx);
    float *misc_f = reinterpret_cast<float *>(smem + p.misc);                  // [0..3] x maxima then scales, [4..7] shared logits
    uint32_t *misc_u = reinterpret_cast<uint32_t *>(smem + p.misc) + 16;       // [1] the guess is usable, [2] sources
    uint8_t *tokmask = smem + p.tokmask, *slotmap = smem + p.slotmap;
    Src *srcs = reinterpret_cast<Src *>(smem + p.src);
    uint8_t *region = smem + p.region;
    uint8_t *xq = region + p.xq;
    int2 *xsum = reinterpret_cast<int2 *>(region + p.xsum);
    unsigned long long *clocks = reinterpret_cast<unsigned long long *>(a.sync + S_CLOCKS);
    const bool clocked = sc == 0 && tid == 0;

    if (tid < FW * FNS + 4 + FW * FNC) {                                       // the barriers lie one after the other: one thread each
        fbar_init(&ringbar[tid], 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (tid < 8) misc_f[tid] = 0.0f;
    float4 *xconsts = reinterpret_cast<float4 *>(smem + p.misc + 512);
    __syncthreads();

    // ================================ phase A ================================
    const uint32_t n_rows = sc <= E ? (E - sc) / NS + 1 : 0;                  // router rows sc, sc + NS, ... <= E
    uint8_t *xf = region + p.xf;
    uint8_t *rows = region + p.rows;
    // weights first: nothing another launch writes
    if (warp == 0) {
        if (lane == 0) fbar_expect(rowbar, n_rows * H * 4u);
        __syncwarp();
        if (lane < n_rows) {
            const uint32_t r = sc + lane * NS;
            const uint8_t *src = r < E ? a.w[0].data + (uint64_t)r * a.w[0].row_bytes : a.w[7].data;
            fbulk(rows + lane * p.row_pitch, src, H * 4u, rowbar);
        }
    } else if (warp == 1 && lane < 3) {                                        // the shared expert's tensors -> L2: one request per tensor
        const uint32_t m = 4 + lane;
        const uint32_t bytes = (uint32_t)a.w[m].expert_bytes & ~15u;            // shared tensors are far below 4 GB
        const uint32_t sub = ((bytes / NS) + 16u) & ~15u;
        const uint32_t from = sc * sub;
        if (from < bytes) fprefetch_l2(a.w[m].data + from, from + sub <= bytes ? sub : bytes - from);
    }
    asm volatile("griddepcontrol.wait;" ::: "memory");
    if (tid == 0) a.t0 = clock64();
    CLOCK(0);
    if (warp == 0) {
        if (lane == 0) fbar_expect(xbar, T * H * 4u);
        __syncwarp();
        if (lane < T) fbulk(xf + lane * p.xf_pitch, a.x + (uint64_t)lane * H, H * 4u, xbar);
    }
    // x -> shared memory (float, one bulk copy per row) with the row maxima, then digits; token rows beyond T stay zero
    bool alive = fbar_wait(xbar, 0, a.status);
    CLOCK(1);
    {
        float m[FTOK] = {0.f, 0.f, 0.f, 0.f};
        if (alive) {
#pragma unroll 1
            for (uint32_t c4 = tid; c4 < (H >> 2); c4 += FT) {                  // the rows' loads of one column are in flight together
#pragma unroll
                for (int q = 0; q < FTOK; q++) {
                    if ((uint32_t)q < T) {
                        const float4 v = *reinterpret_cast<const float4 *>(xf + q * p.xf_pitch + c4 * 16);
                        m[q] = fmaxf(m[q], fmaxf(fmaxf(fabsf(v.x), fabsf(v.y)), fmaxf(fabsf(v.z), fabsf(v.w))));
                    }
                }
            }
        }
#pragma unroll
        for (int q = 0; q < FTOK; q++) {
            if ((uint32_t)q >= T) break;
            const uint32_t v = __reduce_max_sync(0xffffffffu, __float_as_uint(m[q]));        // no sign, no NaN: ordered as integers
            if (lane == 0 && v) atomicMax(reinterpret_cast<uint32_t *>(misc_f) + q, v);
        }
#pragma unroll 1
        for (uint32_t i = tid; i < (FTOK - T) * 2 * (p.kp >> 4); i += FT)       // digit rows of absent tokens
            reinterpret_cast<uint4 *>(xq + 2 * T * p.kp)[i] = make_uint4(0, 0, 0, 0);
#pragma unroll 1
        for (uint32_t i = tid; i < (FTOK - T) * (H >> 5); i += FT) xsum[T * (H >> 5) + i] = make_int2(0, 0);
    }
    __syncthreads();
    // tree-summed logits of this CTA's rows: eight warps split K, each holds its columns of x in registers
    // and reads every router row once; sixteen (row, token) sums per warp, then eight partial sums each
    if (alive) alive = fbar_wait(rowbar, 0, a.status);
    float *lpart = reinterpret_cast<float *>(region + p.rows + FRMAX * p.row_pitch);    // [8 warps][16]
    if (warp < 8 && alive) {
        float acc[FRMAX][FTOK];
#pragma unroll
        for (int j = 0; j < FRMAX; j++)
#pragma unroll
            for (int q = 0; q < FTOK; q++) acc[j][q] = 0.0f;
        const uint32_t per_warp = H >> 3;                                      // columns of this warp
#pragma unroll 1
        for (uint32_t c0 = 0; c0 < per_warp; c0 += 128) {
            const uint32_t col = warp * per_warp + c0 + lane * 4;
            float4 xv[FTOK];
#pragma unroll
            for (int q = 0; q < FTOK; q++)
                xv[q] = (uint32_t)q < T ? *reinterpret_cast<const float4 *>(xf + q * p.xf_pitch + col * 4) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int j = 0; j < FRMAX; j++) {
                if ((uint32_t)j < n_rows) {
                    const float4 w4 = *reinterpret_cast<const float4 *>(rows + j * p.row_pitch + col * 4);
#pragma unroll
                    for (int q = 0; q < FTOK; q++)
                        acc[j][q] = fmaf(w4.x, xv[q].x, fmaf(w4.y, xv[q].y, fmaf(w4.z, xv[q].z, fmaf(w4.w, xv[q].w, acc[j][q]))));
                }
            }
        }
        // sixteen sums over the lanes in sixteen shuffles: at each step a lane keeps half of its sums and hands the other half to its partner,
        // so that lanes 2i and 2i + 1 end with sum i.  The same pairs are added as by a butterfly per sum, whose eighty shuffles took a one-token
        // step 1.1 k cycles longer (with the maxima above by one instruction each: 86.4 -> 84.1 us for four Q4_K layers)
        static_assert(FRMAX * FTOK == 16, "one sum for every two lanes");
        float *v = &acc[0][0];
#pragma unroll
        for (int o = 16; o > 1; o >>= 1)
#pragma unroll
            for (int i = 0; i < o / 2; i++) {
                const bool up = lane & o;
                const float keep = up ? v[i + o / 2] : v[i], send = up ? v[i] : v[i + o / 2];
                v[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
            }
        v[0] += __shfl_xor_sync(0xffffffffu, v[0], 1);
        if (!(lane & 1u)) lpart[warp * 16 + (lane >> 1)] = v[0];
    }
    __syncthreads();
    if (tid < n_rows * FTOK && (tid % FTOK) < T && alive) {
        float v = 0.0f;
#pragma unroll
        for (int w = 0; w < 8; w++) v += lpart[w * 16 + tid];
        a.logits_fast[(uint64_t)(tid % FTOK) * a.fast_pitch + sc + (tid / FTOK) * NS] = v;
    }
    CLOCK(2);
    if (tid < FMAXE / 4) reinterpret_cast<uint32_t *>(tokmask)[tid] = 0;      // for the lists
    static_assert(FMAXE / 4 <= FT, "one word a thread");
    if (tid == 0) misc_u[1] = 1;                                               // the guess is usable
    arrive_counter(a.sync + S_FAST);                                          // (its CTA barrier also orders the reads of xf before the digits' consts)
    digitise_rows(reinterpret_cast<const float *>(xf), p.xf_pitch >> 2, T, H, misc_f, xq, p.kp, xsum, H >> 5, xconsts);
    CLOCK(3);
    if (!wait_counter(a.sync + S_FAST, NS, a.status)) return;
    CLOCK(4);
    MARK(0);

    // ================================ phase B ================================
    float *zs = reinterpret_cast<float *>(region + p.zs);
    if (warp < T) {
        const float *logits = a.logits_fast + (uint64_t)warp * a.fast_pitch;
        if (a.router_mode == 1 && lane == 0) misc_f[4 + warp] = __ldcg(logits + E);     // the shared router's tree sum
        const bool fine = speculate_row(logits, reinterpret_cast<uint32_t *>(zs + warp * FZP), E, k, a.router_mode == 2 && warp == 0, ids_s + warp * k, lane);
        if (!fine && lane == 0) misc_u[1] = 0;
        CLOCK(15);
    }
    const bool all_alive = __syncthreads_and(alive);
    bool lists_ok = misc_u[1] != 0 && all_alive;
    CLOCK(5);

    uint32_t ring_count = 0;                                                   // slices this warp has pushed through its ring
    // phase C: this warp's sources and (tile, source) steps, the next one to issue, steps and digit images read before (a repaired step comes here
    // twice), and whether its first copies are on their way
    uint8_t *aq = region + p.aq, *tiles = region + p.tiles + warp * FNC * FSTAGE;
    float2 *asc = reinterpret_cast<float2 *>(region + p.asc);
    uint32_t n_src = 0, my_src = 0, steps = 0, next_tile = 0, next_src = 0, tiles_read = 0, digits_read = 0;
    bool begun = false;
    auto issue_down = [&](uint32_t n) {                                        // in step order; the phase has ring barriers of its own
        const uint32_t tile = next_tile, j = next_src, at = tiles_read + n;
        next_src += FW;
        if (next_src >= n_src) { next_src = warp; next_tile += NS; }
        const Src s = srcs[j];
        uint8_t *stage = tiles + (at % FNC) * FSTAGE;
        if (s.shared) issue_down_tile<ST>(a.w[6].data, H, IS >> 8, tile * 16, stage, &tilebar[at % FNC], lane);
        else issue_down_tile<RT>(a.w[3].data + (uint64_t)s.expert * a.w[3].expert_bytes, H, I >> 8, tile * 16, stage, &tilebar[at % FNC], lane);
    };
    const bool down_here = sc < (H >> 4);
    auto begin_down = [&]() {                                                  // behind a CTA barrier: phase B's use of the region is over
        if (!down_here || !lists_ok) return;
        asm volatile("fence.proxy.async;" ::: "memory");                          // the digits were written through the generic proxy, by other CTAs
        fproxy_fence();
        const uint32_t aq_bytes = rows_c * 2u * p.ap, asc_bytes = rows_c * (imax >> 5) * 8u;
        if (tid == 0) {
            fbar_expect(abar, aq_bytes + asc_bytes);
            fbulk(aq, a.aq, aq_bytes, abar);
            fbulk(asc, a.asc, asc_bytes, abar);
        }
        alive = __all_sync(0xffffffffu, alive);
        if (alive) for (uint32_t n = 0; n < FNC && n < steps; n++) issue_down(n);
    };
    auto drain_down = [&]() {                                                  // what begin_down sent for has landed, and is not wanted
        if (!down_here || !lists_ok) return;
        bool landed = fbar_wait(abar, digits_read & 1u, a.status);
        const uint32_t sent = alive ? min(steps, (uint32_t)FNC) : 0;
        for (uint32_t n = 0; n < sent; n++) landed &= fbar_wait(&tilebar[(tiles_read + n) % FNC], ((tiles_read + n) / FNC) & 1u, a.status);
        digits_read++; tiles_read += sent;
        alive = __all_sync(0xffffffffu, alive && landed);
    };
    uint64_t *bar = ringbar + warp * FNS;
    const uint32_t gs = IS >> 5, gr = I >> 5;                                  // granules (32 activation columns) per expert
    const uint32_t nbh = H >> 8;
    const uint32_t spu_s = nbh / FGeo<ST>::SLICE_BLOCKS, spu_r = nbh / FGeo<RT>::SLICE_BLOCKS;
#pragma unroll 1
    for (uint32_t attempt = 0; attempt < 2; attempt++) {
        // ---- lists from ids_s: token masks and slots per expert, distinct experts in ascending order behind the shared expert ----
        if (lists_ok) {
            if (warp == 0) {                                                   // one warp, warp-level synchronisation only
#pragma unroll 1
                for (uint32_t pr = lane; pr < pairs; pr += 32) {
                    const uint32_t e = ids_s[pr], tok = pr / k;
                    atomicOr(reinterpret_cast<uint32_t *>(tokmask) + (e >> 2), (1u << tok) << (8 * (e & 3u)));
                    slotmap[e * 4 + tok] = (uint8_t)(pr % k);
                }
                __syncwarp();
                if (lane == 0) { Src s0; s0.expert = 0xffffu; s0.mask = (uint8_t)((1u << T) - 1u); s0.shared = 1; s0.slots = 0; srcs[0] = s0; }
                // lane = sixteen experts in turn: which of them have tokens, the experts before them, then their entries one by one (one or two a lane;
                // a ballot for every 32 experts took 3.2 k cycles, this 1.1 k with one token and 1.4 k with four)
                uint32_t mine = 0;
                const uint4 marks = reinterpret_cast<const uint4 *>(tokmask)[lane];
                const uint32_t word[4] = {marks.x, marks.y, marks.z, marks.w};
#pragma unroll
                for (uint32_t i = 0; i < 16; i++) mine |= ((word[i >> 2] >> (8 * (i & 3u))) & 0xffu ? 1u : 0u) << i;
                uint32_t running = __popc(mine);
                for (int o = 1; o < 32; o <<= 1) { const uint32_t v = __shfl_up_sync(0xffffffffu, running, o); if (lane >= (uint32_t)o) running += v; }
                uint32_t at = 1 + running - __popc(mine);
                for (uint32_t left = mine; left; left &= left - 1, at++) {
                    const uint32_t e = lane * 16 + __ffs(left) - 1;
                    Src sn; sn.expert = (uint16_t)e; sn.mask = tokmask[e]; sn.shared = 0;
                    sn.slots = *reinterpret_cast<const uint32_t *>(slotmap + e * 4);
                    srcs[at] = sn;
                }
                running = 1 + __shfl_sync(0xffffffffu, running, 31);
                if (lane == 0) misc_u[2] = running;
            }
            __syncthreads();
            n_src = misc_u[2];
        }
        CLOCK(6);
        if (lists_ok) {
            // ---- gate/up: whole granules per CTA, the shared expert's first ----
            const uint32_t total = gs + (n_src - 1) * gr;
            const uint32_t g0 = total * sc / NS, g1 = total * (sc + 1) / NS;               // total <= 65 * 32: no overflow
            const uint32_t n_shg = g0 < gs ? min(gs, g1) - g0 : 0;               // shared granules of this CTA come first
            const uint32_t n_shu = n_shg * 4;
            const uint32_t slices = min(n_shu * spu_s + ((g1 - g0) * 4 - n_shu) * spu_r, a.partial_slices);
            const uint32_t mine = slices > warp ? (slices - 1 - warp) / FW + 1 : 0;
            uint8_t *ring = region + p.ring + warp * FNS * FSTAGE;
            float2 *partial = reinterpret_cast<float2 *>(region + p.partial);
            alive = __all_sync(0xffffffffu, alive);
            // CTA slice n -> local unit, slice, kind.  Both formats cut a unit into the same number of slices; the
            // divisors are powers of two for every shape met so far, and a runtime division costs a lone lane as
            // much as a quarter of a slice's arithmetic.
            const uint32_t spu = spu_r, spu_sh = (spu & (spu - 1u)) ? 32u : 31u - (uint32_t)__clz(spu);
            const uint32_t ur = gr * 4, ur_sh = (ur & (ur - 1u)) ? 32u : 31u - (uint32_t)__clz(ur);
            auto locate = [&](uint32_t n, uint32_t &ul, uint32_t &s, bool &sh) {
                if (spu_sh < 32u) { ul = n >> spu_sh; s = n & (spu - 1u); } else { ul = n / spu; s = n - ul * spu; }
                sh = ul < n_shu;
            };
            auto issue = [&](uint32_t i) {
                uint32_t ul, s; bool sh;
                locate(warp + i * FW, ul, s, sh);
                const uint32_t u = g0 * 4 + ul;                                    // unit index over all sources
                const uint32_t at = ring_count + i;
                uint8_t *stage = ring + (at % FNS) * FSTAGE;
                if (sh) issue_unit_slice<ST>(&map_sg, &map_su, a.w[4].data, a.w[5].data, 0, IS, nbh, u * 8, s, stage, &bar[at % FNS], lane);
                else {
                    const uint32_t v = u - gs * 4, vq = ur_sh < 32u ? v >> ur_sh : v / ur, e = srcs[1 + vq].expert;
                    issue_unit_slice<RT>(&map_g, &map_u, a.w[1].data, a.w[2].data, e, I, nbh, (v - vq * ur) * 8, s, stage, &bar[at % FNS], lane);
                }
            };
            __syncthreads();                                                       // the keys in zs are dead: the ring may be written
            fproxy_fence();
            if (alive) for (uint32_t i = 0; i < FNS && i < mine; i++) issue(i);
            // down tiles of this CTA's columns -> L2, ahead of phase C
#pragma unroll 1
            for (uint32_t tile = sc; tile < (H >> 4); tile += NS)
                for (uint32_t j = warp * 4 + lane; lane < 4 && j < n_src; j += FW * 4) {      // a few requests per warp: none of them falls behind
                    const Src s = srcs[j];
                    const uint32_t bytes = s.shared ? (IS >> 9) * FGeo<ST>::SLICE_BYTES : (I >> 9) * FGeo<RT>::SLICE_BYTES;
                    const uint8_t *mat = s.shared ? a.w[6].data : a.w[3].data + (uint64_t)s.expert * a.w[3].expert_bytes;
                    fprefetch_l2(mat + tile * bytes, bytes);
                }
            const uint8_t *xq_lane = xq + g * p.kp + 8 * t;
            const int2 *xsum_tok = xsum + t * (H >> 5);
#pragma unroll 1
            for (uint32_t i = 0; i < mine; i++) {
                uint32_t ul, s; bool sh;
                locate(warp + i * FW, ul, s, sh);
                const uint32_t at = ring_count + i;
                if (alive) alive = fbar_wait(&bar[at % FNS], (at / FNS) & 1u, a.status);
                alive = __all_sync(0xffffffffu, alive);
                const uint8_t *stage = ring + (at % FNS) * FSTAGE;
                float f0 = 0.0f, f1 = 0.0f;
                if (alive) {
                    // one copy of the code where the formats are the same: what a phase costs at one token is partly its code's first fetch
                    if (RT != ST && sh) consume_unit_slice<ST>(stage, nbh, s, xq_lane, xsum_tok, g, t, f0, f1);
                    else consume_unit_slice<RT>(stage, nbh, s, xq_lane, xsum_tok, g, t, f0, f1);
                }
                partial[(warp + i * FW) * 32 + lane] = make_float2(f0, f1);
                __syncwarp();
                fproxy_fence();
                if (alive && i + FNS < mine) issue(i + FNS);
            }
            if (alive) ring_count += mine;
            CLOCK(7);
            MARK(1);
            __syncthreads();
            // granules: slices added in order (the four units' sums side by side, or each read's latency shows: 89.3 against 90.4 us), SwiGLU, digit
            // pairs with one scale per chunk
#pragma unroll 1
            for (uint32_t gl = warp; gl < g1 - g0; gl += FW) {
                const bool sh = gl < n_shg;
                const uint32_t spu = sh ? spu_s : spu_r;
                const uint32_t gi = g0 + gl;                                       // granule over all sources
                const Src sr = sh ? srcs[0] : srcs[1 + (gi - gs) / gr];
                const uint32_t chunk = sh ? gi : (gi - gs) % gr;
                const bool live = t < T && ((sr.mask >> t) & 1u);
                const uint32_t row = sh ? pairs + t : t * k + sr.slot(t);
                float v[4], f0[4] = {0.0f, 0.0f, 0.0f, 0.0f}, f1[4] = {0.0f, 0.0f, 0.0f, 0.0f};
                float m = 0.0f;
                const uint32_t n0 = sh ? gl * 4 * spu_s : n_shu * spu_s + (gl * 4 - n_shu) * spu_r;
                const bool whole = n0 + 4 * spu <= slices;                         // beyond the partial buffer: never for supported shapes
                const float2 *from = partial + n0 * 32 + lane;
#pragma unroll 1
                for (uint32_t s = 0; s < spu && whole; s++)
#pragma unroll
                    for (uint32_t u = 0; u < 4; u++) { const float2 q = from[(u * spu + s) * 32]; f0[u] += q.x; f1[u] += q.y; }
                const float dx = misc_f[t];
#pragma unroll
                for (uint32_t u = 0; u < 4; u++) {
                    const float gate = f0[u] * dx, upv = f1[u] * dx;
                    v[u] = live ? gate * fast_sigmoid(gate) * upv : 0.0f;
                    m = fmaxf(m, fabsf(v[u]));
                }
                if (!whole) { if (lane == 0) atomicOr(a.status, QW4SH_ERR_STATE); continue; }
                for (int o = 4; o < 32; o <<= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));   // over the eight rows of every unit
                if (live && !finite_f32(m)) atomicOr(a.status, QW4SH_ERR_NONFINITE);
                const bool usable = finite_f32(m) && m > 0.0f;
                const float inv = usable ? __fdividef(127.0f, m) : 0.0f, d = usable ? m * (1.0f / 127.0f) : 0.0f;
                const float4 c = make_float4(d, inv, 254.0f * inv, 0.0f);
                int s1 = 0, s2 = 0;
                uint8_t *out = a.aq + (uint64_t)row * 2u * p.ap + chunk * 32u + g;
#pragma unroll
                for (uint32_t u = 0; u < 4; u++) {
                    uint32_t ra, rb;
                    digit_pair(v[u], c, ra, rb);
                    s1 += (int)(int8_t)(ra & 0xffu); s2 += (int)(int8_t)(rb & 0xffu);
                    if (live) { out[u * 8] = (uint8_t)ra; out[p.ap + u * 8] = (uint8_t)rb; }
                }
                for (int o = 4; o < 32; o <<= 1) { s1 += __shfl_xor_sync(0xffffffffu, s1, o); s2 += __shfl_xor_sync(0xffffffffu, s2, o); }
                if (live && g == 0) a.asc[(uint64_t)row * (imax >> 5) + chunk] = make_float2(d, d * fmaf((float)s2, 1.0f / 254.0f, (float)s1));
            }
        }
        CLOCK(8);
        arrive_counter(a.sync + (attempt ? S_ACT1 : S_ACT0));
        if (!wait_counter(a.sync + (attempt ? S_ACT1 : S_ACT0), NS, a.status)) return;
        // ---- the first copies of phase C, which needs the activations alone: under the comparison below.  The digits and each warp's first tiles come
        // from memory in 1.8 k cycles (one token) to 2.6 k (four), and behind the comparison nothing hid them: 97.6 -> 96.1 us for four Q4_K layers with
        // one token, 154.0 -> 150.0 for four IQ2_XXS layers with four, together with the lists above.  (The products as well, before the routes are
        // known, made it slower: their weights then arrive while the chains still read the router.) ----
        my_src = n_src > warp ? (n_src - 1 - warp) / FW + 1 : 0;
        steps = sc < (H >> 4) && lists_ok ? my_src * (((H >> 4) - sc + NS - 1) / NS) : 0;
        next_tile = sc; next_src = warp;
        begun = a.clear || attempt == 1;
        if (begun) begin_down();
        if (attempt == 1) break;
        if (!wait_counter(a.sync + S_ROUTED, T, a.status)) { if (begun) drain_down(); return; }
        CLOCK(9);
        MARK(2);
        // ---- the exact routes against the speculation ----
        // all words in one round trip (thread 0's acquire above and the barrier behind it order them for every thread); ids, logits and the flag one
        // after another took 2.5 k cycles, this 1.4 k: 93.3 against 96.4 us, four IQ2_XXS tokens 146.9 against 150.8
        const bool takes_logit = tid >= 64 && tid < 64 + T && a.router_mode != 1;
        const uint32_t my_id = tid < pairs ? __ldcg(a.ids + tid) : 0;
        const float my_weight = tid < pairs ? __ldcg(a.weights + tid) : takes_logit ? __ldcg(a.shared_logit + tid - 64) : 0.0f;
        const uint32_t failed = tid == FT - 1 ? __ldcg(a.sync + S_ROUTE_FAIL) : 0;
        if (tid < pairs) { ids_x[tid] = my_id; wts_x[tid] = my_weight; }
        if (takes_logit) misc_f[4 + tid - 64] = my_weight;
        if (__syncthreads_or(failed != 0)) {                                          // a nonfinite logit: y stays untouched
            if (begun) drain_down();
            leave();
            return;
        }
        bool same = lists_ok;
        if (lists_ok && tid < pairs) same = ((tokmask[ids_x[tid]] >> (tid / k)) & 1u) != 0;   // k distinct ids on both sides: contained = equal
        same = __syncthreads_and(same);
        if (same) {
            if (tid < pairs) { const uint32_t e = ids_x[tid], tok = tid / k; wts_s[tok * k + slotmap[e * 4 + tok]] = wts_x[tid]; }
            __syncthreads();
            break;
        }
        // repair: phase B again with the exact ids (every CTA takes this branch together: same data, same test)
        if (begun) drain_down();
        if (tid < pairs) { ids_s[tid] = ids_x[tid]; wts_s[tid] = wts_x[tid]; }
        if (tid < FMAXE / 4) reinterpret_cast<uint32_t *>(tokmask)[tid] = 0;
        if (sc == 0 && tid == 0) atomicAdd(a.sync + S_REPAIRS, 1u);             // repaired launches since the workspace was cleared (diagnostic)
        lists_ok = __syncthreads_and(alive);
    }
    CLOCK(10);

    // ================================ phase C ================================
    if (sc < (H >> 4) && lists_ok) {
        float2 *cpartial = reinterpret_cast<float2 *>(region + p.cpartial);
        const uint32_t n_tiles = ((H >> 4) - sc + NS - 1) / NS;
        if (!begun) {
            __syncthreads();                                                   // phase B's use of the region is over
            begin_down();
        }
        bool ok = __syncthreads_and(alive);
        if (ok) ok = __syncthreads_and(fbar_wait(abar, digits_read & 1u, a.status));
        if (!ok) drain_down();
        alive = ok;
        CLOCK(11);
        uint32_t n = 0;
#pragma unroll 1
        for (uint32_t ti = 0; ti < n_tiles; ti++) {
            const uint32_t tile = sc + ti * NS;
            float acc0 = 0.0f, acc1 = 0.0f;
#pragma unroll 1
            for (uint32_t si = 0; si < my_src; si++, n++) {
                const Src s = srcs[warp + si * FW];
                const uint32_t tokg = g >> 1;
                const uint32_t row_g = s.shared ? pairs + (tokg < T ? tokg : 0) : (((s.mask >> tokg) & 1u) ? tokg * k + s.slot(tokg) : 0);
                const bool live_t = t < T && ((s.mask >> t) & 1u);
                const uint32_t row_t = s.shared ? pairs + (t < T ? t : 0) : (live_t ? t * k + s.slot(t) : 0);
                const uint8_t *aq_lane = aq + (2 * row_g + (g & 1u)) * p.ap + 8 * t;
                const float2 *asc_tok = asc + row_t * (imax >> 5);
                const uint32_t at = tiles_read + n;
                if (alive) alive = fbar_wait(&tilebar[at % FNC], (at / FNC) & 1u, a.status);
                alive = __all_sync(0xffffffffu, alive);
                const uint8_t *stage = tiles + (at % FNC) * FSTAGE;
                float f0 = 0.0f, f1 = 0.0f;
                if (alive) {
                    if (RT != ST && s.shared) consume_down_tile<ST>(stage, IS >> 8, aq_lane, asc_tok, g, t, f0, f1);
                    else consume_down_tile<RT>(stage, (s.shared ? IS : I) >> 8, aq_lane, asc_tok, g, t, f0, f1);
                }
                __syncwarp();
                fproxy_fence();
                if (alive && n + FNC < steps) issue_down(n + FNC);
                if (live_t) {
                    const float coef = s.shared ? fast_sigmoid(misc_f[4 + t]) : wts_s[t * k + s.slot(t)];
                    acc0 = fmaf(coef, f0, acc0); acc1 = fmaf(coef, f1, acc1);
                }
            }
            cpartial[warp * 32 + lane] = make_float2(acc0, acc1);
            __syncthreads();
            if (tid < 64) {                                                    // rows g (threads 0-31) and g + 8 (32-63), warps added in order
                const uint32_t l = tid & 31u, gg = l >> 2, tt = l & 3u, hi = tid >> 5;
                float sum = 0.0f;
                const float *from = reinterpret_cast<const float *>(cpartial) + 2 * l + hi;
#pragma unroll
                for (uint32_t w = 0; w < FW; w++) sum += from[w * 64];
                if (tt < T && alive) {
                    if (!finite_f32(sum)) atomicOr(a.status, QW4SH_ERR_NONFINITE);
                    a.y[(uint64_t)tt * H + tile * 16 + hi * 8 + gg] = sum;
                    if (!hc_add(a.hc, tt, tile * 16 + hi * 8 + gg, H, sum)) atomicOr(a.status, QW4SH_ERR_NONFINITE);
                }
            }
            __syncthreads();
        }
    }
    CLOCK(12);
    MARK(3);
    leave();
#undef CLOCK
#undef MARK
}

}  // namespace qw4

using namespace qw4;

extern "C" int qw4sh_note_launch(const char *name);

static DevTensor fdev(const QW4ShTensor &s) {
    DevTensor t;
    t.data = s.data; t.type = s.type; t.k_storage = s.k_storage; t.k_logical = s.k_logical;
    t.n_out = s.n_out; t.n_experts = s.n_experts; t.row_bytes = s.row_bytes; t.expert_bytes = s.expert_bytes;
    return t;
}

static int g_fused_mode = -1;                          // -1 automatic, 0 never
extern "C" void qw4sh_set_fused_decode(int mode) { g_fused_mode = mode; }
static int g_wrong_speculation = 0;
extern "C" void qw4sh_set_wrong_speculation(int on) { g_wrong_speculation = on ? 1 : 0; }

static int g_marks = 0;
extern "C" void qw4sh_set_decode_marks(int on) { g_marks = on ? 1 : 0; }

static bool fused_type(uint32_t type) { return type == T_Q4_K || type == T_IQ2_XXS; }
static uint32_t slice_blocks(uint32_t) { return FGeo<T_Q4_K>::SLICE_BLOCKS; }          // both formats of this path: 512 columns per slice

// Chain CTAs: one per 32 rows of the router (the shared expert's router is row E), and at least
// one per token (chain CTA t routes token t).  The fast mode keeps only the routing CTAs.
static uint32_t chain_ctas(const QW4ShLayer *l, size_t tokens, int router_mode) {
    const uint32_t by_rows = router_mode == 1 ? 0 : (l->experts + 1 + CROWS - 1) / CROWS;
    return by_rows > tokens ? by_rows : (uint32_t)tokens;
}

// Most slices one streaming CTA can get: its share of the granules (whole granules of four units,
// the shared expert's first), each unit cut into its format's number of slices.
static uint32_t partial_capacity(const QW4ShLayer *l, size_t tokens, uint32_t streaming) {
    const uint32_t nbh = l->hidden >> 8, spu_s = nbh / slice_blocks(l->w[4].type), spu_r = nbh / slice_blocks(l->w[1].type);
    const uint64_t total = (l->shared_inter >> 5) + (uint64_t)tokens * l->top_k * (l->inter >> 5);
    const uint32_t per_cta = (uint32_t)((total + streaming - 1) / streaming) + 1;
    return per_cta * 4 * (spu_s > spu_r ? spu_s : spu_r);
}

// Phase C clear of the digit image of x where there is room: everywhere but at hidden 4096 with four tokens and more than fifteen experts each, where
// the two lie over each other and phase C's first copies wait for the comparison.
static FPlan plan_for(const QW4ShLayer *l, size_t tokens, uint32_t streaming, bool *clear) {
    const uint32_t imax = l->inter > l->shared_inter ? l->inter : l->shared_inter, rows = (uint32_t)tokens * l->top_k + (uint32_t)tokens;
    const FPlan p = make_fplan(l->hidden, imax, rows, partial_capacity(l, tokens, streaming), true);
    *clear = p.total <= FSMEM;
    return *clear ? p : make_fplan(l->hidden, imax, rows, partial_capacity(l, tokens, streaming), false);
}

// Bytes of the workspace arrays the kernel needs beyond the common ones (for `cap` tokens, at most FTOK used).
extern "C" void qw4sh_fused_scratch_sizes(const QW4ShLayer *l, size_t *aq_bytes, size_t *asc_bytes, size_t *fast_bytes) {
    const uint32_t imax = l->inter > l->shared_inter ? l->inter : l->shared_inter;
    const size_t rows = (size_t)FTOK * l->top_k + FTOK;
    *aq_bytes = rows * 2 * (imax + 32) + 256;
    *asc_bytes = rows * (imax / 32 + 1) * 8 + 256;
    *fast_bytes = (size_t)FTOK * ((l->experts + 1 + 3) & ~3u) * 4 + 256;
}

// ---- tensor maps of the gate / up matrices ---------------------------------------------------------------------------
typedef CUresult (*EncodeTiled)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *, const cuuint64_t *,
                                const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle,
                                CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
// The tensor this path streams for resident tensor i: the tensor itself (Q4_K) or its expanded image (IQ2_XXS).
static DevTensor fused_view(const QW4ShLayer *l, int i) {
    DevTensor t = fdev(l->w[i]);
    const int holder = (i == 2 || i == 5) ? i - 1 : i;                     // gate and up share the gate's image
    if (t.type == T_IQ2_XXS && l->fused_alt[holder]) {
        t.data = (const uint8_t *)l->fused_alt[holder];
        t.type = T_IQ2N;
        t.row_bytes = (t.k_storage >> 9) * (IQ2N_BLOCK / 16);
        t.expert_bytes = (uint64_t)t.row_bytes * t.n_out;
    }
    return t;
}
// {32-bit words of a row's packed payload, rows of an expert, experts}; box = one slice (288 bytes) of eight rows.
static int rows_map(const DevTensor &t, CUtensorMap *map) {
    static EncodeTiled encode = nullptr;
    if (!encode) {
        void *fn = nullptr;
        cudaDriverEntryPointQueryResult status;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &status) != cudaSuccess || !fn) return -1;
        encode = (EncodeTiled)fn;
    }
    constexpr uint32_t slice = FGeo<T_Q4_K>::SLICE_BYTES / 16;
    const cuuint64_t dims[3] = {(cuuint64_t)t.row_bytes / 4, t.n_out, t.n_experts};
    const cuuint64_t strides[2] = {(cuuint64_t)t.row_bytes, t.expert_bytes};
    const cuuint32_t box[3] = {slice / 4, 8, 1}, elem[3] = {1, 1, 1};
    const CUresult r = encode(map, CU_TENSOR_MAP_DATA_TYPE_UINT32, 3, (void *)t.data, dims, strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE,
                              CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? 0 : -2;
}
static bool fused_type(uint32_t type);
extern "C" void qw4sh_fused_release(QW4ShLayer *l) {
    for (int i = 0; i < 8; i++) { if (l->fused_alt[i]) cudaFree(l->fused_alt[i]); l->fused_alt[i] = nullptr; }
    l->fused_alt_bytes = 0;
    l->fused_maps_ready = 0;
}
// Called once the images are resident.  A layer the path cannot take simply gets no maps and no expanded images; 0
// unless a CUDA call failed.
extern "C" int qw4sh_fused_prepare(QW4ShLayer *l) {
    l->fused_maps_ready = 0;
    l->fused_alt_bytes = 0;
    for (int i = 0; i < 8; i++) l->fused_alt[i] = nullptr;
    static_assert(sizeof(CUtensorMap) == 128, "tensor map size");
    if (g_fused_mode == 0) return 0;                                            // switched off before create: no maps, no expanded images
    if (l->w[2].type != l->w[1].type || l->w[3].type != l->w[1].type || l->w[5].type != l->w[4].type || l->w[6].type != l->w[4].type) return 0;
    for (int i = 1; i <= 6; i++) {
        const QW4ShTensor *t = &l->w[i];
        if (!fused_type(t->type) || t->k_storage % 512 || t->k_logical != t->k_storage || t->n_out % 32 || ((uintptr_t)t->data & 15u) ||
            t->expert_bytes % 16) return 0;
    }
    // expanded images: gate and up of a group share one (unit slices interleaved, held by the gate's slot), down has its own
    for (int i = 1; i <= 6; i++) {
        if (l->w[i].type != T_IQ2_XXS || i == 2 || i == 5) continue;
        const bool pair = i == 1 || i == 4;
        const DevTensor src = fdev(l->w[i]);
        if (pair && (l->w[i + 1].n_out != src.n_out || l->w[i + 1].k_storage != src.k_storage || l->w[i + 1].n_experts != src.n_experts)) return 0;
        const size_t bytes = (size_t)src.n_experts * src.n_out * (src.k_storage >> 9) * (IQ2N_BLOCK / 16) * (pair ? 2 : 1);
        cudaError_t e = cudaMalloc(&l->fused_alt[i], bytes);
        if (e == cudaSuccess) e = cudaMemset(l->fused_alt[i], 0, bytes);
        if (e == cudaSuccess) {
            const uint64_t halves = (uint64_t)src.n_experts * src.n_out * (src.k_storage >> 7);
            iq2_expand_kernel<<<(unsigned)((halves + 255) / 256), 256>>>(src, (uint8_t *)l->fused_alt[i], pair ? 0 : -1);
            if (pair) iq2_expand_kernel<<<(unsigned)((halves + 255) / 256), 256>>>(fdev(l->w[i + 1]), (uint8_t *)l->fused_alt[i], 1);
            e = cudaDeviceSynchronize();
        }
        if (e != cudaSuccess) { qw4sh_fused_release(l); return -1; }
        l->fused_alt_bytes += bytes;
    }
    const int which[4] = {1, 2, 4, 5};
    for (int i = 0; i < 4; i++) {
        alignas(64) CUtensorMap map = {};
        const DevTensor view = fused_view(l, which[i]);
        if (view.type == T_Q4_K && rows_map(view, &map)) { qw4sh_fused_release(l); return -1; }
        memcpy(l->fused_maps[i], &map, sizeof map);
    }
    l->fused_maps_ready = 1;
    return 0;
}

// Probe entry: decode rows of tensor i (1-6) from its expanded image; -3 when the tensor has none.
extern "C" int qw4sh_fused_decode_rows_expanded(const QW4ShLayer *l, int i, size_t expert, size_t row0, size_t rows, float *out, void *stream) {
    if (i < 1 || i > 6 || l->w[i].type != T_IQ2_XXS) return -3;
    const int holder = (i == 2 || i == 5) ? i - 1 : i;
    if (!l->fused_alt[holder]) return -3;
    const int which = i == 3 || i == 6 ? -1 : (i == holder ? 0 : 1);
    const uint64_t total = (uint64_t)rows * l->w[i].k_storage;
    if (!total) return 0;
    iq2n_decode_rows_kernel<<<(unsigned)((total + 255) / 256), 256, 0, (cudaStream_t)stream>>>((const uint8_t *)l->fused_alt[holder], l->w[i].k_storage,
                                                                                          l->w[i].n_out, (uint32_t)expert, (uint32_t)row0, (uint32_t)rows,
                                                                                          which, out);
    return qw4sh_note_launch("iq2n_decode_rows_kernel");
}

// Whether the one-kernel decode path covers this layer and batch.
extern "C" int qw4sh_fused_supported(const QW4ShLayer *l, size_t tokens, const float *x, const float *y, int grid) {
    if (g_fused_mode == 0 || !l->fused_maps_ready) return 0;
    if (!tokens || tokens > FTOK || l->top_k > FMAXK || l->experts > FMAXE || l->top_k > l->experts) return 0;
    const uint32_t H = l->hidden, I = l->inter, IS = l->shared_inter;
    if (H % 1024 || H > 4096 || I % 256 || IS % 256 || !I || !IS) return 0;
    if (((uintptr_t)x | (uintptr_t)y) & 15u) return 0;
    if (l->w[0].type != T_F32 || l->w[7].type != T_F32) return 0;
    const uint32_t rt = l->w[1].type, st = l->w[4].type;
    if (!fused_type(rt) || !fused_type(st)) return 0;
    if (l->w[2].type != rt || l->w[3].type != rt || l->w[5].type != st || l->w[6].type != st) return 0;
    for (int i = 1; i <= 6; i++) if (l->w[i].k_logical != l->w[i].k_storage) return 0;
    // a down tile (16 rows) must fit one ring stage
    if (I > 512 || IS > 512 || I % 512 || IS % 512) return 0;
    const uint32_t nc = chain_ctas(l, tokens, 0);
    if (grid < 1 || (uint32_t)grid <= nc) return 0;
    const uint32_t streaming = (uint32_t)grid - nc;
    if (streaming * FRMAX < l->experts + 1) return 0;
    bool clear;
    if (plan_for(l, tokens, streaming, &clear).total > FSMEM || make_cplan(H).total > FSMEM) return 0;
    return 1;
}

template <uint32_t RT, uint32_t ST, bool MARKS>
static int launch_fused_as(const FusedArgs &a, const QW4ShLayer *layer, uint32_t smem, int grid, cudaStream_t stream) {
    static bool configured[64] = {false};                 // per device: the attribute and the residency check
    int device = 0;
    cudaError_t e = cudaGetDevice(&device);
    if (e != cudaSuccess || device < 0 || device >= 64) return (int)cudaErrorInvalidDevice;
    if (!configured[device]) {
        e = cudaFuncSetAttribute(fused_decode_kernel<RT, ST, MARKS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)FSMEM);
        if (e != cudaSuccess) return (int)e;
        // the grid barriers need every CTA resident: one per SM, and an SM must take one
        int resident = 0;
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&resident, fused_decode_kernel<RT, ST, MARKS>, FT, FSMEM);
        if (e != cudaSuccess) return (int)e;
        if (resident < 1) return (int)cudaErrorCooperativeLaunchTooLarge;
        configured[device] = true;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)grid); cfg.blockDim = dim3(FT); cfg.dynamicSmemBytes = smem; cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization; attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr; cfg.numAttrs = 1;
    alignas(64) CUtensorMap maps[4];
    memcpy(maps, layer->fused_maps, sizeof maps);
    e = cudaLaunchKernelEx(&cfg, fused_decode_kernel<RT, ST, MARKS>, a, maps[0], maps[1], maps[2], maps[3]);
    if (e != cudaSuccess) return (int)e;
    return qw4sh_note_launch("fused_decode_kernel");
}
template <uint32_t RT, uint32_t ST>
static int launch_fused(const FusedArgs &a, const QW4ShLayer *layer, uint32_t smem, int grid, cudaStream_t stream) {
    return g_marks ? launch_fused_as<RT, ST, true>(a, layer, smem, grid, stream) : launch_fused_as<RT, ST, false>(a, layer, smem, grid, stream);
}

extern "C" int qw4sh_fused_decode(const QW4ShLayer *layer, const QW4ShWork *work, const float *x, float *y, size_t tokens,
                                  uint32_t *ids_out, float *weights_out, int router_mode, int sm_count) {
    if (!work->fused_aq || !work->fused_asc || !work->logits_fast) return -5;
    FusedArgs a;
    for (int i = 0; i < 8; i++) a.w[i] = fused_view(layer, i);
    a.x = x; a.y = y;
    a.hc = HcAdd{work->hc_residual, work->hc_inject, work->hc_streams};
    a.status_mirror = work->status_mirror;
    a.tokens = (uint32_t)tokens; a.hidden = layer->hidden; a.experts = layer->experts; a.top_k = layer->top_k;
    a.inter = layer->inter; a.shared_inter = layer->shared_inter; a.norm = layer->norm; a.router_mode = router_mode == 0 && g_wrong_speculation ? 2 : router_mode;
    a.logits = work->logits; a.shared_logit = work->shared_logit; a.ids = work->ids; a.weights = work->weights;
    a.logits_fast = work->logits_fast; a.fast_pitch = (layer->experts + 1 + 3) & ~3u;
    a.aq = (uint8_t *)work->fused_aq; a.asc = (float2 *)work->fused_asc;
    a.ids_out = ids_out; a.weights_out = weights_out;
    a.sync = work->sync; a.status = work->status;
    const uint32_t rt = layer->w[1].type, st = layer->w[4].type;
    const uint32_t streaming = (uint32_t)sm_count - chain_ctas(layer, tokens, 0);     // the same split in every mode (plans, capacity)
    a.chain_ctas = (uint32_t)sm_count - streaming;
    a.partial_slices = partial_capacity(layer, tokens, streaming);
    bool clear;
    const FPlan p = plan_for(layer, tokens, streaming, &clear);
    a.clear = clear;
    const CPlan c = make_cplan(layer->hidden);
    const uint32_t smem = p.total > c.total ? p.total : c.total;
    if (smem > FSMEM) return -4;
    cudaStream_t s = (cudaStream_t)work->stream;
    if (rt == T_Q4_K) return st == T_Q4_K ? launch_fused<T_Q4_K, T_Q4_K>(a, layer, smem, sm_count, s) : launch_fused<T_Q4_K, T_IQ2N>(a, layer, smem, sm_count, s);
    return st == T_Q4_K ? launch_fused<T_IQ2N, T_Q4_K>(a, layer, smem, sm_count, s) : launch_fused<T_IQ2N, T_IQ2N>(a, layer, smem, sm_count, s);
}
