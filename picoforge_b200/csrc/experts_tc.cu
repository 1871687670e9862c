// Launches of the tensor-core expert products (experts_tc.cuh holds the kernel's body and its reasons), and what they
// need beside them: tensor maps of the resident images, the split of the layer's input rows, the groups of the dispatch
// lists, and the wide images of tensors in formats that have no dequantiser.
#include <cuda.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include <string.h>

#include "experts_tc.cuh"

namespace qw4 {

// Two names for one body: the Q4_K launches of large batches, and every other format and size.
template <uint32_t F, int MODE>
__global__ void __launch_bounds__(XRole<F>::THREADS, 1) expert_tile_kernel(const __grid_constant__ XMaps maps, const __grid_constant__ XArgs a) {
    extern __shared__ __align__(1024) uint8_t smem[];
    expert_tc_body<F, MODE>(maps, a, smem);
}
template <int MODE>
__global__ void __launch_bounds__(XRole<T_Q4_K>::THREADS, 1) prefill_tc_kernel(const __grid_constant__ XMaps maps, const __grid_constant__ XArgs a) {
    extern __shared__ __align__(1024) uint8_t smem[];
    expert_tc_body<T_Q4_K, MODE>(maps, a, smem);
}

// x [rows][k], `pitch` floats apart -> fp16 hi / lo of x * 2^e (the kernel's column order), sums over 16 columns (hi / lo),
// and 2^-e per row; e puts the row's largest value into [512, 1024).  One CTA of 128 threads per row, 16 columns a thread.
template <bool ALIGNED>
__global__ void __launch_bounds__(128) split_rows_kernel(const float *__restrict__ x, uint32_t pitch, uint32_t k, __half *__restrict__ hi, __half *__restrict__ lo,
                                                         __half *__restrict__ sum_hi, __half *__restrict__ sum_lo, float *__restrict__ scale) {
    __shared__ float red[4];
    const uint32_t r = blockIdx.x, segs = k >> 4, tid = threadIdx.x;
    const float *src = x + (uint64_t)r * pitch;
    float top = 0.0f;
    for (uint32_t i = tid; i < segs * 4; i += 128) { const float4 v = load_quad<ALIGNED>(src + 4 * i); top = fmaxf(top, fmaxf(fmaxf(fabsf(v.x), fabsf(v.y)), fmaxf(fabsf(v.z), fabsf(v.w)))); }
    for (int o = 16; o; o >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, o));
    if ((tid & 31u) == 0) red[tid >> 5] = top;
    __syncthreads();
    top = fmaxf(fmaxf(red[0], red[1]), fmaxf(red[2], red[3]));
    float up, down;
    xscale_of(top, up, down);
    if (tid == 0) scale[r] = down;
    for (uint32_t s = tid; s < segs; s += 128) {
        float sum = 0.0f;
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const float4 p = load_quad<ALIGNED>(src + s * 16 + 8 * h), q = load_quad<ALIGNED>(src + s * 16 + 8 * h + 4);
            const float v[8] = {p.x * up, p.y * up, p.z * up, p.w * up, q.x * up, q.y * up, q.z * up, q.w * up};
            uint32_t a[4], b[4];
#pragma unroll
            for (int i = 0; i < 8; i++) sum += v[i];
            xsplit8(v, a, b);
            const uint64_t at = (uint64_t)r * k + s * 16 + 8 * h;
            *reinterpret_cast<uint4 *>(hi + at) = make_uint4(a[0], a[1], a[2], a[3]);
            *reinterpret_cast<uint4 *>(lo + at) = make_uint4(b[0], b[1], b[2], b[3]);
        }
        const __half sh = __float2half_rn(sum);
        sum_hi[(uint64_t)r * segs + s] = sh;
        sum_lo[(uint64_t)r * segs + s] = __float2half_rn(sum - __half2float(sh));
    }
}

// Groups of at most 32 rows out of the expert-sorted lists: one CTA, thread i owns active expert i (then i + 1024, ...), a
// block-wide exclusive scan of the group counts gives every expert its place: active experts in ascending order, each
// expert's groups by ascending row.
__global__ void __launch_bounds__(1024) build_tile_groups_kernel(const uint32_t *__restrict__ offsets, const uint32_t *__restrict__ active,
                                                                 XGroup *groups, uint32_t *n_groups) {
    __shared__ uint32_t wsum[32];
    __shared__ uint32_t s_base;
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5, n_active = active[0];
    if (tid == 0) s_base = 0;
    __syncthreads();
    for (uint32_t i0 = 0; i0 < n_active; i0 += 1024) {
        const uint32_t i = i0 + tid;
        uint32_t e = 0, first = 0, end = 0;
        if (i < n_active) { e = active[1 + i]; first = offsets[e]; end = offsets[e + 1]; }
        const uint32_t count = (end - first + XTOK - 1) / XTOK;
        uint32_t scan = count;
        for (int o = 1; o < 32; o <<= 1) { const uint32_t v = __shfl_up_sync(0xffffffffu, scan, o); if (lane >= (uint32_t)o) scan += v; }
        if (lane == 31) wsum[warp] = scan;
        __syncthreads();
        if (warp == 0) {
            const uint32_t v = wsum[lane];
            uint32_t sc = v;
            for (int o = 1; o < 32; o <<= 1) { const uint32_t u = __shfl_up_sync(0xffffffffu, sc, o); if (lane >= (uint32_t)o) sc += u; }
            wsum[lane] = sc - v;
        }
        __syncthreads();
        uint32_t at = s_base + wsum[warp] + scan - count;
        for (uint32_t r = first; r < end; r += XTOK) groups[at++] = XGroup{e, r, min(XTOK, end - r), 0};
        __syncthreads();
        if (tid == 1023) s_base = at;                                // end of the last thread = end of this pass
        __syncthreads();
    }
    if (tid == 0) *n_groups = s_base;
}
__global__ void build_dense_tile_groups_kernel(uint32_t tokens, XGroup *groups, uint32_t *n_groups) {
    const uint32_t n = (tokens + XTOK - 1) / XTOK;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        groups[i] = XGroup{0, i * XTOK, min(XTOK, tokens - i * XTOK), 0};
    if (blockIdx.x == 0 && threadIdx.x == 0) *n_groups = n;
}

// One row of a tensor in any format -> its wide form: fp16 hi / lo of w * 2^e in the kernel's column order, and 2^-e.  Exact
// for F16, BF16 (8 bits), Q8_0 (11 x 7 bits) and MXFP4 weights within 2^34 of the row's largest; half a unit in the last place
// of FP32 for F32 weights.
__global__ void __launch_bounds__(128) widen_rows_kernel(DevTensor t, __half *__restrict__ hi, __half *__restrict__ lo, float *__restrict__ scale) {
    __shared__ float red[4];
    const uint64_t grow = blockIdx.x;
    const uint32_t expert = (uint32_t)(grow / t.n_out), row = (uint32_t)(grow % t.n_out), k = t.k_logical, tid = threadIdx.x;
    float top = 0.0f;
    for (uint32_t c = tid; c < k; c += 128) top = fmaxf(top, fabsf(decode_value(t, expert, row, c)));
    for (int o = 16; o; o >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, o));
    if ((tid & 31u) == 0) red[tid >> 5] = top;
    __syncthreads();
    top = fmaxf(fmaxf(red[0], red[1]), fmaxf(red[2], red[3]));
    float up, down;
    xscale_of(top, up, down);
    if (tid == 0) scale[grow] = down;
    for (uint32_t c = tid; c < k; c += 128) {
        const float v = decode_value(t, expert, row, c) * up;
        const __half h = __float2half_rn(v);
        hi[grow * k + xperm(c)] = h;
        lo[grow * k + xperm(c)] = __float2half_rn(v - __half2float(h));
    }
}

}  // namespace qw4

using namespace qw4;

extern "C" int qw4sh_note_launch(const char *name);

static DevTensor xdev(const QW4ShTensor &s) {
    DevTensor t;
    t.data = s.data; t.type = s.type; t.k_storage = s.k_storage; t.k_logical = s.k_logical;
    t.n_out = s.n_out; t.n_experts = s.n_experts; t.row_bytes = s.row_bytes; t.expert_bytes = s.expert_bytes;
    return t;
}

// ---- tensor maps --------------------------------------------------------------------------------
typedef CUresult (*TileEncode)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *, const cuuint64_t *, const cuuint32_t *,
                               const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
static TileEncode tile_encode() {
    static TileEncode encode = nullptr;
    if (!encode) {
        void *fn = nullptr;
        cudaDriverEntryPointQueryResult status;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &status) != cudaSuccess || !fn) return nullptr;
        encode = (TileEncode)fn;
    }
    return encode;
}
// 128 rows x `box` bytes out of rows `pitch` bytes apart; rank 2 counts all rows of all experts, rank 3 {bytes, rows, experts}.
static int rows_map(const void *base, int rank, uint64_t pitch, uint64_t rows, uint64_t experts, uint64_t expert_bytes, uint32_t box, CUtensorMapSwizzle swizzle,
                    bool halves, CUtensorMap *map) {
    TileEncode encode = tile_encode();
    if (!encode) return -1;
    if (pitch % 16 || ((uintptr_t)base & 15u) || (rank == 3 && expert_bytes % 16)) return -2;
    const uint32_t size = halves ? 2 : 1;
    const cuuint64_t dims[3] = {pitch / size, rows, experts}, strides[2] = {pitch, expert_bytes};
    const cuuint32_t boxes[3] = {box / size, XROWS, 1}, elem[3] = {1, 1, 1};
    return encode(map, halves ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_UINT8, rank, const_cast<void *>(base), dims, strides, boxes, elem,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS ? 0 : -3;
}

// Whether the kernel's geometry takes the tensor in this role: whole tiles of rows (two of them per item for down), whole
// units of columns; stored columns beyond the logical ones (down) are never multiplied.
static bool tile_shape(const QW4ShTensor *t, bool down) {
    if (t->type != T_Q4_K && t->k_storage > 4096) return false;                // room for the scales that lie apart from the codes
    if (t->k_logical % (down ? 128 : 256) || t->n_out % (down ? 256 : 128)) return false;
    return down || t->k_logical == t->k_storage;
}
static int packed_maps(QW4ShTensor *t) {
    const uint32_t nb = t->k_storage >> 8;
    alignas(64) CUtensorMap maps[2];
    int rc = -4;
    if (t->type == T_Q4_K && t->k_storage % 256 == 0)
        rc = rows_map(t->data, 2, t->row_bytes, (uint64_t)t->n_out * t->n_experts, 1, 0, 144, CU_TENSOR_MAP_SWIZZLE_NONE, false, &maps[0]);
    else if (t->type == T_Q2_K && t->k_storage % 256 == 0) {
        rc = rows_map(t->data, 3, nb * 64u, t->n_out, t->n_experts, t->expert_bytes, 64, CU_TENSOR_MAP_SWIZZLE_64B, false, &maps[0]);
        if (!rc) rc = rows_map(t->data + (uint64_t)t->n_out * nb * 64u, 3, nb * 16u, t->n_out, t->n_experts, t->expert_bytes, 16, CU_TENSOR_MAP_SWIZZLE_NONE, false, &maps[1]);
    } else if (t->type == T_IQ2_XXS && t->k_storage % 512 == 0)
        rc = rows_map(t->data, 3, nb * 64u, t->n_out, t->n_experts, t->expert_bytes, 128, CU_TENSOR_MAP_SWIZZLE_128B, false, &maps[0]);
    if (rc) return rc;
    memcpy(t->tc_maps, maps, sizeof maps);
    t->tc_format = t->type;
    return 0;
}
static int widen(QW4ShTensor *t) {
    const size_t rows = (size_t)t->n_out * t->n_experts, image = rows * t->k_logical * sizeof(__half), scale_at = 2 * image;
    if (rows > 0x7fffffffu || t->k_logical % 64) return -4;
    char *block = nullptr;
    if (cudaMalloc(&block, scale_at + rows * sizeof(float)) != cudaSuccess) { (void)cudaGetLastError(); return -1; }
    alignas(64) CUtensorMap maps[2];
    int rc = 0;
    for (int i = 0; i < 2 && !rc; i++)
        rc = rows_map(block + i * image, 2, t->k_logical * 2ull, rows, 1, 0, 128, CU_TENSOR_MAP_SWIZZLE_128B, true, &maps[i]);
    if (!rc) {
        widen_rows_kernel<<<(unsigned)rows, 128>>>(xdev(*t), (__half *)block, (__half *)(block + image), (float *)(block + scale_at));
        if (cudaGetLastError() != cudaSuccess || cudaDeviceSynchronize() != cudaSuccess) rc = -1;
    }
    if (rc) { cudaFree(block); return rc; }
    memcpy(t->tc_maps, maps, sizeof maps);
    t->wide = block; t->wide_scale = (float *)(block + scale_at); t->wide_bytes = scale_at + rows * sizeof(float);
    t->tc_format = T_WIDE;
    return 0;
}
// Called once the images are resident.  Tensors that the kernel can take get their maps; the shared expert's in another
// format (the checkpoint's is Q8_0, 640 columns) a wide image beside the packed one: about 4 bytes a weight, once a layer,
// where a dequantiser for 34-byte blocks that start on no word boundary would run for one expert in 512.  Routed tensors in
// such formats stay on the CUDA-core kernels.  Never fails the create.
extern "C" int qw4sh_tile_prepare(QW4ShLayer *l) {
    static_assert(sizeof(CUtensorMap) == 128, "tensor map size");
    for (int i = 1; i <= 6; i++) {
        QW4ShTensor *t = &l->w[i];
        t->tc_format = 0;
        if (tile_shape(t, i == 3 || i == 6)) (void)packed_maps(t);
    }
    if (!l->w[1].tc_format || !l->w[2].tc_format || !l->w[3].tc_format) return 0;
    for (int i = 4; i <= 6; i++) {
        QW4ShTensor *t = &l->w[i];
        if (!t->tc_format && tile_shape(t, i == 6)) (void)widen(t);
    }
    return 0;
}
extern "C" void qw4sh_tile_release(QW4ShLayer *l) {
    for (int i = 4; i <= 6; i++) { if (l->w[i].wide) cudaFree(l->w[i].wide); l->w[i].wide = nullptr; l->w[i].tc_format = 0; }
}
extern "C" int qw4sh_tile_supported(const QW4ShTensor *w) { return w->tc_format != 0; }

// ---- launches -----------------------------------------------------------------------------------
extern "C" int qw4sh_split_rows(const float *x, uint32_t pitch, uint32_t rows, uint32_t k, const QW4ShSplit *to, void *stream) {
    if (!rows) return 0;
    (rows_aligned(x, pitch) ? split_rows_kernel<true> : split_rows_kernel<false>)<<<rows, 128, 0, (cudaStream_t)stream>>>(x, pitch, k, (__half *)to->hi, (__half *)to->lo, (__half *)to->sum_hi, (__half *)to->sum_lo, to->scale);
    return qw4sh_note_launch("split_rows_kernel");
}
// Groups of <= 32 rows (16-byte records {expert, first row, rows, 0}) for qw4sh_expert_tc: from the expert-sorted lists, or
// dense (the shared expert: rows in token order).
extern "C" int qw4sh_build_tile_groups(const uint32_t *offsets, const uint32_t *active, void *groups, uint32_t *n_groups, void *stream) {
    build_tile_groups_kernel<<<1, 1024, 0, (cudaStream_t)stream>>>(offsets, active, (XGroup *)groups, n_groups);
    return qw4sh_note_launch("build_tile_groups_kernel");
}
extern "C" int qw4sh_build_dense_tile_groups(uint32_t tokens, void *groups, uint32_t *n_groups, void *stream) {
    build_dense_tile_groups_kernel<<<(tokens / XTOK + 256) / 256, 256, 0, (cudaStream_t)stream>>>(tokens, (XGroup *)groups, n_groups);
    return qw4sh_note_launch("build_dense_tile_groups_kernel");
}

static unsigned long long *g_prefill_debug = nullptr;
extern "C" void qw4sh_prefill_debug(void *words) { g_prefill_debug = (unsigned long long *)words; }

template <typename Kernel>
static int launch_tc(Kernel kernel, bool (&configured)[64], bool early, size_t smem, int threads, const XMaps &maps, const XArgs &a, int ctas, cudaStream_t stream,
                     const char *name) {
    int device = 0;
    cudaError_t e = cudaGetDevice(&device);
    if (e != cudaSuccess || device < 0 || device >= 64) return (int)cudaErrorInvalidDevice;
    if (!configured[device]) {                                               // the attribute stays with the function
        e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return (int)e;
        configured[device] = true;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)ctas); cfg.blockDim = dim3((unsigned)threads); cfg.dynamicSmemBytes = smem; cfg.stream = stream;
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization; attr.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &attr; cfg.numAttrs = early ? 1 : 0;
    e = cudaLaunchKernelEx(&cfg, kernel, maps, a);
    if (e != cudaSuccess) return (int)e;
    return qw4sh_note_launch(name);
}
// Down products are launched early, the shared expert's only with few CTAs: they run beside other kernels, whose SMs they would hold
// (148 of them made a four-token step 14% slower).
static const int EARLY_SHARED = 32;
template <uint32_t F, int MODE>
static int launch_tile(const XMaps &maps, const XArgs &a, int ctas, cudaStream_t stream) {
    static bool configured[64] = {false};
    return launch_tc(expert_tile_kernel<F, MODE>, configured, MODE == 1 && (a.row_to_pair || ctas <= EARLY_SHARED), xm_total<F>(), XRole<F>::THREADS, maps, a, ctas, stream, "expert_tile_kernel");
}
template <int MODE>
static int launch_prefill(const XMaps &maps, const XArgs &a, int ctas, cudaStream_t stream) {
    static bool configured[64] = {false};
    return launch_tc(prefill_tc_kernel<MODE>, configured, MODE == 1 && (a.row_to_pair || ctas <= EARLY_SHARED), xm_total<T_Q4_K>(), XRole<T_Q4_K>::THREADS, maps, a, ctas, stream, "prefill_tc_kernel");
}

// mode 0: gate (w0) + up (w1) + SwiGLU, `in` the split rows of x, `act` receives the split activation (row = pair);
// mode 1: down (w0), `in` that activation, -> out [pairs][n_out].  `prefill`: the launch belongs to a large all-Q4_K batch.
extern "C" int qw4sh_expert_tc(int mode, int prefill, const QW4ShTensor *w0, const QW4ShTensor *w1, const void *groups, const uint32_t *n_groups,
                               const uint32_t *row_to_pair, uint32_t k_div, const QW4ShSplit *in, const QW4ShSplit *act, float *out, uint32_t *status,
                               int ctas, void *stream) {
    alignas(64) XMaps maps;
    memcpy(maps.m[0], w0->tc_maps, sizeof maps.m[0]);
    memcpy(maps.m[1], (w1 ? w1 : w0)->tc_maps, sizeof maps.m[1]);
    XArgs a;
    a.w0 = xdev(*w0); a.w1 = xdev(w1 ? *w1 : *w0);
    a.row_scale0 = w0->wide_scale; a.row_scale1 = (w1 ? w1 : w0)->wide_scale;
    a.units = w0->k_logical / (mode == 0 ? 256 : 128); a.tiles = w0->n_out / (mode == 0 ? 128 : 256); a.k_div = k_div;
    a.groups = (const XGroup *)groups; a.n_groups = n_groups; a.row_to_pair = row_to_pair;
    a.in_hi = (const __half *)in->hi; a.in_lo = (const __half *)in->lo; a.sum_hi = (const __half *)in->sum_hi; a.sum_lo = (const __half *)in->sum_lo;
    a.in_scale = in->scale; a.in_pitch = w0->k_logical;
    a.out_hi = act ? (__half *)act->hi : nullptr; a.out_lo = act ? (__half *)act->lo : nullptr;
    a.osum_hi = act ? (__half *)act->sum_hi : nullptr; a.osum_lo = act ? (__half *)act->sum_lo : nullptr; a.out_scale = act ? act->scale : nullptr;
    a.out = out; a.status = status; a.debug = g_prefill_debug ? g_prefill_debug + 32 * mode : nullptr;
    cudaStream_t s = (cudaStream_t)stream;
    const uint32_t f = w0->tc_format;
    if (w1 && w1->tc_format != f) return (int)cudaErrorInvalidValue;
    if (f == T_Q4_K && prefill) return mode == 0 ? launch_prefill<0>(maps, a, ctas, s) : launch_prefill<1>(maps, a, ctas, s);
    if (f == T_Q4_K) return mode == 0 ? launch_tile<T_Q4_K, 0>(maps, a, ctas, s) : launch_tile<T_Q4_K, 1>(maps, a, ctas, s);
    if (f == T_Q2_K) return mode == 0 ? launch_tile<T_Q2_K, 0>(maps, a, ctas, s) : launch_tile<T_Q2_K, 1>(maps, a, ctas, s);
    if (f == T_IQ2_XXS) return mode == 0 ? launch_tile<T_IQ2_XXS, 0>(maps, a, ctas, s) : launch_tile<T_IQ2_XXS, 1>(maps, a, ctas, s);
    if (f == T_WIDE) return mode == 0 ? launch_tile<T_WIDE, 0>(maps, a, ctas, s) : launch_tile<T_WIDE, 1>(maps, a, ctas, s);
    return (int)cudaErrorNotSupported;
}
