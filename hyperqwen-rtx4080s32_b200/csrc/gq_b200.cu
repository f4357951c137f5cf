// B200 (sm_100a) GGUF quantized-linear path: load-time repack / un-repack / dequantise kernels, the
// activation preparation, the grouped small-batch GEMV/GEMM kernel, the split-K partial sum, and the C ABI
// declared in include/gq_b200.h.
#include <cuda_runtime.h>
#include <stdio.h>
#include <stdlib.h>
#include <atomic>
#include <mutex>
#include <unordered_map>
#include "../../include/gq_b200.h"
#include "gq_decode.cuh"
#include "gq_decode8.cuh"
#include "gq_scale16.cuh"
#include <type_traits>
#include "_generated/gq_tables.h"

using namespace gq;

// ---------------------------------------------------------------------------------------------------
// host bookkeeping
// ---------------------------------------------------------------------------------------------------
static thread_local char g_cuda_err[256] = "";
static std::atomic<long long> g_launches{0};

static int cuda_fail(cudaError_t e, const char *what) {
    snprintf(g_cuda_err, sizeof g_cuda_err, "%s: %s", what, cudaGetErrorString(e));
    return GQ_ERR_CUDA;
}
#define GQ_CUDA(call)                                          \
    do {                                                       \
        cudaError_t e_ = (call);                               \
        if (e_ != cudaSuccess) return cuda_fail(e_, #call);    \
    } while (0)
#define GQ_LAUNCHED()                                                    \
    do {                                                                 \
        cudaError_t e_ = cudaGetLastError();                             \
        if (e_ != cudaSuccess) return cuda_fail(e_, "kernel launch");    \
        g_launches.fetch_add(1, std::memory_order_relaxed);              \
    } while (0)

extern "C" const char *gq_last_cuda_error(void) { return g_cuda_err; }
extern "C" int64_t gq_launch_count(void) { return (int64_t)g_launches.load(); }
extern "C" int gq_bytes_per_256(int type) { return gq_type_bytes(type); }

extern "C" int64_t gq_packed_bytes(int type, int64_t n_out, int64_t K) {
    const int B = gq_type_bytes(type);
    if (!B) return GQ_ERR_TYPE;
    if (n_out < 0 || K <= 0 || K % GQ_QK) return GQ_ERR_SHAPE;
    return ((n_out + 63) / 64) * (K / GQ_QK) * 64 * (int64_t)B;
}

extern "C" int gq_slab_map(int type, int32_t *map) {
    const int B = gq_type_bytes(type);
    if (!B) return GQ_ERR_TYPE;
    if (!map) return GQ_ERR_ARG;
    for (int p = 0; p < 16 * B; ++p) {
        int row, byte;
        if (gq_slab_src(type, p, &row, &byte)) return GQ_ERR_TYPE;
        map[p] = row * B + byte;
    }
    return GQ_OK;
}

// ---------------------------------------------------------------------------------------------------
// un-repack: one CTA per (16-row slab, k-block); the slab's raw image goes through shared memory
// ---------------------------------------------------------------------------------------------------
#define GQ_MAX_SLAB (16 * 272)

// fills img[16][B] (raw order) from a packed slab
__device__ __forceinline__ void slab_to_raw_image(int type, int B, const uint8_t *__restrict__ src, uint8_t *img) {
    for (int w = threadIdx.x; w < 4 * B; w += blockDim.x) {
        const uint32_t v = reinterpret_cast<const uint32_t *>(src)[w];
#pragma unroll
        for (int z = 0; z < 4; ++z) {
            int row, byte;
            gq_slab_src(type, 4 * w + z, &row, &byte);
            img[row * B + byte] = (uint8_t)(v >> (8 * z));
        }
    }
}

__global__ void __launch_bounds__(256) unrepack_kernel(int type, int B, const uint8_t *__restrict__ tiles, int64_t n_out, int nb,
                                                       uint8_t *__restrict__ raw, int64_t row_stride) {
    __shared__ __align__(16) uint8_t img[GQ_MAX_SLAB];
    const int slab = blockIdx.x, kb = blockIdx.y;
    const uint8_t *src = tiles + (((int64_t)(slab >> 2) * nb + kb) * 4 + (slab & 3)) * (int64_t)(16 * B);
    slab_to_raw_image(type, B, src, img);
    __syncthreads();
    const int64_t row0 = (int64_t)slab * 16;
    for (int i = threadIdx.x; i < 16 * B; i += 256) {
        const int r = i / B, b = i - r * B;
        if (row0 + r < n_out) raw[(row0 + r) * row_stride + (int64_t)kb * B + b] = img[i];
    }
}

// The codebook grids live in global memory, not in constant memory: the kernels copy them into shared memory with one
// index per thread, which the constant cache would serve one address at a time.
__device__ uint32_t c_iq3s_grid[512];
__device__ uint32_t c_iq3xxs_grid[256];
__device__ uint32_t c_iq2xxs_grid[512], c_iq2xs_grid[1024], c_iq2s_grid[2048];    // two words per entry
__device__ uint32_t c_iq1_grid[4096];      // two words per entry, a byte is 8 g + 16
__constant__ int8_t c_iq4_kvalues[16];

// A bounded wait that runs out is reported twice: in the status word of the launch's workspace (gq_read_status) and in
// this per-device word, which keeps the largest code seen since it was last read (gq_device_status) — a caller that
// drops its workspace after every call, or has none to read (the no-allocation entry point), still learns of it.
__device__ int g_sticky_status;
__device__ __forceinline__ void report_status(int *status, int code) {
    atomicExch(status, code);
    atomicMax(&g_sticky_status, code);
}
// time limit of the waits on data from another GPU (the fused and the separate all-reduce), nanoseconds
static std::atomic<unsigned long long> g_peer_wait_ns{GQ_WAIT_LIMIT_NS};

#include "gq_load.cuh"
#include "gq_prefill.cuh"

struct Workspace {
    int *status;
    uint8_t *xt;      // [nb] tiles of the prepared activations of one k-block (gq_x_tile_bytes)
    float *partials;  // [S][M][n_total]
};

__host__ __device__ inline int64_t align256(int64_t v) { return (v + 255) & ~(int64_t)255; }

// One batch row of one k-block of the staged activation tile, in the form that the kernel multiplies: 512 bytes of activations, then the
// sixteen 16-weight run sums as fp16 hi and lo parts (64 bytes).  576 = 64 mod 128, so the two rows a quarter-warp reads with one 16-byte
// load each sit in different banks.  After the rows of a k-block come their scales (fp32, one per batch row, padded to a multiple of 16
// bytes): what the products have to be multiplied by.
//
// fp16 form (above GQ_GEMV8_MAX_ROWS rows): x * 2^e as fp16, e chosen per row and k-block so that the largest magnitude lands in
// [512, 1024).  16-byte unit 4*P + t holds, of run pair (2P, 2P + 1), the quads 4t..4t+3: one load serves two MMAs.  The sums: unit t
// holds the hi parts of runs 4t..4t+3, then their lo parts.
//
// Integer form (up to GQ_GEMV8_MAX_ROWS rows): the activations as 16-bit
// fixed point (x * 2^e, e chosen per row and k-block so that the largest magnitude lands in [2^14, 2^15)), split into
// two signed bytes, x = 256 hi - lo (with the minus sign they hold -32895 .. 32640, both signs of 255 * 2^7, the largest 8-bit
// significand at that scale; 256 hi + lo ends at 32639): a plane of high bytes (256 B) and one of low bytes (256 B), then the sixteen 16-weight run sums
// (times 2^-6) as fp16 hi parts (32 B) and lo parts (32 B).  Inside a plane the bytes are ordered for the lane that
// reads them: 16-byte unit 4*i + t holds, for runs 4i..4i+3, the quad 4t..4t+3 with bytes in the order (0,2,1,3).
#define GQ_PRE_NONE 0
#define GQ_PRE_SILU_MUL 1
#define GQ_PRE_ADD_RMSNORM 2
#define GQ_X_ROW 576
#define GQ_X_SUMS 512
#ifndef GQ_GEMV8_MAX_ROWS
#define GQ_GEMV8_MAX_ROWS 16      // up to here the integer form runs; above it the fp16 form
#endif

__host__ __device__ inline int gq_x_tile_bytes(int M) { return M * GQ_X_ROW + ((4 * M + 15) & ~15); }

static int64_t ws_layout(int64_t M, int64_t K, int64_t n_total, int split, void *base, Workspace *ws) {
    int64_t off = 256;
    const int64_t o_xt = off; off = align256(off + (K / GQ_QK) * gq_x_tile_bytes((int)M));
    const int64_t o_p = off; if (split > 1) off = align256(off + (int64_t)split * M * n_total * 4);
    if (ws && base) {
        uint8_t *b = (uint8_t *)base;
        ws->status = (int *)b; ws->xt = b + o_xt; ws->partials = (float *)(b + o_p);
    }
    return off;
}

// ---------------------------------------------------------------------------------------------------
// activation preparation: one warp per (batch row, k-block).  The 256 activations become 16-bit fixed point (integer form: exact for every
// value within 2^-7 of the block's largest magnitude, rounded to 2^-16 of it below) or fp16 (fp16 form: exact within 2^-26 of it) at a
// power-of-two scale of their own, stored with the run sums and the scale as described at GQ_X_ROW.  Plays the role of the reference's quantize_activations_256
// (gguf-plugin/gluon/tiles_grouped.py:110-139), which keeps 8 bits per activation; this keeps 16.
// ---------------------------------------------------------------------------------------------------
#define GQ_PREP_WARPS 8

// The op in front of a linear layer, folded into its activation preparation: what vLLM runs as a kernel of its own
// between two linears reads its input here, on the way into the fixed-point planes, instead of writing a bf16 tensor
// that the preparation reads back.  The arithmetic repeats the unfused kernels' (bf16 wherever they round to bf16).
//   GQ_PRE_SILU_MUL     x = silu(gate) * up with gate = in[:, :K], up = in[:, K:2K]: vLLM's silu_and_mul in front of
//                       down_proj
//   GQ_PRE_ADD_RMSNORM  z = in + residual (stored to residual_out), x = z * rsqrt(mean(z^2) + eps) * weight: vLLM's
//                       fused_add_rms_norm in front of qkv_proj / gate_up_proj; without a residual, plain RMSNorm
// (The reference serves the model with the unfused ops of stock vLLM; its own fusion is the kernel's batching of
// shards, gguf-plugin/gluon/tiles_grouped.py:1204-1313.)
struct PreOp {
    int kind, K;
    const __nv_bfloat16 *weight;          // [K]
    const __nv_bfloat16 *residual;        // [M, ld_res] or null
    __nv_bfloat16 *residual_out;          // [M, ld_res], written when residual is given; never the same memory
    int64_t ld_res;
    float eps;
};

__device__ __forceinline__ void load8(const __nv_bfloat16 *p, float (&v)[8]) {
    if ((reinterpret_cast<uintptr_t>(p) & 15) == 0) {
        const uint4 raw = __ldg(reinterpret_cast<const uint4 *>(p));
        const __nv_bfloat162 *b = reinterpret_cast<const __nv_bfloat162 *>(&raw);
#pragma unroll
        for (int j = 0; j < 4; ++j) { const float2 f = __bfloat1622float2(b[j]); v[2 * j] = f.x; v[2 * j + 1] = f.y; }
    } else {
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] = __bfloat162float(p[j]);
    }
}
__device__ __forceinline__ float bf16_round(float f) { return __bfloat162float(__float2bfloat16_rn(f)); }

// one warp: the 256 activations of batch row m, k-block kb (8 per lane, consecutive) -> planes, run sums, scale
__device__ __forceinline__ void prep8_store(const float (&v)[8], int kb, int m, int M, uint8_t *__restrict__ xt, int lane) {
    float amax = 0.0f;
#pragma unroll
    for (int j = 0; j < 8; ++j) amax = fmaxf(amax, fabsf(v[j]));
    bool bad = false;
#pragma unroll
    for (int j = 0; j < 8; ++j) bad |= !(fabsf(v[j]) <= 3.0e38f);      // NaN or infinity
#pragma unroll
    for (int o = 16; o; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
    bad = __any_sync(0xffffffffu, bad);
    // scale = 2^(14 - e) with 2^e <= amax < 2^(e+1); a zero block keeps scale 1; a block holding a NaN or an infinity
    // gets a NaN scale, so that every output of that batch row is NaN as it would be in floating point
    int e = 14;
    if (amax > 0.0f) { e = (int)((__float_as_uint(amax) >> 23) & 0xFF) - 127; if (e < -100) e = -100; }
    const float scale = __uint_as_float((uint32_t)(127 + 14 - e) << 23);
    const float inv = bad ? __uint_as_float(0x7fc00000u) : __uint_as_float((uint32_t)(127 - 14 + e) << 23);
    int xi[8], sum = 0;
#pragma unroll
    for (int j = 0; j < 8; ++j) { xi[j] = bad ? 0 : __float2int_rn(v[j] * scale); sum += xi[j]; }
    uint8_t *row = xt + (int64_t)kb * gq_x_tile_bytes(M) + (int64_t)m * GQ_X_ROW;
    // this lane holds quads 2*(lane & 1) and 2*(lane & 1) + 1 of run lane >> 1
    const int r = lane >> 1, tq = 2 * (lane & 1);
#pragma unroll
    for (int qd = 0; qd < 2; ++qd) {
        const int *q = xi + 4 * qd;
        uint32_t h4[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) h4[j] = (uint32_t)((q[j] + 127) >> 8) & 0xFFu;
        const uint32_t hi = h4[0] | (h4[2] << 8) | (h4[1] << 16) | (h4[3] << 24);
        const uint32_t lo = ((uint32_t)-q[0] & 0xFFu) | (((uint32_t)-q[2] & 0xFFu) << 8) | (((uint32_t)-q[1] & 0xFFu) << 16) | (((uint32_t)-q[3] & 0xFFu) << 24);
        const int off = 64 * (r >> 2) + 16 * (tq + qd) + 4 * (r & 3);
        *reinterpret_cast<uint32_t *>(row + off) = hi;
        *reinterpret_cast<uint32_t *>(row + 256 + off) = lo;
    }
    sum += __shfl_xor_sync(0xffffffffu, sum, 1);
    if (!(lane & 1)) {
        const float f = (float)sum * 0.015625f;          // exact: |sum| < 2^20
        const __half hi = __float2half_rn(f);
        const __half lo = __float2half_rn(f - __half2float(hi));
        __half *so = reinterpret_cast<__half *>(row + GQ_X_SUMS);
        so[r] = hi;
        so[16 + r] = lo;
    }
    if (lane == 0) *reinterpret_cast<float *>(xt + (int64_t)kb * gq_x_tile_bytes(M) + (int64_t)M * GQ_X_ROW + 4 * m) = inv;
}

// the same into the fp16 form
__device__ __forceinline__ void prep16_store(const float (&v)[8], int kb, int m, int M, uint8_t *__restrict__ xt, int lane) {
    float amax = 0.0f;
#pragma unroll
    for (int j = 0; j < 8; ++j) amax = fmaxf(amax, fabsf(v[j]));
#pragma unroll
    for (int o = 16; o; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
    // scale = 2^(9 - e) with 2^e <= amax < 2^(e+1); a zero block and one holding an infinity keep scale 1: its infinities and NaNs (which
    // fmaxf passes over) reach the products as such
    int e = 9;
    if (amax > 0.0f && amax < 3.0e38f) { e = (int)((__float_as_uint(amax) >> 23) & 0xFF) - 127; if (e < -100) e = -100; }
    const float scale = __uint_as_float((uint32_t)(127 + 9 - e) << 23);
    uint32_t o[4];
    float sum = 0.0f;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const __half2 h = __floats2half2_rn(v[2 * j] * scale, v[2 * j + 1] * scale);
        o[j] = h2_as_u32(h);
        sum += __low2float(h) + __high2float(h);
    }
    uint8_t *row = xt + (int64_t)kb * gq_x_tile_bytes(M) + (int64_t)m * GQ_X_ROW;
    const int r = lane >> 1, tq = 2 * (lane & 1);            // this lane holds quads tq and tq + 1 of run r
    uint8_t *dst = row + 64 * (r >> 1) + 16 * tq + 8 * (r & 1);
    *reinterpret_cast<uint2 *>(dst) = make_uint2(o[0], o[1]);
    *reinterpret_cast<uint2 *>(dst + 16) = make_uint2(o[2], o[3]);
    sum += __shfl_xor_sync(0xffffffffu, sum, 1);
    if (!(lane & 1)) {
        const __half hi = __float2half_rn(sum);
        __half *so = reinterpret_cast<__half *>(row + GQ_X_SUMS + 16 * (r >> 2) + 2 * (r & 3));
        so[0] = hi;
        so[4] = __float2half_rn(sum - __half2float(hi));
    }
    if (lane == 0) *reinterpret_cast<float *>(xt + (int64_t)kb * gq_x_tile_bytes(M) + (int64_t)M * GQ_X_ROW + 4 * m) = __uint_as_float((uint32_t)(127 - 9 + e) << 23);
}
template <int FORM>
__device__ __forceinline__ void prep_store(const float (&v)[8], int kb, int m, int M, uint8_t *__restrict__ xt, int lane) {
    if constexpr (FORM) prep8_store(v, kb, m, M, xt, lane);
    else prep16_store(v, kb, m, M, xt, lane);
}

template <int PRE, int FORM>
__global__ void __launch_bounds__(32 * GQ_PREP_WARPS) prep_x_kernel(const __nv_bfloat16 *__restrict__ x, int64_t ldx, int M, uint8_t *__restrict__ xt,
                                                                      int *status, const PreOp pre) {
    const int lane = threadIdx.x & 31, kb = blockIdx.x;
    const int m = blockIdx.y * GQ_PREP_WARPS + (threadIdx.x >> 5);
    pdl_trigger();    // the grouped kernel behind this one may start fetching weights
    pdl_wait();       // whatever ran before (possibly still reading this workspace) has finished
    if (blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0) *status = 0;
    if (m >= M) return;
    const __nv_bfloat16 *xr = x + (int64_t)m * ldx + (int64_t)kb * GQ_QK + 8 * lane;
    float v[8];
    load8(xr, v);
    if constexpr (PRE == GQ_PRE_SILU_MUL) {
        float u[8];
        load8(xr + pre.K, u);
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] = bf16_round(bf16_round(v[j] / (1.0f + expf(-v[j]))) * u[j]);
    }
    prep_store<FORM>(v, kb, m, M, xt, lane);
}

// eight bf16 values as they are, wherever they start (CONST: nothing writes them while the kernel runs)
template <bool CONST = true>
__device__ __forceinline__ uint4 load8_raw(const __nv_bfloat16 *p) {
    if ((reinterpret_cast<uintptr_t>(p) & 15) == 0) return CONST ? __ldg(reinterpret_cast<const uint4 *>(p)) : *reinterpret_cast<const uint4 *>(p);
    const unsigned short *h = reinterpret_cast<const unsigned short *>(p);
    return make_uint4(h[0] | (uint32_t)h[1] << 16, h[2] | (uint32_t)h[3] << 16, h[4] | (uint32_t)h[5] << 16, h[6] | (uint32_t)h[7] << 16);
}
__device__ __forceinline__ void unpack8(const uint4 &raw, float (&v)[8]) {
    const uint32_t r[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) { v[2 * j] = __uint_as_float(r[j] << 16); v[2 * j + 1] = __uint_as_float(r[j] & 0xffff0000u); }
}
__device__ __forceinline__ uint32_t pack2(float a, float b) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<const uint32_t *>(&v);
}
__device__ __forceinline__ uint4 pack8(const float (&v)[8]) { return make_uint4(pack2(v[0], v[1]), pack2(v[2], v[3]), pack2(v[4], v[5]), pack2(v[6], v[7])); }
__device__ __forceinline__ void store8_raw(__nv_bfloat16 *p, const uint4 &o) {
    if ((reinterpret_cast<uintptr_t>(p) & 15) == 0) {
        *reinterpret_cast<uint4 *>(p) = o;
    } else {
        unsigned short *h = reinterpret_cast<unsigned short *>(p);
        const uint32_t r[4] = {o.x, o.y, o.z, o.w};
#pragma unroll
        for (int j = 0; j < 4; ++j) { h[2 * j] = (unsigned short)r[j]; h[2 * j + 1] = (unsigned short)(r[j] >> 16); }
    }
}

// RMSNorm (with the residual add) in front of the layer, one CTA per batch row: x, residual and weight are requested together and stay in registers,
// as bf16, between the sum of squares and the scaling, two k-blocks to a warp (of rows beyond 64 k-blocks the rest is read again).
// PREP: into the integer form's workspace (up to GQ_GEMV8_MAX_ROWS rows); else as bf16 to `out`.  A warp to a k-block where they last, two k-blocks
// to a warp where there are more rows than SMs.  Bound by its latency chain at few rows (one trip to memory, two reductions, the stores), at many by
// waiting for memory with six CTAs to an SM (2,048 rows of 5,120: 84 MB in 19.6 us from a cold cache).  With a CTA to eight k-blocks that each
// summed the whole row and read its own part again, 13 rows of 5,120 took 0.5 to 1 us longer; torch's operations at 24 rows take 32 us more than this,
// at 2,048 rows 80 to 100.
// A thread reads and writes the same columns of its row, each before it writes it, so that the new residual may take the old one's place; the
// entry point of the op by itself accepts that (the folded call never did).
#define GQ_NORM_MAX_WARPS 32
#define GQ_NORM_KEEP 2
template <bool PREP>
__global__ void __launch_bounds__(32 * GQ_NORM_MAX_WARPS) norm_rows_kernel(const __nv_bfloat16 *__restrict__ x, int64_t ldx, int M, uint8_t *__restrict__ xt, int *status,
                                                                           __nv_bfloat16 *__restrict__ out, int64_t ldo, const PreOp pre) {
    __shared__ float red[GQ_NORM_MAX_WARPS];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5, m = blockIdx.x, nb = pre.K / GQ_QK;
    pdl_trigger();
    pdl_wait();
    if (PREP && blockIdx.x == 0 && threadIdx.x == 0) *status = 0;
    const __nv_bfloat16 *row = x + (int64_t)m * ldx;
    const __nv_bfloat16 *res = pre.residual ? pre.residual + (int64_t)m * pre.ld_res : nullptr;
    // the k-block's values after the add, rounded to bf16
    const auto load = [&](int kb) {
        const int64_t col = (int64_t)kb * GQ_QK + 8 * lane;
        uint4 z = load8_raw(row + col);
        if (res) {
            float a[8], r[8];
            unpack8(load8_raw<PREP>(res + col), r);
            unpack8(z, a);
#pragma unroll
            for (int j = 0; j < 8; ++j) a[j] += r[j];
            z = pack8(a);
        }
        return z;
    };
    const auto squares = [](const uint4 &z, float s) {
        float a[8];
        unpack8(z, a);
#pragma unroll
        for (int j = 0; j < 8; ++j) s = fmaf(a[j], a[j], s);
        return s;
    };
    const auto use = [&](int kb, const uint4 &z, float rs, const uint4 &w) {
        const int64_t col = (int64_t)kb * GQ_QK + 8 * lane;
        if (res) store8_raw(pre.residual_out + (int64_t)m * pre.ld_res + col, z);
        float v[8], u[8];
        unpack8(z, v);
        unpack8(w, u);
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] = bf16_round(v[j] * rs) * u[j];
        if constexpr (PREP) {
#pragma unroll
            for (int j = 0; j < 8; ++j) v[j] = bf16_round(v[j]);
            prep8_store(v, kb, m, M, xt, lane);
        } else {
            store8_raw(out + (int64_t)m * ldo + col, pack8(v));
        }
    };
    uint4 z[GQ_NORM_KEEP], w[GQ_NORM_KEEP];
#pragma unroll
    for (int i = 0; i < GQ_NORM_KEEP; ++i) {
        const int kb = warp + i * warps;
        z[i] = w[i] = make_uint4(0u, 0u, 0u, 0u);
        if (kb < nb) { z[i] = load(kb); w[i] = load8_raw(pre.weight + (int64_t)kb * GQ_QK + 8 * lane); }
    }
    float ss = 0.0f;
#pragma unroll
    for (int i = 0; i < GQ_NORM_KEEP; ++i) ss = squares(z[i], ss);
    for (int kb = warp + GQ_NORM_KEEP * warps; kb < nb; kb += warps) ss = squares(load(kb), ss);
#pragma unroll
    for (int o = 16; o; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    if (lane == 0) red[warp] = ss;
    __syncthreads();
    ss = lane < warps ? red[lane] : 0.0f;
#pragma unroll
    for (int o = 16; o; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    const float rs = rsqrtf(ss / (float)pre.K + pre.eps);
#pragma unroll
    for (int i = 0; i < GQ_NORM_KEEP; ++i) {
        const int kb = warp + i * warps;
        if (kb < nb) use(kb, z[i], rs, w[i]);
    }
    for (int kb = warp + GQ_NORM_KEEP * warps; kb < nb; kb += warps) use(kb, load(kb), rs, load8_raw(pre.weight + (int64_t)kb * GQ_QK + 8 * lane));
}

// silu(in[:, :K]) * in[:, K:2K] as bf16, for batches whose preparation does not fold it: eight elements to a thread, at many rows bound by memory and
// its own instructions alike (2,048 rows of 5,120: 63 MB in 17.2 us, SM 62 % busy; torch's two operations: 5 us more at 24 rows of 4,352, 40 at 2,048)
__global__ void __launch_bounds__(256) silu_mul_kernel(const __nv_bfloat16 *__restrict__ x, int64_t ldx, int K, __nv_bfloat16 *__restrict__ out, int64_t ldo) {
    pdl_trigger();
    pdl_wait();
    const int c = (blockIdx.x * blockDim.x + threadIdx.x) * 8;
    if (c >= K) return;
    const __nv_bfloat16 *xr = x + (int64_t)blockIdx.y * ldx + c;
    float v[8], u[8];
    load8(xr, v);
    load8(xr + K, u);
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] = bf16_round(v[j] / (1.0f + expf(-v[j]))) * u[j];
    store8_raw(out + (int64_t)blockIdx.y * ldo + c, pack8(v));
}

// ---------------------------------------------------------------------------------------------------
// grouped small-batch kernel.  One CTA per descriptor row (64 output columns of one shard x a k-range):
// a producer warp streams the tile's k-blocks (one bulk copy each) plus the matching activation rows through
// an mbarrier ring; four consumer warps each own a 16-row slab, dequantise it in registers and run m16n8k16
// MMAs with the weights on the M side and the batch rows on the N side (8 batch rows per MMA, MT MMAs deep).
// Replaces tiles_grouped_kernel / _run (gguf-plugin/gluon/tiles_grouped.py:343-1201).
// ---------------------------------------------------------------------------------------------------
#define GQ_CONSUMER_WARPS 4
#define GQ_AR_MAX_WORLD 8

// Peer buffers of the fused multiply + all-reduce (row-parallel layers under tensor parallelism).  A rank's buffer:
// [per-unit call counters u32] padded to 4096, then data: 2 sets x world slots of slot_bytes, a slot being an image
// [M][n_total / 2] of 8-byte words {two bf16 values, call number} of one rank's partial output.  A unit is (output
// tile, consumer warp): 16 output columns of all batch rows — the grain at which ranks exchange and sum.
struct ArFused {
    int world, rank, units;          // world == 0: plain output, no exchange
    unsigned long long wait_ns;      // time limit of the wait for the peers' words
    int64_t slot_bytes;
    uint8_t *buf[GQ_AR_MAX_WORLD];
    uint32_t *counters;
};

struct GemvParams {
    const uint8_t *packed;
    const int32_t *desc;
    const uint8_t *xt;
    __nv_bfloat16 *y;
    float *partials;
    int *status;
    int M, K, nb, split, stages;
    int64_t ldy, n_total;
    int wbytes_max;      // largest tile bytes in the launch (stage stride of the weight buffers)
    int cb_bytes;                    // shared-memory bytes of the codebook-table region (0: the run has no codebook type)
    int reverse;         // 1: tiles from the last to the first
    int cluster;         // 1: the `split` CTAs of a tile form a thread-block cluster and reduce through shared memory
    int cluster_push;    // 1: the others store their accumulators into slots of the split-0 CTA's shared memory (one cluster barrier)
    const __nv_bfloat16 *x;  // FORM 2, one row: the activations themselves, converted by the producer warp (null: xt is prepared)
    const uint8_t *pf_ptr;   // weights the caller will multiply next (or null): prefetched into L2 while this launch computes
    int64_t pf_bytes;
    ArFused ar;
};

template <int I, int N, typename F>
__device__ __forceinline__ void static_for(F &&f) {
    if constexpr (I < N) {
        f(std::integral_constant<int, I>{});
        static_for<I + 1, N>(f);
    }
}

// The stage ring of one CTA: per stage the weight tile of one k-block and the matching activation tile, filled by two
// bulk copies that complete on the stage's "full" mbarrier; the four consumer warps hand a stage back through its
// "empty" mbarrier, on which the producer warp waits before it refills the stage.  (Letting the last consumer warp to
// finish a stage issue the refill itself — no producer warp, nobody polling — was measured 15 % slower: the arrival
// whose returned state tells a warp that it is the last one, and the copy issue behind it, then sit on the consumer's
// critical path every k-block.)
struct Ring {
    uint8_t *smem;
    uint64_t *full, *empty;
    int stages, stage_bytes, wmax, nk;
    const uint32_t *ar_counter;      // fused all-reduce: this warp's call counter (null: none), read early into ar_prev
};

// Fused all-reduce: lane 0 reads the warp's call counter as soon as the first stage is full — that stage holds
// activations, so every launch in front of this one has finished and the counter is final — and the load's latency
// passes during the multiplication instead of at the start of the exchange.  (The loop below waits on the same phase
// again, which then returns at once.)
__device__ __forceinline__ bool ring_read_counter(const Ring &r, int lane, uint32_t &ar_prev) {
    if (!r.ar_counter) return true;
    if (!mbar_wait(r.full, 0)) return false;
    if (lane == 0) ar_prev = *reinterpret_cast<const volatile uint32_t *>(r.ar_counter);
    return true;
}

// ---- integer form (1..16 batch rows): mma.sync m16n8k32 / m16n8k16 on 8-bit operands ----------------------
// D (int32, 16 x 8) = A (16 weight rows x 32 k, 8-bit) . B (32 k x 8 columns, signed 8-bit) [+ C].  AS: A is signed.
template <bool AS>
__device__ __forceinline__ void imma32(int (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1, int c0, int c1, int c2, int c3) {
    if constexpr (AS)
        asm volatile("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%11,%12,%13};"
                     : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "r"(c0), "r"(c1), "r"(c2), "r"(c3));
    else
        asm volatile("mma.sync.aligned.m16n8k32.row.col.s32.u8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%11,%12,%13};"
                     : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "r"(c0), "r"(c1), "r"(c2), "r"(c3));
}
template <bool AS>
__device__ __forceinline__ void imma16(int (&d)[4], const uint32_t (&a)[2], uint32_t b0) {
    if constexpr (AS)
        asm volatile("mma.sync.aligned.m16n8k16.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%7,%7,%7,%7};"
                     : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3]) : "r"(a[0]), "r"(a[1]), "r"(b0), "r"(0));
    else
        asm volatile("mma.sync.aligned.m16n8k16.row.col.s32.u8.s8.s32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%7,%7,%7,%7};"
                     : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3]) : "r"(a[0]), "r"(a[1]), "r"(b0), "r"(0));
}

// one k-block of one slab in the integer form.  `xs` is the staged activation tile of the k-block (rows of GQ_X_ROW
// bytes, then the batch rows' scales at xs_off).  Per MMA the weights are 8-bit integers and the activations one of the
// two byte planes (x = 256 hi - lo); int32 sums per plane are exact.  At the end of the
// k-block:  acc += 2^-e[n] * ( d[row] * (256 sumH - sumL) - f[row] * 64 * sum_run A''[row][run] * Sx[run][n] ).
// ST (1..4 batch rows): the two planes sit side by side on the MMA's eight columns, the high bytes of row n in column n and the low
// bytes in column n + 4, so that one MMA and one set of scale multiplications serve both; the factors 256 and -1 and the sum of the two
// columns come at the end.
template <int TYPE, int MT, bool ST>
__device__ __forceinline__ void slab_kblock8(const uint8_t *slab, const uint8_t *xs, int xs_off, const DecAux8 &aux, int lane, float (&acc)[MT][4]) {
    using D = Dec8<TYPE>;
    constexpr bool AS = D::A_SIGNED;
    D dec;
    dec.load(slab, lane, aux);
    const int g = lane >> 2, t = lane & 3;
    // unit (i, t) of batch row g; + 8 nt rows, + 256 for the low plane
    const uint8_t *xb = ST ? xs + (g & 3) * GQ_X_ROW + 256 * (g >> 2) + 16 * t : xs + g * GQ_X_ROW + 16 * t;
    int aH[MT][4], aL[MT][4], bH[MT][4], bL[MT][4];
    float bf[MT][4];
#pragma unroll
    for (int nt = 0; nt < MT; ++nt)
#pragma unroll
        for (int j = 0; j < 4; ++j) { aH[nt][j] = 0; aL[nt][j] = 0; bH[nt][j] = 0; bL[nt][j] = 0; bf[nt][j] = 0.f; }
    static_for<0, 4>([&](auto i_) {
        constexpr int I = decltype(i_)::value;
        uint4 xh[MT], xl[MT];
#pragma unroll
        for (int nt = 0; nt < MT; ++nt) {
            xh[nt] = ld16(xb + nt * 8 * GQ_X_ROW + 64 * I);
            if constexpr (!ST) xl[nt] = ld16(xb + nt * 8 * GQ_X_ROW + 64 * I + 256);
        }
        if constexpr (D::SCHEME == GQ_S16) {
            static_for<0, 4>([&](auto r_) {
                constexpr int RR = decltype(r_)::value, R = 4 * I + RR;
                uint32_t a[2];
                dec.template step16<R>(a);
                int s0, s1;
                dec.template iscale16<R>(s0, s1);
#pragma unroll
                for (int nt = 0; nt < MT; ++nt) {
                    int th[4], tl[4];
                    imma16<AS>(th, a, w4(xh[nt], RR));
                    aH[nt][0] += s0 * th[0]; aH[nt][1] += s0 * th[1]; aH[nt][2] += s1 * th[2]; aH[nt][3] += s1 * th[3];
                    if constexpr (!ST) {
                        imma16<AS>(tl, a, w4(xl[nt], RR));
                        aL[nt][0] += s0 * tl[0]; aL[nt][1] += s0 * tl[1]; aL[nt][2] += s1 * tl[2]; aL[nt][3] += s1 * tl[3];
                    }
                }
            });
        } else {
            static_for<0, 2>([&](auto v_) {
                constexpr int V = decltype(v_)::value, S = 2 * I + V;
                uint32_t a[4];
                dec.template step<S>(a);
                int s0 = 1, s1 = 1;
                float f0 = 1.f, f1 = 1.f;
                if constexpr (D::SCHEME == GQ_S32) dec.template iscale<S>(s0, s1);
                if constexpr (D::SCHEME == GQ_F32) dec.template fscale<S>(f0, f1);
#pragma unroll
                for (int nt = 0; nt < MT; ++nt) {
                    const uint32_t bh0 = V ? xh[nt].z : xh[nt].x, bh1 = V ? xh[nt].w : xh[nt].y;
                    const uint32_t bl0 = ST ? 0u : V ? xl[nt].z : xl[nt].x, bl1 = ST ? 0u : V ? xl[nt].w : xl[nt].y;
                    if constexpr (D::SCHEME == GQ_FOLD) {
                        // two accumulator chains per plane (even / odd k-steps): half the dependent MMAs in a row
                        if constexpr (V == 0) {
                            imma32<AS>(aH[nt], a, bh0, bh1, aH[nt][0], aH[nt][1], aH[nt][2], aH[nt][3]);
                            if constexpr (!ST) imma32<AS>(aL[nt], a, bl0, bl1, aL[nt][0], aL[nt][1], aL[nt][2], aL[nt][3]);
                        } else {
                            imma32<AS>(bH[nt], a, bh0, bh1, bH[nt][0], bH[nt][1], bH[nt][2], bH[nt][3]);
                            if constexpr (!ST) imma32<AS>(bL[nt], a, bl0, bl1, bL[nt][0], bL[nt][1], bL[nt][2], bL[nt][3]);
                        }
                    } else {
                        int th[4], tl[4];
                        imma32<AS>(th, a, bh0, bh1, 0, 0, 0, 0);
                        if constexpr (!ST) imma32<AS>(tl, a, bl0, bl1, 0, 0, 0, 0);
                        if constexpr (D::SCHEME == GQ_S32) {
                            aH[nt][0] += s0 * th[0]; aH[nt][1] += s0 * th[1]; aH[nt][2] += s1 * th[2]; aH[nt][3] += s1 * th[3];
                            if constexpr (!ST) { aL[nt][0] += s0 * tl[0]; aL[nt][1] += s0 * tl[1]; aL[nt][2] += s1 * tl[2]; aL[nt][3] += s1 * tl[3]; }
                        } else if constexpr (ST) {
                            bf[nt][0] = fmaf(f0, (float)th[0], bf[nt][0]);
                            bf[nt][1] = fmaf(f0, (float)th[1], bf[nt][1]);
                            bf[nt][2] = fmaf(f1, (float)th[2], bf[nt][2]);
                            bf[nt][3] = fmaf(f1, (float)th[3], bf[nt][3]);
                        } else {
                            bf[nt][0] = fmaf(f0, (float)(th[0] * 256 - tl[0]), bf[nt][0]);
                            bf[nt][1] = fmaf(f0, (float)(th[1] * 256 - tl[1]), bf[nt][1]);
                            bf[nt][2] = fmaf(f1, (float)(th[2] * 256 - tl[2]), bf[nt][2]);
                            bf[nt][3] = fmaf(f1, (float)(th[3] * 256 - tl[3]), bf[nt][3]);
                        }
                    }
                }
            });
        }
    });
    float d0, d1;
    dec.kscale(d0, d1);
    uint32_t ac[4] = {0u, 0u, 0u, 0u};
    float fc[2] = {0.f, 0.f};
    if constexpr (D::NCORR > 0) {
        dec.corr(ac, fc);
        fc[0] *= -64.0f; fc[1] *= -64.0f;
    }
    const float z[4] = {0.f, 0.f, 0.f, 0.f};
    const float plane = t < 2 ? 256.0f : -1.0f;          // ST: lanes t < 2 hold columns 0 .. 3
#pragma unroll
    for (int nt = 0; nt < MT; ++nt) {
        float tot[4];
        if constexpr (D::SCHEME == GQ_F32) {
#pragma unroll
            for (int j = 0; j < 4; ++j) tot[j] = ST ? plane * bf[nt][j] : bf[nt][j];
        } else {
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                if constexpr (D::SCHEME == GQ_FOLD) {
                    // the even and the odd k-steps together: below 2^24 (128 weights of at most 180, and 4 * 45, times 255), exact as float
                    const int h = (aH[nt][j] << D::ODD_SHIFT) + bH[nt][j], l = (aL[nt][j] << D::ODD_SHIFT) + bL[nt][j];
                    tot[j] = (j < 2 ? d0 : d1) * ((ST ? plane * (float)h : fmaf((float)h, 256.0f, -(float)l)) * (1.0f / (1 << D::ODD_SHIFT)));
                } else {
                    tot[j] = (j < 2 ? d0 : d1) * (ST ? plane * (float)aH[nt][j] : fmaf((float)aH[nt][j], 256.0f, -(float)aL[nt][j]));
                }
            }
        }
        if constexpr (D::NCORR > 0) {
            float mm[4];
            if constexpr (ST) {
                const uint2 b = *reinterpret_cast<const uint2 *>(xs + (g & 3) * GQ_X_ROW + GQ_X_SUMS + 32 * (g >> 2) + 8 * t);
                mma16816_z(mm, ac, b.x, b.y, z);
            } else {
                const uint8_t *sb = xs + (nt * 8 + g) * GQ_X_ROW + GQ_X_SUMS + 8 * t;
                const uint2 bh = *reinterpret_cast<const uint2 *>(sb);
                const uint2 bl = *reinterpret_cast<const uint2 *>(sb + 32);
                mma16816_z(mm, ac, bh.x, bh.y, z);
                mma16816(mm, ac, bl.x, bl.y);
            }
#pragma unroll
            for (int j = 0; j < 4; ++j) tot[j] = fmaf(fc[j >> 1], mm[j], tot[j]);
        }
        const float2 sx = *reinterpret_cast<const float2 *>(xs + xs_off + (ST ? (2 * t) & 3 : nt * 8 + 2 * t) * 4);
        acc[nt][0] = fmaf(sx.x, tot[0], acc[nt][0]);
        acc[nt][1] = fmaf(sx.y, tot[1], acc[nt][1]);
        acc[nt][2] = fmaf(sx.x, tot[2], acc[nt][2]);
        acc[nt][3] = fmaf(sx.y, tot[3], acc[nt][3]);
    }
}


// the consumer loop of one warp for a CTA whose shard is of TYPE: waits for each stage, processes its slab,
// releases the stage.  Returns false if a bounded wait ran out.
template <int TYPE, int MT, bool ST>
__device__ __forceinline__ bool consume8(const Ring &r, int xs_off, int slab_off, const DecAux8 &aux, int lane, float (&acc)[MT][4], uint32_t &ar_prev) {
    if (!ring_read_counter(r, lane, ar_prev)) return false;
    for (int i = 0, s = 0, round = 0; i < r.nk; ++i) {
        if (!mbar_wait(r.full + s, round & 1)) return false;
        const uint8_t *st = r.smem + (size_t)s * r.stage_bytes;
        slab_kblock8<TYPE, MT, ST>(st + slab_off, st + r.wmax, xs_off, aux, lane, acc);
        __syncwarp();
        if (lane == 0) mbar_arrive(r.empty + s);
        if (++s == r.stages) { s = 0; ++round; }
    }
    return true;
}

// One warp's share of the fused all-reduce.  `blk` (shared memory) holds the warp's bf16 block [M][16] of this
// rank's partial output (columns col .. col + ncols - 1 of every batch row; col and ncols even).  Push based, one
// shot, and free of fences: every pair of bf16 values travels as one 8-byte word {values, call number}, stored
// whole (an aligned 64-bit store is single-copy atomic) into this rank's slot of every rank's buffer — plain stores
// through peer pointers, own buffer included.  The receiver polls the words of its OWN memory until their call
// number is this call's (with a time limit), adds the ranks' values in rank order in fp32 and rounds once into y:
// the data is its own flag, so no release / acquire at system scope is needed (on a busy SM those cost several
// microseconds per warp).  No loads from remote memory, no multicast.  The call number lives in device memory per
// (tile, warp) and selects one of two slot sets; a stale word of the same set carries an older number, and a rank
// cannot run two calls ahead of a peer because each call needs every peer's words of that call.
__device__ __noinline__ void fused_allreduce_block(const GemvParams &p, const uint32_t *blk, int unit, int col, int ncols, int lane, uint32_t prev) {
    const ArFused &a = p.ar;
    // the call number: one more than the counter, which lane 0 read while the first k-block was being multiplied
    const uint32_t seq = __shfl_sync(0xffffffffu, prev, 0) + 1;
    const uint32_t set = seq & 1u;
    const int M = p.M, half = ncols >> 1;
    const int64_t row_words = p.n_total >> 1, slot_words = a.slot_bytes >> 3;
    const int64_t first = (int64_t)(col >> 1);
    const int n_el = M * half;
    for (int pr = 0; pr < a.world; ++pr) {
        unsigned long long *dst = reinterpret_cast<unsigned long long *>(a.buf[pr]) + ((int64_t)set * a.world + a.rank) * slot_words + first;
        for (int e = lane; e < n_el; e += 32) {
            const int n = e / half, c2 = e - n * half;
            const unsigned long long w = (unsigned long long)blk[n * 8 + c2] | ((unsigned long long)seq << 32);
            asm volatile("st.volatile.global.u64 [%0], %1;" ::"l"(dst + n * row_words + c2), "l"(w) : "memory");
        }
    }
    const unsigned long long *src = reinterpret_cast<const unsigned long long *>(a.buf[a.rank]) + (int64_t)set * a.world * slot_words + first;
    bool fail = false;
    uint64_t t0 = 0;
    // Two elements per lane and pass; the words of all ranks for both are requested before any is looked at, so a pass
    // costs one trip to the L2 whatever the number of ranks (polled one after the other, the 2 x 8 dependent loads of an
    // 8-rank exchange took longer than the kernel in front of them).
    for (int e0 = lane; e0 < n_el; e0 += 64) {
        const int e1 = e0 + 32;
        const bool has1 = e1 < n_el;
        const int n0 = e0 / half, c0 = e0 - n0 * half, n1 = has1 ? e1 / half : n0, c1 = has1 ? e1 - n1 * half : c0;
        const unsigned long long *q0 = src + n0 * row_words + c0, *q1 = src + n1 * row_words + c1;
        unsigned long long w0[GQ_AR_MAX_WORLD], w1[GQ_AR_MAX_WORLD];
        const uint32_t all = (1u << a.world) - 1u;
        uint32_t pending = all | (has1 ? all << 8 : 0u);
        for (uint32_t it = 0; pending; ++it) {
#pragma unroll
            for (int r = 0; r < GQ_AR_MAX_WORLD; ++r) {
                if ((pending >> r) & 1u) asm volatile("ld.volatile.global.u64 %0, [%1];" : "=l"(w0[r]) : "l"(q0 + (int64_t)r * slot_words) : "memory");
                if ((pending >> (8 + r)) & 1u) asm volatile("ld.volatile.global.u64 %0, [%1];" : "=l"(w1[r]) : "l"(q1 + (int64_t)r * slot_words) : "memory");
            }
#pragma unroll
            for (int r = 0; r < GQ_AR_MAX_WORLD; ++r) {
                if (((pending >> r) & 1u) && (uint32_t)(w0[r] >> 32) == seq) pending &= ~(1u << r);
                if (((pending >> (8 + r)) & 1u) && (uint32_t)(w1[r] >> 32) == seq) pending &= ~(1u << (8 + r));
            }
            if (pending && (it & 255u) == 255u) {      // the clock is read only once a wait has become long
                const uint64_t now = global_timer_ns();
                if (t0 == 0) t0 = now;
                if (now - t0 > a.wait_ns) { fail = true; break; }
            }
        }
        if (fail) break;
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            if (k == 1 && !has1) break;
            float s0 = 0.f, s1 = 0.f;
#pragma unroll
            for (int r = 0; r < GQ_AR_MAX_WORLD; ++r) {
                if (r < a.world) {
                    const uint32_t v = (uint32_t)(k ? w1[r] : w0[r]);
                    const float2 f = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162 *>(&v));
                    s0 += f.x; s1 += f.y;
                }
            }
            __nv_bfloat16 *yp = p.y + (int64_t)(k ? n1 : n0) * p.ldy + col + 2 * (k ? c1 : c0);
            if (!(reinterpret_cast<uintptr_t>(yp) & 3)) *reinterpret_cast<__nv_bfloat162 *>(yp) = __floats2bfloat162_rn(s0, s1);
            else { yp[0] = __float2bfloat16_rn(s0); yp[1] = __float2bfloat16_rn(s1); }
        }
    }
    fail = __any_sync(0xffffffffu, fail);
    if (lane == 0) {
        if (fail) report_status(p.status, GQ_DEV_TIMEOUT);
        a.counters[unit] = seq;
    }
}

#include "gq_fp16.cuh"

// MINB = CTAs per SM the compiler must leave room for (0: its own choice).  For the M <= 8 form 4 gives it 96
// registers, which it turns into more loads and MMAs in flight per warp: measured 14 % faster than the 72-register
// build when a CTA walks ten or more k-blocks, a little slower on launches of many short CTAs, 2 % faster on the
// mixed stack.  (Compiling both and choosing per call was slower than either alone: alternating between two large
// kernels costs more in instruction-cache misses at every launch than the better fit gains.)  The fp16 form has room for two CTAs (168
// registers); three were slower up to two waves.
//
// FORM 1: activations as two byte planes, weights decoded to 8-bit quads, m16n8k32 / m16n8k16 integer MMAs: about half the
// instructions per weight of the fp16 form.  (At 9..16 rows the fp16 form is faster where a run is scaled per 16 weights, slower elsewhere:
// 2 x 17,408 x 5,120 at 16 rows, integer / fp16, IQ3_S + Q2_K 41.9 / 37.3 us, Q3_K + IQ3_S 39.8 / 41.7, IQ4_XS 41 / 47; 7,168 x 5,120
// 13.3 / 15.6.)
// FORM 2: the integer form with both planes in one MMA, used for 1..4 batch rows.
// FORM 0: activations as fp16, weights as exact fp16 integers (gq_fp16.cuh), used above GQ_GEMV8_MAX_ROWS rows.
// ONLY: 0 compiles the decoders of all types (the branch is per CTA); a GGML type id compiles that type alone,
// for launches whose shards all share it (a smaller kernel; most launches of a real model are such).
template <int MT, int FORM>
__host__ __device__ constexpr int gq_stage_xbytes() { return FORM == 2 ? 4 * GQ_X_ROW + 16 : 8 * MT * GQ_X_ROW + 32 * MT; }

template <int MT>
__host__ __device__ constexpr bool gq_red_in_ring() { return MT == 8; }

template <int MT, int MINB, int FORM, int ONLY>
__global__ void __launch_bounds__(32 * (GQ_CONSUMER_WARPS + 1), MINB) gemv_grouped_kernel(const __grid_constant__ GemvParams p) {
    extern __shared__ __align__(128) uint8_t smem[];
    // layout: [stages x (weights wbytes_max | activation tile)] [full barriers] [empty barriers] [codebook table] [reduction scratch]
    const int stages = p.stages, wmax = p.wbytes_max, M = p.M;
    constexpr int xbytes = gq_stage_xbytes<MT, FORM>();
    const int stage_bytes = wmax + xbytes;
    uint64_t *full = reinterpret_cast<uint64_t *>(smem + (size_t)stages * stage_bytes);
    uint64_t *empty = full + stages;
    uint64_t *parts = empty + stages;          // push-form split-K: per consumer warp, the other splits' sums have landed
    uint32_t *grid_s = reinterpret_cast<uint32_t *>(parts + GQ_CONSUMER_WARPS);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // the table row: the tile (and of a cluster, which is one, the part), perhaps counted from the last
    const int row = p.reverse ? (int)((gridDim.x - 1 - blockIdx.x) / (unsigned)p.split) * p.split + (int)(blockIdx.x % (unsigned)p.split) : (int)blockIdx.x;
    const int32_t *d = p.desc + (int64_t)row * GQ_DESC_WORDS;
    const int64_t off = (int64_t)d[0] * 16;
    const int type = ONLY ? ONLY : d[1];
    const int col0 = d[2], nvalid = d[3], kb0 = d[4], kb1 = d[5], split_idx = d[6];
    const int B = gq_type_bytes(type);
    const int tile_bytes = 64 * B;
    const int nk = kb1 - kb0;

    // a tile whose type contradicts the call's run_info (not the single type that this kernel is for; fp16 form: no type at all, or one of
    // wider tiles than a stage holds; a codebook type without table space): report and leave (every CTA of a cluster works on the same
    // tile, so a cluster leaves as one)
    if ((ONLY != 0 && d[1] != ONLY) || (FORM == 0 && (B == 0 || tile_bytes > wmax)) || (gq_cb_kind(type) >= 0 && gq_cb_bytes(gq_cb_kind(type)) > p.cb_bytes)) {
        if (threadIdx.x == 0) { pdl_wait(); report_status(p.status, GQ_DEV_BAD_SHAPE); }      // after the preparation kernel has cleared the word
        return;
    }
    Ring ring;
    ring.smem = smem; ring.full = full; ring.empty = empty;
    ring.stages = stages; ring.stage_bytes = stage_bytes; ring.wmax = wmax; ring.nk = nk;
    ring.ar_counter = (p.ar.world > 0 && (p.split == 1 || p.cluster) && split_idx == 0 && warp < GQ_CONSUMER_WARPS)
                          ? p.ar.counters + (int64_t)(blockIdx.x / (unsigned)p.split) * GQ_CONSUMER_WARPS + warp : nullptr;

    if (threadIdx.x == 0) {
        for (int s = 0; s < stages; ++s) { mbar_init(full + s, 1); mbar_init(empty + s, GQ_CONSUMER_WARPS); }
        if (p.cluster_push)
            for (int w = 0; w < GQ_CONSUMER_WARPS; ++w) mbar_init(parts + w, 1);
        fence_barrier_init();
    }
    __syncthreads();
    // the codebook table of this CTA's type, at the start of the table region: filled by the consumer warps while the
    // producer's first copies are already on their way, closed by a barrier among the consumers only
    if (p.cb_bytes && warp < GQ_CONSUMER_WARPS) {
        uint32_t *g32 = grid_s;
        if constexpr (FORM == 0) {
            fill_codebook(type, reinterpret_cast<uint8_t *>(grid_s), threadIdx.x, 32 * GQ_CONSUMER_WARPS);
        } else {
            if ((ONLY == 0 || ONLY == GQ_IQ3_S) && type == GQ_IQ3_S) {
                for (int i = threadIdx.x; i < 512; i += 32 * GQ_CONSUMER_WARPS) g32[i] = iq3s_grid_entry8(c_iq3s_grid[i]);
            }
            if ((ONLY == 0 || ONLY == GQ_IQ3_XXS) && type == GQ_IQ3_XXS) {
                for (int i = threadIdx.x; i < 256; i += 32 * GQ_CONSUMER_WARPS) g32[i] = iq3s_grid_entry8(c_iq3xxs_grid[i]);
            }
            if ((ONLY == 0 || ONLY == GQ_IQ2_XXS) && type == GQ_IQ2_XXS) {
                for (int i = threadIdx.x; i < 512; i += 32 * GQ_CONSUMER_WARPS) g32[i] = iq3s_grid_entry8(c_iq2xxs_grid[i]);
            }
            if ((ONLY == 0 || ONLY == GQ_IQ2_XS) && type == GQ_IQ2_XS) {
                for (int i = threadIdx.x; i < 1024; i += 32 * GQ_CONSUMER_WARPS) g32[i] = iq3s_grid_entry8(c_iq2xs_grid[i]);
            }
            if ((ONLY == 0 || ONLY == GQ_IQ2_S) && type == GQ_IQ2_S) {
                for (int i = threadIdx.x; i < 2048; i += 32 * GQ_CONSUMER_WARPS) g32[i] = iq3s_grid_entry8(c_iq2s_grid[i]);
            }
            if ((ONLY == 0 || ONLY == GQ_IQ1_M) && type == GQ_IQ1_M) {
                for (int i = threadIdx.x; i < 4096; i += 32 * GQ_CONSUMER_WARPS) g32[i] = iq3s_grid_entry8(c_iq1_grid[i]);
            }
        }
        asm volatile("bar.sync 1, %0;" ::"n"(32 * GQ_CONSUMER_WARPS) : "memory");
    }
    // push-form split-K: a CTA may store into the split-0 CTA's shared memory only once that CTA is known to run and has
    // initialised its barriers;
    // every thread enters this rendezvous here and collects it just before its first remote store (or before the
    // closing barrier), long after everyone has arrived
    const bool push = p.cluster && p.cluster_push;
    if (push) cluster_arrive_relaxed();

    if (FORM == 2 && warp == GQ_CONSUMER_WARPS && p.x) {
        // ---- producer of a small launch for one row: the whole warp.  It copies the weight tiles like the one below, and
        // converts the activations of each k-block straight into the stage (what prep_x_kernel would have left in the workspace),
        // one k-block requested ahead.  Every CTA of a k-range repeats that, 0.7 us per k-block; for it the preparation kernel falls
        // away: 2 us of host time (1024 x 5120 Q4_K, called one by one: 8.2 -> 6.4 us) and a kernel boundary on the GPU ----
        const uint8_t *src = p.packed + off + (int64_t)kb0 * tile_bytes;
        const __nv_bfloat16 *xr = p.x + (int64_t)kb0 * GQ_QK + 8 * lane;
        const int pre = nk < stages ? nk : stages;
        if (lane == 0)
            for (int i = 0; i < pre; ++i) bulk_g2s(smem + (size_t)i * stage_bytes, src + (int64_t)i * tile_bytes, (uint32_t)tile_bytes, full + i);
        pdl_wait();
        float nxt[8];
        load8(xr, nxt);
        for (int i = 0, s = 0, round = 0; i < nk; ++i) {
            if (i >= pre) {
                if (!mbar_wait_parked(empty + s, (round - 1) & 1)) { if (lane == 0) report_status(p.status, GQ_DEV_TIMEOUT); break; }
                if (lane == 0) bulk_g2s(smem + (size_t)s * stage_bytes, src + (int64_t)i * tile_bytes, (uint32_t)tile_bytes, full + s);
            }
            float v[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) v[j] = nxt[j];
            if (i + 1 < nk) load8(xr + (i + 1) * GQ_QK, nxt);
            prep8_store(v, 0, 0, 1, smem + (size_t)s * stage_bytes + wmax, lane);
            __syncwarp();
            if (lane == 0) mbar_expect_tx(full + s, (uint32_t)tile_bytes);      // arrives: the rows are there, the tile is counted
            if (i == nk - 3 || (i == 0 && nk < 3)) pdl_trigger();
            if (++s == stages) { s = 0; ++round; }
        }
        if (!p.cluster) return;
        if (push) { cluster_wait(); return; }
        cluster_sync_all();
        cluster_sync_all();
        return;
    }
    if (warp == GQ_CONSUMER_WARPS) {
        // ---- producer: one thread; per k-block one bulk copy of the weight tile and one of the activation tile.
        // The weights do not depend on the kernel in front of this one, so the first stages' weight copies go out
        // before the dependency wait; the activation tiles (written by the preparation kernel) follow it.  The
        // kernel behind this one is allowed to start launching when this CTA has two k-blocks left. ----
        if (lane == 0) {
            const uint8_t *src = p.packed + off + (int64_t)kb0 * tile_bytes;
            const uint32_t abytes = (uint32_t)gq_x_tile_bytes(M);
            const uint8_t *xsrc = p.xt + (int64_t)kb0 * abytes;
            const int pre = nk < stages ? nk : stages;
            for (int i = 0; i < pre; ++i) {
                mbar_expect_tx(full + i, (uint32_t)tile_bytes + abytes);
                bulk_g2s(smem + (size_t)i * stage_bytes, src + (int64_t)i * tile_bytes, (uint32_t)tile_bytes, full + i);
            }
            pdl_wait();
            for (int i = 0; i < pre; ++i) bulk_g2s(smem + (size_t)i * stage_bytes + wmax, xsrc + (int64_t)i * abytes, abytes, full + i);
            if (nk - pre <= 2) pdl_trigger();
            for (int i = pre, s = 0, round = 1; i < nk; ++i) {
                if (!mbar_wait_parked(empty + s, (round - 1) & 1)) { report_status(p.status, GQ_DEV_TIMEOUT); break; }
                uint8_t *st = smem + (size_t)s * stage_bytes;
                mbar_expect_tx(full + s, (uint32_t)tile_bytes + abytes);
                bulk_g2s(st, src + (int64_t)i * tile_bytes, (uint32_t)tile_bytes, full + s);
                bulk_g2s(st + wmax, xsrc + (int64_t)i * abytes, abytes, full + s);
                if (i == nk - 3) pdl_trigger();
                if (++s == stages) { s = 0; ++round; }
            }
        }
        else if (p.pf_ptr) {
            // the producer warp's other lanes: this CTA's share of the next layer's weights, 16 KB per request
            const int64_t chunk = 16384;
            const int64_t n_chunks = (p.pf_bytes + chunk - 1) / chunk;
            for (int64_t c = (int64_t)blockIdx.x * 31 + (lane - 1); c < n_chunks; c += (int64_t)gridDim.x * 31) {
                const int64_t o = c * chunk;
                const int64_t sz = (p.pf_bytes - o < chunk ? p.pf_bytes - o : chunk) & ~(int64_t)15;
                if (sz > 0) prefetch_l2_bulk(p.pf_ptr + o, (uint32_t)sz);
            }
        }
        if (!p.cluster) return;
        if (push) { cluster_wait(); return; }
        cluster_sync_all();     // the pull form's cluster barriers need every thread of every CTA
        cluster_sync_all();
        return;
    }

    // ---- consumers ----
    float acc[MT][4];
#pragma unroll
    for (int nt = 0; nt < MT; ++nt) acc[nt][0] = acc[nt][1] = acc[nt][2] = acc[nt][3] = 0.f;

    bool ok = true;
    uint32_t ar_prev = 0;
    const int slab_off = warp * 16 * B;
    const int xs_off = M * GQ_X_ROW;
#define GQ_EACH_CONSUME \
        switch (type) { \
            GQ_CONSUME(GQ_Q4_0) GQ_CONSUME(GQ_Q5_0) GQ_CONSUME(GQ_Q8_0) GQ_CONSUME(GQ_Q2_K) GQ_CONSUME(GQ_Q3_K) GQ_CONSUME(GQ_Q4_K) \
            GQ_CONSUME(GQ_Q5_K) GQ_CONSUME(GQ_Q6_K) GQ_CONSUME(GQ_IQ4_NL) GQ_CONSUME(GQ_IQ3_S) GQ_CONSUME(GQ_IQ4_XS) GQ_CONSUME(GQ_IQ3_XXS) \
            GQ_CONSUME(GQ_IQ2_XXS) GQ_CONSUME(GQ_IQ2_XS) GQ_CONSUME(GQ_IQ2_S) GQ_CONSUME(GQ_IQ1_M) \
        }
    if constexpr (FORM == 0) {
        DecAux aux;
        aux.grid = grid_s;
        aux.iq4 = iq4_table_biased();
#define GQ_CONSUME(T) case T: ok = consume<T, MT>(ring, xs_off, slab_off, aux, lane, acc, ar_prev); break;
        GQ_EACH_CONSUME
#undef GQ_CONSUME
    } else {
        DecAux8 aux;
        aux.grid = grid_s;
        // the IQ4 codebook in four registers, as signed bytes
        uint32_t tb[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            tb[j] = 0;
#pragma unroll
            for (int i = 0; i < 4; ++i) tb[j] |= (uint32_t)(uint8_t)c_iq4_kvalues[4 * j + i] << (8 * i);
        }
        aux.iq4 = {tb[0], tb[1], tb[2], tb[3]};
#define GQ_CONSUME(T) case T: ok = consume8<T, MT, FORM == 2>(ring, xs_off, slab_off, aux, lane, acc, ar_prev); break;
        if constexpr (ONLY != 0) ok = consume8<(ONLY ? ONLY : GQ_Q4_K), MT, FORM == 2>(ring, xs_off, slab_off, aux, lane, acc, ar_prev);
        else { GQ_EACH_CONSUME }
#undef GQ_CONSUME
    }
#undef GQ_EACH_CONSUME
    if constexpr (FORM == 2) {      // columns n and n + 4: lanes t and t + 2
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[0][j] += __shfl_xor_sync(0xffffffffu, acc[0][j], 2);
    }
    if (!ok && lane == 0) report_status(p.status, GQ_DEV_TIMEOUT);   // the result is then incomplete; the status word says so

    // ---- epilogue: rows of the MMA are output columns, columns of the MMA are batch rows ----
    const int g = lane >> 2, t = lane & 3;
    // scratch of its own behind the ring (a slower warp may still read the ring): GQ_CONSUMER_WARPS x MT x 512 bytes.  Of eight column tiles
    // it would cost a resident CTA, and takes the ring's place once all four warps are through.
    float4 *red = reinterpret_cast<float4 *>(gq_red_in_ring<MT>() ? smem : reinterpret_cast<uint8_t *>(grid_s) + p.cb_bytes);
    if constexpr (gq_red_in_ring<MT>()) asm volatile("bar.sync 1, %0;" ::"n"(32 * GQ_CONSUMER_WARPS) : "memory");
    if (push) {
        cluster_wait();         // the rendezvous entered at the start: every CTA of the cluster is running
        // split-K inside a cluster, push form: the warps of splits 1.. store their accumulators into their slot of the split-0
        // CTA's scratch through distributed shared memory; that CTA's warp of the same columns adds the slots from its own shared
        // memory, in split order, and writes bf16 once.  No partial sums in HBM, no second kernel, fixed order of the additions.
        // The stores are st.async, whose bytes the receiving warp's mbarrier counts: neither side needs a fence or a barrier at
        // cluster scope, and the senders leave at once.
        if (split_idx != 0) {
            const uint32_t dst = map_to_rank(smem_u32(red), 0u) + (uint32_t)((split_idx - 1) * GQ_CONSUMER_WARPS * MT * 512);
            const uint32_t bar = map_to_rank(smem_u32(parts + warp), 0u);
#pragma unroll
            for (int nt = 0; nt < MT; ++nt)
                st_async_f4(dst + (uint32_t)(((warp * MT + nt) * 32 + lane) * 16), acc[nt][0], acc[nt][1], acc[nt][2], acc[nt][3], bar);
            return;
        }
        if (lane == 0) mbar_expect_tx(parts + warp, (uint32_t)((p.split - 1) * MT * 512));
        __syncwarp();
        if (!__all_sync(0xffffffffu, mbar_wait(parts + warp, 0))) {
            // A part is late.  Its CTA may still be inside a bounded wait of its own and store here afterwards, so this CTA must not
            // leave before it: the barrier completes when every other thread of the cluster has left (or failed and come here too);
            // what they stored then has a bounded time to land.
            cluster_sync_all();
            bool landed = false;
            for (int i = 0; i < 100 && !landed; ++i) {
                __nanosleep(10000);
                landed = __all_sync(0xffffffffu, mbar_try_wait(parts + warp, 0));
            }
            if (!landed) { ok = false; if (lane == 0) report_status(p.status, GQ_DEV_TIMEOUT); }
        }
        for (int s = 1; s < p.split; ++s) {
#pragma unroll
            for (int nt = 0; nt < MT; ++nt) {
                const float4 v = red[((s - 1) * GQ_CONSUMER_WARPS * MT + warp * MT + nt) * 32 + lane];
                acc[nt][0] += v.x; acc[nt][1] += v.y; acc[nt][2] += v.z; acc[nt][3] += v.w;
            }
        }
        __syncwarp();       // the warp's part of slot 0 becomes its scratch again below
    } else if (p.cluster) {
        // pull form (when the slots do not fit without costing a resident CTA): every CTA parks its accumulators in
        // its own shared memory, the CTA of split 0 adds the others' in split order through distributed shared
        // memory between two cluster barriers
#pragma unroll
        for (int nt = 0; nt < MT; ++nt) red[(warp * MT + nt) * 32 + lane] = make_float4(acc[nt][0], acc[nt][1], acc[nt][2], acc[nt][3]);
        cluster_sync_all();
        if (split_idx == 0) {
            const uint32_t my = smem_u32(red);
            for (int s = 1; s < p.split; ++s) {
                const uint32_t peer = map_to_rank(my, (uint32_t)s);
#pragma unroll
                for (int nt = 0; nt < MT; ++nt) {
                    const float4 v = ld_cluster_f4(peer + (uint32_t)(((warp * MT + nt) * 32 + lane) * 16));
                    acc[nt][0] += v.x; acc[nt][1] += v.y; acc[nt][2] += v.z; acc[nt][3] += v.w;
                }
            }
        }
        cluster_sync_all();      // peers stay resident until their shared memory has been read
        if (split_idx != 0) return;
    }
    if (p.ar.world > 0 && (p.split == 1 || p.cluster)) {
        // tensor parallel, row-parallel layer: this rank's partial output does not go to y but, as bf16, through
        // the warp's scratch to every rank; y receives the sum over ranks (fused_allreduce_block)
        __nv_bfloat16 *blk = reinterpret_cast<__nv_bfloat16 *>(reinterpret_cast<uint8_t *>(red) + warp * MT * 512);
#pragma unroll
        for (int nt = 0; nt < MT; ++nt)
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int rl = g + 8 * (j >> 1), n = nt * 8 + 2 * t + (j & 1);
                const bool valid = ok && warp * 16 + rl < nvalid && n < p.M;
                blk[n * 16 + rl] = __float2bfloat16_rn(valid ? acc[nt][j] : 0.0f);
            }
        __syncwarp();
        const int ncols = nvalid - warp * 16 < 16 ? nvalid - warp * 16 : 16;
        if (ncols > 0) {
            if (((col0 | ncols | (int)p.n_total) & 1) && lane == 0) report_status(p.status, GQ_DEV_BAD_SHAPE);    // pairs of columns travel together
            else fused_allreduce_block(p, reinterpret_cast<const uint32_t *>(blk), (int)(blockIdx.x / (unsigned)p.split) * GQ_CONSUMER_WARPS + warp,
                                       col0 + warp * 16, ncols, lane, ar_prev);
        }
        return;
    }
#pragma unroll
    for (int nt = 0; nt < MT; ++nt)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int r = warp * 16 + g + 8 * (j >> 1);      // row inside the 64-row tile
            const int n = nt * 8 + 2 * t + (j & 1);          // batch row
            if (ok && r < nvalid && n < p.M) {
                if (p.split == 1 || p.cluster) p.y[(int64_t)n * p.ldy + col0 + r] = __float2bfloat16_rn(acc[nt][j]);
                else p.partials[((int64_t)split_idx * p.M + n) * p.n_total + col0 + r] = acc[nt][j];
            }
        }
}

// Y = sum over splits of the fp32 partials, rounded once to bf16 (reference: sum_partials,
// gguf-plugin/gluon/tiles_grouped.py:142-162)
__global__ void __launch_bounds__(256) sum_partials_kernel(const float *__restrict__ P, int S, int64_t M, int64_t n_total,
                                                           __nv_bfloat16 *__restrict__ y, int64_t ldy) {
    const int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x;
    if (i >= M * n_total) return;
    float a = 0.f;
    for (int s = 0; s < S; ++s) a += P[(int64_t)s * M * n_total + i];
    const int64_t m = i / n_total, c = i - m * n_total;
    y[m * ldy + c] = __float2bfloat16_rn(a);
}

// ---------------------------------------------------------------------------------------------------
// C ABI
// ---------------------------------------------------------------------------------------------------
static int ensure_tables() {
    // per-device one-time upload of the format tables
    static std::atomic<unsigned long long> done_mask{0};
    int dev = 0;
    GQ_CUDA(cudaGetDevice(&dev));
    if (dev < 64 && (done_mask.load() >> dev) & 1ull) return GQ_OK;
    GQ_CUDA(cudaMemcpyToSymbol(c_iq3s_grid, GQ_IQ3S_GRID, sizeof GQ_IQ3S_GRID));
    GQ_CUDA(cudaMemcpyToSymbol(c_iq3xxs_grid, GQ_IQ3XXS_GRID, sizeof GQ_IQ3XXS_GRID));
    GQ_CUDA(cudaMemcpyToSymbol(c_iq2xxs_grid, GQ_IQ2XXS_GRID, sizeof GQ_IQ2XXS_GRID));
    GQ_CUDA(cudaMemcpyToSymbol(c_iq2xs_grid, GQ_IQ2XS_GRID, sizeof GQ_IQ2XS_GRID));
    GQ_CUDA(cudaMemcpyToSymbol(c_iq2s_grid, GQ_IQ2S_GRID, sizeof GQ_IQ2S_GRID));
    GQ_CUDA(cudaMemcpyToSymbol(c_iq1_grid, GQ_IQ1_GRID, sizeof GQ_IQ1_GRID));
    GQ_CUDA(cudaMemcpyToSymbol(c_iq4_kvalues, GQ_IQ4_KVALUES, sizeof GQ_IQ4_KVALUES));
    if (dev < 64) done_mask.fetch_or(1ull << dev);
    return GQ_OK;
}

static int device_sms() {
    static std::atomic<int> cached[64];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 148;
    int v = cached[dev].load();
    if (v <= 0) {
        if (cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || v <= 0) v = 148;
        cached[dev].store(v);
    }
    return v;
}

// opts a kernel in, once per device, to the dynamic shared memory it is launched with (more than 48 KB needs it)
template <auto KERNEL>
static int allow_smem(int bytes) {
    if (bytes <= 48 * 1024) return GQ_OK;
    static std::atomic<unsigned long long> done_mask{0};
    int dev = 0;
    GQ_CUDA(cudaGetDevice(&dev));
    if (dev < 64 && ((done_mask.load() >> dev) & 1ull)) return GQ_OK;
    GQ_CUDA(cudaFuncSetAttribute(KERNEL, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
    if (dev < 64) done_mask.fetch_or(1ull << dev);
    return GQ_OK;
}
// The matrix kernels are launched programmatically, one behind the other, and read tables and weights before they wait for the
// kernel in front: what a load kernel has written is formally visible to them only if something on the stream has waited for that
// kernel.  This launch is that something: an ordinary one, so it starts after the load kernel has completed, and whatever is
// launched behind it starts later still.
__global__ void publish_kernel() {}
static int publish(cudaStream_t st) {
    publish_kernel<<<1, 32, 0, st>>>();
    GQ_LAUNCHED();
    return GQ_OK;
}
#define GQ_EACH_TYPE(X)                                                                                                     \
    X(GQ_Q4_0) X(GQ_Q5_0) X(GQ_Q8_0) X(GQ_Q2_K) X(GQ_Q3_K) X(GQ_Q4_K) X(GQ_Q5_K) X(GQ_Q6_K) X(GQ_IQ4_NL) X(GQ_IQ3_S) X(GQ_IQ4_XS) \
    X(GQ_IQ3_XXS) X(GQ_IQ2_XXS) X(GQ_IQ2_XS) X(GQ_IQ2_S) X(GQ_IQ1_M)

static int check_tensor_args(int type, int64_t n_out, int64_t K) {
    if (!gq_type_bytes(type)) return GQ_ERR_TYPE;
    if (n_out < 0 || K <= 0 || K % GQ_QK || K / GQ_QK > 65535) return GQ_ERR_SHAPE;
    return GQ_OK;
}

extern "C" int gq_repack(int type, const void *raw_dev, int64_t n_out, int64_t K, int64_t raw_row_stride, void *out_dev, void *stream) {
    if (int rc = check_tensor_args(type, n_out, K)) return rc;
    const int B = gq_type_bytes(type);
    const int nb = (int)(K / GQ_QK);
    if (n_out == 0) return GQ_OK;
    if (!raw_dev || !out_dev || ((uintptr_t)out_dev & 15) || raw_row_stride < (int64_t)nb * B) return GQ_ERR_ARG;
    const int64_t slabs = ((n_out + 63) / 64) * 4;
    if (slabs > 0x7fffffff) return GQ_ERR_LIMIT;
    switch (type) {
#define GQ_ONE(T) case T: {                                                                                                        \
            if (int rc = allow_smem<repack_kernel<T>>(16 * stage_pitch(repack_kc<T>() * gq_type_bytes(T)))) return rc;                \
            repack_kernel<T><<<dim3((unsigned)slabs, (unsigned)((nb + repack_kc<T>() - 1) / repack_kc<T>())), GQ_LOAD_THREADS,        \
                               16 * stage_pitch(repack_kc<T>() * gq_type_bytes(T)), (cudaStream_t)stream>>>(                         \
                (const uint8_t *)raw_dev, n_out, nb, raw_row_stride, (uint8_t *)out_dev); break; }
        GQ_EACH_TYPE(GQ_ONE)
#undef GQ_ONE
    }
    GQ_LAUNCHED();
    return publish((cudaStream_t)stream);
}

extern "C" int gq_unrepack(int type, const void *tiles_dev, int64_t n_out, int64_t K, void *raw_dev, int64_t raw_row_stride, void *stream) {
    if (int rc = check_tensor_args(type, n_out, K)) return rc;
    const int B = gq_type_bytes(type);
    const int nb = (int)(K / GQ_QK);
    if (n_out == 0) return GQ_OK;
    if (!raw_dev || !tiles_dev || ((uintptr_t)tiles_dev & 15) || raw_row_stride < (int64_t)nb * B) return GQ_ERR_ARG;
    const int64_t slabs = ((n_out + 63) / 64) * 4;
    if (slabs > 0x7fffffff) return GQ_ERR_LIMIT;
    unrepack_kernel<<<dim3((unsigned)slabs, (unsigned)nb), 256, 0, (cudaStream_t)stream>>>(type, B, (const uint8_t *)tiles_dev, n_out, nb,
                                                                                       (uint8_t *)raw_dev, raw_row_stride);
    GQ_LAUNCHED();
    return GQ_OK;
}

extern "C" int gq_dequant(int type, const void *tiles_dev, int64_t n_out, int64_t K, void *out_dev, int out_dtype, int64_t ld, void *stream) {
    if (int rc = check_tensor_args(type, n_out, K)) return rc;
    const int B = gq_type_bytes(type);
    const int nb = (int)(K / GQ_QK);
    if (n_out == 0) return GQ_OK;
    if (!out_dev || !tiles_dev || ((uintptr_t)tiles_dev & 15) || ld < K || (out_dtype != 0 && out_dtype != 1)) return GQ_ERR_ARG;
    if (int rc = ensure_tables()) return rc;
    const int64_t slabs = ((n_out + 63) / 64) * 4;
    if (slabs > 0x7fffffff) return GQ_ERR_LIMIT;
    // a CTA walks as many of its slab's k-blocks as leave about six CTAs per SM: the codebook table it fills is then shared
    // by up to a whole row of k-blocks
    const int groups = (nb + GQ_LOAD_WARPS - 1) / GQ_LOAD_WARPS;
    int64_t parts = (6 * (int64_t)device_sms() + slabs - 1) / slabs;
    if (parts > groups) parts = groups;
    const int kc = (int)((groups + parts - 1) / parts) * GQ_LOAD_WARPS;
    const dim3 grid((unsigned)slabs, (unsigned)((nb + kc - 1) / kc));
    switch (type) {
#define GQ_ONE_DT(T, BF) {                                                                                                          \
            if (int rc = allow_smem<dequant_kernel<T, BF>>(dequant_smem<T, BF>())) return rc;                                        \
            dequant_kernel<T, BF><<<grid, GQ_LOAD_THREADS, dequant_smem<T, BF>(), (cudaStream_t)stream>>>((const uint8_t *)tiles_dev, \
                                                                                                        n_out, nb, kc, out_dev, ld); }
#define GQ_ONE(T) case T: if (out_dtype == 0) GQ_ONE_DT(T, false) else GQ_ONE_DT(T, true) break;
        GQ_EACH_TYPE(GQ_ONE)
#undef GQ_ONE
#undef GQ_ONE_DT
    }
    GQ_LAUNCHED();
    return GQ_OK;
}

extern "C" int gq_dequant_rows(int type, const void *raw_dev, int64_t n_rows, int64_t K, int64_t raw_row_stride, const void *ids_dev, int ids_bytes,
                               int64_t n_ids, void *out_dev, int out_dtype, int64_t ld, void *stream) {
    if (int rc = check_tensor_args(type, n_rows, K)) return rc;
    const int B = gq_type_bytes(type);
    const int nb = (int)(K / GQ_QK);
    if (n_ids < 0) return GQ_ERR_SHAPE;
    if (n_ids == 0) return GQ_OK;
    if (!raw_dev || !ids_dev || !out_dev || raw_row_stride < (int64_t)nb * B || ld < K || (out_dtype != 0 && out_dtype != 1) ||
        (ids_bytes != 4 && ids_bytes != 8)) return GQ_ERR_ARG;
    if ((n_ids + 15) / 16 > 0x7fffffff) return GQ_ERR_LIMIT;
    if (int rc = ensure_tables()) return rc;
    const dim3 grid((unsigned)((n_ids + 15) / 16), (unsigned)((nb + GQ_LOAD_WARPS - 1) / GQ_LOAD_WARPS));
    switch (type) {
#define GQ_ONE_DT(T, BF) {                                                                                                          \
            if (int rc = allow_smem<dequant_rows_kernel<T, BF>>(dequant_rows_smem<T>())) return rc;                                  \
            dequant_rows_kernel<T, BF><<<grid, GQ_LOAD_THREADS, dequant_rows_smem<T>(), (cudaStream_t)stream>>>(                     \
                (const uint8_t *)raw_dev, n_rows, nb, raw_row_stride, ids_dev, ids_bytes == 8, n_ids, out_dev, ld); }
#define GQ_ONE(T) case T: if (out_dtype == 0) GQ_ONE_DT(T, false) else GQ_ONE_DT(T, true) break;
        GQ_EACH_TYPE(GQ_ONE)
#undef GQ_ONE
#undef GQ_ONE_DT
    }
    GQ_LAUNCHED();
    return GQ_OK;
}

extern "C" int64_t gq_desc_rows(int n_shards, const int64_t *n_outs, int split) {
    if (n_shards <= 0 || !n_outs || split < 1) return GQ_ERR_ARG;
    int64_t tiles = 0;
    for (int i = 0; i < n_shards; ++i) { if (n_outs[i] < 0) return GQ_ERR_SHAPE; tiles += (n_outs[i] + 63) / 64; }
    return tiles * split;
}

// One row of the table, computed from its index alone (host and device).  first_tile / base16 / col0 are the shard's.
struct DescShard {
    int type, n_tiles, n_out, col0, base16;
};
__host__ __device__ inline void desc_row(const DescShard &s, int64_t nb, int split, int tile, int part, int32_t *r) {
    r[0] = (int32_t)(s.base16 + (int64_t)tile * nb * 4 * gq_type_bytes(s.type));       // 64 * bytes / 16
    r[1] = s.type;
    r[2] = s.col0 + tile * 64;
    r[3] = s.n_out - tile * 64 < 64 ? s.n_out - tile * 64 : 64;
    r[4] = (int32_t)((part * nb) / split);
    r[5] = (int32_t)(((part + 1) * nb) / split);
    r[6] = part;
    r[7] = 0;
}
// The shards of a run back to back, one after the other, checked against what a row's 32-bit fields can hold.
struct DescWalk {
    int64_t base16 = 0, col0 = 0, rows = 0;
    int next(int type, int64_t n_out, int64_t nb, int split, DescShard *out) {
        const int B = gq_type_bytes(type);
        if (!B) return GQ_ERR_TYPE;
        if (n_out < 0) return GQ_ERR_SHAPE;
        const int64_t n_tiles = (n_out + 63) / 64;
        // the largest values are those of the shard's last tile; an empty shard writes none
        if (n_tiles && (base16 + (n_tiles - 1) * nb * 4 * B > 0x7fffffff || col0 + (n_tiles - 1) * 64 > 0x7fffffff)) return GQ_ERR_LIMIT;
        if (n_tiles) *out = {type, (int)n_tiles, (int)n_out, (int)col0, (int)base16};
        else *out = {type, 0, 0, 0, 0};
        base16 += n_tiles * nb * 4 * B;
        col0 += n_out;
        rows += n_tiles * split;
        return GQ_OK;
    }
};
static int desc_args(int n_shards, const int32_t *types, const int64_t *n_outs, int64_t K, int split) {
    if (n_shards <= 0 || !types || !n_outs) return GQ_ERR_ARG;
    if (K <= 0 || K % GQ_QK) return GQ_ERR_SHAPE;
    return split < 1 || split > K / GQ_QK ? GQ_ERR_ARG : GQ_OK;
}

extern "C" int64_t gq_build_descs(int n_shards, const int32_t *types, const int64_t *n_outs, int64_t K, int split, int32_t *desc_host) {
    if (!desc_host) return GQ_ERR_ARG;
    if (int rc = desc_args(n_shards, types, n_outs, K, split)) return rc;
    DescShard s;
    DescWalk check;         // nothing is written for a run that is refused
    for (int i = 0; i < n_shards; ++i)
        if (int rc = check.next(types[i], n_outs[i], K / GQ_QK, split, &s)) return rc;
    DescWalk walk;
    for (int i = 0; i < n_shards; ++i) {
        walk.next(types[i], n_outs[i], K / GQ_QK, split, &s);
        for (int t = 0; t < s.n_tiles; ++t)
            for (int p = 0; p < split; ++p, desc_host += GQ_DESC_WORDS) desc_row(s, K / GQ_QK, split, t, p, desc_host);
    }
    return walk.rows;
}

struct DescShards {
    DescShard s[GQ_MAX_DEVICE_SHARDS];
    int n;
};
struct DescSplits {
    int split[GQ_MAX_DEVICE_SPLITS], n;
};
__global__ void __launch_bounds__(256) build_descs_kernel(const DescShards sh, const DescSplits sp, int nb, int tiles, int rows, int32_t *__restrict__ desc) {
    const int row = blockIdx.x * 256 + threadIdx.x;
    if (row >= rows) return;
    int r0 = row, i = 0, k = 0;
    while (k + 1 < sp.n && r0 >= tiles * sp.split[k]) r0 -= tiles * sp.split[k++];      // the table, then the row in it
    const int split = sp.split[k];
    int tile = r0 / split;
    const int part = r0 - tile * split;
    while (i + 1 < sh.n && tile >= sh.s[i].n_tiles) tile -= sh.s[i++].n_tiles;
    __align__(16) int32_t r[GQ_DESC_WORDS];
    desc_row(sh.s[i], nb, split, tile, part, r);
    int4 *o = reinterpret_cast<int4 *>(desc + (int64_t)row * GQ_DESC_WORDS);
    o[0] = make_int4(r[0], r[1], r[2], r[3]);
    o[1] = make_int4(r[4], r[5], r[6], r[7]);
}

extern "C" int64_t gq_build_descs_device(int n_shards, const int32_t *types, const int64_t *n_outs, int64_t K, int n_splits, const int32_t *splits,
                                         int32_t *desc_dev, void *stream) {
    if (n_shards > GQ_MAX_DEVICE_SHARDS || n_splits > GQ_MAX_DEVICE_SPLITS) return GQ_ERR_LIMIT;
    if (!desc_dev || ((uintptr_t)desc_dev & 15) || n_splits <= 0 || !splits) return GQ_ERR_ARG;
    DescShards sh;
    DescSplits sp;
    if (int rc = desc_args(n_shards, types, n_outs, K, 1)) return rc;
    DescWalk walk;
    for (int i = 0; i < n_shards; ++i)
        if (int rc = walk.next(types[i], n_outs[i], K / GQ_QK, 1, sh.s + i)) return rc;
    const int64_t tiles = walk.rows;
    int64_t rows = 0;
    for (int i = 0; i < n_splits; ++i) {
        if (splits[i] < 1 || splits[i] > K / GQ_QK) return GQ_ERR_ARG;
        sp.split[i] = splits[i];
        rows += tiles * splits[i];
    }
    if (rows == 0) return 0;
    if (rows > 0x7ffffff0) return GQ_ERR_LIMIT;
    sh.n = n_shards; sp.n = n_splits;
    build_descs_kernel<<<(unsigned)((rows + 255) / 256), 256, 0, (cudaStream_t)stream>>>(sh, sp, (int)(K / GQ_QK), (int)tiles, (int)rows, desc_dev);
    GQ_LAUNCHED();
    if (int rc = publish((cudaStream_t)stream)) return rc;
    return rows;
}

// CTAs of the grouped kernel that an SM holds by their registers, by the batch rows of a call
static int gemv_ctas_per_sm(int64_t M) { return M <= 8 ? 4 : M <= 16 ? 3 : 2; }

// How many thread-block clusters of 1 .. 8 CTAs the GPU holds side by side with one to four CTAs to an SM (cudaOccupancyMaxActiveClusters on
// 148 SMs: a cluster lies within one of the GPU's processing clusters, and what is left of each stays empty).  Another chip may spread its SMs over
// them differently: a launch planned as one wave may then take two, which costs time and changes no result.
static int64_t cluster_places(int per_sm, int split, int sms) {
    static const short places[4][8] = {{148, 74, 45, 33, 26, 22, 15, 15}, {296, 148, 93, 71, 56, 45, 37, 33}, {444, 222, 142, 104, 82, 71, 56, 48},
                                       {592, 296, 187, 142, 112, 93, 78, 71}};
    return (int64_t)places[per_sm - 1][split - 1] * sms / 148;
}
// The fewest CTAs to an SM (at most `most`) with which `tiles` clusters of `split` find places side by side; 0: they take more than one wave.
// The last places are not counted on: 136 clusters of three for 142 places, and 112 of five for 112, ran as two waves.
static int ctas_per_sm_for(int64_t tiles, int split, int most, int sms) {
    for (int r = 1; r <= most; ++r)
        if (tiles * 100 <= cluster_places(r, split, sms) * 93) return r;
    return 0;
}

// An SM's time for a launch is what its CTAs need together, so up to 16 rows the split is chosen with the number of CTAs to an SM, which
// launch_grouped then holds every SM to: left to the hardware, a launch of fewer CTAs than places fills some SMs and leaves others idle, because
// under programmatic launch the SMs that finish first take all they can hold (and a cluster of eight fits on two SMs).  The costs are in k-blocks'
// times of a CTA alone on its SM, fitted to sweeps of all splits at 4 .. 544 tiles x 5 .. 68 k-blocks of Q4_K, IQ3_S and IQ4_XS, over which calls
// take 0.92 (up to 8 rows) and 0.91 (to 16) of the time under the rule before (the largest split of a single wave that leaves three k-blocks to a
// CTA, the CTAs placed by the hardware).  Microseconds, before / now: 8,704 x 5,120 IQ3_S at 8 / 12 rows 13.5 / 11.7 and 17.1 / 13.6;
// 1,280 x 17,408 IQ4_XS at 8 rows 13.8 / 9.5; 5,120 x 5,120 Q4_K 7.5 / 7.5; 17,408 x 5,120 Q4_K at 1 row 13.3 / 13.4.
struct SplitCost {
    double kb[4];                      // a k-block of a CTA, by the CTAs on its SM
    double split, part;                // a split at all, and per part
    double work, tail, start, crowd;   // more than one wave: the whole work over all SMs, the last CTA's, its start, per part
};
extern "C" int gq_split_for(int64_t n_tiles, int64_t nb, int64_t M, int avg_bytes_per_256, int sm_count) {
    if (n_tiles <= 0 || nb <= 0) return 1;
    if (sm_count <= 0) sm_count = 148;
    const int most = gemv_ctas_per_sm(M);
    const int64_t slots = (int64_t)most * sm_count;
    int s = 1;
    if (most == 2) {
        // the largest split up to 8 that leaves a CTA three k-blocks and the launch one wave, clusters of S filling 1 - 0.03 (S - 1) of the
        // places (the sweeps above 16 rows left little to a finer rule: 0.97 of the time)
        for (int S = 2; S <= 8 && S <= nb / 3; ++S)
            if (S * n_tiles * 100 <= slots * (100 - 3 * (S - 1))) s = S;
        return s;
    }
    static const SplitCost costs[2] = {{{0.80, 1.08, 1.47, 1.95}, 0.72, 0.04, 1.67, 0.96, 0.32, 0.46}, {{0.90, 1.21, 1.80, 0.0}, 0.29, 0.033, 1.94, 0.64, 0.34, 0.67}};
    const SplitCost &c = costs[most == 4 ? 0 : 1];
    double best = 1e300, held = 0.0;
    // 9 .. 16 rows: the largest split of one wave that leaves a CTA three k-blocks stays unless another is to save more than an eighth.  Below
    // that, which types the launch behind finds on an SM counts for more (o_proj and down_proj before 34,816 x 5,120, whose 544 CTAs are a wave and
    // a quarter): four / three parts, o + gate_up of IQ4_XS, IQ4_XS + IQ3_S
    // 52.1 / 60.5 us, stacks of two blocks 191 / 199 to 199 / 189, where the single layers with three take 0.95 to 0.99 of the time.  (That effect
    // depends on the next launch, which is not known here; up to 8 rows the unsharded layers get the same splits either way.)
    int wave = 0;
    if (most == 3)
        for (int S = 1; S <= 8 && (S == 1 || S <= nb / 3); ++S)
            if (S * n_tiles * 100 <= slots * (100 - 3 * (S - 1))) wave = S;
    for (int S = 1; S <= 8 && S <= nb; ++S) {
        const int r = ctas_per_sm_for(n_tiles, S, most, sm_count);
        const double kb = 0.5 * (double)((nb + S - 1) / S) + 0.5 * (double)nb / S;      // parts differ by one k-block
        double cost;
        // (tiles of 13 KB and more: four CTAs to an SM have no room for the pushed reduction, and short parts do not repay the other:
        // 5,120 x 4,352 Q6_K at 4 rows with 5 / 6 parts 7.8 / 9.2 us)
        if (avg_bytes_per_256 >= 200 && r == 4 && nb >= 8 && S > nb / 3) continue;
        if (r) cost = kb * c.kb[r - 1];
        else if (S > 1 && n_tiles * S * 10 > slots * 14) continue;
        else cost = (double)n_tiles * (double)nb / sm_count * c.kb[most - 1] / most * c.work + kb * c.tail + c.start + c.crowd * (S - 1);
        cost += (S > 1 ? c.split : 0.0) + c.part * S;
        if (S == wave) held = cost;
        if (cost < best * (1.0 - 1e-9)) { best = cost; s = S; }
    }
    return 8.0 * best > 7.0 * held && held > 0.0 ? wave : s;
}

extern "C" int64_t gq_workspace_bytes(int64_t M, int64_t K, int64_t n_total, int split) {
    if (M < 0 || K <= 0 || K % GQ_QK || n_total < 0 || split < 1) return GQ_ERR_SHAPE;
    return ws_layout(M, K, n_total, split, nullptr, nullptr);
}

template <int MT, int MINB, int FORM, int ONLY>
static int launch_gemv(const GemvParams &p, int64_t n_desc, int apart, cudaStream_t stream) {
    constexpr int xbytes = gq_stage_xbytes<MT, FORM>();
    const int stage_bytes = p.wbytes_max + xbytes;
    size_t smem = (size_t)p.stages * stage_bytes + (size_t)p.stages * 16 + 8 * GQ_CONSUMER_WARPS + (size_t)p.cb_bytes +
                        (gq_red_in_ring<MT>() ? 0 : (size_t)GQ_CONSUMER_WARPS * MT * 512 * (p.cluster_push ? p.split - 1 : 1));
    if (smem > 232448) return GQ_ERR_LIMIT;
    // `apart` CTAs to an SM and not one more (0: as many as fit): they ask for so much shared memory
    if (apart) {
        const size_t least = ((size_t)(228 * 1024) / (apart + 1) - 1024 + 16) & ~(size_t)15;
        if (smem < least) smem = least;
    }
    // opt in once per device to the largest dynamic shared memory a CTA can have
    static std::atomic<unsigned long long> done_mask{0};
    int dev = 0;
    GQ_CUDA(cudaGetDevice(&dev));
    if (dev >= 64 || !((done_mask.load() >> dev) & 1ull)) {
        GQ_CUDA(cudaFuncSetAttribute(gemv_grouped_kernel<MT, MINB, FORM, ONLY>, cudaFuncAttributeMaxDynamicSharedMemorySize, 232448));
        if (dev < 64) done_mask.fetch_or(1ull << dev);
    }
    {
        cudaLaunchConfig_t cfg = {};
        cudaLaunchAttribute attr[2];
        int na = 0;
        if (p.cluster) {
            attr[na].id = cudaLaunchAttributeClusterDimension;
            attr[na].val.clusterDim.x = (unsigned)p.split; attr[na].val.clusterDim.y = 1; attr[na].val.clusterDim.z = 1;
            ++na;
        }
        attr[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[na].val.programmaticStreamSerializationAllowed = 1;
        ++na;
        cfg.gridDim = dim3((unsigned)n_desc); cfg.blockDim = dim3(32 * (GQ_CONSUMER_WARPS + 1)); cfg.dynamicSmemBytes = smem; cfg.stream = stream;
        cfg.attrs = attr; cfg.numAttrs = na;
        GQ_CUDA(cudaLaunchKernelEx(&cfg, gemv_grouped_kernel<MT, MINB, FORM, ONLY>, p));
    }
    GQ_LAUNCHED();
    return GQ_OK;
}

// integer form, M <= 8 (FORM 1) and M <= 4 (FORM 2): one instantiation per type for runs of a single type, the all-types one otherwise
template <int FORM>
static int launch_gemv8_m8(const GemvParams &p, int64_t n_desc, int apart, cudaStream_t st, int only) {
    switch (only) {
#define GQ_ONE(T) case T: return launch_gemv<1, 4, FORM, T>(p, n_desc, apart, st);
        GQ_EACH_TYPE(GQ_ONE)
#undef GQ_ONE
        default: return launch_gemv<1, 4, FORM, 0>(p, n_desc, apart, st);
    }
}

extern "C" int gq_run_info(int n_shards, const int32_t *types) {
    if (n_shards <= 0 || !types) return GQ_ERR_ARG;
    int maxb = 0, cb = 0, single = types[0];
    for (int i = 0; i < n_shards; ++i) {
        const int B = gq_type_bytes(types[i]);
        if (!B) return GQ_ERR_TYPE;
        if (B > maxb) maxb = B;
        if (gq_cb_kind(types[i]) >= 0) cb |= 1 << gq_cb_kind(types[i]);     // a codebook type: the kernels keep its grid in shared memory
        if (types[i] != single) single = 0;
    }
    return maxb | ((cb ? 1 : 0) << 16) | (single << 17) | (cb << 22);
}

// A run's tiles may be worked on from the last to the first.  Which types first: the CTAs of an SM are neighbours of the launch's order, and those
// that start last, on the SMs that the kernel in front leaves last or in what is left of a wave, should be the quick ones.  2 x 17,408 x 5,120 with
// the slower type first / second: IQ3_S and Q4_K at 1 / 8 rows 28.6 / 33.5 and 31.4 / 36.2 us, at 64 52.3 / 54.4; IQ3_S and Q2_K 29.6 / 32.7, 32.7 / 36.1
// and 50.9 / 53.4.  From 9 to 32 rows, of one and a quarter to two waves, neither order is the better one (IQ3_S and Q4_K at 13 rows 46.2 / 40.0), nor is
// it with CTA pairs.  Costs: 17,408 x 5,120 at 8 rows, 34,816 x 5,120 at 64, in tenths of a microsecond.
static int order_cost(int type, bool tcgen05) {
    switch (type) {
        case GQ_Q4_0: return tcgen05 ? 348 : 123; case GQ_Q5_0: return tcgen05 ? 484 : 175; case GQ_Q8_0: return tcgen05 ? 400 : 212;
        case GQ_Q2_K: return tcgen05 ? 394 : 117; case GQ_Q3_K: return tcgen05 ? 457 : 159; case GQ_Q4_K: return tcgen05 ? 380 : 124;
        case GQ_Q5_K: return tcgen05 ? 469 : 151; case GQ_Q6_K: return tcgen05 ? 435 : 179; case GQ_IQ4_NL: return tcgen05 ? 456 : 176;
        case GQ_IQ3_S: return tcgen05 ? 529 : 170; case GQ_IQ4_XS: return tcgen05 ? 487 : 191; case GQ_IQ3_XXS: return tcgen05 ? 598 : 204;
        case GQ_IQ2_XXS: return tcgen05 ? 598 : 196; case GQ_IQ2_XS: return tcgen05 ? 617 : 221; case GQ_IQ2_S: return tcgen05 ? 588 : 213;
        default: return tcgen05 ? 567 : 220;
    }
}
extern "C" int gq_run_order(int n_shards, const int32_t *types, const int64_t *n_outs) {
    if (n_shards <= 0 || !types || !n_outs) return GQ_ERR_ARG;
    int64_t tiles = 0;
    for (int i = 0; i < n_shards; ++i) {
        if (!gq_type_bytes(types[i])) return GQ_ERR_TYPE;
        if (n_outs[i] < 0) return GQ_ERR_SHAPE;
        tiles += (n_outs[i] + 63) / 64;
    }
    int flags = 0;
    for (int form = 0; form < 2; ++form) {
        // what the first and the second half of the tiles cost
        double first = 0.0, second = 0.0, at = 0.0;
        for (int i = 0; i < n_shards; ++i) {
            const double n = (double)((n_outs[i] + 63) / 64), mid = 0.5 * (double)tiles, in = at + n <= mid ? n : at >= mid ? 0.0 : mid - at, c = order_cost(types[i], form == 1);
            first += in * c; second += (n - in) * c; at += n;
        }
        if (second > 1.03 * first) flags |= GQ_ORDER_8 << form;
    }
    return flags;
}

// the activation preparation of `rows` batch rows (form 1: integer, 0: fp16, which has no folded op: the entry points end those at
// GQ_GEMV8_MAX_ROWS)
static int launch_prep(const __nv_bfloat16 *x, int64_t rows, int64_t K, int64_t ldx, uint8_t *xt, int *status, int form, const PreOp *pre, cudaStream_t st) {
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.dynamicSmemBytes = 0; cfg.stream = st; cfg.attrs = attr; cfg.numAttrs = 1;
    cfg.gridDim = dim3((unsigned)(K / GQ_QK), (unsigned)((rows + GQ_PREP_WARPS - 1) / GQ_PREP_WARPS)); cfg.blockDim = dim3(32 * GQ_PREP_WARPS);
    const PreOp po = pre ? *pre : PreOp{};
    if (po.kind == GQ_PRE_ADD_RMSNORM) {
        const int64_t nb = K / GQ_QK;
        cfg.gridDim = dim3((unsigned)rows); cfg.blockDim = dim3(32 * (unsigned)(nb < GQ_NORM_MAX_WARPS ? nb : GQ_NORM_MAX_WARPS));
        GQ_CUDA(cudaLaunchKernelEx(&cfg, norm_rows_kernel<true>, x, ldx, (int)rows, xt, status, (__nv_bfloat16 *)nullptr, (int64_t)0, po));
    } else {
        auto *kern = po.kind == GQ_PRE_SILU_MUL ? prep_x_kernel<GQ_PRE_SILU_MUL, 1> : form ? prep_x_kernel<GQ_PRE_NONE, 1> : prep_x_kernel<GQ_PRE_NONE, 0>;
        GQ_CUDA(cudaLaunchKernelEx(&cfg, kern, x, ldx, (int)rows, xt, status, po));
    }
    GQ_LAUNCHED();
    return GQ_OK;
}

// an SM has 228 KB of shared memory, of which the system keeps 1 KB per resident CTA
static int resident_ctas(int smem, int cap) { const int n = (228 * 1024) / (smem + 1024); return n < cap ? n : cap; }

// One tile to a CTA.  Rings: integer form, the deepest of three or four stages that leaves room for the CTAs that an SM is to hold (swept on
// the 64-layer stack: deeper rings with fewer resident CTAs were slower); fp16 form, whose activation tiles are larger, of two to four; where
// its launch fits one CTA per SM it takes four, beside which few types leave room for a second CTA.
// The fp16 form with two tiles and eight consumer warps to a CTA (96 registers) was 4 - 9 % faster on 34,816 x 5,120 of Q2_K, Q4_K or Q8_0
// and slower elsewhere: 5,120 x 5,120 at 17 rows Q4_K 10.5 -> 13.9, Q5_0 12.2 -> 16.4, 1,024 x 5,120 at 27 rows Q8_0 8.0 -> 13.4.
static int launch_grouped(GemvParams &p, int run_info, int64_t n_desc, cudaStream_t st) {
    const bool fp16 = p.M > GQ_GEMV8_MAX_ROWS;
    const int mt = p.M <= 8 ? 1 : p.M <= 16 ? 2 : p.M <= 24 ? 3 : p.M <= 32 ? 4 : 8, low = fp16 ? 2 : 3;
    // as many CTAs to an SM as the launch needs and no more (gq_split_for); a launch of more than one wave takes all places
    const int most = gemv_ctas_per_sm(p.M), S = p.cluster ? p.split : 1, sms = device_sms();
    const int need = ctas_per_sm_for(n_desc / S, S, most, sms), cap = need ? need : most;
    // (a launch that leaves a tenth of its places empty is as fast or faster in its own order: q, k, v of 5,120 + 2 x 1,024 rows)
    if (n_desc * 10 < 9 * (int64_t)cap * sms) p.reverse = 0;
    // fp16 form, short parts of a launch that leaves SMs idle in any case: starting under the kernel in front is worth more (1,024 x 5,120
    // IQ4_XS at 32 rows 7.8 / 7.6 us, 5,120 x 1,280 7.0 / 6.7)
    const int apart = cap < most && !(fp16 && p.nb <= 6 * p.split) ? cap : 0;
    const int stage_bytes = p.wbytes_max + (p.M <= 4 ? gq_stage_xbytes<1, 2>() : 8 * mt * GQ_X_ROW + 32 * mt), red1 = mt == 8 ? 0 : GQ_CONSUMER_WARPS * mt * 512;
    const auto resident = [&](int stages, int red, int most) { return resident_ctas(stages * stage_bytes + 64 + 8 * GQ_CONSUMER_WARPS + p.cb_bytes + red, most); };
    // split-K in a cluster: the push form of the reduction needs a scratch slot per other split in every CTA; it is used when that
    // costs no resident CTA at the shallowest ring
    p.cluster_push = p.cluster && red1 && resident(low, red1 * (p.split - 1), cap) >= resident(low, red1, cap) ? 1 : 0;
    const int red = p.cluster_push ? red1 * (p.split - 1) : red1;
    if (fp16) {
        for (p.stages = 2; p.stages < 4 && resident(p.stages + 1, red, cap) >= resident(2, red, cap);) ++p.stages;
    } else {
        p.stages = resident(4, red, cap) >= cap ? 4 : 3;
    }
    switch (mt) {
        case 1: return p.M <= 4 ? launch_gemv8_m8<2>(p, n_desc, apart, st, (run_info >> 17) & 31) : launch_gemv8_m8<1>(p, n_desc, apart, st, (run_info >> 17) & 31);
        case 2: return launch_gemv<2, 3, 1, 0>(p, n_desc, apart, st);
        case 3: return launch_gemv<3, 2, 0, 0>(p, n_desc, apart, st);
        case 4: return launch_gemv<4, 2, 0, 0>(p, n_desc, apart, st);
        default: return launch_gemv<8, 2, 0, 0>(p, n_desc, apart, st);
    }
}

static int gemv_grouped_impl(const void *x_dev, int64_t M, int64_t K, int64_t ldx, const void *packed_dev, const int32_t *desc_dev,
                             int64_t n_desc, int split, int run_info, void *y_dev, int64_t ldy, int64_t n_total, void *workspace_dev,
                             int64_t workspace_bytes, void *stream, int phases, const void *next_packed_dev, int64_t next_bytes,
                             const ArFused *ar = nullptr, const PreOp *pre = nullptr) {
    if (M < 0 || M > GQ_MAX_GEMV_ROWS || K <= 0 || K % GQ_QK || n_total < 0 || n_desc < 0 || split < 1) return GQ_ERR_SHAPE;
    if (M == 0 || n_total == 0 || n_desc == 0) return GQ_OK;
    if (!x_dev || !packed_dev || !desc_dev || !y_dev || !workspace_dev) return GQ_ERR_ARG;
    if (((uintptr_t)packed_dev & 15) || ((uintptr_t)workspace_dev & 255) || ((uintptr_t)x_dev & 3) || ldx < K || ldy < n_total) return GQ_ERR_ARG;
    if (n_desc > 0x7fffffff) return GQ_ERR_LIMIT;
    Workspace ws;
    const int64_t need = ws_layout(M, K, n_total, split, workspace_dev, &ws);
    if (workspace_bytes < need) return GQ_ERR_WORKSPACE;
    if (int rc = ensure_tables()) return rc;
    cudaStream_t st = (cudaStream_t)stream;

    const int maxb = run_info & 0xFFFF;
    if ((phases & 6) && (maxb < 56 || maxb > 272 || (maxb & 1))) return GQ_ERR_ARG;
    // split-K up to 8 reduces inside a thread-block cluster (portable cluster size); larger splits keep the fp32
    // partials and the separate sum
    const int cluster = (split > 1 && split <= 8 && n_desc % split == 0) ? 1 : 0;
    if (ar && (phases & 6)) {
        if (split > 1 && !cluster) return GQ_ERR_ARG;        // the exchange needs the whole tile sum in one CTA
        if (n_desc / split * GQ_CONSUMER_WARPS > ar->units) return GQ_ERR_LIMIT;
    }
    // Whether the grouped kernel converts the activations itself: one row, nothing folded in front, and at most four k-blocks to a
    // CTA, up to where the conversions, one after the other, take no longer than the boundary they save (graphs of 24 layers, Q4_K:
    // 5120 x 5120, 3.3 k-blocks, 6.8 -> 6.5 us; 7168 x 5120, 5 k-blocks, 7.4 -> 8.3; a second row adds 2 us)
    const bool direct = (phases & 8) && M == 1 && !ar && !(pre && pre->kind) && (K / GQ_QK + split - 1) / split <= 4;

    if ((phases & 1) && !direct)
        if (int rc = launch_prep((const __nv_bfloat16 *)x_dev, M, K, ldx, ws.xt, ws.status, M > GQ_GEMV8_MAX_ROWS ? 0 : 1, pre, st)) return rc;
    if (phases & 2) {
        GemvParams p;
        p.packed = (const uint8_t *)packed_dev; p.desc = desc_dev; p.xt = ws.xt;
        p.y = (__nv_bfloat16 *)y_dev; p.partials = ws.partials; p.status = ws.status;
        p.M = (int)M; p.K = (int)K; p.nb = (int)(K / GQ_QK); p.split = split; p.ldy = ldy; p.n_total = n_total;
        p.wbytes_max = 64 * maxb;   // every stage can hold a tile of any shard of the run
        p.cb_bytes = gq_cb_region_max((run_info >> 22) & 63);
        p.cluster = cluster;
        p.reverse = M <= 8 && (run_info & GQ_ORDER_8) && !ar && n_desc % split == 0 ? 1 : 0;      // (launch_grouped has the last word)
        p.x = direct ? (const __nv_bfloat16 *)x_dev : nullptr;
        p.pf_ptr = (next_packed_dev && next_bytes > 0 && !((uintptr_t)next_packed_dev & 15)) ? (const uint8_t *)next_packed_dev : nullptr;
        p.pf_bytes = next_bytes;
        p.ar = ar ? *ar : ArFused{};
        if (int rc = launch_grouped(p, run_info, n_desc, st)) return rc;
    }
    if (split > 1 && !cluster && (phases & 4)) {
        const int64_t n = M * n_total;
        sum_partials_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(ws.partials, split, M, n_total, (__nv_bfloat16 *)y_dev, ldy);
        GQ_LAUNCHED();
    }
    return GQ_OK;
}

extern "C" int gq_gemv_grouped_phases(const void *x_dev, int64_t M, int64_t K, int64_t ldx, const void *packed_dev, const int32_t *desc_dev,
                                      int64_t n_desc, int split, int run_info, void *y_dev, int64_t ldy, int64_t n_total,
                                      void *workspace_dev, int64_t workspace_bytes, void *stream, int phases) {
    return gemv_grouped_impl(x_dev, M, K, ldx, packed_dev, desc_dev, n_desc, split, run_info, y_dev, ldy, n_total, workspace_dev,
                             workspace_bytes, stream, phases, nullptr, 0);
}

extern "C" int gq_gemv_grouped_prefetch(const void *x_dev, int64_t M, int64_t K, int64_t ldx, const void *packed_dev, const int32_t *desc_dev,
                                        int64_t n_desc, int split, int run_info, void *y_dev, int64_t ldy, int64_t n_total,
                                        void *workspace_dev, int64_t workspace_bytes, void *stream, const void *next_packed_dev,
                                        int64_t next_bytes) {
    return gemv_grouped_impl(x_dev, M, K, ldx, packed_dev, desc_dev, n_desc, split, run_info, y_dev, ldy, n_total, workspace_dev,
                             workspace_bytes, stream, 7, next_packed_dev, next_bytes);
}

extern "C" int gq_gemv_grouped(const void *x_dev, int64_t M, int64_t K, int64_t ldx, const void *packed_dev, const int32_t *desc_dev,
                               int64_t n_desc, int split, int run_info, void *y_dev, int64_t ldy, int64_t n_total, void *workspace_dev,
                               int64_t workspace_bytes, void *stream) {
    return gq_gemv_grouped_phases(x_dev, M, K, ldx, packed_dev, desc_dev, n_desc, split, run_info, y_dev, ldy, n_total, workspace_dev,
                                  workspace_bytes, stream, 7);
}

// in_place: residual_out may be residual_in
static int make_pre_op(PreOp &po, int64_t K, int64_t ldx, int pre_op, const void *norm_weight_dev, const void *residual_in_dev, void *residual_out_dev, int64_t ld_res,
                       float eps, bool in_place) {
    po.kind = pre_op; po.K = (int)K; po.eps = eps;
    if (pre_op == GQ_PRE_SILU_MUL) {
        if (ldx < 2 * K) return GQ_ERR_ARG;
    } else if (pre_op == GQ_PRE_ADD_RMSNORM) {
        if (!norm_weight_dev || ((uintptr_t)norm_weight_dev & 1)) return GQ_ERR_ARG;
        if ((residual_in_dev == nullptr) != (residual_out_dev == nullptr)) return GQ_ERR_ARG;
        if (residual_in_dev && ((residual_in_dev == residual_out_dev && !in_place) || ld_res < K)) return GQ_ERR_ARG;
        po.weight = (const __nv_bfloat16 *)norm_weight_dev;
        po.residual = (const __nv_bfloat16 *)residual_in_dev; po.residual_out = (__nv_bfloat16 *)residual_out_dev; po.ld_res = ld_res;
    } else if (pre_op != GQ_PRE_NONE) {
        return GQ_ERR_ARG;
    }
    return GQ_OK;
}

// the op by itself, for batches of more rows than the preparation folds
extern "C" int gq_pre_op(const void *x_dev, int64_t M, int64_t K, int64_t ldx, int pre_op, const void *norm_weight_dev, const void *residual_in_dev,
                         void *residual_out_dev, int64_t ld_res, float eps, void *out_dev, int64_t ldo, void *stream) {
    if (M < 0 || K <= 0 || K % GQ_QK || K > 0x3fffffff) return GQ_ERR_SHAPE;
    if (pre_op != GQ_PRE_SILU_MUL && pre_op != GQ_PRE_ADD_RMSNORM) return GQ_ERR_ARG;
    if (M == 0) return GQ_OK;
    if (!x_dev || !out_dev || ldo < K || ldx < K || (((uintptr_t)x_dev | (uintptr_t)out_dev | (uintptr_t)residual_in_dev | (uintptr_t)residual_out_dev) & 1)) return GQ_ERR_ARG;
    PreOp po{};
    if (int rc = make_pre_op(po, K, ldx, pre_op, norm_weight_dev, residual_in_dev, residual_out_dev, ld_res, eps, true)) return rc;
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.stream = (cudaStream_t)stream; cfg.attrs = attr; cfg.numAttrs = 1;
    if (pre_op == GQ_PRE_ADD_RMSNORM) {
        if (M > 0x7fffffff) return GQ_ERR_LIMIT;
        // two k-blocks to a warp where there are rows for every SM (more CTAs to it), else one
        const int64_t nb = K / GQ_QK, warps = M > device_sms() ? (nb + 1) / 2 : nb;
        cfg.gridDim = dim3((unsigned)M); cfg.blockDim = dim3(32 * (unsigned)(warps < GQ_NORM_MAX_WARPS ? warps : GQ_NORM_MAX_WARPS));
        GQ_CUDA(cudaLaunchKernelEx(&cfg, norm_rows_kernel<false>, (const __nv_bfloat16 *)x_dev, ldx, (int)M, (uint8_t *)nullptr, (int *)nullptr,
                                   (__nv_bfloat16 *)out_dev, ldo, po));
        GQ_LAUNCHED();
        return GQ_OK;
    }
    // a row over CTAs of equal size, whole warps (a grid has 65,535 rows of CTAs)
    const unsigned parts = (unsigned)((K / 8 + 255) / 256), threads = (unsigned)((K / 8 + 32 * parts - 1) / (32 * parts)) * 32;
    for (int64_t m = 0; m < M; m += 65535) {
        cfg.gridDim = dim3(parts, (unsigned)(M - m < 65535 ? M - m : 65535)); cfg.blockDim = dim3(threads);
        GQ_CUDA(cudaLaunchKernelEx(&cfg, silu_mul_kernel, (const __nv_bfloat16 *)x_dev + m * ldx, ldx, (int)K, (__nv_bfloat16 *)out_dev + m * ldo, ldo));
        GQ_LAUNCHED();
    }
    return GQ_OK;
}

// ---- the same call with the op in front of the layer folded into the activation preparation -----------------
// pre_op GQ_PRE_SILU_MUL: x_dev is the [M, 2K] output of gate_up_proj (ldx >= 2K), the layer multiplies
// silu(x[:, :K]) * x[:, K:].  GQ_PRE_ADD_RMSNORM: x_dev is [M, K]; norm_weight [K]; residual_in / residual_out [M, ld_res]
// both or neither (the same memory is refused here; gq_pre_op takes it).  1..GQ_GEMV8_MAX_ROWS rows.
extern "C" int gq_gemv_grouped_pre(const void *x_dev, int64_t M, int64_t K, int64_t ldx, int pre_op, const void *norm_weight_dev,
                                   const void *residual_in_dev, void *residual_out_dev, int64_t ld_res, float eps, const void *packed_dev,
                                   const int32_t *desc_dev, int64_t n_desc, int split, int run_info, void *y_dev, int64_t ldy,
                                   int64_t n_total, void *workspace_dev, int64_t workspace_bytes, void *stream) {
    if (M < 0 || M > GQ_GEMV8_MAX_ROWS) return GQ_ERR_SHAPE;
    PreOp po{};
    if (int rc = make_pre_op(po, K, ldx, pre_op, norm_weight_dev, residual_in_dev, residual_out_dev, ld_res, eps, false)) return rc;
    return gemv_grouped_impl(x_dev, M, K, ldx, packed_dev, desc_dev, n_desc, split, run_info, y_dev, ldy, n_total, workspace_dev,
                             workspace_bytes, stream, 7, nullptr, 0, nullptr, &po);
}

// ---- the same call for callers that cannot allocate device memory -------------------------------------
// Scratch lives in this fixed array, part of the library's device image: every GPU that loads the library
// holds it until the process exits.  All calls of gq_gemv_grouped_static on a device share it.
#define GQ_STATIC_WS_BYTES (8ll << 20)
static __device__ __align__(256) unsigned char g_static_ws[GQ_STATIC_WS_BYTES];

extern "C" int64_t gq_static_workspace_limit(void) { return GQ_STATIC_WS_BYTES; }

extern "C" int gq_gemv_grouped_static(const void *x_dev, int64_t M, int64_t K, int64_t ldx, const void *packed_dev, const int32_t *desc_dev,
                                      int64_t n_desc, int split, int run_info, void *y_dev, int64_t ldy, int64_t n_total, void *stream) {
    if (M < 0 || M > GQ_MAX_GEMV_ROWS || K <= 0 || K % GQ_QK || n_total < 0 || n_desc < 0 || split < 1) return GQ_ERR_SHAPE;
    const int64_t need = ws_layout(M, K, n_total, split, nullptr, nullptr);
    if (need > GQ_STATIC_WS_BYTES) {
        snprintf(g_cuda_err, sizeof g_cuda_err, "gq_gemv_grouped_static: this call needs %lld bytes of scratch, the built-in buffer holds %lld",
                 (long long)need, (long long)GQ_STATIC_WS_BYTES);
        return GQ_ERR_LIMIT;
    }
    // In host code `g_static_ws` is only a handle for the symbol; the address the kernels may use is looked up
    // once per device, with that device current.
    static void *dev_ptr[64] = {nullptr};
    int dev = 0;
    GQ_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64) return GQ_ERR_LIMIT;
    void *ws = dev_ptr[dev];
    if (!ws) {
        GQ_CUDA(cudaGetSymbolAddress(&ws, g_static_ws));
        if (!ws) return GQ_ERR_CUDA;
        dev_ptr[dev] = ws;
    }
    return gq_gemv_grouped_phases(x_dev, M, K, ldx, packed_dev, desc_dev, n_desc, split, run_info, y_dev, ldy, n_total, ws,
                                  GQ_STATIC_WS_BYTES, stream, 7);
}

// ---- the same call fused with the all-reduce of a row-parallel layer ---------------------------------------
// Every rank multiplies its K shard; the kernel's epilogue exchanges the bf16 partial outputs through peer memory
// and leaves the sum over ranks in y on every rank (fused_allreduce_block).  Same arithmetic as the grouped call
// followed by gq_allreduce_push, without the second launch and its latency.
static int64_t fused_ar_units(int64_t max_n_total) { return (max_n_total / 64 + 64) * GQ_CONSUMER_WARPS; }
static int64_t fused_ar_header(int64_t max_n_total) { return (4 * fused_ar_units(max_n_total) + 4095) & ~(int64_t)4095; }

extern "C" int64_t gq_fused_allreduce_buffer_bytes(int world, int64_t max_m, int64_t max_n_total) {
    if (world < 1 || world > GQ_AR_MAX_WORLD || max_m < 1 || max_m > GQ_MAX_GEMV_ROWS || max_n_total < 1) return GQ_ERR_ARG;
    return fused_ar_header(max_n_total) + 2 * (int64_t)world * align256(max_m * max_n_total * 4);
}

static int gemv_grouped_allreduce_impl(const void *x_dev, int64_t M, int64_t K, int64_t ldx, const void *packed_dev, const int32_t *desc_dev,
                                       int64_t n_desc, int split, int run_info, void *y_dev, int64_t ldy, int64_t n_total,
                                       void *workspace_dev, int64_t workspace_bytes, int rank, int world, const uint64_t *peer_buffers,
                                       int64_t max_m, int64_t max_n_total, void *stream, const PreOp *pre) {
    if (world < 1 || world > GQ_AR_MAX_WORLD || rank < 0 || rank >= world || !peer_buffers) return GQ_ERR_ARG;
    if (max_m < 1 || max_m > GQ_MAX_GEMV_ROWS || M > max_m || n_total > max_n_total) return GQ_ERR_SHAPE;
    ArFused ar = {};
    ar.world = world; ar.rank = rank; ar.units = (int)fused_ar_units(max_n_total);
    ar.wait_ns = g_peer_wait_ns.load();
    if (n_total & 1) return GQ_ERR_SHAPE;
    if (world > 1 && M > 0 && n_total > 0 && n_desc > 0) {
        // a buffer serves one output width: the words' positions depend on n_total while the call numbers are kept per
        // (tile, warp), so a second width on the same buffer could meet a stale word that carries a current number
        static std::mutex mu;
        static std::unordered_map<uint64_t, int64_t> bound;
        std::lock_guard<std::mutex> lock(mu);
        auto it = bound.find(peer_buffers[rank]);
        if (it == bound.end()) bound.emplace(peer_buffers[rank], n_total);
        else if (it->second != n_total) {
            snprintf(g_cuda_err, sizeof g_cuda_err, "gq_gemv_grouped_allreduce: this buffer exchanges outputs of %lld columns, the call has %lld",
                     (long long)it->second, (long long)n_total);
            return GQ_ERR_ARG;
        }
    }
    ar.slot_bytes = align256(max_m * max_n_total * 4);
    const int64_t header = fused_ar_header(max_n_total);
    for (int p = 0; p < world; ++p) {
        if (!peer_buffers[p] || (peer_buffers[p] & 255)) return GQ_ERR_ARG;
        uint8_t *b = reinterpret_cast<uint8_t *>(peer_buffers[p]);
        ar.buf[p] = b + header;
    }
    ar.counters = reinterpret_cast<uint32_t *>(peer_buffers[rank]);
    return gemv_grouped_impl(x_dev, M, K, ldx, packed_dev, desc_dev, n_desc, split, run_info, y_dev, ldy, n_total, workspace_dev,
                             workspace_bytes, stream, 7, nullptr, 0, &ar, pre);
}

extern "C" int gq_gemv_grouped_allreduce(const void *x_dev, int64_t M, int64_t K, int64_t ldx, const void *packed_dev, const int32_t *desc_dev,
                                         int64_t n_desc, int split, int run_info, void *y_dev, int64_t ldy, int64_t n_total,
                                         void *workspace_dev, int64_t workspace_bytes, int rank, int world, const uint64_t *peer_buffers,
                                         int64_t max_m, int64_t max_n_total, void *stream) {
    return gemv_grouped_allreduce_impl(x_dev, M, K, ldx, packed_dev, desc_dev, n_desc, split, run_info, y_dev, ldy, n_total, workspace_dev,
                                       workspace_bytes, rank, world, peer_buffers, max_m, max_n_total, stream, nullptr);
}

// the fused multiply + all-reduce of a row-parallel down_proj with silu_and_mul folded into its activation preparation:
// x_dev is this rank's [M, 2K] slice pair (gate | up of its K columns, ldx >= 2K), 1..GQ_GEMV8_MAX_ROWS rows
extern "C" int gq_gemv_grouped_allreduce_silu_mul(const void *x_dev, int64_t M, int64_t K, int64_t ldx, const void *packed_dev,
                                                  const int32_t *desc_dev, int64_t n_desc, int split, int run_info, void *y_dev, int64_t ldy,
                                                  int64_t n_total, void *workspace_dev, int64_t workspace_bytes, int rank, int world,
                                                  const uint64_t *peer_buffers, int64_t max_m, int64_t max_n_total, void *stream) {
    if (M < 0 || M > GQ_GEMV8_MAX_ROWS) return GQ_ERR_SHAPE;
    if (ldx < 2 * K) return GQ_ERR_ARG;
    PreOp po{};
    po.kind = GQ_PRE_SILU_MUL; po.K = (int)K;
    return gemv_grouped_allreduce_impl(x_dev, M, K, ldx, packed_dev, desc_dev, n_desc, split, run_info, y_dev, ldy, n_total, workspace_dev,
                                       workspace_bytes, rank, world, peer_buffers, max_m, max_n_total, stream, &po);
}

// ---- small-message all-reduce over peer memory (tensor-parallel row-parallel layers) ---------------------
// One-shot, push based: every rank stores its bf16 vector into its slot of every peer's buffer (plain stores
// over NVLink into memory the peers mapped for each other), publishes a per-CTA flag, waits — with a limit —
// for the peers' flags, and sums the slots from its OWN memory in rank order (deterministic, fp32, one bf16
// rounding).  No loads from remote memory, no multicast.  Two slot sets alternate by call parity; the call
// number lives in device memory (one counter per CTA) so a captured CUDA graph replays correctly.
// The reference has no collective of its own on this path (docs/multi-gpu.md:8-13 leaves it to vLLM's NCCL).
#define GQ_AR_CTAS 32

struct ArPeers {
    uint8_t *buf[GQ_AR_MAX_WORLD];      // data area of each rank's buffer: [2 sets][world][slot_bytes]
    uint32_t *flags[GQ_AR_MAX_WORLD];   // flag area of each rank's buffer: [2 sets][world][GQ_AR_CTAS]
};

__global__ void __launch_bounds__(256) allreduce_push_kernel(const uint4 *__restrict__ in, uint4 *__restrict__ out, int64_t n_vec, int rank,
                                                             int world, ArPeers peers, int64_t slot_bytes, uint32_t *counters, int *status,
                                                             unsigned long long wait_ns) {
    __shared__ uint32_t s_seq;
    __shared__ int s_fail;
    const int c = blockIdx.x, G = gridDim.x;
    if (threadIdx.x == 0) { s_seq = counters[c] + 1; s_fail = 0; }
    __syncthreads();
    const uint32_t seq = s_seq, set = seq & 1u;
    const int64_t per = (n_vec + G - 1) / G, v0 = (int64_t)c * per, v1 = v0 + per < n_vec ? v0 + per : n_vec;
    // push this CTA's share of the vector into slot `rank` of every rank's buffer (own included)
    for (int p = 0; p < world; ++p) {
        uint4 *dst = reinterpret_cast<uint4 *>(peers.buf[p] + ((int64_t)set * world + rank) * slot_bytes);
        for (int64_t i = v0 + threadIdx.x; i < v1; i += 256) dst[i] = in[i];
    }
    __syncthreads();
    if ((int)threadIdx.x < world) {
        // release at system scope: the stores of this CTA (ordered before by the barrier) are visible to the peer
        // before the flag is; the matching acquire load on the peer's side orders its reads of the slot after it
        uint32_t *f = peers.flags[threadIdx.x] + ((int64_t)set * world + rank) * G + c;
        asm volatile("st.release.sys.global.u32 [%0], %1;" ::"l"(f), "r"(seq) : "memory");
        const uint32_t *mine = peers.flags[rank] + ((int64_t)set * world + threadIdx.x) * G + c;
        uint32_t v;
        uint64_t t0 = 0;
        for (uint32_t it = 0;; ++it) {
            asm volatile("ld.acquire.sys.global.u32 %0, [%1];" : "=r"(v) : "l"(mine) : "memory");
            if (v == seq) break;
            if ((it & 255u) == 255u) {      // the clock is read only once a wait has become long
                const uint64_t now = global_timer_ns();
                if (t0 == 0) t0 = now;
                if (now - t0 > wait_ns || it > GQ_SPIN_LIMIT) { s_fail = 1; break; }
            }
        }
    }
    __syncthreads();
    if (s_fail) {
        if (threadIdx.x == 0) { report_status(status, GQ_DEV_TIMEOUT); counters[c] = seq; }
        return;
    }
    const uint8_t *base = peers.buf[rank] + (int64_t)set * world * slot_bytes;
    for (int64_t i = v0 + threadIdx.x; i < v1; i += 256) {
        float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
        // all ranks' vectors are requested before any is added (one trip to the L2 instead of one per rank)
        uint4 v[GQ_AR_MAX_WORLD];
#pragma unroll
        for (int r = 0; r < GQ_AR_MAX_WORLD; ++r)
            if (r < world) v[r] = __ldcg(reinterpret_cast<const uint4 *>(base + (int64_t)r * slot_bytes) + i);
#pragma unroll
        for (int r = 0; r < GQ_AR_MAX_WORLD; ++r) {
            if (r < world) {
                const __nv_bfloat162 *b = reinterpret_cast<const __nv_bfloat162 *>(&v[r]);
#pragma unroll
                for (int j = 0; j < 4; ++j) { const float2 f = __bfloat1622float2(b[j]); acc[2 * j] += f.x; acc[2 * j + 1] += f.y; }
            }
        }
        uint4 o;
        __nv_bfloat162 *ob = reinterpret_cast<__nv_bfloat162 *>(&o);
#pragma unroll
        for (int j = 0; j < 4; ++j) ob[j] = __floats2bfloat162_rn(acc[2 * j], acc[2 * j + 1]);
        out[i] = o;
    }
    if (threadIdx.x == 0) counters[c] = seq;
}

extern "C" int64_t gq_allreduce_buffer_bytes(int world, int64_t max_bytes) {
    if (world < 1 || world > GQ_AR_MAX_WORLD || max_bytes <= 0) return GQ_ERR_ARG;
    const int64_t slot = align256(max_bytes);
    // [flags 2*world*CTAS u32 | counters CTAS u32 | status] padded to 4096, then data 2 * world * slot
    return 4096 + 2 * (int64_t)world * slot;
}

extern "C" int gq_allreduce_push(const void *in_dev, void *out_dev, int64_t n_bytes, int rank, int world, const uint64_t *peer_buffers,
                                 int64_t max_bytes, void *stream) {
    if (world < 1 || world > GQ_AR_MAX_WORLD || rank < 0 || rank >= world) return GQ_ERR_ARG;
    if (n_bytes < 0 || n_bytes > max_bytes || (n_bytes & 15)) return GQ_ERR_SHAPE;
    if (n_bytes == 0) return GQ_OK;
    if (!in_dev || !out_dev || !peer_buffers || ((uintptr_t)in_dev & 15) || ((uintptr_t)out_dev & 15)) return GQ_ERR_ARG;
    ArPeers peers;
    for (int p = 0; p < GQ_AR_MAX_WORLD; ++p) { peers.buf[p] = nullptr; peers.flags[p] = nullptr; }
    for (int p = 0; p < world; ++p) {
        if (!peer_buffers[p] || (peer_buffers[p] & 255)) return GQ_ERR_ARG;
        peers.flags[p] = reinterpret_cast<uint32_t *>(peer_buffers[p]);
        peers.buf[p] = reinterpret_cast<uint8_t *>(peer_buffers[p]) + 4096;
    }
    uint8_t *own = reinterpret_cast<uint8_t *>(peer_buffers[rank]);
    uint32_t *counters = reinterpret_cast<uint32_t *>(own + 2 * GQ_AR_MAX_WORLD * GQ_AR_CTAS * 4);
    int *status = reinterpret_cast<int *>(own + 2 * GQ_AR_MAX_WORLD * GQ_AR_CTAS * 4 + GQ_AR_CTAS * 4);
    allreduce_push_kernel<<<GQ_AR_CTAS, 256, 0, (cudaStream_t)stream>>>((const uint4 *)in_dev, (uint4 *)out_dev, n_bytes / 16, rank, world, peers,
                                                                     align256(max_bytes), counters, status, g_peer_wait_ns.load());
    GQ_LAUNCHED();
    return GQ_OK;
}

// ---- prefill ----------------------------------------------------------------------------------------
// Dynamic shared memory of a CTA: two CTAs (SETS = 1) or one fill the SM, so that no third user of tensor memory joins them:
// the CTAs of a cluster wait for one another while they hold theirs.
#define GQ_PF_SMEM_1 (111 * 1024)
#define GQ_PF_SMEM_2 (225 * 1024)

// How a prefill launch is cut: N batch rows per CTA (a multiple of 16, tiles balanced), the cluster split of K, and which of
// the kernel's shapes runs it.
struct PrefillPlan {
    int sets, wide, N, tiles, split;
};
static PrefillPlan prefill_shape(int64_t M, int64_t tiles) {
    PrefillPlan p;
    const int64_t rows = (M + tiles - 1) / tiles;
    p.wide = rows > 256;
    p.N = (int)(p.wide ? (rows + 31) & ~31 : (rows + 15) & ~15);
    p.tiles = (int)((M + p.N - 1) / p.N);       // (the steps of N may make the last of many tiles superfluous: each has a row of the batch)
    p.sets = p.N <= 128 ? 1 : 2;
    p.split = 1;
    return p;
}
// CTAs of one batch tile and one part of K: two 64-row tiles each, in pairs where the MMAs span a pair
static int64_t prefill_ctas(int64_t n_desc, const PrefillPlan &p) { return p.sets == 1 ? (n_desc + 1) / 2 : (n_desc + 3) / 4 * 2; }
// Every batch tile decodes the weights again, so there are as few as fit (384 rows each) up to what 256-row tiles would need;
// K is split over a cluster, at least four k-blocks to a CTA and eight in the run.  Both are chosen by the cycles that the waves
// of the launch take: a k-block costs a CTA its MMAs (7.8 N cycles) or its share of the decoding (2700 cycles alone on an SM,
// 4200 where two CTAs share one), whichever is longer, and a wave its start-up and its drain (5000 cycles and 25 a batch row).
static PrefillPlan prefill_plan(int64_t n_desc, int64_t M, int64_t nb, int sms) {
    PrefillPlan best = prefill_shape(M, (M + 255) / 256);
    if (sms <= 0) sms = 148;
    double best_cost = 1e300;
    for (int64_t tiles = (M + 383) / 384; tiles <= (M + 255) / 256; ++tiles) {
        PrefillPlan p = prefill_shape(M, tiles);
        const int64_t ctas = prefill_ctas(n_desc, p) * p.tiles;
        const double mma = 7.8 * p.N + 300.0, decode = p.sets == 1 ? 4200.0 : 2700.0, per_kb = mma > decode ? mma : decode;
        for (int S = 1; S * p.sets <= 8 && (S == 1 || (int64_t)S * 4 <= nb); ++S) {
            // clusters of a unit's parts that the GPU holds side by side: of CTAs short of the last places (ctas_per_sm_for), of pairs, one
            // CTA to an SM, all (32 of 33 and 14 of 15 run as one wave; 34 of two pairs, 8,704 x 5,120 Q4_K at 300 rows, took 55 us where 34
            // whole pairs take 31)
            const int64_t places = cluster_places(p.sets == 1 ? 2 : 1, S * p.sets, sms);
            if (places == 0 && S > 1) break;        // so few SMs hold no such cluster, and no larger one
            const int64_t held = (places ? places : 1) * (p.sets == 1 && S > 1 ? 93 : 100), clusters = ctas / p.sets * 100;
            const int64_t waves = (clusters + held - 1) / held;
            const double cost = (double)waves * ((double)((nb + S - 1) / S) * per_kb + 5000.0 + 25.0 * p.N + (S > 1 ? 6000.0 : 0.0));
            if (cost < best_cost * (1.0 - 1e-9)) { best_cost = cost; best = p; best.split = S; }
        }
    }
    return best;
}

// CTAs to a row of the activation preparation (prep_x_prefill_kernel; `rows` of the padded batch): as many as hold it, up to four of them per
// SM in all, and two while the GPU holds twice the rows (nine CTAs per SM; short of the last of them unless a row fills three).  One up to
// 8,192 activations, where a cluster costs more than the second reading of what one CTA does not keep, unless all of them get an SM of
// their own.  Whole calls with 1 / 2 / 3 / 4 CTAs: 5,120 x 17,408 at 64 rows 32.3 / 30.2 / 29.4 / 29.0 us, at 384 71.1 / 66.5 / 66.7 / 66.9,
// at 600 113.3 / 109.3; 2,048 x 17,408 at 384 57.8 / 55.9 / 58.4; 2,048 x 8,704 at 600 54.4 / 57.4; 5,120 x 6,144 at 160 18.9 / 20.5;
// 2,048 x 7,680 at 64 15.5 / 13.5, at 128 17.4 / 19.5.
static int prefill_prep_parts(int64_t K, int64_t rows, int sms) {
    const int64_t per = GQ_PF_PREP_THREADS * GQ_PF_PREP_VECS * 8;
    if (K < 8192 && !(K >= per + per / 2 && 2 * rows <= sms)) return 1;
    int64_t parts = 4 * (int64_t)sms / rows;
    if (parts < 2) parts = 2 * rows <= (int64_t)sms * (K >= 3 * per ? GQ_PF_PREP_CTAS : GQ_PF_PREP_CTAS - 1) ? 2 : 1;
    if (parts > (K + per - 1) / per) parts = (K + per - 1) / per;
    return (int)(parts > 8 ? 8 : parts);
}

static int64_t pf_ws_layout(int64_t K, const PrefillPlan &pl, void *base, int **status, float **ex, uint8_t **xp) {
    const int64_t rows = (int64_t)pl.tiles * pl.N;
    int64_t off = 256;
    const int64_t o_ex = off; off = align256(off + rows * 4);
    off = (off + 1023) & ~(int64_t)1023;
    const int64_t o_xp = off; off += rows * K * 2;
    if (base) { uint8_t *b = (uint8_t *)base; *status = (int *)b; *ex = (float *)(b + o_ex); *xp = b + o_xp; }
    return off;
}

extern "C" int gq_prefill_plan(int64_t M, int64_t K, int64_t n_desc, int sm_count, int32_t *plan) {
    if (M <= 0 || K <= 0 || K % GQ_QK || n_desc <= 0) return GQ_ERR_SHAPE;
    if (!plan) return GQ_ERR_ARG;
    const PrefillPlan p = prefill_plan(n_desc, M, K / GQ_QK, sm_count);
    plan[0] = p.N; plan[1] = p.tiles; plan[2] = p.split; plan[3] = p.sets; plan[4] = p.wide;
    return GQ_OK;
}

extern "C" int64_t gq_prefill_workspace_bytes(int64_t M, int64_t K, int64_t n_total, int64_t n_desc) {
    if (M < 0 || K <= 0 || K % GQ_QK || n_total < 0 || n_desc < 0) return GQ_ERR_SHAPE;
    if (M == 0) return 256;
    return pf_ws_layout(K, prefill_plan(n_desc, M, K / GQ_QK, device_sms()), nullptr, nullptr, nullptr, nullptr);
}

template <int SETS, bool WIDE, int SL>
static int launch_prefill_kernel(PrefillParams &p, const PrefillPlan &pl, int smem, bool reverse, cudaStream_t st) {
    if (int rc = allow_smem<gemm_prefill_kernel<SETS, WIDE, SL>>(smem)) return rc;
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[2];
    int na = 0;
    if (pl.split * SETS > 1) {
        attr[na].id = cudaLaunchAttributeClusterDimension;
        attr[na].val.clusterDim.x = (unsigned)(pl.split * SETS); attr[na].val.clusterDim.y = 1; attr[na].val.clusterDim.z = 1;
        ++na;
    }
    attr[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[na].val.programmaticStreamSerializationAllowed = 1;
    ++na;
    cfg.blockDim = dim3(32 * (8 * SETS + 3)); cfg.dynamicSmemBytes = (size_t)smem; cfg.stream = st; cfg.attrs = attr; cfg.numAttrs = na;
    // a grid has room for 65,535 units (8.4 or 16.8 million output columns): a run of more takes several launches
    const int64_t n_desc = p.n_desc, step = (int64_t)65535 * 2 * SETS;
    for (int64_t d = 0; d < n_desc; d += step, p.desc += step * GQ_DESC_WORDS) {
        p.n_desc = (int)(n_desc - d < step ? n_desc - d : step);
        cfg.gridDim = dim3((unsigned)(pl.split * SETS), (unsigned)(prefill_ctas(p.n_desc, pl) / SETS), (unsigned)pl.tiles);
        p.unit0 = reverse ? (int)cfg.gridDim.y - 1 : 0; p.unit_step = reverse ? -1 : 1;
        GQ_CUDA(cudaLaunchKernelEx(&cfg, gemm_prefill_kernel<SETS, WIDE, SL>, p));
        GQ_LAUNCHED();
    }
    return GQ_OK;
}

template <int SETS, bool WIDE>
static int launch_prefill(PrefillParams &p, const PrefillPlan &pl, int maxb, int run_info, cudaStream_t st) {
    const int total = SETS == 1 ? GQ_PF_SMEM_1 : GQ_PF_SMEM_2, tables = gq_cb_region_sum(p.cb_mask), bbytes = pl.N * 128 / SETS;
    p.wstage_bytes = 128 * maxb;
    // the activation ring takes four slices (one k-block), the weight ring the rest; a run whose widest type leaves no two
    // weight stages beside them takes activation stages away, down to two
    int left = total - 1024 - tables;
    p.bstages = 4;
    while (p.bstages > 2 && (left - p.bstages * bbytes) / p.wstage_bytes < 2) --p.bstages;
    p.wstages = (left - p.bstages * bbytes) / p.wstage_bytes;
    if (p.wstages > GQ_PF_MAX_STAGES) p.wstages = GQ_PF_MAX_STAGES;
    p.wstages -= p.wstages % SETS;        // each set walks stages of its own
    if (p.wstages < 1) return GQ_ERR_LIMIT;
    left -= p.wstages * p.wstage_bytes + p.bstages * bbytes;
    while (p.bstages < GQ_PF_SLOTS * (WIDE ? 1 : SETS) && left >= bbytes) { ++p.bstages; left -= bbytes; }
    const bool reverse = SETS == 1 && (run_info & GQ_ORDER_128);
    if constexpr (SETS == 1) {
        if ((p.bstages == GQ_PF_SLOTS || p.cb_mask) && !(((run_info >> 17) & 31) == GQ_Q4_0 && pl.N > 64))
            return launch_prefill_kernel<SETS, WIDE, 2>(p, pl, total, reverse, st);
    }
    return launch_prefill_kernel<SETS, WIDE, 1>(p, pl, total, reverse, st);
}

extern "C" int gq_gemm_prefill(const void *x_dev, int64_t M, int64_t K, int64_t ldx, const void *packed_dev, const int32_t *desc_dev,
                               int64_t n_desc, int run_info, void *y_dev, int64_t ldy, int64_t n_total, void *workspace_dev,
                               int64_t workspace_bytes, void *stream) {
    if (M < 0 || K <= 0 || K % GQ_QK || n_total < 0 || n_desc < 0) return GQ_ERR_SHAPE;
    if (M == 0 || n_total == 0 || n_desc == 0) return GQ_OK;
    if (!x_dev || !packed_dev || !desc_dev || !y_dev || !workspace_dev) return GQ_ERR_ARG;
    if (((uintptr_t)packed_dev & 15) || ((uintptr_t)workspace_dev & 1023) || ((uintptr_t)x_dev & 15) || (ldx & 7) || ldx < K || ldy < n_total)
        return GQ_ERR_ARG;
    if (n_desc > 0x7ffffffe || M > (int64_t)65535 * 64) return GQ_ERR_LIMIT;
    const int maxb = run_info & 0xFFFF;
    if (maxb < 56 || maxb > 272 || (maxb & 1)) return GQ_ERR_ARG;
    const PrefillPlan pl = prefill_plan(n_desc, M, K / GQ_QK, device_sms());
    int *status; float *ex; uint8_t *xp;
    const int64_t need = pf_ws_layout(K, pl, workspace_dev, &status, &ex, &xp);
    if (workspace_bytes < need) return GQ_ERR_WORKSPACE;
    if (int rc = ensure_tables()) return rc;
    PrefillParams p = {};
    p.packed = (const uint8_t *)packed_dev; p.desc = desc_dev; p.n_desc = (int)n_desc; p.xp = xp; p.ex = ex;
    p.y = (__nv_bfloat16 *)y_dev; p.ldy = ldy; p.M = (int)M; p.nb = (int)(K / GQ_QK); p.N = pl.N; p.status = status;
    p.split = pl.split; p.cb_mask = (run_info >> 22) & 63;
    for (int t = 0; t < 32; ++t) {
        const int kind = gq_cb_kind(t);
        p.half_bytes[t] = (uint8_t)(gq_type_bytes(t) / 2);
        p.cb_at[t] = (uint16_t)(kind < 0 ? 0 : (p.cb_mask >> kind) & 1 ? gq_cb_offset(p.cb_mask, kind) / 16 + 2 : 1);
    }
    cudaStream_t st = (cudaStream_t)stream;
    {
        cudaLaunchConfig_t cfg = {};
        cudaLaunchAttribute attr[2];
        attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[0].val.programmaticStreamSerializationAllowed = 1;
        const int parts = prefill_prep_parts(K, (int64_t)pl.tiles * pl.N, device_sms());
        attr[1].id = cudaLaunchAttributeClusterDimension;
        attr[1].val.clusterDim.x = 1; attr[1].val.clusterDim.y = (unsigned)parts; attr[1].val.clusterDim.z = 1;
        cfg.gridDim = dim3((unsigned)(pl.tiles * pl.N), (unsigned)parts); cfg.blockDim = dim3(GQ_PF_PREP_THREADS); cfg.stream = st; cfg.attrs = attr;
        cfg.numAttrs = parts > 1 ? 2 : 1;
        GQ_CUDA(cudaLaunchKernelEx(&cfg, prep_x_prefill_kernel, (const __nv_bfloat16 *)x_dev, ldx, (int)K, (int)M, pl.N, pl.sets == 1 ? 0 : pl.wide ? pl.N / 2 : pl.N, ex, xp, status));
        GQ_LAUNCHED();
    }
    if (pl.wide) return launch_prefill<2, true>(p, pl, maxb, run_info, st);
    return pl.sets == 1 ? launch_prefill<1, false>(p, pl, maxb, run_info, st) : launch_prefill<2, false>(p, pl, maxb, run_info, st);
}

extern "C" int gq_device_status(int clear, void *stream) {
    int v = 0;
    GQ_CUDA(cudaMemcpyFromSymbolAsync(&v, g_sticky_status, sizeof v, 0, cudaMemcpyDeviceToHost, (cudaStream_t)stream));
    GQ_CUDA(cudaStreamSynchronize((cudaStream_t)stream));
    if (clear && v != 0) {
        const int zero = 0;
        GQ_CUDA(cudaMemcpyToSymbolAsync(g_sticky_status, &zero, sizeof zero, 0, cudaMemcpyHostToDevice, (cudaStream_t)stream));
        GQ_CUDA(cudaStreamSynchronize((cudaStream_t)stream));
    }
    return v;
}

extern "C" int gq_set_peer_wait_limit_ns(int64_t ns) {
    if (ns < 1000 || ns > 60000000000ll) return GQ_ERR_ARG;
    g_peer_wait_ns.store((unsigned long long)ns);
    return GQ_OK;
}

extern "C" int gq_read_status(const void *workspace_dev, int64_t workspace_bytes, void *stream) {
    if (!workspace_dev || workspace_bytes < 256) return GQ_ERR_ARG;
    int v = 0;
    GQ_CUDA(cudaMemcpyAsync(&v, workspace_dev, sizeof v, cudaMemcpyDeviceToHost, (cudaStream_t)stream));
    GQ_CUDA(cudaStreamSynchronize((cudaStream_t)stream));
    return v;
}
