// Load-time and lookup kernels: raw GGUF rows -> tile-major slabs, slabs -> row-major weights, and the quantized embedding
// lookup (raw rows -> row-major weights, nothing stored in between).  All are bound by HBM; see each kernel for its split.
//
// Bit-exactness of the dequantisers.  The format reference computes fp32 (d * sc) * q, then - (dmin * m).  d has 11
// significant bits, a scale at most 8 and a weight at most 8, and the products that reach 24 bits still fit fp32, so
// (d * sc) * q is exact in any order of its factors and the only rounding is the final subtraction of the types that have a
// minimum.  The register decoders of gq_decode.cuh deliver q as an exact fp16 integer and sc as an exact float, so they
// serve here as they do in the matrix kernels.
// (included after gq_decode.cuh and the codebook tables)
#pragma once
#include "gq_decode.cuh"

namespace gq {

#define GQ_LOAD_THREADS 256
#define GQ_LOAD_WARPS (GQ_LOAD_THREADS / 32)

// the codebook table of TYPE for the fp16 decoders of gq_decode.cuh (gq_cb_bytes(kind) bytes of shared memory)
__device__ __forceinline__ void fill_codebook(int type, uint8_t *dst, int tid, int nthreads) {
    uint32_t *t32 = reinterpret_cast<uint32_t *>(dst);
    switch (type) {
        case GQ_IQ3_S: for (int i = tid; i < 512; i += nthreads) t32[i] = iq3s_grid_entry(c_iq3s_grid[i]); break;
        case GQ_IQ3_XXS: for (int i = tid; i < 256; i += nthreads) t32[i] = prmt(c_iq3xxs_grid[i], 0u, 0x3120u); break;
        case GQ_IQ2_XXS: for (int i = tid; i < 512; i += nthreads) t32[i] = prmt(c_iq2xxs_grid[i], 0u, 0x3120u); break;
        case GQ_IQ2_XS: for (int i = tid; i < 1024; i += nthreads) t32[i] = prmt(c_iq2xs_grid[i], 0u, 0x3120u); break;
        case GQ_IQ2_S: for (int i = tid; i < 2048; i += nthreads) t32[i] = prmt(c_iq2s_grid[i], 0u, 0x3120u); break;
        case GQ_IQ1_M: for (int i = tid; i < 4096; i += nthreads) t32[i] = prmt(c_iq1_grid[i], 0u, 0x3120u); break;
        default: break;
    }
}
// the IQ4 codebook as unsigned bytes (value + 128)
__device__ __forceinline__ Iq4Table iq4_table_biased() {
    uint32_t tb[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        tb[j] = 0;
#pragma unroll
        for (int i = 0; i < 4; ++i) tb[j] |= (uint32_t)(uint8_t)(c_iq4_kvalues[4 * j + i] + 128) << (8 * i);
    }
    return {tb[0], tb[1], tb[2], tb[3]};
}

// Sixteen rows' byte ranges [p_r, p_r + len) into shared memory, one warp per row and 16 bytes per lane whatever the rows'
// alignment: what is copied are the aligned 16-byte granules that hold the range, so byte b of row r lands at
// img + r * pitch + (p_r & 15) + b.  (A granule that holds a byte of an allocation lies inside it: device allocations start
// and end on 16-byte boundaries.)  row(r) == nullptr: zeros.
template <typename Row>
__device__ __forceinline__ void stage_rows(uint8_t *img, int pitch, int len, int warp, int lane, Row row) {
#pragma unroll
    for (int r = warp; r < 16; r += GQ_LOAD_WARPS) {
        const uint8_t *p = row(r);
        const int off = (int)(reinterpret_cast<uintptr_t>(p) & 15);
        const uint4 *a = reinterpret_cast<const uint4 *>(p - off);
        const int n = (off + len + 15) >> 4;
        uint4 *dst = reinterpret_cast<uint4 *>(img + r * pitch);
#pragma unroll 4
        for (int j = lane; j < n; j += 32) dst[j] = p ? __ldg(a + j) : make_uint4(0u, 0u, 0u, 0u);
    }
}
// row pitch for len bytes at any alignment: an odd number of 16-byte units, so that the rows start in different banks
__host__ __device__ constexpr int stage_pitch(int len) { return (((len + 15 + 15) >> 4) | 1) * 16; }

// the staged rows of n_kb k-blocks -> n_kb slabs of 16 * B bytes, one 4-byte word per thread and step.  The four source
// offsets of a word do not depend on the k-block: they are computed once (gq_slab_src with the type known at compile time)
// and serve all of them.
template <int TYPE, typename Row>
__device__ __forceinline__ void permute_slabs(const uint8_t *img, int pitch, int n_kb, uint8_t *dst, int64_t dst_stride, Row row) {
    constexpr int B = gq_type_bytes(TYPE);
    for (int w = threadIdx.x; w < 4 * B; w += GQ_LOAD_THREADS) {
        int s[4];
#pragma unroll
        for (int z = 0; z < 4; ++z) {
            int r, byte;
            gq_slab_src(TYPE, 4 * w + z, &r, &byte);
            s[z] = r * pitch + (int)(reinterpret_cast<uintptr_t>(row(r)) & 15) + byte;
        }
        // most words are four neighbouring bytes in another order; at an even address two halfword loads fetch them
        const int lo = min(min(s[0], s[1]), min(s[2], s[3])), hi = max(max(s[0], s[1]), max(s[2], s[3]));
        if (hi - lo == 3 && !(lo & 1)) {
            uint32_t sel = 0;
#pragma unroll
            for (int z = 0; z < 4; ++z) sel |= (uint32_t)(s[z] - lo + ((s[z] - lo) & 2)) << (4 * z);      // 0 1 | 4 5: bytes of the two halfwords
            const uint8_t *a = img + lo;
#pragma unroll 4
            for (int kb = 0; kb < n_kb; ++kb)
                *reinterpret_cast<uint32_t *>(dst + kb * dst_stride + 4 * w) =
                    prmt(*reinterpret_cast<const uint16_t *>(a + kb * B), *reinterpret_cast<const uint16_t *>(a + kb * B + 2), sel);
        } else {
#pragma unroll 4
            for (int kb = 0; kb < n_kb; ++kb) {
                const uint8_t *b = img + kb * B;
                *reinterpret_cast<uint32_t *>(dst + kb * dst_stride + 4 * w) =
                    (uint32_t)b[s[0]] | (uint32_t)b[s[1]] << 8 | (uint32_t)b[s[2]] << 16 | (uint32_t)b[s[3]] << 24;
            }
        }
    }
}

// k-blocks a repack CTA takes: about 2 KB of every row
template <int TYPE>
constexpr int repack_kc() { return gq_type_bytes(TYPE) > 128 ? 8 : 16; }

// ---- repack: one CTA per (16-row slab, up to KC k-blocks) ------------------------------------------------------
// Bound by HBM (raw bytes in and out).  A CTA reads KC * B contiguous bytes of each row with 16-byte loads and writes its
// slabs as full 128-byte lines; the previous kernel took one k-block of 56..272 bytes per row byte by byte and evaluated the
// layout function for every byte.  17408 x 5120 IQ3_S / Q5_K: 23 / 46 us = 3.3 / 2.7 TB/s in and out (before: 223 on
// average); what remains is the byte gather from shared memory.
template <int TYPE>
__global__ void __launch_bounds__(GQ_LOAD_THREADS) repack_kernel(const uint8_t *__restrict__ raw, int64_t n_out, int nb, int64_t row_stride,
                                                                 uint8_t *__restrict__ out) {
    extern __shared__ __align__(16) uint8_t img[];
    constexpr int B = gq_type_bytes(TYPE), KC = repack_kc<TYPE>();
    const int slab = blockIdx.x, kb0 = blockIdx.y * KC, n_kb = nb - kb0 < KC ? nb - kb0 : KC;
    const int pitch = stage_pitch(KC * B);
    const int64_t row0 = (int64_t)slab * 16;
    const auto row = [&](int r) -> const uint8_t * {
        return row0 + r < n_out ? raw + (row0 + r) * row_stride + (int64_t)kb0 * B : (const uint8_t *)nullptr;
    };
    stage_rows(img, pitch, n_kb * B, threadIdx.x >> 5, threadIdx.x & 31, row);
    __syncthreads();
    // packed address: tile = slab / 4, slab-in-tile = slab % 4
    uint8_t *dst = out + (((int64_t)(slab >> 2) * nb + kb0) * 4 + (slab & 3)) * (int64_t)(16 * B);
    permute_slabs<TYPE>(img, pitch, n_kb, dst, (int64_t)64 * B, row);
}

// ---- dequantise: one warp per (slab, k-block) ------------------------------------------------------------------
// the fp32 weights of run pair P (32 weights, the lane's four of each run, rows g and g + 8): v[u][h][0..3]
template <int TYPE, int P>
__device__ __forceinline__ void dequant_pair(const Dec<TYPE> &dec, float (&v)[2][2][4]) {
    uint32_t a[2][4];
    dec.template pair<P>(a);
    float d[2];
    dec.kscale(d[0], d[1]);
#pragma unroll
    for (int u = 0; u < 2; ++u) {
        float s[2], m[2] = {0.f, 0.f};
        constexpr bool G32 = Dec<TYPE>::GROUP == 32;
        if (u == 0) {
            dec.template scale<G32 ? P : 2 * P>(s[0], s[1]);
            if constexpr (Dec<TYPE>::HAS_MIN) dec.template minterm<G32 ? P : 2 * P>(m[0], m[1]);
        } else {
            dec.template scale<G32 ? P : 2 * P + 1>(s[0], s[1]);
            if constexpr (Dec<TYPE>::HAS_MIN) dec.template minterm<G32 ? P : 2 * P + 1>(m[0], m[1]);
        }
        constexpr float off = Dec<TYPE>::template offs<2 * P>();
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const float ds = __fmul_rn(d[h], s[h]);
            uint32_t w01 = a[u][h], w23 = a[u][2 + h];
            if constexpr (off != 0.0f) { w01 = hsub2(w01, h2k(off)); w23 = hsub2(w23, h2k(off)); }
            const float q[4] = {f16lo(w01), f16hi(w01), f16lo(w23), f16hi(w23)};
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                v[u][h][j] = __fmul_rn(ds, q[j]);
                if constexpr (Dec<TYPE>::HAS_MIN) v[u][h][j] = __fsub_rn(v[u][h][j], m[h]);
            }
        }
    }
}

// Row pitch of a warp's staging area for 128 bf16 columns of 16 rows: 288 bytes = 8 banks mod 32, so the 8-byte stores of
// four rows fill the 32 banks once; read back it gives whole rows, two of 256 contiguous bytes per store instruction.
#define GQ_DEQ_PITCH 288
#define GQ_DEQ_STAGE (16 * GQ_DEQ_PITCH)

// one slab's k-block as rows of the output: out points at (row 0 of the slab, first column of the k-block)
template <int TYPE, bool BF16>
__device__ __forceinline__ void dequant_slab(const uint8_t *slab, const DecAux &aux, int lane, uint8_t *stage, void *out, int64_t ld, int rows, bool vec) {
    Dec<TYPE> dec;
    dec.load(slab, lane, aux);
    const int g = lane >> 2, t = lane & 3;
#define GQ_DEQ_PAIR(P)                                                                                                       \
    {                                                                                                                        \
        float v[2][2][4];                                                                                                    \
        dequant_pair<TYPE, P>(dec, v);                                                                                       \
        _Pragma("unroll") for (int u = 0; u < 2; ++u) _Pragma("unroll") for (int h = 0; h < 2; ++h) {                         \
            if constexpr (BF16) {                                                                                            \
                __nv_bfloat162 b[2] = {__floats2bfloat162_rn(v[u][h][0], v[u][h][1]), __floats2bfloat162_rn(v[u][h][2], v[u][h][3])}; \
                *reinterpret_cast<uint2 *>(stage + (g + 8 * h) * GQ_DEQ_PITCH + 2 * (32 * ((P) & 3) + 16 * u + 4 * t)) =     \
                    *reinterpret_cast<uint2 *>(b);                                                                           \
            } else if (g + 8 * h < rows) {                                                                                   \
                float *o = reinterpret_cast<float *>(out) + (g + 8 * h) * ld + 32 * (P) + 16 * u + 4 * t;                    \
                if (vec) *reinterpret_cast<float4 *>(o) = make_float4(v[u][h][0], v[u][h][1], v[u][h][2], v[u][h][3]);       \
                else { o[0] = v[u][h][0]; o[1] = v[u][h][1]; o[2] = v[u][h][2]; o[3] = v[u][h][3]; }                         \
            }                                                                                                                \
        }                                                                                                                    \
    }
    const auto flush = [&](int half) {
        if constexpr (BF16) {
            __syncwarp();
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const int r = 2 * i + (lane >> 4), c = 8 * (lane & 15);
                const uint4 w = *reinterpret_cast<const uint4 *>(stage + r * GQ_DEQ_PITCH + 2 * c);
                if (r < rows) {
                    __nv_bfloat16 *o = reinterpret_cast<__nv_bfloat16 *>(out) + r * ld + 128 * half + c;
                    if (vec) *reinterpret_cast<uint4 *>(o) = w;
                    else {
                        const __nv_bfloat16 *e = reinterpret_cast<const __nv_bfloat16 *>(&w);
#pragma unroll
                        for (int j = 0; j < 8; ++j) o[j] = e[j];
                    }
                }
            }
            __syncwarp();
        }
    };
    GQ_DEQ_PAIR(0) GQ_DEQ_PAIR(1) GQ_DEQ_PAIR(2) GQ_DEQ_PAIR(3)
    flush(0);
    GQ_DEQ_PAIR(4) GQ_DEQ_PAIR(5) GQ_DEQ_PAIR(6) GQ_DEQ_PAIR(7)
    flush(1);
#undef GQ_DEQ_PAIR
}

// packed tiles -> row-major fp32 or bf16.  grid (slabs, k parts); a CTA's warps take the k-blocks of its part in turn.
// Bound by HBM (the bf16 output is 3.6x the packed bytes of a 4.5-bit type); the previous kernel turned the slab back into
// raw order in shared memory and decoded every weight on its own from there.  17408 x 5120 Q5_K to bf16: 50 us = 4.8 TB/s
// (before: 406 us).
// (CTAs per SM that the compiler leaves registers for: its own choice, except where that is four with a spill: 17,408 x 5,120 IQ2_S 49.2 us,
// with three 46.5)
template <int TYPE, bool BF16>
__global__ void __launch_bounds__(GQ_LOAD_THREADS, BF16 && TYPE == GQ_IQ2_S ? 3 : 0) dequant_kernel(const uint8_t *__restrict__ tiles, int64_t n_out, int nb, int kc, void *__restrict__ out,
                                                                  int64_t ld) {
    constexpr int B = gq_type_bytes(TYPE), CB = gq_cb_kind(TYPE) >= 0 ? gq_cb_bytes(gq_cb_kind(TYPE)) : 0;
    extern __shared__ __align__(16) uint8_t sm[];       // [codebook][the warps' output staging]
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, slab = blockIdx.x;
    if constexpr (CB > 0) {
        fill_codebook(TYPE, sm, threadIdx.x, GQ_LOAD_THREADS);
        __syncthreads();
    }
    DecAux aux;
    aux.grid = reinterpret_cast<const uint32_t *>(sm);
    aux.iq4 = iq4_table_biased();
    const int64_t row0 = (int64_t)slab * 16;
    const int rows = n_out - row0 < 16 ? (n_out - row0 > 0 ? (int)(n_out - row0) : 0) : 16;
    if (rows == 0) return;
    const int k1 = ((int)blockIdx.y + 1) * kc < nb ? ((int)blockIdx.y + 1) * kc : nb;
    const bool vec = !((reinterpret_cast<uintptr_t>(out) & 15) | ((ld * (BF16 ? 2 : 4)) & 15));
    for (int kb = blockIdx.y * kc + warp; kb < k1; kb += GQ_LOAD_WARPS) {
        const uint8_t *src = tiles + (((int64_t)(slab >> 2) * nb + kb) * 4 + (slab & 3)) * (int64_t)(16 * B);
        uint8_t *o = reinterpret_cast<uint8_t *>(out) + (row0 * ld + (int64_t)kb * 256) * (BF16 ? 2 : 4);
        dequant_slab<TYPE, BF16>(src, aux, lane, sm + CB + warp * (BF16 ? GQ_DEQ_STAGE : 0), o, ld, rows, vec);
    }
}

template <int TYPE, bool BF16>
constexpr int dequant_smem() { return (gq_cb_kind(TYPE) >= 0 ? gq_cb_bytes(gq_cb_kind(TYPE)) : 0) + (BF16 ? GQ_LOAD_WARPS * GQ_DEQ_STAGE : 0); }
template <int TYPE>
constexpr int dequant_rows_smem() {
    const int img = 16 * stage_pitch(GQ_LOAD_WARPS * gq_type_bytes(TYPE)), st = GQ_LOAD_WARPS * GQ_DEQ_STAGE;
    return (img > st ? img : st) + GQ_LOAD_WARPS * 16 * gq_type_bytes(TYPE) + (gq_cb_kind(TYPE) >= 0 ? gq_cb_bytes(gq_cb_kind(TYPE)) : 0);
}
// ---- embedding lookup: rows `ids` of a raw table -> row-major weights --------------------------------------------
// One CTA takes sixteen ids and up to eight k-blocks: the raw bytes are gathered into shared memory, permuted into slabs
// there, and each warp decodes one k-block.  One launch and one pass over memory; gathering, repacking and dequantising as
// three kernels cost 80 us for 2048 IQ2_S rows of 5120 (24 MB), this one 10.6.  An id outside the table is reported, its row is not read,
// its output is NaN.
template <int TYPE, bool BF16>
__global__ void __launch_bounds__(GQ_LOAD_THREADS) dequant_rows_kernel(const uint8_t *__restrict__ raw, int64_t n_rows, int nb, int64_t row_stride,
                                                                       const void *__restrict__ ids, int ids64, int64_t n_ids, void *__restrict__ out,
                                                                       int64_t ld) {
    extern __shared__ __align__(16) uint8_t dyn[];      // [rows as staged | later the warps' output staging][slabs][codebook]
    constexpr int B = gq_type_bytes(TYPE), KC = GQ_LOAD_WARPS;
    constexpr int pitch = stage_pitch(KC * B), IMG = 16 * pitch > KC * GQ_DEQ_STAGE ? 16 * pitch : KC * GQ_DEQ_STAGE;
    __shared__ int64_t s_id[16];
    uint8_t *slabs = dyn + IMG, *cb = slabs + KC * 16 * B;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int kb0 = blockIdx.y * KC, n_kb = nb - kb0 < KC ? nb - kb0 : KC;
    const int64_t i0 = (int64_t)blockIdx.x * 16;
    const int rows = n_ids - i0 < 16 ? (int)(n_ids - i0) : 16;
    if (threadIdx.x < 16) {
        int64_t id = -1;
        if ((int)threadIdx.x < rows) {
            id = ids64 ? reinterpret_cast<const int64_t *>(ids)[i0 + threadIdx.x] : (int64_t)reinterpret_cast<const int32_t *>(ids)[i0 + threadIdx.x];
            if (id < 0 || id >= n_rows) { atomicMax(&g_sticky_status, GQ_DEV_BAD_SHAPE); id = -1; }
        }
        s_id[threadIdx.x] = id;
    }
    fill_codebook(TYPE, cb, threadIdx.x, GQ_LOAD_THREADS);
    __syncthreads();
    const auto row = [&](int r) -> const uint8_t * { return s_id[r] >= 0 ? raw + s_id[r] * row_stride + (int64_t)kb0 * B : (const uint8_t *)nullptr; };
    stage_rows(dyn, pitch, n_kb * B, warp, lane, row);
    __syncthreads();
    permute_slabs<TYPE>(dyn, pitch, n_kb, slabs, 16 * B, row);
    __syncthreads();
    if (warp >= n_kb) return;
    DecAux aux;
    aux.grid = reinterpret_cast<const uint32_t *>(cb);
    aux.iq4 = iq4_table_biased();
    const bool vec = !((reinterpret_cast<uintptr_t>(out) & 15) | ((ld * (BF16 ? 2 : 4)) & 15));
    uint8_t *o = reinterpret_cast<uint8_t *>(out) + (i0 * ld + (int64_t)(kb0 + warp) * 256) * (BF16 ? 2 : 4);
    dequant_slab<TYPE, BF16>(slabs + warp * 16 * B, aux, lane, dyn + warp * GQ_DEQ_STAGE, o, ld, rows, vec);
    __syncwarp();
    for (int r = 0; r < rows; ++r)
        if (s_id[r] < 0)
            for (int c = lane; c < 256; c += 32) {
                if constexpr (BF16) reinterpret_cast<uint16_t *>(o)[r * ld + c] = 0x7fc0u;
                else reinterpret_cast<uint32_t *>(o)[r * ld + c] = 0x7fc00000u;
            }
}

}  // namespace gq
