// Large-batch (prefill) path: packed weights are dequantised in registers, stored into TENSOR MEMORY as the A operand of
// tcgen05.mma, and multiplied there; the accumulator lives in tensor memory too.  Replaces the reference's wide forms and its
// dequantise-then-cuBLAS path (gguf-plugin/gluon/interface.py:159-188, gguf-plugin/gluon/tiles.py:141-149): the dequantised
// weights touch neither HBM nor shared memory.
//
// Why tensor memory.  The lane-ordered slab layout was made for mma.sync fragments: lane 4g + t holds rows g and g + 8,
// weights 4t .. 4t+3 of a 16-weight run.  tcgen05.st.16x256b writes exactly that fragment — a run is one 256-bit row segment
// of sixteen TMEM lanes — so a slab's 64-wide k-slice is ONE store instruction of sixteen registers, without a swizzle, bank
// conflicts or a proxy fence, and the tensor core reads A at no shared-memory bandwidth: an MMA of M = 128, K = 16 takes
// 12 / 17 / 32 / 63 / 125 cycles at N = 16 / 32 / 64 / 128 / 256, with A in shared memory 40 / 40 / 48 / 63 / 125.
//
// One CTA computes a 128 (weight rows: two 64-row tiles of the packed run) x N (batch rows, a multiple of 16 up to 384) tile
// over a range of k-blocks:
//   dequantiser warps   SETS groups of eight; a warp owns a 16-row slab and every SETS-th k-block.  It loads the slab from
//                       the weight ring, releases the stage at once, and stores four k-slices into its set's four A slots
//   weight producer     one thread; a k-block of both tiles per stage, bulk copies
//   activation producer one thread; a 64-wide k-slice per stage, in the MMA's shared-memory layout (K-major, 128-byte
//                       swizzle) as the preparation kernel stored it
//   MMA issuer          one warp; four tcgen05.mma (M = 128, K = 16, A in TMEM, B in shared memory) per k-slice
// Three shapes, all with sixteen dequantiser warps on an SM: SETS = 1 for N <= 128, two CTAs per SM of 256 TMEM columns (128
// accumulator + a ring of four A slots of 32 columns); SETS = 2 for N <= 256, one CTA with all 512 columns (256 + a ring of four
// slots per set); and WIDE for N <= 384 (384 + one ring that the two sets fill in turn), where a weight is decoded once for half
// as many rows again and the tensor core needs 3000 cycles a k-block against 1300 of decoding.  The SETS = 2 shapes run as CTA
// pairs (cta_group::2): the MMAs span both CTAs' 128 rows and each CTA holds half of the batch rows, because the activation
// slices are read once per 128 weight rows otherwise, 65 bytes a cycle and SM out of the L2, which is more than it gives.
// Weights sit on the MMA's M side (D rows = output features), batch rows on N, as in the small-batch kernel.
//
// Split-K: the S CTAs of a tile form a thread-block cluster.  When their accumulators are done each CTA sends column part r
// of its own to CTA r through distributed shared memory (which the rings no longer need) and adds the S parts of its own
// columns in split order: no fp32 partials in HBM, no second kernel, the additions in a fixed order.
// Every wait is bounded; a wait that runs out sets the status word, and the CTA still frees its tensor memory.
#pragma once
#include "gq_decode.cuh"
#include "gq_scale16.cuh"

// (included after the codebook tables and gq_load.cuh)
namespace gq {

#define GQ_PF_SLOTS 4                        // A slots of a ring: the four 64-wide k-slices of a k-block
// k-slices that share a barrier (a dequantiser's wait, store and announcement; the MMA issuer's wait and commit): SL.  Up to 128 batch rows
// (SETS = 1) the MMAs of a slice are short beside its decoding and the hand-over counts: two a barrier, 34,816 x 5,120 at 64 rows, one / two /
// four, Q4_K 41.3 / 38.0 / 44.6 us, IQ3_S 59.0 / 55.4 / 56.5, Q2_K 43.9 / 39.9 / 45.4.  Above, the MMAs have to follow the slices closely: Q4_K
// at 517 rows, one / two, 153 / 173 us.  Two also need an activation ring of the whole k-block, or the copies of a pair wait for the MMAs of
// the pair before (Q8_0 at 96 to 128 rows, Q6_K at 128): 34,816 x 5,120 at 128 rows, one / two, Q8_0 58.9 / 71.1 us, 1,024 x 5,120 at 112 rows
// 13.2 / 15.3 — except in a run with a codebook type, whose decoding takes longer still (Q8_0 beside IQ2_S at 112 rows 76.3 / 68.9).  And Q4_0,
// which has the least to decode, hands over singly beyond 64 rows: 1,024 x 5,120 at 128 rows 13.1 / 13.8 us.
#define GQ_PF_MAX_STAGES 6                   // upper bound of the weight ring

struct PrefillParams {
    const uint8_t *packed;
    const int32_t *desc;      // split-1 descriptor table: one row per 64-row tile
    int n_desc;
    const uint8_t *xp;        // [m_tile][K/64][N rows][128 B]: fp16 activations in MMA layout
    const float *ex;          // [m_tiles * N] row scales
    __nv_bfloat16 *y;
    int64_t ldy;
    int M, nb, N;             // N: batch rows of a CTA's tile
    int *status;
    int split;                // CTAs of a cluster, each with its part of the k-blocks
    int unit0, unit_step;     // one set: the first unit and +1, or the last and -1
    int wstages, bstages;     // ring depths
    int wstage_bytes;         // both tiles of the widest type of the run
    int cb_mask;              // the codebook types of the run (bit gq_cb_kind): their tables sit side by side in shared memory
    // per GGML type, read from the parameter bank: the size functions of gq_layout.h are switches, and at the start of a CTA every
    // jump is an instruction-cache miss (they and the divisions of a flat block index cost 2500 .. 4000 cycles per CTA)
    uint8_t half_bytes[32];   // bytes_per_256 / 2
    uint16_t cb_at[32];       // 0: no codebook; 1: one the run did not announce; else offset of its table / 16 + 2
};

__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// shared-memory matrix descriptor: K-major, 128-byte swizzle, 8-row groups 1024 bytes apart
__device__ __forceinline__ uint64_t umma_desc(uint32_t smem_addr) {
    const uint32_t lo = ((smem_addr >> 4) & 0x3FFFu) | (1u << 16);
    const uint32_t hi = 64u | (1u << 14) | (2u << 29);
    return ((uint64_t)hi << 32) | lo;
}
// instruction descriptor: D fp32, A and B fp16, both K-major
__device__ __forceinline__ uint32_t umma_idesc(int m, int n) { return (1u << 4) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24); }
// D[128 CG, N] (+)= A[128 CG, 16] (tensor memory) . B[16, N] (shared memory); CG = 2: of both CTAs of a pair, half of B's rows each
template <int CG>
__device__ __forceinline__ void umma_ts_f16(uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
    if constexpr (CG == 1)
        asm volatile(
            "{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\ntcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n}"
            :
            : "r"(tmem_d), "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(accumulate)
            : "memory");
    else
        asm volatile(
            "{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\ntcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %2, %3, p;\n}"
            :
            : "r"(tmem_d), "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(accumulate)
            : "memory");
}
// one thread of the warp, chosen so that the compiler knows the branch to be uniform
__device__ __forceinline__ bool elect_one() {
    uint32_t p;
    asm volatile("{\n.reg .pred p;\nelect.sync _|p, 0xffffffff;\nselp.b32 %0, 1, 0, p;\n}" : "=r"(p));
    return p != 0;
}
// arrive on `bar` when the MMAs issued so far are done; CG = 2: on the barrier at the same place in both CTAs of the pair (`ctas`: their bits)
template <int CG>
__device__ __forceinline__ void umma_commit(uint64_t *bar, uint16_t ctas) {
    if constexpr (CG == 1)
        asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
    else
        asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(smem_u32(bar)), "h"(ctas)
                     : "memory");
}
template <int CG>
__device__ __forceinline__ void tmem_alloc(uint32_t *slot, uint32_t cols) {
    if constexpr (CG == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(slot)), "r"(cols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    } else {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(slot)), "r"(cols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
}
template <int CG>
__device__ __forceinline__ void tmem_dealloc(uint32_t tmem, uint32_t cols) {
    if constexpr (CG == 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(cols) : "memory");
    else asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(cols) : "memory");
}
// an arrival on a barrier of the cluster, by its shared::cluster address.  No fence at cluster scope (release.cluster costs a
// memory barrier of hundreds of cycles, measured 1.6x on the whole kernel): what it announces is tensor memory, ordered by
// tcgen05.fence, or bulk copies, which their own barrier has completed.
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t addr) { asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(addr) : "memory"); }
// sixteen lanes (rows) x 32 columns of tensor memory from the fragments of four 16-weight runs
__device__ __forceinline__ void tmem_st_16x256b_x4(uint32_t taddr, const uint32_t (&r)[16]) {
    asm volatile("tcgen05.st.sync.aligned.16x256b.x4.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};" ::"r"(taddr), "r"(r[0]),
                 "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]),
                 "r"(r[13]), "r"(r[14]), "r"(r[15])
                 : "memory");
}
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_ld_32x32b_x8(uint32_t taddr, uint32_t (&v)[8]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
                 : "r"(taddr)
                 : "memory");
}
// the registers of a load in flight pass through its wait, so that nothing reads, copies or merges them before it
__device__ __forceinline__ void tmem_wait_ld(uint32_t (&v)[8]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(v[0]), "+r"(v[1]), "+r"(v[2]), "+r"(v[3]), "+r"(v[4]), "+r"(v[5]), "+r"(v[6]), "+r"(v[7])
                 :
                 : "memory");
}

// ---- k-slice J (runs 4J .. 4J+3) of one slab: decode, scale -> fp16 weights as the registers of one 16x256b.x4 store --------
template <int TYPE, int J>
__device__ __forceinline__ void pf_slice(const Dec<TYPE> &dec, uint32_t (&o)[16]) {
    uint32_t s[2][2], m[2][2], a[2][2][4];
    constexpr int G = Dec<TYPE>::GROUP;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        hscales<J>(dec, h, s[h]);
        if constexpr (Dec<TYPE>::HAS_MIN) hmins<J>(dec, h, m[h]);
    }
    dec.template pair<2 * J>(a[0]);
    dec.template pair<2 * J + 1>(a[1]);
    const auto run = [&](auto r_) {
        constexpr int R = decltype(r_)::value;
        constexpr float off = Dec<TYPE>::template offs<4 * J + R>();
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int k = 0; k < 2; ++k) {
                __half2 w = u32_as_h2(a[R >> 1][R & 1][2 * k + h]);
                if constexpr (off != 0.0f) w = __hsub2(w, u32_as_h2(h2k(off)));
                if constexpr (Dec<TYPE>::HAS_MIN) w = __hfma2(w, scale_of<G, R>(s[h]), scale_of<G, R>(m[h]));
                else w = __hmul2(w, scale_of<G, R>(s[h]));
                o[4 * R + 2 * h + k] = h2_as_u32(w);       // 32-bit column 2t + k of row g + 8h of the run's eight columns
            }
    };
    run(std::integral_constant<int, 0>{}); run(std::integral_constant<int, 1>{}); run(std::integral_constant<int, 2>{}); run(std::integral_constant<int, 3>{});
}

struct PfRings {
    uint8_t *wring;
    int wstage_bytes, wstages;
    uint64_t *wfull, *wfree, *afree;
    uint32_t afull;                  // shared::cluster address: in a CTA pair, of the CTA that issues the MMAs
};

// the dequantiser loop of one warp for a tile of TYPE: k-blocks set, set + SETS, ... of this CTA's nkb; k-block kb fills the
// A ring kb % RINGS once the MMAs of k-block kb - RINGS have read it.  Barriers are waited on phase by phase: wfull because the
// weight ring has a multiple of SETS stages, afree because it belongs to a set's k-blocks, not to the ring.
template <int TYPE, int SETS, int RINGS, int SL>
__device__ __forceinline__ bool pf_dequant(const PfRings &r, int slab_off, int set, int nkb, uint32_t ta, const DecAux &aux, int lane) {
    int ws = set % r.wstages, wround = set / r.wstages;
    for (int kb = set; kb < nkb; kb += SETS) {
        const int prev = kb - RINGS;
        uint64_t *afree = r.afree + GQ_PF_SLOTS / SL * ((kb + SETS - RINGS) % SETS);
        if (!mbar_wait(r.wfull + ws, wround & 1)) return false;
        Dec<TYPE> dec;
        dec.load(r.wring + (size_t)ws * r.wstage_bytes + slab_off, lane, aux);
        __syncwarp();
        if (lane == 0) mbar_arrive(r.wfree + ws);          // everything the decoder needs is in registers
        ws += SETS;
        while (ws >= r.wstages) { ws -= r.wstages; ++wround; }
        const auto slice = [&](auto j_) -> bool {
            constexpr int J = decltype(j_)::value;
            uint32_t o[16];
            pf_slice<TYPE, J>(dec, o);
            if constexpr (J % SL == 0) {
                if (prev >= 0 && !mbar_wait(afree + J / SL, (prev / SETS) & 1)) return false;
                __syncwarp();
                tc_fence_after();
            }
            tmem_st_16x256b_x4(ta + 32 * J, o);
            if constexpr (J % SL == SL - 1) {
                tmem_wait_st();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive_cluster(r.afull + 8 * (J / SL));
            }
            return true;
        };
        if (!slice(std::integral_constant<int, 0>{}) || !slice(std::integral_constant<int, 1>{}) || !slice(std::integral_constant<int, 2>{}) ||
            !slice(std::integral_constant<int, 3>{})) return false;
    }
    return true;
}

// eight accumulator columns (batch rows n0..n0+7) of the lane's feature row to y.  Two neighbouring lanes hold
// neighbouring columns of y: they trade values so that each stores both of one batch row (four bytes instead of two).
__device__ __forceinline__ void pf_store8(const PrefillParams &p, const float (&v)[8], int n0, int64_t col, bool row_ok, bool pair_ok, int lane) {
#pragma unroll
    for (int j = 0; j < 8; j += 2) {
        const bool odd = lane & 1;
        const float got = __shfl_xor_sync(0xffffffffu, odd ? v[j] : v[j + 1], 1);
        if (pair_ok) {
            const int n = n0 + j + (odd ? 1 : 0);
            if (n < p.M) *reinterpret_cast<__nv_bfloat162 *>(p.y + (int64_t)n * p.ldy + col - (odd ? 1 : 0)) =
                odd ? __floats2bfloat162_rn(got, v[j + 1]) : __floats2bfloat162_rn(v[j], got);
        } else if (row_ok) {
            if (n0 + j < p.M) p.y[(int64_t)(n0 + j) * p.ldy + col] = __float2bfloat16_rn(v[j]);
            if (n0 + j + 1 < p.M) p.y[(int64_t)(n0 + j + 1) * p.ldy + col] = __float2bfloat16_rn(v[j + 1]);
        }
    }
}

// batch rows of tile mt that enter the MMAs: all N, of the last tile those that the batch has, in steps of 16 (517 rows are tiles of 288 and 240)
__host__ __device__ inline int pf_rows(int M, int N, int mt) { const int left = (M - mt * N + 15) & ~15; return left < N ? left : N; }

template <int SETS, bool WIDE, int SL>
__global__ void __launch_bounds__(32 * (8 * SETS + 3), SETS == 1 ? 2 : 1) gemm_prefill_kernel(const __grid_constant__ PrefillParams p) {
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    // layout: [activation ring][weight ring][codebook tables of the run's types]; the reduction of a split reuses the rings
    __shared__ __align__(8) uint64_t bars[2 * GQ_PF_MAX_STAGES + 2 * GQ_PF_SLOTS * SETS + 1];
    __shared__ uint32_t tmem_slot;
    __shared__ int s_out[2][2];          // first output column and columns of the two tiles: the epilogue does not wait for global memory
    uint8_t *smem = reinterpret_cast<uint8_t *>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    const int N = p.N, bbytes = N * 128 / SETS;          // a CTA of a pair holds half of the batch rows of a slice
    uint8_t *wring = smem + p.bstages * bbytes;
    uint8_t *tables = wring + p.wstages * p.wstage_bytes;
    constexpr int RINGS = WIDE ? 1 : SETS, CG = SETS, GROUPS = GQ_PF_SLOTS / SL;
    uint64_t *wfull = bars, *wfree = bars + GQ_PF_MAX_STAGES;
    uint64_t *afull = bars + 2 * GQ_PF_MAX_STAGES, *afree = afull + GROUPS * RINGS, *done = afree + GROUPS * SETS;
    constexpr uint32_t TMEM_COLS = 256u * SETS, D_COLS = TMEM_COLS - 32u * GQ_PF_SLOTS * RINGS;      // the A slots follow the accumulator
    constexpr int DEQ = 8 * SETS;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // grid (CG * split, units, batch tiles): a cluster is the parts of one unit, CG groups of two tiles each
    const int half = (int)blockIdx.x % CG, part = (int)blockIdx.x / CG, unit = SETS == 1 ? p.unit0 + p.unit_step * (int)blockIdx.y : (int)blockIdx.y, mt = blockIdx.z;
    const int kb0 = (int)((uint32_t)(part * p.nb) / (uint32_t)p.split), nkb = (int)((uint32_t)((part + 1) * p.nb) / (uint32_t)p.split) - kb0;
    const int rows = SETS == 1 ? N : pf_rows(p.M, N, mt);        // of the batch tile, those that are multiplied (one set: all, up to 15 past the batch)
    const uint32_t leader = (uint32_t)(part * CG);       // cluster rank of the CTA that issues the pair's MMAs
    __shared__ __align__(16) float s_ex[SETS == 1 ? 128 : 384];

    // the two 64-row tiles of this CTA (neither, in the second CTA of a last pair; only one, in the last CTA with any)
    const int first = 2 * (unit * CG + half);
    const bool has0 = first < p.n_desc, has1 = first + 1 < p.n_desc;
    const int32_t *d0 = p.desc + (int64_t)(has0 ? first : p.n_desc - 1) * GQ_DESC_WORDS;
    const int32_t *d1 = has1 ? d0 + GQ_DESC_WORDS : d0;
    int types[2 * CG];                  // of all tiles of the pair, requested together (a load from global memory costs 700 cycles)
#pragma unroll
    for (int t = 0; t < 2 * CG; ++t) types[t] = p.desc[(int64_t)min(2 * unit * CG + t, p.n_desc - 1) * GQ_DESC_WORDS + 1];
    const int off0 = d0[0], off1 = d1[0];
    const int type0 = CG > 1 && half && has0 ? types[2 * CG - 2] : types[0], type1 = !has1 ? type0 : CG > 1 && half ? types[2 * CG - 1] : types[1];
    const int wb0 = has0 ? 128 * p.half_bytes[type0 & 31] : 0, wb1 = has1 ? 128 * p.half_bytes[type1 & 31] : 0;

    // a codebook type the call's run_info did not announce has no table space, a wider type no stage: report and leave
    // (nothing is allocated yet; every CTA of a cluster looks at all of its tiles, so a cluster leaves as one)
    bool bad = false;
#pragma unroll
    for (int t = 0; t < 2 * CG; ++t) {
        const int hb = p.half_bytes[types[t] & 31];
        bad |= hb == 0 || 256 * hb > p.wstage_bytes || p.cb_at[types[t] & 31] == 1;
    }
    if (bad) {
        if (threadIdx.x == 0) { pdl_wait(); report_status(p.status, GQ_DEV_BAD_SHAPE); }      // after the preparation kernel has cleared the word
        return;
    }
    const uint8_t *wsrc0 = p.packed + (int64_t)off0 * 16 + (int64_t)kb0 * wb0, *wsrc1 = p.packed + (int64_t)off1 * 16 + (int64_t)kb0 * wb1;
    const auto load_weights = [&](int kb, int st) {
        uint8_t *dst = wring + (size_t)st * p.wstage_bytes;
        mbar_expect_tx(wfull + st, (uint32_t)(wb0 + wb1));
        bulk_g2s(dst, wsrc0 + (int64_t)kb * wb0, (uint32_t)wb0, wfull + st);
        if (wb1) bulk_g2s(dst + wb0, wsrc1 + (int64_t)kb * wb1, (uint32_t)wb1, wfull + st);
    };
    if (threadIdx.x == 32 * DEQ) {
        const uint32_t slabs = has1 ? 8 : has0 ? 4 : 0;
        // an A slot is full when all slabs of the pair are stored and each CTA's rows of the activation slice are there; the
        // second CTA's own barrier sees its copy only, and its relay warp passes that on
        const int in_pair = p.n_desc - 2 * unit * CG;
        const uint32_t pair_slabs = (uint32_t)(in_pair < 2 * CG ? in_pair : 2 * CG) * 4;
        for (int s = 0; s < p.wstages; ++s) { mbar_init(wfull + s, 1); mbar_init(wfree + s, slabs ? slabs : 1); }
        for (int s = 0; s < GROUPS * RINGS; ++s) mbar_init(afull + s, half ? SL : pair_slabs + SL + CG - 1);
        for (int s = 0; s < GROUPS * SETS; ++s) mbar_init(afree + s, 1);
        mbar_init(done, 1);
        fence_barrier_init();
        fence_proxy_async();
        // the first weights do not wait for anything: on their way while the rest is set up
        if (has0)
            for (int kb = 0; kb < SETS && kb < nkb; ++kb) load_weights(kb, kb);
    }
    if (threadIdx.x < 4) s_out[threadIdx.x >> 1][threadIdx.x & 1] = (threadIdx.x >> 1 ? d1 : d0)[2 + (threadIdx.x & 1)];
    __syncwarp();
    if (warp == DEQ + 2) tmem_alloc<CG>(&tmem_slot, TMEM_COLS);
    // the codebook tables of the two tiles' types, each at its place among the tables of the run's types
    const int cb0 = p.cb_at[type0 & 31], cb1 = p.cb_at[type1 & 31];
    if (cb0) fill_codebook(type0, tables + 16 * (cb0 - 2), threadIdx.x, blockDim.x);
    if (cb1 && type1 != type0) fill_codebook(type1, tables + 16 * (cb1 - 2), threadIdx.x, blockDim.x);
    tc_fence_before();
    __syncwarp();
    if constexpr (CG > 1) cluster_sync_all();      // the other CTA's barriers exist before anything arrives on them
    else __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_slot;
    bool ok = true;

    if (warp == DEQ) {
        // ---- weight producer (the rest of the k-blocks): does not depend on the kernel in front of this one ----
        if (lane == 0 && has0) {
            for (int kb = SETS, st = SETS % p.wstages, round = SETS / p.wstages; kb < nkb; ++kb) {
                if (round > 0 && !mbar_wait_parked(wfree + st, (round - 1) & 1)) { ok = false; break; }
                load_weights(kb, st);
                if (++st == p.wstages) { st = 0; ++round; }
            }
        }
        __syncwarp();
    } else if (warp == DEQ + 1) {
        // ---- activation producer.  Slice i takes stage i % bstages; the MMAs of slice i - bstages have read it when that
        // slice's A slot comes free (bstages <= 4 RINGS, so the slot cannot have been used again by then).  The copy completes on
        // the barrier of the slice's A slot, so that the MMA issuer waits once per slice ----
        if (lane == 0) {
            pdl_wait();
            const uint8_t *src = p.xp + (((int64_t)mt * p.nb + kb0) * 4 * CG + half) * bbytes;
            for (int i = 0, st = 0; i < 4 * nkb; ++i) {
                const int o = i - p.bstages;
                if (o >= 0 && !mbar_wait_parked(afree + ((o >> 2) % SETS) * GROUPS + (o & 3) / SL, ((o >> 2) / SETS) & 1)) { ok = false; break; }
                uint64_t *full = afull + ((i >> 2) % RINGS) * GROUPS + (i & 3) / SL;
                mbar_expect_tx(full, (uint32_t)bbytes);
                bulk_g2s(smem + (size_t)st * bbytes, src + (int64_t)i * CG * bbytes, (uint32_t)bbytes, full);
                if (++st == p.bstages) st = 0;
            }
            pdl_trigger();
        }
        __syncwarp();
    } else if (warp == DEQ + 2 && half) {
        // ---- relay of the pair's second CTA: its activation rows are there -> the issuing CTA's barrier ----
        for (int kb = 0; kb < nkb && ok; ++kb) {
            const int slot0 = GROUPS * (kb % RINGS);
#pragma unroll
            for (int j = 0; j < GROUPS; ++j) {
                if (!mbar_wait(afull + slot0 + j, (uint32_t)(kb / RINGS) & 1u)) { ok = false; break; }
                if (lane == 0) mbar_arrive_cluster(map_to_rank(smem_u32(afull + slot0 + j), leader));
            }
            __syncwarp();
        }
    } else if (warp == DEQ + 2) {
        // ---- MMA issuer: the warp waits as one and a thread chosen by elect.sync issues, so that addresses and descriptors
        // stay in uniform registers (issued from a `lane == 0` branch an MMA cost the thread a hundred cycles) ----
        // an MMA takes up to 256 batch rows: the wide tile is two of them, of a last tile's rows the second has what is left, if anything
        const int nmma = WIDE ? N >> 1 : N, n0 = rows < nmma ? rows : nmma, n1 = rows - n0;
        const uint32_t idesc = umma_idesc(128 * CG, n0), idesc1 = umma_idesc(128 * CG, n1);
        const uint16_t ctas = (uint16_t)(3u << leader);
        const uint64_t bdesc0 = umma_desc(smem_u32(smem));
        const uint32_t bstep = (uint32_t)bbytes >> 4, bwrap = bstep * (uint32_t)p.bstages;
        uint32_t boff = 0;
        for (int kb = 0; kb < nkb && ok; ++kb) {
            const int ring = kb % RINGS;
            const uint32_t parity = (uint32_t)(kb / RINGS) & 1u;
            uint64_t *full = afull + GROUPS * ring, *free = afree + GROUPS * (kb % SETS);
            const uint32_t ta = tmem + D_COLS + 32u * GQ_PF_SLOTS * ring;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                if (j % SL == 0) {
                    if (!mbar_wait(full + j / SL, parity)) { ok = false; break; }
                    tc_fence_after();
                }
                if (elect_one()) {
                    const uint64_t bd = bdesc0 + boff;
#pragma unroll
                    for (int kk = 0; kk < 4; ++kk) {
                        const uint32_t acc = (j > 0 || kk > 0) ? 1u : (uint32_t)(kb > 0);
                        umma_ts_f16<CG>(tmem, ta + 32 * j + 8 * kk, bd + 2 * kk, idesc, acc);
                        if constexpr (WIDE)
                            if (n1 > 0) umma_ts_f16<CG>(tmem + nmma, ta + 32 * j + 8 * kk, bd + 8 / CG * nmma + 2 * kk, idesc1, acc);      // 128 bytes a row
                    }
                    // the slot and the activation stage may be overwritten once these MMAs have read them
                    if (j % SL == SL - 1) umma_commit<CG>(j == 3 && kb + 1 == nkb ? done : free + j / SL, ctas);
                }
                boff += bstep;
                if (boff == bwrap) boff = 0;
            }
            __syncwarp();
        }
    } else {
        // ---- dequantisers: warp w reaches the TMEM lanes of partition w % 4, which hold slabs 2 (w % 4) and + 1 ----
        const int w = warp & 7, slab = 2 * (w & 3) + (w >> 2), set = warp >> 3, ring = set % RINGS;
        const int type = slab < 4 ? type0 : type1;
        if (slab < 4 ? has0 : has1) {
            DecAux aux;
            const int cb = slab < 4 ? cb0 : cb1;
            aux.grid = reinterpret_cast<const uint32_t *>(tables + (cb ? 16 * (cb - 2) : 0));
            aux.iq4 = iq4_table_biased();
            PfRings r;
            r.wring = wring; r.wstage_bytes = p.wstage_bytes; r.wstages = p.wstages;
            r.wfull = wfull; r.wfree = wfree; r.afree = afree;
            r.afull = map_to_rank(smem_u32(afull + GROUPS * ring), CG > 1 ? leader : cluster_ctarank());
            const int slab_off = (slab < 4 ? 0 : wb0) + (slab & 3) * 32 * p.half_bytes[type & 31];
            const uint32_t ta = tmem + D_COLS + 32u * GQ_PF_SLOTS * ring + ((uint32_t)(16 * slab) << 16);
#define GQ_PF(T) case T: ok = pf_dequant<T, SETS, RINGS, SL>(r, slab_off, set, nkb, ta, aux, lane); break;
            switch (type) {
                GQ_PF(GQ_Q4_0) GQ_PF(GQ_Q5_0) GQ_PF(GQ_Q8_0) GQ_PF(GQ_Q2_K) GQ_PF(GQ_Q3_K) GQ_PF(GQ_Q4_K)
                GQ_PF(GQ_Q5_K) GQ_PF(GQ_Q6_K) GQ_PF(GQ_IQ4_NL) GQ_PF(GQ_IQ3_S) GQ_PF(GQ_IQ4_XS) GQ_PF(GQ_IQ3_XXS)
                GQ_PF(GQ_IQ2_XXS) GQ_PF(GQ_IQ2_XS) GQ_PF(GQ_IQ2_S) GQ_PF(GQ_IQ1_M)
            }
#undef GQ_PF
        }
        pdl_wait();       // y may be read, and ex is written, by what runs in front
        for (int i = threadIdx.x; i < N; i += 32 * DEQ) s_ex[i] = p.ex[mt * N + i];
        if (ok && !mbar_wait(done, 0)) ok = false;
        __syncwarp();
        asm volatile("bar.sync 1, %0;" ::"n"(32 * DEQ) : "memory");
        tc_fence_after();
    }

    // ---- epilogue: warps 0 .. DEQ-1; lane l of partition q is row 32 q + l of the pair of tiles ----
    const int q = warp & 3, e = warp >> 2, feat = 32 * q + lane;
    const int rt = feat & 63, n_cols = s_out[feat >> 6][1];
    const bool tile_ok = feat < 64 ? has0 : has1, row_ok = tile_ok && rt < n_cols;
    const int64_t col = (int64_t)s_out[feat >> 6][0] + rt;
    const bool pair_ok = tile_ok && (rt | 1) < n_cols && !(p.ldy & 1) && !((reinterpret_cast<uintptr_t>(p.y) + 2 * (uintptr_t)(col - (lane & 1))) & 3);
    const uint32_t td = tmem + ((uint32_t)(32 * q) << 16);
    if (p.split == 1) {
        if (warp < DEQ && ok) {
#pragma unroll 1
            for (int c = 8 * e; c < rows; c += 8 * (DEQ / 4)) {
                uint32_t a[8];
                tmem_ld_32x32b_x8(td + c, a);
                const float4 e0 = *reinterpret_cast<const float4 *>(s_ex + c), e1 = *reinterpret_cast<const float4 *>(s_ex + c + 4);
                const float es[8] = {e0.x, e0.y, e0.z, e0.w, e1.x, e1.y, e1.z, e1.w};
                float v[8];
                tmem_wait_ld(a);
#pragma unroll
                for (int j = 0; j < 8; ++j) v[j] = __uint_as_float(a[j]) * es[j];
                pf_store8(p, v, mt * N + c, col, row_ok, pair_ok, lane);
            }
        }
    } else {
        // columns [r ch, (r + 1) ch) are summed and stored by the CTA of part r; slot s of its buffer is part s's share, as
        // [ch / 4][128 rows] of four columns each: 16-byte stores and loads, one per lane side by side
        const int S = p.split, ch = ((rows + S - 1) / S + 7) & ~7;
        float4 *buf = reinterpret_cast<float4 *>(smem);
        cluster_sync_all();                 // every CTA of the cluster has finished with its rings
        if (warp < DEQ) {
            const uint32_t mine = smem_u32(buf) + (uint32_t)(part * (ch >> 2) * 128 + feat) * 16;
#pragma unroll 1
            for (int c = 8 * e; c < rows; c += 8 * (DEQ / 4)) {
                uint32_t a[8];
                tmem_ld_32x32b_x8(td + c, a);
                const int r = c / ch;
                const uint32_t dst = map_to_rank(mine, (uint32_t)(r * CG + half)) + (uint32_t)((c - r * ch) >> 2) * 2048;
                tmem_wait_ld(a);
                st_cluster_f4(dst, __uint_as_float(a[0]), __uint_as_float(a[1]), __uint_as_float(a[2]), __uint_as_float(a[3]));
                st_cluster_f4(dst + 2048, __uint_as_float(a[4]), __uint_as_float(a[5]), __uint_as_float(a[6]), __uint_as_float(a[7]));
            }
            __syncwarp();
        }
        const bool any_bad = __syncthreads_or(!ok);
        cluster_sync_all();
        const int c1 = (part + 1) * ch < rows ? (part + 1) * ch : rows;
        if (warp < DEQ && !any_bad) {
#pragma unroll 1
            for (int c = part * ch + 8 * e; c < c1; c += 8 * (DEQ / 4)) {
                float v[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
                for (int s = 0; s < S; ++s) {
                    const float4 *b = buf + ((s * ch + (c - part * ch)) >> 2) * 128 + feat;
                    const float4 x = b[0], y = b[128];
                    v[0] += x.x; v[1] += x.y; v[2] += x.z; v[3] += x.w;
                    v[4] += y.x; v[5] += y.y; v[6] += y.z; v[7] += y.w;
                }
                const float4 e0 = *reinterpret_cast<const float4 *>(s_ex + c), e1 = *reinterpret_cast<const float4 *>(s_ex + c + 4);
                const float es[8] = {e0.x, e0.y, e0.z, e0.w, e1.x, e1.y, e1.z, e1.w};
#pragma unroll
                for (int j = 0; j < 8; ++j) v[j] *= es[j];
                pf_store8(p, v, mt * N + c, col, row_ok, pair_ok, lane);
            }
        }
    }
    if (!ok) {
        // a bounded wait ran out: report it, and give copies and MMAs still in flight a bounded time to land
        if (lane == 0) report_status(p.status, GQ_DEV_TIMEOUT);
        for (int i = 0; i < 100; ++i) __nanosleep(10000);
    }
    tc_fence_before();
    __syncwarp();
    if constexpr (CG > 1) cluster_sync_all();      // tensor memory is given back by both CTAs, after both have read theirs
    else __syncthreads();
    if (warp == DEQ + 2) {
        tc_fence_after();
        tmem_dealloc<CG>(tmem, TMEM_COLS);
    }
}

__device__ __forceinline__ float amax8(const uint4 &v) {
    const __nv_bfloat162 *b = reinterpret_cast<const __nv_bfloat162 *>(&v);
    float a = 0.0f;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const float2 f = __bfloat1622float2(b[j]);
        a = fmaxf(a, fmaxf(fabsf(f.x), fabsf(f.y)));
    }
    return a;
}

// activation preparation for the prefill path: bf16 row -> fp16 scaled by an exact power of two, stored in the
// MMA's shared-memory layout (tiles of N rows x 64 k, K-major, 16-byte chunks XOR-swizzled by row % 8) so the
// kernel's producer moves a whole k-slice with one bulk copy.  For CTA pairs a slice holds the rows of the first CTA, then
// those of the second: of every `nmma` rows that an MMA takes, the first half is the first CTA's.  The row is read once and kept in
// registers between the maximum and the conversion: 5120 activations to a CTA of 128 threads, long rows over a cluster of up to eight CTAs
// (prefill_prep_parts), which exchange their maxima (what they do not hold is read twice).  128 threads of few
// registers, so that these CTAs fit beside those of a matrix kernel: they are in place when the kernel in front ends, and the
// matrix kernel behind them gets its SMs, fetches weights and decodes while they run (with 512 threads a CTA kept it off its SM).
// Bound by the latency of its loads and, beyond a few hundred rows, by how many of these CTAs an SM holds: rows of 17,408 in one CTA each
// took 6 us at 64 rows and 17 at 517, a sixth of the layer.
#define GQ_PF_PREP_THREADS 128
#define GQ_PF_PREP_VECS 5
#define GQ_PF_PREP_CTAS 9        // of them that an SM holds
__global__ void __launch_bounds__(GQ_PF_PREP_THREADS, GQ_PF_PREP_CTAS) prep_x_prefill_kernel(const __nv_bfloat16 *__restrict__ x, int64_t ldx, int K, int M, int N, int nmma,
                                                                            float *__restrict__ ex, uint8_t *__restrict__ xp, int *status) {
    __shared__ float red[GQ_PF_PREP_THREADS / 32], peers[8];
    const int part = blockIdx.y, parts = gridDim.y, m = blockIdx.x, mt = m / N, n = m - mt * N, nvec = K >> 3;
    // of a pair's tile each MMA (rows [0, nmma) and the rest) has its first half in the first CTA
    const int rows = pf_rows(M, N, mt), second = nmma && n >= nmma, in = second ? n - nmma : n, of = !nmma ? 0 : second ? rows - nmma : rows < nmma ? rows : nmma;
    const int r = !nmma || n >= rows ? n : in / (of >> 1) * (N >> 1) + (second ? nmma >> 1 : 0) + in % (of >> 1);
    uint8_t *dst = xp + (int64_t)mt * (K / 64) * (N * 128) + r * 128;
    const int phase = r & 7;
    if (parts > 1) cluster_arrive_relaxed();      // collected before the first store into another CTA: by then it runs
    pdl_trigger();    // the kernel behind this one may start fetching weights
    pdl_wait();       // whatever ran before (possibly still reading this workspace) has finished
    if (m == 0 && part == 0 && threadIdx.x == 0) *status = 0;
    const int first = part * GQ_PF_PREP_THREADS + threadIdx.x, step = parts * GQ_PF_PREP_THREADS;       // the thread's chunks of the row
    const auto put = [&](int c, const uint4 &o) { *reinterpret_cast<uint4 *>(dst + (int64_t)(c >> 3) * (N * 128) + (((c & 7) ^ phase) << 4)) = o; };
    if (n >= rows) return;      // no MMA reads it
    if (m >= M) {
        // rows past the batch among the last 16: zeros (their outputs are never stored)
        for (int c = first; c < nvec; c += step) put(c, make_uint4(0, 0, 0, 0));
        return;
    }
    const uint4 *xr = reinterpret_cast<const uint4 *>(x + (int64_t)m * ldx);
    uint4 v[GQ_PF_PREP_VECS];
    float amax = 0.0f;
#pragma unroll
    for (int i = 0; i < GQ_PF_PREP_VECS; ++i) {
        const int c = first + i * step;
        v[i] = c < nvec ? __ldg(xr + c) : make_uint4(0u, 0u, 0u, 0u);
    }
#pragma unroll
    for (int i = 0; i < GQ_PF_PREP_VECS; ++i) amax = fmaxf(amax, amax8(v[i]));
    for (int c = first + GQ_PF_PREP_VECS * step; c < nvec; c += step) amax = fmaxf(amax, amax8(__ldg(xr + c)));
#pragma unroll
    for (int o = 16; o; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = amax;
    __syncthreads();
    float a = red[0];
#pragma unroll
    for (int i = 1; i < GQ_PF_PREP_THREADS / 32; ++i) a = fmaxf(a, red[i]);
    if (parts > 1) {      // the cluster is the row: every CTA puts its maximum into all of them
        cluster_wait();
        if ((int)threadIdx.x < parts) st_cluster_f32(map_to_rank(smem_u32(peers + part), threadIdx.x), a);
        cluster_sync_all();
        for (int i = 0; i < parts; ++i) a = fmaxf(a, peers[i]);
    }
    // scale = 2^(9 - e), amax * scale in [512, 1024); identity for a zero, tiny or non-finite row
    int e = 9;
    if (a > 0.0f && a < 3.0e38f) { e = (int)((__float_as_uint(a) >> 23) & 0xFF) - 127; if (e < -100) e = -100; }
    const float scale = __uint_as_float((uint32_t)(127 + 9 - e) << 23);
    if (part == 0 && threadIdx.x == 0) ex[m] = __uint_as_float((uint32_t)(127 - 9 + e) << 23);
    const auto convert = [&](int c, const uint4 &w) {
        const __nv_bfloat162 *b = reinterpret_cast<const __nv_bfloat162 *>(&w);
        uint4 o;
        uint32_t *oo = reinterpret_cast<uint32_t *>(&o);
#pragma unroll
        for (int j = 0; j < 4; ++j) { const float2 f = __bfloat1622float2(b[j]); oo[j] = h2_as_u32(__floats2half2_rn(f.x * scale, f.y * scale)); }
        put(c, o);
    };
#pragma unroll
    for (int i = 0; i < GQ_PF_PREP_VECS; ++i) {
        const int c = first + i * step;
        if (c < nvec) convert(c, v[i]);
    }
    for (int c = first + GQ_PF_PREP_VECS * step; c < nvec; c += step) convert(c, __ldg(xr + c));
}

}  // namespace gq
