// The grouped kernel's fp16 form: batches of more rows than the integer form takes, up to 32 (above, the C ABI runs it twice).
// mma.sync m16n8k16 with the weights on M as exact fp16 integers and the activations as fp16 on N.
// (included after GemvParams, the workspace layout, gq_load.cuh and fused_allreduce_block)
#pragma once
#include "gq_scale16.cuh"

// One k-block of one slab:  acc += sx[n] * ( d[row] * sum_runs(scale * (W_int . x)) - f[row] * (A'' . run sums) ).
// Types whose field x scale is an exact fp16 integer (gq_folds) enter the MMA with the scale multiplied in, and the MMAs of a k-block
// accumulate: one packed multiply-add per two weights, whatever the number of batch rows, in place of four fp32 multiply-adds per scale
// group and column tile.  The others (an fp16 d per 32 weights, or a product of more than eleven bits) scale each group's MMA result.
template <int TYPE, int MT>
__device__ __forceinline__ void slab_kblock(const uint8_t *slab, const uint8_t *xs, int xs_off, const DecAux &aux, int lane, float (&acc)[MT][4],
                                            const float (&z)[4]) {
    Dec<TYPE> dec;
    dec.load(slab, lane, aux);
    const int g = lane >> 2, t = lane & 3;
    const uint8_t *xb = xs + g * GQ_X_ROW + 16 * t;              // unit (P, t) of batch row g; + 8 nt rows, + 64 P
    float blk[MT][4];
#pragma unroll
    for (int nt = 0; nt < MT; ++nt) blk[nt][0] = blk[nt][1] = blk[nt][2] = blk[nt][3] = 0.f;
    if constexpr (gq_folds<TYPE>()) {
        static_for<0, 4>([&](auto j_) {
            constexpr int J = decltype(j_)::value;
            uint32_t a[4][4];
            fold_slice<TYPE, J>(dec, a);
#pragma unroll
            for (int p = 0; p < 2; ++p) {
                // the MMAs of the two runs of a pair accumulate into the same registers: the other column tiles stand between them
                uint4 b[MT];
#pragma unroll
                for (int nt = 0; nt < MT; ++nt) {
                    b[nt] = ld16(xb + nt * 8 * GQ_X_ROW + 64 * (2 * J + p));
                    mma16816(blk[nt], a[2 * p], b[nt].x, b[nt].y);
                }
#pragma unroll
                for (int nt = 0; nt < MT; ++nt) mma16816(blk[nt], a[2 * p + 1], b[nt].z, b[nt].w);
            }
        });
    } else {
        static_for<0, 8>([&](auto p_) {
            constexpr int P = decltype(p_)::value;
            constexpr bool G32 = Dec<TYPE>::GROUP == 32;
            uint32_t a[2][4];
            dec.template pair<P>(a);
            float sc[2][2];
            if constexpr (G32) dec.template scale<P>(sc[0][0], sc[0][1]);
            else { dec.template scale<2 * P>(sc[0][0], sc[0][1]); dec.template scale<2 * P + 1>(sc[1][0], sc[1][1]); }
#pragma unroll
            for (int nt = 0; nt < MT; ++nt) {
                const uint4 b = ld16(xb + nt * 8 * GQ_X_ROW + 64 * P);
                float tmp[4];
                mma16816_z(tmp, a[0], b.x, b.y, z);
                if constexpr (G32) {
                    mma16816(tmp, a[1], b.z, b.w);
                } else {
#pragma unroll
                    for (int j = 0; j < 4; ++j) blk[nt][j] = fmaf(sc[0][j >> 1], tmp[j], blk[nt][j]);
                    mma16816_z(tmp, a[1], b.z, b.w, z);
                }
#pragma unroll
                for (int j = 0; j < 4; ++j) blk[nt][j] = fmaf(sc[G32 ? 0 : 1][j >> 1], tmp[j], blk[nt][j]);
            }
        });
    }
    float d[2];
    dec.kscale(d[0], d[1]);
    // the correction sets: all of them, or of a folded type the last one (the first removes the bias that the fold has taken off)
    constexpr int NC = Dec<TYPE>::NCORR, C0 = gq_folds<TYPE>() ? (fold_has_corr<TYPE>() ? NC - 1 : NC) : 0;
    uint32_t ac[NC ? NC : 1][4];
    float fc[NC ? NC : 1][2];
    if constexpr (C0 < NC) dec.corr(ac, fc);
#pragma unroll
    for (int nt = 0; nt < MT; ++nt) {
        float tot[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) tot[j] = d[j >> 1] * blk[nt][j];
        if constexpr (C0 < NC) {
            const uint4 b = ld16(xs + (nt * 8 + g) * GQ_X_ROW + GQ_X_SUMS + 16 * t);
#pragma unroll
            for (int c = C0; c < NC; ++c) {
                float mm[4];
                mma16816_z(mm, ac[c], b.x, b.y, z);
                mma16816(mm, ac[c], b.z, b.w);
#pragma unroll
                for (int j = 0; j < 4; ++j) tot[j] = fmaf(-fc[c][j >> 1], mm[j], tot[j]);
            }
        }
        const float2 sx = *reinterpret_cast<const float2 *>(xs + xs_off + (nt * 8 + 2 * t) * 4);
        acc[nt][0] = fmaf(sx.x, tot[0], acc[nt][0]);
        acc[nt][1] = fmaf(sx.y, tot[1], acc[nt][1]);
        acc[nt][2] = fmaf(sx.x, tot[2], acc[nt][2]);
        acc[nt][3] = fmaf(sx.y, tot[3], acc[nt][3]);
    }
}

template <int TYPE, int MT>
__device__ __forceinline__ bool consume(const Ring &r, int x_at, int xs_off, int slab_off, const DecAux &aux, int lane, float (&acc)[MT][4]) {
    const float z[4] = {0.f, 0.f, 0.f, 0.f};
    for (int i = 0, s = 0, round = 0; i < r.nk; ++i) {
        if (!mbar_wait(r.full + s, round & 1)) return false;
        const uint8_t *st = r.smem + (size_t)s * r.stage_bytes;
        slab_kblock<TYPE, MT>(st + slab_off, st + x_at, xs_off, aux, lane, acc, z);
        __syncwarp();
        if (lane == 0) mbar_arrive(r.empty + s);
        if (++s == r.stages) { s = 0; ++round; }
    }
    return true;
}

// One CTA: two 64-row tiles of the run (128 output columns) x a k-range; a producer warp and eight consumer warps, a 16-column slab each.
// Bound by the tensor pipe as mma.sync reaches it (18 MMAs of 8 cycles per slab, k-block and column tile) and by the decoders' instructions,
// which the four warps of a scheduler overlap only in part: 34,816 x 5,120 at 27 rows takes 22 us of MMAs and 46 us.  Two tiles share a
// staged activation tile (18 KB at 32 rows, twice a Q4_K tile).  Measured at 27 rows, before (64-row CTAs, scales applied to the MMA
// results) and now: gate_up Q4_K 56 -> 46 us, IQ3_S 71 -> 57, Q2_K 63 -> 48, Q3_K 67 -> 54; two slabs to a warp (half the loads of
// activations, half the warps) 47, 58, 50, 59, and 67 against 53 where the two halves of the run differ in type.
#define GQ_WIDE_WARPS 8                   // consumer warps
template <int MT>
__global__ void __launch_bounds__(32 * (GQ_WIDE_WARPS + 1), 2) gemv_wide_kernel(const __grid_constant__ GemvParams p) {
    constexpr int xbytes = gq_stage_xbytes<MT, 0>();
    extern __shared__ __align__(128) uint8_t smem[];
    // layout: [stages x (tile 0 | tile 1 | activation tile)] [full barriers] [empty barriers] [codebook tables of the two tiles]; the
    // reduction of a split reuses the ring
    const int stages = p.stages, wmax = p.wbytes_max, M = p.M;
    const int stage_bytes = 2 * wmax + xbytes;
    uint64_t *full = reinterpret_cast<uint64_t *>(smem + (size_t)stages * stage_bytes);
    uint64_t *empty = full + stages;
    uint8_t *tables = reinterpret_cast<uint8_t *>(empty + stages);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int unit = (int)(blockIdx.x / (unsigned)p.split), part = (int)blockIdx.x - unit * p.split;
    // tile `unit` of the first half of the run and its counterpart of the second: in a run of several types every CTA gets its share of each
    const int half = (p.n_tiles + 1) >> 1;
    const bool two = unit + half < p.n_tiles;
    const int32_t *d0 = p.desc + ((int64_t)unit * p.split + part) * GQ_DESC_WORDS, *d1 = two ? d0 + (int64_t)half * p.split * GQ_DESC_WORDS : d0;
    const int type0 = d0[1], type1 = d1[1], kb0 = d0[4], kb1 = d0[5], nk = kb1 - kb0;
    const int tb0 = 64 * gq_type_bytes(type0), tb1 = two ? 64 * gq_type_bytes(type1) : 0;

    // a tile whose type contradicts the call's run_info (a wider stage, or a codebook type it did not announce, which has no table space):
    // report and leave (every CTA of a cluster works on the same tiles, so a cluster leaves as one)
    const auto bad = [&](int type) { return gq_type_bytes(type) == 0 || 64 * gq_type_bytes(type) > wmax || (gq_cb_kind(type) >= 0 && gq_cb_bytes(gq_cb_kind(type)) > p.cb_bytes); };
    if (bad(type0) || bad(type1)) {
        if (threadIdx.x == 0) { pdl_wait(); report_status(p.status, GQ_DEV_BAD_SHAPE); }      // after the preparation kernel has cleared the word
        return;
    }
    if (threadIdx.x == 0) {
        for (int s = 0; s < stages; ++s) { mbar_init(full + s, 1); mbar_init(empty + s, two ? GQ_WIDE_WARPS : GQ_WIDE_WARPS / 2); }
        fence_barrier_init();
    }
    __syncthreads();

    if (warp == GQ_WIDE_WARPS) {
        // ---- producer: one thread.  The weights do not depend on the kernel in front of this one, so the first stages' weight copies
        // go out before the dependency wait; the activation tiles (written by the preparation kernel) follow it ----
        if (lane == 0) {
            const uint8_t *src0 = p.packed + (int64_t)d0[0] * 16 + (int64_t)kb0 * tb0, *src1 = p.packed + (int64_t)d1[0] * 16 + (int64_t)kb0 * tb1;
            const uint32_t abytes = (uint32_t)gq_x_tile_bytes(M);
            const uint8_t *xsrc = p.xt + (int64_t)kb0 * abytes;
            const auto weights = [&](int i, int s) {
                uint8_t *st = smem + (size_t)s * stage_bytes;
                mbar_expect_tx(full + s, (uint32_t)(tb0 + tb1) + abytes);
                bulk_g2s(st, src0 + (int64_t)i * tb0, (uint32_t)tb0, full + s);
                if (tb1) bulk_g2s(st + wmax, src1 + (int64_t)i * tb1, (uint32_t)tb1, full + s);
            };
            const int pre = nk < stages ? nk : stages;
            for (int i = 0; i < pre; ++i) weights(i, i);
            pdl_wait();
            for (int i = 0; i < pre; ++i) bulk_g2s(smem + (size_t)i * stage_bytes + 2 * wmax, xsrc + (int64_t)i * abytes, abytes, full + i);
            if (nk - pre <= 2) pdl_trigger();
            for (int i = pre, s = 0, round = 1; i < nk; ++i) {
                if (!mbar_wait_parked(empty + s, (round - 1) & 1)) { report_status(p.status, GQ_DEV_TIMEOUT); break; }
                weights(i, s);
                bulk_g2s(smem + (size_t)s * stage_bytes + 2 * wmax, xsrc + (int64_t)i * abytes, abytes, full + s);
                if (i == nk - 3) pdl_trigger();
                if (++s == stages) { s = 0; ++round; }
            }
        } else if (p.pf_ptr) {
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
        __syncwarp();
        cluster_sync_all();     // the cluster barriers of the reduction need every thread of every CTA
        cluster_sync_all();
        return;
    }

    // ---- consumers ----
    const int tile = warp >> 2, row0 = 16 * (warp & 3);
    const bool live = tile == 0 || two;
    const int32_t *d = tile ? d1 : d0;
    const int type = tile ? type1 : type0;
    float acc[MT][4];
#pragma unroll
    for (int nt = 0; nt < MT; ++nt) acc[nt][0] = acc[nt][1] = acc[nt][2] = acc[nt][3] = 0.f;
    if (p.cb_bytes) {       // both tables (of a run of one type: the same one twice over, at the same place)
        uint8_t *mine = tables + tile * p.cb_stride;
        if (p.cb_stride) { if (live) fill_codebook(type, mine, threadIdx.x % (16 * GQ_WIDE_WARPS), 16 * GQ_WIDE_WARPS); }
        else fill_codebook(type0, tables, threadIdx.x, 32 * GQ_WIDE_WARPS);
        asm volatile("bar.sync 1, %0;" ::"n"(32 * GQ_WIDE_WARPS) : "memory");
    }
    bool ok = true;
    if (live) {
        DecAux aux;
        aux.grid = reinterpret_cast<const uint32_t *>(tables + tile * p.cb_stride);
        aux.iq4 = iq4_table_biased();
        Ring ring;
        ring.smem = smem; ring.full = full; ring.empty = empty;
        ring.stages = stages; ring.stage_bytes = stage_bytes; ring.wmax = wmax; ring.nk = nk;
        ring.ar_counter = nullptr;
        const int slab_off = tile * wmax + row0 * gq_type_bytes(type);
#define GQ_CONSUME(T) case T: ok = consume<T, MT>(ring, 2 * wmax, M * GQ_X_ROW, slab_off, aux, lane, acc); break;
        switch (type) {
            GQ_CONSUME(GQ_Q4_0) GQ_CONSUME(GQ_Q5_0) GQ_CONSUME(GQ_Q8_0) GQ_CONSUME(GQ_Q2_K) GQ_CONSUME(GQ_Q3_K) GQ_CONSUME(GQ_Q4_K)
            GQ_CONSUME(GQ_Q5_K) GQ_CONSUME(GQ_Q6_K) GQ_CONSUME(GQ_IQ4_NL) GQ_CONSUME(GQ_IQ3_S) GQ_CONSUME(GQ_IQ4_XS) GQ_CONSUME(GQ_IQ3_XXS)
            GQ_CONSUME(GQ_IQ2_XXS) GQ_CONSUME(GQ_IQ2_XS) GQ_CONSUME(GQ_IQ2_S) GQ_CONSUME(GQ_IQ1_M)
        }
#undef GQ_CONSUME
    }
    if (!ok && lane == 0) report_status(p.status, GQ_DEV_TIMEOUT);   // the result is then incomplete; the status word says so

    // ---- epilogue: rows of the MMA are output columns, columns of the MMA are batch rows ----
    if (p.cluster) {
        // split-K inside a cluster: every CTA parks its accumulators in its ring, which all its consumers have finished with; the slabs
        // are dealt out over the CTAs, and the warp that owns slab i in CTA i % split adds the parts in split order through distributed
        // shared memory.  No partial sums in HBM, no second kernel, a fixed order of the additions.
        asm volatile("bar.sync 1, %0;" ::"n"(32 * GQ_WIDE_WARPS) : "memory");
        float4 *park = reinterpret_cast<float4 *>(smem) + warp * MT * 32 + lane;
#pragma unroll
        for (int nt = 0; nt < MT; ++nt) park[nt * 32] = make_float4(acc[nt][0], acc[nt][1], acc[nt][2], acc[nt][3]);
        cluster_sync_all();
        const bool mine = live && warp % p.split == part;
        if (mine) {
#pragma unroll
            for (int nt = 0; nt < MT; ++nt) acc[nt][0] = acc[nt][1] = acc[nt][2] = acc[nt][3] = 0.f;
            for (int r = 0; r < p.split; ++r) {
                const uint32_t peer = map_to_rank(smem_u32(park), (uint32_t)r);
#pragma unroll
                for (int nt = 0; nt < MT; ++nt) {
                    const float4 v = ld_cluster_f4(peer + (uint32_t)(nt * 512));
                    acc[nt][0] += v.x; acc[nt][1] += v.y; acc[nt][2] += v.z; acc[nt][3] += v.w;
                }
            }
        }
        cluster_sync_all();      // the peers have read this CTA's shared memory
        if (!mine) return;
    }
    if (!live) return;
    const int g = lane >> 2, t = lane & 3;
    const int col0 = d[2], nvalid = d[3];
    if (p.ar.world > 0 && (p.split == 1 || p.cluster)) {
        // tensor parallel, row-parallel layer: this rank's partial output does not go to y but, as bf16, through the warp's scratch to
        // every rank; y receives the sum over ranks (fused_allreduce_block)
        uint32_t prev = 0;
        const int ar_unit = (unit + tile * half) * GQ_CONSUMER_WARPS + (warp & 3);
        if (lane == 0) prev = *reinterpret_cast<const volatile uint32_t *>(p.ar.counters + ar_unit);
        __nv_bfloat16 *blk = reinterpret_cast<__nv_bfloat16 *>(smem + p.ar_at + warp * MT * 512);
#pragma unroll
        for (int nt = 0; nt < MT; ++nt)
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int rl = g + 8 * (j >> 1), n = nt * 8 + 2 * t + (j & 1);
                const bool valid = ok && row0 + rl < nvalid && n < p.M;
                blk[n * 16 + rl] = __float2bfloat16_rn(valid ? acc[nt][j] : 0.0f);
            }
        __syncwarp();
        const int ncols = nvalid - row0 < 16 ? nvalid - row0 : 16;
        if (ncols > 0) {
            if (((col0 | ncols | (int)p.n_total) & 1) && lane == 0) report_status(p.status, GQ_DEV_BAD_SHAPE);    // pairs of columns travel together
            else fused_allreduce_block(p, reinterpret_cast<const uint32_t *>(blk), ar_unit, col0 + row0, ncols, lane, prev);
        }
        return;
    }
#pragma unroll
    for (int nt = 0; nt < MT; ++nt)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int r = row0 + g + 8 * (j >> 1);           // row inside the 64-row tile
            const int n = nt * 8 + 2 * t + (j & 1);          // batch row
            if (ok && r < nvalid && n < p.M) {
                if (p.split == 1 || p.cluster) p.y[(int64_t)n * p.ldy + col0 + r] = __float2bfloat16_rn(acc[nt][j]);
                else p.partials[((int64_t)part * p.part_rows + n) * p.n_total + col0 + r] = acc[nt][j];
            }
        }
}
