// The grouped kernel's fp16 form, for batches of more rows than the integer form takes: the consumer side of a CTA.
// mma.sync m16n8k16 with the weights on M as exact fp16 integers and the activations as fp16 on N.
// (included after Ring and the workspace layout)
#pragma once
#include "gq_scale16.cuh"

// Pairs of runs whose MMAs follow one another in one accumulator before it is added in fp32: the tensor core truncates where an fp32 add rounds,
// so a chain over the whole k-block (eight pairs) left the codebook types with two to three times the error of a form that adds up each
// scale group's sum in fp32 (rms over the norm of the products, N(0, 1) activations: IQ2_S 1.85e-7 against 7.6e-8, by pairs 7.3e-8; IQ3_S 1.4e-7
// against 6.3e-8, 6.7e-8).  The types with a minimum or an offset lose far more in that form (Q4_K 6.8e-6, with the fold 1.4e-7) and keep the
// long chain.  Whole calls at 27 rows, eight pairs / one: 34,816 x 5,120 IQ3_S 56 / 60 us, IQ2_XS 64 / 65.
template <int TYPE>
constexpr int gq_fold_chain() { return gq_cb_kind(TYPE) >= 0 ? 1 : 8; }

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
        constexpr int CHAIN = gq_fold_chain<TYPE>(), GRP = CHAIN == 1 && MT > 4 ? 4 : MT;      // short chains: four column tiles' sums at a time
        float sum[GRP][4];
        static_for<0, 4>([&](auto j_) {
            constexpr int J = decltype(j_)::value;
            uint32_t a[4][4];
            fold_slice<TYPE, J>(dec, a);
            static_for<0, 2 * (MT / GRP)>([&](auto p_) {
                constexpr int P = decltype(p_)::value / (MT / GRP), N0 = decltype(p_)::value % (MT / GRP) * GRP, Q = 2 * J + P;
                // the MMAs of the two runs of a pair accumulate into the same registers: the other column tiles stand between them
                uint4 b[GRP];
#pragma unroll
                for (int n = 0; n < GRP; ++n) {
                    b[n] = ld16(xb + (N0 + n) * 8 * GQ_X_ROW + 64 * Q);
                    if constexpr (Q % CHAIN == 0) mma16816_z(sum[n], a[2 * P], b[n].x, b[n].y, z);
                    else mma16816(sum[n], a[2 * P], b[n].x, b[n].y);
                }
#pragma unroll
                for (int n = 0; n < GRP; ++n) mma16816(sum[n], a[2 * P + 1], b[n].z, b[n].w);
                if constexpr (Q % CHAIN == CHAIN - 1) {
#pragma unroll
                    for (int n = 0; n < GRP; ++n)
#pragma unroll
                        for (int j = 0; j < 4; ++j) blk[N0 + n][j] = Q < CHAIN ? sum[n][j] : blk[N0 + n][j] + sum[n][j];
                }
            });
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
        const float2 sx = *reinterpret_cast<const float2 *>(xs + xs_off + (nt * 8 + 2 * t) * 4);
        if constexpr (C0 == NC) {           // sx is a power of two: d * sx is exact
#pragma unroll
            for (int j = 0; j < 4; ++j) acc[nt][j] = fmaf(d[j >> 1] * (j & 1 ? sx.y : sx.x), blk[nt][j], acc[nt][j]);
        } else {
            float tot[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) tot[j] = d[j >> 1] * blk[nt][j];
            const uint4 b = ld16(xs + (nt * 8 + g) * GQ_X_ROW + GQ_X_SUMS + 16 * t);
#pragma unroll
            for (int c = C0; c < NC; ++c) {
                float mm[4];
                mma16816_z(mm, ac[c], b.x, b.y, z);
                mma16816(mm, ac[c], b.z, b.w);
#pragma unroll
                for (int j = 0; j < 4; ++j) tot[j] = fmaf(-fc[c][j >> 1], mm[j], tot[j]);
            }
#pragma unroll
            for (int j = 0; j < 4; ++j) acc[nt][j] = fmaf(j & 1 ? sx.y : sx.x, tot[j], acc[nt][j]);
        }
    }
}

template <int TYPE, int MT>
__device__ __forceinline__ bool consume(const Ring &r, int xs_off, int slab_off, const DecAux &aux, int lane, float (&acc)[MT][4], uint32_t &ar_prev) {
    const float z[4] = {0.f, 0.f, 0.f, 0.f};
    if (!ring_read_counter(r, lane, ar_prev)) return false;
    for (int i = 0, s = 0, round = 0; i < r.nk; ++i) {
        if (!mbar_wait(r.full + s, round & 1)) return false;
        const uint8_t *st = r.smem + (size_t)s * r.stage_bytes;
        slab_kblock<TYPE, MT>(st + slab_off, st + r.wmax, xs_off, aux, lane, acc, z);
        __syncwarp();
        if (lane == 0) mbar_arrive(r.empty + s);
        if (++s == r.stages) { s = 0; ++round; }
    }
    return true;
}
