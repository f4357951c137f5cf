// Sub-block scales of the register decoders (gq_decode.cuh) as fp16, for the path that multiplies them into the weights.
// hscales<J>(dec, h, s): the scales d * sc of the 16-weight runs 4J .. 4J+3 of row half h, each rounded once to fp16, two to a
// register: types with a scale per 32 weights leave both in s[0], the others use s[0] and s[1].  hmins<J>: minus the minimum
// terms, - dmin * m, likewise.  scale_of<GROUP, R>(s): run R's scale in both halves (a swizzle of the multiply's operand).
// Everything is packed fp16 arithmetic: a scale field is dropped into the mantissa of a constant (exact integer), the constant
// is taken off (exact, `iscales`) and the product with d is the only rounding — the value of the fp32 product rounded to fp16, at about
// two instructions per scale instead of four or five.
#pragma once
#include <type_traits>
#include "gq_decode.cuh"

namespace gq {

__device__ __forceinline__ __half2 lo2(uint32_t v) { return __low2half2(u32_as_h2(v)); }
__device__ __forceinline__ __half2 hi2(uint32_t v) { return __high2half2(u32_as_h2(v)); }
// fp16 constants of both halves
constexpr uint32_t h2two(double lo, double hi) { return hc(lo) | (hc(hi) << 16); }
__device__ __forceinline__ uint32_t mul_d(uint32_t sc, __half2 d) { return h2_as_u32(__hmul2(u32_as_h2(sc), d)); }

template <int GROUP, int R>
__device__ __forceinline__ __half2 scale_of(const uint32_t (&s)[2]) {
    if constexpr (GROUP == 32) return R < 2 ? lo2(s[0]) : hi2(s[0]);
    else return (R & 1) ? hi2(s[R >> 1]) : lo2(s[R >> 1]);
}

// scales given as one byte per run (stored plus bias): word = the four runs' bytes
template <int BIAS>
__device__ __forceinline__ void ints_of_bytes(uint32_t word, uint32_t (&s)[2]) {
    s[0] = hsub2(bytes_h2(word, 0x5150u), h2k(1024 + BIAS));
    s[1] = hsub2(bytes_h2(word, 0x5352u), h2k(1024 + BIAS));
}

// the scale fields themselves, as exact fp16 integers; of the types with a constant factor besides d (a quarter, an eighth) times that
// factor, or without it (FACTOR = false).  Not for the types whose only scale is an fp16 d per 32 weights.
template <int J, bool FACTOR, int TYPE>
__device__ __forceinline__ void iscales(const Dec<TYPE> &dec, int h, uint32_t (&s)[2]) {
    if constexpr (TYPE == GQ_Q4_K || TYPE == GQ_Q5_K) {
        s[0] = hsub2(bytes_h2(dec.sc[h][J >> 1], (J & 1) ? 0x5352u : 0x5150u), h2k(1024));
    } else if constexpr (TYPE == GQ_Q6_K) {
        ints_of_bytes<128>(w4(dec.sc[h], J), s);
    } else if constexpr (TYPE == GQ_Q2_K) {
        ints_of_bytes<0>(w4(dec.sc[h], J), s);
    } else if constexpr (TYPE == GQ_Q3_K) {
        ints_of_bytes<32>(dec.sv[h][J], s);
    } else if constexpr (TYPE == GQ_IQ4_XS) {
        s[0] = hsub2(bytes_h2(dec.ls[h][J >> 1], (J & 1) ? 0x5352u : 0x5150u), h2k(1056));
    } else if constexpr (TYPE == GQ_IQ3_S) {
        // bytes J of the even and the odd sub-blocks' words side by side
        const uint32_t x = and_or(prmt(dec.sce[h], dec.sco[h], 0x11u * J + 0x1100u * (4 + J)), 0x000f000fu, GQ_MAGIC_B0);
        s[0] = hfma2(x, h2k(2), h2k(-2047));
    } else if constexpr (TYPE == GQ_IQ3_XXS || TYPE == GQ_IQ2_XXS) {
        constexpr double c = !FACTOR ? 1.0 : TYPE == GQ_IQ3_XXS ? 0.25 : 0.125;
        const uint32_t x = (dec.sw[h][2 * J] >> 28) | and_or(dec.sw[h][2 * J + 1] >> 12, 0x000f0000u, GQ_MAGIC_B0);
        s[0] = hfma2(x, h2k(2 * c), h2k(-2047 * c));
    } else if constexpr (TYPE == GQ_IQ2_XS || TYPE == GQ_IQ2_S) {
        // a byte holds the nibbles of two runs: repeated in both halves, the low one is read at bit 0, the high one at bit 4
        constexpr double c = FACTOR ? 0.125 : 1.0;
        const uint32_t w = J < 2 ? dec.sc[h].x : dec.sc[h].y;
        const uint32_t a = and_or(prmt(w, w, (J & 1) ? 0x2222u : 0x0000u), 0x00f0000fu, 0x54006400u);
        const uint32_t b = and_or(prmt(w, w, (J & 1) ? 0x3333u : 0x1111u), 0x00f0000fu, 0x54006400u);
        s[0] = hfma2(a, h2k(2 * c), h2two(-2047 * c, -127 * c));
        s[1] = hfma2(b, h2k(2 * c), h2two(-2047 * c, -127 * c));
    } else if constexpr (TYPE == GQ_IQ1_M) {
        // four 3-bit fields in halfword J: two at bits 0 and 3, two more six bits higher
        constexpr double c = FACTOR ? 0.125 : 1.0;
        const uint32_t w = J < 2 ? dec.sc[h].x : dec.sc[h].y, y = prmt(w, w, (J & 1) ? 0x3232u : 0x1010u);
        const uint32_t a = and_or(y, 0x00380007u, 0x58006400u), b = and_or(y >> 6, 0x00380007u, 0x58006400u);
        s[0] = hfma2(a, h2k(2 * c), h2two(-2047 * c, -255 * c));
        s[1] = hfma2(b, h2k(2 * c), h2two(-2047 * c, -255 * c));
    }
}

template <int J, int TYPE>
__device__ __forceinline__ void hscales(const Dec<TYPE> &dec, int h, uint32_t (&s)[2]) {
    if constexpr (TYPE == GQ_Q8_0 || TYPE == GQ_Q4_0 || TYPE == GQ_Q5_0 || TYPE == GQ_IQ4_NL) {
        s[0] = w4(dec.d8[h], J);
    } else {
        iscales<J, true>(dec, h, s);
        s[0] = mul_d(s[0], lo2(dec.dd[h]));
        if constexpr (Dec<TYPE>::GROUP == 16) s[1] = mul_d(s[1], lo2(dec.dd[h]));
    }
}

template <int J, int TYPE>
__device__ __forceinline__ void hmins(const Dec<TYPE> &dec, int h, uint32_t (&m)[2]) {
    const __half2 nd = __hneg2(hi2(dec.dd[h]));
    if constexpr (TYPE == GQ_Q2_K) {
        ints_of_bytes<0>(w4(dec.mn[h], J), m);
        m[0] = mul_d(m[0], nd); m[1] = mul_d(m[1], nd);
    } else {
        m[0] = mul_d(hsub2(bytes_h2(dec.mn[h][J >> 1], (J & 1) ? 0x5352u : 0x5150u), h2k(1024)), nd);
    }
}

// ---- integer weights with their scale multiplied in, for the kernels that apply d once per k-block ----------------------------
// Of the types below, field x sub-block scale is an integer of at most eleven bits (Q4_K 15 x 63, Q5_K 31 x 63, Q2_K 3 x 15, Q3_K 7 x 32,
// IQ3_S 15 x 31, IQ3_XXS 62 x 31, IQ2_* 43 x 31, IQ1_M 9 x 15), so its fp16 form is exact.  The bias that the decoder leaves on a field is a
// power of two (1152 = 9 * 128 of IQ3_S), bias x scale is therefore exact too, and one fused multiply-add takes it off and multiplies.
template <int TYPE>
constexpr bool gq_folds() {
    return TYPE == GQ_Q4_K || TYPE == GQ_Q5_K || TYPE == GQ_Q2_K || TYPE == GQ_Q3_K || TYPE == GQ_IQ3_S || TYPE == GQ_IQ3_XXS || TYPE == GQ_IQ2_XXS ||
           TYPE == GQ_IQ2_XS || TYPE == GQ_IQ2_S || TYPE == GQ_IQ1_M;
}
template <int TYPE, int P>
constexpr double fold_bias() {
    return TYPE == GQ_Q4_K || TYPE == GQ_Q5_K ? ((P & 1) ? 64.0 : 1024.0) : TYPE == GQ_Q2_K || TYPE == GQ_Q3_K ? double(1024 >> (2 * (P & 3))) : TYPE == GQ_IQ3_S ? 1152.0 : 1024.0;
}
// the A operands of runs 4J .. 4J+3
template <int TYPE, int J>
__device__ __forceinline__ void fold_slice(const Dec<TYPE> &dec, uint32_t (&a)[4][4]) {
    constexpr int G = Dec<TYPE>::GROUP;
    constexpr double B0 = fold_bias<TYPE, 2 * J>(), B1 = fold_bias<TYPE, 2 * J + 1>();
    uint32_t s[2][2], nb[2][2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        iscales<J, false>(dec, h, s[h]);
        if constexpr (TYPE != GQ_IQ1_M) {
            if constexpr (G == 32) nb[h][0] = hmul2(s[h][0], h2two(-B0, -B1));
            else { nb[h][0] = hmul2(s[h][0], h2k(-B0)); nb[h][1] = hmul2(s[h][1], h2k(-B1)); }
        }
    }
    const auto run = [&](auto r_) {
        constexpr int R = decltype(r_)::value, R4 = 4 * J + R;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const __half2 sc = scale_of<G, R>(s[h]);
            if constexpr (TYPE == GQ_IQ3_XXS || TYPE == GQ_IQ2_XXS || TYPE == GQ_IQ2_XS || TYPE == GQ_IQ2_S) {
                const MagSign v = dec.template mags<R4>(h);
                const __half2 n = scale_of<G, R>(nb[h]);
                a[R][h] = xor_and(h2_as_u32(__hfma2(u32_as_h2(v.m01), sc, n)), v.s01, 0x80008000u);
                a[R][2 + h] = xor_and(h2_as_u32(__hfma2(u32_as_h2(v.m23), sc, n)), v.s23, 0x80008000u);
            } else if constexpr (TYPE == GQ_IQ1_M) {       // its bias is odd: the decoder takes it off
                a[R][h] = h2_as_u32(__hmul2(u32_as_h2(a[R][h]), sc));
                a[R][2 + h] = h2_as_u32(__hmul2(u32_as_h2(a[R][2 + h]), sc));
            } else {
                const __half2 n = scale_of<G, R>(nb[h]);
                a[R][h] = h2_as_u32(__hfma2(u32_as_h2(a[R][h]), sc, n));
                a[R][2 + h] = h2_as_u32(__hfma2(u32_as_h2(a[R][2 + h]), sc, n));
            }
        }
    };
    if constexpr (!(TYPE == GQ_IQ3_XXS || TYPE == GQ_IQ2_XXS || TYPE == GQ_IQ2_XS || TYPE == GQ_IQ2_S)) {
        uint32_t p[2][2][4];
        dec.template pair<2 * J>(p[0]);
        dec.template pair<2 * J + 1>(p[1]);
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int k = 0; k < 4; ++k) a[i][k] = p[i >> 1][i & 1][k];
    }
    run(std::integral_constant<int, 0>{}); run(std::integral_constant<int, 1>{}); run(std::integral_constant<int, 2>{}); run(std::integral_constant<int, 3>{});
}
// what is left for the correction MMA (the minimum term; Q3_K: the -4 of its field)
template <int TYPE>
constexpr bool fold_has_corr() { return TYPE == GQ_Q4_K || TYPE == GQ_Q5_K || TYPE == GQ_Q2_K || TYPE == GQ_Q3_K; }

}  // namespace gq
