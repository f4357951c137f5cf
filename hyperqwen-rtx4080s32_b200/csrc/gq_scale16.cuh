// Sub-block scales of the register decoders (gq_decode.cuh) as fp16 pairs, for the path that multiplies them into the weights.
// hscales<J>(dec, h, s): the scales of the four 16-weight runs 4J .. 4J+3 of row half h, d * sc each rounded once to fp16 and
// repeated in both halves of s[r]; hmins<J>: minus the minimum terms, - dmin * m, likewise.
// Everything is packed fp16 arithmetic: a scale field is dropped into the mantissa of a constant (exact integer), the constant
// is taken off (exact) and the product with d is the only rounding — the value of the fp32 product rounded to fp16, at about
// two instructions per scale instead of four or five.
#pragma once
#include "gq_decode.cuh"

namespace gq {

__device__ __forceinline__ uint32_t splat_lo(uint32_t v) { return prmt(v, v, 0x1010u); }
__device__ __forceinline__ uint32_t splat_hi(uint32_t v) { return prmt(v, v, 0x3232u); }
// fp16 constants of both halves
constexpr uint32_t h2two(double lo, double hi) { return hc(lo) | (hc(hi) << 16); }

// scales given as one byte per run (stored plus bias): word = the four runs' bytes
template <int BIAS>
__device__ __forceinline__ void scales_of_bytes(uint32_t word, uint32_t d2, uint32_t (&s)[4]) {
    constexpr uint32_t b2 = h2k(1024 + BIAS);
    const uint32_t a = hmul2(hsub2(bytes_h2(word, 0x5150u), b2), d2), b = hmul2(hsub2(bytes_h2(word, 0x5352u), b2), d2);
    s[0] = splat_lo(a); s[1] = splat_hi(a); s[2] = splat_lo(b); s[3] = splat_hi(b);
}
// one scale per 32 weights: a = the fp16 pair (groups 2J, 2J + 1)
__device__ __forceinline__ void scales_of_pair(uint32_t a, uint32_t (&s)[4]) {
    s[0] = s[1] = splat_lo(a);
    s[2] = s[3] = splat_hi(a);
}
template <int J, int TYPE>
__device__ __forceinline__ void hscales(const Dec<TYPE> &dec, int h, uint32_t (&s)[4]) {
    if constexpr (TYPE == GQ_Q4_K || TYPE == GQ_Q5_K) {
        const uint32_t a = bytes_h2(dec.sc[h][J >> 1], (J & 1) ? 0x5352u : 0x5150u);
        scales_of_pair(hmul2(hsub2(a, h2k(1024)), splat_lo(dec.dd[h])), s);
    } else if constexpr (TYPE == GQ_Q6_K) {
        scales_of_bytes<128>(w4(dec.sc[h], J), splat_lo(dec.dd[h]), s);
    } else if constexpr (TYPE == GQ_Q2_K) {
        scales_of_bytes<0>(w4(dec.sc[h], J), splat_lo(dec.dd[h]), s);
    } else if constexpr (TYPE == GQ_Q3_K) {
        scales_of_bytes<32>(dec.sv[h][J], splat_lo(dec.dd[h]), s);
    } else if constexpr (TYPE == GQ_IQ4_XS) {
        const uint32_t a = bytes_h2(dec.ls[h][J >> 1], (J & 1) ? 0x5352u : 0x5150u);
        scales_of_pair(hmul2(hsub2(a, h2k(1056)), splat_lo(dec.dd[h])), s);
    } else if constexpr (TYPE == GQ_Q8_0 || TYPE == GQ_Q4_0 || TYPE == GQ_Q5_0 || TYPE == GQ_IQ4_NL) {
        scales_of_pair(w4(dec.d8[h], J), s);
    } else if constexpr (TYPE == GQ_IQ3_S) {
        // bytes J of the even and the odd sub-blocks' words side by side
        const uint32_t x = and_or(prmt(dec.sce[h], dec.sco[h], 0x11u * J + 0x1100u * (4 + J)), 0x000f000fu, GQ_MAGIC_B0);
        scales_of_pair(hmul2(hfma2(x, h2k(2), h2k(-2047)), splat_lo(dec.dd[h])), s);
    } else if constexpr (TYPE == GQ_IQ3_XXS || TYPE == GQ_IQ2_XXS) {
        constexpr double c = TYPE == GQ_IQ3_XXS ? 0.25 : 0.125;
        const uint32_t x = (dec.sw[h][2 * J] >> 28) | and_or(dec.sw[h][2 * J + 1] >> 12, 0x000f0000u, GQ_MAGIC_B0);
        scales_of_pair(hmul2(hfma2(x, h2k(2 * c), h2k(-2047 * c)), splat_lo(dec.dd[h])), s);
    } else if constexpr (TYPE == GQ_IQ2_XS || TYPE == GQ_IQ2_S) {
        // a byte holds the nibbles of two runs: repeated in both halves, the low one is read at bit 0, the high one at bit 4
        const uint32_t w = J < 2 ? dec.sc[h].x : dec.sc[h].y;
        const uint32_t d2 = splat_lo(dec.dd[h]);
        const uint32_t a = and_or(prmt(w, w, (J & 1) ? 0x2222u : 0x0000u), 0x00f0000fu, 0x54006400u);
        const uint32_t b = and_or(prmt(w, w, (J & 1) ? 0x3333u : 0x1111u), 0x00f0000fu, 0x54006400u);
        const uint32_t ea = hmul2(hfma2(a, h2k(0.25), h2two(-2047 * 0.125, -127 * 0.125)), d2);
        const uint32_t eb = hmul2(hfma2(b, h2k(0.25), h2two(-2047 * 0.125, -127 * 0.125)), d2);
        s[0] = splat_lo(ea); s[1] = splat_hi(ea); s[2] = splat_lo(eb); s[3] = splat_hi(eb);
    } else if constexpr (TYPE == GQ_IQ1_M) {
        // four 3-bit fields in halfword J: two at bits 0 and 3, two more six bits higher
        const uint32_t w = J < 2 ? dec.sc[h].x : dec.sc[h].y, y = (J & 1) ? splat_hi(w) : splat_lo(w);
        const uint32_t d2 = splat_lo(dec.dd[h]);
        const uint32_t a = and_or(y, 0x00380007u, 0x58006400u), b = and_or(y >> 6, 0x00380007u, 0x58006400u);
        const uint32_t ea = hmul2(hfma2(a, h2k(0.25), h2two(-2047 * 0.125, -255 * 0.125)), d2);
        const uint32_t eb = hmul2(hfma2(b, h2k(0.25), h2two(-2047 * 0.125, -255 * 0.125)), d2);
        s[0] = splat_lo(ea); s[1] = splat_hi(ea); s[2] = splat_lo(eb); s[3] = splat_hi(eb);
    }
}

template <int J, int TYPE>
__device__ __forceinline__ void hmins(const Dec<TYPE> &dec, int h, uint32_t (&m)[4]) {
    const uint32_t nd = splat_hi(dec.dd[h]) ^ 0x80008000u;
    if constexpr (TYPE == GQ_Q2_K) scales_of_bytes<0>(w4(dec.mn[h], J), nd, m);
    else scales_of_pair(hmul2(hsub2(bytes_h2(dec.mn[h][J >> 1], (J & 1) ? 0x5352u : 0x5150u), h2k(1024)), nd), m);
}

}  // namespace gq
