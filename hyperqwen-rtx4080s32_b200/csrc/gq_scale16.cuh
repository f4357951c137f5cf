// Sub-block scales of the register decoders (gq_decode.cuh) as fp16, for the path that multiplies them into the weights.
// hscales<J>(dec, h, s): the scales d * sc of the 16-weight runs 4J .. 4J+3 of row half h, each rounded once to fp16, two to a
// register: types with a scale per 32 weights leave both in s[0], the others use s[0] and s[1].  hmins<J>: minus the minimum
// terms, - dmin * m, likewise.  scale_of<GROUP, R>(s): run R's scale in both halves (a swizzle of the multiply's operand).
// Everything is packed fp16 arithmetic: a scale field is dropped into the mantissa of a constant (exact integer), the constant
// is taken off (exact) and the product with d is the only rounding — the value of the fp32 product rounded to fp16, at about
// two instructions per scale instead of four or five.
#pragma once
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
__device__ __forceinline__ void scales_of_bytes(uint32_t word, __half2 d, uint32_t (&s)[2]) {
    s[0] = mul_d(hsub2(bytes_h2(word, 0x5150u), h2k(1024 + BIAS)), d);
    s[1] = mul_d(hsub2(bytes_h2(word, 0x5352u), h2k(1024 + BIAS)), d);
}

template <int J, int TYPE>
__device__ __forceinline__ void hscales(const Dec<TYPE> &dec, int h, uint32_t (&s)[2]) {
    if constexpr (TYPE == GQ_Q4_K || TYPE == GQ_Q5_K) {
        const uint32_t a = bytes_h2(dec.sc[h][J >> 1], (J & 1) ? 0x5352u : 0x5150u);
        s[0] = mul_d(hsub2(a, h2k(1024)), lo2(dec.dd[h]));
    } else if constexpr (TYPE == GQ_Q6_K) {
        scales_of_bytes<128>(w4(dec.sc[h], J), lo2(dec.dd[h]), s);
    } else if constexpr (TYPE == GQ_Q2_K) {
        scales_of_bytes<0>(w4(dec.sc[h], J), lo2(dec.dd[h]), s);
    } else if constexpr (TYPE == GQ_Q3_K) {
        scales_of_bytes<32>(dec.sv[h][J], lo2(dec.dd[h]), s);
    } else if constexpr (TYPE == GQ_IQ4_XS) {
        const uint32_t a = bytes_h2(dec.ls[h][J >> 1], (J & 1) ? 0x5352u : 0x5150u);
        s[0] = mul_d(hsub2(a, h2k(1056)), lo2(dec.dd[h]));
    } else if constexpr (TYPE == GQ_Q8_0 || TYPE == GQ_Q4_0 || TYPE == GQ_Q5_0 || TYPE == GQ_IQ4_NL) {
        s[0] = w4(dec.d8[h], J);
    } else if constexpr (TYPE == GQ_IQ3_S) {
        // bytes J of the even and the odd sub-blocks' words side by side
        const uint32_t x = and_or(prmt(dec.sce[h], dec.sco[h], 0x11u * J + 0x1100u * (4 + J)), 0x000f000fu, GQ_MAGIC_B0);
        s[0] = mul_d(hfma2(x, h2k(2), h2k(-2047)), lo2(dec.dd[h]));
    } else if constexpr (TYPE == GQ_IQ3_XXS || TYPE == GQ_IQ2_XXS) {
        constexpr double c = TYPE == GQ_IQ3_XXS ? 0.25 : 0.125;
        const uint32_t x = (dec.sw[h][2 * J] >> 28) | and_or(dec.sw[h][2 * J + 1] >> 12, 0x000f0000u, GQ_MAGIC_B0);
        s[0] = mul_d(hfma2(x, h2k(2 * c), h2k(-2047 * c)), lo2(dec.dd[h]));
    } else if constexpr (TYPE == GQ_IQ2_XS || TYPE == GQ_IQ2_S) {
        // a byte holds the nibbles of two runs: repeated in both halves, the low one is read at bit 0, the high one at bit 4
        const uint32_t w = J < 2 ? dec.sc[h].x : dec.sc[h].y;
        const uint32_t a = and_or(prmt(w, w, (J & 1) ? 0x2222u : 0x0000u), 0x00f0000fu, 0x54006400u);
        const uint32_t b = and_or(prmt(w, w, (J & 1) ? 0x3333u : 0x1111u), 0x00f0000fu, 0x54006400u);
        s[0] = mul_d(hfma2(a, h2k(0.25), h2two(-2047 * 0.125, -127 * 0.125)), lo2(dec.dd[h]));
        s[1] = mul_d(hfma2(b, h2k(0.25), h2two(-2047 * 0.125, -127 * 0.125)), lo2(dec.dd[h]));
    } else if constexpr (TYPE == GQ_IQ1_M) {
        // four 3-bit fields in halfword J: two at bits 0 and 3, two more six bits higher
        const uint32_t w = J < 2 ? dec.sc[h].x : dec.sc[h].y, y = prmt(w, w, (J & 1) ? 0x3232u : 0x1010u);
        const uint32_t a = and_or(y, 0x00380007u, 0x58006400u), b = and_or(y >> 6, 0x00380007u, 0x58006400u);
        s[0] = mul_d(hfma2(a, h2k(0.25), h2two(-2047 * 0.125, -255 * 0.125)), lo2(dec.dd[h]));
        s[1] = mul_d(hfma2(b, h2k(0.25), h2two(-2047 * 0.125, -255 * 0.125)), lo2(dec.dd[h]));
    }
}

template <int J, int TYPE>
__device__ __forceinline__ void hmins(const Dec<TYPE> &dec, int h, uint32_t (&m)[2]) {
    const __half2 nd = __hneg2(hi2(dec.dd[h]));
    if constexpr (TYPE == GQ_Q2_K) scales_of_bytes<0>(w4(dec.mn[h], J), nd, m);
    else m[0] = mul_d(hsub2(bytes_h2(dec.mn[h][J >> 1], (J & 1) ? 0x5352u : 0x5150u), h2k(1024)), nd);
}

}  // namespace gq
