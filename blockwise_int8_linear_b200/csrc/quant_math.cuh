// The arithmetic of one quantisation block (reference kernel triton_functions.py:397-403), shared by the standalone
// quantizers and by the GEMM that quantizes its activations on load.
#pragma once

#include "bi8_common.cuh"

namespace bi8 {

constexpr float kMagic = 12582912.0f;  // 1.5 * 2^23: adding it rounds to integer (RNE) in the low mantissa bits

// Quantizer of one block: scale and the reciprocal used by the exact-division shortcut.
//
// For operands with at most 11 significant bits (bf16, fp16) the correctly rounded fp32 quotient a/b is
//   q0 = a*r;  e = fma(-b, q0, a);  q1 = fma(e, r, q0)        with r = RN(1/b):
// e is exact, q0 + e/b is the exact quotient, and the quotient of two such short operands is either
// representable or at least 2^-13 ulp away from a rounding boundary, far more than the error of e*r.
// For fp32 operands, and for scales outside [2^-100, 2^100], the IEEE division is used directly.
//
// `once`: the byte needs no quotient.  With X and S the significands of x and the scale as integers below 2^11 and 2^k the ratio of their
// units, 127 x / s lies at least 2^-19 of its value away from every n + 1/2 that it does not equal: |254 X 2^k - (2n + 1) S| is an integer, or
// one divided by 2^-k, and 254 X < 2^19.  Both fl(127 fl(x / s)) (off by less than 2^-23 of its value) and x * r, r within 2^-21 above 127 / s,
// then round to the same integer.  Equality, 254 X 2^k = (2n + 1) S, asks for a factor of 127 on the right.  In 2n + 1: n = 63 and
// x = s / 2, where the quotient is exact and 63.5 goes to 64, as does x * r, which is 63.5 or more.  Or in S, the scale's 11 significant bits a
// multiple of 127: there fl(127 fl(x / s)) goes to the even neighbour (all pairs of 11-bit numbers tried), and x * r does too where 127 / s is a
// power of two and r exactly that (S = 2032, the only such bf16 scale); the other seven fp16 ones have no `once`.  One fused operation replaces
// five, which at two issue cycles a packed pair were most of the tile quantizer; taken there and in the streaming row-wise kernel, not where
// fp16 would need the code of both (rows of any alignment, 8192 x 12289: 98.4 us without, 100.4 with) or few values are quantized.
struct BlockQ {
    float scale;
    float rcp;
    bool fast, once;
    __device__ __forceinline__ void set(float amax, bool short_mantissa) {
        scale = amax;
        fast = short_mantissa && amax > 7.8886090522101181e-31f && amax < 1.2676506002282294e30f;
        rcp = fast ? __frcp_rn(amax) : 0.0f;
        const uint32_t sig = significand();
        once = fast && (sig == 2032u || sig % 127u != 0u);
    }
    __device__ __forceinline__ uint32_t significand() const { return ((__float_as_uint(scale) >> 13) & 0x3ffu) | 0x400u; }
    // 127 / scale, too large by less than 2^-21 of it and never too small, or exact (computed where it is used: not kept beside rcp)
    __device__ __forceinline__ float r127() const {
        return significand() == 2032u ? __fmul_rn(127.0f, rcp) : __fmul_ru(__fmul_ru(127.0f, rcp), 1.00000011920928955f);
    }
    // returns fl32(127 * fl32(x / scale)) + magic, whose low byte is the int8 result
    __device__ __forceinline__ uint32_t q(float x) const {
        if (fast) {
            float q0 = __fmul_rn(x, rcp);
            float e = __fmaf_rn(-scale, q0, x);
            float y = __fmaf_rn(e, rcp, q0);
            return __float_as_uint(__fadd_rn(__fmul_rn(127.0f, y), kMagic));
        }
        if (scale == 0.0f) return 0u;                 // 0/0: the reference stores 0
        float z = __fmul_rn(127.0f, __fdiv_rn(x, scale));
        if (!(z == z)) return 0u;                     // NaN converts to 0 in the int8 store
        return __float_as_uint(__fadd_rn(z, kMagic));
    }
};

__device__ __forceinline__ uint32_t pack4(uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
    // low bytes of a,b,c,d -> one word (a in byte 0)
    uint32_t ab = __byte_perm(a, b, 0x0040);
    uint32_t cd = __byte_perm(c, d, 0x0040);
    return __byte_perm(ab, cd, 0x5410);
}

// packed pairs of fp32 values (one 64-bit register), every operation rounded on its own
__device__ __forceinline__ uint64_t f2_pack(float lo, float hi) {
    uint64_t d;
    asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(lo), "f"(hi));
    return d;
}
__device__ __forceinline__ void f2_bits(uint64_t v, uint32_t& lo, uint32_t& hi) { asm("mov.b64 {%0, %1}, %2;" : "=r"(lo), "=r"(hi) : "l"(v)); }
__device__ __forceinline__ void f2_unpack(uint64_t v, float& lo, float& hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v)); }
__device__ __forceinline__ uint64_t f2_mul(uint64_t a, uint64_t b) {
    uint64_t d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ uint64_t f2_fma(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}

// the value a kernel storing `v` in the activation type would have left in memory
__device__ __forceinline__ float round_to(float v, int dt) {
    if (dt == BI8_BF16) return __bfloat162float(__float2bfloat16_rn(v));
    if (dt == BI8_F16) return __half2float(__float2half_rn(v));
    return v;
}

// silu(g) as the separate kernel stores it: one fp32 exponential, an IEEE division, one rounding to the activation type.
__device__ __forceinline__ float silu_exact(float g, int dt) { return round_to(__fdiv_rn(g, __fadd_rn(1.0f, expf(-g))), dt); }

// two values rounded to a 16-bit activation type and packed; and back
__device__ __forceinline__ uint32_t pack16(float lo, float hi, bool bf) { return bf ? pack_bf16x2(lo, hi) : pack_f16x2(lo, hi); }
__device__ __forceinline__ float2 unpack16(uint32_t w, bool bf) {
    return bf ? make_float2(bf16lo(w), bf16hi(w)) : __half22float2(*reinterpret_cast<const __half2*>(&w));
}

// g = cast(cast(silu(g)) * v), the gated activation as its two separate kernels would leave it, bit for bit.
//
// What is stored of silu(g) is its 16-bit rounding, so an approximate value decides it unless it lies next to a rounding
// boundary: s = g * rcp(1 + ex2(-g log2 e)) with the hardware's approximations (2^-22 and 2^-23 relative) is within
// eps = (|t| + 16) * 1.25 * 2^-24 of silu_exact's fp32 value before rounding, t = g log2 e (the rounding of t costs |t| 2^-24, the exponential
// 4 units of 2^-24, the reciprocal 2, the sum and the product 1 each, and silu_exact's own error is at most 4), and where s (1 - eps) and
// s (1 + eps) round to the same value, that is the value.  Elsewhere (1 in 1400 values of bf16, 1 in 180 of fp16) and for
// |g| > 60 (in any of the eight) silu_exact is evaluated.  65 instructions per value became 20; the products and sums run on packed
// pairs, each rounded on its own (4096 x 11008: 62.3 -> 60.4 us).
__device__ __forceinline__ void silu_mul8(float (&g)[8], const float (&v)[8], int dt) {
    if (dt == BI8_F32) {
#pragma unroll
        for (int e = 0; e < 8; ++e) g[e] = __fmul_rn(silu_exact(g[e], dt), v[e]);
        return;
    }
    const bool bf = dt == BI8_BF16;
    float most = 0.0f;
#pragma unroll
    for (int e = 0; e < 8; ++e) most = fmaxf(most, fabsf(g[e]));
    const bool far = !(most <= 60.0f);
    const uint64_t log2e = f2_pack(-1.4426950408889634f, -1.4426950408889634f), one = f2_pack(1.0f, 1.0f);
#pragma unroll
    for (int h = 0; h < 4; ++h) {
        const uint64_t x = f2_pack(g[2 * h], g[2 * h + 1]);
        float t[2], ex[2], sum[2], r[2], eps[2], lo[2], hi[2], y[2];
        f2_unpack(f2_mul(x, log2e), t[0], t[1]);
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(ex[u]) : "f"(t[u]));
            eps[u] = __fmaf_rn(fabsf(t[u]), 1.25f * 5.9604644775390625e-8f, 20.0f * 5.9604644775390625e-8f);
        }
        f2_unpack(f2_fma(f2_pack(ex[0], ex[1]), one, one), sum[0], sum[1]);
#pragma unroll
        for (int u = 0; u < 2; ++u) asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r[u]) : "f"(sum[u]));
        const uint64_t s = f2_mul(x, f2_pack(r[0], r[1]));
        f2_unpack(f2_fma(s, f2_pack(eps[0], eps[1]), s), hi[0], hi[1]);
        f2_unpack(f2_fma(s, f2_pack(-eps[0], -eps[1]), s), lo[0], lo[1]);
        uint32_t w = pack16(lo[0], lo[1], bf);
        if (far || w != pack16(hi[0], hi[1], bf)) w = pack16(silu_exact(g[2 * h], dt), silu_exact(g[2 * h + 1], dt), bf);
        const float2 silu = unpack16(w, bf);
        f2_unpack(f2_mul(f2_pack(silu.x, silu.y), f2_pack(v[2 * h], v[2 * h + 1])), y[0], y[1]);
        const float2 z = unpack16(pack16(y[0], y[1], bf), bf);
        g[2 * h] = z.x;
        g[2 * h + 1] = z.y;
    }
}

// Quantizes eight values of one block (scale amax) on packed pairs: the same operations, each rounded on its own, as BlockQ::q.
// Returns the bytes of values 0-3 and 4-7.
__device__ __forceinline__ void quantize8(const float (&v)[8], const BlockQ& bq, uint32_t& lo, uint32_t& hi) {
    uint32_t b[8];
    if (bq.fast) {
        const uint64_t r2 = f2_pack(bq.rcp, bq.rcp), ns2 = f2_pack(-bq.scale, -bq.scale);
        const uint64_t c127 = f2_pack(127.0f, 127.0f), cmagic = f2_pack(kMagic, kMagic), cone = f2_pack(1.0f, 1.0f);
#pragma unroll
        for (int h = 0; h < 4; ++h) {
            const uint64_t v2 = f2_pack(v[2 * h], v[2 * h + 1]);
            const uint64_t q0 = f2_mul(v2, r2);
            const uint64_t e = f2_fma(ns2, q0, v2);
            const uint64_t y = f2_fma(e, r2, q0);
            f2_bits(f2_fma(f2_mul(c127, y), cone, cmagic), b[2 * h], b[2 * h + 1]);
        }
    } else {
#pragma unroll
        for (int e = 0; e < 8; ++e) b[e] = bq.q(v[e]);
    }
    lo = pack4(b[0], b[1], b[2], b[3]);
    hi = pack4(b[4], b[5], b[6], b[7]);
}

}  // namespace bi8
