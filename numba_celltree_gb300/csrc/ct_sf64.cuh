// ct_sf64.cuh -- float64 products and quotients on the integer pipes.
//
// The GPU's float64 unit takes 20 cycles per warp addition or multiplication
// and SM and 144 per division (2.07 GHz; measured on chains of independent
// operations), 40 times as long as the float32 unit.  Kernels whose float64
// results are fixed bit for bit and whose time is that unit's compute their
// quotients, and as many products as the integer pipes have room for, here
// and leave it the rest, so that both kinds of unit work at once.  Measured
// the same way: sf_mul 16.6 cycles (20.4 for a product and an addition side
// by side, against 40 on the float64 unit alone), sf_div 25.
//
// Both return the IEEE 754 binary64 result rounded to nearest even, the bits
// of `a * b` and `a / b`: the significands are multiplied (divided) exactly
// as integers and rounded once.  Zero operands (a zero numerator) are
// handled; other operands or results outside the normal range (subnormals,
// infinities, NaN, a zero divisor, overflow, underflow) set `bad`, and the
// caller repeats the computation with the hardware's operators.  Neither
// branches, so independent operations interleave.
#pragma once

#include <cstdint>
#include <cstring>

#ifdef __CUDACC__
#define SF_FN __host__ __device__ __forceinline__
#else
#define SF_FN static inline
#endif

SF_FN uint64_t sf_bits(double x) {
#ifdef __CUDA_ARCH__
    uint64_t b;  // opaque: the compiler turns tests on reinterpreted bits into float64 comparisons
    asm("mov.b64 %0, %1;" : "=l"(b) : "d"(x));
    return b;
#else
    uint64_t b;
    memcpy(&b, &x, 8);
    return b;
#endif
}
SF_FN double sf_value(uint64_t b) {
#ifdef __CUDA_ARCH__
    return __longlong_as_double((long long)b);
#else
    double x;
    memcpy(&x, &b, 8);
    return x;
#endif
}
SF_FN uint32_t sf_shr64(uint32_t lo, uint32_t hi, uint32_t s) {  // low word of (hi:lo) >> s, 0 < s < 32
#ifdef __CUDA_ARCH__
    return __funnelshift_r(lo, hi, s);
#else
    return (lo >> s) | (hi << (32 - s));
#endif
}
SF_FN uint32_t sf_umulhi(uint32_t a, uint32_t b) { return (uint32_t)(((uint64_t)a * b) >> 32); }
SF_FN bool sf_zero(double x) { return (sf_bits(x) << 1) == 0u; }

// Rounds the significand at bit `s` (1 <= s <= 31) of (h:l) to nearest even,
// `sticky` for set bits below l, and adds it to sign and exponent `head`
// (exponent one less: the significand's leading bit adds the one).
SF_FN double sf_round(uint32_t h, uint32_t l, uint32_t s, uint32_t sticky, uint32_t head) {
    const uint32_t ml = sf_shr64(l, h, s), mh = h >> s;
    const uint32_t rest = (l << (32 - s)) | sticky;
    const uint32_t up = (rest + (ml & 1u)) > 0x80000000u ? 1u : 0u;
    return sf_value((((uint64_t)head << 32) | 0u) + (((uint64_t)mh << 32) | ml) + up);
}

// a * b
SF_FN double sf_mul(double a, double b, bool* bad) {
    const uint64_t x = sf_bits(a), y = sf_bits(b);
    const uint32_t xh = (uint32_t)(x >> 32), yh = (uint32_t)(y >> 32);
    const uint32_t ex = (xh >> 20) & 0x7ffu, ey = (yh >> 20) & 0x7ffu;
    const uint32_t e = ex + ey - 1023u;  // of a product of significands in [1, 2)
    const bool zero = sf_zero(a) || sf_zero(b);
    const uint32_t px = ex - 1u, py = ey - 1u, pe = e + 1u;  // pe < 2: underflow
    const bool in = (px > py ? px : py) < 2046u && pe - 2u < 2043u;
    *bad = *bad || (!in && !(zero && (ex > ey ? ex : ey) < 2047u));
    // significands with their top bit at bit 63; product in [2^126, 2^128)
    const uint64_t A = (x << 11) | 0x8000000000000000ull, B = (y << 11) | 0x8000000000000000ull;
#ifdef __CUDA_ARCH__
    const uint64_t h = __umul64hi(A, B), l = A * B;
#else
    const unsigned __int128 P = (unsigned __int128)A * B;
    const uint64_t h = (uint64_t)(P >> 64), l = (uint64_t)P;
#endif
    const uint32_t up = (uint32_t)(h >> 63);
    const uint32_t sign = (xh ^ yh) & 0x80000000u;
    const double r = sf_round((uint32_t)(h >> 32), (uint32_t)h, 10u + up, l != 0u ? 1u : 0u,
                              sign | ((e + up - 1u) << 20));
    return zero ? sf_value((uint64_t)sign << 32) : r;
}

// a / b.  The quotient of the significands is found as floor(ma 2^54 / mb) in
// two digits of 27 bits with a reciprocal that is never too large and at most
// 2^-30 too small: 23 bits of the float32 reciprocal and one Newton step in
// integers (R0 (1 + e) <= R0 / (1 - e) for the residual e of R0).  Each digit
// is then the true one or one less (errors: 2^28 (2^-30 + 2^-31) + 1 < 2 for
// the first, 2^27.5 2^-30 + 2^-3 + 1 < 2 for the second), so the remainder
// stays within [0, 2 mb) and one conditional subtraction makes it exact.
SF_FN double sf_div(double a, double b, bool* bad) {
    const uint64_t x = sf_bits(a), y = sf_bits(b);
    const uint32_t xh = (uint32_t)(x >> 32), yh = (uint32_t)(y >> 32);
    const uint32_t ex = (xh >> 20) & 0x7ffu, ey = (yh >> 20) & 0x7ffu;
    const uint32_t e = ex - ey + 1023u;  // of a quotient in [1, 2); one less below 1
    const bool zero = sf_zero(a);
    const uint32_t px = ex - 1u, py = ey - 1u;
    const bool in = (px > py ? px : py) < 2046u && e - 2u < 2044u;
    *bad = *bad || (!in && !(zero && py < 2046u));
    const uint32_t mah = (xh & 0xfffffu) | 0x100000u, mbh = (yh & 0xfffffu) | 0x100000u;
    const uint64_t ma = ((uint64_t)mah << 32) | (uint32_t)x, mb = ((uint64_t)mbh << 32) | (uint32_t)y;
    const uint32_t bh = sf_shr64((uint32_t)y, mbh, 21);  // b 2^31, truncated, b in [1, 2)
    // R0 = 2^32 / b to 23 bits: the reciprocal of b rounded up to 24 bits,
    // which lies in [1/2, 1)
    const uint32_t fb = 0x3f800001u + ((bh >> 8) & 0x7fffffu);
#ifdef __CUDA_ARCH__
    float rf;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(rf) : "f"(__uint_as_float(fb)));
    uint32_t rb = __float_as_uint(rf);
#else
    float ff;
    memcpy(&ff, &fb, 4);
    const float rf = 1.0f / ff;
    uint32_t rb;
    memcpy(&rb, &rf, 4);
#ifdef SF_TEST_RCP
    rb += SF_TEST_RCP;
#endif
#endif
    rb = rb > 0x3f7fffffu ? 0x3f7fffffu : rb < 0x3f000000u ? 0x3f000000u : rb;
    const uint32_t R0 = (rb << 8) | 0x80000000u;
    const int32_t res = (int32_t)((0x8000000000000000ull - ((uint64_t)R0 * bh + R0)) >> 20);
    const uint32_t R = R0 + (uint32_t)(int32_t)(((int64_t)res * (int64_t)R0) >> 43);
    const uint32_t q1 = sf_umulhi(sf_shr64((uint32_t)x, mah, 21), R) >> 4;
    const uint64_t r1 = (ma << 27) - (uint64_t)q1 * mb;
    const uint32_t q2 = sf_umulhi((uint32_t)(r1 >> 22), R) >> 3;
    uint64_t r2 = (r1 << 27) - (uint64_t)q2 * mb;
    const bool more = r2 >= mb;
    const uint64_t q = (((uint64_t)q1 << 27) + q2) + (more ? 1u : 0u);
    r2 -= more ? mb : 0u;
    // q in (2^53, 2^55)
    const uint32_t up = (uint32_t)(q >> 54);
    const uint32_t sign = (xh ^ yh) & 0x80000000u;
    const double r = sf_round((uint32_t)(q >> 32), (uint32_t)q, 1u + up, r2 != 0u ? 1u : 0u,
                              sign | ((e + up - 2u) << 20));
    return zero ? sf_value((uint64_t)sign << 32) : r;
}
