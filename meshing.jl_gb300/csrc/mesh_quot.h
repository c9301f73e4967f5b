// Correctly rounded Float64 quotients whose divisor has at most 32 significant
// bits, on the integer pipes.
//
// (iso - v1) / (v2 - v1) is a Float64 division whenever iso is a Float64 (the
// default) or an Int on integer samples, but v2 - v1 is a Float32, a Float16 or a
// small integer.  GB300 executes two Float64 operations per SM and cycle, and a
// division takes several; 32-bit integer operations run 64 times as fast.  The
// dividend's 64-bit significand is divided by the divisor's normalised 32 bits in
// two steps of 64 by 32 bits with a precomputed reciprocal (Moeller and Granlund,
// "Improved division by invariant integers", IEEE Trans. Comput. 60(2), 2011,
// algorithm 4), which leaves 63 or 64 quotient bits and the remainder: the
// rounding to 53 bits is then exact.  The reciprocal comes from a Float32 estimate
// and one exact correction.
//
// Zeros, subnormals, Inf, NaN and results outside the normal range are left to the
// caller (quot_narrow returns false).
#pragma once
#include <stdint.h>
#include <string.h>

#ifdef __CUDACC__
#define MESH_QUOT static __device__ __forceinline__
#else
#define MESH_QUOT static inline
#endif

namespace mesh {

MESH_QUOT float quot_seed(float x) {  // about 1 / x, x in [1, 2)
#ifdef __CUDACC__
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
#else
    return MESH_QUOT_SEED(x);
#endif
}
MESH_QUOT float quot_float(uint32_t u) {
    float f;
    memcpy(&f, &u, 4);
    return f;
}

// v with 2^64 - d (2^32 + v) in [1, d], for d with its top bit set.
MESH_QUOT uint32_t quot_reciprocal(uint32_t d) {
    const float r = quot_seed(quot_float((d >> 8 & 0x7fffffu) | 0x3f800000u));  // of d / 2^31, within 2^-21
    const float t = (r + r - 1.0f) * 4294967296.0f;
    uint32_t v = t >= 4294967040.0f ? 0xffffff00u : t <= 0.0f ? 0u : (uint32_t)t;
    int64_t e = (int64_t)(0ull - (uint64_t)d * v - ((uint64_t)d << 32));  // |e| < 2^45
    // e / d, within 1: e in units of 2^22 and r give it to 2^-9 and a rounding
    const int c = (int)((float)(int32_t)(e >> 22) * r * (1.0f / 512.0f));
    v += (uint32_t)c;
    e -= (int64_t)c * (int64_t)d;
    if (e <= 0) {
        v -= 1;
        e += d;
    }
    if (e > (int64_t)d) {
        v += 1;
        e -= d;
    }
    if (e > (int64_t)d) v += 1;
    return v;
}

// (u1 2^32 + u0) / d for u1 < d; u1 becomes the remainder.
MESH_QUOT uint32_t quot_step(uint32_t &u1, uint32_t u0, uint32_t d, uint32_t v) {
    const uint64_t q = (uint64_t)v * u1 + (((uint64_t)u1 << 32) | u0);
    uint32_t q1 = (uint32_t)(q >> 32) + 1u;
    uint32_t r = u0 - q1 * d;
    if (r > (uint32_t)q) {
        q1 -= 1;
        r += d;
    }
    if (r >= d) {
        q1 += 1;
        r -= d;
    }
    u1 = r;
    return q1;
}

// RN((-1)^neg n 2^ne / (d 2^de)) for n and d with their top bits set.
MESH_QUOT bool quot_bits(uint32_t neg, uint64_t n, int ne, uint32_t d, int de, uint64_t &out) {
    const uint32_t v = quot_reciprocal(d);
    uint32_t r = (uint32_t)(n >> 33);  // n / 2, so that the first digit fits
    // (n has at least one zero low bit: its significand is 53 bits long at most)
    const uint32_t q1 = quot_step(r, (uint32_t)(n >> 1), d, v);
    const uint32_t q0 = quot_step(r, 0u, d, v);
    uint64_t q = ((uint64_t)q1 << 32) | q0;  // n / 2 * 2^32 / d, at least 2^62
    int x = ne - de - 31;                    // the quotient is q 2^x and the remainder
    if (!(q >> 63)) {
        q <<= 1;
        x -= 1;
    }
    const uint32_t low = (uint32_t)q & 0x7ffu;
    uint64_t m = q >> 11;
    // ties are exact only with a zero remainder
    m += low > 0x400u || (low == 0x400u && (r != 0u || (m & 1u)));
    const int b = x + 1086;  // biased exponent of 2^52 <= m < 2^53
    if (b < 1 || b > 2045) return false;
    out = ((uint64_t)neg << 63) + ((uint64_t)(b - 1) << 52) + m;
    return true;
}

// a / f for a normal Float64 (bits a) and a normal Float32 (bits f).
MESH_QUOT bool quot_f64_f32(uint64_t a, uint32_t f, uint64_t &out) {
    const uint32_t ea = (uint32_t)(a >> 52) & 0x7ffu, ef = (f >> 23) & 0xffu;
    if (ea - 1u >= 2046u || ef - 1u >= 254u) return false;
    return quot_bits((uint32_t)(a >> 63) ^ (f >> 31), (a << 11) | (1ull << 63), (int)ea - 1086, (f << 8) | 0x80000000u,
                     (int)ef - 158, out);
}
// a / f for two normal Float32.
MESH_QUOT bool quot_f32_f32(uint32_t a, uint32_t f, uint64_t &out) {
    const uint32_t ea = (a >> 23) & 0xffu, ef = (f >> 23) & 0xffu;
    if (ea - 1u >= 254u || ef - 1u >= 254u) return false;
    return quot_bits((a >> 31) ^ (f >> 31), (uint64_t)((a << 8) | 0x80000000u) << 32, (int)ea - 190,
                     (f << 8) | 0x80000000u, (int)ef - 158, out);
}
// a / d for integers, both nonzero.
MESH_QUOT bool quot_i32_i32(int32_t a, int32_t d, uint64_t &out) {
    if (a == 0 || d == 0) return false;
    const uint32_t ua = a < 0 ? 0u - (uint32_t)a : (uint32_t)a, ud = d < 0 ? 0u - (uint32_t)d : (uint32_t)d;
#ifdef __CUDACC__
    const int sa = __clz((int)ua), sd = __clz((int)ud);
#else
    const int sa = __builtin_clz(ua), sd = __builtin_clz(ud);
#endif
    return quot_bits(((uint32_t)a ^ (uint32_t)d) >> 31, (uint64_t)(ua << sa) << 32, -32 - sa, ud << sd, -sd, out);
}
// a / d for a normal Float64 (bits a) and a nonzero integer.
MESH_QUOT bool quot_f64_i32(uint64_t a, int32_t d, uint64_t &out) {
    const uint32_t ea = (uint32_t)(a >> 52) & 0x7ffu;
    if (ea - 1u >= 2046u || d == 0) return false;
    const uint32_t ud = d < 0 ? 0u - (uint32_t)d : (uint32_t)d;
#ifdef __CUDACC__
    const int sd = __clz((int)ud);
#else
    const int sd = __builtin_clz(ud);
#endif
    return quot_bits((uint32_t)(a >> 63) ^ ((uint32_t)d >> 31), (a << 11) | (1ull << 63), (int)ea - 1086, ud << sd, -sd,
                     out);
}

}  // namespace mesh
