// exact_round.cuh -- quotients and square roots rounded to nearest from an
// estimate and its exact integer remainder (the ray tracer's plain path).
#pragma once

namespace fair {

// Rare operations are calls: inlined they would be predicated, and an FP64
// instruction holds its pipe for 64 cycles whether or not a lane executes it.
static __device__ __noinline__ double div_slow(double n, double a) { return __ddiv_rn(n, a); }
static __device__ __noinline__ double sqrt_slow(double v) { return __dsqrt_rn(v); }

// n / a rounded to nearest, y = 1/a rounded to nearest. q = n y is within 1.5
// units in the last place (half a unit from the product, up to one from y);
// the remainder n - a q in units of ulp(a) ulp(q) is below 2^55, so its low 64
// bits give it exactly, and the quotient is the neighbour that leaves at most
// |a|/2 (no quotient of two doubles lies half way between doubles). Zero, a
// result at a power of two from below and exponents off the usual two go to
// the division itself.
__device__ __forceinline__ double div_by(double n, double a, double y) {
    const unsigned long long M52 = 1ull << 52, mask = M52 - 1;
    const double q = __dmul_rn(n, y);
    const unsigned long long nb = __double_as_longlong(n), ab = __double_as_longlong(a),
                             qb = __double_as_longlong(q);
    const unsigned long long mn = (nb & mask) | M52, ma = (ab & mask) | M52, mq = (qb & mask) | M52;
    const int en = (int)(nb >> 52) & 0x7ff, ea = (int)(ab >> 52) & 0x7ff, eq = (int)(qb >> 52) & 0x7ff;
    const int sh = en - ea - eq + 1075;
    const long long R = (long long)((mn << (sh & 63)) - ma * mq);
    const long long R2 = 2 * R, A = (long long)ma;
    if ((unsigned)(sh - 51) > 3u || eq == 0 || (mq == M52 && R < 0)) return div_slow(n, a);
    const int k = (R2 > A ? 1 : 0) - (R2 < -A ? 1 : 0);
    return __longlong_as_double((long long)qb + k);
}

// sqrt(v) rounded to nearest, s0 close to it (the difference of the ray
// parameters): one Newton step with a 22-bit 1/(2 s0), then the neighbour whose
// exact integer remainder v - s^2 lies in (-s, s] (units of ulp(s)^2). Where the
// step leaves s further off than one unit (|v - s^2| > 2 s: its neighbour need
// not be the nearest then, above all next to a power of two, below which the
// units are half as large), and on short segments, the root itself.
__device__ __forceinline__ double sqrt_near(double v, double s0) {
    const unsigned long long M52 = 1ull << 52, mask = M52 - 1;
    const double e = fma(-s0, s0, v);
    const unsigned long long sb0 = __double_as_longlong(s0);
    // s0 as a float (truncated) and its reciprocal back as a double, by the bits
    const unsigned fb = (unsigned)((sb0 >> 29) - (896ull << 23));
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(__uint_as_float(fb)));
    const double h = __longlong_as_double((long long)(((unsigned long long)__float_as_uint(r) << 29) +
                                                      ((896ull - 1) << 52)));  // r / 2
    const double s = fma(e, h, s0);
    const unsigned long long vb = __double_as_longlong(v), sb = __double_as_longlong(s);
    const unsigned long long mv = (vb & mask) | M52, ms = (sb & mask) | M52;
    const int ev = (int)(vb >> 52), es = (int)(sb >> 52);
    const int sh = ev - 2 * es + 1075;  // v in units of ulp(s)^2
    const long long R = (long long)((mv << (sh & 63)) - ms * ms), S = (long long)ms;
    if ((int)(sb0 >> 52) < 1023 - 12 || (unsigned)(sh - 50) > 5u || R > 2 * S || R < -2 * S || (ms == M52 && R < 0))
        return sqrt_slow(v);
    const int k = (R > S ? 1 : 0) - (R <= -S ? 1 : 0);
    return __longlong_as_double((long long)sb + k);
}

}  // namespace fair
