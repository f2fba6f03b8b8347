// IEEE-754 binary64 arithmetic, round to nearest even, computed on the integer and FP32 pipes.
//
// GB300 issues FP64 at 2 lanes per clock per SM (a warp instruction every 16 SM cycles), and a
// double division or square root is a sequence of about eight FP64 instructions.  The functions
// here return the same bits as the hardware's correctly rounded operations (they are the IEEE
// operations, computed another way) from 64-bit integer arithmetic, so a kernel bound by FP64 issue
// can move part of its work off the FP64 pipe without changing any result.
//
// Each function handles the common case -- normal finite operands and a normal result -- itself and
// passes everything else (zeros, subnormals, infinities, NaNs, results that overflow or underflow)
// to the hardware operation, so every input gets the IEEE result.
//
// Methods:
//   mul   the 106-bit product of the significands from four 32x32 -> 64-bit multiply-adds (the high
//         words hold 21 bits, so the partial sums never carry out of 64), rounded.
//   add   significands aligned with 10 guard bits and a sticky bit, added or subtracted,
//         renormalised (count of leading zeros), rounded.
//   div   reciprocal of the divisor: the approximate FP32 reciprocal, refined in FP32 on a two-term
//         divisor (~42 bits), then one Newton-Raphson step r <- r + r (1 - y r) in fixed point, whose
//         residual fits one word; the quotient from the reciprocal, its last bit from the exact
//         integer remainder.  The reciprocal (a Divisor) serves any number of dividends.
//   sqrt  reciprocal square root: the approximate FP32 one, refined in FP32 on a two-term argument
//         (~43 bits); the root from it with one Newton-Raphson step on the root's own residual, its last
//         bit from the exact integer remainder.  The same reciprocal root, refined against the
//         rounded root, is that root's reciprocal: dividing by a square root (sqrt_divisor) costs no
//         second reciprocal.
//   widen / narrow  float <-> double by moving the fields (narrow: round to nearest even on the
//         29 dropped bits).
// Floats enter the integers through their bit fields and through 32-bit conversions only: conversions
// with a 64-bit operand issue on the FP64 pipe, at its rate.
// Measured against the former sequences (64-bit conversions for the seeds, two Newton-Raphson steps, up
// to three corrections) at 100k cells: FP64 force kernel 0.435 -> 0.410 ms, corner phase 0.148 -> 0.133
// ms, cells 34 -> 31 us; one 396-vertex force launch 45 -> 40 us.
// (Newton-Raphson refinement of reciprocals and the final correction by an exact remainder are the
// classical methods of P. Markstein, "IA-64 and Elementary Functions", 2000, and of integer
// division by invariant integers, T. Granlund and P. Montgomery, PLDI 1994.)
#pragma once
#include <cstdint>

#if defined(__CUDACC__)
#define SF_HD __host__ __device__ __forceinline__
// the fallbacks of operands outside the fast paths stay out of line (code size)
#define SF_SLOW static __host__ __device__ __noinline__
#else
#define SF_HD inline
#define SF_SLOW inline
#endif

namespace sf {

constexpr unsigned long long kMant = 0xFFFFFFFFFFFFFull, kHid = 0x10000000000000ull, kSign = 0x8000000000000000ull;

SF_HD unsigned long long bits(double x) {
#if defined(__CUDA_ARCH__)
    return (unsigned long long)__double_as_longlong(x);
#else
    unsigned long long u;
    __builtin_memcpy(&u, &x, 8);
    return u;
#endif
}
SF_HD double dbl(unsigned long long u) {
#if defined(__CUDA_ARCH__)
    return __longlong_as_double((long long)u);
#else
    double x;
    __builtin_memcpy(&x, &u, 8);
    return x;
#endif
}
SF_HD int clz64(unsigned long long x) {
#if defined(__CUDA_ARCH__)
    return __clzll((long long)x);
#else
    return __builtin_clzll(x);
#endif
}
// FP32 seeds: the approximate reciprocal (1 ulp) and reciprocal square root (2 ulp) instructions.  Any
// seed within 4 ulp gives the same results; the host build's are moved by SF_HOST_SEED_ULPS (0 unless a test
// sets it, to -4 or 4) to check that.
#ifndef SF_HOST_SEED_ULPS
#define SF_HOST_SEED_ULPS 0
#endif
SF_HD float ulps_off(float x, int n) {
    unsigned u;
    __builtin_memcpy(&u, &x, 4);
    u += (unsigned)n;
    __builtin_memcpy(&x, &u, 4);
    return x;
}
SF_HD float rcp32(float x) {
#if defined(__CUDA_ARCH__)
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
#else
    return ulps_off(1.0f / x, SF_HOST_SEED_ULPS);
#endif
}
SF_HD float rsqrt32(float x) {
#if defined(__CUDA_ARCH__)
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
#else
    return ulps_off(1.0f / __builtin_sqrtf(x), SF_HOST_SEED_ULPS);
#endif
}
SF_HD float f32_of(unsigned u) {
#if defined(__CUDA_ARCH__)
    return __uint_as_float(u);
#else
    float x;
    __builtin_memcpy(&x, &u, 4);
    return x;
#endif
}
SF_HD unsigned u32_of(float x) {
#if defined(__CUDA_ARCH__)
    return __float_as_uint(x);
#else
    unsigned u;
    __builtin_memcpy(&u, &x, 4);
    return u;
#endif
}
SF_HD int round32(float x) {  // to the nearest int (ties even on the device; either tie serves)
#if defined(__CUDA_ARCH__)
    return __float2int_rn(x);
#else
    return (int)__builtin_rintf(x);
#endif
}
SF_HD float clamp32(float x, float lo, float hi) {
#if defined(__CUDA_ARCH__)
    return fminf(fmaxf(x, lo), hi);
#else
    return x < lo ? lo : (x > hi ? hi : x);
#endif
}
// a b and a b + c of unsigned words in 64 bits; the left funnel shift's high word (0 < n < 32)
SF_HD unsigned long long wide(unsigned a, unsigned b) { return (unsigned long long)a * b; }
SF_HD unsigned long long wide_add(unsigned a, unsigned b, unsigned long long c) { return (unsigned long long)a * b + c; }
SF_HD unsigned shl2(unsigned hi, unsigned lo, unsigned n) {
#if defined(__CUDA_ARCH__)
    return __funnelshift_l(lo, hi, n);
#else
    return (hi << n) | (lo >> (32 - n));
#endif
}
SF_HD unsigned hi32(unsigned long long x) { return (unsigned)(x >> 32); }
SF_HD unsigned lo32(unsigned long long x) { return (unsigned)x; }
// a b / 2^64 without the low words' product and carries: 0 to 3 below the exact high word
SF_HD unsigned long long mulhi_near(unsigned long long a, unsigned long long b) {
    const unsigned long long x = wide(hi32(a), lo32(b)), y = wide(lo32(a), hi32(b));
    return wide_add(hi32(a), hi32(b), (unsigned long long)hi32(x) + hi32(y));
}
SF_HD float fma32(float a, float b, float c) {
#if defined(__CUDA_ARCH__)
    return __fmaf_rn(a, b, c);
#else
    return __builtin_fmaf(a, b, c);
#endif
}
// The hardware operations (the fallback for operands and results outside the fast paths).
SF_SLOW double hw_mul(double a, double b) {
#if defined(__CUDA_ARCH__)
    return __dmul_rn(a, b);
#else
    volatile double r = a * b;
    return r;
#endif
}
SF_SLOW double hw_add(double a, double b) {
#if defined(__CUDA_ARCH__)
    return __dadd_rn(a, b);
#else
    volatile double r = a + b;
    return r;
#endif
}
SF_SLOW double hw_div(double a, double b) {
#if defined(__CUDA_ARCH__)
    return __ddiv_rn(a, b);
#else
    volatile double r = a / b;
    return r;
#endif
}
SF_SLOW double hw_sqrt(double a) {
#if defined(__CUDA_ARCH__)
    return __dsqrt_rn(a);
#else
    volatile double r = __builtin_sqrt(a);
    return r;
#endif
}

// Rounds the significand m (hidden bit at 52) with the rest `rest` (2^63 = one half of the last
// place) to nearest even and packs it with the biased exponent E (the carry of a round-up into
// bit 53 increments the exponent, up to infinity) and the sign.
SF_HD double pack(unsigned long long sign, int E, unsigned long long m, unsigned long long rest) {
    const unsigned long long up = (rest > kSign) | ((rest == kSign) & (m & 1ull));
    return dbl(sign | ((((unsigned long long)(E - 1)) << 52) + m + up));
}

SF_HD double mul(double a, double b) {
    const unsigned long long ia = bits(a), ib = bits(b);
    const unsigned ha = hi32(ia), hb = hi32(ib);
    const unsigned ea = (ha >> 20) & 0x7ffu, eb = (hb >> 20) & 0x7ffu;
    const int E = (int)ea + (int)eb - 1023;
    if (ea - 1u < 2046u && eb - 1u < 2046u && (unsigned)(E - 1) < 2045u) {
        const unsigned ah = (ha & 0xfffffu) | 0x100000u, bh = (hb & 0xfffffu) | 0x100000u;
        const unsigned al = lo32(ia), bl = lo32(ib);
        const unsigned long long p0 = wide(al, bl);
        const unsigned long long p1 = wide_add(al, bh, wide_add(ah, bl, p0 >> 32));  // < 2^55
        const unsigned long long p2 = wide_add(ah, bh, p1 >> 32);   // product in [2^104, 2^106): below 2^42
        const unsigned n = hi32(p2) >> 9;                           // 1: product >= 2^105
        const unsigned sh = 12u - n;
        const unsigned mh = shl2(hi32(p2), lo32(p2), sh), ml = shl2(lo32(p2), lo32(p1), sh);
        unsigned g = shl2(lo32(p1), lo32(p0), sh);                  // the dropped bits: 2^31 = half
        g |= (lo32(p0) << sh) != 0u ? 1u : 0u;
        // to nearest even: up when g > half, or g == half and the last bit is odd
        const unsigned up = hi32((unsigned long long)g + 0x7fffffffu + (ml & 1u));
        const unsigned top = ((ha ^ hb) & 0x80000000u) + ((unsigned)(E + (int)n - 1) << 20) + mh;
        return dbl((((unsigned long long)top << 32) | ml) + up);
    }
    return hw_mul(a, b);
}

// x x
SF_HD double sqr(double x) {
    const unsigned long long ix = bits(x);
    const unsigned hx = hi32(ix), ex = (hx >> 20) & 0x7ffu;
    if (ex - 512u < 1023u) {   // 2 ex - 1023 in [1, 2045]
        const unsigned xh = (hx & 0xfffffu) | 0x100000u, xl = lo32(ix);
        const unsigned long long p0 = wide(xl, xl), c = wide(xh, xl);       // c < 2^53
        const unsigned long long p1 = 2ull * c + (p0 >> 32);                // < 2^55
        const unsigned long long p2 = wide_add(xh, xh, p1 >> 32);           // product in [2^104, 2^106)
        const unsigned n = hi32(p2) >> 9, sh = 12u - n;
        const unsigned mh = shl2(hi32(p2), lo32(p2), sh), ml = shl2(lo32(p2), lo32(p1), sh);
        unsigned g = shl2(lo32(p1), lo32(p0), sh);
        g |= (lo32(p0) << sh) != 0u ? 1u : 0u;
        const unsigned up = hi32((unsigned long long)g + 0x7fffffffu + (ml & 1u));
        const unsigned top = ((2u * ex - 1023u + n - 1u) << 20) + mh;
        return dbl((((unsigned long long)top << 32) | ml) + up);
    }
    return hw_mul(x, x);
}
// mul out of line, for kernels with dozens of products, whose code would not fit the instruction caches.
SF_SLOW double mul_call(double a, double b) { return mul(a, b); }

// -x and, if c, -x: a bit flip (the hardware's negation, where it is not an operand's modifier, is an
// addition).
SF_HD double negate_if(bool c, double x) {
#if defined(__CUDA_ARCH__)
    return __hiloint2double(__double2hiint(x) ^ (c ? (int)0x80000000u : 0), __double2loint(x));
#else
    return c ? -x : x;
#endif
}

// 2 x (exact; zeros, subnormals, the largest binade, infinities and NaN take the hardware)
SF_HD double twice(double x) {
    const unsigned long long u = bits(x);
    if (((unsigned)(u >> 52) & 0x7ffu) - 1u < 2045u) return dbl(u + (1ull << 52));
    return hw_add(x, x);
}

SF_HD double add(double a, double b) {
    unsigned long long ia = bits(a), ib = bits(b);
    unsigned long long aa = ia & ~kSign, ab = ib & ~kSign;
    if (aa < ab) {
        unsigned long long t = ia; ia = ib; ib = t;
        t = aa; aa = ab; ab = t;
    }
    const unsigned ea = (unsigned)(aa >> 52), eb = (unsigned)(ab >> 52);
    if (ea - 1u < 2046u && eb - 1u < 2046u) {
        const unsigned d = ea - eb;
        const unsigned long long A = ((aa & kMant) | kHid) << 10;
        unsigned long long B = ((ab & kMant) | kHid) << 10;
        if (d) B = d < 64 ? ((B >> d) | (unsigned long long)((B << (64 - d)) != 0)) : 1ull;
        int E = (int)ea;
        unsigned long long S;
        if (!((ia ^ ib) >> 63)) {
            S = A + B;
            if (S >> 63) { S = (S >> 1) | (S & 1ull); E += 1; }
        } else {
            S = A - B;
            if (S == 0) return 0.0;
            const int lz = clz64(S) - 1;
            S <<= lz;
            E -= lz;
        }
        if ((unsigned)(E - 1) < 2046u) return pack(ia & kSign, E, S >> 10, S << 54);
    }
    return hw_add(a, b);
}

SF_HD double sub(double a, double b) { return add(a, dbl(bits(b) ^ kSign)); }

// A divisor with the reciprocal of its significand: R ~ 2^63 / y, y = the significand in [1, 2).
// R = 0 marks a divisor outside the fast path (zero, subnormal, infinite, NaN).
struct Divisor {
    double d;
    unsigned long long R;
};

// One Newton-Raphson step on R ~ 2^63 / y (relative error below 2^-42) for the 53-bit significand m
// (y = m / 2^52): the residual 2^62 (1 - y R / 2^63) is below 2^20, so the correction is one 32 x 32-bit
// product.  The result's error is below 2^-60 relative (8 units of 2^-63).
SF_HD unsigned long long refine_rcp(unsigned long long m, unsigned long long R) {
    const unsigned long long phi = mulhi_near(m << 11, R);          // 0 to 3 low
    const int e = (int)(lo32(0x4000000000000000ull - phi)) - 1;     // 2^62 (1 - y R / 2^63)
    return R + (unsigned long long)(((long long)e * (int)(hi32(R) >> 1)) >> 29);
}
// The two leading parts of a significand's fraction as floats: 1.f (23 bits, exact) and the next 23
// bits scaled to [0, 1).
SF_HD float lead(unsigned long long m, unsigned one) { return f32_of(one | ((unsigned)(m >> 29) & 0x7fffffu)); }
SF_HD float next(unsigned long long m) { return f32_of(0x3f800000u | (((unsigned)m >> 6) & 0x7fffffu)) - 1.0f; }
// r (1 + c) 2^63 for r in [1/2, 1) and |c| < 2^-20, with c r given
SF_HD unsigned long long fixed63(float r, float cr) {
    const unsigned long long t = (unsigned long long)((u32_of(r) & 0x7fffffu) | 0x800000u) << 39;
    return t + ((unsigned long long)(long long)round32(cr * 0x1p47f) << 16);
}

SF_HD Divisor divisor(double b) {
    const unsigned long long ib = bits(b);
    Divisor D{b, 0ull};
    if (((unsigned)(ib >> 52) & 0x7ffu) - 1u < 2046u) {
        const unsigned long long mb = (ib & kMant) | kHid;
        // y = yh + yl 2^-23; r = 1 / yh nearly (kept in [1/2, 1)); e = 1 - r y to ~2^-44
        const float yh = lead(mb, 0x3f800000u), yl = next(mb);
        const float r = clamp32(rcp32(yh), 0.5f, 0.99999994f);
        const float e = fma32(-r * 0x1p-23f, yl, fma32(-r, yh, 1.0f));
        D.R = refine_rcp(mb, fixed63(r, r * fma32(e, e, e)));
    }
    return D;
}

SF_HD double div(double a, const Divisor& b) {
    const unsigned long long ia = bits(a), ib = bits(b.d);
    const unsigned ea = (unsigned)(ia >> 52) & 0x7ffu, eb = (unsigned)(ib >> 52) & 0x7ffu;
    if (b.R != 0ull && ea - 1u < 2046u) {
        const unsigned long long ma = (ia & kMant) | kHid, mb = (ib & kMant) | kHid;
        // quotient q = ma / mb in (1/2, 2) in units of 2^-54: its estimate (in units of 2^-62 off by -6 to
        // +9 from the exact quotient) less 8, truncated, is the floor or one below
        unsigned long long Q = (mulhi_near(ma << 11, b.R) - 8ull) >> 8;
        const unsigned long long rem = (ma << 54) - Q * mb;          // exact, in [0, 2 mb)
        Q += rem >= mb ? 1ull : 0ull;
        // q >= 1 has two bits below its 53, q < 1 one; a quotient is never halfway between two doubles
        const unsigned n = (unsigned)(Q >> 54);
        const int E = (int)ea - (int)eb + 1022 + (int)n;
        if ((unsigned)(E - 1) < 2045u) {
            const unsigned long long m = (Q + (1ull + n)) >> (1u + n);
            return dbl(((ia ^ ib) & kSign) + ((unsigned long long)(unsigned)(E - 1) << 52) + m);
        }
    }
    return hw_div(a, b.d);
}
SF_HD double div(double a, double b) { return div(a, divisor(b)); }

// The square root's parts for a in (0, inf), normal: R ~ 2^63 / sqrt(m) to ~43 bits, m = M / 2^52 in
// [1, 4), and S = the floor of sqrt(m) 2^53.
SF_HD unsigned long long root_floor(unsigned long long ma, unsigned odd, unsigned long long& R) {
    const float mh = lead(ma, odd ? 0x40000000u : 0x3f800000u), ml = next(ma) * (odd ? 0x1p-22f : 0x1p-23f);
    const float r = clamp32(rsqrt32(mh), 0.5f, 0.99999994f);
    const float p = r * r, pe = fma32(r, r, -p);
    const float e = fma32(-ml, p, fma32(-mh, pe, fma32(-mh, p, 1.0f)));   // 1 - m r^2 to ~2^-43
    R = fixed63(r, r * (e * fma32(0.375f, e, 0.5f)));
    const unsigned long long M = ma << odd;
    const unsigned long long S0 = mulhi_near(M << 10, R);                 // sqrt(m) 2^61
    // residual m - s^2 in units of 2^-58 (below 2^20), times r / 2: the root to a few 2^-61
    const int d = (int)lo32((M << 6) - mulhi_near(S0, S0)) - 1;
    const unsigned long long S1 = S0 + (unsigned long long)(((long long)d * (int)(hi32(R) >> 1)) >> 28);
    unsigned long long S = (S1 - 24ull) >> 8;                             // the floor or one below
    const unsigned long long rem = (M << 54) - S * S;                     // exact, in [0, 4 S + 4)
    S += rem > 2ull * S ? 1ull : 0ull;
    return S;
}
SF_HD double sqrt(double a) {
    const unsigned long long ia = bits(a);
    const unsigned ea = (unsigned)(ia >> 52);  // sign bit included: negatives take the fallback
    if (ea - 1u < 2046u) {
        const unsigned odd = (ea + 1u) & 1u;          // unbiased exponent odd: the root of 2 ma
        unsigned long long R;
        const unsigned long long S = root_floor((ia & kMant) | kHid, odd, R);
        const unsigned E = (ea + 1023u - odd) >> 1;   // (ea - 1023 - odd) / 2 + 1023
        return dbl(((unsigned long long)(E - 1u) << 52) + ((S + 1ull) >> 1));  // a root is never halfway
    }
    return hw_sqrt(a);
}
// The square root as a divisor.
SF_HD Divisor sqrt_divisor(double a) {
    const unsigned long long ia = bits(a);
    const unsigned ea = (unsigned)(ia >> 52);
    Divisor D;
    if (ea - 1u < 2046u) {
        const unsigned odd = (ea + 1u) & 1u;
        unsigned long long R;
        const unsigned long long S = root_floor((ia & kMant) | kHid, odd, R);
        const unsigned E = (ea + 1023u - odd) >> 1;
        const unsigned long long m = (S + 1ull) >> 1;
        D.d = dbl(((unsigned long long)(E - 1u) << 52) + m);
        // (a root that rounds up to 2 has significand 1: its reciprocal is exact)
        D.R = m == 2ull * kHid ? kSign : refine_rcp(m, R);
        return D;
    }
    D.d = hw_sqrt(a);
    return divisor(D.d);
}

// Conversions between float and double, on the integer pipes (conversion instructions with a 64-bit
// operand issue on GB300's FP64 pipe, at its rate).  widen is exact; narrow rounds to nearest even.
// Zeros, subnormals, infinities and NaN -- and doubles outside the normal float range -- take the
// hardware conversion.
SF_HD unsigned f32bits(float f) { return u32_of(f); }
SF_HD float f32of(unsigned u) { return f32_of(u); }
// (Out of line, as all fallbacks here: an inlined conversion or addition is evaluated on every call, beside
// the fast path, and selected from.)
SF_SLOW double hw_widen(float f) {
#if defined(__CUDA_ARCH__)
    return (double)f;
#else
    volatile double r = (double)f;
    return r;
#endif
}
SF_SLOW float hw_narrow(double d) {
#if defined(__CUDA_ARCH__)
    return __double2float_rn(d);
#else
    volatile float r = (float)d;
    return r;
#endif
}
SF_HD double widen(float f) {
    const unsigned u = f32bits(f), e = (u >> 23) & 0xffu;
    if (e == 0u || e == 0xffu) return hw_widen(f);
    // sign, exponent rebiased by 1023 - 127, the 23 significand bits on top of the double's 52
    return dbl(((unsigned long long)(u & 0x80000000u) << 32) | ((unsigned long long)(e + 896u) << 52) |
               ((unsigned long long)(u & 0x7fffffu) << 29));
}
// The product of two floats as a double: exact (48 bits).
SF_SLOW double hw_mul32(float a, float b) { return hw_mul(hw_widen(a), hw_widen(b)); }
SF_HD double mul32(float a, float b) {
    const unsigned u = f32bits(a), w = f32bits(b);
    const unsigned ea = (u >> 23) & 0xffu, eb = (w >> 23) & 0xffu;
    if (ea - 1u < 254u && eb - 1u < 254u) {
        const unsigned long long p = wide((u & 0x7fffffu) | 0x800000u, (w & 0x7fffffu) | 0x800000u);   // [2^46, 2^48)
        const unsigned n = hi32(p) >> 15, sh = 6u - n;
        const unsigned top = ((u ^ w) & 0x80000000u) + ((ea + eb + n + 768u) << 20) + shl2(hi32(p), lo32(p), sh);
        return dbl(((unsigned long long)top << 32) | (lo32(p) << sh));
    }
    return hw_mul32(a, b);
}
SF_HD float narrow(double d) {
    const unsigned long long b = bits(d);
    const int e = (int)((b >> 52) & 0x7ff);
    if (e < 1023 - 126 || e > 1023 + 127) return hw_narrow(d);
    // 23 significand bits kept, 29 rounded: to nearest, ties to even; a carry out of the
    // significand raises the exponent (up to infinity from the largest binade), as IEEE rounding does
    const unsigned m = (unsigned)((b >> 29) & 0x7fffffu), r = (unsigned)(b & 0x1fffffffu);
    unsigned f = ((unsigned)(b >> 32) & 0x80000000u) | ((unsigned)(e - 896) << 23) | m;
    if (r > 0x10000000u || (r == 0x10000000u && (m & 1u))) f += 1u;
    return f32of(f);
}

}  // namespace sf
