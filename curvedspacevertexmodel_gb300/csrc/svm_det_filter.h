// The sign of det(v1, v2, v3) (sphericalDomain.h:395-402 flips a triangle's gradient by it) in FP32 where
// that is certain: the FP64 determinant is 14 instructions of GB300's scarce FP64 pipe (2 lanes per
// clock per SM) and its sign is all that is used.  Host and device builds evaluate the same IEEE FP32
// operations, so tests/native/det_filter_check.cpp checks the bound on the CPU.
#pragma once
#include "svm_softf64.cuh"

namespace svm_det {

struct F3 { float x, y, z; };

// x as a float, truncated to 24 significant bits, on the integer pipes (sign kept; magnitudes below
// 2^-126 read as 0, those of 2^128 or more, infinities and NaN as NaN).
SF_HD float near32(double x) {
    const unsigned long long u = sf::bits(x);
    const unsigned hi = sf::hi32(u), e = (hi >> 20) & 0x7ffu;
    // sign and exponent rebiased by 127 - 1023 = -896, which is +128 modulo 256, and 23 mantissa bits
    const unsigned f = ((sf::shl2(hi, sf::lo32(u), 3) + (128u << 23)) & 0x7fffffffu) | (hi & 0x80000000u);
    if (e - 897u < 254u) return sf::f32_of(f);
    return e < 897u ? 0.f : sf::f32_of(0x7fc00000u);
}
SF_HD F3 near3(double x, double y, double z) { return F3{near32(x), near32(y), near32(z)}; }
SF_HD F3 diff(F3 a, F3 b) { return F3{a.x - b.x, a.y - b.y, a.z - b.z}; }
SF_HD float abs32(float x) { return sf::f32_of(sf::u32_of(x) & 0x7fffffffu); }
SF_HD float norm1(F3 a) { return abs32(a.x) + abs32(a.y) + abs32(a.z); }

// Whether det(v, v + b, v + c), as the FP64 formula evaluates it, is below 0, from the FP32 differences
// b, c of near3 points: 1 or 0 where that is certain, else -1.  With s = |v|_1 + |b|_1 + |c|_1 (no
// smaller than any of the three points): truncation moves a difference by at most 2.4e-7 s and the
// FP32 products and sums add a few 6e-8 relative, so D = v . (b x c) is within
// s^2 (1e-6 (|b|_1 + |c|_1) + 1e-13 s) of the exact determinant, and the FP64 formula within 5e-15 s^3
// of it; a |D| beyond four times the former fixes the sign of both (a NaN or an overflow decides
// nothing; coordinates so small that FP32 products could underflow neither).
SF_HD int below_zero(F3 v, F3 b, F3 c) {
    const float D = v.x * (b.y * c.z - b.z * c.y) + v.y * (b.z * c.x - b.x * c.z) + v.z * (b.x * c.y - b.y * c.x);
    const float l = norm1(b) + norm1(c), s = norm1(v) + l;
    if (abs32(D) > 4e-6f * s * s * (l + 1e-6f * s) && s < 1e12f && s > 1e-6f) return D < 0.f ? 1 : 0;
    return -1;
}

}  // namespace svm_det
