// Host check of the special products of csrc/svm_softf64.cuh against the host's IEEE operations: the square of
// a double and the exact product of two floats, on random bits, the edges of the exponent range, significands of
// few bits and squares next to a rounding tie.  Prints the mismatches as JSON.
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <random>
#include "svm_softf64.cuh"

static bool same(double x, double y) { return (std::isnan(x) && std::isnan(y)) || sf::bits(x) == sf::bits(y); }

int main(int argc, char** argv) {
    const long cases = argc > 1 ? std::atol(argv[1]) : 2000000;
    std::mt19937_64 g(argc > 2 ? std::strtoull(argv[2], nullptr, 10) : 1);
    long badS = 0, badM = 0, badN = 0;
    for (long i = 0; i < cases; ++i) {
        unsigned long long u = g();
        if (i % 3) u = (u & (sf::kMant | sf::kSign)) | ((1023ull + g() % 81 - 40) << 52);
        if (i % 5 == 0) u &= ~0x3FFFFFFull;                            // 27 bits: squares with exact ties
        if (i % 7 == 0) u = (u & ~sf::kMant) | (g() & 0xF);
        if (i % 11 == 0) u = (u | sf::kMant) ^ (g() & 0xF);
        if (i % 13 == 0) u = (u & ~(0x7FFull << 52)) | ((g() % 2 ? 509ull + g() % 6 : 1532ull + g() % 6) << 52);
        if (i % 17 == 0) u = (u & ~(0x7FFull << 52)) | ((g() % 2 ? 0ull : 2047ull) << 52);
        const double x = sf::dbl(u);
        badS += !same(sf::sqr(x), sf::hw_mul(x, x));
        unsigned a = (unsigned)g(), b = (unsigned)g();
        if (i % 3) a = (a & 0x807fffffu) | ((127u + (unsigned)(g() % 41) - 20u) << 23);
        if (i % 5 == 0) b &= 0xfff00000u;
        if (i % 7 == 0) b = (b & 0xff800000u) | (unsigned)(g() & 3u);
        if (i % 11 == 0) a |= 0x7fffffu;
        if (i % 13 == 0) b = (b & 0x807fffffu) | ((g() % 2 ? 0u : 255u) << 23);
        if (i % 17 == 0) a = (a & 0x807fffffu) | ((g() % 2 ? 1u : 254u) << 23);
        const float p = sf::f32of(a), q = sf::f32of(b);
        badM += !same(sf::mul32(p, q), sf::hw_mul((double)p, (double)q));
        badN += !same(sf::negate_if(i & 1, x), (i & 1) ? -x : x);
    }
    std::printf("{\"cases\": %ld, \"sqr\": %ld, \"mul32\": %ld, \"negate\": %ld}\n", cases, badS, badM, badN);
    return 0;
}
