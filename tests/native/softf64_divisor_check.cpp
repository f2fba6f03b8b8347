// Host check of the divisor forms of csrc/svm_softf64.cuh against the host's IEEE operations: a quotient by
// a kept divisor, a quotient by a square root (sqrt_divisor), and the exact doubling.  Built with
// -DSF_HOST_SEED_ULPS=k, whose seeds are k ulp off: the results may not depend on the seed.
//   Usage: softf64_divisor_check [cases]
#include "svm_softf64.cuh"
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <random>

static bool same(double x, double y) { return (std::isnan(x) && std::isnan(y)) || sf::bits(x) == sf::bits(y); }

int main(int argc, char** argv) {
    const long n = argc > 1 ? std::atol(argv[1]) : 1000000;
    std::mt19937_64 g(7);
    long bad[5] = {0, 0, 0, 0, 0};
    auto draw = [&](bool any) {
        const unsigned long long u = g();
        if (any) return sf::dbl(u);
        return sf::dbl((u & (sf::kMant | sf::kSign)) | ((1023ull + (long long)(g() % 81) - 40) << 52));
    };
    for (long i = 0; i < n; ++i) {
        double a = draw(i % 5 == 0), c = draw(i % 7 == 0), b = draw(i % 6 == 0);
        if (i % 11 == 0) b = sf::dbl((sf::bits(b) & ~sf::kMant) | (g() & 0xFull));       // just above 2^k
        if (i % 13 == 0) b = sf::dbl((sf::bits(b) | sf::kMant) ^ (g() & 0xFull));        // just below 2^k
        if (i % 17 == 0) b = sf::dbl((sf::bits(b) & ~sf::kMant) | ((g() & 0x7FFFFF) << 29) | (i % 2 ? 0x1FFFFFFF : g() & 63));
        if (i % 19 == 0) b = sf::hw_mul(b, b);                                            // an exact root, often
        if (i % 23 == 0) b = i % 2 ? 0.0 : (i % 3 ? INFINITY : 1e-310);
        const sf::Divisor d = sf::divisor(b), r = sf::sqrt_divisor(b);
        const double root = sf::hw_sqrt(b);
        bad[0] += !same(sf::div(a, d), sf::hw_div(a, b)) + !same(sf::div(c, d), sf::hw_div(c, b));
        bad[1] += !same(sf::div(a, r), sf::hw_div(a, root)) + !same(sf::div(c, r), sf::hw_div(c, root));
        bad[2] += !same(r.d, root);
        bad[3] += !same(sf::twice(a), sf::hw_add(a, a));
        bad[4] += !same(sf::mul(a, b), sf::hw_mul(a, b));
    }
    std::printf("{\"div\": %ld, \"div_root\": %ld, \"root\": %ld, \"twice\": %ld, \"mul\": %ld}\n", bad[0], bad[1], bad[2],
                bad[3], bad[4]);
    return (bad[0] | bad[1] | bad[2] | bad[3] | bad[4]) ? 1 : 0;
}
