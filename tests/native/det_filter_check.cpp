// Host check of csrc/svm_det_filter.h: wherever it decides, the sign is that of the FP64 determinant as
// the force kernel's formula evaluates it.  Triangles of spheres of radius 0.01 to 1e9 and free points,
// from ordinary ones to slivers, repeated points and coordinates with zeros; counts the undecided of
// ordinary triangles.   Usage: det_filter_check [cases]
#include "svm_det_filter.h"
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <random>

struct P { double x, y, z; };
static double det3(P a, P b, P c) {
    return a.x * (b.y * c.z - b.z * c.y) + a.y * (b.z * c.x - b.x * c.z) + a.z * (b.x * c.y - b.y * c.x);
}

int main(int argc, char** argv) {
    const long n = argc > 1 ? std::atol(argv[1]) : 2000000;
    std::mt19937_64 g(3);
    std::normal_distribution<double> nd;
    std::uniform_real_distribution<double> un(0.0, 1.0);
    long wrong = 0, ordinary = 0, undecided = 0;
    for (long i = 0; i < n; ++i) {
        const double R = i % 3 ? std::sqrt(std::exp(un(g) * 9.6 + 4.0) / 12.566) : std::pow(10.0, -2.0 + 11.0 * un(g));
        P v{nd(g), nd(g), nd(g)};
        const double r = std::sqrt(v.x * v.x + v.y * v.y + v.z * v.z);
        v = P{R * v.x / r, R * v.y / r, R * v.z / r};
        if (i % 29 == 0) v = P{R, 0.0, -0.0};
        const bool plain = i % 3 && i % 5;
        const double len = i % 5 ? 0.3 + 0.5 * un(g) : R * std::pow(10.0, -12.0 * un(g));
        auto near = [&](double l) {
            P q{v.x + l * nd(g), v.y + l * nd(g), v.z + l * nd(g)};
            if (i % 7 == 0) return q;   // off the sphere
            const double t = R / std::sqrt(q.x * q.x + q.y * q.y + q.z * q.z);
            return P{t * q.x, t * q.y, t * q.z};
        };
        P b = near(len), c = near(len);
        if (i % 11 == 0) { const double t = un(g), e = std::pow(10.0, -15.0 * un(g)); c = P{v.x + t * (b.x - v.x) + e * nd(g), v.y + t * (b.y - v.y), v.z + t * (b.z - v.z) + e * nd(g)}; }
        if (i % 97 == 0) c = b;
        if (i % 101 == 0) b = v;
        const svm_det::F3 v32 = svm_det::near3(v.x, v.y, v.z);
        const int k = svm_det::below_zero(v32, svm_det::diff(svm_det::near3(b.x, b.y, b.z), v32),
                                          svm_det::diff(svm_det::near3(c.x, c.y, c.z), v32));
        if (k >= 0) wrong += (k == 1) != (det3(v, b, c) < 0);
        if (plain && i % 11 && i % 7 && i % 97 && i % 101 && i % 29) { ++ordinary; undecided += k < 0; }
    }
    for (double x : {0.0, -0.0, 1e-320, 1e-39, 1e39, (double)INFINITY, (double)NAN, -1e300}) {  // out of FP32's range
        const float f = svm_det::near32(x);
        const float want = std::fabs(x) < 0x1p-126 ? 0.f : NAN;
        wrong += !(f == want || (f != f && want != want));
    }
    std::printf("{\"wrong\": %ld, \"ordinary\": %ld, \"undecided\": %ld}\n", wrong, ordinary, undecided);
    return wrong ? 1 : 0;
}
