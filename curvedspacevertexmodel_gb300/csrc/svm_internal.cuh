// Internal state and FP64 device math of libsvm.
//
// Device layout (structure of arrays, one GPU):
//   pos[2]      double4_32a[Nv]   vertex positions (x,y,z,0); two buffers so the fused
//                             force+integrate+move kernel reads old and writes new positions
//   vsph        double4_32a[Nv]   per-vertex spherical coordinates (cos t, sin t, cos p, sin p)
//   vcell/vnbr  int4[Nv]      vertex->cell and vertex->vertex slots (w unused)
//   vlast/vnext int4[Nv]      ring predecessor / successor of the vertex in each of its cells
//   vrpos       int4[Nv]      position of the vertex in each of its cells' rings
//   ring        int[N*Wc]     clockwise ring of each cell, capacity Wc; ringCount int[N]
//   corner      double2[N*Wc] per ring position k: (arc(ring[k-1], ring[k]), included angle at k)
//   cellPos     double4_32a[N]    renormalised ring centroid; cellSph double4_32a[N] its (cos t, ...)
//   ap, pref    double2[N]    (area, perimeter) and (A0, P0)
//   force, vel  double4_32a[Nv]
// The reference keeps AoS double[3] vertices and scatters (last, cur, next) vertex copies into
// per-(vertex, cell) slots every step (src/model/sphericalVertexModel.cu:94-96); here the force
// kernel gathers them through vlast/vnext instead, which removes 3 x 24 B x 3Nv of writes.
#pragma once
#include <cuda_runtime.h>
#include <cstdint>
#include <vector>
#include "../../include/svm.h"
#include "svm_acos.h"
#include "svm_softf64.cuh"
#include "svm_edge_filter.h"
#include "svm_det_filter.h"

namespace svm {

constexpr double kPI = 3.141592653589793115997963468544185161590576171875;
// pi - kPI (the next term of pi's double-double expansion)
constexpr double kPILo = 1.2246467991473532e-16;

struct D3 { double x, y, z; };

// Division and square root of the FP64 kernels.  Both are the IEEE correctly rounded operations
// either way; by default they run on the integer and FP32 pipes (svm_softf64.cuh), which leaves
// GB300's FP64 pipe -- 2 lanes per clock per SM, the bound of these kernels -- to the products and
// sums, where a hardware division or square root would take about eight FP64 instructions.  kHw
// (the T1 pass's kernels, where one warp's chain of dependent operations, not the FP64 pipe's
// issue rate, sets the time) takes the hardware sequences, whose latency is shorter; so does a
// build with -DSVM_NATIVE_FP64_DIV.  The results are the same bits.
template <bool kHw = false>
__device__ __forceinline__ double f64_div(double a, double b) {
#ifdef SVM_NATIVE_FP64_DIV
    return __ddiv_rn(a, b);
#else
    if constexpr (kHw) return __ddiv_rn(a, b);
    else return sf::div(a, b);
#endif
}
template <bool kHw = false>
__device__ __forceinline__ double f64_sqrt(double a) {
#ifdef SVM_NATIVE_FP64_DIV
    return __dsqrt_rn(a);
#else
    if constexpr (kHw) return __dsqrt_rn(a);
    else return sf::sqrt(a);
#endif
}

// A divisor used more than once, and a square root used as a divisor: the quotients are f64_div's.
#ifdef SVM_NATIVE_FP64_DIV
struct F64Divisor { double d; };
__device__ __forceinline__ F64Divisor f64_root_divisor(double a) { return F64Divisor{__dsqrt_rn(a)}; }
__device__ __forceinline__ F64Divisor kept_divisor(double b) { return F64Divisor{b}; }
__device__ __forceinline__ double f64_div(double a, const F64Divisor& b) { return __ddiv_rn(a, b.d); }
#else
using F64Divisor = sf::Divisor;
__device__ __forceinline__ F64Divisor f64_root_divisor(double a) { return sf::sqrt_divisor(a); }
__device__ __forceinline__ F64Divisor kept_divisor(double b) { return sf::divisor(b); }
__device__ __forceinline__ double f64_div(double a, const F64Divisor& b) { return sf::div(a, b); }
#endif
// a / sqrt(b)
template <bool kHw = false>
__device__ __forceinline__ double f64_div_root(double a, double b) {
    if constexpr (kHw) return __ddiv_rn(a, __dsqrt_rn(b));
    else return f64_div(a, f64_root_divisor(b));
}

// The arccosine of the FP64 geometry (arcs, included angles, triangle areas, T1 length tests).
// The default build uses CUDA's acos; a build with -DSVM_PORTABLE_ACOS uses svm_portable::acos,
// the same operations as the CPU restatement's portable mode, which makes GPU and CPU trajectories
// comparable bit for bit.
__device__ __forceinline__ double svm_acos(double x) {
#ifdef SVM_PORTABLE_ACOS
    return svm_portable::acos(x);
#else
    return acos(x);
#endif
}

__device__ __forceinline__ D3 ld3(const double4_32a* p, int i) {
    double4_32a t = p[i];
    return D3{t.x, t.y, t.z};
}
__device__ __forceinline__ void st3(double4_32a* p, int i, D3 v) { p[i] = make_double4_32a(v.x, v.y, v.z, 0.0); }
// FP32 positions (mixed-precision form): widened exactly on load, rounded to nearest on store (the
// conversions on the integer pipes: sf::widen, sf::narrow).
__device__ __forceinline__ D3 ld3(const float4* p, int i) {
    const float4 t = p[i];
    return D3{sf::widen(t.x), sf::widen(t.y), sf::widen(t.z)};
}
__device__ __forceinline__ void st3(float4* p, int i, D3 v) {
    p[i] = make_float4(sf::narrow(v.x), sf::narrow(v.y), sf::narrow(v.z), 0.f);
}
// In the mixed form the w component of a vertex's FP32 position holds its replica index (0 for a
// single sphere); rounded stores of a vertex keep it.
__device__ __forceinline__ void st3_keep(float4* p, int i, D3 v) {
    p[i] = make_float4(sf::narrow(v.x), sf::narrow(v.y), sf::narrow(v.z), p[i].w);
}
__device__ __forceinline__ int rep_of(const float4& p) { return (int)p.w; }
__device__ __forceinline__ int rep_of(const double4_32a&) { return 0; }
__device__ __forceinline__ D3 add3(D3 a, D3 b) { return D3{a.x + b.x, a.y + b.y, a.z + b.z}; }
__device__ __forceinline__ D3 sub3(D3 a, D3 b) { return D3{a.x - b.x, a.y - b.y, a.z - b.z}; }
__device__ __forceinline__ D3 scl3(double s, D3 a) { return D3{s * a.x, s * a.y, s * a.z}; }
// dot (inc/functions.h:131-138): accumulated in component order
__device__ __forceinline__ double dot3(D3 a, D3 b) { double s = a.x * b.x; s += a.y * b.y; s += a.z * b.z; return s; }
__device__ __forceinline__ D3 cross3(D3 p1, D3 p2) {          // inc/functions.h:160-167
    return D3{p1.y * p2.z - p1.z * p2.y, p1.z * p2.x - p1.x * p2.z, p1.x * p2.y - p1.y * p2.x};
}
// A product on the integer pipes (sf::mul: the same bits as the hardware multiply), for products the
// FP64 pipe -- the bound of these kernels -- can be spared: the cross and dot products ahead of the
// geometry's divisions and arccosines (corner phase 0.159 -> 0.151 ms at 100k cells when they moved), the
// norms ahead of the centroids', vertices' and fan triangles' square roots (cells and fallback phases
// 2-3% shorter).  The gradients' products are grad_mul.
// (kHw: the hardware multiply, for the T1 pass's latency-bound chains and for small models: kFewHwMul.)
template <bool kHw = false>
__device__ __forceinline__ double early_mul(double x, double y) {
    if constexpr (kHw) return __dmul_rn(x, y);
    else return sf::mul(x, y);
}
// dot3 and cross3 with their products on the integer pipes (the same bits)
template <bool kHw = false>
__device__ __forceinline__ double dot3e(D3 a, D3 b) {
    double s = early_mul<kHw>(a.x, b.x);
    s += early_mul<kHw>(a.y, b.y);
    s += early_mul<kHw>(a.z, b.z);
    return s;
}
// dot3e(a, a)
template <bool kHw = false>
__device__ __forceinline__ double norm2e(D3 a) {
    if constexpr (kHw) return dot3e<true>(a, a);
    double s = sf::sqr(a.x);
    s += sf::sqr(a.y);
    s += sf::sqr(a.z);
    return s;
}
// cross3 of FP32 points: the products are exact
__device__ __forceinline__ D3 cross32(float4 a, float4 b) {
    return D3{sf::mul32(a.y, b.z) - sf::mul32(a.z, b.y), sf::mul32(a.z, b.x) - sf::mul32(a.x, b.z),
              sf::mul32(a.x, b.y) - sf::mul32(a.y, b.x)};
}
template <bool kHw = false>
__device__ __forceinline__ D3 cross3e(D3 p1, D3 p2) {
    return D3{early_mul<kHw>(p1.y, p2.z) - early_mul<kHw>(p1.z, p2.y),
              early_mul<kHw>(p1.z, p2.x) - early_mul<kHw>(p1.x, p2.z),
              early_mul<kHw>(p1.x, p2.y) - early_mul<kHw>(p1.y, p2.x)};
}
__device__ __forceinline__ double det3(D3 a, D3 b, D3 c) {    // a . (b x c), sphericalDomain.h:123-125
    return a.x * (b.y * c.z - b.z * c.y) + a.y * (b.z * c.x - b.x * c.z) + a.z * (b.x * c.y - b.y * c.x);
}

// putInBoxReal (sphericalDomain.h:183-187): p <- R p / |p|
template <bool kHwMul = false, bool kHwScale = true>
__device__ __forceinline__ D3 renorm(D3 p, double R) {
    const auto M = [](double x, double y) { return early_mul<kHwScale>(x, y); };
    const double inv = f64_div_root(1.0, norm2e<kHwMul>(p));
    return D3{M(R, M(inv, p.x)), M(R, M(inv, p.y)), M(R, M(inv, p.z))};
}
// move(p, v) (sphericalDomain.h:203-209): project v onto the tangent plane at p, add, renormalise
__device__ __forceinline__ D3 sphere_move(D3 p, D3 v, double R) {
    double s = f64_div(dot3(v, p), dot3(p, p));
    D3 d = sub3(v, scl3(s, p));
    return renorm(add3(p, d), R);
}
// geodesicDistance (sphericalDomain.h:94-112)
template <bool kHw = false>
__device__ __forceinline__ double geodesic(D3 p1, D3 p2, double R) {
    double num = p1.x * p2.x + p1.y * p2.y + p1.z * p2.z;
    double den = f64_sqrt<kHw>(p1.x * p1.x + p1.y * p1.y + p1.z * p1.z) *
                 f64_sqrt<kHw>(p2.x * p2.x + p2.y * p2.y + p2.z * p2.z);
    return R * svm_acos(f64_div<kHw>(num, den));
}
// |p| as geodesic and sph_coords evaluate it (same operations, so the same value)
template <bool kHw = false, bool kHwMul = kHw>
__device__ __forceinline__ double pos_norm(D3 p) { return f64_sqrt<kHw>(norm2e<kHwMul>(p)); }
// geodesic with the two norms given (n1 = pos_norm(p1), n2 = pos_norm(p2)): the same value
template <bool kHwMul = false>
__device__ __forceinline__ double geodesic_n(D3 p1, D3 p2, double n1, double n2, double R) {
    return R * svm_acos(f64_div(dot3e<kHwMul>(p1, p2), early_mul<kHwMul>(n1, n2)));
}
// The T1 length test geodesic(p1, p2) < t, i.e. R acos(c) < t with c = p1.p2 / (|p1||p2|).  acos
// is decreasing, so away from c = cos(t / R) the answer is c > cos(t / R); the formula itself is
// evaluated only when c lies within [cosLo, cosHi], a bracket around cos(t / R) of half-width
// 1e-9, which is many orders wider than the error of acos and of the rounding of c, or when c > 1.
__host__ __device__ inline void t1_bracket(double t, double R, double* lo, double* hi) {
    if (!(t > 0.0)) {   // an arc is never below a threshold of 0 or less: every c < lo decides "no"
        *lo = *hi = 2.0;
        return;
    }
    const double c = cos(t / R);
    *lo = c - 1e-9;
    *hi = c + 1e-9;
}
// A pre-test decides the edges away from the threshold without square roots or divisions:
// sin^2(angle) = |p1 x p2|^2 / (|p1|^2 |p2|^2) against sin^2(a) (1 -/+ eps) (s2Lo, s2Hi), a = t / R,
// for angles below pi / 2 (p1.p2 > 0) and above 3e-7 (|p1 x p2|^2 > 1e-13 |p1|^2 |p2|^2: closer
// to 0, c can round to 1 or past it, where the reference's acos is 0 or NaN).  The formula's
// decision is c > c* with c* within 1e-30 of cos(a), and c within 5e-16 of the cosine of the angle;
// outside the band, the cosine differs from cos(a) by at least a^2 eps / 2 >= 5e-13, and the
// pre-test's own relative error is below 1e-9 / a, so every decision it takes is the formula's.
// eps = max(1e-6, 1e-12 / a^2); thresholds of 0 or of 1 radian or more skip the pre-test.
__host__ inline void t1_sin2_bracket(double t, double R, double* lo, double* hi) {
    const double a = t / R;
    if (!(a > 0.0 && a < 1.0)) {   // never decides: xx < -d and xx > 2 d are impossible
        *lo = -1.0;
        *hi = 2.0;
        return;
    }
    const double s = sin(a);
    double eps = 1e-12 / (a * a);
    if (eps < 1e-6) eps = 1e-6;
    *lo = s * s * (1.0 - eps);
    *hi = s * s * (1.0 + eps);
}
template <bool kHw = false>
__device__ __forceinline__ bool shorter_than(D3 p1, D3 p2, double R, double t, double cosLo, double cosHi,
                                             double s2Lo, double s2Hi) {
    if (svm_edge::clearly_longer(p1.x, p1.y, p1.z, p2.x, p2.y, p2.z, R, t)) return false;
    const double num = p1.x * p2.x + p1.y * p2.y + p1.z * p2.z;
    if (num > 0) {
        const D3 x = cross3(p1, p2);
        const double xx = dot3(x, x), d = dot3(p1, p1) * dot3(p2, p2);
        if (xx < s2Lo * d && xx > 1e-13 * d) return true;
        if (xx > s2Hi * d) return false;
    }
    const double den = f64_sqrt<kHw>(p1.x * p1.x + p1.y * p1.y + p1.z * p1.z) *
                       f64_sqrt<kHw>(p2.x * p2.x + p2.y * p2.y + p2.z * p2.z);
    const double c = f64_div<kHw>(num, den);
    if (c > cosHi && c <= 1.0) return true;   // c > 1 (rounding) makes acos NaN: not shorter
    if (c < cosLo) return false;
    return R * svm_acos(c) < t;
}
// Arc length in the mixed-precision form: 2 R asin(|q - p| / 2R) in FP32 from the raw chord
// (exact for nearby FP32 points), well conditioned for the short arcs of the model (the acos form
// loses half its digits there).
__device__ __forceinline__ float arc32(float4 p, float4 q, float R) {
    const float dx = q.x - p.x, dy = q.y - p.y, dz = q.z - p.z;
    return 2.0f * R * asinf(sqrtf(dx * dx + dy * dy + dz * dz) / (2.0f * R));
}
// includedAngle (sphericalDomain.h:114-133)
template <bool kHw = false>
__device__ __forceinline__ double included_angle(D3 p1, D3 p2, D3 p3) {
    D3 ci = cross3(p2, p3), cim1 = cross3(p1, p2);
    double det = det3(p1, p2, p3);
    double a = svm_acos(f64_div<kHw>(-dot3(ci, cim1), f64_sqrt<kHw>(dot3(ci, ci)) * f64_sqrt<kHw>(dot3(cim1, cim1))));
    if (det > 0) a = -a;
    if (a < 0) a += 2. * kPI;
    return a;
}
// includedAngle(pl, p, px) from the cross products Cx = p x px and Cl = p x pl and their norms,
// computed once per neighbour of p: cross(pl, p) = -(p x pl) exactly, the negations cancel exactly
// in the dot product and the norms, and det(pl, p, px) = pl . (p x px) in the same operation
// order, so the result is bitwise included_angle(pl, p, px).
//
// With `clamp` (the mixed form) the cosine is clamped to [-1, 1]: for a nearly straight corner its
// rounding can leave the domain, where acos is NaN (the reference does not clamp, and the FP64
// form keeps that behaviour).  In two parts, around the arccosine; comparisons on the integer pipes.
__device__ __forceinline__ bool positive(double x) {   // x > 0
    return (unsigned long long)__double_as_longlong(x) - 1ull < 0x7ff0000000000000ull;
}
template <bool clamp = false, bool kHwMul = false>
__device__ __forceinline__ double included_cos(D3 Cx, D3 Cl, double nx, double nl) {
    double c = f64_div(dot3e<kHwMul>(Cx, Cl), early_mul<kHwMul>(nx, nl));
    // fmin(1, fmax(-1, c)), a NaN to -1
    if (clamp) {
        const unsigned long long b = (unsigned long long)__double_as_longlong(c), m = b & 0x7fffffffffffffffull;
        if (m > 0x3ff0000000000000ull) c = (b >> 63) || m > 0x7ff0000000000000ull ? -1.0 : 1.0;
    }
    return c;
}
// the angle from its arccosine a (in [0, pi], or NaN) and whether det(pl, p, px) > 0: a, or 2 pi - a
__device__ __forceinline__ double included_finish(double a, bool detPositive) {
    if (detPositive) a = positive(a) ? 2. * kPI - a : sf::negate_if(true, a);
    return a;
}

// det(pl, p, px) > 0, the side of the corner (p x px = X): in FP32 where that is certain (svm_det), else as the
// FP64 formula.  det(p, pl, px) is its negative.
static __device__ __noinline__ bool det_positive_exact(D3 pl, D3 X) { return positive(dot3e(pl, X)); }
__device__ __forceinline__ bool det_positive(svm_det::F3 pl, svm_det::F3 p, svm_det::F3 px, D3 pl64, D3 X) {
    const int n = svm_det::below_zero(p, svm_det::diff(pl, p), svm_det::diff(px, p));
    return n >= 0 ? n != 0 : det_positive_exact(pl64, X);
}
// Arccosines of a block's cosines with like magnitudes on the same warps.  An arccosine evaluates one of
// two expansions by the magnitude of its argument, and the angles of a vertex model (60 to 180 degrees)
// fall on both sides, so a warp of them in vertex order runs both: about 50 FP64 instructions instead of
// 25.  The block's kPer values per thread are dealt out with the magnitudes below kAcosSplit first and the
// others last (one warp's worth mixed), evaluated, and dealt back: the same value for each.
// val: kPer blockDim.x doubles, src: as many shorts, warpHigh: an int per warp.  Every thread of the
// block calls it.
// The boundary is where the measured time is least; the corner phase against one arccosine per thread in
// vertex order: FP32 positions 1M cells 800 -> 589 us, 100k 100 -> 74.5 (with the boundary at 0.5 84.4, 0.55
// 82.7, 0.6 89.6, 0.625 94.2), FP64 100k 123 -> 102.
constexpr unsigned kAcosSplit = 0x3fe26666u;   // high word of the boundary, 0.575
template <int kPer>
__device__ __forceinline__ void block_acos(double (&c)[kPer], double* val, unsigned short* src, int* warpHigh) {
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5, n = blockDim.x;
    unsigned high[kPer];
    int before[kPer], mine = 0;   // high values of the warp ahead of this one, by (j, lane)
#pragma unroll
    for (int j = 0; j < kPer; ++j) {
        high[j] = ((unsigned)__double2hiint(c[j]) & 0x7fffffffu) >= kAcosSplit;
        const unsigned m = __ballot_sync(0xffffffffu, high[j]);
        before[j] = mine + __popc(m & ((1u << lane) - 1u));
        mine += __popc(m);
    }
    if (lane == 0) warpHigh[warp] = mine;
    __syncthreads();
    int ahead = 0;   // high values of the warps ahead
    for (int w = 0; w < warp; ++w) ahead += warpHigh[w];
#pragma unroll
    for (int j = 0; j < kPer; ++j) {
        const int h = ahead + before[j], k = 32 * kPer * warp + 32 * j + lane;
        const int at = high[j] ? kPer * n - 1 - h : k - h;
        val[at] = c[j];
        src[at] = (unsigned short)(j * n + t);
    }
    __syncthreads();
    double a[kPer];
    int from[kPer];
#pragma unroll
    for (int j = 0; j < kPer; ++j) {
        a[j] = svm_acos(val[j * n + t]);
        from[j] = src[j * n + t];
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < kPer; ++j) val[from[j]] = a[j];
    __syncthreads();
#pragma unroll
    for (int j = 0; j < kPer; ++j) c[j] = val[j * n + t];
}
// element j of a three-element register array (selects, no local-memory indexing)
template <class T>
__device__ __forceinline__ T pick3(const T* a, int j) { return j == 0 ? a[0] : (j == 1 ? a[1] : a[2]); }
// slot of vertex u among the three neighbour slots nb (-1 if absent)
__device__ __forceinline__ int nbr_slot(int4 nb, int u) { return u == nb.x ? 0 : (u == nb.y ? 1 : (u == nb.z ? 2 : -1)); }
// included_angle with the cosine clamped to [-1, 1] (the mixed form)
template <bool kHw = false>
__device__ __forceinline__ double included_angle_clamped(D3 p1, D3 p2, D3 p3) {
    D3 ci = cross3(p2, p3), cim1 = cross3(p1, p2);
    double det = det3(p1, p2, p3);
    double c = f64_div<kHw>(-dot3(ci, cim1), f64_sqrt<kHw>(dot3(ci, ci)) * f64_sqrt<kHw>(dot3(cim1, cim1)));
    double a = svm_acos(fmin(1.0, fmax(-1.0, c)));
    if (det > 0) a = -a;
    if (a < 0) a += 2. * kPI;
    return a;
}
// sphericalTriangleArea (sphericalDomain.h:135-166)
// q / |q| as sphericalTriangleArea normalises each corner
__device__ __forceinline__ D3 unit_corner(D3 q) { return scl3(f64_div_root(1.0, norm2e(q)), q); }
__device__ __forceinline__ double triangle_area_unit(D3 p1, D3 p2, D3 p3, double R);
__device__ __forceinline__ double triangle_area(D3 q1, D3 q2, D3 q3, double R) {
    return triangle_area_unit(unit_corner(q1), unit_corner(q2), unit_corner(q3), R);
}
// the cosines of the three angles, from the normalised corners
__device__ __forceinline__ void triangle_cosines(D3 p1, D3 p2, D3 p3, double (&c)[3]) {
    const double d12 = dot3e(p1, p2), d13 = dot3e(p1, p3), d23 = dot3e(p2, p3);
    const auto M = [](double x, double y) { return early_mul(x, y); };
    const double s12 = f64_sqrt(1 - sf::sqr(d12)), s13 = f64_sqrt(1 - sf::sqr(d13)), s23 = f64_sqrt(1 - sf::sqr(d23));
    c[0] = f64_div(d23 - M(d12, d13), M(s12, s13));
    c[1] = f64_div(d12 - M(d13, d23), M(s13, s23));
    c[2] = f64_div(d13 - M(d12, d23), M(s12, s23));
}
// the area from the three angles
__device__ __forceinline__ double triangle_sum(const double (&a)[3], double R) {
    double area = -kPI;
    area += a[0];
    area += a[1];
    area += a[2];
    return area * (R * R);
}
__device__ __forceinline__ double triangle_area_unit(D3 p1, D3 p2, D3 p3, double R) {
    double c[3];
    triangle_cosines(p1, p2, p3, c);
    const double a[3] = {svm_acos(c[0]), svm_acos(c[1]), svm_acos(c[2])};
    return triangle_sum(a, R);
}

// The total-area check of the mixed form (sphericalVertexModel.cpp:304-310 compares with 1e-6): the areas
// of nC cells on a sphere of radius R sum to 4 pi R^2 plus whole turns of R^2 -- what the check is after --
// plus the rounding of 6 nC angles, which grows with nC R^2.  At 1M cells of unit density the check failed by
// rounding alone on nearly every state and replaced the areas by the triangle fan's, which there are the less
// accurate ones (1e-5 each: the fan's cosines cancel) and took 2.1 ms of a 3.4 ms step.  The limit is therefore
// 2^-53 R^2 an angle where that is above 1e-6: for nC R^2 above 1.5e9, which at unit density is 137,000
// cells; below, it is the reference's.  It is an empirical limit, not a bound (roundings that all erred one way,
// an ulp of the angle and more each, would pass it): sheets of 20k to 1M cells in steps at T = 0.01 and of up to
// 900 times the unit density's area sum to 0 to 0.07 of it as a rule and to 0.45 at most, and a turn of one
// angle is pi R^2 or more, nine orders above.
__host__ __device__ inline double mixed_area_limit(int nC, double R) {
    const double rounding = 6.0 * nC * R * R * 0x1p-53;
    return rounding > 1e-6 ? rounding : 1e-6;
}

// Spherical coordinates of a point as the reference's gradients compute them
// (sphericalDomain.h:218-232, 251-261): cos t = z/|p|, sin t = sqrt(1 - cos^2 t),
// cos p = x / sqrt(x^2+y^2), sin p = y / sqrt(x^2+y^2).
template <bool kHw = false, bool kHwMul = kHw>
__device__ __forceinline__ double4_32a sph_coords_n(D3 p, double r) {  // r = pos_norm(p)
    double cosT = f64_div<kHw>(p.z, r);
    double sinT = f64_sqrt<kHw>(1. - cosT * cosT);
    const double rxy2 = kHwMul ? __dadd_rn(__dmul_rn(p.x, p.x), __dmul_rn(p.y, p.y)) : __dadd_rn(sf::sqr(p.x), sf::sqr(p.y));
    if constexpr (kHw) {
        const double rxy = f64_sqrt<kHw>(rxy2);
        return make_double4_32a(cosT, sinT, f64_div<kHw>(p.x, rxy), f64_div<kHw>(p.y, rxy));
    } else {
        const F64Divisor rxy = f64_root_divisor(rxy2);
        return make_double4_32a(cosT, sinT, f64_div(p.x, rxy), f64_div(p.y, rxy));
    }
}
template <bool kHw = false, bool kHwMul = kHw>
__device__ __forceinline__ double4_32a sph_coords(D3 p) { return sph_coords_n<kHw, kHwMul>(p, pos_norm<kHw, kHwMul>(p)); }

// The gradients' products on the integer pipes, out of line: some sixty to a slot, whose inlined code
// (56 KB for the Brownian force kernel) did not fit the instruction caches.
template <bool kHwMul = false>
__device__ __forceinline__ double grad_mul(double x, double y) {
    if constexpr (kHwMul) return __dmul_rn(x, y);
    else return sf::mul_call(x, y);
}

// The terms of a pair of points (a, b), in spherical coordinates, that the gradients at a of both
// gradientGeodesicDistance (sphericalDomain.h:248-273) and gradientTriangleArea (347-411) evaluate:
// sin(phi_a - phi_b), s = cos of the arc, d = its derivative by theta_a, s s and s s - 1.  A pair is
// evaluated once and serves its edge and both triangles it is a side of.
struct PairTerms { double sP, s, d, ss, q; };
template <bool kHwMul = false>
__device__ __forceinline__ PairTerms pair_terms(const double4_32a& a, const double4_32a& b) {
    const auto E = [](double x, double y) { return grad_mul<kHwMul>(x, y); };
    PairTerms p;
    p.sP = E(a.w, b.z) - E(a.z, b.w);
    const double cP = E(a.z, b.z) + E(a.w, b.w);
    p.s = E(a.x, b.x) + E(E(cP, a.y), b.y);
    p.d = E(E(a.x, cP), b.y) - E(b.x, a.y);
    p.ss = E(p.s, p.s);
    p.q = -1. + p.ss;
    return p;
}
// cos of the arc between b and c alone (the third side of a triangle at a)
template <bool kHwMul = false>
__device__ __forceinline__ double pair_cos(const double4_32a& b, const double4_32a& c) {
    const auto E = [](double x, double y) { return grad_mul<kHwMul>(x, y); };
    const double cP = E(b.z, c.z) + E(b.w, c.w);
    return E(b.x, c.x) + E(E(cP, b.y), c.y);
}

// gradientGeodesicDistance (sphericalDomain.h:248-273) in the (theta, phi) basis of v1, from the
// pair's terms and sin(theta) of the other point: returns (d/dtheta, d/dphi) components.
template <bool kHwMul = false>
__device__ __forceinline__ double2 grad_geodesic(const PairTerms& p, double sinT2) {
    const double dinv = f64_div_root(1., -p.q);   // 1 - s s = -(s s - 1) exactly
    return make_double2(-p.d * dinv, grad_mul<kHwMul>(sinT2, p.sP) * dinv);
}

// grad_triangle's products that stay on the FP64 pipe, which balances the two: the roots' arguments
// (chains of up to five products, ahead of everything else) and the last scaling.
__device__ __forceinline__ double tri_mul(double x, double y) { return __dmul_rn(x, y); }
// gradientTriangleArea (sphericalDomain.h:347-411) in the (theta, phi) basis of v1 for the triangle
// (v1, v2, v3), without the sign of det(v1, v2, v3), from the terms of the pairs (v1, v2) and
// (v1, v3), s23 = pair_cos(v2, v3) and sin(theta) of v2 and v3.  Returns (d/dtheta, d/dphi)
// components.  Every product and sum rounds as the reference's expressions evaluate them (left to
// right, products first); equal subexpressions, and those that differ by an exact sign or a power
// of two, are evaluated once.  Each denominator is a square root and divides two numerators: its
// reciprocal comes with the root (f64_root_divisor) and serves both.
template <bool kHwMul = false>
__device__ __forceinline__ double2 grad_triangle(const PairTerms& p12, const PairTerms& p13, double s23, double sinT2,
                                                 double sinT3, double R) {
    const auto M = tri_mul;
    const auto E = [](double x, double y) { return grad_mul<kHwMul>(x, y); };
    const double s12s13 = E(p12.s, p13.s);
    // 2 s12 s13 s23 = 2 ((s12 s13) s23): the factor two is exact wherever it is applied
    const double g = ((-p12.q - p13.ss) - M(s23, s23)) + sf::twice(M(s12s13, s23));
    const F64Divisor den1 = f64_root_divisor(M(M(p12.q, p12.q), g));
    const F64Divisor den2 = f64_root_divisor(M(M(p13.q, p13.q), g));
    const F64Divisor den3 = f64_root_divisor(M(M(M(M(p12.q, p13.q), p12.q), p13.q), g));
    const double t = s23 - s12s13, u = p13.s - E(p12.s, s23), w = p12.s - E(p13.s, s23);
    // the d/dtheta numerators are formed while the square roots of the denominators run: integer pipes
    const double d12q13 = E(p12.d, p13.q), d13q12 = E(p13.d, p12.q);
    double gT = f64_div(d13q12 + E(p12.d, t), den1) + f64_div(d12q13 + E(p13.d, t), den2)
              - f64_div(E(d12q13, u) + E(d13q12, w), den3);
    gT = M(gT, R);
    double gP = f64_div(-E(E(t, p12.sP), sinT2) - E(E(p12.q, p13.sP), sinT3), den1)
              - f64_div(E(E(p13.q, p12.sP), sinT2) + E(E(t, p13.sP), sinT3), den2)
              + f64_div(E(E(E(p13.q, u), p12.sP), sinT2) + E(E(E(p12.q, w), p13.sP), sinT3), den3);
    gP = M(gP, R);
    return make_double2(gT, gP);
}

// (theta, phi) components to Cartesian with the basis of sphericalDomain.h:218-232:
// thetaHat = (cos t cos p, cos t sin p, -sin t), phiHat = (-sin p, cos p, 0).
__device__ __forceinline__ D3 from_basis(double4_32a s, double2 g) {
    double z = g.x * (-s.y);   // + g.y * 0, which changes it only for an infinite or NaN g.y: to NaN
    if ((((unsigned)__double2hiint(g.y) >> 20) & 0x7ffu) == 0x7ffu) z = __hiloint2double(0x7fffffff, -1);
    return D3{g.x * (s.x * s.z) + g.y * (-s.w), g.x * (s.x * s.w) + g.y * s.z, z};
}

// ---- host-side state -----------------------------------------------------------------------
// Old values of everything one T1 flip overwrites, so a parallel pass can be rolled back.
struct UndoEntry {
    int v1, v2, b, c;              // vertices whose vertex->vertex slots change
    int cells[4];                  // cells i, j, k, l whose rings change
    double4_32a p1, p2;            // old positions of v1, v2
    int4 vc1, vc2;                 // old vertex->cell slots of v1, v2
    int4 vn[4];                    // old vertex->vertex slots of v1, v2, b, c
    int counts[4];                 // old ring sizes
    int logIdx;                    // the flip's entry in the flip log
};

// Counters of one parallel T1 pass: in shared memory for a single-block pass, in global memory
// (T1Scratch::ctl) for a pass spread over a cooperative grid, with the grid barrier's words.
struct T1Ctl {
    int undo, late, rollback, exec, flips, next[2];
    unsigned barCount, barGen;
};
constexpr int kT1CtlInts = sizeof(T1Ctl) / sizeof(int);

struct T1Scratch {
    unsigned* bits = nullptr;      // one bit per (vertex, slot) position, 3*Nv bits
    unsigned* summary = nullptr;   // one bit per word of `bits`: set only for a replay
    int* count = nullptr;          // positions that rolled-back segments left to the replay
    int* segCount = nullptr;       // per segment (the sphere, or each replica): positions the test flagged
    const int* segOff = nullptr;   // first vertex of each segment [segments + 1] (null: one sphere)
    int listPad = 0;               // list slack per segment
    const int* stop = nullptr;     // device flag: while it is set the test flags nothing (a minimisation that has ended)
    int* flipLog = nullptr;        // (pass, position, v1, v2) per flip, capacity flipLogCap
    int* flipCount = nullptr;
    int* pass = nullptr;           // T1 passes so far (orders the flip log across passes)
    int* touched = nullptr;        // cells whose rings changed (batches, and replays)
    int nWords = 0, nSummary = 0, flipLogCap = 0, touchedCap = 0;
    // parallel pass (deterministic reservations), capacity `cap` pending positions
    int* listA = nullptr;          // pending positions of this round (the first: as the test flags them)
    int* listB = nullptr;          // pending positions of the next round
    int* listOrig = nullptr;       // the candidates as flagged by the test (for a rollback)
    int* fp = nullptr;             // footprint of each pending position, kFootprint ints
    int* resV = nullptr;           // per vertex: lowest position reserving it this round
    int* resC = nullptr;           // per cell: same
    int* comV = nullptr;           // per vertex: highest position that has executed on it
    int* comC = nullptr;           // per cell: same
    int* comList = nullptr;        // footprints of executed positions (to clear comV/comC)
    UndoEntry* undo = nullptr;     // one entry per committed flip
    int* undoRings = nullptr;      // old rings of the four cells, 4*Wc ints per entry
    int* ctr = nullptr;            // [5] touched cells, [6] most rounds, [7] blocks finished (batches); then the T1Ctl
    int* stats = nullptr;          // svm_model_t1_stats counters
    unsigned long long* clocks = nullptr;  // svm_model_t1_clocks: SM cycles per phase (null: off)
    T1Ctl* ctl = nullptr;          // counters of a cooperative pass (inside the ctr allocation)
    int cap = 0, undoCap = 0;
};
constexpr int kFootprint = 14;     // 8 vertex slots + 6 cell slots (duplicates allowed)
constexpr int kListPad = 1024;     // list slack of a single-sphere parallel pass
constexpr int kListPadBatch = 64;  // list slack per replica of a batch's parallel pass
constexpr int kResFree = 0x7f7f7f7f;

#ifdef __CUDACC__
// Footprint of the edge (v1, v2): every vertex and cell that testing, flipping and re-testing after
// the flip can read or write (v1, v2 and their neighbours; the cells of v1 and v2).  Two positions
// with disjoint footprints commute.
__device__ __forceinline__ void t1_footprint(int v1, int v2, const int4& n1, const int4& n2, const int4& c1, const int4& c2,
                                             int* f) {
    f[0] = v1; f[1] = v2; f[2] = n1.x; f[3] = n1.y; f[4] = n1.z; f[5] = n2.x; f[6] = n2.y; f[7] = n2.z;
    f[8] = c1.x; f[9] = c1.y; f[10] = c1.z; f[11] = c2.x; f[12] = c2.y; f[13] = c2.z;
}
// Before a T1 pass, by the test kernel (whose own work touches none of it): the touched cells, the most
// rounds, the ticket, and the T1Ctl of a cooperative pass.
__device__ __forceinline__ void t1_clear(const T1Scratch& t1) {
    if (blockIdx.x != 0 || threadIdx.x >= 3 + kT1CtlInts) return;
    t1.ctr[5 + threadIdx.x] = 0;
}
// The T1 test's record of a short edge (position p = 3 v + slot, neighbour u, replica seg): its flag, its
// place in the pass's first list, its footprint, and its reservation of it -- so that the pass starts
// with its first round's reservations made.  Short edges are a few in ten thousand.
inline __device__ __noinline__ void t1_flag(const T1Scratch& t1, int p, int v, int u, int seg, const int4* __restrict__ vnbr,
                                     const int4* __restrict__ vcell) {
    if (t1.stop && *t1.stop) return;
    const unsigned bit = 1u << (p & 31);
    if (atomicOr(&t1.bits[p >> 5], bit) & bit) return;   // listed by an earlier test whose pass did not run
    const int lo = t1.segOff ? 3 * t1.segOff[seg] : 0;
    const int i = atomicAdd(t1.segCount + seg, 1);
    const int at = lo / 2 + t1.listPad * seg + i;
    // (a segment's slice holds one position per edge and more: the bounds only guard a broken state)
    if (at >= t1.cap || (t1.segOff && i >= 3 * (t1.segOff[seg + 1] - t1.segOff[seg]) / 2 + t1.listPad)) return;
    t1.listA[at] = p;
    int* f = t1.fp + (long)at * kFootprint;
    t1_footprint(v, u, vnbr[v], vnbr[u], vcell[v], vcell[u], f);
    for (int k = 0; k < 8; ++k) atomicMin(t1.resV + f[k], p);
    for (int k = 8; k < kFootprint; ++k) atomicMin(t1.resC + f[k], p);
}
#endif

}  // namespace svm

struct svm_model {
    int nCells = 0, nVertices = 0, Wc = 0;
    // Ring capacity grows as the reference's growCellVerticesList widens its ring storage: the T1
    // commits keep the largest ring count in ringMax, every T1 pass copies it to the page-locked
    // ringMaxHost, and before a pass the host grows the capacity whenever ringHeadroom or fewer
    // slots are free in the largest ring.  passEv: the ends of the last two passes launched outside
    // a capture (the host waits for the older before the next pass, so its reading is recent).
    int* ringMax = nullptr;            // device
    int* ringMaxHost = nullptr;        // page-locked, mapped
    int* ringMaxHostDev = nullptr;     // its device address
    int ringHeadroom = 2;
    int ringGrowths = 0;
    cudaEvent_t passEv[2] = {nullptr, nullptr};
    int passSlot = 0;
    bool passChecks = true;            // false: the caller checks the headroom itself, between groups of passes
    double R = 1.0, Kr = 1.0, t1Threshold = 0.1;
    bool restricted = false;
    bool ownStream = false;
    cudaStream_t stream = nullptr;
    int cur = 0;                       // index of the current position buffer
    bool cornersValid = false;         // corner/vsph arrays match the current state
    int t1Blocks = 0;                  // svm_model_set_t1_blocks (0: automatic)
    int t1WaitLimit = 1 << 20;         // polls of a cooperative T1 pass's grid-barrier wait
    double4_32a* pos[2] = {nullptr, nullptr};
    double4_32a* vsph = nullptr;
    double* vnorm = nullptr;           // |p| per vertex, from the last corner pass (FP64 form)
    double4_32a* dir = nullptr;        // directors (self-propelled updater; single spheres only)
    double4_32a* dirTarget = nullptr;  // the Vicsek updater's target directors (allocated on first use)
    double4_32a* cellRef = nullptr;    // reference cell positions of the dynamical observables
    double4_32a* edgeC = nullptr;      // per owned edge slot 3v+j (v < u): p_v x p_u and its norm
    double* edgeArc = nullptr;         // and the arc (FP64 corner pass; single spheres only)
    int4 *vcell = nullptr, *vnbr = nullptr, *vlast = nullptr, *vnext = nullptr, *vrpos = nullptr;
    int* ring = nullptr;
    int* ringCount = nullptr;
    double2* corner = nullptr;
    double4_32a* cellPos = nullptr;
    double4_32a* cellSph = nullptr;
    double2* ap = nullptr;
    double2* pref = nullptr;
    double4_32a* force = nullptr;
    double4_32a* vel = nullptr;
    // mixed-precision form (SVM_PRECISION_MIXED): FP32 positions, centroids and forces
    int precision = SVM_PRECISION_FP64;
    float4* pos32[2] = {nullptr, nullptr};
    float4* cellPos32 = nullptr;
    float4* force32 = nullptr;
    float2* dap32 = nullptr;           // per cell (A - A0, P - P0) in FP32, written with the geometry
    // replicas (mixed form): per-replica radius, noise amplitude and reductions.  A single sphere
    // is one replica; vertex v of replica r has pos32[v].w = r, replica r owns cells
    // [repCellOff[r], repCellOff[r+1]) and vertices [repVertOff[r], repVertOff[r+1]).
    int nRep = 1;
    double* repR = nullptr;            // device [nRep]
    float* repNp = nullptr;            // device [nRep], sqrt(2 dt mu T_r) of the batch's last step
    int* repCellOff = nullptr;         // device [nRep + 1]
    int* repVertOff = nullptr;         // device [nRep + 1]
    int* repFlag = nullptr;            // device [nRep], area-check fallback flags
    int* repList = nullptr;            // device [1 + nRep]: how many of a batch's replicas failed the check, which
    double* repScal = nullptr;         // device [3 nRep]: total area, excess, energy
    std::vector<double> repT;          // host, per-replica temperatures of a batch
    std::vector<int> hRepCellOff, hRepVertOff;
    double repNpDt = -1, repNpMu = -1; // (dt, mu) repNp was computed for
    unsigned repTVersion = 0, repNpVersion = ~0u;
    // block sizes of the batch's per-element kernels (picked by the autotuner)
    int blkCorners = 256, blkCells = 256, blkForce = 256;
    void* tuners = nullptr;            // svm::BatchTuners when autotuning is on
    // FIRE minimizers created on this model; destroying the model detaches them
    std::vector<svm_fire*> fires;
    double* noiseBuf = nullptr;        // [3*Nv] staging for host-supplied noise / displacements
    double* dispBuf = nullptr;         // [3*Nv]
    double* ioHostOut = nullptr;       // while a host-buffer step is issued: the caller's mapped output
                                       // positions (AoS), written by the force kernel and the T1 patch
    // reductions: per-block partials + ticket (last-block-done pattern)
    double* partials = nullptr;
    double* dotPartials = nullptr;     // svm_reduce_dots: 4 per block of 64 vertices (allocated on first use)
    unsigned* ticket = nullptr;
    double* scalars = nullptr;         // [0] total area, [1] excess, [2] energy ...
    int* fallbackFlag = nullptr;
    int* status = nullptr;             // SVM_DEV_* bits
    unsigned long long* stepCounter = nullptr;
    svm::T1Scratch t1;
    int maxPartialBlocks = 0;
    int sms = 152;                     // SMs of the model's device
    // graph cache for svm_brownian_run
    // captured pairs of steps, one per role of the position buffers at its start (an odd run swaps them)
    struct StepGraph {
        cudaGraphExec_t exec = nullptr;
        double T = 0, dt = 0, mu = 0;
        uint64_t seed = 0;
        unsigned version = ~0u;
    } bdGraph[2];
    cudaEvent_t runEv[2] = {nullptr, nullptr};   // svm_brownian_run: ends of the last two chunks
    // per-phase event timing (svm_model_profile)
    bool prof = false;
    int profMask = 0xff;               // phases bracketed by events while profiling (bit per phase)
    std::vector<cudaEvent_t> profEvents[SVM_PHASE_COUNT];   // start/stop pairs, in launch order
    int profUsed[SVM_PHASE_COUNT] = {0};
    double profMs[SVM_PHASE_COUNT] = {0};
    int profLaunches[SVM_PHASE_COUNT] = {0};   // kernel launches (a bracket may hold several)
    std::vector<int> profKernels[SVM_PHASE_COUNT];
    // bumped by every setter whose value a captured graph bakes in (Kr, threshold, restriction)
    unsigned paramsVersion = 0;
    // graph cache for svm_brownian_step_io with pinned host buffers, one per position-buffer role
    struct IoGraph {
        cudaGraphExec_t exec = nullptr;
        double T = 0, dt = 0, mu = 0;
        uint64_t seed = 0;
        const void *in = nullptr, *out = nullptr;
        const void* outDev = nullptr;   // the output's mapped device address the kernels write, or null
        unsigned version = ~0u;
        int precision = -1;
    } ioGraph[2];
    double* ioEnergy = nullptr;        // page-locked landing slot of the graph's energy copy
};

namespace svm {
// Brackets one phase launch with profiling events when profiling is on and the stream is not
// being captured.
struct PhaseTimer {
    svm_model* m;
    int phase;
    bool on;       // profiling on: the phase's launches are counted
    bool timed;    // and bracketed by events (the phase is in the profile mask)
    PhaseTimer(svm_model* m_, int phase_, int kernels = 1);
    ~PhaseTimer();
};
#ifdef __CUDACC__
// The kernels of a step may be launched with programmatic stream serialisation: a kernel's blocks are set
// up while the previous kernel's last blocks still run, and wait for it (its completion and its writes)
// in step_begin, which every such kernel calls before anything else.  It then lets the next kernel's
// blocks be set up in turn.  A kernel launched the ordinary way waits for the previous one's completion
// as always, and step_begin does nothing in it.
// It hides part of the gap between short kernels: 200 cells 52.4 -> 50.8 us a graph-replayed step, 5k
// cells 91.7 -> 89.7; 20k-cell Vicsek steps, launched one by one, 195 -> 176 us.  Blocks that wait early
// cost a graph of longer kernels more than that (20k cells: FIRE iteration 121 -> 128 us, step 139.5 ->
// 142.3), so larger models launch the ordinary way: from 20,000 vertices in a captured graph, whose
// launches follow one another closely anyway, from 100,000 otherwise.
inline bool early_launch(const svm_model* m) {
    if (m->nVertices < 20000) return true;
    cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone;
    return m->nVertices < 100000 && cudaStreamIsCapturing(m->stream, &st) == cudaSuccess && st == cudaStreamCaptureStatusNone;
}
__device__ __forceinline__ void step_begin() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
template <class... Params, class... Args>
inline void launch_next_with(const svm_model* m, void (*kernel)(Params...), int grid, int cluster, int block, int smem,
                             Args&&... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = m->stream;
    cudaLaunchAttribute attr[2];
    int n = 0;
    if (early_launch(m)) {
        attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[n++].val.programmaticStreamSerializationAllowed = 1;
    }
    if (cluster > 1) {
        attr[n].id = cudaLaunchAttributeClusterDimension;
        attr[n].val.clusterDim.x = cluster;
        attr[n].val.clusterDim.y = attr[n].val.clusterDim.z = 1;
        ++n;
    }
    cfg.attrs = attr;
    cfg.numAttrs = n;
    // (an error stays with the runtime for check_launch)
    (void)cudaLaunchKernelEx(&cfg, kernel, static_cast<Params>(args)...);
}
template <class... Params, class... Args>
inline void launch_next_smem(const svm_model* m, void (*kernel)(Params...), int grid, int block, int smem, Args&&... args) {
    launch_next_with(m, kernel, grid, 1, block, smem, static_cast<Args&&>(args)...);
}
// One cluster or more of `cluster` blocks each.
template <class... Params, class... Args>
inline void launch_next_cluster(const svm_model* m, void (*kernel)(Params...), int grid, int cluster, int block, Args&&... args) {
    launch_next_with(m, kernel, grid, cluster, block, 0, static_cast<Args&&>(args)...);
}
template <class... Params, class... Args>
inline void launch_next(const svm_model* m, void (*kernel)(Params...), int grid, int block, Args&&... args) {
    launch_next_smem(m, kernel, grid, block, 0, static_cast<Args&&>(args)...);
}
#endif
// launch helpers shared across translation units (svm_model.cu)
int launch_geometry(svm_model* m);
// vnormReady: the kernel that last moved every vertex also wrote its norm (pos_norm) to m->vnorm, so
// the corner pass skips k_vnorm.
int launch_corners(svm_model* m, bool t1test, bool vnormReady = false);
int launch_t1_apply(svm_model* m, int bump);
int grow_rings(svm_model* m, int newCapacity);
// Threads per block for a one-thread-per-item FP64 kernel over n items: the largest of 256, 128, 64
// and 32 that still gives every SM four blocks (or 32).  An SM's FP64 pipe -- one warp instruction
// per 16 clocks -- is kept busy by a few warps, so a small grid goes over all SMs in small blocks
// rather than over some of them in full ones.
inline int spread_block(const svm_model* m, long n) {
    int bs = 256;
    while (bs > 32 && n < 4L * m->sms * bs) bs >>= 1;
    return bs;
}
// Small models' corner and force kernels take the hardware multiply in place of sf::mul (the same bits):
// they wait on the chain of a thread's operations, not on the FP64 pipe, and the hardware's is the shorter.
// A step, soft / hardware: 200 cells 40.6 / 35.1 us (force phase 20.8 / 18.0, corners 13.1 / 12.6), 1000
// 55.6 / 50.0, 5000 70.6 / 70.4.  The line lies where three models on three streams, whose work adds up on the pipe,
// are even; 8 steps: 150 cells 122 / 108 us, 1000 150 / 143, 1500 166 / 166, 2000 183 / 189, 5000 256 / 298.
constexpr int kFewHwMul = 3000;   // vertices
inline bool few_hw_mul(const svm_model* m) { return m->nVertices < kFewHwMul; }
int ensure_ring_headroom(svm_model* m);
int check_launch();
void fire_detach(svm_fire* F);          // svm_fire.cu: the model is going away
int model_alloc(int nCells, int nVertices, int Wc, const double* radius, int nRep, void* stream, svm_model** out);
// replicas (svm_batch.cu)
int launch_rep_check(svm_model* m);
int update_rep_noise(svm_model* m, double dt, double mu);
void batch_release(svm_model* m);
int batch_tuned_corners(svm_model* m, bool t1test);
int batch_tuned_cells(svm_model* m, int (*launch)(svm_model*));
int batch_tuned_force_bd(svm_model* m, double T, double dt, double mu, int noiseMode, const double* noise,
                         uint64_t seed, int nxt);
bool batch_tuning(svm_model* m);
int mixed_max_block_corners();
int mixed_max_block_force();
int max_block_cells_batch();
void batch_tuner_untimed(svm_model* m, int calls);
// FP64 force kernels (svm_force_kernels.cu)
int zig_init();  // the device's normal-sampling table (svm_force_kernels.cu), before the first Brownian step
int launch_force_fp64(svm_model* m);
int launch_force_bd_fp64(svm_model* m, double np, double fp, int noiseMode, const double* noise, uint64_t seed,
                         int nxt);
// mixed-precision kernels (svm_mixed.cu)
int mixed_launch_corners(svm_model* m, bool t1test);
int mixed_launch_force(svm_model* m);
int mixed_launch_force_bd(svm_model* m, double T, double dt, double mu, int noiseMode, const double* noise,
                          uint64_t seed, int nxt);
int mixed_launch_move(svm_model* m, const double* disp, double scale);
int mixed_upload_positions(svm_model* m, const double* deviceAos);
int mixed_download(svm_model* m, const float4* src, int n, double* deviceAos);
}  // namespace svm
