// The initial topology on the device: the convex hull of the cell centres (a spherical Delaunay
// triangulation) and the vertex-model arrays built from it, with the contract of svm_hull.h
// (convexHullCGAL.cpp:82-186: one vertex per facet at the normalised centroid, CCW facet corners,
// neighbours across facet edges, clockwise rings) and the same canonical numbering, so the result
// equals svm_topology_from_points array for array.
//
// A hull built point by point instead of by incremental insertion:
//   k_hb_*        the centres sorted into bins (counts, a scan, each bin's centres in ascending index)
//   k_hull_star   a warp per centre p.  Candidates are the centres in the bins within w of p's
//                 bin (a ball of radius w h around p lies inside them).  The nearest candidate q0
//                 spans a hull edge (for points on a sphere, the plane through p and q0 with
//                 normal p + q0 has every other point strictly below it).  Gift wrapping around p
//                 from the edge p -> q0: the next corner s of edge p -> q is the candidate that no
//                 other candidate lies above, found by the lanes' scans and a tree over them with
//                 the test "orient(p, q, s, x) > 0", the lower candidate kept in a tie, until the
//                 wrap returns to q0.  Each triangle of the star is then certified: its
//                 circumcircle's cap (the part of the sphere above its plane, smaller than a
//                 hemisphere) lies within 2 rho of p, rho the triangle's circumradius, so when
//                 2 rho < w h every point that could lie in the cap was a candidate and the
//                 triangle is a hull facet.  A star with an uncertified triangle is computed
//                 again with w + 1 (in a second launch over the centres that need it).  A closed
//                 cycle of hull facets around p is p's whole star.
//   k_hull_check  every triangle of a star appears, rotated, in the stars of its other two corners
//                 (the stars form one triangulated sphere), and counts the triangles whose
//                 smallest corner is the star's own point.
//   (scan)        facet offsets: the facets of the smallest corner a are numbered in (b, c) order
//                 after those of smaller a -- the lexicographic order of the host builder.
//   k_hull_emit   writes each point's facets (a, b, c), sorted by (b, c).
//   k_hull_vertex per facet: position (radius / |c|) c with c = (p_a + p_b + p_c) / 3 summed and
//                 scaled as convexHullCGAL.cpp:118-127, cells, and the facets across its edges.
//   k_hull_ring   per cell: its facets clockwise from the lowest-numbered one.
// The orientation test is the host hull's: the FP64 determinant with a relative filter, and a
// double-double evaluation where the filter cannot decide (the host uses long double there).
#include <algorithm>
#include <cmath>
#include "svm_internal.cuh"
#include "svm_hull.h"

using namespace svm;

namespace {
constexpr int kHB = 128;          // threads per block of the star kernel: four centres
constexpr int kFewCand = 128;     // candidates of a star in the first launch (about 70 at w = 1)
constexpr int kMaxCand = 512;     // candidates a star may draw on
constexpr int kMaxDeg = 32;       // facets around one centre
constexpr int kMaxW = 4;          // widest search, in bins
constexpr int kB = 256;
constexpr int kOutside = 16;      // error bit: a centre outside the bins' grid, or not finite

struct DD { double hi, lo; };

__device__ __forceinline__ DD two_sum(double a, double b) {
    const double s = a + b, bb = s - a;
    return {s, (a - (s - bb)) + (b - bb)};
}
__device__ __forceinline__ DD quick_two_sum(double a, double b) {
    const double s = a + b;
    return {s, b - (s - a)};
}
__device__ __forceinline__ DD dd_add(DD a, DD b) {
    const DD s = two_sum(a.hi, b.hi);
    return quick_two_sum(s.hi, s.lo + a.lo + b.lo);
}
__device__ __forceinline__ DD dd_neg(DD a) { return {-a.hi, -a.lo}; }
__device__ __forceinline__ DD dd_mul(DD a, DD b) {
    const double p = a.hi * b.hi;
    double e = fma(a.hi, b.hi, -p);
    e += a.hi * b.lo + a.lo * b.hi;
    return quick_two_sum(p, e);
}
__device__ __forceinline__ DD dd_diff(double a, double b) { return two_sum(a, -b); }  // a - b, exactly

__device__ double orient_dd(const double* A, const double* B, const double* C, const double* D) {
    DD b[3], c[3], d[3];
    for (int k = 0; k < 3; ++k) { b[k] = dd_diff(B[k], A[k]); c[k] = dd_diff(C[k], A[k]); d[k] = dd_diff(D[k], A[k]); }
    const DD nx = dd_add(dd_mul(b[1], c[2]), dd_neg(dd_mul(b[2], c[1])));
    const DD ny = dd_add(dd_mul(b[2], c[0]), dd_neg(dd_mul(b[0], c[2])));
    const DD nz = dd_add(dd_mul(b[0], c[1]), dd_neg(dd_mul(b[1], c[0])));
    const DD det = dd_add(dd_add(dd_mul(nx, d[0]), dd_mul(ny, d[1])), dd_mul(nz, d[2]));
    return det.hi + det.lo;
}

// Positive when D lies on the side the normal (B - A) x (C - A) points to; the FP64 value and
// filter of the host hull's orient.
__device__ double orient(const double* A, const double* B, const double* C, const double* D) {
    const double bx = B[0] - A[0], by = B[1] - A[1], bz = B[2] - A[2];
    const double cx = C[0] - A[0], cy = C[1] - A[1], cz = C[2] - A[2];
    const double dx = D[0] - A[0], dy = D[1] - A[1], dz = D[2] - A[2];
    const double nx = by * cz - bz * cy, ny = bz * cx - bx * cz, nz = bx * cy - by * cx;
    const double det = nx * dx + ny * dy + nz * dz;
    const double perm = (fabs(by * cz) + fabs(bz * cy)) * fabs(dx) + (fabs(bz * cx) + fabs(bx * cz)) * fabs(dy) +
                        (fabs(bx * cy) + fabs(by * cx)) * fabs(dz);
    if (fabs(det) > 1e-13 * perm) return det;
    return orient_dd(A, B, C, D);
}

__device__ __forceinline__ void load3(const double* P, int i, double* o) {
    o[0] = P[3 * i]; o[1] = P[3 * i + 1]; o[2] = P[3 * i + 2];
}

// The cap above the plane of (p, q, s) lies within `reach` of p.
__device__ bool cap_within(const double* p, const double* q, const double* s, double reach) {
    double a[3], b[3], ab[3];
    for (int k = 0; k < 3; ++k) { a[k] = q[k] - p[k]; b[k] = s[k] - p[k]; ab[k] = a[k] - b[k]; }
    const double nx = a[1] * b[2] - a[2] * b[1], ny = a[2] * b[0] - a[0] * b[2], nz = a[0] * b[1] - a[1] * b[0];
    if (nx * p[0] + ny * p[1] + nz * p[2] <= 0.0) return false;  // cap not smaller than a hemisphere
    const double la = sqrt(a[0] * a[0] + a[1] * a[1] + a[2] * a[2]);
    const double lb = sqrt(b[0] * b[0] + b[1] * b[1] + b[2] * b[2]);
    const double lab = sqrt(ab[0] * ab[0] + ab[1] * ab[1] + ab[2] * ab[2]);
    const double ln = sqrt(nx * nx + ny * ny + nz * nz);
    const double diameter = la * lb * lab / ln;  // twice the circumradius
    return diameter * (1.0 + 1e-9) < reach;
}

// The plane of (p, q, s) for the pivot's FP32 sign test: n = b x c with b = q - p, c = s - p in
// FP32, and the coefficients of the filter's permanent (|b1 c2| + |b2 c1|, ...).
struct Plane32 { float n[3], k[3]; };
__device__ __forceinline__ Plane32 plane32(const float* b, const float* c) {
    Plane32 t;
    t.n[0] = b[1] * c[2] - b[2] * c[1]; t.n[1] = b[2] * c[0] - b[0] * c[2]; t.n[2] = b[0] * c[1] - b[1] * c[0];
    t.k[0] = fabsf(b[1] * c[2]) + fabsf(b[2] * c[1]);
    t.k[1] = fabsf(b[2] * c[0]) + fabsf(b[0] * c[2]);
    t.k[2] = fabsf(b[0] * c[1]) + fabsf(b[1] * c[0]);
    return t;
}

// FP32 form of cap_within for the triangle (p, p + a, p + b), n p's offset from the centre: 1 or 0 where a
// margin of 1e-3 makes it certain (FP32 is good to 1e-5 for triangles this far from flat), else -1.
__device__ __forceinline__ int cap_within32(const float* p, const float* a, const float* b, float reach) {
    const float nx = a[1] * b[2] - a[2] * b[1], ny = a[2] * b[0] - a[0] * b[2], nz = a[0] * b[1] - a[1] * b[0];
    const float la = sqrtf(a[0] * a[0] + a[1] * a[1] + a[2] * a[2]), lb = sqrtf(b[0] * b[0] + b[1] * b[1] + b[2] * b[2]);
    const float c0 = a[0] - b[0], c1 = a[1] - b[1], c2 = a[2] - b[2], lab = sqrtf(c0 * c0 + c1 * c1 + c2 * c2);
    const float ln = sqrtf(nx * nx + ny * ny + nz * nz), lp = sqrtf(p[0] * p[0] + p[1] * p[1] + p[2] * p[2]);
    const float up = nx * p[0] + ny * p[1] + nz * p[2];
    if (!(ln > 0.02f * la * lb && lab > 0.02f * (la + lb) && fabsf(up) > 0.1f * ln * lp && la * lb > 1e-12f)) return -1;
    if (up < 0.f) return 0;
    const float diameter = la * lb * lab / ln;
    return diameter * 1.001f < reach ? 1 : (diameter * 0.999f > reach ? 0 : -1);
}

// The bins: centres list[off[bin] .. off[bin + 1]) of bin x + y nside + z nside^2, side h over
// [-radius, radius]^3.
struct BinGrid {
    const int* off;
    const int* list;
    int nside;
    double h, radius;
};

// Centres list[0..*count) (all n centres when list is null), a warp each, with searches of wFirst..wLast
// bins and at most kCap candidates.  A centre whose stars all fail certification in that range, or that
// has more candidates, is queued in retry (when given) for a second launch with the wider searches and
// kMaxCand candidates, so that warps of the first launch do not wait on them.
// What bounds it: issue slots and shared memory (about 1,700 FP32 instructions a warp to pivot six times
// over 70 candidates); the FP64 pipe holds only the offsets x - p.  One centre per thread, candidates in
// local memory: 4.5 ms at 100k centres.  Seven and six blocks an SM: the whole build at 100k centres 1.30 -> 1.18
// ms, 1M 10.8 -> 9.4 (93 registers, five blocks, before; eight blocks 1.20, ten 1.29).
template <int kCap>
__global__ void __launch_bounds__(kHB, kCap == kFewCand ? 7 : 6) k_hull_star(const double* __restrict__ P, const int* __restrict__ list,
                                                  const int* __restrict__ countPtr, int n, int wFirst, int wLast, BinGrid g,
                                                  int* __restrict__ deg, int* __restrict__ star,
                                                  int* __restrict__ retry, int* __restrict__ retryCount,
                                                  int* __restrict__ err) {
    constexpr int kWarps = kHB / 32;
    constexpr unsigned kAll = 0xffffffffu;
    __shared__ float dvS[kWarps][kCap][3];   // offsets from p, fl32(x - p) of the FP64 difference
    __shared__ int candS[kWarps][kCap];
    __shared__ int stS[kWarps][kMaxDeg];     // the star, as candidate indices
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    float (*dv)[3] = dvS[warp];
    int* cand = candS[warp];
    int* st = stS[warp];
    const int count = list ? *countPtr : n;
    for (int t = blockIdx.x * kWarps + warp; t < count; t += gridDim.x * kWarps) {
        // (a queued centre: as ~p if it had too many candidates, else its first search cannot be certified)
        const int entry = list ? list[t] : t, p = entry < 0 ? ~entry : entry;
        double pp[3];
        load3(P, p, pp);
        const float p32[3] = {(float)pp[0], (float)pp[1], (float)pp[2]};
        int c[3];
        for (int d = 0; d < 3; ++d) c[d] = max(0, min(g.nside - 1, (int)floor((pp[d] + g.radius) / g.h)));
        bool hard = false, done = false, full = false;  // hard: a failure no wider search can repair
        for (int w = list && entry >= 0 ? wFirst + 1 : wFirst; w <= wLast && !done && !hard; ++w) {
            int lo[3], ext[3];
            bool whole = true;
            for (int d = 0; d < 3; ++d) {
                lo[d] = max(0, c[d] - w);
                ext[d] = min(g.nside - 1, c[d] + w) - lo[d] + 1;
                whole &= ext[d] == g.nside;
            }
            // candidates in the order of the bins (x fastest) and of each bin's list
            const int nb = ext[0] * ext[1] * ext[2];
            int nc = 0;
            __syncwarp();
            for (int b0 = 0; b0 < nb; b0 += 32) {
                const int b = b0 + lane;
                int first = 0, m = 0;
                if (b < nb) {
                    const int x = lo[0] + b % ext[0], y = lo[1] + (b / ext[0]) % ext[1], z = lo[2] + b / (ext[0] * ext[1]);
                    const long cell = x + (long)y * g.nside + (long)z * g.nside * g.nside;
                    first = g.off[cell];
                    m = g.off[cell + 1] - first;
                }
                int incl = m;
                for (int o = 1; o < 32; o <<= 1) {
                    const int v = __shfl_up_sync(kAll, incl, o);
                    if (lane >= o) incl += v;
                }
                const int excl = incl - m, total = __shfl_sync(kAll, incl, 31);
                for (int k0 = 0; k0 < total; k0 += 32) {
                    const int k = k0 + lane;
                    int owner = 0;  // the last lane whose bin starts at or before k
                    for (int step = 16; step > 0; step >>= 1) {
                        const int e = __shfl_sync(kAll, excl, owner + step);
                        if (e <= k) owner += step;
                    }
                    const int slot = k - __shfl_sync(kAll, excl, owner), from = __shfl_sync(kAll, first, owner);
                    const int j = k < total ? g.list[from + slot] : p;
                    const bool valid = j != p;
                    const unsigned mask = __ballot_sync(kAll, valid);
                    const int at = nc + __popc(mask & ((1u << lane) - 1u));
                    if (valid && at < kCap) {
                        double xx[3];
                        load3(P, j, xx);
                        cand[at] = j;
                        dv[at][0] = (float)(xx[0] - pp[0]);
                        dv[at][1] = (float)(xx[1] - pp[1]);
                        dv[at][2] = (float)(xx[2] - pp[2]);
                    }
                    nc += __popc(mask);
                }
            }
            __syncwarp();
            if (nc > kCap) { if (kCap == kMaxCand) hard = true; full = true; break; }
            if (nc < 3) { if (whole) hard = true; continue; }
            // the nearest in FP32 (squared length within 5 2^-24 relative of the exact one); a near tie: the
            // FP64 squared lengths of those near it, lowest index on ties
            float b1 = INFINITY;
            for (int i = lane; i < nc; i += 32) b1 = fminf(b1, dv[i][0] * dv[i][0] + dv[i][1] * dv[i][1] + dv[i][2] * dv[i][2]);
            for (int o = 16; o > 0; o >>= 1) b1 = fminf(b1, __shfl_xor_sync(kAll, b1, o));
            int iq0 = kCap, near = 0;
            for (int i = lane; i < nc; i += 32) {
                const float d2 = dv[i][0] * dv[i][0] + dv[i][1] * dv[i][1] + dv[i][2] * dv[i][2];
                if (!(d2 > b1 * (1.0f + 1e-5f))) {
                    ++near;
                    if (d2 == b1) iq0 = min(iq0, i);
                }
            }
            near = __reduce_add_sync(kAll, near);
            iq0 = __reduce_min_sync(kAll, iq0);
            if (near != 1) {
                double best = INFINITY;
                int bi = -1;
                for (int i = lane; i < nc; i += 32) {
                    if (dv[i][0] * dv[i][0] + dv[i][1] * dv[i][1] + dv[i][2] * dv[i][2] > b1 * (1.0f + 1e-5f)) continue;
                    double xx[3];
                    load3(P, cand[i], xx);
                    const double dx = xx[0] - pp[0], dy = xx[1] - pp[1], dz = xx[2] - pp[2];
                    const double d2 = dx * dx + dy * dy + dz * dz;
                    if (bi < 0 || d2 < best || (d2 == best && cand[i] < cand[bi])) { best = d2; bi = i; }
                }
                for (int o = 16; o > 0; o >>= 1) {
                    const double ob = __shfl_xor_sync(kAll, best, o);
                    const int oi = __shfl_xor_sync(kAll, bi, o);
                    if (oi >= 0 && (bi < 0 || ob < best || (ob == best && cand[oi] < cand[bi]))) { best = ob; bi = oi; }
                }
                iq0 = __shfl_sync(kAll, bi, 0);   // (none at worst)
            }
            if (iq0 < 0 || iq0 >= nc) { hard = true; break; }
            // gift wrapping around p from the edge to the nearest candidate.  The pivot's sign test runs in
            // FP32: with every input within 2^-24 relative, |det32 - det| <= 8 2^-24 perm, so |det32| > 1e-5
            // perm32 fixes the sign; anything closer (or so small that FP32 could underflow) takes the FP64
            // test.
            int d = 0, iq = iq0;
            bool ok = true;
            do {
                if (d >= kMaxDeg) { ok = false; break; }
                if (lane == 0) st[d] = iq;
                ++d;
                const float b[3] = {dv[iq][0], dv[iq][1], dv[iq][2]};
                // whether candidate x lies above the plane of (p, q, s)
                const auto above = [&](const Plane32& pl, int s, int x) {
                    const float det = pl.n[0] * dv[x][0] + pl.n[1] * dv[x][1] + pl.n[2] * dv[x][2];
                    const float perm = pl.k[0] * fabsf(dv[x][0]) + pl.k[1] * fabsf(dv[x][1]) + pl.k[2] * fabsf(dv[x][2]);
                    if (perm > 1e-30f && fabsf(det) > 1e-5f * perm) return det > 0.f;
                    double qq[3], ss[3], xx[3];
                    load3(P, cand[iq], qq); load3(P, cand[s], ss); load3(P, cand[x], xx);
                    return orient(pp, qq, ss, xx) > 0.0;
                };
                int is = -1;
                Plane32 pl;
                for (int i = lane; i < nc; i += 32) {
                    if (i == iq) continue;
                    if (is < 0 || above(pl, is, i)) { is = i; pl = plane32(b, dv[i]); }
                }
                for (int o = 16; o > 0; o >>= 1) {
                    const int other = __shfl_xor_sync(kAll, is, o);
                    if (other < 0 || other == is) continue;
                    if (is < 0) { is = other; continue; }
                    const int s = min(is, other), x = max(is, other);
                    is = above(plane32(b, dv[s]), s, x) ? x : s;
                }
                is = __shfl_sync(kAll, is, 0);
                if (is < 0) { ok = false; break; }
                iq = is;
            } while (iq != iq0);
            __syncwarp();
            if (ok && d < 3) ok = false;
            if (ok && !whole) {
                const double reach = w * g.h;
                bool in = true;
                if (lane < d) {
                    const int i1 = st[lane], i2 = st[lane + 1 < d ? lane + 1 : 0];
                    const int r = cap_within32(p32, dv[i1], dv[i2], (float)reach);
                    in = r > 0;
                    if (r < 0) {
                        double a[3], b[3];
                        load3(P, cand[i1], a);
                        load3(P, cand[i2], b);
                        in = cap_within(pp, a, b, reach);
                    }
                }
                ok = __all_sync(kAll, in);
            }
            if (ok) {
                if (lane == 0) deg[p] = d;
                if (lane < d) star[(long)p * kMaxDeg + lane] = cand[st[lane]];
                done = true;
            } else if (whole) {
                hard = true;
            }
        }
        if (!done && lane == 0) {
            deg[p] = 0;
            if (retry && !hard) retry[atomicAdd(retryCount, 1)] = full ? ~p : p;
            else atomicOr(err, 1);
        }
    }
}

// Bins: the count of each, then (after the scan of the counts) each centre at a provisional place of
// its bin, then at its rank in the bin.
__device__ __forceinline__ int hb_bin(const double* P, int i, int nside, double h, double radius) {
    int b[3];
    for (int d = 0; d < 3; ++d) b[d] = max(0, min(nside - 1, (int)floor((P[3 * (long)i + d] + radius) / h)));
    return b[0] + b[1] * nside + b[2] * nside * nside;
}
__global__ void k_hb_count(const double* __restrict__ P, int n, int nside, double h, double radius, int* __restrict__ binOf,
                           int* __restrict__ off, int* __restrict__ err) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    for (int d = 0; d < 3; ++d)
        if (!(fabs(P[3 * (long)i + d]) <= radius)) atomicOr(err, kOutside);
    const int b = hb_bin(P, i, nside, h, radius);
    binOf[i] = b;
    atomicAdd(off + b, 1);
}
__global__ void k_hb_place(const int* __restrict__ binOf, int n, const int* __restrict__ off, int* __restrict__ cursor,
                           int* __restrict__ tmp) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int b = binOf[i];
    tmp[off[b] + atomicAdd(cursor + b, 1)] = i;
}
__global__ void k_hb_order(const int* __restrict__ binOf, int n, const int* __restrict__ off, const int* __restrict__ tmp,
                           int* __restrict__ list) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int b = binOf[i], first = off[b], last = off[b + 1];
    int rank = 0;
    for (int k = first; k < last; ++k) rank += tmp[k] < i;
    list[first + rank] = i;
}

__device__ __forceinline__ int star_next(const int* star, const int* deg, int a, int b) {
    // in a's star, the corner after b (-1 if b is not a neighbour of a)
    const int da = deg[a];
    const int* s = star + (long)a * kMaxDeg;
    for (int i = 0; i < da; ++i)
        if (s[i] == b) return s[i + 1 < da ? i + 1 : 0];
    return -1;
}

__global__ void k_hull_check(const int* __restrict__ star, const int* __restrict__ deg, int n,
                             int* __restrict__ own, int* __restrict__ err) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= n) return;
    const int d = deg[p];
    const int* s = star + (long)p * kMaxDeg;
    int count = 0;
    bool ok = d >= 3;
    for (int i = 0; i < d && ok; ++i) {
        const int a = s[i], b = s[i + 1 < d ? i + 1 : 0];
        ok = star_next(star, deg, a, b) == p && star_next(star, deg, b, p) == a;
        count += p < a && p < b;
    }
    own[p] = count;
    if (!ok) atomicOr(err, 2);
}

__global__ void k_hull_emit(const int* __restrict__ star, const int* __restrict__ deg, int n,
                            const int* __restrict__ off, int* __restrict__ F) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= n) return;
    const int d = deg[p];
    const int* s = star + (long)p * kMaxDeg;
    int b[kMaxDeg], c[kMaxDeg], m = 0;
    for (int i = 0; i < d; ++i) {
        const int u = s[i], v = s[i + 1 < d ? i + 1 : 0];
        if (p < u && p < v) {
            int k = m++;
            while (k > 0 && (b[k - 1] > u || (b[k - 1] == u && c[k - 1] > v))) { b[k] = b[k - 1]; c[k] = c[k - 1]; --k; }
            b[k] = u; c[k] = v;
        }
    }
    const int o = off[p];
    for (int k = 0; k < m; ++k) { F[3 * (o + k)] = p; F[3 * (o + k) + 1] = b[k]; F[3 * (o + k) + 2] = c[k]; }
}

// Index of the facet with corners u, v, w (CCW), in canonical numbering.
__device__ int facet_of(int u, int v, int w, const int* off, const int* F) {
    int a = u, b = v, c = w;
    if (v < u && v < w) { a = v; b = w; c = u; }
    else if (w < u && w < v) { a = w; b = u; c = v; }
    for (int k = off[a]; k < off[a + 1]; ++k)
        if (F[3 * k + 1] == b && F[3 * k + 2] == c) return k;
    return -1;
}

__global__ void k_hull_vertex(const double* __restrict__ P, const int* __restrict__ F, int nf,
                              const int* __restrict__ off, const int* __restrict__ star, const int* __restrict__ deg,
                              double radius, double* __restrict__ vpos, int* __restrict__ vcells,
                              int* __restrict__ vnbrs, int* __restrict__ err) {
    const int f = blockIdx.x * blockDim.x + threadIdx.x;
    if (f >= nf) return;
    const int t[3] = {F[3 * f], F[3 * f + 1], F[3 * f + 2]};
    double c[3] = {0.0, 0.0, 0.0};
    for (int k = 0; k < 3; ++k)
        for (int d = 0; d < 3; ++d) c[d] += P[3 * t[k] + d];
    for (int d = 0; d < 3; ++d) c[d] = (1.0 / 3.0) * c[d];
    const double nrm = sqrt(c[0] * c[0] + c[1] * c[1] + c[2] * c[2]);
    for (int d = 0; d < 3; ++d) vpos[3 * (long)f + d] = (radius / nrm) * c[d];
    for (int k = 0; k < 3; ++k) {
        vcells[3 * (long)f + k] = t[k];
        const int from = t[(k + 2) % 3], to = t[k];  // the facet across the edge ending at corner k
        const int x = star_next(star, deg, to, from);
        const int gidx = x < 0 ? -1 : facet_of(to, from, x, off, F);
        if (gidx < 0) atomicOr(err, 4);
        vnbrs[3 * (long)f + k] = gidx;
    }
}

__global__ void k_hull_ring(const int* __restrict__ star, const int* __restrict__ deg, int n,
                            const int* __restrict__ off, const int* __restrict__ F,
                            const int* __restrict__ ringOff, int* __restrict__ ring, int* __restrict__ err) {
    const int x = blockIdx.x * blockDim.x + threadIdx.x;
    if (x >= n) return;
    const int d = deg[x];
    const int* s = star + (long)x * kMaxDeg;
    int gi[kMaxDeg];
    int start = 0;
    for (int i = 0; i < d; ++i) {
        gi[i] = facet_of(x, s[i], s[i + 1 < d ? i + 1 : 0], off, F);
        if (gi[i] < 0) atomicOr(err, 8);
        if (gi[i] < gi[start]) start = i;
    }
    const int o = ringOff[x];
    for (int j = 0; j < d; ++j) ring[o + j] = gi[(start - j + d) % d];  // clockwise: decreasing i
}

// Exclusive scan of n ints in place; a block scans 2 kB entries, the block totals are scanned the
// same way, then added back.
__global__ void k_scan_block(int* a, int n, int* sums) {
    __shared__ int sh[2 * kB];
    const int base = blockIdx.x * 2 * kB;
    const int i0 = base + threadIdx.x, i1 = base + kB + threadIdx.x;
    sh[threadIdx.x] = i0 < n ? a[i0] : 0;
    sh[kB + threadIdx.x] = i1 < n ? a[i1] : 0;
    __syncthreads();
    for (int o = 1; o < 2 * kB; o <<= 1) {  // Hillis-Steele over the block's 2 kB entries
        int v0 = 0, v1 = 0;
        if (threadIdx.x >= o) v0 = sh[threadIdx.x - o];
        if (kB + threadIdx.x >= o) v1 = sh[kB + threadIdx.x - o];
        __syncthreads();
        sh[threadIdx.x] += v0;
        sh[kB + threadIdx.x] += v1;
        __syncthreads();
    }
    const int e0 = threadIdx.x == 0 ? 0 : sh[threadIdx.x - 1];
    const int e1 = sh[kB + threadIdx.x - 1];
    if (i0 < n) a[i0] = e0;
    if (i1 < n) a[i1] = e1;
    if (threadIdx.x == 0) sums[blockIdx.x] = sh[2 * kB - 1];
}
__global__ void k_scan_add(int* a, int n, const int* sums) {
    const int i = blockIdx.x * 2 * kB + threadIdx.x;
    const int add = sums[blockIdx.x];
    if (i < n) a[i] += add;
    if (i + kB < n) a[i + kB] += add;
}

// (sums: scan_ints(n) ints of workspace)
size_t scan_ints(size_t n) {
    const size_t nb = (n + 2 * kB - 1) / (2 * kB);
    return nb + 1 + (nb > 1 ? scan_ints(nb) : 0);
}
int exclusive_scan(int* a, int n, cudaStream_t s, int* sums) {
    const int nb = (n + 2 * kB - 1) / (2 * kB);
    k_scan_block<<<nb, kB, 0, s>>>(a, n, sums);
    int rc = check_launch();
    if (!rc && nb > 1) rc = exclusive_scan(sums, nb, s, sums + nb + 1);
    else if (!rc) rc = cudaMemsetAsync(sums, 0, sizeof(int), s) == cudaSuccess ? SVM_OK : SVM_ERR_CUDA;
    if (!rc) { k_scan_add<<<nb, kB, 0, s>>>(a, n, sums); rc = check_launch(); }
    return rc;
}

// Each cell's ring in a row of `stride` (-1 past its end), with the counts.
__global__ void k_hull_rows(const int* __restrict__ ringOff, const int* __restrict__ ring, int n, int stride,
                            int* __restrict__ rows) {
    const long e = blockIdx.x * (long)blockDim.x + threadIdx.x;
    if (e >= (long)n * stride) return;
    const int c = (int)(e / stride), k = (int)(e % stride), b = ringOff[c], m = ringOff[c + 1] - b;
    rows[e] = k < m ? ring[b + k] : -1;
}
__global__ void k_hull_max(const int* __restrict__ deg, int n, int* __restrict__ maxDeg) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int m = __reduce_max_sync(0xffffffffu, i < n ? deg[i] : 0);
    if ((threadIdx.x & 31) == 0) atomicMax(maxDeg, m);
}

// One device allocation cut into 256-byte aligned arrays.
struct Arena {
    char* base = nullptr;
    size_t used = 0;
    template <typename T> T* cut(size_t count) {   // with base null: counts the bytes
        T* p = reinterpret_cast<T*>(base + used);
        used += (sizeof(T) * std::max<size_t>(count, 1) + 255) & ~(size_t)255;
        return p;
    }
};
}  // namespace

// The arrays stay on the device, where they were computed, until svm_topology_get copies them straight
// into the caller's; the workspace they were computed with is given back when the build returns.
// Fetching and freeing them take no part in what other threads have under way: the copies run on a stream of
// the handle's own, which the default stream's work and captures do not order, and the thread's calls are not
// counted among those that another thread's capture forbids.
namespace {
struct OutsideCaptures {
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    OutsideCaptures() { cudaThreadExchangeStreamCaptureMode(&mode); }
    ~OutsideCaptures() { cudaThreadExchangeStreamCaptureMode(&mode); }
};
}  // namespace
struct svm::DeviceTopology {
    void* base = nullptr;
    cudaStream_t stream = nullptr;
    const double* vpos = nullptr;
    const int *vcells = nullptr, *vnbrs = nullptr, *rows = nullptr, *deg = nullptr;
    ~DeviceTopology() {
        OutsideCaptures guard;
        cudaFree(base);
        if (stream) cudaStreamDestroy(stream);
    }
};
svm_topology::~svm_topology() { delete dev; }

namespace svm {
// svm_topology_get of a device-built topology.
int device_topology_get(const svm_topology* t, double* vp, int* rings, int stride, unsigned* counts, int* vc, int* vn) {
    const DeviceTopology& D = *t->dev;
    const size_t nC = t->t.nCells, nV = t->t.nVertices, W = t->t.maxRing;
    OutsideCaptures guard;
    const auto copy = [&](void* dst, const void* src, size_t bytes) {
        return cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, D.stream) == cudaSuccess;
    };
    bool ok = (!vp || copy(vp, D.vpos, sizeof(double) * 3 * nV)) && (!vc || copy(vc, D.vcells, sizeof(int) * 3 * nV)) &&
              (!vn || copy(vn, D.vnbrs, sizeof(int) * 3 * nV)) && (!counts || copy(counts, D.deg, sizeof(int) * nC)) &&
              (!rings || copy(rings, D.rows, sizeof(int) * nC * W));
    ok = cudaStreamSynchronize(D.stream) == cudaSuccess && ok;
    if (ok && rings && (size_t)stride > W)   // wider rows than the rings need: spread them, the last first
        for (size_t c = nC; c-- > 0;)
            for (size_t k = stride; k-- > 0;) rings[c * stride + k] = k < W ? rings[c * W + k] : -1;
    return ok ? SVM_OK : SVM_ERR_CUDA;
}
}  // namespace svm

extern "C" int svm_topology_from_points_gpu(const double* pts, int n, void* stream, svm_topology** out) {
    if (!pts || n < 4 || !out) return SVM_ERR_ARG;
    cudaStream_t s = (cudaStream_t)stream;
    // bins of side 2.5 mean spacings (a unit-density sphere has ~70 candidates at w = 1)
    double r2 = 0.0;
    for (int i = 0; i < n; ++i)
        r2 = std::max(r2, pts[3 * i] * pts[3 * i] + pts[3 * i + 1] * pts[3 * i + 1] + pts[3 * i + 2] * pts[3 * i + 2]);
    const double rmax = std::sqrt(r2);
    const double gridR = rmax * (1.0 + 1e-6) + 1e-3;
    const double spacing = std::sqrt(4.0 * 3.141592653589793 * rmax * rmax / n);
    const double side = std::min(2.5 * spacing, gridR);
    if (!(side > 0) || !std::isfinite(gridR)) return SVM_ERR_ARG;
    BinGrid g;
    g.nside = (int)std::floor(2.0 * gridR / side);
    g.nside -= g.nside % 2;
    if (g.nside < 1 || g.nside > 1024) return SVM_ERR_ARG;
    g.h = 2.0 * gridR / g.nside;
    g.radius = gridR;
    const size_t bins = (size_t)g.nside * g.nside * g.nside, nf = 2 * (size_t)n - 4;
    // the workspace, one allocation
    Arena A;
    double* P;
    int *deg, *star, *own, *ctl, *retry, *F, *ringOff, *ring, *off, *cursor, *binOf, *list, *tmp, *sums;
    const auto lay = [&] {
        A.used = 0;
        deg = A.cut<int>(n);
        star = A.cut<int>((size_t)n * kMaxDeg);
        P = A.cut<double>(3 * (size_t)n);
        own = A.cut<int>((size_t)n + 1); retry = A.cut<int>(n); F = A.cut<int>(3 * nf);
        ringOff = A.cut<int>((size_t)n + 1); ring = A.cut<int>(3 * nf);
        binOf = A.cut<int>(n); list = A.cut<int>(n); tmp = A.cut<int>(n);
        sums = A.cut<int>(scan_ints(std::max(bins + 1, (size_t)n + 1)));
        ctl = A.cut<int>(4);   // [0] error bits, [1] centres queued for the wider search, [2] largest ring
        off = A.cut<int>(bins + 1); cursor = A.cut<int>(bins);   // (cleared together, to the end)
    };
    lay();
    const size_t bytes = A.used;
    svm_topology* t = new svm_topology();
    t->dev = new DeviceTopology();
    if (cudaStreamCreateWithFlags(&t->dev->stream, cudaStreamNonBlocking) != cudaSuccess ||
        cudaMalloc((void**)&A.base, bytes) != cudaSuccess) {
        cudaGetLastError();
        delete t;
        return SVM_ERR_CUDA;
    }
    lay();
    const auto fail = [&](int rc) { cudaStreamSynchronize(s); cudaFree(A.base); delete t; return rc; };
    if (cudaMemcpyAsync(P, pts, sizeof(double) * 3 * n, cudaMemcpyHostToDevice, s) != cudaSuccess ||
        cudaMemsetAsync(ctl, 0, (char*)A.base + bytes - (char*)ctl, s) != cudaSuccess ||
        cudaMemsetAsync(own + n, 0, sizeof(int), s) != cudaSuccess)
        return fail(SVM_ERR_CUDA);
    const int nb = (n + kB - 1) / kB;
    k_hb_count<<<nb, kB, 0, s>>>(P, n, g.nside, g.h, g.radius, binOf, off, ctl);
    if (check_launch() || exclusive_scan(off, (int)bins + 1, s, sums)) return fail(SVM_ERR_CUDA);
    k_hb_place<<<nb, kB, 0, s>>>(binOf, n, off, cursor, tmp);
    k_hb_order<<<nb, kB, 0, s>>>(binOf, n, off, tmp, list);
    g.off = off;
    g.list = list;
    const int warps = kHB / 32;
    k_hull_star<kFewCand><<<(n + warps - 1) / warps, kHB, 0, s>>>(P, nullptr, nullptr, n, 1, 1, g, deg, star, retry, ctl + 1, ctl);
    // the queued centres, however many there are (their count stays on the device): six blocks per SM
    k_hull_star<kMaxCand><<<std::min((n + warps - 1) / warps, 6 * 152), kHB, 0, s>>>(P, retry, ctl + 1, n, 1, kMaxW, g, deg,
                                                                                   star, nullptr, nullptr, ctl);
    k_hull_check<<<nb, kB, 0, s>>>(star, deg, n, own, ctl);
    if (check_launch() || exclusive_scan(own, n + 1, s, sums)) return fail(SVM_ERR_CUDA);
    // the stars have to close into one triangulated sphere before facets are numbered from them
    k_hull_max<<<nb, kB, 0, s>>>(deg, n, ctl + 2);
    // what svm_topology_get copies, in an allocation of its own: made while the device works, with rows for rings of up
    // to kKeptRow
    constexpr int kKeptRow = 16;
    double* vpos;
    int *vcells, *vnbrs, *counts, *rows;
    const auto keep = [&](int row) {
        Arena K;
        const auto cut = [&] {
            K.used = 0;
            vpos = K.cut<double>(3 * nf);
            vcells = K.cut<int>(3 * nf); vnbrs = K.cut<int>(3 * nf); counts = K.cut<int>(n);
            rows = K.cut<int>((size_t)n * row);
        };
        cut();
        cudaFree(t->dev->base);
        t->dev->base = nullptr;
        if (cudaMalloc(&t->dev->base, K.used) != cudaSuccess) { cudaGetLastError(); return false; }
        K.base = (char*)t->dev->base;
        cut();
        return true;
    };
    if (check_launch() || !keep(kKeptRow)) return fail(SVM_ERR_CUDA);
    int got[3], facets = 0;
    if (cudaMemcpyAsync(got, ctl, sizeof(got), cudaMemcpyDeviceToHost, s) != cudaSuccess ||
        cudaMemcpyAsync(&facets, own + n, sizeof(int), cudaMemcpyDeviceToHost, s) != cudaSuccess ||
        cudaStreamSynchronize(s) != cudaSuccess)
        return fail(SVM_ERR_CUDA);
    if (got[0] & kOutside) return fail(SVM_ERR_DEVICE);
    if (got[0] || (size_t)facets != nf) return fail(SVM_ERR_HULL);
    const int W = got[2];
    if (W > kKeptRow && !keep(W)) return fail(SVM_ERR_CUDA);
    const double radius = std::sqrt(pts[0] * pts[0] + pts[1] * pts[1] + pts[2] * pts[2]);
    k_hull_emit<<<nb, kB, 0, s>>>(star, deg, n, own, F);
    k_hull_vertex<<<((int)nf + kB - 1) / kB, kB, 0, s>>>(P, F, (int)nf, own, star, deg, radius, vpos, vcells, vnbrs, ctl);
    if (check_launch() || cudaMemcpyAsync(counts, deg, sizeof(int) * n, cudaMemcpyDeviceToDevice, s) != cudaSuccess ||
        cudaMemcpyAsync(ringOff, deg, sizeof(int) * n, cudaMemcpyDeviceToDevice, s) != cudaSuccess ||
        cudaMemsetAsync(ringOff + n, 0, sizeof(int), s) != cudaSuccess || exclusive_scan(ringOff, n + 1, s, sums))
        return fail(SVM_ERR_CUDA);
    // (a triangulated sphere of nf facets has rings of 3 nf entries)
    k_hull_ring<<<nb, kB, 0, s>>>(star, deg, n, own, F, ringOff, ring, ctl);
    k_hull_rows<<<(int)(((long)n * W + kB - 1) / kB), kB, 0, s>>>(ringOff, ring, n, W, rows);
    int e = 0, nr = 0;
    if (check_launch() || cudaMemcpyAsync(&e, ctl, sizeof(int), cudaMemcpyDeviceToHost, s) != cudaSuccess ||
        cudaMemcpyAsync(&nr, ringOff + n, sizeof(int), cudaMemcpyDeviceToHost, s) != cudaSuccess ||
        cudaStreamSynchronize(s) != cudaSuccess)
        return fail(SVM_ERR_CUDA);
    if (e || (size_t)nr != 3 * nf) return fail(SVM_ERR_HULL);
    t->t.nCells = n;
    t->t.nVertices = (int)nf;
    t->t.maxRing = W;
    t->dev->vpos = vpos; t->dev->vcells = vcells; t->dev->vnbrs = vnbrs; t->dev->rows = rows; t->dev->deg = counts;
    cudaFree(A.base);
    *out = t;
    return SVM_OK;
}
