// Per-vertex force of the quadratic spherical vertex model, shared by the Brownian, FIRE and
// plain force kernels.
//
// Restates computeForceCPU (src/model/sphericalVertexModel.cpp:356-420) /
// gpu_quadratic_spherical_cellular_force_kernel (src/model/sphericalVertexModel.cu:141-195):
// for each of the vertex's three cells,
//   fSet = -2 dP [grad d(v,last) + grad d(v,next)] - 2 Kr dA [grad A(v,last,c) + grad A(v,c,next)]
// in the spherical basis at v, skipping a cell whose contribution is NaN.  (last, next) are the
// ring neighbours of v in that cell, c the cell's renormalised centroid.
#pragma once
#include "svm_internal.cuh"

namespace svm {

struct ForceArgs {
    const double4_32a* pos;
    const double4_32a* vsph;
    const int4* vcell;
    const int4* vlast;
    const int4* vnext;
    const double4_32a* cellPos;
    const double4_32a* cellSph;
    const double2* ap;
    const double2* pref;
    double Kr, R;
};

__device__ __forceinline__ int comp(const int4& a, int s) { return s == 0 ? a.x : (s == 1 ? a.y : a.z); }

// The force form of a kernel (the closed forms of the reference, or SVM_PRECISION_FP64_VECTOR's exact gradient as
// vectors: grad_geo_vec, grad_tri_vec), fixed at compile time, which lets each drop the other's registers.
constexpr int kFormVector = 1, kFormReference = 2;

// Block-level force of kVerts vertices by six threads a vertex: thread (role, vi, s) with s one of the
// vertex's three cell slots and a role per triangle of the slot's fan.  Role 0 holds the slot's ring
// predecessor L and the triangle (v, L, c), role 1 the cell's centroid c and the triangle (v, c, X), X
// the successor.  Each thread first evaluates its point's terms -- every neighbour of v is the
// predecessor in one of its cells, so the six threads cover the vertex's six pairs once -- and then,
// with the other's through shared memory, its triangle.  The roles are whole warps.
//
// What bounds it: at large N the FP64 pipe (2 lanes per clock per SM) and the instruction caches; at
// small N one warp's chain of dependent operations, which two threads a slot halve.  Measured for the
// Brownian kernel (k_force_bd) against three threads a vertex, 64 vertices a block, three blocks per SM
// and every product but the chains' first ones on the FP64 pipe:
//   100k cells  265 us -> 266 (six threads) -> 251 (all of the triangle's products but the roots'
//               arguments on the integer pipes, FP64 pipe 67% busy) -> 226 (those products out of
//               line, normals drawn by role 1 beside the edge gradients)
//   20k cells   78 -> 58 us;   200 cells  28.7 -> 20.5 us.
// Also tried at 100k cells: the roots' arguments on the integer pipes too 231 us, the quotients out of
// line too 230, four blocks per SM 240; blocks of 10 vertices at 200 cells 20.3, at 20k cells 72.
constexpr int kSlotVerts = 32;
constexpr int slot_role_threads(int verts) { return (3 * verts + 31) / 32 * 32; }
constexpr int slot_threads(int verts) { return 2 * slot_role_threads(verts); }
// Blocks per SM the slot-force kernels are compiled for (64 registers: 30 warps per SM).
constexpr int kSlotMinBlocks = 5;
template <int kVerts = kSlotVerts>
struct SlotShared {
    double l[7][3 * kVerts];   // predecessor terms: (sin dphi, s, d, s s, s s - 1) or (beta, a x beta, beta^2)
    double c[7][3 * kVerts];   // centroid terms, the same
    double g[3][3 * kVerts];   // edge gradients towards the predecessors, then the slots' forces
    double t[3][3 * kVerts];   // role 1's triangle terms
};

struct SlotIndex { int v, vi, s, at, c, L, X, jx; bool live; };
template <int kVerts>
__device__ __forceinline__ SlotIndex slot_index(const ForceArgs& A, int nV, int k) {
    SlotIndex q;
    q.vi = k / 3; q.s = k - 3 * q.vi; q.at = k;
    q.v = blockIdx.x * kVerts + q.vi;
    q.live = q.vi < kVerts && q.v < nV;
    q.c = q.L = q.X = q.jx = 0;
    if (q.live) {
        const int4 cells = A.vcell[q.v], lasts = A.vlast[q.v], nexts = A.vnext[q.v];
        q.c = comp(cells, q.s); q.L = comp(lasts, q.s); q.X = comp(nexts, q.s);
        // the slot whose predecessor X is (-1: inconsistent lists)
        q.jx = q.X == lasts.x ? 0 : (q.X == lasts.y ? 1 : (q.X == lasts.z ? 2 : -1));
    }
    return q;
}
template <int kVerts>
__device__ __forceinline__ void put_pair(double (*a)[3 * kVerts], int k, const PairTerms& p) {
    a[0][k] = p.sP; a[1][k] = p.s; a[2][k] = p.d; a[3][k] = p.ss; a[4][k] = p.q;
}
template <int kVerts>
__device__ __forceinline__ PairTerms get_pair(const double (*a)[3 * kVerts], int k) {
    return PairTerms{a[0][k], a[1][k], a[2][k], a[3][k], a[4][k]};
}
template <int kVerts>
__device__ __forceinline__ void put3(double (*a)[3 * kVerts], int k, D3 p) { a[0][k] = p.x; a[1][k] = p.y; a[2][k] = p.z; }
template <int kVerts>
__device__ __forceinline__ D3 get3(const double (*a)[3 * kVerts], int k) { return D3{a[0][k], a[1][k], a[2][k]}; }

static __device__ __noinline__ bool det_negative_exact(D3 p, D3 a, D3 b) { return det3(p, a, b) < 0; }
// det(p, a, b) < 0: in FP32 where that is certain (all but nearly flat triangles).
__device__ __forceinline__ bool det_negative(D3 p, D3 a, D3 b) {
    const svm_det::F3 v32 = svm_det::near3(p.x, p.y, p.z);
    const int n = svm_det::below_zero(v32, svm_det::diff(svm_det::near3(a.x, a.y, a.z), v32),
                                      svm_det::diff(svm_det::near3(b.x, b.y, b.z), v32));
    return n >= 0 ? n != 0 : det_negative_exact(p, a, b);
}

// The slot forces of the reference form, left in sh.g for the block: per slot
//   -pp (grad d(v, L) + grad d(v, X)) - aa (grad A(v, L, c) + grad A(v, c, X)), pp = 2 dP, aa = 2 Kr dA,
// each term subtracted in the reference's order.  `side(q)` is work that does not depend on the force: one
// call per slot, by role 1's threads while role 0 evaluates the edge gradients.  Every thread of the block calls it.
template <bool kHwMul, int kVerts, class Side>
__device__ __forceinline__ void slot_forces_reference(const ForceArgs& A, int nV, SlotShared<kVerts>& sh, Side side) {
    constexpr int kRole = slot_role_threads(kVerts);
    const bool role0 = threadIdx.x < kRole;
    const SlotIndex q = slot_index<kVerts>(A, nV, role0 ? threadIdx.x : threadIdx.x - kRole);
    double4_32a sv, s2;   // the spherical coordinates of v and of the thread's own point
    PairTerms own;
    D3 gL;
    if (q.live) {
        sv = A.vsph[q.v];
        s2 = role0 ? A.vsph[q.L] : A.cellSph[q.c];
        own = pair_terms<kHwMul>(sv, s2);
        if (role0) {
            gL = from_basis(sv, grad_geodesic<kHwMul>(own, s2.y));
            put3<kVerts>(sh.g, q.at, gL);
        } else {
            side(q);
        }
        put_pair<kVerts>(role0 ? sh.l : sh.c, q.at, own);
    }
    __syncthreads();
    D3 fs;
    if (q.live) {
        const double2 apc = A.ap[q.c], pr = A.pref[q.c];
        const double aa = 2.0 * A.Kr * (apc.x - pr.x);
        // the triangle's third corner: the centroid (role 0) or the successor (role 1)
        const double4_32a s3 = role0 ? A.cellSph[q.c] : A.vsph[q.X];
        PairTerms other;
        D3 gX;
        const int tx = 3 * q.vi + q.jx;
        if (role0) {
            other = get_pair<kVerts>(sh.c, q.at);
            const double pp = sf::twice(apc.y - pr.y);
            if (q.jx >= 0) gX = get3<kVerts>(sh.g, tx);
            else {
                const double4_32a sx = A.vsph[q.X];
                gX = from_basis(sv, grad_geodesic<kHwMul>(pair_terms<kHwMul>(sv, sx), sx.y));
            }
            fs = sub3(scl3(-pp, gL), scl3(pp, gX));
        } else {
            other = q.jx >= 0 ? get_pair<kVerts>(sh.l, tx) : pair_terms<kHwMul>(sv, s3);
        }
        double2 g = grad_triangle<kHwMul>(own, other, pair_cos<kHwMul>(s2, s3), s2.y, s3.y, A.R);
        const D3 p = ld3(A.pos, q.v), cp = ld3(A.cellPos, q.c), pn = ld3(A.pos, role0 ? q.L : q.X);
        const bool negative = det_negative(p, role0 ? pn : cp, role0 ? cp : pn);
        g = make_double2(sf::negate_if(negative, g.x), sf::negate_if(negative, g.y));
        const D3 t = scl3(aa, from_basis(sv, g));
        if (role0) fs = sub3(fs, t);
        else put3<kVerts>(sh.t, q.at, t);
    }
    __syncthreads();
    if (q.live) {
        if (role0) put3<kVerts>(sh.g, q.at, sub3(fs, get3<kVerts>(sh.t, q.at)));
    }
    __syncthreads();
}

// The vector form (the exact gradient as vectors, well conditioned where the reference's closed
// forms lose digits -- short edges, thin fan triangles), the same way.  Products and sums contract to
// multiply-adds here: the form's values are pinned to its formulas, not to the CPU's sequence of
// roundings.  The products that are not part of a multiply-add run on the integer pipes, which the form
// leaves idle (early_mul; kHwMul: on the FP64 pipe), a third of its FP64 instructions: a FIRE iteration of 20k cells
// 115 -> 105 us, of 100k 391 -> 344.
template <bool kHwMul>
__device__ __forceinline__ double dot3f(D3 a, D3 b) { return fma(a.z, b.z, fma(a.y, b.y, early_mul<kHwMul>(a.x, b.x))); }
template <bool kHwMul>
__device__ __forceinline__ D3 cross3f(D3 a, D3 b) {
    return D3{fma(a.y, b.z, -early_mul<kHwMul>(a.z, b.y)), fma(a.z, b.x, -early_mul<kHwMul>(a.x, b.z)),
              fma(a.x, b.y, -early_mul<kHwMul>(a.y, b.x))};
}
template <bool kHwMul>
__device__ __forceinline__ D3 scl3f(double k, D3 a) {
    return D3{early_mul<kHwMul>(k, a.x), early_mul<kHwMul>(k, a.y), early_mul<kHwMul>(k, a.z)};
}
__device__ __forceinline__ D3 axpy3f(double s, D3 x, D3 y) { return D3{fma(s, x.x, y.x), fma(s, x.y, y.y), fma(s, x.z, y.z)}; }
// Unit tangent at a pointing away from the neighbour at v + d: gradient of the geodesic length
// (any radius), from the raw position difference d.
template <bool kHwMul>
__device__ __forceinline__ D3 grad_geo_vec(D3 a, D3 d) {
    const D3 t = axpy3f(-dot3f<kHwMul>(d, a), a, d);
    return scl3f<kHwMul>(f64_div_root(-1.0, dot3f<kHwMul>(t, t)), t);
}
// scale / 2 times the gradient w.r.t. v = |v| a of the signed spherical triangle area
// R^2 E(a, a + beta, a + gamma), over R and without its projection onto the tangent plane: tan(E/2) = N/D (Van
// Oosterom and Strackee, 1983) differentiated, beta and gamma the raw differences to the other corners over
// |v|, ab = a x beta, ag = a x gamma, and the squares of beta and gamma given.
template <bool kHwMul>
__device__ __forceinline__ D3 grad_tri_vec(D3 a, D3 beta, D3 gamma, D3 ab, D3 ag, double beta2, double gamma2,
                                              double scale) {
    const D3 bg = cross3f<kHwMul>(beta, gamma);
    const D3 bxc = add3(sub3(ag, ab), bg);
    const double N = dot3f<kHwMul>(a, bg);
    const double D = fma(beta.z, gamma.z, fma(beta.y, gamma.y, fma(beta.x, gamma.x, 4.0 - beta2 - gamma2)));
    const double w = f64_div(scale, fma(N, N, early_mul<kHwMul>(D, D)));
    return scl3f<kHwMul>(w, axpy3f(-N, add3(beta, gamma), scl3f<kHwMul>(D, bxc)));
}
template <bool kHwMul, int kVerts, class Side>
__device__ __forceinline__ void slot_forces_vector(const ForceArgs& A, int nV, SlotShared<kVerts>& sh, Side side) {
    constexpr int kRole = slot_role_threads(kVerts);
    const bool role0 = threadIdx.x < kRole;
    const SlotIndex q = slot_index<kVerts>(A, nV, role0 ? threadIdx.x : threadIdx.x - kRole);
    D3 a, b, ab, gL;
    double b2, inv;
    if (q.live) {
        const D3 P = ld3(A.pos, q.v), d = sub3(role0 ? ld3(A.pos, q.L) : ld3(A.cellPos, q.c), P);
        inv = f64_div_root(1.0, dot3f<kHwMul>(P, P));
        a = scl3f<kHwMul>(inv, P);
        b = scl3f<kHwMul>(inv, d);
        ab = cross3f<kHwMul>(a, b);
        b2 = dot3f<kHwMul>(b, b);
        double (*o)[3 * kVerts] = role0 ? sh.l : sh.c;
        put3<kVerts>(o, q.at, b);
        put3<kVerts>(o + 3, q.at, ab);
        o[6][q.at] = b2;
        if (role0) {
            gL = grad_geo_vec<kHwMul>(a, d);
            put3<kVerts>(sh.g, q.at, gL);
        } else {
            side(q);
        }
    }
    __syncthreads();
    D3 fs;
    if (q.live) {
        const double2 apc = A.ap[q.c], pr = A.pref[q.c];
        const double aaR = 2.0 * A.Kr * (apc.x - pr.x) * A.R;
        D3 o, ao, gX;   // the triangle's third corner: the centroid (role 0) or the successor (role 1)
        double o2;
        const int tx = 3 * q.vi + q.jx;
        if (role0 || q.jx >= 0) {
            const double (*p)[3 * kVerts] = role0 ? sh.c : sh.l;
            const int k = role0 ? q.at : tx;
            o = get3<kVerts>(p, k);
            ao = get3<kVerts>(p + 3, k);
            o2 = p[6][k];
        } else {  // inconsistent lists
            o = scl3f<kHwMul>(inv, sub3(ld3(A.pos, q.X), ld3(A.pos, q.v)));
            ao = cross3f<kHwMul>(a, o);
            o2 = dot3f<kHwMul>(o, o);
        }
        const D3 t = grad_tri_vec<kHwMul>(a, b, o, ab, ao, b2, o2, 2.0 * aaR);
        if (role0) {
            const double pp = 2.0 * (apc.y - pr.y);
            gX = q.jx >= 0 ? get3<kVerts>(sh.g, tx) : grad_geo_vec<kHwMul>(a, sub3(ld3(A.pos, q.X), ld3(A.pos, q.v)));
            fs = sub3(scl3f<kHwMul>(-pp, add3(gL, gX)), t);
        } else {
            put3<kVerts>(sh.t, q.at, t);
        }
    }
    __syncthreads();
    if (q.live) {
        if (role0) {   // the slot's sum, projected onto the tangent plane (the edge gradients lie in it)
            const D3 f = sub3(fs, get3<kVerts>(sh.t, q.at));
            put3<kVerts>(sh.g, q.at, axpy3f(-dot3f<kHwMul>(f, a), a, f));
        }
    }
    __syncthreads();
}

// The force of vertex threadIdx.x of the block's kVerts vertices (threads from kVerts on: zero).  The
// slots' contributions are added in slot order, a NaN term skipped, as the reference's loop over the
// three cells does.
template <int kForm, bool kHwMul, int kVerts, class Side>
__device__ __forceinline__ D3 block_slot_force(const ForceArgs& A, int nV, SlotShared<kVerts>& sh, Side side) {
    if (kForm == kFormVector) slot_forces_vector<kHwMul>(A, nV, sh, side);
    else slot_forces_reference<kHwMul>(A, nV, sh, side);
    const int t = threadIdx.x;
    D3 f{0.0, 0.0, 0.0};
    if (t < kVerts && blockIdx.x * kVerts + t < nV) {
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const D3 fq = get3<kVerts>(sh.g, 3 * t + k);
            if (!isnan(fq.x)) f = add3(f, fq);
        }
    }
    return f;
}
struct NoSide { __device__ void operator()(const SlotIndex&) const {} };

// Philox4x32-10 (Salmon, Moraes, Dror, Shaw, "Parallel random numbers: as easy as 1, 2, 3",
// SC'11): ten rounds of two 32x32->64 multiplies with a Weyl-sequence key schedule.
__device__ __forceinline__ uint4 philox4x32_10(uint4 ctr, uint2 key) {
    const unsigned M0 = 0xD2511F53u, M1 = 0xCD9E8D57u, W0 = 0x9E3779B9u, W1 = 0xBB67AE85u;
#pragma unroll
    for (int r = 0; r < 10; ++r) {
        if (r) { key.x += W0; key.y += W1; }
        const unsigned hi0 = __umulhi(M0, ctr.x), lo0 = M0 * ctr.x;
        const unsigned hi1 = __umulhi(M1, ctr.z), lo1 = M1 * ctr.z;
        ctr = make_uint4(hi1 ^ ctr.y ^ key.x, lo1, hi0 ^ ctr.w ^ key.y, lo0);
    }
    return ctr;
}
// 53-bit uniform in (0, 1) from two 32-bit words.
__device__ __forceinline__ double u53(unsigned a, unsigned b) {
    const unsigned long long x = ((unsigned long long)a << 21) ^ (unsigned long long)(b >> 11);
    return ((double)(x & ((1ull << 53) - 1)) + 0.5) * 0x1.0p-53;
}

// Standard normals by the ziggurat method (G. Marsaglia and W. W. Tsang, "The Ziggurat Method for
// Generating Random Variables", J. Stat. Softw. 5(8), 2000) with 256 layers of equal area v under
// f(x) = exp(-x^2/2): layer i >= 1 is the box [0, x_i) x [f(x_i), f(x_{i+1})), layer 0 the box
// [0, v / f(r)) x [0, f(r)) together with the tail beyond r = x_1.  A uniform layer, sign and
// u in [0, 1) give x = u x_i, accepted at once when x < x_{i+1} (98.5% of draws); otherwise layer 0
// samples the tail (Marsaglia's x = -ln(u1) / r, y = -ln(u2), accepted when 2y > x^2) and the other
// layers test the wedge against f(x), starting over on rejection.  The bits: one Philox draw's
// 64-bit halves for the fast path, a fresh draw per retry.
struct ZigTable {
    double x[257];  // x_0 = v / f(r), x_1 = r, ..., x_256 = 0
    double f[257];  // f(x_i) (f_0 unused)
};
constexpr double kZigR = 3.654152885361009;  // r for 256 layers
// Layer, sign and a 53-bit u in [0, 1) from 64 bits.
__device__ __forceinline__ double zig_draw(const ZigTable* __restrict__ Z, unsigned a, unsigned b, int& i, bool& neg) {
    i = (int)(a & 255u);
    neg = (a >> 8) & 1u;
    const unsigned long long n = ((unsigned long long)(a >> 9) << 30) | (unsigned long long)(b >> 2);
    return (double)n * 0x1.0p-53 * __ldg(Z->x + i);
}
static __device__ __noinline__ double zig_slow(const ZigTable* __restrict__ Z, int i, double x, bool neg, uint4 ctr, uint2 key) {
    for (int attempt = 0; attempt < 32; ++attempt) {  // each round fails with probability < 0.02
        ctr.w += 1u;
        const uint4 r = philox4x32_10(ctr, key);
        if (i == 0) {
            const double xt = -log(u53(r.x, r.y)) / kZigR, y = -log(u53(r.z, r.w));
            if (y + y > xt * xt) return neg ? -(kZigR + xt) : kZigR + xt;
            continue;
        }
        const double y = __ldg(Z->f + i) + u53(r.x, r.y) * (__ldg(Z->f + i + 1) - __ldg(Z->f + i));
        // y < exp(-x^2 / 2) in FP32 where that is certain: the FP32 exponential is within 2e-6 of it
        const float xf = svm_det::near32(x), yf = svm_det::near32(y), ef = expf(-0.5f * xf * xf);
        const bool under = fabsf(yf - ef) > 2e-5f * ef ? yf < ef : y < exp(-0.5 * x * x);
        if (under) return sf::negate_if(neg, x);
        x = zig_draw(Z, r.z, r.w, i, neg);
        if (x < __ldg(Z->x + i + 1)) return sf::negate_if(neg, x);
    }
    return sf::negate_if(neg, x);
}
__device__ __forceinline__ double zig_normal(const ZigTable* __restrict__ Z, unsigned a, unsigned b, uint4 ctr, uint2 key) {
    int i;
    bool neg;
    const double x = zig_draw(Z, a, b, i, neg);
    if (x < __ldg(Z->x + i + 1)) return sf::negate_if(neg, x);
    return zig_slow(Z, i, x, neg, ctr, key);
}
// Component k of the three standard normals for (vertex, step): two Philox draws (counter words 0 and 1)
// give the three fast-path draws; normal k retries on counter words 64 (k + 1) + 1, 2, ...
__device__ __forceinline__ double philox_normal(const ZigTable* __restrict__ Z, uint64_t seed, unsigned long long step, int v,
                                                int k) {
    const uint2 key = make_uint2((unsigned)seed, (unsigned)(seed >> 32));
    uint4 c = make_uint4((unsigned)v, (unsigned)step, (unsigned)(step >> 32), k == 2 ? 1u : 0u);
    const uint4 r = philox4x32_10(c, key);
    c.w = 64u * (unsigned)(k + 1);
    return zig_normal(Z, k == 1 ? r.z : r.x, k == 1 ? r.w : r.y, c, key);
}

// disp_d = xi_d sqrt(2 dt mu T) + F_d dt mu (brownianDynamics.cpp:37-44), products rounded
// before the sum as on the CPU.
__device__ __forceinline__ double bd_disp(double xi, double np, double f, double fp) {
    return __dadd_rn(__dmul_rn(xi, np), __dmul_rn(f, fp));
}
// sphericalDomain::move with every product and sum rounded separately (no contraction), so the
// renormalised positions follow the CPU's sequence of roundings.
// kHwMul: its products on the FP64 pipe (k_force_bd, whose force part already fills the integer pipes, and
// small models), or on the integer pipes.
template <bool kHwMul = true>
__device__ __forceinline__ D3 move_exact(D3 p, D3 v, double R) {
    const auto M = [](double x, double y) { return early_mul<kHwMul>(x, y); };
    const double s = f64_div(dot3e<kHwMul>(v, p), norm2e<kHwMul>(p));
    D3 q{__dadd_rn(p.x, __dsub_rn(v.x, M(s, p.x))), __dadd_rn(p.y, __dsub_rn(v.y, M(s, p.y))),
         __dadd_rn(p.z, __dsub_rn(v.z, M(s, p.z)))};
    const double inv = f64_div_root(1.0, norm2e<kHwMul>(q));
    return D3{M(R, M(inv, q.x)), M(R, M(inv, q.y)), M(R, M(inv, q.z))};
}
// a projected onto the tangent plane at p and normalised (projectToTangentPlaneAndNormalize,
// sphericalDomain.h:173-177), every product and sum rounded.
template <bool kHwMul>
__device__ __forceinline__ D3 tangent_unit(D3 a, D3 p) {
    const auto M = [](double x, double y) { return early_mul<kHwMul>(x, y); };
    const double s = f64_div(dot3e<kHwMul>(a, p), norm2e<kHwMul>(p));
    a = D3{__dsub_rn(a.x, M(s, p.x)), __dsub_rn(a.y, M(s, p.y)), __dsub_rn(a.z, M(s, p.z))};
    const double inv = f64_div_root(1.0, norm2e<kHwMul>(a));
    return D3{M(inv, a.x), M(inv, a.y), M(inv, a.z)};
}

inline ForceArgs force_args(svm_model* m, int buf) {
    ForceArgs A;
    A.pos = m->pos[buf]; A.vsph = m->vsph; A.vcell = m->vcell; A.vlast = m->vlast; A.vnext = m->vnext;
    A.cellPos = m->cellPos; A.cellSph = m->cellSph; A.ap = m->ap; A.pref = m->pref; A.Kr = m->Kr; A.R = m->R;
    return A;
}
}  // namespace svm
