// Cell list of points on (or near) the sphere: hyperrectangularCellList on the GPU.
//
// Restates setGridSize and computeCPU of src/utilities/hyperrectangularCellList.cpp:27-51,
// 165-214: a cubic grid over [-r, r]^3 with floor(2r / a) cells per side made even,
// h = 2r / cells, bin_d = floor((x_d + r) / h), flat index x + y n + z n^2
// (inc/indexer.h:170-176).  The reference GPU kernel (hyperrectangularCellList.cu:14-51) fills
// slots in atomic order; here the slots of a bin are put in ascending point index, as the CPU
// loop leaves them, so the table is deterministic.  Kernels:
//   k_cl_clear   zero the counts of the bins the previous call used (not the whole grid), and the
//                call's scalars
//   k_cl_bin     bin each point, take a provisional slot with an atomic; a neighbour list's FP32 copies
//   k_cl_order   rank each point among its bin's entries by index, write the final slot;
//                Nmax = max(Nmax, largest occupancy), the grow-only width of the reference
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <vector>
#include "svm_internal.cuh"

using namespace svm;

struct svm_cell_list {
    double a = 1.0, radius = 1.0, h = 1.0;
    int nside = 0, cap = 0, nPoints = 0;
    long total = 0;
    cudaStream_t stream = nullptr;
    bool ownStream = false;
    unsigned* counts = nullptr;   // [total]
    int* tmp = nullptr;           // [total * cap] provisional slots
    int* slots = nullptr;         // [total * cap] ordered slots
    int* binOf = nullptr;         // [nPoints]
    // [0] max occupancy this call, [1] Nmax (grow-only), [2] overflow, [3] out of grid, [4] the neighbour
    // list's longest row
    int* scalars = nullptr;
    int* hostScalars = nullptr;   // page-locked, what the host reads of them
    bool first = true;
};

namespace {
constexpr int kB = 256;
constexpr int kClScalars = 5;

__device__ __forceinline__ int bin_of(double x, double y, double z, double r, double h, int n, int* bad) {
    const F64Divisor H = kept_divisor(h);   // (the quotients on the integer pipes, the same bits)
    int bx = (int)floor(f64_div(x + r, H)), by = (int)floor(f64_div(y + r, H)), bz = (int)floor(f64_div(z + r, H));
    if (bx < 0 || by < 0 || bz < 0 || bx >= n || by >= n || bz >= n) {
        atomicExch(bad, 1);
        bx = min(max(bx, 0), n - 1); by = min(max(by, 0), n - 1); bz = min(max(bz, 0), n - 1);
    }
    return bx + by * n + bz * n * n;
}

__global__ void k_cl_clear(const int* __restrict__ binOf, unsigned* counts, int np, int* __restrict__ scalars) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < kClScalars && i != 1) scalars[i] = 0;  // (np >= 1: the grid has the threads)
    if (i < np && binOf[i] >= 0) counts[binOf[i]] = 0u;
}

template <typename P>
__global__ void k_cl_bin(P pts, int np, double r, double h, int n, int cap, int* __restrict__ binOf,
                         unsigned* __restrict__ counts, int* __restrict__ tmp, int* __restrict__ scalars,
                         float4* __restrict__ p32) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    int occ = 0;
    if (i < np) {
        double x, y, z;
        pts(i, x, y, z);
        if (p32) p32[i] = make_float4((float)x, (float)y, (float)z, 0.f);
        const int b = bin_of(x, y, z, r, h, n, scalars + 3);
        binOf[i] = b;
        const unsigned s = atomicAdd(counts + b, 1u);
        if ((int)s < cap) tmp[(long)b * cap + s] = i;
        else atomicExch(scalars + 2, 1);
        occ = (int)s + 1;
    }
    // one atomic per warp: a per-point atomic on this one word serialises in L2
    occ = __reduce_max_sync(0xffffffffu, occ);
    if ((threadIdx.x & 31) == 0 && occ > 0) atomicMax(scalars, occ);
}

__global__ void k_cl_order(const int* __restrict__ binOf, const unsigned* __restrict__ counts,
                           const int* __restrict__ tmp, int* __restrict__ slots, int np, int cap, int* __restrict__ scalars) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i == 0) scalars[1] = max(scalars[1], scalars[0]);
    if (i >= np) return;
    const int b = binOf[i];
    const int c = min((int)counts[b], cap);
    const int* t = tmp + (long)b * cap;
    int rank = 0;
    bool present = false;
    for (int k = 0; k < c; ++k) {
        const int j = t[k];
        rank += j < i;
        present |= j == i;
    }
    if (present) slots[(long)b * cap + rank] = i;
}

struct ModelPoints {
    const double4_32a* p;
    __device__ void operator()(int i, double& x, double& y, double& z) const { const double4_32a q = p[i]; x = q.x; y = q.y; z = q.z; }
};
struct ModelPoints32 {
    const float4* p;
    __device__ void operator()(int i, double& x, double& y, double& z) const { const float4 q = p[i]; x = q.x; y = q.y; z = q.z; }
};
struct AosPoints {
    const double* p;
    __device__ void operator()(int i, double& x, double& y, double& z) const { x = p[3 * i]; y = p[3 * i + 1]; z = p[3 * i + 2]; }
};

// A bin took more points than it has slots: give every bin `cap` slots, as the reference's cell
// list widens its Nmax and bins again (hyperrectangularCellList.cpp:165-214).  The counts of the
// overflowing call stay valid for the next call's incremental clear.
// (On failure the list has no slots, and the next call allocates them.)
int cl_grow(svm_cell_list* cl, int cap) {
    if (cudaStreamSynchronize(cl->stream) != cudaSuccess) return SVM_ERR_CUDA;
    const auto release = [&] {
        cudaFree(cl->tmp); cudaFree(cl->slots);
        cl->tmp = nullptr; cl->slots = nullptr;
    };
    release();
    if (cudaMalloc(&cl->tmp, sizeof(int) * cl->total * cap) != cudaSuccess ||
        cudaMalloc(&cl->slots, sizeof(int) * cl->total * cap) != cudaSuccess) {
        release();
        cudaGetLastError();
        return SVM_ERR_CUDA;
    }
    cl->cap = cap;
    return SVM_OK;
}

// `p32`: where to leave FP32 copies of the points, or null
template <typename P>
int compute(svm_cell_list* cl, P pts, int np, float4* p32 = nullptr) {
    if (np != cl->nPoints) return SVM_ERR_ARG;
    if (!cl->slots)
        if (int rc = cl_grow(cl, cl->cap)) return rc;
    const int nb = (np + kB - 1) / kB;
    k_cl_clear<<<nb, kB, 0, cl->stream>>>(cl->binOf, cl->counts, np, cl->scalars);
    k_cl_bin<<<nb, kB, 0, cl->stream>>>(pts, np, cl->radius, cl->h, cl->nside, cl->cap, cl->binOf, cl->counts, cl->tmp,
                                        cl->scalars, p32);
    k_cl_order<<<nb, kB, 0, cl->stream>>>(cl->binOf, cl->counts, cl->tmp, cl->slots, np, cl->cap, cl->scalars);
    return check_launch();
}

// The model's points, ordered after the model's pending work.
int compute_model(svm_cell_list* cl, svm_model* m, float4* p32 = nullptr) {
    if (cl->stream != m->stream) {
        cudaEvent_t e;
        cudaEventCreateWithFlags(&e, cudaEventDisableTiming);
        cudaEventRecord(e, m->stream);
        cudaStreamWaitEvent(cl->stream, e, 0);
        cudaEventDestroy(e);
    }
    if (m->precision == SVM_PRECISION_MIXED) return compute(cl, ModelPoints32{m->pos32[m->cur]}, m->nVertices, p32);
    return compute(cl, ModelPoints{m->pos[m->cur]}, m->nVertices, p32);
}

// This call's scalars, in cl->hostScalars, once the stream has finished.
int read_scalars(svm_cell_list* cl) {
    return cudaMemcpyAsync(cl->hostScalars, cl->scalars, sizeof(int) * kClScalars, cudaMemcpyDeviceToHost, cl->stream) == cudaSuccess &&
                   cudaStreamSynchronize(cl->stream) == cudaSuccess ? SVM_OK : SVM_ERR_CUDA;
}

// neighborList (src/utilities/neighborList.cpp:6-18, 96-151; kernels neighborList.cu:108-357): per
// point, over the adjacent bins of its (clamped) bin in the mask's order and each bin's points in
// slot order, every other point whose minimum-image displacement (periodic box of side 2 radius,
// periodicBoundaryConditions.h:124-132) is shorter than `range`; the first nmax are stored, the
// rest of each row is zero, and the count is kept whole (the host grows nmax and recomputes when a
// count exceeds it).
//
// FP64 issues at a sixty-fourth of the FP32 rate here, so a candidate is first classified in FP32
// and only neighbours (and the rare borderline candidate) see FP64.  kNlLanes threads a point:
//   phase 1: each thread takes kNlBins consecutive bins of the mask and classifies their candidates
//     with FP32 copies of the positions.  With E a bound on |d32 - d64| per component (coordinates
//     within the grid, |x| <= radius, rounded to FP32 and subtracted: E = radius 2^-21 covers both
//     roundings with a factor of two), a candidate whose |d32| components all stay below radius - 2E
//     cannot wrap in FP64, and then
//       dd32 > thrHi (> ((range + 2E)(1 + 2^-20))^2)  => |d64| > range      => not a neighbour
//       dd32 < thrLo (< ((range - 2E)(1 - 2^-20))^2)  => |d64| < range      => a neighbour
//     (dd32's own rounding is below 3 2^-24 relative, inside the 2^-20 factors).  Any other
//     candidate takes the reference's FP64 test.  The point's threads add up their counts in bin
//     order, and each writes its neighbours' indices at its place in the row.
//   phase 2, the block: the rows of its points, an entry a thread: displacement, squared length and
//     root in FP64 exactly as the reference does, or zeros past the row's end.
// What bounds it: phase 1 is a chain of dependent loads (count, slot, position) per candidate, which
// one thread a point walked for all ~25 candidates with 8 warps on an SM; eight threads a point walk
// it for three or four candidates each, with 64 warps' loads in flight.  The call on the device, of
// 39,996 points at two per unit area, range 1: 114 -> 60 us; of 300 points, where launches, clears and
// the read-back of five scalars are all of it (eleven stream operations, now five): 100 -> 37 us.  Longer rows
// are bound by phase 2's FP64, whose roots and the bins' quotients run on the integer pipes: 199,996 vertices
// with rows of 22 214 -> 164 us.
// The minimum-image loops run at most kWrapIters times: points inside the grid need one, and a
// point outside it is an error the host reports (the cell list's flag).
constexpr int kNlLanes = 8;                 // threads a point
constexpr int kNlBins = 4;                  // consecutive bins a thread: 32 a round, the usual mask has 27
constexpr int kNlPoints = kB / kNlLanes;    // points a block
constexpr int kWrapIters = 8;
constexpr unsigned kNlWrapped = 0x80000000u;  // between the phases: the displacement wrapped

struct NlParams {
    int np, cap, nside, K, nmax;
    double radius, range, range2Hi;
    float wrapLim, thrLo, thrHi;
};

__device__ __forceinline__ bool min_image(double& d, double radius) {
    bool w = false;
    for (int i = 0; i < kWrapIters && d < -radius; ++i) { d += 2. * radius; w = true; }
    for (int i = 0; i < kWrapIters && d > radius; ++i) { d -= 2. * radius; w = true; }
    return w;
}

template <typename P>
__global__ void __launch_bounds__(kB, 6) k_nl(P pts, const float4* __restrict__ p32, NlParams prm,
                                          const unsigned* __restrict__ counts, const int* __restrict__ slots,
                                          const int* __restrict__ binOf, const int* __restrict__ mask,
                                          unsigned* __restrict__ npp, int* __restrict__ idx,
                                          double* __restrict__ vec, double* __restrict__ dist,
                                          int* __restrict__ maxCount) {
    __shared__ double own[kNlPoints][3];
    __shared__ int stored[kNlPoints];
    const int sub = threadIdx.x % kNlLanes, row = threadIdx.x / kNlLanes;
    const int p0 = blockIdx.x * kNlPoints, pp = p0 + row;
    const bool active = pp < prm.np;
    float4 t32 = make_float4(0.f, 0.f, 0.f, 0.f);
    int c[3] = {0, 0, 0};
    if (active) {
        t32 = p32[pp];
        const int b = binOf[pp], q = b / prm.nside;  // the (clamped) bin the cell list found
        c[0] = b - q * prm.nside; c[2] = q / prm.nside; c[1] = q - c[2] * prm.nside;
        if (sub == 0) pts(pp, own[row][0], own[row][1], own[row][2]);
    }
    int have = 0;
    for (int k0 = 0; k0 < prm.K; k0 += kNlLanes * kNlBins) {
        // this thread's bins: their first slots and, running, the candidates up to each one's end
        long first[kNlBins];
        int end[kNlBins], n[kNlBins];
#pragma unroll
        for (int i = 0; i < kNlBins; ++i) {
            const int k = k0 + sub * kNlBins + i;
            first[i] = 0;
            n[i] = 0;
            if (active && k < prm.K) {
                int nb[3];
                for (int d = 0; d < 3; ++d) {
                    nb[d] = c[d] + mask[3 * k + d];
                    // the mask's offsets may exceed the grid's side (few bins): the true remainder then
                    if (nb[d] < 0 || nb[d] >= prm.nside) {
                        nb[d] %= prm.nside;
                        if (nb[d] < 0) nb[d] += prm.nside;
                    }
                }
                const long cell = nb[0] + (long)nb[1] * prm.nside + (long)nb[2] * prm.nside * prm.nside;
                first[i] = cell * prm.cap;
                n[i] = min((int)counts[cell], prm.cap);
            }
        }
        int total = 0;
#pragma unroll
        for (int i = 0; i < kNlBins; ++i) {
            first[i] -= total;
            total += n[i];
            end[i] = total;
        }
        const auto candidate = [&](int t) {
            long at = first[0];
#pragma unroll
            for (int i = 1; i < kNlBins; ++i)
                if (t >= end[i - 1]) at = first[i];
            return slots[at + t];
        };
        // the neighbours among candidates [t0, t0 + 32), and which of them wrapped
        const auto classify = [&](int t0, unsigned& yes, unsigned& wrapped) {
            const int m = min(32, total - t0);
            unsigned open = 0;
            yes = wrapped = 0;
#pragma unroll 4
            for (int t = 0; t < m; ++t) {
                const int j = candidate(t0 + t);
                const float4 q = p32[j];
                const float d0 = t32.x - q.x, d1 = t32.y - q.y, d2 = t32.z - q.z;
                const bool inside = fabsf(d0) <= prm.wrapLim && fabsf(d1) <= prm.wrapLim && fabsf(d2) <= prm.wrapLim;
                const float dd32 = d0 * d0 + d1 * d1 + d2 * d2;
                const bool no = (inside && dd32 > prm.thrHi) || j == pp, is = inside && dd32 < prm.thrLo && !no;
                yes |= (unsigned)is << t;
                open |= (unsigned)(!is && !no) << t;
            }
            while (open) {  // the reference's test, in FP64 (rare: the points are reloaded)
                const int t = __ffs(open) - 1;
                open &= open - 1;
                double a[3], b[3], disp[3];
                pts(pp, a[0], a[1], a[2]);
                pts(candidate(t0 + t), b[0], b[1], b[2]);
                bool w = false;
                for (int d = 0; d < 3; ++d) {
                    disp[d] = a[d] - b[d];
                    w |= min_image(disp[d], prm.radius);
                }
                const double dd = disp[0] * disp[0] + disp[1] * disp[1] + disp[2] * disp[2];
                if (dd > prm.range2Hi || sqrt(dd) >= prm.range) continue;
                yes |= 1u << t;
                if (w) wrapped |= 1u << t;
            }
        };
        // counts first (a thread past 32 candidates classifies the later ones twice), then the places
        unsigned yes, wrapped;
        classify(0, yes, wrapped);
        int cnt = __popc(yes);
        for (int t0 = 32; t0 < total; t0 += 32) {
            unsigned y, w;
            classify(t0, y, w);
            cnt += __popc(y);
        }
        __syncwarp();
        int incl = cnt;
#pragma unroll
        for (int o = 1; o < kNlLanes; o <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, incl, o, kNlLanes);
            if (sub >= o) incl += v;
        }
        int at = have + incl - cnt;
        have += __shfl_sync(0xffffffffu, incl, kNlLanes - 1, kNlLanes);
        for (int t0 = 0; t0 < total && at < prm.nmax; t0 += 32) {
            if (t0) classify(t0, yes, wrapped);
            for (; yes && at < prm.nmax; yes &= yes - 1, ++at) {
                const int t = __ffs(yes) - 1;
                idx[(long)pp * prm.nmax + at] = (int)((unsigned)candidate(t0 + t) | (wrapped >> t & 1 ? kNlWrapped : 0u));
            }
        }
        __syncwarp();
    }
    if (sub == 0) {
        stored[row] = min(have, prm.nmax);
        if (active) npp[pp] = (unsigned)have;
    }
    const int most = __reduce_max_sync(0xffffffffu, have);  // one atomic per warp on the shared word
    if ((threadIdx.x & 31) == 0 && most > 0) atomicMax(maxCount, most);
    __syncthreads();
    // ---- phase 2, with the rest of each row zero (resetNeighbors)
    const long entries = (long)min(kNlPoints, prm.np - p0) * prm.nmax;
    for (long e = threadIdx.x; e < entries; e += kB) {
        const int o = (int)(e / prm.nmax), k = (int)(e - (long)o * prm.nmax);
        const long at = (long)p0 * prm.nmax + e;
        int j = 0;
        double disp[3] = {0., 0., 0.}, len = 0.;
        if (k < stored[o]) {
            j = idx[at];
            const bool w = j < 0;
            j &= (int)~kNlWrapped;
            double b[3];
            pts(j, b[0], b[1], b[2]);
            for (int d = 0; d < 3; ++d) disp[d] = own[o][d] - b[d];
            if (w)
                for (int d = 0; d < 3; ++d) min_image(disp[d], prm.radius);
            len = f64_sqrt(disp[0] * disp[0] + disp[1] * disp[1] + disp[2] * disp[2]);
        }
        idx[at] = j;
        vec[3 * at] = disp[0]; vec[3 * at + 1] = disp[1]; vec[3 * at + 2] = disp[2];
        dist[at] = len;
    }
}
}  // namespace

struct svm_neighbor_list {
    svm_cell_list* cl = nullptr;
    double range = 1.0, radius = 1.0;
    int nPoints = 0, nmax = 4, K = 0;   // Nmax starts at 4 (neighborList.cpp:17)
    int* mask = nullptr;                // [3 K] adjacent-bin offsets
    unsigned* npp = nullptr;            // [nPoints]
    int* idx = nullptr;                 // [nPoints * nmax]
    double* vec = nullptr;              // [nPoints * nmax * 3]
    double* dist = nullptr;             // [nPoints * nmax]
    float4* p32 = nullptr;              // [nPoints] FP32 copies for the candidate scan
};

namespace {
// Rows of nmax entries.  (On failure the list has no rows, and the next call allocates them.)
int nl_alloc(svm_neighbor_list* nl, int nmax) {
    const auto release = [&] {
        cudaFree(nl->idx); cudaFree(nl->vec); cudaFree(nl->dist);
        nl->idx = nullptr; nl->vec = nullptr; nl->dist = nullptr;
    };
    release();
    const size_t e = (size_t)nl->nPoints * nmax;
    if (cudaMalloc(&nl->idx, sizeof(int) * e) != cudaSuccess || cudaMalloc(&nl->vec, sizeof(double) * 3 * e) != cudaSuccess ||
        cudaMalloc(&nl->dist, sizeof(double) * e) != cudaSuccess) {
        release();
        cudaGetLastError();
        return SVM_ERR_CUDA;
    }
    nl->nmax = nmax;
    return SVM_OK;
}

// The scan's FP32 thresholds for points within [-radius, radius]^3, rounded outward.
void nl_thresholds(NlParams& p) {
    const double E = p.radius * 0x1p-21;
    auto down = [](double v) { float f = (float)v; if ((double)f > v) f = std::nextafter(f, -INFINITY); return f; };
    auto up = [](double v) { float f = (float)v; if ((double)f < v) f = std::nextafter(f, INFINITY); return f; };
    p.wrapLim = p.radius > 2 * E ? down(p.radius - 2 * E) : -1.f;
    const double hi = (p.range + 2 * E) * (1 + 0x1p-20), lo = (p.range - 2 * E) * (1 - 0x1p-20);
    p.thrHi = up(hi * hi);
    p.thrLo = lo > 0 ? down(lo * lo) : -1.f;
}

// After the cell list's own launches: the points are binned and their FP32 copies written.
template <typename P>
int nl_compute(svm_neighbor_list* nl, P pts, int np) {
    svm_cell_list* cl = nl->cl;
    const int* sc = cl->hostScalars;
    if (!nl->dist)
        if (int rc = nl_alloc(nl, nl->nmax)) return rc;
    for (int pass = 0; pass < 64; ++pass) {   // a third pass at most: slots widened, then nmax grown
        NlParams prm;
        prm.np = np; prm.cap = cl->cap; prm.nside = cl->nside; prm.K = nl->K; prm.nmax = nl->nmax;
        prm.radius = cl->radius; prm.range = nl->range;
        prm.range2Hi = nl->range * nl->range * (1.0 + 0x1p-48);
        nl_thresholds(prm);
        k_nl<<<(np + kNlPoints - 1) / kNlPoints, kB, 0, cl->stream>>>(pts, nl->p32, prm, cl->counts, cl->slots, cl->binOf,
                                                                      nl->mask, nl->npp, nl->idx, nl->vec, nl->dist,
                                                                      cl->scalars + 4);
        if (check_launch() || read_scalars(cl)) return SVM_ERR_CUDA;
        if (sc[3]) return SVM_ERR_DEVICE;  // a point lay outside the grid (or was not finite)
        if (sc[2]) {                       // a bin overflowed its slots: widen them, bin again
            if (cl_grow(cl, sc[0]) || compute(cl, pts, np, nl->p32)) return SVM_ERR_CUDA;
            continue;
        }
        const int longest = sc[4];         // (of the same points at any nmax: the next pass finds it again)
        if (longest <= nl->nmax) return SVM_OK;
        if (nl_alloc(nl, longest)) return SVM_ERR_CUDA;   // grow-only, then recompute
    }
    return SVM_ERR_DEVICE;
}
}  // namespace

extern "C" {

int svm_neighbor_list_create(double range, double radius, int subGridReduction, int nPoints, int slotCapacity,
                             void* stream, svm_neighbor_list** out) {
    if (!(range > 0) || !(radius > 0) || subGridReduction < 1 || nPoints <= 0 || !out) return SVM_ERR_ARG;
    svm_neighbor_list* nl = new svm_neighbor_list();
    nl->range = range; nl->radius = radius; nl->nPoints = nPoints;
    int rc = svm_cell_list_create(range * (1. / (double)subGridReduction), radius, nPoints, slotCapacity, stream, &nl->cl);
    if (rc) { delete nl; return rc; }
    // computeAdjacentCells (hyperrectangularCellList.cpp:219-262): offsets in iVecIterate order
    // (x fastest) whose nearest corner lies within `width` bins
    const int width = subGridReduction;
    const double h = nl->cl->h;
    std::vector<int> mask;
    for (int z = -width; z <= width; ++z)
        for (int y = -width; y <= width; ++y)
            for (int x = -width; x <= width; ++x) {
                const int g[3] = {x, y, z};
                double rmin = 0.0;
                for (int d = 0; d < 3; ++d) {
                    const double t = h * (std::max(std::abs(g[d]) - 1., 0.0));
                    rmin += t * t;
                }
                rmin = std::sqrt(rmin);
                if (rmin < h * width + 1e-6) { mask.push_back(x); mask.push_back(y); mask.push_back(z); }
            }
    nl->K = (int)mask.size() / 3;
    bool ok = cudaMalloc(&nl->mask, sizeof(int) * mask.size()) == cudaSuccess &&
              cudaMalloc(&nl->npp, sizeof(unsigned) * nPoints) == cudaSuccess &&
              cudaMalloc(&nl->p32, sizeof(float4) * nPoints) == cudaSuccess && nl_alloc(nl, nl->nmax) == SVM_OK;
    if (ok) ok = cudaMemcpy(nl->mask, mask.data(), sizeof(int) * mask.size(), cudaMemcpyHostToDevice) == cudaSuccess;
    if (!ok) { svm_neighbor_list_destroy(nl); return SVM_ERR_CUDA; }
    *out = nl;
    return SVM_OK;
}

int svm_neighbor_list_destroy(svm_neighbor_list* nl) {
    if (!nl) return SVM_ERR_ARG;
    if (nl->cl) svm_cell_list_destroy(nl->cl);
    void* ptrs[] = {nl->mask, nl->npp, nl->idx, nl->vec, nl->dist, nl->p32};
    for (void* p : ptrs) if (p) cudaFree(p);
    delete nl;
    return SVM_OK;
}

int svm_neighbor_list_compute(svm_neighbor_list* nl, const double* pts, int n) {
    if (!nl || !pts) return SVM_ERR_ARG;
    int rc = compute(nl->cl, AosPoints{pts}, n, nl->p32);
    return rc ? rc : nl_compute(nl, AosPoints{pts}, n);
}

int svm_neighbor_list_compute_model(svm_neighbor_list* nl, svm_model* m) {
    if (!nl || !m) return SVM_ERR_ARG;
    int rc = compute_model(nl->cl, m, nl->p32);
    if (rc) return rc;
    if (m->precision == SVM_PRECISION_MIXED) return nl_compute(nl, ModelPoints32{m->pos32[m->cur]}, m->nVertices);
    return nl_compute(nl, ModelPoints{m->pos[m->cur]}, m->nVertices);
}

int svm_neighbor_list_get(svm_neighbor_list* nl, int* nmax, unsigned* npp, int* idx, double* vec, double* dist,
                          long capacity) {
    if (!nl) return SVM_ERR_ARG;
    if (nmax) *nmax = nl->nmax;
    const size_t e = (size_t)nl->nPoints * nl->nmax;
    if ((idx || vec || dist) && (long)e > capacity) return SVM_ERR_ARG;
    if ((idx || vec || dist) && !nl->dist) return SVM_ERR_CUDA;   // the last call found no room for its rows
    cudaStream_t s = nl->cl->stream;
    if (npp && cudaMemcpyAsync(npp, nl->npp, sizeof(unsigned) * nl->nPoints, cudaMemcpyDeviceToHost, s) != cudaSuccess)
        return SVM_ERR_CUDA;
    if (idx && cudaMemcpyAsync(idx, nl->idx, sizeof(int) * e, cudaMemcpyDeviceToHost, s) != cudaSuccess) return SVM_ERR_CUDA;
    if (vec && cudaMemcpyAsync(vec, nl->vec, sizeof(double) * 3 * e, cudaMemcpyDeviceToHost, s) != cudaSuccess)
        return SVM_ERR_CUDA;
    if (dist && cudaMemcpyAsync(dist, nl->dist, sizeof(double) * e, cudaMemcpyDeviceToHost, s) != cudaSuccess)
        return SVM_ERR_CUDA;
    return cudaStreamSynchronize(s) == cudaSuccess ? SVM_OK : SVM_ERR_CUDA;
}

int svm_cell_list_create(double a, double radius, int nPoints, int cap, void* stream, svm_cell_list** out) {
    if (!(a > 0) || !(radius > 0) || nPoints <= 0 || cap < 2 || !out) return SVM_ERR_ARG;
    svm_cell_list* cl = new svm_cell_list();
    cl->a = a; cl->radius = radius; cl->nPoints = nPoints; cl->cap = cap;
    const double b = 2. * radius;  // setGridSize (hyperrectangularCellList.cpp:31-41)
    unsigned n = (unsigned)std::floor(b / a);
    if (n % 2 == 1) n -= 1;
    if (n == 0) { delete cl; return SVM_ERR_ARG; }
    cl->nside = (int)n;
    cl->h = b / n;
    cl->total = (long)n * n * n;
    if (stream) cl->stream = (cudaStream_t)stream;
    else { cudaStreamCreateWithFlags(&cl->stream, cudaStreamNonBlocking); cl->ownStream = true; }
    bool ok = cudaMalloc(&cl->counts, sizeof(unsigned) * cl->total) == cudaSuccess &&
              cudaMalloc(&cl->tmp, sizeof(int) * cl->total * cap) == cudaSuccess &&
              cudaMalloc(&cl->slots, sizeof(int) * cl->total * cap) == cudaSuccess &&
              cudaMalloc(&cl->binOf, sizeof(int) * nPoints) == cudaSuccess &&
              cudaMalloc(&cl->scalars, sizeof(int) * kClScalars) == cudaSuccess &&
              cudaMallocHost(&cl->hostScalars, sizeof(int) * kClScalars) == cudaSuccess;
    if (!ok) { svm_cell_list_destroy(cl); return SVM_ERR_CUDA; }
    cudaMemsetAsync(cl->counts, 0, sizeof(unsigned) * cl->total, cl->stream);
    cudaMemsetAsync(cl->binOf, 0xff, sizeof(int) * nPoints, cl->stream);
    const int init[kClScalars] = {0, 2};  // Nmax starts at 2 (hyperrectangularCellList.cpp:17,47)
    cudaMemcpyAsync(cl->scalars, init, sizeof(init), cudaMemcpyHostToDevice, cl->stream);
    if (cudaStreamSynchronize(cl->stream) != cudaSuccess) { svm_cell_list_destroy(cl); return SVM_ERR_CUDA; }
    *out = cl;
    return SVM_OK;
}

int svm_cell_list_destroy(svm_cell_list* cl) {
    if (!cl) return SVM_ERR_ARG;
    if (cl->stream) cudaStreamSynchronize(cl->stream);
    void* ptrs[] = {cl->counts, cl->tmp, cl->slots, cl->binOf, cl->scalars};
    for (void* p : ptrs) if (p) cudaFree(p);
    if (cl->hostScalars) cudaFreeHost(cl->hostScalars);
    if (cl->ownStream && cl->stream) cudaStreamDestroy(cl->stream);
    delete cl;
    return SVM_OK;
}

int svm_cell_list_compute_model(svm_cell_list* cl, svm_model* m) {
    return !cl || !m ? SVM_ERR_ARG : compute_model(cl, m);
}

int svm_cell_list_compute(svm_cell_list* cl, const double* pts, int n) {
    if (!cl || !pts) return SVM_ERR_ARG;
    return compute(cl, AosPoints{pts}, n);
}

int svm_cell_list_get(svm_cell_list* cl, int* nside, int* nmax, unsigned* counts, int* slots, long cap) {
    if (!cl) return SVM_ERR_ARG;
    int sc[4];
    if (cudaMemcpyAsync(sc, cl->scalars, sizeof(sc), cudaMemcpyDeviceToHost, cl->stream) != cudaSuccess ||
        cudaStreamSynchronize(cl->stream) != cudaSuccess) return SVM_ERR_CUDA;
    if (nside) *nside = cl->nside;
    if (nmax) *nmax = sc[1];
    if (sc[2] || sc[3]) return SVM_ERR_DEVICE;  // a bin overflowed its slots, or a point left the grid
    const int Nmax = sc[1];
    if (counts) {
        if (cudaMemcpy(counts, cl->counts, sizeof(unsigned) * cl->total, cudaMemcpyDeviceToHost) != cudaSuccess) return SVM_ERR_CUDA;
    }
    if (slots) {
        if (cap < cl->total * Nmax) return SVM_ERR_ARG;
        if (!cl->slots) return SVM_ERR_CUDA;
        std::vector<unsigned> cnt(cl->total);
        std::vector<int> s((size_t)cl->total * cl->cap);
        if (cudaMemcpy(cnt.data(), cl->counts, sizeof(unsigned) * cl->total, cudaMemcpyDeviceToHost) != cudaSuccess ||
            cudaMemcpy(s.data(), cl->slots, sizeof(int) * s.size(), cudaMemcpyDeviceToHost) != cudaSuccess)
            return SVM_ERR_CUDA;
        for (long b = 0; b < cl->total; ++b)
            for (int k = 0; k < Nmax; ++k)
                slots[b * Nmax + k] = (k < (int)cnt[b] && k < cl->cap) ? s[(size_t)b * cl->cap + k] : -1;
    }
    return SVM_OK;
}

int svm_cell_list_bins(svm_cell_list* cl, int* binOfPoint) {
    if (!cl || !binOfPoint) return SVM_ERR_ARG;
    if (cudaMemcpyAsync(binOfPoint, cl->binOf, sizeof(int) * cl->nPoints, cudaMemcpyDeviceToHost, cl->stream) != cudaSuccess ||
        cudaStreamSynchronize(cl->stream) != cudaSuccess) return SVM_ERR_CUDA;
    return SVM_OK;
}

}  // extern "C"
