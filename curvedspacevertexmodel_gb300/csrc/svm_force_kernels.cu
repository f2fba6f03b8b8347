// The FP64 force kernels of the plain form: computeForce (sphericalVertexModel.cpp:356-420) alone
// and fused with the Brownian displacement and the move (brownianDynamics.cpp:37-44,
// sphericalDomain.h:203-209).  Kept in its own translation unit so that its contraction setting
// can differ from the geometry's; it is built without FMA contraction like the rest (the force's
// rounding then differs from the CPU's only through acos), and the displacement and the move spell
// out every product and sum with __dmul_rn / __dadd_rn.
#include <mutex>
#include <type_traits>

#include "svm_force.cuh"

namespace svm {
int check_launch();
}

namespace {
// The ziggurat table of this device, built once by k_zig_init (zig_init) from r alone:
// v = r f(r) + sqrt(pi/2) erfc(r / sqrt 2), then f(x_{i+1}) = v / x_i + f(x_i).
__device__ svm::ZigTable gZig;

__global__ void k_zig_init() {
    const double r = svm::kZigR, fr = exp(-0.5 * r * r);
    const double v = r * fr + sqrt(0.5 * svm::kPI) * erfc(r / sqrt(2.0));
    gZig.x[0] = v / fr;
    gZig.f[0] = 0.0;
    gZig.x[1] = r;
    gZig.f[1] = fr;
    for (int i = 1; i < 255; ++i) {
        const double f1 = v / gZig.x[i] + gZig.f[i];
        gZig.f[i + 1] = f1;
        gZig.x[i + 1] = sqrt(-2.0 * log(f1));
    }
    gZig.x[256] = 0.0;
    gZig.f[256] = 1.0;
}
}  // namespace

namespace {
using namespace svm;

// One instantiation per form (one that held both spilled more: 100k cells 231 -> 227 us, 200 cells 18 -> 17).
constexpr int form_min_blocks(int form) { return form == kFormVector ? 6 : kSlotMinBlocks; }

template <int kForm, bool kHwMul>
__global__ void __launch_bounds__(slot_threads(kSlotVerts), form_min_blocks(kForm))
    k_force(ForceArgs A, int nV, double4_32a* __restrict__ force) {
    step_begin();
    __shared__ SlotShared<> sh;
    const D3 f = block_slot_force<kForm, kHwMul>(A, nV, sh, NoSide());
    const int v = blockIdx.x * kSlotVerts + threadIdx.x;
    if (threadIdx.x >= kSlotVerts || v >= nV) return;
    st3(force, v, f);
}

// Fused Brownian step: force, displacement, move; reads `A.pos`, writes posNext (and hostOut, when
// non-null).  Role 1's threads draw the vertex's three normals, one each, while role 0 evaluates the
// edge gradients.
// (Writing the moved vertex's norm here as well, which would spare the corner pass its k_vnorm, made
// this FP64-bound kernel as much slower as the corner pass got faster.)
template <int kNoise, int kForm, bool kHwMul>
__global__ void __launch_bounds__(slot_threads(kSlotVerts), form_min_blocks(kForm))
    k_force_bd(ForceArgs A, int nV, double4_32a* __restrict__ force, double4_32a* __restrict__ posNext,
               const double* __restrict__ noise, uint64_t seed, const unsigned long long* __restrict__ stepCounter,
               double np, double fp, const ZigTable* __restrict__ zig, double* __restrict__ hostOut) {
    step_begin();
    __shared__ SlotShared<> sh;
    __shared__ double xi[3 * kSlotVerts];
    const D3 f = block_slot_force<kForm, kHwMul>(A, nV, sh, [&](const SlotIndex& q) {
        xi[q.at] = kNoise == SVM_NOISE_BUFFER ? noise[3 * q.v + q.s] : philox_normal(zig, seed, *stepCounter, q.v, q.s);
    });
    const int t = threadIdx.x, v = blockIdx.x * kSlotVerts + t;
    if (t >= kSlotVerts || v >= nV) return;
    st3(force, v, f);
    const D3 d{bd_disp(xi[3 * t], np, f.x, fp), bd_disp(xi[3 * t + 1], np, f.y, fp), bd_disp(xi[3 * t + 2], np, f.z, fp)};
    const D3 p = move_exact(ld3(A.pos, v), d, A.R);
    st3(posNext, v, p);
    // a host-buffer step's output, straight into the caller's mapped page-locked array (AoS)
    if (hostOut) { hostOut[3 * v] = p.x; hostOut[3 * v + 1] = p.y; hostOut[3 * v + 2] = p.z; }
}

int slot_blocks(int nV) { return (nV + kSlotVerts - 1) / kSlotVerts; }

}  // namespace

namespace svm {

// f(form, hwMul) with the two as compile-time constants
template <class F>
static void with_form(const svm_model* m, F f) {
    using T = std::true_type;
    using N = std::false_type;
    if (m->precision == SVM_PRECISION_FP64_VECTOR) {
        using V = std::integral_constant<int, kFormVector>;
        few_hw_mul(m) ? f(V(), T()) : f(V(), N());
    } else {
        using R = std::integral_constant<int, kFormReference>;
        few_hw_mul(m) ? f(R(), T()) : f(R(), N());
    }
}

int launch_force_fp64(svm_model* m) {
    with_form(m, [&](auto form, auto hw) {
        launch_next(m, k_force<form.value, hw.value>, slot_blocks(m->nVertices), slot_threads(kSlotVerts),
                    force_args(m, m->cur), m->nVertices, m->force);
    });
    return check_launch();
}

// Builds this device's ziggurat table once (outside any stream capture: called at model creation).
static ZigTable* gZigAddr[64] = {};  // per device, once built
int zig_init() {
    static std::mutex mu;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return SVM_ERR_CUDA;
    std::lock_guard<std::mutex> lock(mu);
    if (gZigAddr[dev]) return SVM_OK;
    ZigTable* addr = nullptr;
    if (cudaGetSymbolAddress((void**)&addr, gZig) != cudaSuccess) return SVM_ERR_CUDA;
    k_zig_init<<<1, 1>>>();
    if (check_launch() || cudaDeviceSynchronize() != cudaSuccess) return SVM_ERR_CUDA;
    gZigAddr[dev] = addr;
    return SVM_OK;
}

int launch_force_bd_fp64(svm_model* m, double np, double fp, int noiseMode, const double* noise, uint64_t seed,
                         int nxt) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64 || !gZigAddr[dev]) return SVM_ERR_CUDA;
    const ZigTable* zig = gZigAddr[dev];
    const auto go = [&](auto kernel) {
        launch_next(m, kernel, slot_blocks(m->nVertices), slot_threads(kSlotVerts),
            force_args(m, m->cur), m->nVertices, m->force, m->pos[nxt], noise, seed, m->stepCounter, np, fp, zig,
            m->ioHostOut);
    };
    with_form(m, [&](auto form, auto hw) {
        if (noiseMode == SVM_NOISE_BUFFER) go(k_force_bd<SVM_NOISE_BUFFER, form.value, hw.value>);
        else go(k_force_bd<SVM_NOISE_PHILOX, form.value, hw.value>);
    });
    return check_launch();
}

}  // namespace svm
