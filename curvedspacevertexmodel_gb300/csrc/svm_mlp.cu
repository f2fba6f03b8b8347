// Learned warm start for FIRE (svm_mlp_* in include/svm.h): a per-vertex MLP 24 -> 64 -> 64 -> 2
// (ReLU hidden layers, BF16 weights, FP32 accumulation) that reads the local tangent-frame
// geometry of a vertex and predicts its displacement to the relaxed state.  No counterpart in the
// reference.
//
// Features of vertex v (FP32, from the FP64 model state after geometry and forces):
//   frame: n = v/|v|, e1 = unit tangent projection of (nbr0 - v), e2 = n x e1;
//   [0..5]   offsets to the three neighbours (vnbr slots) in (e1, e2);
//   [6..11]  offsets to the three adjacent cells' centroids (vcell slots) in (e1, e2);
//   [12..17] (A - A0, P - P0) of the three cells;
//   [18..20] (ring size - 6) of the three cells;
//   [21..22] the force in (e1, e2);  [23] |force|.
// Output: the displacement in (e1, e2), in units of the network's output scale.
//
// Parameters (FP32 master copy, kParams floats): W1[64][24], b1[64], W2[64][64], b2[64],
// W3[2][64], b3[2], row-major (out, in).  The forward pass uses their BF16 roundings; gradients
// are taken with respect to those (straight-through) and applied to the master copy by Adam.
//
// Every layer runs as register tiles over shared memory: a block of kTT threads takes kTS samples, a
// thread four samples by two units, each output one chain of FP32 multiply-adds over the inputs in
// ascending order.  Training takes kTB samples per cluster of four such blocks: each block runs its
// quarter of the samples forward and back, then, with the cluster's activations and deltas gathered
// through distributed shared memory, sums a quarter of the parameters' gradients over all kTB samples
// in sample order; a second kernel sums the clusters' partials in order and applies Adam, so gradients
// are deterministic and do not depend on how the work is spread.
// What bounds it: FP32 multiply-adds (35k per sample and step, 2 us for 4096 samples at 128 a clock on
// 152 SMs) and, far above that, the latency of the chains; a batch of 4096 is 128 blocks.  The batch's loss stays on
// the device until the epoch ends.  A batch, both kernels: 4096 samples 35.6 -> 24.8 us, 512 samples 27.9 -> 16.2 with
// the weights read eight at a time, the remote reads of a cluster all in flight together, and each kernel set up,
// with the batch's samples fetched, while the previous one ends.
#include <algorithm>
#include <cmath>
#include <mutex>
#include <cstdio>
#include <random>
#include <vector>
#include <cooperative_groups.h>
#include <cuda_bf16.h>
#include "svm_internal.cuh"

namespace {
using namespace svm;

constexpr int kIn = 24, kH = 64, kOut = 2;
constexpr int oW1 = 0, oB1 = oW1 + kH * kIn, oW2 = oB1 + kH, oB2 = oW2 + kH * kH, oW3 = oB2 + kH,
              oB3 = oW3 + kOut * kH, kParams = oB3 + kOut;
constexpr int kTB = 128;       // samples per training cluster (one partial gradient)
constexpr int kTC = 4;         // blocks per training cluster
constexpr int kTS = 32;        // samples per tile
constexpr int kTT = 256;       // threads per tile
constexpr int kQ = kH / kTC;   // hidden units whose gradients one block of a cluster sums
static_assert(kTS * kTC == kTB, "a cluster's tiles cover its samples");
// Shared-memory row strides (floats): 16-byte rows whose starts fall on distinct banks, so that a
// warp's 8 sample rows and 4 unit rows load as 16-byte vectors without conflicts.
constexpr int kSX = kIn + 4, kSH = kH + 4, kSQ = kQ + 4;
// the weights in shared memory: W1[64][kSX] | W2[64][kSH] | W3[2][64] | b1 | b2 | b3
constexpr int sW1 = 0, sW2 = sW1 + kH * kSX, sW3 = sW2 + kH * kSH, sB1 = sW3 + kOut * kH, sB2 = sB1 + kH, sB3 = sB2 + kH,
              kWeights = sB3 + 4;

__device__ __forceinline__ int c3(const int4& a, int s) { return s == 0 ? a.x : (s == 1 ? a.y : a.z); }

struct FeatArgs {
    const double4_32a* pos;
    const int4* vnbr;
    const int4* vcell;
    const double4_32a* cellPos;
    const double2* ap;
    const double2* pref;
    const int* ringCount;
    const double4_32a* force;
};

// features and tangent frame of vertex v
__device__ void vertex_features(const FeatArgs& A, int v, float* x, D3& e1, D3& e2, D3& p) {
    p = ld3(A.pos, v);
    const D3 n = scl3(1.0 / sqrt(dot3(p, p)), p);
    const int4 nb = A.vnbr[v], cells = A.vcell[v];
    D3 d0 = sub3(ld3(A.pos, nb.x), p);
    d0 = sub3(d0, scl3(dot3(d0, n), n));
    e1 = scl3(1.0 / sqrt(dot3(d0, d0)), d0);
    e2 = cross3(n, e1);
#pragma unroll
    for (int s = 0; s < 3; ++s) {
        const D3 d = sub3(ld3(A.pos, c3(nb, s)), p);
        x[2 * s] = (float)dot3(d, e1);
        x[2 * s + 1] = (float)dot3(d, e2);
        const int c = c3(cells, s);
        const D3 dc = sub3(ld3(A.cellPos, c), p);
        x[6 + 2 * s] = (float)dot3(dc, e1);
        x[7 + 2 * s] = (float)dot3(dc, e2);
        const double2 apc = A.ap[c], pr = A.pref[c];
        x[12 + 2 * s] = (float)(apc.x - pr.x);
        x[13 + 2 * s] = (float)(apc.y - pr.y);
        x[18 + s] = (float)(A.ringCount[c] - 6);
    }
    const D3 f = ld3(A.force, v);
    x[21] = (float)dot3(f, e1);
    x[22] = (float)dot3(f, e2);
    x[23] = (float)sqrt(dot3(f, f));
}

__global__ void k_features(FeatArgs A, int nV, float* __restrict__ X, double* __restrict__ frames) {
    const int v = blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= nV) return;
    float x[kIn];
    D3 e1, e2, p;
    vertex_features(A, v, x, e1, e2, p);
    for (int k = 0; k < kIn; ++k) X[(long)v * kIn + k] = x[k];
    if (frames) {
        double* fr = frames + 6L * v;
        fr[0] = e1.x; fr[1] = e1.y; fr[2] = e1.z; fr[3] = e2.x; fr[4] = e2.y; fr[5] = e2.z;
    }
}

// BF16 weights -> FP32 in shared memory, rows at their strides: eight at a time (every section and row starts
// on a multiple of eight; the two output biases are left over), all of a thread's loads ahead of its stores.
constexpr int kW8 = oB3 / 8;
static_assert(oB3 % 8 == 0 && oB1 % 8 == 0 && oW2 % 8 == 0 && oB2 % 8 == 0 && oW3 % 8 == 0 && kIn % 8 == 0, "vectors of eight");
__device__ __forceinline__ float2 bf2(unsigned u) { return make_float2(__uint_as_float(u << 16), __uint_as_float(u & 0xffff0000u)); }
__device__ __forceinline__ void load_weights(const __nv_bfloat16* __restrict__ wb, float* w) {
    constexpr int kPer = (kW8 + kTT - 1) / kTT;
    const uint4* src = reinterpret_cast<const uint4*>(wb);
    uint4 q[kPer];
#pragma unroll
    for (int r = 0; r < kPer; ++r) {
        const int e = threadIdx.x + r * kTT;
        if (e < kW8) q[r] = src[e];
    }
#pragma unroll
    for (int r = 0; r < kPer; ++r) {
        const int i = 8 * (threadIdx.x + r * kTT);
        if (i >= oB3) break;
        int at;
        if (i < oB1) at = sW1 + (i / kIn) * kSX + i % kIn;
        else if (i < oW2) at = sB1 + (i - oB1);
        else if (i < oB2) at = sW2 + ((i - oW2) / kH) * kSH + (i - oW2) % kH;
        else if (i < oW3) at = sB2 + (i - oB2);
        else at = sW3 + (i - oW3);
        const float2 a = bf2(q[r].x), b = bf2(q[r].y), c = bf2(q[r].z), d = bf2(q[r].w);
        *reinterpret_cast<float4*>(w + at) = make_float4(a.x, a.y, b.x, b.y);
        *reinterpret_cast<float4*>(w + at + 4) = make_float4(c.x, c.y, d.x, d.y);
    }
    if (threadIdx.x < kOut) w[sB3 + threadIdx.x] = __bfloat162float(wb[oB3 + threadIdx.x]);
}

__device__ __forceinline__ float4 ld4(const float* p) { return *reinterpret_cast<const float4*>(p); }
// s + a . b over four consecutive inputs, one multiply-add after the other
__device__ __forceinline__ float chain4(float4 a, float4 b, float s) {
    return fmaf(a.w, b.w, fmaf(a.z, b.z, fmaf(a.y, b.y, fmaf(a.x, b.x, s))));
}

// One hidden layer of a tile: out[s][j] = relu(b[j] + sum_k W[j][k] in[s][k]).  Thread t computes
// samples t % 8 + 8 i (i < 4) of units t / 8 + 32 u (u < 2) and keeps them in h.  Samples from `count`
// on are written as zeros.
template <int kK, int kSIn>
__device__ __forceinline__ void tile_layer(const float* W, const float* b, const float* in, float* out, int count,
                                           float (&h)[4][2]) {
    const int sg = threadIdx.x & 7, jg = threadIdx.x >> 3;
    float acc[4][2];
#pragma unroll
    for (int u = 0; u < 2; ++u)
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[i][u] = b[jg + 32 * u];
#pragma unroll 4
    for (int k = 0; k < kK; k += 4) {
        const float4 w0 = ld4(W + jg * kSIn + k), w1 = ld4(W + (jg + 32) * kSIn + k);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float4 x = ld4(in + (sg + 8 * i) * kSIn + k);
            acc[i][0] = chain4(w0, x, acc[i][0]);
            acc[i][1] = chain4(w1, x, acc[i][1]);
        }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            h[i][u] = sg + 8 * i < count ? fmaxf(acc[i][u], 0.f) : 0.f;
            out[(sg + 8 * i) * kSH + jg + 32 * u] = h[i][u];
        }
}
// The network on a tile of kTS samples (x: rows of kSX in shared memory; every thread of the block
// calls it, after a barrier): activations to h1, h2 (rows of kSH; this thread's in a1, a2), and the
// outputs y[s][o] held by threads t < 2 kTS (s = t / 2, o = t % 2) as the return value.
__device__ __forceinline__ float tile_forward(const float* w, const float* x, float* h1, float* h2, int count,
                                              float (&a1)[4][2], float (&a2)[4][2]) {
    tile_layer<kIn, kSX>(w + sW1, w + sB1, x, h1, count, a1);
    __syncthreads();
    tile_layer<kH, kSH>(w + sW2, w + sB2, h1, h2, count, a2);
    __syncthreads();
    float y = 0.f;
    if (threadIdx.x < 2 * kTS) {
        const int s = threadIdx.x >> 1, o = threadIdx.x & 1;
        y = w[sB3 + o];
#pragma unroll
        for (int j = 0; j < kH; j += 4) y = chain4(ld4(w + sW3 + o * kH + j), ld4(h2 + s * kSH + j), y);
    }
    return y;
}

// Shared memory of a training block: the weights, this tile's x | h1 | h2 | d2 | d1 | dy, and the
// cluster's H1 | X and, of the block's kQ units, D2 | D1 | H2, and DY.
constexpr int tX = kWeights, tH1 = tX + kTS * kSX, tH2 = tH1 + kTS * kSH, tD2 = tH2 + kTS * kSH, tD1 = tD2 + kTS * kSH,
              tDY = tD1 + kTS * kSH, gH1 = tDY + kTS * 2, gX = gH1 + kTB * kSH, gD2 = gX + kTB * kSX, gD1 = gD2 + kTB * kSQ,
              gH2 = gD1 + kTB * kSQ, gDY = gH2 + kTB * kSQ, kTrainFloats = gDY + kTB * 2;

// Forward + backward of kTB samples per cluster of kTC blocks; the cluster's partial gradients and each
// tile's loss.
__global__ void __cluster_dims__(kTC, 1, 1) __launch_bounds__(kTT)
    k_train_block(const __nv_bfloat16* __restrict__ wb, const float* __restrict__ X, const float* __restrict__ Y,
                  const int* __restrict__ order, int first, int count, float invBatch, float* __restrict__ partials,
                  double* __restrict__ lossPartials) {
    namespace cg = cooperative_groups;
    extern __shared__ float4 smem4[];
    float* sm = reinterpret_cast<float*>(smem4);
    cg::cluster_group cluster = cg::this_cluster();
    const int t = threadIdx.x, rank = (int)cluster.block_rank();
    const int base = blockIdx.x * kTS;                 // tiles of a cluster are consecutive
    const int live = max(0, min(kTS, count - base));
    // the tile's samples on their way first: they do not depend on the previous batch's update
    constexpr int kXPer = kTS * kIn / kTT;
    static_assert(kTS * kIn % kTT == 0, "whole rounds");
    float xr[kXPer];
#pragma unroll
    for (int r = 0; r < kXPer; ++r) {
        const int e = t + r * kTT, s = e / kIn, k = e - s * kIn;
        xr[r] = 0.f;
        if (s < live) xr[r] = X[(long)(order ? order[first + base + s] : first + base + s) * kIn + k];
    }
    step_begin();
    load_weights(wb, sm);
#pragma unroll
    for (int r = 0; r < kXPer; ++r) {
        const int e = t + r * kTT, s = e / kIn, k = e - s * kIn;
        sm[tX + s * kSX + k] = xr[r];
    }
    __syncthreads();
    float a1[4][2], a2[4][2];
    const float y = tile_forward(sm, sm + tX, sm + tH1, sm + tH2, live, a1, a2);
    if (t < 2 * kTS) {
        const int s = t >> 1, o = t & 1;
        float r = 0.f;
        if (s < live) {
            const int sIdx = order ? order[first + base + s] : first + base + s;
            r = y - Y[2L * sIdx + o];
        }
        sm[tDY + t] = 2.f * r * invBatch;
        // (y0 - t0)^2 + (y1 - t1)^2 of sample s on its even thread, summed over the tile as a warp's
        // shuffle tree over its samples does: the even threads of two warps hold 16 samples each
        const double rd = (double)r * r;
        const double ro = __shfl_xor_sync(0xffffffffu, rd, 1);
        double* lossSh = reinterpret_cast<double*>(sm + gDY);   // (not yet in use)
        if (o == 0) lossSh[s] = rd + ro;
    }
    __syncthreads();
    if (t < 32) {
        double loss = reinterpret_cast<const double*>(sm + gDY)[t];
        for (int o = 16; o > 0; o >>= 1) loss += __shfl_down_sync(0xffffffffu, loss, o);
        if (t == 0) lossPartials[blockIdx.x] = loss;
    }
    const int sg = t & 7, jg = t >> 3;
    // deltas of layer 2's pre-activations
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int s = sg + 8 * i;
        const float dy0 = sm[tDY + 2 * s], dy1 = sm[tDY + 2 * s + 1];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const int j = jg + 32 * u;
            const float g = sm[sW3 + j] * dy0 + sm[sW3 + kH + j] * dy1;
            sm[tD2 + s * kSH + j] = a2[i][u] > 0.f ? g : 0.f;
        }
    }
    __syncthreads();
    // deltas of layer 1's pre-activations
    {
        float g[4][2] = {};
#pragma unroll 4
        for (int i = 0; i < kH; i += 4) {
            float4 d[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) d[q] = ld4(sm + tD2 + (sg + 8 * q) * kSH + i);
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const float* w = sm + sW2 + i * kSH + jg + 32 * u;
                const float4 wv = make_float4(w[0], w[kSH], w[2 * kSH], w[3 * kSH]);
#pragma unroll
                for (int q = 0; q < 4; ++q) g[q][u] = chain4(wv, d[q], g[q][u]);
            }
        }
#pragma unroll
        for (int q = 0; q < 4; ++q)
#pragma unroll
            for (int u = 0; u < 2; ++u) sm[tD1 + (sg + 8 * q) * kSH + jg + 32 * u] = a1[q][u] > 0.f ? g[q][u] : 0.f;
    }
    cluster.sync();
    // The cluster's activations and deltas, in sample order: a block's loads are all on their way before the
    // first is stored (the four blocks one after another were a chain of remote loads, a quarter of the kernel).
    const int u0 = rank * kQ;
    {
        constexpr int kH4 = kTS * (kH / 4) / kTT, kQ4 = (3 * kTS * (kQ / 4) + kTT - 1) / kTT;
        static_assert(kTS * (kH / 4) % kTT == 0 && kTS * (kIn / 4) <= kTT, "whole rounds");
        float4 h[kTC][kH4], x[kTC], d[kTC][kQ4];
        float dy[kTC];
#pragma unroll
        for (int p = 0; p < kTC; ++p) {
            const float* src = cluster.map_shared_rank(sm, p);
#pragma unroll
            for (int r = 0; r < kH4; ++r) {
                const int e = t + r * kTT;
                h[p][r] = ld4(src + tH1 + (e / (kH / 4)) * kSH + 4 * (e % (kH / 4)));
            }
            if (t < kTS * (kIn / 4)) x[p] = ld4(src + tX + (t / (kIn / 4)) * kSX + 4 * (t % (kIn / 4)));
#pragma unroll
            for (int r = 0; r < kQ4; ++r) {
                const int e = t + r * kTT, a = e / (kTS * (kQ / 4)), q = e % (kTS * (kQ / 4));
                if (a < 3) d[p][r] = ld4(src + (a == 0 ? tD2 : (a == 1 ? tD1 : tH2)) + (q / (kQ / 4)) * kSH + u0 + 4 * (q % (kQ / 4)));
            }
            if (t < 2 * kTS) dy[p] = src[tDY + t];
        }
#pragma unroll
        for (int p = 0; p < kTC; ++p) {
#pragma unroll
            for (int r = 0; r < kH4; ++r) {
                const int e = t + r * kTT;
                *reinterpret_cast<float4*>(sm + gH1 + (p * kTS + e / (kH / 4)) * kSH + 4 * (e % (kH / 4))) = h[p][r];
            }
            if (t < kTS * (kIn / 4))
                *reinterpret_cast<float4*>(sm + gX + (p * kTS + t / (kIn / 4)) * kSX + 4 * (t % (kIn / 4))) = x[p];
#pragma unroll
            for (int r = 0; r < kQ4; ++r) {
                const int e = t + r * kTT, a = e / (kTS * (kQ / 4)), q = e % (kTS * (kQ / 4));
                if (a < 3)
                    *reinterpret_cast<float4*>(sm + (a == 0 ? gD2 : (a == 1 ? gD1 : gH2)) + (p * kTS + q / (kQ / 4)) * kSQ +
                                               4 * (q % (kQ / 4))) = d[p][r];
            }
            if (t < 2 * kTS) sm[gDY + p * 2 * kTS + t] = dy[p];
        }
    }
    cluster.sync();  // (no block leaves while another still reads its shared memory)
    float* out = partials + (long)(blockIdx.x / kTC) * kParams;
    {   // dW2 rows u0 .. u0 + kQ: thread (column j, four rows)
        const int j = t & (kH - 1), ig = 4 * (t >> 6);
        float s0 = 0.f, s1 = 0.f, s2 = 0.f, s3 = 0.f;
#pragma unroll 8
        for (int q = 0; q < kTB; ++q) {
            const float4 d = ld4(sm + gD2 + q * kSQ + ig);
            const float h = sm[gH1 + q * kSH + j];
            s0 = fmaf(d.x, h, s0); s1 = fmaf(d.y, h, s1); s2 = fmaf(d.z, h, s2); s3 = fmaf(d.w, h, s3);
        }
        float* o = out + oW2 + (u0 + ig) * kH + j;
        o[0] = s0; o[kH] = s1; o[2 * kH] = s2; o[3 * kH] = s3;
    }
    if (t < 192) {  // dW1 rows u0 .. u0 + kQ: thread (column k, two rows)
        const int k = t % kIn, ig = 2 * (t / kIn);
        float s0 = 0.f, s1 = 0.f;
#pragma unroll 8
        for (int q = 0; q < kTB; ++q) {
            const float x = sm[gX + q * kSX + k];
            s0 = fmaf(sm[gD1 + q * kSQ + ig], x, s0);
            s1 = fmaf(sm[gD1 + q * kSQ + ig + 1], x, s1);
        }
        out[oW1 + (u0 + ig) * kIn + k] = s0;
        out[oW1 + (u0 + ig + 1) * kIn + k] = s1;
    } else if (t < 224) {  // dW3 columns u0 .. u0 + kQ
        const int o = (t - 192) / kQ, j = (t - 192) % kQ;
        float s = 0.f;
#pragma unroll 8
        for (int q = 0; q < kTB; ++q) s = fmaf(sm[gDY + 2 * q + o], sm[gH2 + q * kSQ + j], s);
        out[oW3 + o * kH + u0 + j] = s;
    } else {  // db2, db1 of the kQ units
        const int i = (t - 224) % kQ, which = (t - 224) / kQ;
        const float* d = sm + (which ? gD1 : gD2) + i;
        float s = 0.f;
#pragma unroll 8
        for (int q = 0; q < kTB; ++q) s += d[q * kSQ];
        out[(which ? oB1 : oB2) + u0 + i] = s;
    }
    if (rank == 0 && t < kOut) {
        float s = 0.f;
        for (int q = 0; q < kTB; ++q) s += sm[gDY + 2 * q + t];
        out[oB3 + t] = s;
    }
}

struct AdamStep { float lr, b1, b2, eps, c1, c2; };
// grad[i] = sum over clusters (in order) of the partials; with kAdam the update of the FP32 master
// weights (Adam, Kingma and Ba, 2015) and their BF16 copy follows.  loss: the samples' sum, each
// cluster's four tiles in order, then the clusters; added to *loss with kAdam, else stored there.
template <bool kAdam>
__global__ void k_reduce_grad(const float* __restrict__ partials, int nBlocks, float* __restrict__ grad,
                              const double* __restrict__ lossPartials, double* __restrict__ loss, float* __restrict__ w,
                              float* __restrict__ m, float* __restrict__ v, __nv_bfloat16* __restrict__ wb, AdamStep A) {
    step_begin();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < kParams) {
        float gi = 0.f;
#pragma unroll 8
        for (int b = 0; b < nBlocks; ++b) gi += partials[(long)b * kParams + i];
        grad[i] = gi;
        if (kAdam) {
            const float mi = A.b1 * m[i] + (1.f - A.b1) * gi;
            const float vi = A.b2 * v[i] + (1.f - A.b2) * gi * gi;
            m[i] = mi;
            v[i] = vi;
            const float wi = w[i] - A.lr * (mi / A.c1) / (sqrtf(vi / A.c2) + A.eps);
            w[i] = wi;
            wb[i] = __float2bfloat16_rn(wi);
        }
    } else if (i == kParams) {
        double l = 0.0;
#pragma unroll 4
        for (int b = 0; b < nBlocks; ++b) {
            double lb = 0.0;
            for (int q = 0; q < kTC; ++q) lb += lossPartials[b * kTC + q];
            l += lb;
        }
        *loss = kAdam ? *loss + l : l;
    }
}

__global__ void k_to_bf16(const float* __restrict__ w, __nv_bfloat16* __restrict__ wb) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < kParams) wb[i] = __float2bfloat16_rn(w[i]);
}

// Dynamic shared memory of the inference kernels: the weights, x[kSamples] rows, h1, h2 of one tile.
constexpr size_t infer_floats(int samples) { return kWeights + (size_t)samples * kSX + 2 * kTS * kSH; }

// Outputs of n samples, a tile at a time per block.
__global__ void __launch_bounds__(kTT) k_predict(const __nv_bfloat16* __restrict__ wb, const float* __restrict__ X,
                                                 int n, float* __restrict__ Y) {
    extern __shared__ float4 smem4[];
    float* sm = reinterpret_cast<float*>(smem4);
    float *x = sm + kWeights, *h1 = x + kTS * kSX, *h2 = h1 + kTS * kSH;
    load_weights(wb, sm);
    for (int base = blockIdx.x * kTS; base < n; base += gridDim.x * kTS) {
        const int live = min(kTS, n - base);
        __syncthreads();  // (the weights; the previous tile's x)
        for (int e = threadIdx.x; e < kTS * kIn; e += kTT) {
            const int s = e / kIn, k = e - s * kIn;
            x[s * kSX + k] = s < live ? X[(long)base * kIn + e] : 0.f;
        }
        __syncthreads();
        float a1[4][2], a2[4][2];
        const float y = tile_forward(sm, x, h1, h2, live, a1, a2);
        if (threadIdx.x < 2 * live) Y[2L * base + threadIdx.x] = y;
    }
}

// Fused inference: features of the current state (a thread per vertex), the network (kTT / kTS tiles),
// and the move of every vertex by scale * (y0 e1 + y1 e2) onto the sphere (sphericalDomain::move),
// written to the other buffer.
__global__ void __launch_bounds__(kTT) k_warm_start(const __nv_bfloat16* __restrict__ wb, FeatArgs A, int nV, double scale,
                                                    double R, double4_32a* __restrict__ posOut) {
    extern __shared__ float4 smem4[];
    float* sm = reinterpret_cast<float*>(smem4);
    float *x = sm + kWeights, *h1 = x + kTT * kSX, *h2 = h1 + kTS * kSH;
    __shared__ float ySh[2 * kTT];
    load_weights(wb, sm);
    const int v = blockIdx.x * kTT + threadIdx.x;
    D3 e1, e2, p;
    float f[kIn] = {};
    if (v < nV) vertex_features(A, v, f, e1, e2, p);
#pragma unroll
    for (int k = 0; k < kIn; ++k) x[threadIdx.x * kSX + k] = f[k];
    const int live = min(kTT, nV - (int)blockIdx.x * kTT);
    for (int base = 0; base < live; base += kTS) {
        __syncthreads();
        float a1[4][2], a2[4][2];
        const float y = tile_forward(sm, x + base * kSX, h1, h2, min(kTS, live - base), a1, a2);
        if (threadIdx.x < 2 * kTS) ySh[2 * base + threadIdx.x] = y;
    }
    __syncthreads();
    if (v >= nV) return;
    const float y0 = ySh[2 * threadIdx.x], y1 = ySh[2 * threadIdx.x + 1];
    const D3 d = add3(scl3(scale * y0, e1), scl3(scale * y1, e2));
    st3(posOut, v, sphere_move(p, d, R));
}

// The kernels' dynamic shared memory, above the default 48 KB: opted in once per device.
int mlp_opt_in() {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return SVM_ERR_CUDA;
    static std::once_flag once[64];
    static cudaError_t err[64];
    std::call_once(once[dev], [&] {
        const cudaFuncAttribute a = cudaFuncAttributeMaxDynamicSharedMemorySize;
        err[dev] = cudaFuncSetAttribute(k_train_block, a, (int)(kTrainFloats * sizeof(float)));
        if (err[dev] == cudaSuccess) err[dev] = cudaFuncSetAttribute(k_predict, a, (int)(infer_floats(kTS) * sizeof(float)));
        if (err[dev] == cudaSuccess) err[dev] = cudaFuncSetAttribute(k_warm_start, a, (int)(infer_floats(kTT) * sizeof(float)));
    });
    return err[dev] == cudaSuccess ? SVM_OK : SVM_ERR_CUDA;
}

}  // namespace

struct svm_mlp {
    cudaStream_t stream = nullptr;
    float* w = nullptr;       // FP32 master [kParams]
    float* m = nullptr;       // Adam moments
    float* v = nullptr;
    float* g = nullptr;       // gradient
    __nv_bfloat16* wb = nullptr;
    float* partials = nullptr;
    double* lossPartials = nullptr;
    double* loss = nullptr;
    int maxBlocks = 0;
    long adamStep = 0;
    double outScale = 1.0;
    float beta1 = 0.9f, beta2 = 0.999f, eps = 1e-8f;
};

// (on failure both arrays are gone and maxBlocks is 0: the next call reserves again)
static int mlp_reserve(svm_mlp* M, int blocks) {
    if (blocks <= M->maxBlocks) return SVM_OK;
    const auto release = [&] {
        cudaFree(M->partials);
        cudaFree(M->lossPartials);
        M->partials = nullptr; M->lossPartials = nullptr;
        M->maxBlocks = 0;
    };
    release();
    if (cudaMalloc(&M->partials, sizeof(float) * (size_t)blocks * kParams) != cudaSuccess ||
        cudaMalloc(&M->lossPartials, sizeof(double) * kTC * blocks) != cudaSuccess) {
        release();
        cudaGetLastError();
        return SVM_ERR_CUDA;
    }
    M->maxBlocks = blocks;
    return SVM_OK;
}

// A launch on `stream`; with `early` its blocks may be set up while the previous kernel of the stream ends (programmatic
// stream serialisation: the kernel waits for it in step_begin).
template <class... Params, class... Args>
static void launch_early(cudaStream_t stream, bool early, void (*kernel)(Params...), int grid, int block, size_t smem,
                         Args... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = early ? 1 : 0;
    (void)cudaLaunchKernelEx(&cfg, kernel, static_cast<Params>(args)...);   // (an error stays for check_launch)
}

// forward + backward over samples [first, first + count) of `order` (or of X directly): the gradient
// of sum (y - t)^2 * invBatch into M->g and the loss sum into M->loss, or, with an Adam step, the
// step taken and the loss added to M->loss
static int mlp_grad(svm_mlp* M, const float* X, const float* Y, const int* order, int first, int count,
                    float invBatch, const AdamStep* adam) {
    const int blocks = (count + kTB - 1) / kTB;
    int rc = mlp_reserve(M, blocks);
    if (rc || (rc = mlp_opt_in())) return rc;
    // In training each kernel may be set up while the previous one ends (step_begin).  (A gradient on its own may
    // follow a kernel of the caller's that writes X, which k_train_block reads ahead of that wait.)
    const bool early = adam != nullptr;
    launch_early(M->stream, early, k_train_block, kTC * blocks, kTT, kTrainFloats * sizeof(float), M->wb, X, Y, order, first,
                 count, invBatch, M->partials, M->lossPartials);
    // 64-thread blocks: the sums are chains over the partials, and 93 blocks reach most SMs
    const int nb = kParams / 64 + 1;
    if (adam)
        launch_early(M->stream, early, k_reduce_grad<true>, nb, 64, 0, M->partials, blocks, M->g, M->lossPartials, M->loss, M->w,
                     M->m, M->v, M->wb, *adam);
    else
        k_reduce_grad<false><<<nb, 64, 0, M->stream>>>(M->partials, blocks, M->g, M->lossPartials, M->loss, nullptr, nullptr,
                                                       nullptr, nullptr, AdamStep{});
    return check_launch();
}

static FeatArgs feat_args(svm_model* m) {
    FeatArgs A;
    A.pos = m->pos[m->cur]; A.vnbr = m->vnbr; A.vcell = m->vcell; A.cellPos = m->cellPos; A.ap = m->ap;
    A.pref = m->pref; A.ringCount = m->ringCount; A.force = m->force;
    return A;
}

extern "C" {

int svm_mlp_create(unsigned seed, void* stream, svm_mlp** out) {
    if (!out) return SVM_ERR_ARG;
    svm_mlp* M = new svm_mlp();
    M->stream = static_cast<cudaStream_t>(stream);
    bool ok = cudaMalloc(&M->w, sizeof(float) * kParams) == cudaSuccess &&
              cudaMalloc(&M->m, sizeof(float) * kParams) == cudaSuccess &&
              cudaMalloc(&M->v, sizeof(float) * kParams) == cudaSuccess &&
              cudaMalloc(&M->g, sizeof(float) * kParams) == cudaSuccess &&
              cudaMalloc(&M->wb, sizeof(__nv_bfloat16) * kParams) == cudaSuccess &&
              cudaMalloc(&M->loss, sizeof(double)) == cudaSuccess;
    if (!ok) { svm_mlp_destroy(M); return SVM_ERR_CUDA; }
    // He-uniform initialisation from the seed, zero biases
    std::mt19937 gen(seed);
    std::vector<float> w(kParams, 0.f);
    auto fill = [&](int off, int fanOut, int fanIn) {
        std::uniform_real_distribution<float> u(-std::sqrt(6.f / fanIn), std::sqrt(6.f / fanIn));
        for (int i = 0; i < fanOut * fanIn; ++i) w[off + i] = u(gen);
    };
    fill(oW1, kH, kIn);
    fill(oW2, kH, kH);
    fill(oW3, kOut, kH);
    for (int i = oW3; i < oW3 + kOut * kH; ++i) w[i] *= 0.1f;  // small initial outputs
    int rc = svm_mlp_set_weights(M, w.data());
    if (rc) { svm_mlp_destroy(M); return rc; }
    *out = M;
    return SVM_OK;
}

int svm_mlp_destroy(svm_mlp* M) {
    if (!M) return SVM_ERR_ARG;
    if (M->stream) cudaStreamSynchronize(M->stream);
    void* ptrs[] = {M->w, M->m, M->v, M->g, M->wb, M->partials, M->lossPartials, M->loss};
    for (void* p : ptrs) if (p) cudaFree(p);
    delete M;
    return SVM_OK;
}

int svm_mlp_parameter_count(int* n) {
    if (!n) return SVM_ERR_ARG;
    *n = kParams;
    return SVM_OK;
}

int svm_mlp_set_weights(svm_mlp* M, const float* w) {
    if (!M || !w) return SVM_ERR_ARG;
    if (cudaMemcpyAsync(M->w, w, sizeof(float) * kParams, cudaMemcpyHostToDevice, M->stream) != cudaSuccess ||
        cudaMemsetAsync(M->m, 0, sizeof(float) * kParams, M->stream) != cudaSuccess ||
        cudaMemsetAsync(M->v, 0, sizeof(float) * kParams, M->stream) != cudaSuccess)
        return SVM_ERR_CUDA;
    k_to_bf16<<<(kParams + 255) / 256, 256, 0, M->stream>>>(M->w, M->wb);
    M->adamStep = 0;
    if (check_launch()) return SVM_ERR_CUDA;
    return cudaStreamSynchronize(M->stream) == cudaSuccess ? SVM_OK : SVM_ERR_CUDA;
}

int svm_mlp_get_weights(svm_mlp* M, float* w) {
    if (!M || !w) return SVM_ERR_ARG;
    if (cudaMemcpyAsync(w, M->w, sizeof(float) * kParams, cudaMemcpyDeviceToHost, M->stream) != cudaSuccess ||
        cudaStreamSynchronize(M->stream) != cudaSuccess)
        return SVM_ERR_CUDA;
    return SVM_OK;
}

int svm_mlp_set_output_scale(svm_mlp* M, double scale) {
    if (!M || !(scale > 0)) return SVM_ERR_ARG;
    M->outScale = scale;
    return SVM_OK;
}

int svm_mlp_features(svm_model* m, float* X, double* frames) {
    if (!m || !X || m->precision == SVM_PRECISION_MIXED) return SVM_ERR_ARG;
    k_features<<<(m->nVertices + 255) / 256, 256, 0, m->stream>>>(feat_args(m), m->nVertices, X, frames);
    if (check_launch()) return SVM_ERR_CUDA;
    return cudaStreamSynchronize(m->stream) == cudaSuccess ? SVM_OK : SVM_ERR_CUDA;
}

int svm_mlp_gradient(svm_mlp* M, const float* X, const float* Y, int n, float* grad, double* loss) {
    if (!M || !X || !Y || n <= 0 || !grad) return SVM_ERR_ARG;
    int rc = mlp_grad(M, X, Y, nullptr, 0, n, 1.f / n, nullptr);
    if (rc) return rc;
    if (cudaMemcpyAsync(grad, M->g, sizeof(float) * kParams, cudaMemcpyDeviceToHost, M->stream) != cudaSuccess)
        return SVM_ERR_CUDA;
    double l = 0.0;
    if (cudaMemcpyAsync(&l, M->loss, sizeof(double), cudaMemcpyDeviceToHost, M->stream) != cudaSuccess ||
        cudaStreamSynchronize(M->stream) != cudaSuccess)
        return SVM_ERR_CUDA;
    if (loss) *loss = l / n;
    return SVM_OK;
}

int svm_mlp_train(svm_mlp* M, const float* X, const float* Y, const int* order, int n, int batch, float learningRate,
                  double* meanLoss) {
    if (!M || !X || !Y || !order || n <= 0 || batch <= 0) return SVM_ERR_ARG;
    if (cudaMemsetAsync(M->loss, 0, sizeof(double), M->stream) != cudaSuccess) return SVM_ERR_CUDA;
    for (int first = 0; first < n; first += batch) {
        const int count = std::min(batch, n - first);
        const long step = M->adamStep + 1;
        AdamStep A{learningRate, M->beta1, M->beta2, M->eps, 0.f, 0.f};
        A.c1 = 1.f - std::pow(M->beta1, (float)step);
        A.c2 = 1.f - std::pow(M->beta2, (float)step);
        if (int rc = mlp_grad(M, X, Y, order, first, count, 1.f / count, &A)) return rc;
        M->adamStep = step;
    }
    double total = 0.0;
    if (meanLoss && cudaMemcpyAsync(&total, M->loss, sizeof(double), cudaMemcpyDeviceToHost, M->stream) != cudaSuccess)
        return SVM_ERR_CUDA;
    if (cudaStreamSynchronize(M->stream) != cudaSuccess) return SVM_ERR_CUDA;
    if (meanLoss) *meanLoss = total / n;
    return SVM_OK;
}

int svm_mlp_predict(svm_mlp* M, const float* X, int n, float* Y) {
    if (!M || !X || !Y || n <= 0) return SVM_ERR_ARG;
    if (int rc = mlp_opt_in()) return rc;
    // four resident blocks per SM (47 KB of shared memory each), each over several tiles at large n
    const int tiles = (n + kTS - 1) / kTS;
    k_predict<<<std::min(tiles, 4 * 152), kTT, infer_floats(kTS) * sizeof(float), M->stream>>>(M->wb, X, n, Y);
    if (check_launch()) return SVM_ERR_CUDA;
    return cudaStreamSynchronize(M->stream) == cudaSuccess ? SVM_OK : SVM_ERR_CUDA;
}

int svm_mlp_warm_start(svm_mlp* M, svm_model* m) {
    if (!M || !m || m->precision == SVM_PRECISION_MIXED) return SVM_ERR_ARG;
    if (cudaStreamSynchronize(M->stream) != cudaSuccess) return SVM_ERR_CUDA;  // training done
    // geometry and forces of the current state feed the features
    int rc = svm_model_compute_forces(m);
    if (rc) return rc;
    const int nxt = 1 - m->cur;
    if ((rc = mlp_opt_in())) return rc;
    k_warm_start<<<(m->nVertices + kTT - 1) / kTT, kTT, infer_floats(kTT) * sizeof(float), m->stream>>>(
        M->wb, feat_args(m), m->nVertices, M->outScale, m->R, m->pos[nxt]);
    if (check_launch()) return SVM_ERR_CUDA;
    m->cur = nxt;
    m->cornersValid = false;
    m->paramsVersion++;  // captured graphs hold the old buffer roles
    return cudaStreamSynchronize(m->stream) == cudaSuccess ? SVM_OK : SVM_ERR_CUDA;
}

}  // extern "C"
