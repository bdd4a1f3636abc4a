// Learned preconditioner: a message-passing network over the Newton
// matrix's 3x3-block graph that emits a lower block-triangular factor G on
// the IC(0) pattern (the lower block pattern of the matrix itself) of the
// block-Jacobi-scaled matrix
//     Â = S A S^T,  S_i = L_i^-1,  D_i = L_i L_i^T (assembled diagonal block),
// used as a factorised sparse approximate inverse
//     M^-1 = S^T G^T G S        (G = I gives block-Jacobi exactly),
// so applying it is two sparse products over the existing block pattern.
// G is lower triangular with a positive diagonal (softplus), so M^-1 is SPD
// for any weights.
//
// Training minimises the Kaporin condition number of B = G Â G^T,
//     L = log(tr(B)/n) - (2/n) sum_q log G_qq,
// with tr(B)/n estimated from probe vectors w as mean w^T B w / w^T w; the
// minimiser of L over the pattern is the factorised sparse approximate
// inverse of that pattern.  Forward and backward kernels are hand-written;
// the weights are used in BF16 with FP32 accumulation, FP32 masters are
// updated by Adam.
//
// Graph: nodes are vertices; edges are the lower off-diagonal block slots
// (col < row) of the static BSR and of the contact BSR.  Each edge keeps its
// factor block in its own slot and the transpose in the mirror slot (row and
// column swapped), so G x and G^T x are both row-wise products.
//
// No counterpart in CPU-IPC; the closest is the Eigen IncompleteCholesky
// option of NewtonLinearSystem::solve (CPU IPC/NewtonLinearSystem.cpp:186-192).
#include "cipc_device.cuh"
#include "cipc_internal.h"
#include "mpnn.h"
#include "dense_tc.cuh"

#include <cuda_bf16.h>
#include <cub/cub.cuh>

#include <algorithm>
#include <cmath>
#include <string>
#include <vector>

namespace cipc {

namespace {

constexpr int TB = 128;
inline int blocksFor(int n, int tb = TB) { return std::max(1, std::min((n + tb - 1) / tb, 148 * 32)); }

typedef __nv_bfloat16 bf16;
__device__ __forceinline__ float W(const bf16* w, int i) { return __bfloat162float(w[i]); }
__device__ __forceinline__ float relu(float x) { return x > 0.f ? x : 0.f; }
__device__ __forceinline__ float softplus(float x) { return x > 20.f ? x : log1pf(expf(x)); }
__device__ __forceinline__ float sigmoidf(float x) { return 1.f / (1.f + expf(-x)); }

// ---------------------------------------------------------------------------
// scaling and features
// ---------------------------------------------------------------------------
template <class MT>
__device__ void diagBlock(int v, const int* diagSlot, const MT* val, const int* dRowS, const int* dRowE, const int* dCol, const MT* dVal,
                          const double* diagExtra, double D[9], double C[9]) {
    for (int k = 0; k < 9; ++k) { D[k] = diagExtra[9 * v + k]; C[k] = 0.0; }
    int s = diagSlot[v];
    if (s >= 0) for (int k = 0; k < 9; ++k) D[k] += (double)val[(size_t)9 * s + k];
    if (dRowS)
        for (int k = dRowS[v]; k < dRowE[v]; ++k)
            if (dCol[k] == v)
                for (int q = 0; q < 9; ++q) { D[q] += (double)dVal[(size_t)9 * k + q]; C[q] += (double)dVal[(size_t)9 * k + q]; }
}

// S = L^-1 of the Cholesky factor of D (lower entries used); diagonal
// scaling if D is not positive definite.
__device__ void invChol(const double D[9], double S[9]) {
    for (int k = 0; k < 9; ++k) S[k] = 0.0;
    double a00 = D[0], a10 = D[3], a11 = D[4], a20 = D[6], a21 = D[7], a22 = D[8];
    bool ok = a00 > 0;
    double l00 = 0, l10 = 0, l20 = 0, l11 = 0, l21 = 0, l22 = 0;
    if (ok) { l00 = sqrt(a00); l10 = a10 / l00; l20 = a20 / l00; double t = a11 - l10 * l10; ok = t > 0; if (ok) l11 = sqrt(t); }
    if (ok) { l21 = (a21 - l20 * l10) / l11; double t = a22 - l20 * l20 - l21 * l21; ok = t > 0; if (ok) l22 = sqrt(t); }
    if (ok && isfinite(l22)) {
        S[0] = 1 / l00; S[4] = 1 / l11; S[8] = 1 / l22;
        S[3] = -l10 / (l00 * l11);
        S[7] = -l21 / (l11 * l22);
        S[6] = (l10 * l21 - l11 * l20) / (l00 * l11 * l22);
    } else {
        for (int q = 0; q < 3; ++q) S[4 * q] = D[4 * q] > 0 ? 1.0 / sqrt(D[4 * q]) : 1.0;
    }
}

// out = S_i B S_j^T (B row-major 3x3, S lower-triangular row-major)
template <class MT>
__device__ __forceinline__ void scaleBlock(const double* Si, const MT* B, const double* Sj, double out[9]) {
    double T[9];
    for (int a = 0; a < 3; ++a)
        for (int b = 0; b < 3; ++b) T[3 * a + b] = Si[3 * a] * (double)B[b] + Si[3 * a + 1] * (double)B[3 + b] + Si[3 * a + 2] * (double)B[6 + b];
    for (int a = 0; a < 3; ++a)
        for (int d = 0; d < 3; ++d) out[3 * a + d] = T[3 * a] * Sj[3 * d] + T[3 * a + 1] * Sj[3 * d + 1] + T[3 * a + 2] * Sj[3 * d + 2];
}

template <class MT>
__global__ void scaleKernel(int nv, const int* diagSlot, const MT* val, const int* dRowS, const int* dRowE, const int* dCol, const MT* dVal,
                            const double* diagExtra, double* S, float* f5) {
    CIPC_KERNEL_LOOP(v, nv) {
        double D[9], C[9], Sv[9];
        diagBlock(v, diagSlot, val, dRowS, dRowE, dCol, dVal, diagExtra, D, C);
        invChol(D, Sv);
        for (int k = 0; k < 9; ++k) S[9 * v + k] = Sv[k];
        double sc[9];
        scaleBlock(Sv, C, Sv, sc);
        f5[v] = (float)((sc[0] + sc[4] + sc[8]) / 3.0);
    }
}

// per row: sums / max / counts of |Â_vc|_F over off-diagonal slots
template <class MT>
__global__ void nodeFeatKernel(int nv, const int* rowPtr, const int* col, const MT* val, const int* dRowS, const int* dRowE, const int* dCol,
                               const MT* dVal, const double* S, const float* f5, float* f) {
    CIPC_KERNEL_LOOP(v, nv) {
        double sumS = 0, sumD = 0, mx = 0;
        int degS = 0, degD = 0;
        for (int k = rowPtr[v]; k < rowPtr[v + 1]; ++k) {
            int c = col[k];
            if (c == v) continue;
            double b[9];
            scaleBlock(S + 9 * v, val + (size_t)9 * k, S + 9 * c, b);
            double n = 0;
            for (int q = 0; q < 9; ++q) n += b[q] * b[q];
            n = sqrt(n);
            sumS += n; mx = fmax(mx, n); ++degS;
        }
        if (dRowS)
            for (int k = dRowS[v]; k < dRowE[v]; ++k) {
                int c = dCol[k];
                if (c == v) continue;
                double b[9];
                scaleBlock(S + 9 * v, dVal + (size_t)9 * k, S + 9 * c, b);
                double n = 0;
                for (int q = 0; q < 9; ++q) n += b[q] * b[q];
                n = sqrt(n);
                sumD += n; mx = fmax(mx, n); ++degD;
            }
        float* o = f + MPNN_NF * v;
        o[0] = (float)sumS; o[1] = (float)sumD; o[2] = (float)mx;
        o[3] = log1pf((float)degS); o[4] = log1pf((float)degD); o[5] = f5[v];
    }
}

// edge features Â_ij (9, row-major) for lower slots of a row-ranged pattern
template <class MT>
__global__ void edgeFeatKernel(int nv, const int* rowS, const int* rowE, const int* col, const MT* val, const double* S, float* g) {
    CIPC_KERNEL_LOOP(v, nv) {
        for (int k = rowS[v]; k < rowE[v]; ++k) {
            int c = col[k];
            if (c >= v) continue;
            double b[9];
            scaleBlock(S + 9 * v, val + (size_t)9 * k, S + 9 * c, b);
            for (int q = 0; q < 9; ++q) g[(size_t)9 * k + q] = (float)b[q];
        }
    }
}

// mirror slot of (row, col) = slot of (col, row) in a column-sorted pattern
__global__ void mirrorKernel(int nv, const int* rowS, const int* rowE, const int* col, int* mirror) {
    CIPC_KERNEL_LOOP(v, nv) {
        for (int k = rowS[v]; k < rowE[v]; ++k) {
            int c = col[k];
            int lo = rowS[c], hi = rowE[c];
            while (lo < hi) {
                int mid = (lo + hi) >> 1;
                if (col[mid] < v) lo = mid + 1; else hi = mid;
            }
            mirror[k] = (lo < rowE[c] && col[lo] == v) ? lo : -1;
        }
    }
}
__global__ void rowRangeKernel(int nv, const int* rowPtr, int* rs, int* re) {
    CIPC_KERNEL_LOOP(v, nv) { rs[v] = rowPtr[v]; re[v] = rowPtr[v + 1]; }
}

__global__ void degreeKernel(int nv, const int* rowPtr, const int* col, const int* mirS, const int* dRowS, const int* dRowE, const int* dCol,
                             const int* mirD, int* deg) {
    CIPC_KERNEL_LOOP(v, nv) {
        int d = 0;
        for (int k = rowPtr[v]; k < rowPtr[v + 1]; ++k) {
            int c = col[k];
            if (c != v && (c < v || mirS[k] >= 0)) ++d;
        }
        if (dRowS)
            for (int k = dRowS[v]; k < dRowE[v]; ++k) {
                int c = dCol[k];
                if (c != v && (c < v || mirD[k] >= 0)) ++d;
            }
        deg[v] = d;
    }
}

// mean of incident edge states; an edge is read at its lower slot
// Mean of the incident edges' features, one warp per vertex: lane t sums
// feature t over the row's static slots, then its contact slots, in slot
// order (one coalesced 128-byte row per edge).  Each lane first resolves one
// slot of the row (its lower-slot index, or -1 for the diagonal and for
// blocks without an edge), and the warp walks them with shuffles.
__device__ __forceinline__ float aggregateRange(float a, int v, int k0, int k1, const int* col, const int* mir, const float* e, int lane) {
    for (int c0 = k0; c0 < k1; c0 += 32) {
        const int k = c0 + lane;
        int slot = -1;
        if (k < k1) {
            const int c = col[k];
            slot = c == v ? -1 : (c < v ? k : mir[k]);
        }
        const int m = min(32, k1 - c0);
        for (int j = 0; j < m; ++j) {
            const int sj = __shfl_sync(0xffffffffu, slot, j);
            if (sj >= 0) a += e[(size_t)MPNN_H * sj + lane];
        }
    }
    return a;
}

__global__ void aggregateKernel(int nv, const int* rowPtr, const int* col, const int* mirS, const float* eS, const int* dRowS, const int* dRowE,
                                const int* dCol, const int* mirD, const float* eD, const int* deg, float* agg) {
    const int lane = threadIdx.x & 31;
    const int warps = gridDim.x * blockDim.x / 32;
    for (int v = (blockIdx.x * blockDim.x + threadIdx.x) / 32; v < nv; v += warps) {
        float a = aggregateRange(0.f, v, rowPtr[v], rowPtr[v + 1], col, mirS, eS, lane);
        if (dRowS) a = aggregateRange(a, v, dRowS[v], dRowE[v], dCol, mirD, eD, lane);
        const float inv = deg[v] > 0 ? 1.f / deg[v] : 0.f;
        agg[(size_t)MPNN_H * v + lane] = a * inv;
    }
}

// ---------------------------------------------------------------------------
// Tiled dense layers of the forward pass.  A CTA stages one weight matrix
// (transposed, FP32 from the BF16 copy) and a tile of DT_ITEMS input rows in
// shared memory; two threads per item split the outputs and accumulate in
// FP32 registers.  Items are nodes or the lower edges of a flat edge list;
// gather and emit functors read the layer's inputs and write its outputs.
// ---------------------------------------------------------------------------
constexpr int DT_ITEMS = 64;
constexpr int DT_THREADS = 2 * DT_ITEMS;

template <int IN, int OUT, class G, class E>
__global__ void __launch_bounds__(DT_THREADS) denseTiledKernel(int n, G gather, E emit, const bf16* Wm, const bf16* bias) {
    constexpr int HALF = (OUT + 1) / 2;
    __shared__ float sW[IN][OUT + 1];
    __shared__ float sB[OUT];
    __shared__ float sX[DT_ITEMS][IN + 1];
    for (int t = threadIdx.x; t < IN * OUT; t += DT_THREADS) sW[t % IN][t / IN] = W(Wm, t);
    for (int t = threadIdx.x; t < OUT; t += DT_THREADS) sB[t] = W(bias, t);
    for (int base = blockIdx.x * DT_ITEMS; base < n; base += gridDim.x * DT_ITEMS) {
        __syncthreads();
        for (int t = threadIdx.x; t < DT_ITEMS * IN; t += DT_THREADS) {
            int r = t / IN, i = t % IN, item = base + r;
            sX[r][i] = item < n ? gather(item, i) : 0.f;
        }
        __syncthreads();
        const int r = threadIdx.x >> 1, h = threadIdx.x & 1, item = base + r;
        float acc[HALF];
#pragma unroll
        for (int q = 0; q < HALF; ++q) {
            int o = h * HALF + q;
            acc[q] = o < OUT ? sB[o] : 0.f;
        }
        for (int i = 0; i < IN; ++i) {
            float x = sX[r][i];
#pragma unroll
            for (int q = 0; q < HALF; ++q) {
                int o = h * HALF + q;
                if (o < OUT) acc[q] += sW[i][o] * x;
            }
        }
        if (item < n) {
#pragma unroll
            for (int q = 0; q < HALF; ++q) {
                int o = h * HALF + q;
                if (o < OUT) emit(item, o, acc[q]);
            }
        }
    }
}

// flat list of the lower edges of a row-ranged pattern
__global__ void lowerCountKernel(int nv, const int* rowS, const int* rowE, const int* col, int* cnt) {
    CIPC_KERNEL_LOOP(v, nv) {
        int k = 0;
        for (int s = rowS[v]; s < rowE[v]; ++s) k += col[s] < v;
        cnt[v] = k;
    }
}
// edgeOf[slot]: the lower slot's place in the list, -1 for the other slots
__global__ void lowerFillKernel(int nv, const int* rowS, const int* rowE, const int* col, const int* off, int* eSlot, int* eI, int* eJ, int* edgeOf) {
    CIPC_KERNEL_LOOP(v, nv) {
        int o = off[v];
        for (int s = rowS[v]; s < rowE[v]; ++s) {
            const bool low = col[s] < v;
            edgeOf[s] = low ? o : -1;
            if (low) { eSlot[o] = s; eI[o] = v; eJ[o] = col[s]; ++o; }
        }
    }
}

struct NodeFeatGather {
    const float* f;
    __device__ float operator()(int v, int i) const { return f[MPNN_NF * v + i]; }
};
struct EdgeFeatGather {
    const int* slot;
    const float* g;
    __device__ float operator()(int e, int i) const { return g[(size_t)9 * slot[e] + i]; }
};
struct EdgeLayerGather {  // [e_l ; h_i + h_j]
    const int *slot, *ei, *ej;
    const float *e, *h;
    // tensor-core layer: an edge's slot and end vertices, and its inputs
    // lane and MPNN_H + lane
    struct Idx {
        int s, i, j;
    };
    __device__ Idx index(int k) const { return Idx{slot[k], ei[k], ej[k]}; }
    __device__ static Idx shfl(const Idx& x, int src) {
        return Idx{__shfl_sync(0xffffffffu, x.s, src), __shfl_sync(0xffffffffu, x.i, src), __shfl_sync(0xffffffffu, x.j, src)};
    }
    __device__ float2 pair(const Idx& x, int lane) const {
        return make_float2(e[(size_t)MPNN_H * x.s + lane], h[(size_t)MPNN_H * x.i + lane] + h[(size_t)MPNN_H * x.j + lane]);
    }
};
struct NodeLayerGather {  // [h ; agg]
    const float *h, *agg;
    struct Idx {
        int v;
    };
    __device__ Idx index(int v) const { return Idx{v}; }
    __device__ static Idx shfl(const Idx& x, int src) { return Idx{__shfl_sync(0xffffffffu, x.v, src)}; }
    __device__ float2 pair(const Idx& x, int lane) const {
        return make_float2(h[(size_t)MPNN_H * x.v + lane], agg[(size_t)MPNN_H * x.v + lane]);
    }
};
struct HeadEdgeGather {  // [e_L ; g]
    const int* slot;
    const float *e, *g;
    __device__ float operator()(int k, int i) const {
        return i < MPNN_H ? e[(size_t)MPNN_H * slot[k] + i] : g[(size_t)9 * slot[k] + i - MPNN_H];
    }
};
struct NodeHiddenGather {
    const float* h;
    __device__ float operator()(int v, int i) const { return h[(size_t)MPNN_H * v + i]; }
};

__device__ __forceinline__ void reluStore32(float* dst, const float v[32]) {
    float4* p = reinterpret_cast<float4*>(dst);
#pragma unroll
    for (int o = 0; o < 8; ++o) p[o] = make_float4(relu(v[4 * o]), relu(v[4 * o + 1]), relu(v[4 * o + 2]), relu(v[4 * o + 3]));
}
struct ReluEmitNode {
    float* out;
    __device__ void operator()(int v, int o, float a) const { out[(size_t)MPNN_H * v + o] = relu(a); }
    __device__ void emit32(int v, const float a[32]) const { reluStore32(out + (size_t)MPNN_H * v, a); }
};
struct ReluEmitEdge {
    const int* slot;
    float* out;
    __device__ void operator()(int k, int o, float a) const { out[(size_t)MPNN_H * slot[k] + o] = relu(a); }
    __device__ void emit32(int k, const float a[32]) const { reluStore32(out + (size_t)MPNN_H * slot[k], a); }
};
// G_ij into the lower slot and G_ij^T into its mirror; no block touches a
// Dirichlet vertex
struct HeadEdgeEmit {
    const int *slot, *ei, *ej, *mirror, *btype;
    float* gOut;
    __device__ void operator()(int k, int o, float a) const {
        const int s = slot[k];
        const float v = (btype[ei[k]] == 0 && btype[ej[k]] == 0) ? a : 0.f;
        gOut[(size_t)9 * s + o] = v;
        const int m = mirror[s];
        if (m >= 0) gOut[(size_t)9 * m + 3 * (o % 3) + o / 3] = v;
    }
};
// G_ii: lower triangle, softplus diagonal; Dirichlet vertices keep I
struct HeadDiagEmit {
    const int *diagSlot, *btype;
    float *gS, *headD;
    __device__ void operator()(int v, int o, float a) const {
        headD[6 * v + o] = a;
        float* G = gS + (size_t)9 * diagSlot[v];
        const bool fixedV = btype[v] != 0;
        const int pos[6] = {0, 4, 8, 3, 6, 7};
        float val = o < 3 ? softplus(a) : a;
        if (fixedV) val = o < 3 ? 1.f : 0.f;
        G[pos[o]] = val;
        if (o == 0) { G[1] = 0.f; G[2] = 0.f; G[5] = 0.f; }
    }
};

// ---------------------------------------------------------------------------
// factor and scaled operator products of all probe vectors at once (FP32
// vectors, planes of 3 nv): one thread per row and probe, the probes of a row
// in neighbouring lanes, so that a block is fetched once for all of them
//
// ---------------------------------------------------------------------------
// y = G u (transpose = 0: lower slots + diagonal) or y = G^T u (mirror slots + transposed diagonal)
__global__ void factorApplyKernel(int nv, int probes, int transpose, const int* rowPtr, const int* col, const float* gS, const int* dRowS, const int* dRowE,
                                  const int* dCol, const float* gD, const float* uAll, float* yAll) {
    CIPC_KERNEL_LOOP(i, nv * probes) {
        const int v = i / probes;
        const size_t plane = (size_t)(i - v * probes) * 3 * nv;
        const float* u = uAll + plane;
        float* y = yAll + plane;
        float acc[3] = {0.f, 0.f, 0.f};
        for (int k = rowPtr[v]; k < rowPtr[v + 1]; ++k) {
            int c = col[k];
            if (transpose ? c < v : c > v) continue;
            const float* B = gS + (size_t)9 * k;
            float x0 = u[3 * c], x1 = u[3 * c + 1], x2 = u[3 * c + 2];
            if (transpose && c == v)
                for (int a = 0; a < 3; ++a) acc[a] += B[a] * x0 + B[3 + a] * x1 + B[6 + a] * x2;
            else
                for (int a = 0; a < 3; ++a) acc[a] += B[3 * a] * x0 + B[3 * a + 1] * x1 + B[3 * a + 2] * x2;
        }
        if (dRowS)
            for (int k = dRowS[v]; k < dRowE[v]; ++k) {
                int c = dCol[k];
                if (transpose ? c <= v : c >= v) continue;
                const float* B = gD + (size_t)9 * k;
                float x0 = u[3 * c], x1 = u[3 * c + 1], x2 = u[3 * c + 2];
                for (int a = 0; a < 3; ++a) acc[a] += B[3 * a] * x0 + B[3 * a + 1] * x1 + B[3 * a + 2] * x2;
            }
        for (int a = 0; a < 3; ++a) y[3 * v + a] = acc[a];
    }
}

// y = Â u = S A S^T u
template <class MT>
__global__ void scaledSpmvKernel(int nv, int probes, const int* rowPtr, const int* col, const MT* val, const int* dRowS, const int* dRowE,
                                 const int* dCol, const MT* dVal, const double* diagExtra, const double* S, const float* uAll, float* yAll) {
    CIPC_KERNEL_LOOP(i, nv * probes) {
        const int v = i / probes;
        const size_t plane = (size_t)(i - v * probes) * 3 * nv;
        const float* u = uAll + plane;
        float* y = yAll + plane;
        double acc[3] = {0, 0, 0};
        auto stu = [&](int c, double x[3]) {
            // S_c^T u_c (S_c lower triangular)
            const double* Sc = S + 9 * c;
            double u0 = u[3 * c], u1 = u[3 * c + 1], u2 = u[3 * c + 2];
            x[0] = Sc[0] * u0 + Sc[3] * u1 + Sc[6] * u2;
            x[1] = Sc[4] * u1 + Sc[7] * u2;
            x[2] = Sc[8] * u2;
        };
        for (int k = rowPtr[v]; k < rowPtr[v + 1]; ++k) {
            double x[3];
            stu(col[k], x);
            const MT* B = val + (size_t)9 * k;
            for (int a = 0; a < 3; ++a) acc[a] += (double)B[3 * a] * x[0] + (double)B[3 * a + 1] * x[1] + (double)B[3 * a + 2] * x[2];
        }
        if (dRowS)
            for (int k = dRowS[v]; k < dRowE[v]; ++k) {
                double x[3];
                stu(dCol[k], x);
                const MT* B = dVal + (size_t)9 * k;
                for (int a = 0; a < 3; ++a) acc[a] += (double)B[3 * a] * x[0] + (double)B[3 * a + 1] * x[1] + (double)B[3 * a + 2] * x[2];
            }
        {
            double x[3];
            stu(v, x);
            const double* B = diagExtra + 9 * v;
            for (int a = 0; a < 3; ++a) acc[a] += B[3 * a] * x[0] + B[3 * a + 1] * x[1] + B[3 * a + 2] * x[2];
        }
        const double* Sv = S + 9 * v;
        y[3 * v] = (float)(Sv[0] * acc[0]);
        y[3 * v + 1] = (float)(Sv[3] * acc[0] + Sv[4] * acc[1]);
        y[3 * v + 2] = (float)(Sv[6] * acc[0] + Sv[7] * acc[1] + Sv[8] * acc[2]);
    }
}

// probe vectors: four summed uniforms from a splitmix64 stream, unit variance
__global__ void probeKernel(int n, unsigned long long seed, float* w) {
    CIPC_KERNEL_LOOP(i, n) {
        unsigned long long z = seed + 0x9E3779B97F4A7C15ull * (unsigned long long)(i + 1);
        float s = 0.f;
        for (int k = 0; k < 4; ++k) {
            z ^= z >> 30; z *= 0xBF58476D1CE4E5B9ull; z ^= z >> 27; z *= 0x94D049BB133111EBull; z ^= z >> 31;
            s += (float)(z >> 40) * (1.0f / 16777216.0f) - 0.5f;
        }
        w[i] = s * 1.7320508f;
    }
}

// partials of u.v and w.w of probe blockIdx.y (planes of n)
__global__ void probeDotsKernel(int n, const float* uAll, const float* vAll, const float* wAll, double* partAll) {
    const size_t plane = (size_t)blockIdx.y * n;
    const float *u = uAll + plane, *v = vAll + plane, *w = wAll + plane;
    double* part = partAll + (size_t)2 * gridDim.x * blockIdx.y;
    double uv = 0, ww = 0;
    CIPC_KERNEL_LOOP(i, n) {
        uv += (double)u[i] * (double)v[i];
        ww += (double)w[i] * (double)w[i];
    }
    double a = blockReduce(uv, AddOp(), 0.0);
    __syncthreads();
    double b = blockReduce(ww, AddOp(), 0.0);
    if (threadIdx.x == 0) { part[2 * blockIdx.x] = a; part[2 * blockIdx.x + 1] = b; }
}

// partial sums of log G_qq over the diagonal blocks
__global__ void logDiagKernel(int nv, const int* diagSlot, const float* gS, double* part) {
    double s = 0;
    CIPC_KERNEL_LOOP(v, nv) {
        const float* G = gS + (size_t)9 * diagSlot[v];
        s += log((double)G[0]) + log((double)G[4]) + log((double)G[8]);
    }
    double a = blockReduce(s, AddOp(), 0.0);
    if (threadIdx.x == 0) part[blockIdx.x] = a;
}

// The loss's gradient with respect to G, (1/T) sum over probes of
// scale w_i v_j^T, a chunk of probes at a time (first: nothing is summed yet;
// mul: 1/T with the last chunk, else 1): on the lower slots one thread per edge
// and entry, the probes in their order, ...
__global__ void factorGradEdgeKernel(int n, const int* slot, const int* ei, const int* ej, const int* btype, int probes, int n3, const float* w,
                                     const float* vv, const float* scale, bool first, float mul, float* dG) {
    CIPC_KERNEL_LOOP(t, 9 * n) {
        const int e = t / 9, q = t - 9 * e, a = q / 3, b = q - 3 * a;
        const int i = ei[e], j = ej[e];
        float* o = dG + (size_t)9 * slot[e] + q;
        float s = first ? 0.f : *o;
        if (btype[i] == 0 && btype[j] == 0)
            for (int p = 0; p < probes; ++p) s += scale[p] * w[(size_t)p * n3 + 3 * i + a] * vv[(size_t)p * n3 + 3 * j + b];
        *o = s * mul;
    }
}
// ... and on the diagonal slots' lower triangles (zero above), where the log
// term adds -(2/n) / G_qq on the free vertices.
__global__ void factorGradDiagKernel(int nv, const int* diagSlot, const int* btype, int probes, int n3, const float* w, const float* vv,
                                     const float* scale, bool first, float mul, bool last, const float* gS, float coef, float* dG) {
    CIPC_KERNEL_LOOP(t, 9 * nv) {
        const int v = t / 9, q = t - 9 * v, a = q / 3, b = q - 3 * a;
        const size_t o = (size_t)9 * diagSlot[v] + q;
        float s = first ? 0.f : dG[o];
        if (btype[v] == 0 && b <= a) {
            for (int p = 0; p < probes; ++p) s += scale[p] * w[(size_t)p * n3 + 3 * v + a] * vv[(size_t)p * n3 + 3 * v + b];
            s *= mul;
            if (last && a == b) s -= coef / gS[o];
        }
        dG[o] = s;
    }
}

// ---------------------------------------------------------------------------
// backward
//
// Each layer's backward runs in two parts over items: nodes, or the edges of
// the flat lower-edge lists (edge states of the forward pass are read at the
// edge's slot, gradients are stored by edge).  An item kernel forms the
// pre-activation gradient d (written to D[item][OUT]) and propagates W^T d to
// the layer's inputs.  Every row of 32 values is read and written by 32
// neighbouring lanes; one thread per matrix row walking its edges with
// strided rows took most of an evaluation (loss and gradient, 4 probes, 8-cube
// pile, 17,596 vertices: 5.68 -> 1.46 ms on a B200).  Bound now: launches of
// 5-20 us each, the weight gradients among them.  The weight gradient dW = D^T X and db = sum D is then
// a split-K reduction over the items: each CTA stages TI items of D and X in
// shared memory and accumulates its share of the OUT x IN outputs in
// registers, writes one partial per output, and a second kernel sums the
// partials in CTA order - deterministic and free of atomics.
// ---------------------------------------------------------------------------
constexpr int WG_TI = 32;        // items per shared-memory tile
constexpr int WG_THREADS = 256;
constexpr int WG_GRID = 296;     // CTAs of the split-K reduction (2 per SM)

// X = [X1 (IN1 columns) ; X2 (IN2 columns)] per item; dItem and xItem are the
// rows of D and of X1, X2 that belong to an item (null: the item's number).
// partial[cta][OUT*(IN1+IN2) + OUT].  The heads and the embeddings (the
// tensor-core layers use weightGradTcKernel).
template <int OUT, int IN1, int IN2>
__global__ void __launch_bounds__(WG_THREADS) weightGradKernel(int items, const float* D, const int* dItem, const float* X1, const float* X2,
                                                               const int* xItem, float* partial) {
    constexpr int IN = IN1 + IN2;
    constexpr int NW = OUT * IN + OUT;
    constexpr int PER = (NW + WG_THREADS - 1) / WG_THREADS;
    __shared__ float sD[WG_TI][OUT];
    __shared__ float sX[WG_TI][IN + 1];
    float acc[PER];
    for (int q = 0; q < PER; ++q) acc[q] = 0.f;
    for (int base = blockIdx.x * WG_TI; base < items; base += gridDim.x * WG_TI) {
        __syncthreads();
        for (int t = threadIdx.x; t < WG_TI * OUT; t += WG_THREADS) {
            int it = base + t / OUT, o = t % OUT;
            sD[t / OUT][o] = it < items ? D[(size_t)(dItem ? dItem[it] : it) * OUT + o] : 0.f;
        }
        for (int t = threadIdx.x; t < WG_TI * IN; t += WG_THREADS) {
            int r = t / IN, i = t % IN, it = base + r;
            float v = 0.f;
            if (it < items) {
                const size_t row = xItem ? xItem[it] : it;
                v = i < IN1 ? X1[row * IN1 + i] : X2[row * IN2 + (i - IN1)];
            }
            sX[r][i] = v;
        }
        __syncthreads();
        for (int q = 0; q < PER; ++q) {
            int idx = threadIdx.x + q * WG_THREADS;
            if (idx >= NW) break;
            float s = 0.f;
            if (idx < OUT * IN) {
                int o = idx / IN, i = idx % IN;
#pragma unroll 8
                for (int r = 0; r < WG_TI; ++r) s += sD[r][o] * sX[r][i];
            } else {
                int o = idx - OUT * IN;
#pragma unroll 8
                for (int r = 0; r < WG_TI; ++r) s += sD[r][o];
            }
            acc[q] += s;
        }
    }
    for (int q = 0; q < PER; ++q) {
        int idx = threadIdx.x + q * WG_THREADS;
        if (idx < NW) partial[(size_t)blockIdx.x * NW + idx] = acc[q];
    }
}

// gW[w] += sum over CTAs of partial (weights, then `out` biases).  WR_SPLIT
// threads share a weight, each adds every WR_SPLIT-th CTA, and their sums are
// added in a fixed order: a thread that read all 296 partials one after the
// other took 33 us.
constexpr int WR_OUT = 32, WR_SPLIT = 8;
__global__ void __launch_bounds__(WR_OUT * WR_SPLIT) weightGradReduceKernel(int nw, int out, int ctas, const float* partial, float* gW, float* gB) {
    __shared__ float sh[WR_SPLIT][WR_OUT];
    const int o = threadIdx.x % WR_OUT, part = threadIdx.x / WR_OUT, idx = blockIdx.x * WR_OUT + o;
    float s = 0.f;
    if (idx < nw)
        for (int g = part; g < ctas; g += WR_SPLIT) s += partial[(size_t)g * nw + idx];
    sh[part][o] = s;
    __syncthreads();
    if (part == 0 && idx < nw) {
        for (int k = 1; k < WR_SPLIT; ++k) s += sh[k][o];
        if (idx < nw - out) gW[idx] += s;
        else gB[idx - (nw - out)] += s;
    }
}

// one warp per node: lane t forms component t of W^T d
__global__ void headDiagBackKernel(int nv, const float* headD, const int* diagSlot, const float* dGS, const bf16* w, float* D6, float* dhL) {
    const int lane = threadIdx.x & 31, warps = gridDim.x * blockDim.x / 32;
    float wt[6];
    for (int q = 0; q < 6; ++q) wt[q] = W(w + MP_WD, q * MPNN_H + lane);
    for (int v = (blockIdx.x * blockDim.x + threadIdx.x) / 32; v < nv; v += warps) {
        const float* dB = dGS + (size_t)9 * diagSlot[v];
        const float* o = headD + 6 * (size_t)v;
        const float d[6] = {dB[0] * sigmoidf(o[0]), dB[4] * sigmoidf(o[1]), dB[8] * sigmoidf(o[2]), dB[3], dB[6], dB[7]};
        float dh = 0.f;
        for (int q = 0; q < 6; ++q) dh += d[q] * wt[q];
        float mine = d[0];
        for (int q = 1; q < 6; ++q) mine = lane == q ? d[q] : mine;
        if (lane < 6) D6[6 * (size_t)v + lane] = mine;
        dhL[(size_t)MPNN_H * v + lane] = dh;
    }
}

// one warp per edge (its output gradient is the edge's block of dG)
__global__ void headEdgeBackKernel(int n, const int* slot, const float* dG, const bf16* w, float* deL) {
    constexpr int IN = MPNN_H + MPNN_EF;
    const int lane = threadIdx.x & 31, warps = gridDim.x * blockDim.x / 32;
    float wt[9];
    for (int q = 0; q < 9; ++q) wt[q] = W(w + MP_WO + q * IN, lane);
    for (int e = (blockIdx.x * blockDim.x + threadIdx.x) / 32; e < n; e += warps) {
        const float* d = dG + (size_t)9 * slot[e];
        float dh = 0.f;
        for (int q = 0; q < 9; ++q) dh += d[q] * wt[q];
        deL[(size_t)MPNN_H * e + lane] = dh;
    }
}

// Backward of a 64 -> 32 layer over tiles of LB_ITEMS items: the warps form the
// items' pre-activation gradients d (one row of 32 per warp step; also kept in
// shared memory), then two threads per item each form 32 of the 64 components
// of W^T d from the staged weights.
constexpr int LB_ITEMS = 64, LB_THREADS = 2 * LB_ITEMS;

struct NodeBack {  // h' = relu(Wh [h; agg] + b)
    const float *hNext, *dhNext;
    float *dhPrev, *dagg;
    __device__ float pre(int v, int t) const { return hNext[(size_t)MPNN_H * v + t] > 0.f ? dhNext[(size_t)MPNN_H * v + t] : 0.f; }
    __device__ float* out(int v, int half) const { return (half ? dagg : dhPrev) + (size_t)MPNN_H * v; }
};
// e' = relu(We [e; h_i + h_j] + b); the edge's gradient is deNext plus what the
// node layer's mean takes from it, dagg_i / deg_i + dagg_j / deg_j.  Writes the
// gradient with respect to e (dePrev) and to h_i + h_j (ds), and that sum (the
// second input block of the weight gradient).
struct EdgeBack {
    const int *slot, *ei, *ej;
    const float *hPrev, *eNext, *deNext, *dagg;
    const int* deg;
    float *hsum, *dePrev, *ds;
    __device__ float pre(int k, int t) const {
        const int i = ei[k], j = ej[k];
        hsum[(size_t)MPNN_H * k + t] = hPrev[(size_t)MPNN_H * i + t] + hPrev[(size_t)MPNN_H * j + t];
        const float iv = deg[i] > 0 ? 1.f / deg[i] : 0.f, ic = deg[j] > 0 ? 1.f / deg[j] : 0.f;
        const float de = deNext[(size_t)MPNN_H * k + t] + (dagg[(size_t)MPNN_H * i + t] * iv + dagg[(size_t)MPNN_H * j + t] * ic);
        return eNext[(size_t)MPNN_H * slot[k] + t] > 0.f ? de : 0.f;
    }
    __device__ float* out(int k, int half) const { return (half ? ds : dePrev) + (size_t)MPNN_H * k; }
};

template <class B>
__global__ void __launch_bounds__(LB_THREADS) layerBackKernel(int n, B b, const bf16* Wm, float* D32) {
    __shared__ __align__(16) float sW[MPNN_H][2 * MPNN_H];
    __shared__ float sD[LB_ITEMS][MPNN_H + 1];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int t = threadIdx.x; t < MPNN_H * 2 * MPNN_H; t += LB_THREADS) sW[t / (2 * MPNN_H)][t % (2 * MPNN_H)] = W(Wm, t);
    for (int base = blockIdx.x * LB_ITEMS; base < n; base += gridDim.x * LB_ITEMS) {
        __syncthreads();
        for (int r = warp; r < LB_ITEMS; r += LB_THREADS / 32) {
            const int item = base + r;
            float d = 0.f;
            if (item < n) {
                d = b.pre(item, lane);
                D32[(size_t)MPNN_H * item + lane] = d;
            }
            sD[r][lane] = d;
        }
        __syncthreads();
        // lanes 0-15 of a warp take 16 items' first halves, 16-31 the second
        const int r = 16 * warp + (lane & 15), half = lane >> 4, item = base + r;
        float acc[MPNN_H];
#pragma unroll
        for (int i = 0; i < MPNN_H; ++i) acc[i] = 0.f;
#pragma unroll 4
        for (int o = 0; o < MPNN_H; ++o) {
            const float d = sD[r][o];
            const float4* wr = reinterpret_cast<const float4*>(&sW[o][half * MPNN_H]);
#pragma unroll
            for (int i = 0; i < MPNN_H / 4; ++i) {
                const float4 w4 = wr[i];
                acc[4 * i] += w4.x * d;
                acc[4 * i + 1] += w4.y * d;
                acc[4 * i + 2] += w4.z * d;
                acc[4 * i + 3] += w4.w * d;
            }
        }
        if (item < n) {
            float4* out = reinterpret_cast<float4*>(b.out(item, half));
#pragma unroll
            for (int i = 0; i < MPNN_H / 4; ++i) out[i] = make_float4(acc[4 * i], acc[4 * i + 1], acc[4 * i + 2], acc[4 * i + 3]);
        }
    }
}

// sum over the row's edges of feature `lane` of e, slot order (as
// aggregateRange, rows by edge)
__device__ __forceinline__ float edgeSumRange(float a, int v, int k0, int k1, const int* col, const int* mir, const int* edgeOf, const float* e,
                                              int lane) {
    for (int c0 = k0; c0 < k1; c0 += 32) {
        const int k = c0 + lane;
        int edge = -1;
        if (k < k1) {
            const int c = col[k];
            const int slot = c == v ? -1 : (c < v ? k : mir[k]);
            if (slot >= 0) edge = edgeOf[slot];
        }
        const int m = min(32, k1 - c0);
        for (int j = 0; j < m; ++j) {
            const int ej = __shfl_sync(0xffffffffu, edge, j);
            if (ej >= 0) a += e[(size_t)MPNN_H * ej + lane];
        }
    }
    return a;
}

// dh_v += sum of ds over the edges incident to v, one warp per vertex
__global__ void dsGatherKernel(int nv, const int* rowPtr, const int* col, const int* mirS, const int* edgeS, const float* dsS, const int* dRowS,
                               const int* dRowE, const int* dCol, const int* mirD, const int* edgeD, const float* dsD, float* dh) {
    const int lane = threadIdx.x & 31;
    const int warps = gridDim.x * blockDim.x / 32;
    for (int v = (blockIdx.x * blockDim.x + threadIdx.x) / 32; v < nv; v += warps) {
        float s = edgeSumRange(0.f, v, rowPtr[v], rowPtr[v + 1], col, mirS, edgeS, dsS, lane);
        if (dRowS) s = edgeSumRange(s, v, dRowS[v], dRowE[v], dCol, mirD, edgeD, dsD, lane);
        dh[(size_t)MPNN_H * v + lane] += s;
    }
}

// pre-activation gradient of an embedding (relu): items are nodes or edges,
// whose forward state is at their slot
__global__ void reluGradKernel(int n, const int* slot, const float* y, const float* dy, float* D32) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < (size_t)n * MPNN_H; i += (size_t)gridDim.x * blockDim.x) {
        const size_t item = i / MPNN_H, t = i - item * MPNN_H;
        D32[i] = y[(slot ? (size_t)slot[item] : item) * MPNN_H + t] > 0.f ? dy[i] : 0.f;
    }
}

__global__ void toBf16Kernel(int n, const float* w, bf16* o) {
    CIPC_KERNEL_LOOP(i, n) o[i] = __float2bfloat16_rn(w[i]);
}

__global__ void adamKernel(int n, float* w, const float* g, float* m, float* v, float lr, float b1, float b2, float eps, float c1, float c2, float clip) {
    CIPC_KERNEL_LOOP(i, n) {
        float gi = fmaxf(-clip, fminf(clip, g[i]));
        m[i] = b1 * m[i] + (1.f - b1) * gi;
        v[i] = b2 * v[i] + (1.f - b2) * gi * gi;
        w[i] -= lr * (m[i] / c1) / (sqrtf(v[i] / c2) + eps);
    }
}

__global__ void zeroFloatKernel(size_t n, float* a) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)blockDim.x * gridDim.x) a[i] = 0.f;
}

struct DynView {
    const int *rs, *re, *col;
    bool on;
};
DynView dynView(Ctx& c) {
    bool on = c.nDynB > 0;
    return {on ? c.dynRowStart.p : nullptr, on ? c.dynRowEnd.p : nullptr, on ? c.dynCol.p : nullptr, on};
}

void zeroF(Ctx& c, float* p, size_t n) {
    if (n) launch(zeroFloatKernel, (unsigned)std::min<size_t>((n + 255) / 256, 4096), 256, 0, c.s, n, p);
}
const bf16* wbf(Ctx& c) { return reinterpret_cast<const bf16*>(c.mpWb.p); }

}  // namespace

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
void mpnnInitWeights(Ctx& c, unsigned long long seed) {
    std::vector<float> w(MP_NPARAM, 0.f);
    unsigned long long z = seed;
    auto rnd = [&]() {
        z += 0x9E3779B97F4A7C15ull;
        unsigned long long t = z;
        t = (t ^ (t >> 30)) * 0xBF58476D1CE4E5B9ull;
        t = (t ^ (t >> 27)) * 0x94D049BB133111EBull;
        t ^= t >> 31;
        return (double)(t >> 11) * (1.0 / 9007199254740992.0) * 2.0 - 1.0;
    };
    auto fill = [&](int off, int fanOut, int fanIn) {
        double s = std::sqrt(6.0 / (fanIn + fanOut));
        for (int i = 0; i < fanOut * fanIn; ++i) w[off + i] = (float)(s * rnd());
    };
    fill(MP_WN0, MPNN_H, MPNN_NF);
    fill(MP_WE0, MPNN_H, MPNN_EF);
    for (int l = 0; l < MPNN_L; ++l) { fill(mpWe(l), MPNN_H, 2 * MPNN_H); fill(mpWh(l), MPNN_H, 2 * MPNN_H); }
    // heads start at the first-order factor G = I - strict_lower(Â)
    const float inv = (float)std::log(std::exp(1.0) - 1.0);  // softplus^-1(1)
    w[MP_BD + 0] = w[MP_BD + 1] = w[MP_BD + 2] = inv;
    for (int q = 0; q < 9; ++q) w[MP_WO + q * (MPNN_H + MPNN_EF) + MPNN_H + q] = -1.f;
    mpnnSetWeights(c, w.data(), MP_NPARAM);
}

void mpnnSetWeights(Ctx& c, const float* w, int n) {
    if (n != MP_NPARAM) throw InvalidArgument("expected " + std::to_string(MP_NPARAM) + " network parameters, got " + std::to_string(n));
    for (int i = 0; i < n; ++i)
        if (!std::isfinite(w[i])) throw InvalidArgument("network parameter " + std::to_string(i) + " is not finite");
    c.mpW.reserve(MP_NPARAM); c.mpWb.reserve(MP_NPARAM); c.mpG.reserve(MP_NPARAM); c.mpM.reserve(MP_NPARAM); c.mpV.reserve(MP_NPARAM);
    CIPC_CUDA(cudaMemcpyAsync(c.mpW.p, w, sizeof(float) * MP_NPARAM, cudaMemcpyHostToDevice, c.s));
    zeroF(c, c.mpM.p, MP_NPARAM);
    zeroF(c, c.mpV.p, MP_NPARAM);
    zeroF(c, c.mpG.p, MP_NPARAM);
    launch(toBf16Kernel, blocksFor(MP_NPARAM), TB, 0, c.s, MP_NPARAM, (const float*)c.mpW.p, reinterpret_cast<bf16*>(c.mpWb.p));
    hostSync(c);
    c.mpStep = 0;
    c.mpReady = true;
    c.mpFactorReady = false;
}

void mpnnGetWeights(Ctx& c, float* w) {
    if (!c.mpReady) throw InvalidArgument("no network weights set");
    CIPC_CUDA(cudaMemcpyAsync(w, c.mpW.p, sizeof(float) * MP_NPARAM, cudaMemcpyDeviceToHost, c.s));
    hostSync(c);
}

void mpnnGetGrad(Ctx& c, float* g) {
    if (!c.mpReady) throw InvalidArgument("no network weights set");
    CIPC_CUDA(cudaMemcpyAsync(g, c.mpG.p, sizeof(float) * MP_NPARAM, cudaMemcpyDeviceToHost, c.s));
    hostSync(c);
}

// Flat list of the lower edges of a row-ranged pattern: three arrays of
// `count` ints (slot, row, column) packed in `out`, and each slot's place in
// it (edgeOf, -1 for the other slots).  Returns the count.
static int buildLowerList(Ctx& c, const int* rowS, const int* rowE, const int* col, DBuf<int>& out, int* edgeOf) {
    int nv = c.nv;
    c.mpScanTmpI.reserve(2 * (size_t)nv + 2);
    int* cnt = c.mpScanTmpI.p;
    int* off = cnt + nv + 1;
    launch(lowerCountKernel, blocksFor(nv), TB, 0, c.s, nv, rowS, rowE, col, cnt);
    CIPC_CUDA(cudaMemsetAsync(cnt + nv, 0, sizeof(int), c.s));
    size_t bytes = 0;
    CIPC_CUDA(cub::DeviceScan::ExclusiveSum(nullptr, bytes, cnt, off, nv + 1, c.s));
    c.mpScanTmp.reserve(bytes + 16);
    CIPC_CUDA(cub::DeviceScan::ExclusiveSum(c.mpScanTmp.p, bytes, cnt, off, nv + 1, c.s));
    int n = 0;
    CIPC_CUDA(cudaMemcpyAsync(&n, off + nv, sizeof(int), cudaMemcpyDeviceToHost, c.s));
    hostSync(c);
    out.reserve(3 * (size_t)std::max(n, 1));
    launch(lowerFillKernel, blocksFor(nv), TB, 0, c.s, nv, rowS, rowE, col, (const int*)off, out.p, out.p + n, out.p + 2 * (size_t)n, edgeOf);
    return n;
}

template <class MT>
static void prepareT(Ctx& c, const MT* val, const MT* dval, bool features) {
    int nv = c.nv;
    DynView d = dynView(c);
    size_t es = (size_t)std::max(c.nnzb, 1), ed = (size_t)std::max(c.nDynB, 1);
    c.mpS.reserve(9 * (size_t)nv);
    c.mpNodeF.reserve(MPNN_NF * (size_t)nv + nv);
    float* f5 = c.mpNodeF.p + MPNN_NF * (size_t)nv;
    launch(scaleKernel<MT>, blocksFor(nv), TB, 0, c.s, nv, (const int*)c.diagSlot.p, val, d.rs, d.re, d.col, dval, (const double*)c.diagExtra.p,
           c.mpS.p, f5);
    if (features)
        launch(nodeFeatKernel<MT>, blocksFor(nv), TB, 0, c.s, nv, (const int*)c.rowPtr.p, (const int*)c.colIdx.p, val, d.rs, d.re, d.col, dval,
               (const double*)c.mpS.p, (const float*)f5, c.mpNodeF.p);
    if (!c.mpMirrorReady) {
        c.mpMirS.reserve(es);
        c.mpRowS.reserve(nv); c.mpRowE.reserve(nv);
        launch(rowRangeKernel, blocksFor(nv), TB, 0, c.s, nv, (const int*)c.rowPtr.p, c.mpRowS.p, c.mpRowE.p);
        launch(mirrorKernel, blocksFor(nv), TB, 0, c.s, nv, (const int*)c.mpRowS.p, (const int*)c.mpRowE.p, (const int*)c.colIdx.p, c.mpMirS.p);
        c.mpMirrorReady = true;
    }
    c.mpEdgeF.reserve(9 * es);
    if (features)
        launch(edgeFeatKernel<MT>, blocksFor(nv), TB, 0, c.s, nv, (const int*)c.mpRowS.p, (const int*)c.mpRowE.p, (const int*)c.colIdx.p, val,
               (const double*)c.mpS.p, c.mpEdgeF.p);
    c.mpMirD.reserve(ed);
    c.mpEdgeFD.reserve(9 * ed);
    if (d.on) {
        launch(mirrorKernel, blocksFor(nv), TB, 0, c.s, nv, d.rs, d.re, d.col, c.mpMirD.p);
        if (features) launch(edgeFeatKernel<MT>, blocksFor(nv), TB, 0, c.s, nv, d.rs, d.re, d.col, dval, (const double*)c.mpS.p, c.mpEdgeFD.p);
    }
    if (features) {  // the network's flat edge lists
        if (c.nFlatS < 0) {
            c.mpEdgeOfS.reserve(es);
            c.nFlatS = buildLowerList(c, (const int*)c.mpRowS.p, (const int*)c.mpRowE.p, (const int*)c.colIdx.p, c.mpFlatS, c.mpEdgeOfS.p);
        }
        c.mpEdgeOfD.reserve(ed);
        c.nFlatD = d.on ? buildLowerList(c, d.rs, d.re, d.col, c.mpFlatD, c.mpEdgeOfD.p) : 0;
    }
    c.mpDeg.reserve(nv);
    launch(degreeKernel, blocksFor(nv), TB, 0, c.s, nv, (const int*)c.rowPtr.p, (const int*)c.colIdx.p, (const int*)c.mpMirS.p, d.rs, d.re, d.col,
           (const int*)c.mpMirD.p, c.mpDeg.p);
    CIPC_CUDA(cudaGetLastError());
    c.mpFactorReady = false;
}

void mpnnPrepare(Ctx& c, bool features) {
    if (c.mixed) prepareT<float>(c, c.valF.p, c.dynBF.p, features);
    else prepareT<double>(c, c.valD.p, c.dynBD.p, features);
}

static_assert(mpWe(0) % 8 == 0 && mpWh(0) % 8 == 0 && MP_LAYER % 8 == 0,
              "tensor-core layer weights start on 16-byte boundaries");

void mpnnForward(Ctx& c) {
    if (!c.mpReady) throw InvalidArgument("no network weights set");
    if (c.tcFault) throw std::runtime_error("a tensor-core wait timed out earlier on this context; recreate it to use the learned preconditioner");
    int nv = c.nv;
    DynView d = dynView(c);
    size_t es = (size_t)std::max(c.nnzb, 1), ed = (size_t)std::max(c.nDynB, 1);
    c.mpH.reserve((size_t)(MPNN_L + 1) * MPNN_H * nv);
    c.mpAgg.reserve((size_t)MPNN_L * MPNN_H * nv);
    c.mpES.reserve((size_t)(MPNN_L + 1) * MPNN_H * es);
    c.mpED.reserve((size_t)(MPNN_L + 1) * MPNN_H * ed);
    c.mpGS.reserve(9 * es);
    c.mpGD.reserve(9 * ed);
    c.mpHeadD.reserve(6 * (size_t)nv);
    const bf16* w = wbf(c);
    auto H = [&](int l) { return c.mpH.p + (size_t)l * MPNN_H * nv; };
    auto ES = [&](int l) { return c.mpES.p + (size_t)l * MPNN_H * es; };
    auto ED = [&](int l) { return c.mpED.p + (size_t)l * MPNN_H * ed; };
    const int nS = c.nFlatS, nD = d.on ? c.nFlatD : 0;
    const int *sSlot = c.mpFlatS.p, *sI = sSlot + nS, *sJ = sSlot + 2 * (size_t)nS;
    const int *dSlot = c.mpFlatD.p, *dI = dSlot + nD, *dJ = dSlot + 2 * (size_t)nD;
    auto grid = [](int n) { return std::max(1, std::min((n + DT_ITEMS - 1) / DT_ITEMS, 148 * 16)); };
    // embeddings
    launch(denseTiledKernel<MPNN_NF, MPNN_H, NodeFeatGather, ReluEmitNode>, grid(nv), DT_THREADS, 0, c.s, nv, NodeFeatGather{c.mpNodeF.p},
           ReluEmitNode{H(0)}, w + MP_WN0, w + MP_BN0);
    if (nS) launch(denseTiledKernel<MPNN_EF, MPNN_H, EdgeFeatGather, ReluEmitEdge>, grid(nS), DT_THREADS, 0, c.s, nS,
                   EdgeFeatGather{sSlot, c.mpEdgeF.p}, ReluEmitEdge{sSlot, ES(0)}, w + MP_WE0, w + MP_BE0);
    if (nD) launch(denseTiledKernel<MPNN_EF, MPNN_H, EdgeFeatGather, ReluEmitEdge>, grid(nD), DT_THREADS, 0, c.s, nD,
                   EdgeFeatGather{dSlot, c.mpEdgeFD.p}, ReluEmitEdge{dSlot, ED(0)}, w + MP_WE0, w + MP_BE0);
    // the 64 -> 32 message-passing layers run on the tensor cores
    auto tcGrid = [](int n) { return std::max(1, std::min((n + tc::M - 1) / tc::M, 148 * 4)); };
    for (int l = 0; l < MPNN_L; ++l) {
        if (nS) launch(tc::denseTcKernel<EdgeLayerGather, ReluEmitEdge>, tcGrid(nS), tc::THREADS, 0, c.s, nS, EdgeLayerGather{sSlot, sI, sJ, ES(l), H(l)},
                       ReluEmitEdge{sSlot, ES(l + 1)}, w + mpWe(l), w + mpBe(l), c.status.p, (int)CIPC_ST_TC_TIMEOUT);
        if (nD) launch(tc::denseTcKernel<EdgeLayerGather, ReluEmitEdge>, tcGrid(nD), tc::THREADS, 0, c.s, nD, EdgeLayerGather{dSlot, dI, dJ, ED(l), H(l)},
                       ReluEmitEdge{dSlot, ED(l + 1)}, w + mpWe(l), w + mpBe(l), c.status.p, (int)CIPC_ST_TC_TIMEOUT);
        float* agg = c.mpAgg.p + (size_t)l * MPNN_H * nv;
        launch(aggregateKernel, blocksFor(32 * nv), TB, 0, c.s, nv, (const int*)c.rowPtr.p, (const int*)c.colIdx.p, (const int*)c.mpMirS.p,
               (const float*)ES(l + 1), d.rs, d.re, d.col, (const int*)c.mpMirD.p, (const float*)ED(l + 1), (const int*)c.mpDeg.p, agg);
        launch(tc::denseTcKernel<NodeLayerGather, ReluEmitNode>, tcGrid(nv), tc::THREADS, 0, c.s, nv, NodeLayerGather{H(l), agg}, ReluEmitNode{H(l + 1)},
               w + mpWh(l), w + mpBh(l), c.status.p, (int)CIPC_ST_TC_TIMEOUT);
    }
    // heads: contact diagonal slots carry no factor part
    if (d.on) CIPC_CUDA(cudaMemsetAsync(c.mpGD.p, 0, sizeof(float) * 9 * (size_t)c.nDynB, c.s));
    if (nS) launch(denseTiledKernel<MPNN_H + MPNN_EF, 9, HeadEdgeGather, HeadEdgeEmit>, grid(nS), DT_THREADS, 0, c.s, nS,
                   HeadEdgeGather{sSlot, ES(MPNN_L), c.mpEdgeF.p}, HeadEdgeEmit{sSlot, sI, sJ, c.mpMirS.p, c.btype.p, c.mpGS.p}, w + MP_WO, w + MP_BO);
    if (nD) launch(denseTiledKernel<MPNN_H + MPNN_EF, 9, HeadEdgeGather, HeadEdgeEmit>, grid(nD), DT_THREADS, 0, c.s, nD,
                   HeadEdgeGather{dSlot, ED(MPNN_L), c.mpEdgeFD.p}, HeadEdgeEmit{dSlot, dI, dJ, c.mpMirD.p, c.btype.p, c.mpGD.p}, w + MP_WO, w + MP_BO);
    launch(denseTiledKernel<MPNN_H, 6, NodeHiddenGather, HeadDiagEmit>, grid(nv), DT_THREADS, 0, c.s, nv, NodeHiddenGather{H(MPNN_L)},
           HeadDiagEmit{c.diagSlot.p, c.btype.p, c.mpGS.p, c.mpHeadD.p}, w + MP_WD, w + MP_BD);
    CIPC_CUDA(cudaGetLastError());
    c.mpFactorReady = true;
}

template <class MT>
static double lossT(Ctx& c, const MT* val, const MT* dval, int nprobes, const float* hostProbes, unsigned long long seed, bool backward) {
    int nv = c.nv, n3 = 3 * nv;
    DynView d = dynView(c);
    size_t es = (size_t)std::max(c.nnzb, 1), ed = (size_t)std::max(c.nDynB, 1);
    // probes in chunks: planes of 3 nv per probe of w, u = G^T w, v = Â G^T w; then the scales
    constexpr int CHUNK = 8;
    const int chunk = std::min(nprobes, CHUNK);
    const size_t np3 = (size_t)chunk * n3;
    c.mpVec.reserve(3 * np3 + chunk);
    float* w = c.mpVec.p;
    float* u = w + np3;
    float* vv = u + np3;
    float* scaleDev = vv + np3;
    const int nb = std::min(1024, std::max(1, (n3 + 255) / 256));
    c.red.reserve(2 * 1024 * CHUNK + 16);
    std::vector<double> part(std::max<size_t>(2 * (size_t)nb * chunk, 1024));
    float scale[CHUNK];
    const int nS = c.nFlatS, nE = d.on ? c.nFlatD : 0;
    const int *sSlot = c.mpFlatS.p, *sI = sSlot + nS, *sJ = sSlot + 2 * (size_t)nS;
    const int *dSlot = c.mpFlatD.p, *dI = dSlot + nE, *dJ = dSlot + 2 * (size_t)nE;
    if (backward) {
        c.mpDGS.reserve(9 * es);
        c.mpDGD.reserve(9 * ed);
    }
    double T = 0;
    for (int p0 = 0; p0 < nprobes; p0 += chunk) {
        const int np = std::min(chunk, nprobes - p0);
        if (hostProbes)
            CIPC_CUDA(cudaMemcpyAsync(w, hostProbes + (size_t)p0 * n3, sizeof(float) * n3 * np, cudaMemcpyHostToDevice, c.s));
        else
            for (int k = 0; k < np; ++k)
                launch(probeKernel, blocksFor(n3), TB, 0, c.s, n3, seed + 7919ull * (p0 + k), w + (size_t)k * n3);
        launch(factorApplyKernel, blocksFor(nv * np), TB, 0, c.s, nv, np, 1, (const int*)c.rowPtr.p, (const int*)c.colIdx.p, (const float*)c.mpGS.p,
               d.rs, d.re, d.col, (const float*)c.mpGD.p, (const float*)w, u);
        launch(scaledSpmvKernel<MT>, blocksFor(nv * np), TB, 0, c.s, nv, np, (const int*)c.rowPtr.p, (const int*)c.colIdx.p, val, d.rs, d.re, d.col,
               dval, (const double*)c.diagExtra.p, (const double*)c.mpS.p, (const float*)u, vv);
        launch(probeDotsKernel, dim3(nb, np), 256, 0, c.s, n3, (const float*)u, (const float*)vv, (const float*)w, c.red.p);
        CIPC_CUDA(cudaMemcpyAsync(part.data(), c.red.p, sizeof(double) * 2 * nb * np, cudaMemcpyDeviceToHost, c.s));
        hostSync(c);
        for (int k = 0; k < np; ++k) {
            const double* pp = part.data() + (size_t)2 * nb * k;
            double uv = 0, ww = 0;
            for (int q = 0; q < nb; ++q) { uv += pp[2 * q]; ww += pp[2 * q + 1]; }
            if (!(ww > 0)) throw InvalidArgument("probe vector is zero");
            T += uv / ww / nprobes;
            scale[k] = (float)(2.0 / ww / nprobes);
        }
        if (!backward) continue;
        const bool first = p0 == 0, last = p0 + np >= nprobes;
        const float mul = last ? (float)(1.0 / T) : 1.f;
        CIPC_CUDA(cudaMemcpyAsync(scaleDev, scale, sizeof(float) * np, cudaMemcpyHostToDevice, c.s));
        if (nS)
            launch(factorGradEdgeKernel, blocksFor(9 * nS), TB, 0, c.s, nS, sSlot, sI, sJ, (const int*)c.btype.p, np, n3, (const float*)w,
                   (const float*)vv, (const float*)scaleDev, first, mul, c.mpDGS.p);
        if (nE)
            launch(factorGradEdgeKernel, blocksFor(9 * nE), TB, 0, c.s, nE, dSlot, dI, dJ, (const int*)c.btype.p, np, n3, (const float*)w,
                   (const float*)vv, (const float*)scaleDev, first, mul, c.mpDGD.p);
        launch(factorGradDiagKernel, blocksFor(9 * nv), TB, 0, c.s, nv, (const int*)c.diagSlot.p, (const int*)c.btype.p, np, n3, (const float*)w,
               (const float*)vv, (const float*)scaleDev, first, mul, last, (const float*)c.mpGS.p, (float)(2.0 / n3), c.mpDGS.p);
    }
    int nb2 = std::min(1024, std::max(1, (nv + 255) / 256));
    launch(logDiagKernel, nb2, 256, 0, c.s, nv, (const int*)c.diagSlot.p, (const float*)c.mpGS.p, c.red.p);
    CIPC_CUDA(cudaMemcpyAsync(part.data(), c.red.p, sizeof(double) * nb2, cudaMemcpyDeviceToHost, c.s));
    hostSync(c);
    double logDiag = 0;
    for (int k = 0; k < nb2; ++k) logDiag += part[k];
    if (!(T > 0) || !std::isfinite(T) || !std::isfinite(logDiag)) throw std::runtime_error("learned preconditioner loss is not finite");
    double loss = std::log(T) - 2.0 / n3 * logDiag;
    if (!backward) return loss;

    const bf16* wb = wbf(c);
    float* gW = c.mpG.p;
    zeroF(c, gW, MP_NPARAM);
    const size_t fS = (size_t)std::max(nS, 1), fD = (size_t)std::max(nE, 1);
    size_t items = std::max(std::max(fS, fD), (size_t)nv);
    c.mpDH.reserve((size_t)(MPNN_L + 1) * MPNN_H * nv);
    c.mpDES.reserve((size_t)(MPNN_L + 1) * MPNN_H * fS);
    c.mpDED.reserve((size_t)(MPNN_L + 1) * MPNN_H * fD);
    c.mpDAgg.reserve((size_t)MPNN_H * nv);
    c.mpDS.reserve((size_t)MPNN_H * fS);
    c.mpDSD.reserve((size_t)MPNN_H * fD);
    c.mpBD.reserve((size_t)MPNN_H * items);
    c.mpBX.reserve((size_t)MPNN_H * items);
    c.mpPart.reserve((size_t)WG_GRID * (MPNN_H * 2 * MPNN_H + MPNN_H));
    auto H = [&](int l) { return c.mpH.p + (size_t)l * MPNN_H * nv; };
    auto DH = [&](int l) { return c.mpDH.p + (size_t)l * MPNN_H * nv; };
    auto ES = [&](int l) { return c.mpES.p + (size_t)l * MPNN_H * es; };
    auto ED = [&](int l) { return c.mpED.p + (size_t)l * MPNN_H * ed; };
    auto DES = [&](int l) { return c.mpDES.p + (size_t)l * MPNN_H * fS; };
    auto DED = [&](int l) { return c.mpDED.p + (size_t)l * MPNN_H * fD; };
    float* BD = c.mpBD.p;
    float* BX = c.mpBX.p;
    auto reduceWeights = [&](int nw, int out, int ctas, int wOff, int bOff) {
        launch(weightGradReduceKernel, (nw + WR_OUT - 1) / WR_OUT, WR_OUT * WR_SPLIT, 0, c.s, nw, out, ctas, (const float*)c.mpPart.p, gW + wOff,
               gW + bOff);
    };
    // dW += D^T [X1 X2], db += sum D over `n` items (split-K, deterministic)
    auto wgrad = [&](auto kernel, int out, int in, int n, const float* D, const int* dItem, const float* X1, const float* X2, const int* xItem,
                     int wOff, int bOff) {
        if (n <= 0) return;
        int nw = out * in + out;
        int grid = std::max(1, std::min(WG_GRID, (n + WG_TI - 1) / WG_TI));
        launch(kernel, grid, WG_THREADS, 0, c.s, n, D, dItem, X1, X2, xItem, c.mpPart.p);
        reduceWeights(nw, out, grid, wOff, bOff);
    };
    // the 64 -> 32 message-passing layers: the same contraction on the tensor cores
    auto wgradTc = [&](int n, const float* X1, const int* x1Item, const float* X2, int wOff, int bOff) {
        if (n <= 0) return;
        static bool attr = false;
        if (!attr) {
            CIPC_CUDA(cudaFuncSetAttribute(tc::weightGradTcKernel, cudaFuncAttributeMaxDynamicSharedMemorySize, tc::WG_SMEM));
            attr = true;
        }
        const int nw = MPNN_H * 2 * MPNN_H + MPNN_H;
        const int grid = std::max(1, std::min(WG_GRID, (n + tc::WG_K - 1) / tc::WG_K));
        launch(tc::weightGradTcKernel, grid, tc::THREADS, tc::WG_SMEM, c.s, n, (const float*)BD, X1, x1Item, X2, c.mpPart.p, c.status.p,
               (int)CIPC_ST_TC_TIMEOUT);
        reduceWeights(nw, MPNN_H, grid, wOff, bOff);
    };
    const int* none = nullptr;
    const int nodeWarps = blocksFor(32 * nv);
    auto edgeWarps = [](int n) { return std::max(1, (int)std::min<long long>(((long long)n * 32 + TB - 1) / TB, 148 * 32)); };
    auto tiles = [](int n) { return std::max(1, std::min((n + LB_ITEMS - 1) / LB_ITEMS, 148 * 16)); };
    // heads
    launch(headDiagBackKernel, nodeWarps, TB, 0, c.s, nv, (const float*)c.mpHeadD.p, (const int*)c.diagSlot.p, (const float*)c.mpDGS.p, wb, BD,
           DH(MPNN_L));
    wgrad(weightGradKernel<6, MPNN_H, 0>, 6, MPNN_H, nv, (const float*)BD, none, (const float*)H(MPNN_L), (const float*)nullptr, none, MP_WD, MP_BD);
    if (nS) launch(headEdgeBackKernel, edgeWarps(nS), TB, 0, c.s, nS, sSlot, (const float*)c.mpDGS.p, wb, DES(MPNN_L));
    wgrad(weightGradKernel<9, MPNN_H, MPNN_EF>, 9, MPNN_H + MPNN_EF, nS, (const float*)c.mpDGS.p, sSlot, (const float*)ES(MPNN_L),
          (const float*)c.mpEdgeF.p, sSlot, MP_WO, MP_BO);
    if (nE) {
        launch(headEdgeBackKernel, edgeWarps(nE), TB, 0, c.s, nE, dSlot, (const float*)c.mpDGD.p, wb, DED(MPNN_L));
        wgrad(weightGradKernel<9, MPNN_H, MPNN_EF>, 9, MPNN_H + MPNN_EF, nE, (const float*)c.mpDGD.p, dSlot, (const float*)ED(MPNN_L),
              (const float*)c.mpEdgeFD.p, dSlot, MP_WO, MP_BO);
    }
    for (int l = MPNN_L - 1; l >= 0; --l) {
        const float* agg = c.mpAgg.p + (size_t)l * MPNN_H * nv;
        launch(layerBackKernel<NodeBack>, tiles(nv), LB_THREADS, 0, c.s, nv, NodeBack{H(l + 1), DH(l + 1), DH(l), c.mpDAgg.p}, wb + mpWh(l), BD);
        wgradTc(nv, (const float*)H(l), none, agg, mpWh(l), mpBh(l));
        if (nS) {
            launch(layerBackKernel<EdgeBack>, tiles(nS), LB_THREADS, 0, c.s, nS,
                   EdgeBack{sSlot, sI, sJ, H(l), ES(l + 1), DES(l + 1), c.mpDAgg.p, c.mpDeg.p, BX, DES(l), c.mpDS.p}, wb + mpWe(l), BD);
            wgradTc(nS, (const float*)ES(l), sSlot, (const float*)BX, mpWe(l), mpBe(l));
        }
        if (nE) {
            launch(layerBackKernel<EdgeBack>, tiles(nE), LB_THREADS, 0, c.s, nE,
                   EdgeBack{dSlot, dI, dJ, H(l), ED(l + 1), DED(l + 1), c.mpDAgg.p, c.mpDeg.p, BX, DED(l), c.mpDSD.p}, wb + mpWe(l), BD);
            wgradTc(nE, (const float*)ED(l), dSlot, (const float*)BX, mpWe(l), mpBe(l));
        }
        launch(dsGatherKernel, nodeWarps, TB, 0, c.s, nv, (const int*)c.rowPtr.p, (const int*)c.colIdx.p, (const int*)c.mpMirS.p,
               (const int*)c.mpEdgeOfS.p, (const float*)c.mpDS.p, d.rs, d.re, d.col, (const int*)c.mpMirD.p, (const int*)c.mpEdgeOfD.p,
               (const float*)c.mpDSD.p, DH(l));
    }
    // embeddings
    launch(reluGradKernel, nodeWarps, TB, 0, c.s, nv, none, (const float*)H(0), (const float*)DH(0), BD);
    wgrad(weightGradKernel<MPNN_H, MPNN_NF, 0>, MPNN_H, MPNN_NF, nv, (const float*)BD, none, (const float*)c.mpNodeF.p, (const float*)nullptr, none,
          MP_WN0, MP_BN0);
    if (nS) {
        launch(reluGradKernel, edgeWarps(nS), TB, 0, c.s, nS, sSlot, (const float*)ES(0), (const float*)DES(0), BD);
        wgrad(weightGradKernel<MPNN_H, MPNN_EF, 0>, MPNN_H, MPNN_EF, nS, (const float*)BD, none, (const float*)c.mpEdgeF.p, (const float*)nullptr, sSlot,
              MP_WE0, MP_BE0);
    }
    if (nE) {
        launch(reluGradKernel, edgeWarps(nE), TB, 0, c.s, nE, dSlot, (const float*)ED(0), (const float*)DED(0), BD);
        wgrad(weightGradKernel<MPNN_H, MPNN_EF, 0>, MPNN_H, MPNN_EF, nE, (const float*)BD, none, (const float*)c.mpEdgeFD.p, (const float*)nullptr,
              dSlot, MP_WE0, MP_BE0);
    }
    CIPC_CUDA(cudaGetLastError());
    return loss;
}

double mpnnLoss(Ctx& c, int nprobes, const float* probes, unsigned long long seed, bool backward) {
    if (!c.mpFactorReady) throw InvalidArgument("no factor: run the network forward on an assembled system first");
    if (nprobes < 1) throw InvalidArgument("need at least one probe vector");
    if (c.mixed) return lossT<float>(c, c.valF.p, c.dynBF.p, nprobes, probes, seed, backward);
    return lossT<double>(c, c.valD.p, c.dynBD.p, nprobes, probes, seed, backward);
}

void mpnnAdam(Ctx& c, double lr) {
    c.mpStep++;
    const float b1 = 0.9f, b2 = 0.999f;
    float c1 = 1.f - std::pow(b1, (float)c.mpStep), c2 = 1.f - std::pow(b2, (float)c.mpStep);
    launch(adamKernel, blocksFor(MP_NPARAM), TB, 0, c.s, MP_NPARAM, c.mpW.p, (const float*)c.mpG.p, c.mpM.p, c.mpV.p, (float)lr, b1, b2, 1e-8f, c1,
           c2, 1.0f);
    launch(toBf16Kernel, blocksFor(MP_NPARAM), TB, 0, c.s, MP_NPARAM, (const float*)c.mpW.p, reinterpret_cast<bf16*>(c.mpWb.p));
    CIPC_CUDA(cudaGetLastError());
    c.mpFactorReady = false;
}

}  // namespace cipc
