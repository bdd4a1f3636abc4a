// Newton linear solve on the GPU: block-Jacobi preconditioned conjugate
// gradients on A = (static element BSR) + (contact BSR) + (per-vertex
// diagonal: mass, ground, soft), replacing NewtonLinearSystem::solve's
// backends (CPU IPC/NewtonLinearSystem.cpp:21-56, 176-207).  The stopping rule
// is Eigen's: ||r||^2 < tol^2 ||b||^2 with x0 = 0.
//
// A solve is one cooperative launch: rows staged in shared memory where they fit,
// else streamed in tiles or as block-CSR rows.  Groups of 4 lanes own block rows
// and combine with shuffles; partial sums are added in a fixed order, so no host
// round trip is needed inside an iteration and results are reproducible.
//
// Mixed precision: FP32 blocks, FP64 vectors; the stopping rule is decided on the
// true residual b - A x in FP64 (FP32 blocks promoted).
#include "cipc_device.cuh"
#include <cuda_fp16.h>
#include "cipc_gpu.h"
#include "cipc_internal.h"
#include "fsai.h"
#include "mpnn.h"

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdlib>

namespace cipc {

namespace {

constexpr int VB = 256;          // threads per block for vector kernels
constexpr int GROUP = 4;         // lanes per block row (measured: 4 lanes, 128 rows per block, one block per SM beat 8 lanes and two blocks per SM by 10 %)
constexpr int MAXPART = 512;
constexpr int PB = 512;          // threads per block of the persistent PCG
constexpr int PIPE_PMAX = 1024;  // partial-sum slots per array of the pipelined PCG (>= its grid)

inline int vecBlocks(int n) { return std::max(1, std::min((n + VB - 1) / VB, MAXPART)); }

template <class MT, class VT>
__device__ __forceinline__ void blockMulAdd(const MT* B, const VT* xv, VT acc[3]) {
    acc[0] += (VT)B[0] * xv[0] + (VT)B[1] * xv[1] + (VT)B[2] * xv[2];
    acc[1] += (VT)B[3] * xv[0] + (VT)B[4] * xv[1] + (VT)B[5] * xv[2];
    acc[2] += (VT)B[6] * xv[0] + (VT)B[7] * xv[1] + (VT)B[8] * xv[2];
}

// acc += B x for a 3x3 block of FP16 values (row-major)
template <class VT>
__device__ __forceinline__ void blockMulAddH(const __half* B, const VT* xv, VT acc[3]) {
    VT b[9];
#pragma unroll
    for (int e = 0; e < 9; ++e) b[e] = (VT)__half2float(B[e]);
    acc[0] += b[0] * xv[0] + b[1] * xv[1] + b[2] * xv[2];
    acc[1] += b[3] * xv[0] + b[4] * xv[1] + b[5] * xv[2];
    acc[2] += b[6] * xv[0] + b[7] * xv[1] + b[8] * xv[2];
}

// y = A x ; partial[block] = sum over the block's rows of x . y (for p.Ap)
template <class MT, class VT>
__global__ void spmvKernel(int nv, const int* rowPtr, const int* col, const MT* val, const int* dRowS, const int* dRowE, const int* dCol,
                           const MT* dVal, const double* diagExtra, const VT* x, VT* y) {
    int gid = blockIdx.x * blockDim.x + threadIdx.x;
    int lane = threadIdx.x & (GROUP - 1);
    int grp = (threadIdx.x & 31) / GROUP;
    const int RPW = 32 / GROUP;  // rows per warp per pass
    int nWarps = gridDim.x * blockDim.x / 32;
    // the loop bound is uniform across a warp, so every lane reaches the shuffles
    for (int base = (gid / 32) * RPW; base < nv; base += nWarps * RPW) {
        int row = base + grp;
        bool active = row < nv;
        VT acc[3] = {VT(0), VT(0), VT(0)};
        if (active) {
            for (int k = rowPtr[row] + lane; k < rowPtr[row + 1]; k += GROUP) {
                int c = col[k];
                VT xv[3] = {x[3 * c], x[3 * c + 1], x[3 * c + 2]};
                blockMulAdd(val + (size_t)9 * k, xv, acc);
            }
            if (dRowS) {
                for (int k = dRowS[row] + lane; k < dRowE[row]; k += GROUP) {
                    int c = dCol[k];
                    VT xv[3] = {x[3 * c], x[3 * c + 1], x[3 * c + 2]};
                    blockMulAdd(dVal + (size_t)9 * k, xv, acc);
                }
            }
        }
        for (int o = GROUP / 2; o > 0; o >>= 1)
            for (int q = 0; q < 3; ++q) acc[q] += __shfl_xor_sync(0xffffffffu, acc[q], o, GROUP);
        if (active && lane == 0) {
            VT xv[3] = {x[3 * row], x[3 * row + 1], x[3 * row + 2]};
            const double* D = diagExtra + 9 * row;
            for (int q = 0; q < 3; ++q) acc[q] += (VT)(D[3 * q] * (double)xv[0] + D[3 * q + 1] * (double)xv[1] + D[3 * q + 2] * (double)xv[2]);
            for (int q = 0; q < 3; ++q) y[3 * row + q] = acc[q];
        }
    }
}

// block-Jacobi inverse of the assembled diagonal blocks
template <class MT>
__global__ void dinvKernel(int nv, const int* diagSlot, const MT* val, const int* dRowS, const int* dRowE, const int* dCol, const MT* dVal,
                           const double* diagExtra, double* Dinv) {
    CIPC_KERNEL_LOOP(v, nv) {
        double D[9];
        for (int k = 0; k < 9; ++k) D[k] = diagExtra[9 * v + k];
        int s = diagSlot[v];
        if (s >= 0) for (int k = 0; k < 9; ++k) D[k] += (double)val[(size_t)9 * s + k];
        if (dRowS)
            for (int k = dRowS[v]; k < dRowE[v]; ++k)
                if (dCol[k] == v) for (int q = 0; q < 9; ++q) D[q] += (double)dVal[(size_t)9 * k + q];
        double c00 = D[4] * D[8] - D[5] * D[7], c10 = D[5] * D[6] - D[3] * D[8], c20 = D[3] * D[7] - D[4] * D[6];
        double det = D[0] * c00 + D[1] * c10 + D[2] * c20;
        double* o = Dinv + 9 * v;
        if (det == 0.0 || !isfinite(det)) { for (int k = 0; k < 9; ++k) o[k] = 0.0; continue; }
        o[0] = c00 / det; o[3] = c10 / det; o[6] = c20 / det;
        o[1] = (D[2] * D[7] - D[1] * D[8]) / det;
        o[4] = (D[0] * D[8] - D[2] * D[6]) / det;
        o[7] = (D[1] * D[6] - D[0] * D[7]) / det;
        o[2] = (D[1] * D[5] - D[2] * D[4]) / det;
        o[5] = (D[2] * D[3] - D[0] * D[5]) / det;
        o[8] = (D[0] * D[4] - D[1] * D[3]) / det;
    }
}

template <class VT>
__device__ __forceinline__ void applyDinv(const double* Dinv, const VT* r, VT* z, int v) {
    const double* D = Dinv + 9 * v;
    double r0 = r[3 * v], r1 = r[3 * v + 1], r2 = r[3 * v + 2];
    z[3 * v] = (VT)(D[0] * r0 + D[1] * r1 + D[2] * r2);
    z[3 * v + 1] = (VT)(D[3] * r0 + D[4] * r1 + D[5] * r2);
    z[3 * v + 2] = (VT)(D[6] * r0 + D[7] * r1 + D[8] * r2);
}

__global__ void rhsKernel(int nv, const double* g, const int* btype, double* b) {
    CIPC_KERNEL_LOOP(v, nv) {
        bool fr = btype[v] == 0;
        for (int q = 0; q < 3; ++q) b[3 * v + q] = fr ? g[3 * v + q] : 0.0;
    }
}

// r = b - Ax (FP64), rF = (float) r, partial |r|^2
__global__ void residualKernel(int n3, const double* b, const double* Ax, double* r, float* rF, double* part) {
    double rr = 0;
    CIPC_KERNEL_LOOP(i, n3) {
        double v = b[i] - Ax[i];
        r[i] = v;
        rF[i] = (float)v;
        rr += v * v;
    }
    double s = blockReduce(rr, AddOp(), 0.0);
    if (threadIdx.x == 0) part[blockIdx.x] = s;
}

__global__ void accumulateKernel(int n3, const float* d, double* x) {
    CIPC_KERNEL_LOOP(i, n3) x[i] += (double)d[i];
}

// ---------------------------------------------------------------------------
// Persistent PCG: the whole CG loop in one cooperative launch.
//
// Two grid barriers per iteration with block-Jacobi.  The direction update is
// folded into the SpMV phase through A p' = A z + beta A p, so each phase only
// reads vectors that the previous phase finished:
//   phase 1: p = z + beta p, Ap = A z + beta Ap, partial p.Ap     | barrier
//   phase 2: x += alpha p, r -= alpha Ap, z = M r, partial r.r, r.z | barrier
// With the learned factorised approximate inverse M = S^T G^T G S, phase 2
// splits in three (r and S r | t = G S r | z = S^T G^T t), four barriers per
// iteration.  A group of GROUP lanes owns one block row in every phase, so a
// row's x, r, p, Ap are only touched by their owner; z, S r and t are read by
// neighbours after a barrier.  Those reads are plain loads: the barrier's
// acquire (then __syncthreads) orders them after the other blocks' writes
// under the PTX memory model, and they may hit in L1, where the vertices
// that neighbouring rows of one SM share are fetched from L2 once.  Every block sums the
// per-block partials in the same order, so all blocks take the same branch and
// results are reproducible.  The barrier spin is bounded: on timeout it sets
// an error flag and the kernel returns.
// ---------------------------------------------------------------------------
// A matrix in tiles of 8 rows (streaming variant, below): tile t holds steps
// [tile[t], tile[t + 1]); a step holds one 3x3 block for each of a warp's 32
// lanes, its column (-1: none) and its nine values.
struct SellView {
    const int* tile;
    const int* col;
    const void* val;
};

template <class MT, class VT>
struct PcgArgs {
    int nv;
    const int *rowPtr, *col;
    const MT* val;
    const int *dRowS, *dRowE, *dCol;
    const MT* dVal;
    const double* diagExtra;
    const double* Dinv;
    // learned factor (null for block-Jacobi): S 9 per vertex, G slot-aligned
    const double* S;
    const float *gS, *gD;
    VT* t;
    const VT* b;
    VT *x, *r, *z, *p, *Ap;
    VT *u, *w, *mA, *mB, *q, *s;  // pipelined variants over block-CSR rows only
    // streaming variant: gathered vectors padded to 4 entries per row, the
    // tiled matrix and factor parts, whether the recurrence vectors live in
    // shared memory, and else where they live
    VT *g0, *g1, *g2, *g3, *state;
    SellView sA, sL, sU;
    int resident;
    double *partA, *partB, *partC;
    double* pp;                   // pipelined variant: two sets of three partial arrays, PIPE_PMAX each
    int sliceMax;                 // cached variant: static slots of the largest block row range
    int rowsPerBlock;             // cached variant: rows each block owns (<= ROWS_PER_BLOCK)
    int dynCap;                   // cached variant: contact slots a block's window may hold
    int cacheG;                   // cached variant with a factor: G blocks staged in shared memory
    double* scal;  // out: [3] rr, [4] iterations, [6] rhs2
    int* flag;     // out: 1 converged, 2 iteration cap, 3 barrier timeout
    unsigned* bar;  // BAR_WORDS words: grid-barrier counters and generation
    double tol;
    int maxIter;
};

// Two block sums with one pair of __syncthreads; the result is valid in
// every thread.  Partial sums follow a fixed order (reproducible).
__device__ __forceinline__ void blockReduce2(double& a, double& b) {
    __shared__ double s0[32], s1[32], r2[2];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
    for (int o = 16; o > 0; o >>= 1) {
        a += __shfl_xor_sync(0xffffffffu, a, o);
        b += __shfl_xor_sync(0xffffffffu, b, o);
    }
    __syncthreads();  // earlier readers of s0/s1/r2 are done
    if (lane == 0) { s0[w] = a; s1[w] = b; }
    __syncthreads();
    if (w == 0) {
        double x = lane < nw ? s0[lane] : 0.0, y = lane < nw ? s1[lane] : 0.0;
        for (int o = 16; o > 0; o >>= 1) {
            x += __shfl_xor_sync(0xffffffffu, x, o);
            y += __shfl_xor_sync(0xffffffffu, y, o);
        }
        if (lane == 0) { r2[0] = x; r2[1] = y; }
    }
    __syncthreads();
    a = r2[0];
    b = r2[1];
}

// Three block sums with one pair of __syncthreads (as blockReduce2).
__device__ __forceinline__ void blockReduce3(double& a, double& b, double& c) {
    __shared__ double s0[32], s1[32], s2[32], r3[3];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
    for (int o = 16; o > 0; o >>= 1) {
        a += __shfl_xor_sync(0xffffffffu, a, o);
        b += __shfl_xor_sync(0xffffffffu, b, o);
        c += __shfl_xor_sync(0xffffffffu, c, o);
    }
    __syncthreads();
    if (lane == 0) { s0[w] = a; s1[w] = b; s2[w] = c; }
    __syncthreads();
    if (w == 0) {
        double x = lane < nw ? s0[lane] : 0.0, y = lane < nw ? s1[lane] : 0.0, z = lane < nw ? s2[lane] : 0.0;
        for (int o = 16; o > 0; o >>= 1) {
            x += __shfl_xor_sync(0xffffffffu, x, o);
            y += __shfl_xor_sync(0xffffffffu, y, o);
            z += __shfl_xor_sync(0xffffffffu, z, o);
        }
        if (lane == 0) { r3[0] = x; r3[1] = y; r3[2] = z; }
    }
    __syncthreads();
    a = r3[0];
    b = r3[1];
    c = r3[2];
}

// Grid barrier on one arrival counter that only grows within a launch (it is
// zeroed before the launch): barrier number e is complete when the counter
// reaches e * nblocks.  Thread 0 arrives with an acquire-release atomic after
// the block's __syncthreads, which releases every write the block made before
// the barrier; the spin's acquire loads, followed by __syncthreads, order the
// block's later reads after the other blocks' writes.  One flat counter with
// these semantics measured 1.3 us per barrier on B200 for 148-296 blocks,
// against 2.9 us for a two-level tree of counters with full fences.
// The spin is bounded: on timeout the spinning thread sets flag = 3 and the
// barrier returns false; a block that returns early makes every other block
// time out at its next barrier, so no wait is unbounded.
constexpr int BAR_WORDS = 32;  // the counter, alone on its 128-byte line
constexpr long long BAR_SPIN_MAX = 1ll << 25;

__device__ __forceinline__ unsigned atomAddAcqRelGpu(unsigned* p, unsigned v) {
    unsigned old;
    asm volatile("atom.add.acq_rel.gpu.u32 %0, [%1], %2;" : "=r"(old) : "l"(p), "r"(v) : "memory");
    return old;
}
__device__ __forceinline__ unsigned ldAcquireGpu(const unsigned* p) {
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
// spin (acquire loads) until the counter reaches target; false on timeout
__device__ __forceinline__ bool barrierSpin(const unsigned* bar, int* flag, unsigned target) {
    long long spins = 0;
    while ((int)(ldAcquireGpu(bar) - target) < 0) {
        if (++spins > BAR_SPIN_MAX) { atomicExch(flag, 3); return false; }
    }
    return true;
}

__device__ __forceinline__ bool gridBarrier(unsigned* bar, int* flag, unsigned nblocks, unsigned& epoch) {
    const unsigned target = ++epoch * nblocks;
    __shared__ int ok;
    __syncthreads();
    if (threadIdx.x == 0) {
        int good = 1;
        if (atomAddAcqRelGpu(bar, 1u) + 1 != target) good = barrierSpin(bar, flag, target);
        ok = good;
    }
    __syncthreads();
    return ok != 0;
}

// Grid barrier followed by the sums of K per-block partial arrays (array j at
// P + j * stride, one entry per block, written before the barrier).  Warp 0
// waits (every lane spins with its own acquire loads), reads the partials in
// a fixed order and reduces them with shuffles, so every block gets the same
// bits; one __syncthreads hands the sums to the block.
template <int K>
__device__ __forceinline__ bool gridBarrierSum(unsigned* bar, int* flag, unsigned nblocks, unsigned& epoch, const double* P, size_t stride,
                                               double (&out)[K]) {
    const unsigned target = ++epoch * nblocks;
    __shared__ double res[K];
    __shared__ int ok;
    __syncthreads();
    if (threadIdx.x < 32) {
        const int lane = threadIdx.x;
        if (lane == 0) atomAddAcqRelGpu(bar, 1u);
        const bool good = __all_sync(0xffffffffu, barrierSpin(bar, flag, target));
        double v[K];
        for (int j = 0; j < K; ++j) v[j] = 0.0;
        if (good)
            for (int i = lane; i < (int)nblocks; i += 32)
                for (int j = 0; j < K; ++j) v[j] += __ldcg(P + j * stride + i);
        for (int o = 16; o > 0; o >>= 1)
            for (int j = 0; j < K; ++j) v[j] += __shfl_xor_sync(0xffffffffu, v[j], o);
        if (lane == 0) {
            for (int j = 0; j < K; ++j) res[j] = v[j];
            ok = good ? 1 : 0;
        }
    }
    __syncthreads();
    for (int j = 0; j < K; ++j) out[j] = res[j];
    return ok != 0;
}

// Row-group iteration shared by every phase: the same (block, lane group)
// owns the same rows in all phases.
struct RowIter {
    int lane, grp, first, stride, limit;
    __device__ RowIter() {
        int gid = blockIdx.x * blockDim.x + threadIdx.x;
        lane = threadIdx.x & (GROUP - 1);
        grp = (threadIdx.x & 31) / GROUP;
        first = (gid / 32) * (32 / GROUP);
        stride = gridDim.x * blockDim.x / 32 * (32 / GROUP);
        limit = 0x7fffffff;
    }
    // single pass over this block's own rows [blockIdx.x * rows, + rows) of nv
    __device__ RowIter(int nv, int rows) {
        lane = threadIdx.x & (GROUP - 1);
        grp = (threadIdx.x & 31) / GROUP;
        const int row0 = blockIdx.x * rows;
        first = row0 + (threadIdx.x / 32) * (32 / GROUP);
        stride = nv;
        limit = min(nv, row0 + rows);
    }
};

template <class VT>
__device__ __forceinline__ void groupReduce3(VT acc[3]) {
    for (int o = GROUP / 2; o > 0; o >>= 1)
        for (int q = 0; q < 3; ++q) acc[q] += __shfl_xor_sync(0xffffffffu, acc[q], o, GROUP);
}

// acc += (A u)_row over the row's static and contact blocks (lane-strided)
template <class MT, class VT>
__device__ __forceinline__ void rowSpmv(const PcgArgs<MT, VT>& a, int row, int lane, const VT* u, VT acc[3]) {
    for (int k = a.rowPtr[row] + lane; k < a.rowPtr[row + 1]; k += GROUP) {
        int c = a.col[k];
        VT xv[3] = {u[3 * c], u[3 * c + 1], u[3 * c + 2]};
        blockMulAdd(a.val + (size_t)9 * k, xv, acc);
    }
    if (a.dRowS) {
        for (int k = a.dRowS[row] + lane; k < a.dRowE[row]; k += GROUP) {
            int c = a.dCol[k];
            VT xv[3] = {u[3 * c], u[3 * c + 1], u[3 * c + 2]};
            blockMulAdd(a.dVal + (size_t)9 * k, xv, acc);
        }
    }
}

// acc += (G u)_row (TR = false: lower slots and the diagonal block) or
// (G^T u)_row (TR = true: mirror slots and the transposed diagonal block)
template <bool TR, class MT, class VT>
__device__ __forceinline__ void rowFactor(const PcgArgs<MT, VT>& a, int row, int lane, const VT* u, VT acc[3]) {
    for (int k = a.rowPtr[row] + lane; k < a.rowPtr[row + 1]; k += GROUP) {
        int c = a.col[k];
        if (TR ? c < row : c > row) continue;
        VT xv[3] = {u[3 * c], u[3 * c + 1], u[3 * c + 2]};
        const float* B = a.gS + (size_t)9 * k;
        if (TR && c == row) {
            for (int q = 0; q < 3; ++q) acc[q] += (VT)B[q] * xv[0] + (VT)B[3 + q] * xv[1] + (VT)B[6 + q] * xv[2];
        } else {
            blockMulAdd(B, xv, acc);
        }
    }
    if (a.dRowS) {
        for (int k = a.dRowS[row] + lane; k < a.dRowE[row]; k += GROUP) {
            int c = a.dCol[k];
            if (TR ? c <= row : c >= row) continue;
            VT xv[3] = {u[3 * c], u[3 * c + 1], u[3 * c + 2]};
            blockMulAdd(a.gD + (size_t)9 * k, xv, acc);
        }
    }
}

// z = M r for the learned factor, phases after r is final: writes S r into
// z, t = G (S r), z = S^T G^T t; returns this thread's r.z contribution
// (valid on lane 0 of each group).  Three barriers; false on barrier timeout.
template <class MT, class VT>
__device__ bool learnedApply(const PcgArgs<MT, VT>& a, const RowIter& it, double& rz, double* partRR, double rrLocal, unsigned& ep) {
    const unsigned nb = gridDim.x;
    for (int base = it.first; base < a.nv; base += it.stride) {
        int row = base + it.grp;
        if (row < a.nv && it.lane == 0) {
            const double* S = a.S + 9 * row;
            double r0 = a.r[3 * row], r1 = a.r[3 * row + 1], r2 = a.r[3 * row + 2];
            a.z[3 * row] = (VT)(S[0] * r0);
            a.z[3 * row + 1] = (VT)(S[3] * r0 + S[4] * r1);
            a.z[3 * row + 2] = (VT)(S[6] * r0 + S[7] * r1 + S[8] * r2);
        }
    }
    {
        double dummy = 0;
        blockReduce2(rrLocal, dummy);
        if (threadIdx.x == 0) partRR[blockIdx.x] = rrLocal;
    }
    if (!gridBarrier(a.bar, a.flag, nb, ep)) return false;
    for (int base = it.first; base < a.nv; base += it.stride) {
        int row = base + it.grp;
        bool active = row < a.nv;
        VT acc[3] = {VT(0), VT(0), VT(0)};
        if (active) rowFactor<false>(a, row, it.lane, (const VT*)a.z, acc);
        groupReduce3(acc);
        if (active && it.lane == 0)
            for (int q = 0; q < 3; ++q) a.t[3 * row + q] = acc[q];
    }
    if (!gridBarrier(a.bar, a.flag, nb, ep)) return false;
    rz = 0;
    for (int base = it.first; base < a.nv; base += it.stride) {
        int row = base + it.grp;
        bool active = row < a.nv;
        VT acc[3] = {VT(0), VT(0), VT(0)};
        if (active) rowFactor<true>(a, row, it.lane, (const VT*)a.t, acc);
        groupReduce3(acc);
        if (active && it.lane == 0) {
            const double* S = a.S + 9 * row;
            double y0 = acc[0], y1 = acc[1], y2 = acc[2];
            VT z0 = (VT)(S[0] * y0 + S[3] * y1 + S[6] * y2);
            VT z1 = (VT)(S[4] * y1 + S[7] * y2);
            VT z2 = (VT)(S[8] * y2);
            a.z[3 * row] = z0; a.z[3 * row + 1] = z1; a.z[3 * row + 2] = z2;
            rz += (double)a.r[3 * row] * (double)z0 + (double)a.r[3 * row + 1] * (double)z1 + (double)a.r[3 * row + 2] * (double)z2;
        }
    }
    return true;
}

template <class MT, class VT, bool LEARNED>
__global__ void __launch_bounds__(PB) pcgPersistentKernel(PcgArgs<MT, VT> a) {
    const unsigned nb = gridDim.x;
    unsigned ep = 0;
    const int nv = a.nv;
    const RowIter it;
    // init: x = 0, r = b, z = M r, p = 0, Ap = 0 (the first beta is 0)
    double rr = 0, rz = 0;
    for (int base = it.first; base < nv; base += it.stride) {
        int row = base + it.grp;
        if (row < nv && it.lane == 0) {
            for (int q = 0; q < 3; ++q) {
                a.x[3 * row + q] = VT(0); a.p[3 * row + q] = VT(0); a.Ap[3 * row + q] = VT(0);
                a.r[3 * row + q] = a.b[3 * row + q];
                rr += (double)a.r[3 * row + q] * (double)a.r[3 * row + q];
            }
            if (!LEARNED) {
                applyDinv(a.Dinv, a.r, a.z, row);
                for (int q = 0; q < 3; ++q) rz += (double)a.r[3 * row + q] * (double)a.z[3 * row + q];
            }
        }
    }
    if (LEARNED) {
        if (!learnedApply(a, it, rz, a.partA, rr, ep)) return;
        double dummy = 0;
        blockReduce2(rz, dummy);
        if (threadIdx.x == 0) a.partB[blockIdx.x] = rz;
    } else {
        blockReduce2(rr, rz);
        if (threadIdx.x == 0) { a.partA[blockIdx.x] = rr; a.partB[blockIdx.x] = rz; }
    }
    {
        double sums[2];
        if (!gridBarrierSum<2>(a.bar, a.flag, nb, ep, a.partA, a.partB - a.partA, sums)) return;
        rr = sums[0]; rz = sums[1];
    }
    const double rhs2 = rr;
    const double thr = fmax(a.tol * a.tol * rr, 2.2250738585072014e-308);
    int iter = 0;
    int status = (rr == 0.0 || rr < thr) ? 1 : 0;
    VT beta = VT(0);
    while (status == 0) {
        // phase 1: p = z + beta p ; Ap = A z + beta Ap ; p . Ap
        double d = 0;
        for (int base = it.first; base < nv; base += it.stride) {
            int row = base + it.grp;
            bool active = row < nv;
            VT acc[3] = {VT(0), VT(0), VT(0)};
            if (active) rowSpmv(a, row, it.lane, (const VT*)a.z, acc);
            groupReduce3(acc);
            if (active && it.lane == 0) {
                const double* D = a.diagExtra + 9 * row;
                VT zv[3] = {a.z[3 * row], a.z[3 * row + 1], a.z[3 * row + 2]};
                for (int q = 0; q < 3; ++q) acc[q] += (VT)(D[3 * q] * (double)zv[0] + D[3 * q + 1] * (double)zv[1] + D[3 * q + 2] * (double)zv[2]);
                for (int q = 0; q < 3; ++q) {
                    VT pv = zv[q] + beta * a.p[3 * row + q];
                    VT apv = acc[q] + beta * a.Ap[3 * row + q];
                    a.p[3 * row + q] = pv;
                    a.Ap[3 * row + q] = apv;
                    d += (double)pv * (double)apv;
                }
            }
        }
        {
            double dummy = 0;
            blockReduce2(d, dummy);
            if (threadIdx.x == 0) a.partC[blockIdx.x] = d;
        }
        double pAp[1];
        if (!gridBarrierSum<1>(a.bar, a.flag, nb, ep, a.partC, 0, pAp)) return;
        VT alpha = (VT)(rz / pAp[0]);
        // phase 2: x += alpha p ; r -= alpha Ap ; z = M r
        double lrr = 0, lrz = 0;
        for (int base = it.first; base < nv; base += it.stride) {
            int row = base + it.grp;
            if (row < nv && it.lane == 0) {
                for (int q = 0; q < 3; ++q) {
                    a.x[3 * row + q] += alpha * a.p[3 * row + q];
                    a.r[3 * row + q] -= alpha * a.Ap[3 * row + q];
                    lrr += (double)a.r[3 * row + q] * (double)a.r[3 * row + q];
                }
                if (!LEARNED) {
                    applyDinv(a.Dinv, a.r, a.z, row);
                    for (int q = 0; q < 3; ++q) lrz += (double)a.r[3 * row + q] * (double)a.z[3 * row + q];
                }
            }
        }
        if (LEARNED) {
            if (!learnedApply(a, it, lrz, a.partA, lrr, ep)) return;
            double dummy = 0;
            blockReduce2(lrz, dummy);
            if (threadIdx.x == 0) a.partB[blockIdx.x] = lrz;
        } else {
            blockReduce2(lrr, lrz);
            if (threadIdx.x == 0) { a.partA[blockIdx.x] = lrr; a.partB[blockIdx.x] = lrz; }
        }
        double sums[2];
        if (!gridBarrierSum<2>(a.bar, a.flag, nb, ep, a.partA, a.partB - a.partA, sums)) return;
        rr = sums[0];
        const double rzNew = sums[1];
        ++iter;
        if (rr < thr) { status = 1; break; }
        if (iter >= a.maxIter || !isfinite(rr)) { status = 2; break; }
        beta = (VT)(rzNew / rz);
        rz = rzNew;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        a.scal[3] = rr;
        a.scal[4] = iter;
        a.scal[6] = rhs2;
        atomicCAS(a.flag, 0, status);  // a barrier timeout (3) stands
    }
}

// ---------------------------------------------------------------------------
// Pipelined PCG (Ghysels and Vanroose's recurrences): the dot products of an
// iteration are formed in the same pass as its vector updates, and the
// preconditioned direction's product n = A m is carried by recurrences, so
// one iteration is one pass over the rows and ONE grid barrier with
// block-Jacobi (three with a factor: S w | G (S w) | S^T G^T t).
//   gamma = (r,u), delta = (w,u);  beta = gamma/gamma_old,
//   alpha = gamma / (delta - beta gamma / alpha_old)
//   n = A m;  z = n + beta z;  q = m + beta q;  s = w + beta s;  p = u + beta p
//   x += alpha p;  r -= alpha s;  u -= alpha q;  w -= alpha z;  m = M w
// With block-Jacobi the new m is written to the other of two buffers, since
// neighbours read the current one in the same pass; the partial sums also
// alternate between two sets, so a set is rewritten only two barriers after
// its last read.  The recurrences drift from the true residual in finite
// precision; the callers decide every solve on the true FP64 residual.
// ---------------------------------------------------------------------------
// Rows a block owns in a single-pass launch (PB / GROUP consecutive rows),
// staged once per solve in shared memory: the static slots (column and
// block, and with a factor its G block), the rows' contact blocks when the
// block's contact window fits, the diagonal extras, the 3x3 Jacobi inverse
// or the factor's scaling S, and the rows' recurrence vectors.  Every
// iteration then reads the matrix rows from shared memory and only the
// gathered vectors from L2.
constexpr int ROWS_PER_BLOCK = PB / GROUP;
// Rows per block of a small system: fewer and fuller blocks make the grid
// barrier and its sums cheaper, until the SMs left idle cost more.  Up to
// SINGLE_FILL_ROWS rows a block in an even spread over the SMs a block takes
// SINGLE_MIN_ROWS, beyond that the even share.  Measured per solve on a B200, with 64
// rows a block and with the even share (in brackets), ms:
//   even share 3-30: 432 rows 2.59 (2.77), 1,458 FP32 4.22 (4.61), 1,881 0.25
//   (0.27), 2,000 3.82 (4.22), 2,662 with a factor 6.35 (6.46), 4,329 0.49 (0.51),
//   4,394 4.09 (4.14);
//   even share 41-54: 6,001 0.49 (0.49), 6,750 4.55 (4.20), 6,932 2.38 (2.40),
//   7,954 FP32 1.05 (1.00), 8,001 0.56 (0.52).
constexpr int SINGLE_MIN_ROWS = 64, SINGLE_FILL_ROWS = 32;
constexpr int STATE_VECS = 9;  // x r u w z q s p, and the row's own m

struct SmemLayout {
    size_t dex, blk, val, gval, col, rp, drs, dval, dgval, dcol, state, total;
};
__host__ __device__ inline size_t alignUp16(size_t v) { return (v + 15) / 16 * 16; }
// offsets (16-byte aligned) of the cached arrays for a block of
// ROWS_PER_BLOCK rows with at most sliceMax static and dynCap contact slots
__host__ __device__ inline SmemLayout smemLayout(int sliceMax, int dynCap, bool cacheG, int msz, int vsz) {
    SmemLayout L{};
    size_t o = 0;
    L.dex = o;   o = alignUp16(o + (size_t)ROWS_PER_BLOCK * 9 * sizeof(double));
    L.blk = o;   o = alignUp16(o + (size_t)ROWS_PER_BLOCK * 9 * sizeof(double));
    L.val = o;   o = alignUp16(o + (size_t)sliceMax * 9 * msz);
    L.gval = o;  o = alignUp16(o + (cacheG ? (size_t)sliceMax * 9 * sizeof(float) : 0));
    L.col = o;   o = alignUp16(o + (size_t)sliceMax * sizeof(int));
    L.rp = o;    o = alignUp16(o + (size_t)(ROWS_PER_BLOCK + 1) * sizeof(int));
    L.drs = o;   o = alignUp16(o + (size_t)ROWS_PER_BLOCK * 2 * sizeof(int));
    L.dval = o;  o = alignUp16(o + (size_t)dynCap * 9 * msz);
    L.dgval = o; o = alignUp16(o + (cacheG ? (size_t)dynCap * 9 * sizeof(float) : 0));
    L.dcol = o;  o = alignUp16(o + (size_t)dynCap * sizeof(int));
    L.state = o; o = alignUp16(o + (size_t)STATE_VECS * ROWS_PER_BLOCK * 3 * vsz);
    L.total = o;
    return L;
}

template <class MT>
struct RowCache {
    int row0, s0;
    int d0;              // global index of the first cached contact slot; -1: contact blocks are read from global memory
    const int* rp;       // ROWS_PER_BLOCK + 1 static slot offsets (global slot indices)
    const int* col;
    const MT* val;
    const float* gval;   // factor blocks of the static slots (null: read from global memory)
    const int* drs;      // contact slot range [start, end) per row (global slot indices)
    const int* dcol;
    const MT* dval;
    const float* dgval;  // factor blocks of the cached contact slots (null: global)
    const double* dex;   // diagonal extras, 9 per row
    const double* blk;   // 9 per row: the Jacobi inverse, or the factor's scaling S
};

template <class MT, class VT, bool LEARNED>
__device__ RowCache<MT> loadRowCache(const PcgArgs<MT, VT>& a, unsigned char* smem) {
    const bool cacheG = LEARNED && a.cacheG != 0;
    const SmemLayout L = smemLayout(a.sliceMax, a.dynCap, cacheG, (int)sizeof(MT), (int)sizeof(VT));
    double* dex = reinterpret_cast<double*>(smem + L.dex);
    double* blk = reinterpret_cast<double*>(smem + L.blk);
    MT* val = reinterpret_cast<MT*>(smem + L.val);
    float* gval = reinterpret_cast<float*>(smem + L.gval);
    int* col = reinterpret_cast<int*>(smem + L.col);
    int* rp = reinterpret_cast<int*>(smem + L.rp);
    int* drs = reinterpret_cast<int*>(smem + L.drs);
    MT* dval = reinterpret_cast<MT*>(smem + L.dval);
    float* dgval = reinterpret_cast<float*>(smem + L.dgval);
    int* dcol = reinterpret_cast<int*>(smem + L.dcol);
    __shared__ int dlo, dhi;
    RowCache<MT> rc;
    rc.row0 = blockIdx.x * a.rowsPerBlock;
    const int nrows = min(a.rowsPerBlock, a.nv - rc.row0);  // >= 1: the grid is ceil(nv / rowsPerBlock)
    if (threadIdx.x == 0) { dlo = 0x7fffffff; dhi = 0; }
    for (int i = threadIdx.x; i <= nrows; i += blockDim.x) rp[i] = a.rowPtr[rc.row0 + i];
    __syncthreads();
    for (int i = threadIdx.x; i < nrows; i += blockDim.x) {
        int s = 0, e = 0;
        if (a.dRowS) { s = a.dRowS[rc.row0 + i]; e = a.dRowE[rc.row0 + i]; }
        drs[2 * i] = s;
        drs[2 * i + 1] = e;
        if (e > s) { atomicMin(&dlo, s); atomicMax(&dhi, e); }
    }
    rc.s0 = rp[0];
    const int ns = rp[nrows] - rc.s0;  // <= sliceMax (host-computed maximum over blocks)
    for (int k = threadIdx.x; k < ns; k += blockDim.x) col[k] = a.col[rc.s0 + k];
    for (int k = threadIdx.x; k < 9 * ns; k += blockDim.x) val[k] = a.val[(size_t)9 * rc.s0 + k];
    if (cacheG)
        for (int k = threadIdx.x; k < 9 * ns; k += blockDim.x) gval[k] = a.gS[(size_t)9 * rc.s0 + k];
    const double* srcBlk = LEARNED ? a.S : a.Dinv;
    for (int k = threadIdx.x; k < 9 * nrows; k += blockDim.x) {
        dex[k] = a.diagExtra[(size_t)9 * rc.row0 + k];
        blk[k] = srcBlk[(size_t)9 * rc.row0 + k];
    }
    __syncthreads();  // dlo / dhi complete
    // the rows' contact slots are one contiguous window (row-sorted)
    const int nd = dhi > dlo ? dhi - dlo : 0;
    rc.d0 = (nd > 0 && nd <= a.dynCap) ? dlo : -1;
    if (rc.d0 >= 0) {
        for (int k = threadIdx.x; k < nd; k += blockDim.x) dcol[k] = a.dCol[dlo + k];
        for (int k = threadIdx.x; k < 9 * nd; k += blockDim.x) dval[k] = a.dVal[(size_t)9 * dlo + k];
        if (cacheG)
            for (int k = threadIdx.x; k < 9 * nd; k += blockDim.x) dgval[k] = a.gD[(size_t)9 * dlo + k];
    }
    __syncthreads();
    rc.rp = rp; rc.col = col; rc.val = val; rc.gval = cacheG ? gval : nullptr;
    rc.drs = drs; rc.dcol = dcol; rc.dval = dval; rc.dgval = cacheG ? dgval : nullptr;
    rc.dex = dex; rc.blk = blk;
    return rc;
}

// acc = (A u)_row without the diagonal extras, from the cache; every lane of
// the row's group gets the sum
template <class MT, class VT>
__device__ __forceinline__ void rowAxCached(const PcgArgs<MT, VT>& a, const RowCache<MT>& rc, const RowIter& it, int row, const VT* u,
                                            VT acc[3]) {
    const int lr = row - rc.row0;
    if (row < it.limit) {
        const int kb = rc.rp[lr] - rc.s0, ke = rc.rp[lr + 1] - rc.s0;
        // two of the lane's slots per round: both gathers are issued before
        // the products, which stay in slot order
        for (int kk = kb + it.lane; kk < ke; kk += 2 * GROUP) {
            const int k1 = kk + GROUP;
            const bool two = k1 < ke;
            const int c0 = rc.col[kk], c1 = two ? rc.col[k1] : c0;
            const VT x0[3] = {u[3 * c0], u[3 * c0 + 1], u[3 * c0 + 2]};
            const VT x1[3] = {u[3 * c1], u[3 * c1 + 1], u[3 * c1 + 2]};
            blockMulAdd(rc.val + (size_t)9 * kk, x0, acc);
            if (two) blockMulAdd(rc.val + (size_t)9 * k1, x1, acc);
        }
        const int ds = rc.drs[2 * lr], de = rc.drs[2 * lr + 1];
        if (rc.d0 >= 0) {
            for (int k = ds + it.lane; k < de; k += GROUP) {
                int kk = k - rc.d0;
                int c = rc.dcol[kk];
                VT xv[3] = {u[3 * c], u[3 * c + 1], u[3 * c + 2]};
                blockMulAdd(rc.dval + (size_t)9 * kk, xv, acc);
            }
        } else {
            for (int k = ds + it.lane; k < de; k += GROUP) {
                int c = a.dCol[k];
                VT xv[3] = {u[3 * c], u[3 * c + 1], u[3 * c + 2]};
                blockMulAdd(a.dVal + (size_t)9 * k, xv, acc);
            }
        }
    }
    groupReduce3(acc);
}

// (G u)_row (TR false) or (G^T u)_row (TR true) from the cache, as rowFactor
template <bool TR, class MT, class VT>
__device__ __forceinline__ void rowFactorCached(const PcgArgs<MT, VT>& a, const RowCache<MT>& rc, const RowIter& it, int row, const VT* u,
                                                VT acc[3]) {
    const int lr = row - rc.row0;
    const int kb = rc.rp[lr] - rc.s0, ke = rc.rp[lr + 1] - rc.s0;
    // the factor block of slot kk (transposed on the diagonal of G^T)
    auto slotMulAdd = [&](int kk, int c, const VT* xv) {
        const float* B = rc.gval ? rc.gval + (size_t)9 * kk : a.gS + (size_t)9 * (kk + rc.s0);
        if (TR && c == row) {
            for (int q = 0; q < 3; ++q) acc[q] += (VT)B[q] * xv[0] + (VT)B[3 + q] * xv[1] + (VT)B[6 + q] * xv[2];
        } else {
            blockMulAdd(B, xv, acc);
        }
    };
    // two of the lane's slots per round, as rowAxCached; slots outside this
    // pass's triangle are skipped
    for (int kk = kb + it.lane; kk < ke; kk += 2 * GROUP) {
        const int k1 = kk + GROUP;
        const int c0 = rc.col[kk], c1 = k1 < ke ? rc.col[k1] : row;
        const bool on0 = !(TR ? c0 < row : c0 > row), on1 = k1 < ke && !(TR ? c1 < row : c1 > row);
        const int g0 = on0 ? c0 : row, g1 = on1 ? c1 : row;
        const VT x0[3] = {u[3 * g0], u[3 * g0 + 1], u[3 * g0 + 2]};
        const VT x1[3] = {u[3 * g1], u[3 * g1 + 1], u[3 * g1 + 2]};
        if (on0) slotMulAdd(kk, c0, x0);
        if (on1) slotMulAdd(k1, c1, x1);
    }
    const int ds = rc.drs[2 * lr], de = rc.drs[2 * lr + 1];
    for (int k = ds + it.lane; k < de; k += GROUP) {
        const bool cached = rc.d0 >= 0;
        int c = cached ? rc.dcol[k - rc.d0] : a.dCol[k];
        if (TR ? c <= row : c >= row) continue;
        VT xv[3] = {u[3 * c], u[3 * c + 1], u[3 * c + 2]};
        blockMulAdd((cached && rc.dgval) ? rc.dgval + (size_t)9 * (k - rc.d0) : a.gD + (size_t)9 * k, xv, acc);
    }
}

// out = S^T G^T G tmp for the factor, where tmp = S w was written by the
// rows' owners before the call: barrier, t = G tmp, barrier, out = S^T G^T t
// into outG (gathered by neighbours) and into the owner's shared copy
// own[3 * local row + q].  Ends without a barrier; false on timeout.
template <class MT, class VT>
__device__ bool factorCachedPasses(const PcgArgs<MT, VT>& a, const RowCache<MT>& rc, const RowIter& it, const VT* tmp, VT* outG, VT* own,
                                   unsigned& ep) {
    const unsigned nb = gridDim.x;
    if (!gridBarrier(a.bar, a.flag, nb, ep)) return false;
    for (int base = it.first; base < it.limit; base += it.stride) {
        int row = base + it.grp;
        bool active = row < it.limit;
        VT acc[3] = {VT(0), VT(0), VT(0)};
        if (active) rowFactorCached<false>(a, rc, it, row, tmp, acc);
        groupReduce3(acc);
        // lanes 0, 1, 2 of the group store components 0, 1, 2
        const int q = it.lane;
        if (active && q < 3) a.t[3 * row + q] = q == 0 ? acc[0] : (q == 1 ? acc[1] : acc[2]);
    }
    if (!gridBarrier(a.bar, a.flag, nb, ep)) return false;
    for (int base = it.first; base < it.limit; base += it.stride) {
        int row = base + it.grp;
        bool active = row < it.limit;
        VT acc[3] = {VT(0), VT(0), VT(0)};
        if (active) rowFactorCached<true>(a, rc, it, row, (const VT*)a.t, acc);
        groupReduce3(acc);
        const int q = it.lane;
        if (active && q < 3) {
            // component q of S^T y (S lower triangular)
            const int lr = row - rc.row0;
            const double* S = rc.blk + 9 * lr;
            const double y0 = acc[0], y1 = acc[1], y2 = acc[2];
            const VT o = (VT)(q == 0 ? S[0] * y0 + S[3] * y1 + S[6] * y2 : (q == 1 ? S[4] * y1 + S[7] * y2 : S[8] * y2));
            outG[3 * row + q] = o;
            own[3 * lr + q] = o;
        }
    }
    return true;
}

// The single-pass launch: a block owns the same rows for the whole solve.
template <class MT, class VT, bool LEARNED>
__global__ void __launch_bounds__(PB, 2) pcgPipelinedKernel(PcgArgs<MT, VT> a) {
    extern __shared__ __align__(16) unsigned char pipeSmem[];
    // The block's matrix rows and its rows' recurrence vectors live in shared
    // memory: only the gathered vectors (u once; m, and with a factor S w and
    // t, every iteration), the partial sums and the solution at the end touch
    // global memory.  Lanes 0, 1, 2 of a row's group update components 0, 1, 2
    // of the row's vectors.
    const unsigned nb = gridDim.x;
    unsigned ep = 0;
    const RowIter it(a.nv, a.rowsPerBlock);
    const int rEnd = it.limit;  // rows this thread's loops cover end here
    const int q = it.lane;  // the component this lane updates (q < 3)
    const RowCache<MT> rc = loadRowCache<MT, VT, LEARNED>(a, pipeSmem);
    VT* const sv = reinterpret_cast<VT*>(
        pipeSmem + smemLayout(a.sliceMax, a.dynCap, LEARNED && a.cacheG != 0, (int)sizeof(MT), (int)sizeof(VT)).state);
    // component q of own-row vector k (0 x, 1 r, 2 u, 3 w, 4 z, 5 q, 6 s, 7 p)
    auto V = [&](int k, int row) -> VT& { return sv[(k * ROWS_PER_BLOCK + (row - rc.row0)) * 3 + q]; };
    VT* const ownM = sv + 8 * ROWS_PER_BLOCK * 3;  // the rows' own m (shared copy)
    VT* const ownU = sv + 2 * ROWS_PER_BLOCK * 3;
    auto pick = [&](const VT v[3]) { return q == 0 ? v[0] : (q == 1 ? v[1] : v[2]); };
    // component q of D v for a row's 3x3 block D (row-major), v given whole
    auto rowDot = [&](const double* D, const VT v[3]) {
        return (VT)(D[3 * q] * (double)v[0] + D[3 * q + 1] * (double)v[1] + D[3 * q + 2] * (double)v[2]);
    };
    auto dexRow = [&](int row) { return rc.dex + 9 * (row - rc.row0); };
    auto blkRow = [&](int row) { return rc.blk + 9 * (row - rc.row0); };
    // the group's three components of v (held by lanes 0, 1, 2); every lane calls
    auto share3 = [&](VT v, VT out[3]) {
        out[0] = __shfl_sync(0xffffffffu, v, 0, GROUP);
        out[1] = __shfl_sync(0xffffffffu, v, 1, GROUP);
        out[2] = __shfl_sync(0xffffffffu, v, 2, GROUP);
    };
    VT* sw = a.Ap;  // S w, gathered by the factor's first pass
    // the row's M-related output from the group's three components of v:
    // block-Jacobi m = Dinv v into mOut (and the shared copy), or with a
    // factor S v into sw, the input of the factor's first pass; lanes q < 3
    // of active rows store
    auto precondRow = [&](int row, bool active, const VT v[3], VT* mOut) {
        if (!active || q >= 3) return;
        if (!LEARNED) {
            const VT mq = rowDot(blkRow(row), v);
            mOut[3 * row + q] = mq;
            ownM[3 * (row - rc.row0) + q] = mq;
        } else {
            // lower triangular
            const double* S = rc.blk + 9 * (row - rc.row0);
            const double v0 = v[0], v1 = v[1], v2 = v[2];
            sw[3 * row + q] = (VT)(q == 0 ? S[0] * v0 : (q == 1 ? S[3] * v0 + S[4] * v1 : S[6] * v0 + S[7] * v1 + S[8] * v2));
        }
    };
    auto part = [&](int set, int k) { return a.pp + (size_t)(3 * set + k) * PIPE_PMAX; };
    // x = 0, r = b, u = M r; the recurrence vectors start at 0
    double rr = 0;
    for (int base = it.first; base < rEnd; base += it.stride) {
        const int row = base + it.grp;
        const bool active = row < rEnd;
        VT rq = VT(0);
        if (active && q < 3) {
            V(0, row) = VT(0); V(4, row) = VT(0); V(5, row) = VT(0); V(6, row) = VT(0); V(7, row) = VT(0);
            rq = a.b[3 * row + q];
            V(1, row) = rq;
            rr += (double)rq * (double)rq;
        }
        VT rv[3];
        share3(rq, rv);
        if (!LEARNED) {
            if (active && q < 3) {
                const VT uq = rowDot(blkRow(row), rv);
                V(2, row) = uq;
                a.u[3 * row + q] = uq;
            }
        } else {
            precondRow(row, active, rv, nullptr);
        }
    }
    if (LEARNED && !factorCachedPasses(a, rc, it, (const VT*)sw, a.u, ownU, ep)) return;
    if (!gridBarrier(a.bar, a.flag, nb, ep)) return;
    // w = A u, m = M w, gamma = (r,u), delta = (w,u)
    double g = 0, dl = 0;
    for (int base = it.first; base < rEnd; base += it.stride) {
        const int row = base + it.grp;
        const bool active = row < rEnd;
        VT acc[3] = {VT(0), VT(0), VT(0)};
        rowAxCached(a, rc, it, row, (const VT*)a.u, acc);
        VT wq = VT(0);
        if (active && q < 3) {
            const VT* uOwn = ownU + 3 * (row - rc.row0);
            const VT uo[3] = {uOwn[0], uOwn[1], uOwn[2]};
            wq = pick(acc) + rowDot(dexRow(row), uo);
            V(3, row) = wq;
            const VT uq = V(2, row);
            g += (double)V(1, row) * (double)uq;
            dl += (double)wq * (double)uq;
        }
        VT wv[3];
        share3(wq, wv);
        precondRow(row, active, wv, a.mA);
    }
    blockReduce3(rr, g, dl);
    if (threadIdx.x == 0) { part(0, 0)[blockIdx.x] = rr; part(0, 1)[blockIdx.x] = g; part(0, 2)[blockIdx.x] = dl; }
    if (LEARNED && !factorCachedPasses(a, rc, it, (const VT*)sw, a.mA, ownM, ep)) return;
    {
        double sums[3];
        if (!gridBarrierSum<3>(a.bar, a.flag, nb, ep, part(0, 0), PIPE_PMAX, sums)) return;
        rr = sums[0]; g = sums[1]; dl = sums[2];
    }
    const double rhs2 = rr;
    const double thr = fmax(a.tol * a.tol * rr, 2.2250738585072014e-308);
    int iter = 0;
    int status = (rr == 0.0 || rr < thr) ? 1 : 0;
    double gPrev = 1.0, alphaPrev = 1.0;
    while (status == 0) {
        double beta = iter == 0 ? 0.0 : g / gPrev;
        double den = iter == 0 ? dl : dl - beta * g / alphaPrev;
        if (!(den != 0.0) || !isfinite(den)) { status = 2; break; }  // breakdown: the caller's true residual decides
        double alpha = g / den;
        const VT* mCur = (LEARNED || (iter & 1) == 0) ? a.mA : a.mB;
        VT* mNext = LEARNED ? a.mA : ((iter & 1) == 0 ? a.mB : a.mA);
        const VT bt = (VT)beta, al = (VT)alpha;
        double lrr = 0, lg = 0, ld = 0;
        for (int base = it.first; base < rEnd; base += it.stride) {
            const int row = base + it.grp;
            const bool active = row < rEnd;
            VT acc[3] = {VT(0), VT(0), VT(0)};
            rowAxCached(a, rc, it, row, mCur, acc);
            VT wq = VT(0);
            if (active && q < 3) {
                const VT* mOwn = ownM + 3 * (row - rc.row0);
                const VT mo[3] = {mOwn[0], mOwn[1], mOwn[2]};
                const VT zv = pick(acc) + rowDot(dexRow(row), mo) + bt * V(4, row);
                const VT qv = pick(mo) + bt * V(5, row);
                const VT sq = V(3, row) + bt * V(6, row);
                const VT pv = V(2, row) + bt * V(7, row);
                V(4, row) = zv; V(5, row) = qv; V(6, row) = sq; V(7, row) = pv;
                V(0, row) += al * pv;
                const VT rv = V(1, row) - al * sq;
                const VT uv = V(2, row) - al * qv;
                wq = V(3, row) - al * zv;
                V(1, row) = rv; V(2, row) = uv; V(3, row) = wq;
                lrr += (double)rv * (double)rv;
                lg += (double)rv * (double)uv;
                ld += (double)wq * (double)uv;
            }
            VT wv[3];
            share3(wq, wv);
            precondRow(row, active, wv, mNext);
        }
        const int set = (iter + 1) & 1;
        blockReduce3(lrr, lg, ld);
        if (threadIdx.x == 0) { part(set, 0)[blockIdx.x] = lrr; part(set, 1)[blockIdx.x] = lg; part(set, 2)[blockIdx.x] = ld; }
        // the factor's m is replaced only in its last pass, two barriers
        // after every row read it
        if (LEARNED && !factorCachedPasses(a, rc, it, (const VT*)sw, mNext, ownM, ep)) return;
        double sums[3];
        if (!gridBarrierSum<3>(a.bar, a.flag, nb, ep, part(set, 0), PIPE_PMAX, sums)) return;
        gPrev = g;
        alphaPrev = alpha;
        rr = sums[0]; g = sums[1]; dl = sums[2];
        ++iter;
        if (rr < thr) { status = 1; break; }
        if (iter >= a.maxIter || !isfinite(rr)) { status = 2; break; }
    }
    // the solution leaves shared memory
    for (int base = it.first; base < rEnd; base += it.stride) {
        const int row = base + it.grp;
        if (row < rEnd && q < 3) a.x[3 * row + q] = V(0, row);
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        a.scal[3] = rr;
        a.scal[4] = iter;
        a.scal[6] = rhs2;
        atomicCAS(a.flag, 0, status);  // a barrier timeout (3) stands
    }
}

// ---------------------------------------------------------------------------
// Streaming pipelined PCG, for systems whose rows do not fit the chip's shared
// memory: the recurrences of pcgPipelinedKernel over matrices in tiles.
//
// A warp takes 8 rows at a time, 4 lanes to a row.  In block-CSR order each of
// a lane's nine loads of a block touched lines of all 8 rows, at 40 registers
// with 48 warps, and the loads waited for one another.  The tiles hold the
// blocks of one step of the warp lane by lane (16 bytes per lane and load), so
// every load is one contiguous run; a lane without a block has column -1 and
// reads no values.  The gathered vectors have 4 entries per row, one 32-byte
// load each.  A block owns a contiguous run of tiles, the same in every pass,
// and keeps its rows' eight recurrence vectors in shared memory where they fit
// (STREAM_STATE_BYTES): on the 64-cube pile 54 MB less traffic per iteration.
// Sums run in the order of the block-CSR rows.
//
// Bound by memory latency within L2 and by memory beyond it.  Measured per
// solve on a B200, block-CSR rows -> tiles: 13x81 twist (FP64, block-Jacobi, 427
// iterations) 9.3 -> 4.5 ms, 27-cube pile (FP32 blocks) 16.7 -> 7.9 ms, with the
// factor 16.4 -> 10.9 ms, 64-cube pile 27.9 -> 15.0 ms, with the factor 25.9 ->
// 23.8 ms.
// ---------------------------------------------------------------------------
// Warps per block, one block per SM.  A system within L2 waits for latency:
// 16 warps, two steps of a row in flight (128 registers).  One beyond it waits
// for memory: 24 warps, one step each, the next tile fetched ahead (80
// registers).  Measured, in ms per solve: 64-cube pile 14.9 against 16.7 with 16
// warps, with the factor 23.8 against 26.7; 13x81 twist 4.5 without the fetch
// and the priorities against 5.4 with them.
constexpr int streamWarps(bool beyond) { return beyond ? 24 : 16; }
// Beyond when an iteration's data exceed this share of L2 (63 MB): 27-cube pile,
// 45 MB, 7.9 ms within and 9.2 beyond; with the factor, 75 MB, 11.8 and 10.9.
constexpr double STREAM_L2_SHARE = 0.5;
// Tiles suit rows that are alike: their steps past each tile's first (which is
// there even for a single block) hold at most SELL_PAD slots per block.  The meshes of
// the scenes are at 0.8-1.15.  Past it tiles still suit if they lie within L2 and no
// tile is longer than SELL_LONG steps.  Measured per iteration on a B200 in tiles and in
// block-CSR rows (pcgRowsKernel), us, FP64 and FP32 blocks, 40,011 rows unless said:
//   every 8th row joined to 24 others 12.7 and 17.1, 11.8 and 14.9; every 2nd to 30
//   17.0 and 24.4, 15.5 and 20.3 (within L2: 53-118 MB); every 8th to 60 32 and
//   25 (203 MB), 20.9 and 21.0 (111 MB); every 32nd to 100 (26 steps) 21.8 and 20.4,
//   24.4 and 20.2; every 2nd to 200 151 and 96, 96 and 79; 200,011 rows, every 8th to 12
//   66 and 53, 52 and 42 (170 MB).
constexpr double SELL_PAD = 1.5;
constexpr int SELL_LONG = 16;
constexpr size_t STREAM_STATE_BYTES = 192 * 1024;  // recurrence vectors in shared memory, per SM

// fetch [p, p + bytes) into L2 (both multiples of 16)
__device__ __forceinline__ void prefetchL2(const void* p, int bytes, uint64_t pol) {
    asm volatile("cp.async.bulk.prefetch.L2.global.L2::cache_hint [%0], %1, %2;" ::"l"(p), "r"(bytes), "l"(pol));
}

// entries 0-2 of row c of a padded vector, in one 32-byte load
__device__ __forceinline__ void gather3(const double* u, int c, double x[3]) {
    double pad;
    asm volatile("ld.global.v4.f64 {%0, %1, %2, %3}, [%4];" : "=d"(x[0]), "=d"(x[1]), "=d"(x[2]), "=d"(pad) : "l"(u + 4 * (size_t)c));
}

// L2 priority of streamed data in a system beyond L2: the matrix goes first, so
// that the factor and the vectors stay
template <bool FIRST>
__device__ __forceinline__ uint64_t streamPolicy() {
    uint64_t p;
    if (FIRST) asm("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(p));
    else asm("createpolicy.fractional.L2::evict_normal.b64 %0, 1.0;" : "=l"(p));
    return p;
}
// constant data, read once per pass: past L1
__device__ __forceinline__ uint4 streamLoad16(const void* p, uint64_t pol) {
    uint4 v;
    asm("ld.global.nc.L1::no_allocate.L2::cache_hint.v4.u32 {%0, %1, %2, %3}, [%4], %5;"
        : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p), "l"(pol));
    return v;
}
__device__ __forceinline__ void streamLoad(const float* p, uint64_t pol, float& v) {
    asm("ld.global.nc.L1::no_allocate.L2::cache_hint.f32 %0, [%1], %2;" : "=f"(v) : "l"(p), "l"(pol));
}
__device__ __forceinline__ void streamLoad(const double* p, uint64_t pol, double& v) {
    asm("ld.global.nc.L1::no_allocate.L2::cache_hint.f64 %0, [%1], %2;" : "=d"(v) : "l"(p), "l"(pol));
}
__device__ __forceinline__ void streamLoad(const unsigned short* p, uint64_t pol, unsigned short& v) {
    asm("ld.global.nc.L1::no_allocate.L2::cache_hint.u16 %0, [%1], %2;" : "=h"(v) : "l"(p), "l"(pol));
}
__device__ __forceinline__ int streamLoad(const int* p, uint64_t pol) {
    int v;
    asm("ld.global.nc.L1::no_allocate.L2::cache_hint.s32 %0, [%1], %2;" : "=r"(v) : "l"(p), "l"(pol));
    return v;
}

// one lane's block of a step
template <class T>
struct SellBlock;
template <>
struct SellBlock<float> {
    uint4 a, b;
    float c;
    __device__ __forceinline__ void load(const void* step, int lane, uint64_t pol) {
        a = streamLoad16((const uint4*)step + lane, pol);
        b = streamLoad16((const uint4*)step + 32 + lane, pol);
        streamLoad((const float*)step + 256 + lane, pol, c);
    }
    __device__ __forceinline__ void mulAdd(const double x[3], double acc[3]) const {
        const float B[9] = {__uint_as_float(a.x), __uint_as_float(a.y), __uint_as_float(a.z), __uint_as_float(a.w), __uint_as_float(b.x),
                            __uint_as_float(b.y), __uint_as_float(b.z), __uint_as_float(b.w), c};
        blockMulAdd(B, x, acc);
    }
};
template <>
struct SellBlock<double> {
    uint4 a[4];
    double e;
    __device__ __forceinline__ void load(const void* step, int lane, uint64_t pol) {
#pragma unroll
        for (int k = 0; k < 4; ++k) a[k] = streamLoad16((const uint4*)step + 32 * k + lane, pol);
        streamLoad((const double*)step + 256 + lane, pol, e);
    }
    __device__ __forceinline__ void mulAdd(const double x[3], double acc[3]) const {
        double B[9];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            B[2 * k] = __hiloint2double((int)a[k].y, (int)a[k].x);
            B[2 * k + 1] = __hiloint2double((int)a[k].w, (int)a[k].z);
        }
        B[8] = e;
        blockMulAdd(B, x, acc);
    }
};
template <>
struct SellBlock<__half> {
    uint4 a;
    unsigned short b;
    __device__ __forceinline__ void load(const void* step, int lane, uint64_t pol) {
        a = streamLoad16((const uint4*)step + lane, pol);
        streamLoad((const unsigned short*)step + 256 + lane, pol, b);
    }
    __device__ __forceinline__ void mulAdd(const double x[3], double acc[3]) const {
        const unsigned w[4] = {a.x, a.y, a.z, a.w};
        __half B[9];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            B[2 * k] = __ushort_as_half((unsigned short)(w[k] & 0xffffu));
            B[2 * k + 1] = __ushort_as_half((unsigned short)(w[k] >> 16));
        }
        B[8] = __ushort_as_half(b);
        blockMulAddH(B, x, acc);
    }
};

// A warp's way through its tiles of one pass: the step ranges of the current
// and the next tile.  Beyond L2, the next tile's columns and values are fetched
// into it by one bulk prefetch each while a tile is worked on.
template <bool BEYOND>
struct SellCursor {
    static constexpr int W = streamWarps(BEYOND);
    int s, n, sn, nn;
    __device__ __forceinline__ void start(const SellView& m, int tile, int hi) {
        s = n = 0;
        if (tile < hi) { s = __ldcg(m.tile + tile); n = __ldcg(m.tile + tile + 1) - s; }
        sn = nn = 0;
        tile += W;
        if (tile < hi) { sn = __ldcg(m.tile + tile); nn = __ldcg(m.tile + tile + 1) - sn; }
    }
    template <class T, bool FIRST>
    __device__ __forceinline__ void prefetch(const SellView& m, int s, int n) const {
        if (BEYOND && n > 0 && (threadIdx.x & 31) == 0) {
            const uint64_t pol = streamPolicy<FIRST>();
            prefetchL2(m.col + (size_t)s * 32, n * 128, pol);
            prefetchL2((const char*)m.val + (size_t)s * (288 * sizeof(T)), n * (int)(288 * sizeof(T)), pol);
        }
    }
    // at the end of a tile: on to the next, and the range after it
    __device__ __forceinline__ void next(const SellView& m, int tile, int hi) {
        s = sn; n = nn;
        sn = nn = 0;
        tile += 2 * W;
        if (tile < hi) { sn = __ldcg(m.tile + tile); nn = __ldcg(m.tile + tile + 1) - sn; }
    }
};

// acc += (M u)_row over the tile's static blocks of this lane.  A round of two
// steps (one of FP64 blocks, or beyond L2: registers) requests its gathers and values, and
// the next round's columns, before the products.
template <class T, bool BEYOND, bool FIRST>
__device__ __forceinline__ void sellRow(const SellView& m, int s0, int n, const double* u, double acc[3]) {
    constexpr int R = BEYOND || sizeof(T) == 8 ? 1 : 2;
    int wl = threadIdx.x & 31;
    asm volatile("" : "+r"(wl));  // see StreamPlace::first
    int left = n;
    const uint64_t pol = streamPolicy<BEYOND && FIRST>();
    const int* cp = m.col + (size_t)s0 * 32 + wl;
    const char* vp = (const char*)m.val + (size_t)s0 * (288 * sizeof(T));
    int c[R];
#pragma unroll
    for (int j = 0; j < R; ++j) c[j] = j < left ? streamLoad(cp + 32 * j, pol) : -1;
#pragma unroll 1
    for (; left > 0; left -= R) {
        SellBlock<T> b[R];
        double x[R][3];
        int nx[R];
#pragma unroll
        for (int j = 0; j < R; ++j)
            if (c[j] >= 0) { b[j].load(vp + j * 288 * sizeof(T), wl, pol); gather3(u, c[j], x[j]); }
        cp += 32 * R;
        vp += R * 288 * sizeof(T);
#pragma unroll
        for (int j = 0; j < R; ++j) nx[j] = R + j < left ? streamLoad(cp + 32 * j, pol) : -1;
#pragma unroll
        for (int j = 0; j < R; ++j) {
            if (c[j] >= 0) b[j].mulAdd(x[j], acc);
            c[j] = nx[j];
        }
    }
}

// Where a thread of the streaming kernel works: its warp's first tile and the
// block's last, the component it updates, its row in a tile, and the
// recurrence vectors, tile by tile: the 24 entries of x, then r, u, w, z, q,
// s, p (in shared or global memory).
enum StreamVec { SV_X, SV_R, SV_U, SV_W, SV_Z, SV_Q, SV_S, SV_P };
struct StreamPlace {
    int tFirst, tHi;
    double* st;
    // the compiler sees a new value in every pass: the passes' addresses, formed
    // once before the iterations, would spill 60-100 registers
    __device__ __forceinline__ int first() const {
        int t = tFirst;
        asm volatile("" : "+r"(t));
        return t;
    }
    __device__ __forceinline__ int q() const { return threadIdx.x & (GROUP - 1); }
    __device__ __forceinline__ int row(int tile) const { return 8 * tile + (threadIdx.x & 31) / GROUP; }
    // this thread's entry of vector 0 (lanes q < 3); vector k lies 24 k further
    __device__ __forceinline__ double* own(int tile) const { return st + (ptrdiff_t)192 * tile + 3 * ((threadIdx.x & 31) / GROUP) + q(); }
};

__device__ __forceinline__ double pick3(const double v[3], int q) { return q == 0 ? v[0] : (q == 1 ? v[1] : v[2]); }
__device__ __forceinline__ double rowDot3(const double* D, int q, const double v[3]) {
    return D[3 * q] * v[0] + D[3 * q + 1] * v[1] + D[3 * q + 2] * v[2];
}

// The group's sum of (M u)_row over the static blocks and the contact blocks
// (all, or with TRI < 0 / > 0 those left / right of the diagonal), in every lane
template <class T, int TRI, bool BEYOND, class MT>
__device__ __forceinline__ void streamRow(const PcgArgs<MT, double>& a, const SellView& m, const SellCursor<BEYOND>& cur, const float* factor, const MT* matrix,
                                          int row, const double* u, double acc[3]) {
    acc[0] = acc[1] = acc[2] = 0.0;
    sellRow<T, BEYOND, TRI == 0>(m, cur.s, cur.n, u, acc);
    if (a.dRowS && row < a.nv) {
#pragma unroll 1
        for (int k = a.dRowS[row] + (threadIdx.x & (GROUP - 1)), ke = a.dRowE[row]; k < ke; k += GROUP) {
            const int c = a.dCol[k];
            if ((TRI < 0 && c >= row) || (TRI > 0 && c <= row)) continue;
            double xv[3];
            gather3(u, c, xv);
            if (TRI == 0) blockMulAdd(matrix + (size_t)9 * k, xv, acc);
            else blockMulAdd(factor + (size_t)9 * k, xv, acc);
        }
    }
    groupReduce3(acc);
}

// From component q of v in each lane: block-Jacobi Dinv v, or with a factor
// S v (lower triangular), the input of the factor's first pass.  The fourth
// lane writes the pad, so that whole sectors are written.
template <bool LEARNED, class MT>
__device__ __forceinline__ double streamPrecond(const PcgArgs<MT, double>& a, int row, double vq, double* out) {
    const int q = threadIdx.x & (GROUP - 1);
    const double v[3] = {__shfl_sync(0xffffffffu, vq, 0, GROUP), __shfl_sync(0xffffffffu, vq, 1, GROUP), __shfl_sync(0xffffffffu, vq, 2, GROUP)};
    double o = 0.0;
    if (row < a.nv) {
        if (q < 3) {
            if (!LEARNED) {
                o = rowDot3(a.Dinv + 9 * (size_t)row, q, v);
            } else {
                const double* S = a.S + 9 * (size_t)row + 3 * q;
                const double p1 = S[1] * v[1], p2 = S[2] * v[2];
                o = S[0] * v[0] + (q > 0 ? p1 : 0.0) + (q > 1 ? p2 : 0.0);
            }
        }
        out[4 * (size_t)row + q] = o;
    }
    return o;
}

// out = S^T G^T G (S w), with S w in g2 already; ends without a barrier.  The
// result is also the rows' u where ownU.  False on a barrier timeout.
template <class FT, bool BEYOND, class MT>
__device__ __forceinline__ bool streamFactor(const PcgArgs<MT, double>& a, const StreamPlace& at, double* out, bool ownU, unsigned& ep) {
    const int q = at.q();
    constexpr int W = streamWarps(BEYOND);
    SellCursor<BEYOND> cur;
    cur.start(a.sL, at.first(), at.tHi);
    cur.template prefetch<FT, false>(a.sL, cur.s, cur.n);
    if (!gridBarrier(a.bar, a.flag, gridDim.x, ep)) return false;
    for (int tile = at.first(); tile < at.tHi; tile += W) {
        const int row = at.row(tile);
        double acc[3];
        cur.template prefetch<FT, false>(a.sL, cur.sn, cur.nn);
        streamRow<FT, -1, BEYOND>(a, a.sL, cur, a.gD, (const MT*)nullptr, row, a.g2, acc);
        cur.next(a.sL, tile, at.tHi);
        if (row < a.nv) a.g3[4 * (size_t)row + q] = q < 3 ? pick3(acc, q) : 0.0;
    }
    cur.start(a.sU, at.first(), at.tHi);
    cur.template prefetch<FT, false>(a.sU, cur.s, cur.n);
    if (!gridBarrier(a.bar, a.flag, gridDim.x, ep)) return false;
    for (int tile = at.first(); tile < at.tHi; tile += W) {
        const int row = at.row(tile);
        double acc[3];
        cur.template prefetch<FT, false>(a.sU, cur.sn, cur.nn);
        streamRow<FT, 1, BEYOND>(a, a.sU, cur, a.gD, (const MT*)nullptr, row, a.g3, acc);
        cur.next(a.sU, tile, at.tHi);
        if (row < a.nv) {
            double o = 0.0;
            if (q < 3) {
                // component q of S^T y
                const double* S = a.S + 9 * (size_t)row + 4 * q;
                o = S[0] * pick3(acc, q);
                if (q < 2) o += S[3] * (q == 0 ? acc[1] : acc[2]);
                if (q < 1) o += S[6] * acc[2];
                if (ownU) at.own(tile)[24 * SV_U] = o;
            }
            out[4 * (size_t)row + q] = o;
        }
    }
    return true;
}

template <class MT, class FT, bool LEARNED, bool BEYOND>
__global__ void __launch_bounds__(32 * streamWarps(BEYOND), 1) pcgStreamKernel(PcgArgs<MT, double> a) {
    constexpr int W = streamWarps(BEYOND);
    extern __shared__ __align__(16) unsigned char pipeSmem[];
    __shared__ double sc[3];  // the last gamma and alpha, and the stopping threshold
    const unsigned nb = gridDim.x;
    unsigned ep = 0;
    const int nTiles = (a.nv + 7) / 8;
    StreamPlace at;
    const int tLo = (int)((long long)nTiles * blockIdx.x / nb);
    at.tHi = (int)((long long)nTiles * (blockIdx.x + 1) / nb);
    at.tFirst = tLo + (threadIdx.x >> 5);
    at.st = a.resident ? reinterpret_cast<double*>(pipeSmem) - 192 * (ptrdiff_t)tLo : a.state;
    const int q = at.q();
    auto part = [&](int set, int k) { return a.pp + (size_t)(3 * set + k) * PIPE_PMAX; };
    // x = 0, r = b, u = M r (gathered from g1); the recurrence vectors start at 0
    double s0 = 0, s1 = 0, s2 = 0;  // this thread's shares of r.r, gamma = (r,u), delta = (w,u)
    for (int tile = at.first(); tile < at.tHi; tile += W) {
        const int row = at.row(tile);
        double rq = 0.0;
        if (row < a.nv && q < 3) {
            double* v = at.own(tile);
            v[24 * SV_X] = v[24 * SV_Z] = v[24 * SV_Q] = v[24 * SV_S] = v[24 * SV_P] = 0.0;
            rq = a.b[3 * (size_t)row + q];
            v[24 * SV_R] = rq;
            s0 += rq * rq;
        }
        const double u = streamPrecond<LEARNED>(a, row, rq, LEARNED ? a.g2 : a.g1);
        if (!LEARNED && row < a.nv && q < 3) at.own(tile)[24 * SV_U] = u;
    }
    if (LEARNED && !streamFactor<FT, BEYOND>(a, at, a.g1, true, ep)) return;
    if (!gridBarrier(a.bar, a.flag, nb, ep)) return;
    // w = A u, m = M w
    SellCursor<BEYOND> cur;
    cur.start(a.sA, at.first(), at.tHi);
    for (int tile = at.first(); tile < at.tHi; tile += W) {
        const int row = at.row(tile);
        double acc[3];
        streamRow<MT, 0, BEYOND>(a, a.sA, cur, (const float*)nullptr, a.dVal, row, a.g1, acc);
        cur.next(a.sA, tile, at.tHi);
        double wq = 0.0;
        if (row < a.nv && q < 3) {
            double uo[3];
            gather3(a.g1, row, uo);
            wq = pick3(acc, q) + rowDot3(a.diagExtra + 9 * (size_t)row, q, uo);
            double* v = at.own(tile);
            v[24 * SV_W] = wq;
            const double uq = v[24 * SV_U];
            s1 += v[24 * SV_R] * uq;
            s2 += wq * uq;
        }
        streamPrecond<LEARNED>(a, row, wq, LEARNED ? a.g2 : a.g0);
    }
    blockReduce3(s0, s1, s2);
    if (threadIdx.x == 0) { part(0, 0)[blockIdx.x] = s0; part(0, 1)[blockIdx.x] = s1; part(0, 2)[blockIdx.x] = s2; }
    if (LEARNED && !streamFactor<FT, BEYOND>(a, at, a.g0, false, ep)) return;
    double sums[3];  // r.r, gamma, delta
    cur.start(a.sA, at.first(), at.tHi);
    if (!gridBarrierSum<3>(a.bar, a.flag, nb, ep, part(0, 0), PIPE_PMAX, sums)) return;
    if (threadIdx.x == 0) {
        sc[0] = sc[1] = 1.0;
        sc[2] = fmax(a.tol * a.tol * sums[0], 2.2250738585072014e-308);
        if (blockIdx.x == 0) a.scal[6] = sums[0];
    }
    __syncthreads();
    int iter = 0;
    int status = (sums[0] == 0.0 || sums[0] < sc[2]) ? 1 : 0;
    while (status == 0) {
        const double g = sums[1];
        const double bt = iter == 0 ? 0.0 : g / sc[0];
        const double den = iter == 0 ? sums[2] : sums[2] - bt * g / sc[1];
        if (!(den != 0.0) || !isfinite(den)) { status = 2; break; }  // breakdown: the caller's true residual decides
        const double al = g / den;
        const double* mCur = (LEARNED || (iter & 1) == 0) ? a.g0 : a.g1;
        s0 = s1 = s2 = 0.0;
        for (int tile = at.first(); tile < at.tHi; tile += W) {
            const int row = at.row(tile);
            double acc[3];
            cur.template prefetch<MT, true>(a.sA, cur.sn, cur.nn);
            if (BEYOND && (threadIdx.x & 31) == 0 && tile + W < at.tHi && 8 * (tile + W) + 8 <= a.nv) {
                const size_t o = 72 * (size_t)(tile + W);
                const uint64_t pol = streamPolicy<false>();
                prefetchL2(a.diagExtra + o, 576, pol);
                prefetchL2((LEARNED ? a.S : a.Dinv) + o, 576, pol);
            }
            streamRow<MT, 0, BEYOND>(a, a.sA, cur, (const float*)nullptr, a.dVal, row, mCur, acc);
            cur.next(a.sA, tile, at.tHi);
            double wq = 0.0;
            if (row < a.nv && q < 3) {
                double mo[3];
                gather3(mCur, row, mo);
                double* v = at.own(tile);
                const double zv = pick3(acc, q) + rowDot3(a.diagExtra + 9 * (size_t)row, q, mo) + bt * v[24 * SV_Z];
                v[24 * SV_Z] = zv;
                const double w0 = v[24 * SV_W];
                wq = w0 - al * zv;
                v[24 * SV_W] = wq;
                const double sq = w0 + bt * v[24 * SV_S];
                v[24 * SV_S] = sq;
                const double u0 = v[24 * SV_U];
                const double pv = u0 + bt * v[24 * SV_P];
                v[24 * SV_P] = pv;
                v[24 * SV_X] += al * pv;
                const double qv = pick3(mo, q) + bt * v[24 * SV_Q];
                v[24 * SV_Q] = qv;
                const double uv = u0 - al * qv;
                v[24 * SV_U] = uv;
                const double rv = v[24 * SV_R] - al * sq;
                v[24 * SV_R] = rv;
                s0 += rv * rv;
                s1 += rv * uv;
                s2 += wq * uv;
            }
            streamPrecond<LEARNED>(a, row, wq, LEARNED ? a.g2 : ((iter & 1) == 0 ? a.g1 : a.g0));
        }
        const int set = (iter + 1) & 1;
        blockReduce3(s0, s1, s2);
        if (threadIdx.x == 0) {
            part(set, 0)[blockIdx.x] = s0; part(set, 1)[blockIdx.x] = s1; part(set, 2)[blockIdx.x] = s2;
            sc[0] = g;
            sc[1] = al;
        }
        // the factor's m is replaced only in its last pass, two barriers
        // after every row read it
        if (LEARNED && !streamFactor<FT, BEYOND>(a, at, a.g0, false, ep)) return;
        cur.start(a.sA, at.first(), at.tHi);
        cur.template prefetch<MT, true>(a.sA, cur.s, cur.n);
        if (!gridBarrierSum<3>(a.bar, a.flag, nb, ep, part(set, 0), PIPE_PMAX, sums)) return;
        ++iter;
        if (sums[0] < sc[2]) { status = 1; break; }
        if (iter >= a.maxIter || !isfinite(sums[0])) { status = 2; break; }
    }
    // the solution leaves the state
    for (int tile = at.first(); tile < at.tHi; tile += W) {
        const int row = at.row(tile);
        if (row < a.nv && q < 3) a.x[3 * (size_t)row + q] = at.own(tile)[24 * SV_X];
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        a.scal[3] = sums[0];
        a.scal[4] = iter;
        atomicCAS(a.flag, 0, status);  // a barrier timeout (3) stands
    }
}

// The same recurrences with block-Jacobi over block-CSR rows in memory, for
// patterns whose rows differ so much that tiles would be mostly padding
// (SELL_PAD).  A row of some hundred blocks is a chain of loads, so this build
// keeps three blocks of 512 threads on an SM (40 registers) and deals the rows of
// the whole system out in turn.  Measured per iteration on a B200, FP64, here and in
// tiles: 40,011 rows, every 8th joined to 200 others, 50 and 100 us, every 32nd to
// 400, 44 and 141; 200,011 rows, every 8th joined to 80, 101 and 238.  Bound by the
// longest row's chain and by nine scattered loads a block.
template <class MT>
__global__ void __launch_bounds__(PB, 3) pcgRowsKernel(PcgArgs<MT, double> a) {
    const unsigned nb = gridDim.x;
    unsigned ep = 0;
    const int nv = a.nv;
    const RowIter it;
    const int q = it.lane;  // the component this lane updates (q < 3)
    auto part = [&](int set, int k) { return a.pp + (size_t)(3 * set + k) * PIPE_PMAX; };
    auto pick = [&](const double v[3]) { return q == 0 ? v[0] : (q == 1 ? v[1] : v[2]); };
    auto rowDot = [&](const double* D, const double v[3]) { return D[3 * q] * v[0] + D[3 * q + 1] * v[1] + D[3 * q + 2] * v[2]; };
    // m = Dinv v for the row, v held by lanes 0, 1, 2 of its group; every lane calls
    auto precondRow = [&](int row, double vq, double* out) {
        const double v[3] = {__shfl_sync(0xffffffffu, vq, 0, GROUP), __shfl_sync(0xffffffffu, vq, 1, GROUP), __shfl_sync(0xffffffffu, vq, 2, GROUP)};
        double o = 0.0;
        if (row < nv && q < 3) out[3 * (size_t)row + q] = o = rowDot(a.Dinv + 9 * (size_t)row, v);
        return o;
    };
    // x = 0, r = b, u = M r; the recurrence vectors start at 0
    double rr = 0, g = 0, dl = 0;
    for (int base = it.first; base < nv; base += it.stride) {
        const int row = base + it.grp;
        const size_t i = 3 * (size_t)row + q;
        double rq = 0.0;
        if (row < nv && q < 3) {
            a.x[i] = a.z[i] = a.q[i] = a.s[i] = a.p[i] = 0.0;
            a.r[i] = rq = a.b[i];
            rr += rq * rq;
        }
        precondRow(row, rq, a.u);
    }
    if (!gridBarrier(a.bar, a.flag, nb, ep)) return;
    // w = A u, m = M w, gamma = (r,u), delta = (w,u).  The recurrences overwrite
    // u row by row while its neighbours still read m alone.
    for (int base = it.first; base < nv; base += it.stride) {
        const int row = base + it.grp;
        const size_t i = 3 * (size_t)row + q;
        double acc[3] = {0.0, 0.0, 0.0};
        if (row < nv) rowSpmv(a, row, q, (const double*)a.u, acc);
        groupReduce3(acc);
        double wq = 0.0;
        if (row < nv && q < 3) {
            const double uo[3] = {a.u[3 * (size_t)row], a.u[3 * (size_t)row + 1], a.u[3 * (size_t)row + 2]};
            a.w[i] = wq = pick(acc) + rowDot(a.diagExtra + 9 * (size_t)row, uo);
            g += a.r[i] * pick(uo);
            dl += wq * pick(uo);
        }
        precondRow(row, wq, a.mA);
    }
    blockReduce3(rr, g, dl);
    if (threadIdx.x == 0) { part(0, 0)[blockIdx.x] = rr; part(0, 1)[blockIdx.x] = g; part(0, 2)[blockIdx.x] = dl; }
    double sums[3];  // r.r, gamma, delta
    if (!gridBarrierSum<3>(a.bar, a.flag, nb, ep, part(0, 0), PIPE_PMAX, sums)) return;
    const double rhs2 = sums[0];
    const double thr = fmax(a.tol * a.tol * rhs2, 2.2250738585072014e-308);
    int iter = 0;
    int status = (rhs2 == 0.0 || rhs2 < thr) ? 1 : 0;
    double gPrev = 1.0, alPrev = 1.0;
    while (status == 0) {
        g = sums[1];
        const double bt = iter == 0 ? 0.0 : g / gPrev;
        const double den = iter == 0 ? sums[2] : sums[2] - bt * g / alPrev;
        if (!(den != 0.0) || !isfinite(den)) { status = 2; break; }  // breakdown: the caller's true residual decides
        const double al = g / den;
        const double* mCur = (iter & 1) == 0 ? a.mA : a.mB;
        double* mNext = (iter & 1) == 0 ? a.mB : a.mA;
        double lrr = 0, lg = 0, ld = 0;
        for (int base = it.first; base < nv; base += it.stride) {
            const int row = base + it.grp;
            const size_t i = 3 * (size_t)row + q;
            double acc[3] = {0.0, 0.0, 0.0};
            if (row < nv) rowSpmv(a, row, q, mCur, acc);
            groupReduce3(acc);
            double wq = 0.0;
            if (row < nv && q < 3) {
                const double mo[3] = {mCur[3 * (size_t)row], mCur[3 * (size_t)row + 1], mCur[3 * (size_t)row + 2]};
                const double zv = pick(acc) + rowDot(a.diagExtra + 9 * (size_t)row, mo) + bt * a.z[i];
                const double qv = pick(mo) + bt * a.q[i];
                const double w0 = a.w[i], u0 = a.u[i];
                const double sq = w0 + bt * a.s[i];
                const double pv = u0 + bt * a.p[i];
                a.z[i] = zv; a.q[i] = qv; a.s[i] = sq; a.p[i] = pv;
                a.x[i] += al * pv;
                const double rv = a.r[i] - al * sq;
                const double uv = u0 - al * qv;
                wq = w0 - al * zv;
                a.r[i] = rv; a.u[i] = uv; a.w[i] = wq;
                lrr += rv * rv;
                lg += rv * uv;
                ld += wq * uv;
            }
            precondRow(row, wq, mNext);
        }
        const int set = (iter + 1) & 1;
        blockReduce3(lrr, lg, ld);
        if (threadIdx.x == 0) { part(set, 0)[blockIdx.x] = lrr; part(set, 1)[blockIdx.x] = lg; part(set, 2)[blockIdx.x] = ld; }
        if (!gridBarrierSum<3>(a.bar, a.flag, nb, ep, part(set, 0), PIPE_PMAX, sums)) return;
        gPrev = g;
        alPrev = al;
        ++iter;
        if (sums[0] < thr) { status = 1; break; }
        if (iter >= a.maxIter || !isfinite(sums[0])) { status = 2; break; }
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        a.scal[3] = sums[0];
        a.scal[4] = iter;
        a.scal[6] = rhs2;
        atomicCAS(a.flag, 0, status);  // a barrier timeout (3) stands
    }
}

__global__ void accumulateKernelD(int n3, const double* d, double* x) {
    CIPC_KERNEL_LOOP(i, n3) x[i] += d[i];
}

__global__ void zeroKernel(int n3, double* x) {
    CIPC_KERNEL_LOOP(i, n3) x[i] = 0.0;
}

}  // namespace

// One warp per tile copies the tile's blocks into the layout of SellView:
// lane l of step j holds block 4 j + l % 4 of the tile's row l / 4.  slotOf
// lists the rows' source slots (null: the block-CSR slots themselves; ~slot:
// the block is transposed).  Columns are written when col is given.
template <class MT, class OT>
__global__ void packTilesKernel(int nv, const int* ptr, const int* slotOf, const int* srcCol, const MT* src, const int* tile, int* col, OT* out) {
    const int nTiles = (nv + 7) / 8, wl = threadIdx.x & 31;
    const int nWarps = gridDim.x * blockDim.x / 32;
    for (int t = (blockIdx.x * blockDim.x + threadIdx.x) / 32; t < nTiles; t += nWarps) {
        const int row = 8 * t + wl / GROUP;
        int k = 0, ke = 0;
        if (row < nv) { k = ptr[row] + (wl & (GROUP - 1)); ke = ptr[row + 1]; }
        for (int st = tile[t], se = tile[t + 1]; st < se; ++st, k += GROUP) {
            int c = -1;
            if (k < ke) {
                int s = slotOf ? slotOf[k] : k;
                const bool tr = s < 0;
                if (tr) s = ~s;
                if (col) c = srcCol[s];
                const MT* B = src + (size_t)9 * s;
                OT* o = out + (size_t)st * 288;
                // 16-byte runs of each lane, then the ninth values
                constexpr int RUN = 16 / sizeof(OT);
#pragma unroll
                for (int e = 0; e < 8; ++e) o[(e / RUN) * 32 * RUN + wl * RUN + e % RUN] = (OT)B[tr ? 3 * (e % 3) + e / 3 : e];
                o[256 + wl] = (OT)B[8];
            }
            if (col) col[(size_t)st * 32 + wl] = c;
        }
    }
}

// Steps of tile t of 8 rows with the given row offsets.
static int tileSteps(int nv, const std::vector<int>& ptr, int t) {
    int most = 0;
    for (int r = 8 * t; r < std::min(nv, 8 * t + 8); ++r) most = std::max(most, ptr[r + 1] - ptr[r]);
    return (most + GROUP - 1) / GROUP;
}

// Step offsets of the tiles.
static void tileOffsets(Ctx& c, SellRows& m, int nv, const std::vector<int>& ptr) {
    std::vector<int> tile((nv + 7) / 8 + 1, 0);
    for (int t = 0; 8 * t < nv; ++t) tile[t + 1] = tile[t] + tileSteps(nv, ptr, t);
    m.steps = tile.back();
    upload(c, m.tile, tile);
    m.laid = true;
}

// What a block-Jacobi iteration over the tiles reads: matrix, gathered vectors
// and diagonal blocks.
static double tileBytes(const Ctx& c, size_t valueSize) { return (double)c.sellA.steps * (288 * valueSize + 128) + c.nv * (2 * 72.0 + 2 * 32.0); }

// Whether the static pattern goes into tiles (SELL_PAD).
static bool rowsSuitTiles(Ctx& c) {
    SellRows& m = c.sellA;
    const int tiles = (c.nv + 7) / 8;
    if (!m.steps)
        for (int t = 0; t < tiles; ++t) {
            const int n = tileSteps(c.nv, c.hRowPtr, t);
            m.steps += n;
            m.longest = std::max(m.longest, n);
        }
    if (32.0 * (m.steps - tiles) <= SELL_PAD * c.nnzb) return true;
    int dev = 0, l2 = 0;
    CIPC_CUDA(cudaGetDevice(&dev));
    CIPC_CUDA(cudaDeviceGetAttribute(&l2, cudaDevAttrL2CacheSize, dev));
    return m.longest <= SELL_LONG && tileBytes(c, c.mixed ? sizeof(float) : sizeof(double)) <= l2;
}

template <class MT, class OT>
static void packTiles(Ctx& c, SellRows& m, const int* ptr, const int* slotOf, const MT* src) {
    const bool first = !m.hasCols;
    m.col.reserve(std::max<size_t>((size_t)32 * m.steps, 1), true);
    m.val.reserve(std::max<size_t>((size_t)288 * sizeof(OT) * m.steps, 16), true);
    const int nb = std::max(1, std::min(((c.nv + 7) / 8 + VB / 32 - 1) / (VB / 32), 148 * 8));
    launch(packTilesKernel<MT, OT>, nb, VB, 0, c.s, c.nv, ptr, slotOf, (const int*)c.colIdx, src, (const int*)m.tile, first ? m.col.p : (int*)nullptr,
           reinterpret_cast<OT*>(m.val.p));
    CIPC_CUDA(cudaGetLastError());
    m.hasCols = true;
}

// The static matrix and, with a factor, its static blocks in tiles: per row
// the slots with column <= row (G), then those with column >= row (G^T: the
// mirror slots, and the diagonal transposed).  Offsets and columns follow the
// static pattern and are laid out on the first call; values on every call.
template <class MT, class FT>
static void packStream(Ctx& c, const MT* val, bool learned) {
    const int nv = c.nv;
    if (!c.sellA.laid) tileOffsets(c, c.sellA, nv, c.hRowPtr);
    packTiles<MT, MT>(c, c.sellA, c.rowPtr, nullptr, val);
    if (!learned) return;
    if (!c.sellL.laid) {
        std::vector<int> col(c.nnzb);
        CIPC_CUDA(cudaMemcpy(col.data(), c.colIdx.p, sizeof(int) * c.nnzb, cudaMemcpyDeviceToHost));
        std::vector<int> lp(nv + 1, 0), ls, up(nv + 1, 0), us;
        ls.reserve(c.nnzb / 2 + nv); us.reserve(c.nnzb / 2 + nv);
        for (int r = 0; r < nv; ++r) {
            for (int k = c.hRowPtr[r]; k < c.hRowPtr[r + 1]; ++k) {
                if (col[k] <= r) ls.push_back(k);
                if (col[k] >= r) us.push_back(col[k] == r ? ~k : k);
            }
            lp[r + 1] = (int)ls.size();
            up[r + 1] = (int)us.size();
        }
        upload(c, c.sellL.ptr, lp); upload(c, c.sellL.slot, ls); upload(c, c.sellU.ptr, up); upload(c, c.sellU.slot, us);
        tileOffsets(c, c.sellU, nv, up);
        tileOffsets(c, c.sellL, nv, lp);
    }
    packTiles<float, FT>(c, c.sellL, c.sellL.ptr, c.sellL.slot, (const float*)c.mpGS);
    packTiles<float, FT>(c, c.sellU, c.sellU.ptr, c.sellU.slot, (const float*)c.mpGS);
}

void buildRhs(Ctx& c) {
    c.rhs.reserve(3 * c.nv);
    launch(rhsKernel, vecBlocks(c.nv), VB, 0, c.s, c.nv, c.grad, c.btype, c.rhs);
    CIPC_CUDA(cudaGetLastError());
}

// y = A x
template <class MT>
static void spmv(Ctx& c, const MT* val, const MT* dval, const double* x, double* y) {
    const bool dyn = c.nDynB > 0;
    launch(spmvKernel<MT, double>, std::max(1, std::min((c.nv * GROUP + VB - 1) / VB, MAXPART)), VB, 0, c.s, c.nv, c.rowPtr, c.colIdx, val,
           dyn ? c.dynRowStart.p : nullptr, dyn ? c.dynRowEnd.p : nullptr, dyn ? c.dynCol.p : nullptr, dval, c.diagExtra, x, y);
}

static void computeDinv(Ctx& c) {
    int nv = c.nv;
    bool dyn = c.nDynB > 0;
    c.Dinv.reserve(9 * (size_t)nv);
    if (c.mixed)
        launch(dinvKernel<float>, vecBlocks(nv), VB, 0, c.s, nv, c.diagSlot, c.valF, dyn ? c.dynRowStart.p : nullptr, dyn ? c.dynRowEnd.p : nullptr,
               dyn ? c.dynCol.p : nullptr, c.dynBF, c.diagExtra, c.Dinv);
    else
        launch(dinvKernel<double>, vecBlocks(nv), VB, 0, c.s, nv, c.diagSlot, c.valD, dyn ? c.dynRowStart.p : nullptr, dyn ? c.dynRowEnd.p : nullptr,
               dyn ? c.dynCol.p : nullptr, c.dynBD, c.diagExtra, c.Dinv);
}

constexpr int PMAX = 1024;  // max blocks of the persistent PCG

// Blocks per SM of the textbook kernel: CIPC_PCG_BLOCKS_PER_SM (1-8) or 2.
static int pcgBlocksPerSm() {
    static int v = -1;
    if (v < 0) {
        const char* e = std::getenv("CIPC_PCG_BLOCKS_PER_SM");
        int k = e ? std::atoi(e) : 2;
        v = std::min(8, std::max(1, k));
    }
    return v;
}

// CIPC_PCG_CLASSIC=1 selects the textbook recurrences (two barriers per
// iteration with block-Jacobi); the default is the pipelined kernel.
static bool pcgClassic() {
    static int v = -1;
    if (v < 0) { const char* e = std::getenv("CIPC_PCG_CLASSIC"); v = (e && *e == '1') ? 1 : 0; }
    return v == 1;
}

// CIPC_PCG_NOPACK=1 keeps the streaming kernel's factor in FP32.
static bool pcgNoPack() {
    static int v = -1;
    if (v < 0) { const char* e = std::getenv("CIPC_PCG_NOPACK"); v = (e && *e == '1') ? 1 : 0; }
    return v == 1;
}

// CIPC_PCG_NOCACHE=1 keeps the pipelined kernel's matrix rows in global memory.
static bool pcgNoCache() {
    static int v = -1;
    if (v < 0) { const char* e = std::getenv("CIPC_PCG_NOCACHE"); v = (e && *e == '1') ? 1 : 0; }
    return v == 1;
}

// CIPC_DEBUG_PCG=1 prints every inner solve and fallback to stderr.
static bool debugPcg() {
    static int v = -1;
    if (v < 0) { const char* e = std::getenv("CIPC_DEBUG_PCG"); v = (e && *e == '1') ? 1 : 0; }
    return v == 1;
}

// largest static-slot count of `rows` consecutive rows starting at a multiple of rows
static int pcgSliceMax(Ctx& c, int rows) {
    if (c.pcgSliceMax < 0 || c.pcgSliceRows != rows) {
        int m = 0;
        for (int r0 = 0; r0 < c.nv; r0 += rows) {
            int r1 = std::min(c.nv, r0 + rows);
            m = std::max(m, c.hRowPtr[r1] - c.hRowPtr[r0]);
        }
        c.pcgSliceMax = m;
        c.pcgSliceRows = rows;
    }
    return c.pcgSliceMax;
}

// Lets a kernel ask for as much dynamic shared memory as a block can have.  The
// limit belongs to the process, not to the launch: a limit of one system's size
// would be lowered by another thread's smaller system between here and the launch.
static void allowSharedMemory(const void* fn) {
    int dev = 0, optin = 0;
    CIPC_CUDA(cudaGetDevice(&dev));
    CIPC_CUDA(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
    cudaFuncAttributes fa;
    CIPC_CUDA(cudaFuncGetAttributes(&fa, fn));
    CIPC_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, optin - (int)fa.sharedSizeBytes));
}

// The six vectors that the pipelined kernels over block-CSR rows keep beside the
// caller's.
template <class MT, class VT>
static void pipeVectors(Ctx& c, PcgArgs<MT, VT>& a) {
    const size_t n3 = 3 * (size_t)c.nv;
    c.pcgPipe.reserve(6 * n3 * sizeof(VT) / sizeof(double) + 6);
    VT* pv = reinterpret_cast<VT*>(c.pcgPipe.p);
    a.u = pv; a.w = pv + n3; a.mA = pv + 2 * n3; a.mB = pv + 3 * n3; a.q = pv + 4 * n3; a.s = pv + 5 * n3;
}

template <class MT, class VT, bool LEARNED>
static void launchPersistent(Ctx& c, PcgArgs<MT, VT>& a, int smCount, bool classic) {
    int needed = std::max(1, (c.nv * GROUP + PB - 1) / PB);
    int cap = std::min(PMAX, PIPE_PMAX);
    void* args[] = {&a};
    a.dynCap = 0;
    a.cacheG = 0;
    if (!classic && !pcgNoCache() && !c.hRowPtr.empty() && needed <= cap) {
        // single-pass launch: each block owns its rows for the whole solve and
        // stages them in shared memory.  The largest configuration that keeps
        // every block resident is taken: the factor's blocks cached or not, a
        // contact window of 512 down to 0 slots.  Rows are spread evenly over one
        // block per SM or more, in a small system SINGLE_MIN_ROWS.  Where so many wide
        // rows do not fit, the streaming kernel takes a block-Jacobi solve as fast (443
        // rows of 161 blocks on a B200: 0.59 ms with 8 rows a block, 0.58 streamed;
        // FP32 0.74 and 0.51); a factor, which it would round to FP16, stays here
        // with fewer rows a block, down to the even spread.
        const int even = (c.nv + std::max(needed, smCount) - 1) / std::max(needed, smCount);
        const void* fn = (const void*)pcgPipelinedKernel<MT, VT, LEARNED>;
        int maxOptin = 0, dev = 0;
        CIPC_CUDA(cudaGetDevice(&dev));
        CIPC_CUDA(cudaDeviceGetAttribute(&maxOptin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
        allowSharedMemory(fn);
        const bool dyn = a.dRowS != nullptr;
        static const int dynCaps[] = {512, 256, 128, 0};
        for (int cg = LEARNED ? 1 : 0; cg >= 0; --cg) {
            for (int rows = even <= SINGLE_FILL_ROWS ? SINGLE_MIN_ROWS : even, last = 0; !last; rows = std::max(even, rows / 2)) {
                last = !LEARNED || rows == even;
                const int threads = std::min(PB, std::max(256, (rows * GROUP + 31) / 32 * 32));  // half a block at least, to stage wide rows
                const int nbRows = (c.nv + rows - 1) / rows;
                a.rowsPerBlock = rows;
                a.sliceMax = pcgSliceMax(c, rows);
                for (int dc : dynCaps) {
                    if (!dyn && dc > 0) continue;
                    size_t smem = smemLayout(a.sliceMax, dc, cg != 0, (int)sizeof(MT), (int)sizeof(VT)).total;
                    if (smem + 4096 > (size_t)maxOptin) continue;
                    int perSM = 0;
                    CIPC_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&perSM, fn, threads, smem));
                    if (perSM >= 1 && nbRows <= perSM * smCount && nbRows <= cap) {
                        a.dynCap = dc;
                        a.cacheG = cg;
                        pipeVectors(c, a);
                        if (debugPcg())
                            std::fprintf(stderr, "[pcg] single-pass launch: %d blocks of %d rows, slice %d, contact window %d, factor cached %d, %zu B shared\n",
                                         nbRows, rows, a.sliceMax, dc, cg, smem);
                        ++g_kernelLaunches;
                        CIPC_CUDA(cudaLaunchCooperativeKernel(fn, dim3(nbRows), dim3(threads), args, smem, c.s));
                        return;
                    }
                }
            }
        }
    }
    a.sliceMax = 0;
    a.rowsPerBlock = 0;
    if (classic || sizeof(VT) != sizeof(double)) {
        const void* fn = (const void*)pcgPersistentKernel<MT, VT, LEARNED>;
        int perSM = 0;
        CIPC_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&perSM, fn, PB, 0));
        if (perSM < 1) throw std::runtime_error("persistent PCG kernel does not fit on an SM");
        const int grid = std::max(1, std::min(std::min(std::min(perSM, pcgBlocksPerSm()) * smCount, needed), cap));
        ++g_kernelLaunches;
        CIPC_CUDA(cudaLaunchCooperativeKernel(fn, dim3(grid), dim3(PB), args, 0, c.s));
        return;
    }
    if constexpr (sizeof(VT) == sizeof(double) && !LEARNED) {
        // (a factor belongs to a mesh, whose rows are alike)
        if (!rowsSuitTiles(c)) {
            const void* fn = (const void*)pcgRowsKernel<MT>;
            int perSM = 0;
            CIPC_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&perSM, fn, PB, 0));
            if (perSM < 1) throw std::runtime_error("streaming PCG kernel does not fit on an SM");
            const int grid = std::max(1, std::min(std::min(std::min(perSM, 3) * smCount, needed), cap));
            pipeVectors(c, a);
            if (debugPcg()) std::fprintf(stderr, "[pcg] block-CSR launch: %d blocks, %d tile steps for %d blocks\n", grid, c.sellA.steps, c.nnzb);
            ++g_kernelLaunches;
            CIPC_CUDA(cudaLaunchCooperativeKernel(fn, dim3(grid), dim3(PB), args, 0, c.s));
            return;
        }
    }
    if constexpr (sizeof(VT) == sizeof(double)) {
        const bool half = LEARNED && !pcgNoPack();
        if (half) packStream<MT, __half>(c, a.val, true);
        else packStream<MT, float>(c, a.val, LEARNED);
        auto view = [](const SellRows& m) { return SellView{m.tile.p, m.col.p, m.val.p}; };
        a.sA = view(c.sellA); a.sL = view(c.sellL); a.sU = view(c.sellU);
        // padded gathered vectors
        const size_t n4 = 4 * (size_t)c.nv;
        c.pcgGather.reserve(4 * n4, true);
        a.g0 = c.pcgGather.p; a.g1 = a.g0 + n4; a.g2 = a.g1 + n4; a.g3 = a.g2 + n4;
        const int tiles = (c.nv + 7) / 8;
        const int grid = std::max(1, std::min(std::min(smCount, tiles), cap));
        const int tilesPerBlock = (tiles + grid - 1) / grid;  // at most
        // the state vectors in shared memory where all eight fit
        const size_t state = (size_t)tilesPerBlock * 24 * sizeof(double) * 8;
        a.resident = state <= STREAM_STATE_BYTES ? 1 : 0;
        const size_t smem = a.resident ? state : 0;
        if (!a.resident) c.pcgState.reserve(8 * (size_t)tiles * 24, true);
        a.state = c.pcgState.p;
        // what every iteration reads: matrix, factor, gathered vectors, diagonal
        // blocks and the state
        double bytes = tileBytes(c, sizeof(MT)) + (a.resident ? 0.0 : (double)state * grid);
        if (LEARNED) bytes += ((double)c.sellL.steps + c.sellU.steps) * (288.0 * (half ? 2 : 4) + 128) + c.nv * 32.0;
        int dev = 0, l2 = 0;
        CIPC_CUDA(cudaGetDevice(&dev));
        CIPC_CUDA(cudaDeviceGetAttribute(&l2, cudaDevAttrL2CacheSize, dev));
        const bool beyond = bytes > STREAM_L2_SHARE * l2;
        const void* fn = half ? (beyond ? (const void*)pcgStreamKernel<MT, __half, LEARNED, true> : (const void*)pcgStreamKernel<MT, __half, LEARNED, false>)
                              : (beyond ? (const void*)pcgStreamKernel<MT, float, LEARNED, true> : (const void*)pcgStreamKernel<MT, float, LEARNED, false>);
        const int threads = 32 * streamWarps(beyond);
        allowSharedMemory(fn);
        int fit = 0;
        CIPC_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&fit, fn, threads, smem));
        if (fit * smCount < grid) throw std::runtime_error("streaming PCG kernel does not fit on an SM");
        if (debugPcg()) std::fprintf(stderr, "[pcg] streaming launch: %d blocks of %d tiles, state in shared memory %d, beyond L2 %d (%.1f MB)\n", grid, tilesPerBlock, a.resident, (int)beyond, bytes * 1e-6);
        ++g_kernelLaunches;
        CIPC_CUDA(cudaLaunchCooperativeKernel(fn, dim3(grid), dim3(threads), args, smem, c.s));
    }
}

// Whole PCG in one cooperative launch (grid sized to what is co-resident).
// learned: apply the factor in c.mpS / c.mpGS / c.mpGD instead of block-Jacobi.
template <class MT, class VT>
static int runPcgPersistent(Ctx& c, const MT* val, const MT* dval, const VT* b, VT* x, VT* r, VT* z, VT* p, VT* Ap, double tol, int maxIter,
                            int& flagOut, double& relRes, bool learned = false, bool classic = false) {
    static const int smCount = [] {
        int dev = 0, sms = 0;
        CIPC_CUDA(cudaGetDevice(&dev));
        CIPC_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
        return sms;
    }();
    bool dyn = c.nDynB > 0;
    PcgArgs<MT, VT> a;
    a.nv = c.nv; a.rowPtr = c.rowPtr; a.col = c.colIdx; a.val = val;
    a.dRowS = dyn ? c.dynRowStart.p : nullptr; a.dRowE = dyn ? c.dynRowEnd.p : nullptr; a.dCol = dyn ? c.dynCol.p : nullptr; a.dVal = dval;
    a.diagExtra = c.diagExtra; a.Dinv = c.Dinv; a.b = b; a.x = x; a.r = r; a.z = z; a.p = p; a.Ap = Ap;
    a.S = nullptr; a.gS = nullptr; a.gD = nullptr; a.t = nullptr;
    if (learned) {
        c.mpT.reserve(3 * (size_t)c.nv);
        a.S = c.mpS.p; a.gS = c.mpGS.p; a.gD = c.mpGD.p; a.t = reinterpret_cast<VT*>(c.mpT.p);
    }
    a.partA = c.red.p; a.partB = c.red.p + PMAX; a.partC = c.red.p + 2 * PMAX;
    // pipelined kernels: two sets of partial sums
    c.pcgParts.reserve(6 * (size_t)PIPE_PMAX);
    a.pp = c.pcgParts.p;
    a.scal = c.scal.p; a.flag = c.counters.p + 10;
    c.pcgBar.reserve(BAR_WORDS);
    a.bar = c.pcgBar.p;
    a.tol = tol; a.maxIter = maxIter;
    CIPC_CUDA(cudaMemsetAsync(c.counters.p + 10, 0, sizeof(int), c.s));
    CIPC_CUDA(cudaMemsetAsync(c.pcgBar.p, 0, BAR_WORDS * sizeof(unsigned), c.s));
    profBegin(c, PROF_PCG);
    classic = classic || pcgClassic();
    if (learned) launchPersistent<MT, VT, true>(c, a, smCount, classic);
    else launchPersistent<MT, VT, false>(c, a, smCount, classic);
    profEnd(c, PROF_PCG);
    int hflag = 0;
    double hs[8];
    CIPC_CUDA(cudaMemcpyAsync(&hflag, a.flag, sizeof(int), cudaMemcpyDeviceToHost, c.s));
    CIPC_CUDA(cudaMemcpyAsync(hs, c.scal.p, 8 * sizeof(double), cudaMemcpyDeviceToHost, c.s));
    hostSync(c);
    if (hflag == 3) throw std::runtime_error("device status in PCG: grid barrier timed out");
    flagOut = hflag;
    relRes = hs[6] > 0 ? std::sqrt(hs[3] / hs[6]) : 0.0;
    c.lastPcgLaunchIters = (int)hs[4];
    return (int)hs[4];
}

static void reservePcg(Ctx& c) {
    size_t n3 = 3 * (size_t)c.nv;
    c.sol.reserve(n3); c.r.reserve(n3); c.z.reserve(n3); c.p.reserve(n3); c.Ap.reserve(n3);
    c.red.reserve(4 * PMAX + 16);
    c.scal.reserve(16);
    c.counters.reserve(16);
}

// Builds the factor for the current system (network forward, or the exact
// FSAI); false when block-Jacobi is selected.
static bool prepareLearned(Ctx& c) {
    if (c.precond == CIPC_PRECOND_FSAI) {
        mpnnPrepare(c, false);
        fsaiBuild(c);
    } else if (c.precond == CIPC_PRECOND_LEARNED) {
        if (!c.mpReady) mpnnInitWeights(c, 1);
        mpnnPrepare(c);
        mpnnForward(c);
    } else {
        return false;
    }
    return true;
}

// ||rhs - A sol||^2 in FP64 (FP32 blocks promoted in mixed mode)
static double trueResidual2(Ctx& c) {
    int nv = c.nv, n3 = 3 * nv;
    c.rF.reserve(n3);
    double* part = c.red.p + 3 * MAXPART;
    if (c.mixed) spmv<float>(c, c.valF, c.dynBF, c.sol.p, c.Ap.p);
    else spmv<double>(c, c.valD, c.dynBD, c.sol.p, c.Ap.p);
    int nb = vecBlocks(nv);
    launch(residualKernel, nb, VB, 0, c.s, n3, c.rhs.p, c.Ap.p, c.r.p, c.rF.p, part);
    return deviceSum(c, part, nb);
}

// Iteration cap of one solve with a factor preconditioner before block-Jacobi
// takes over (CIPC_FACTOR_CAP, default 1000): a factor that does not reach
// the inner tolerance within it is rejected rather than iterated further.
static int factorCap() {
    static int v = -1;
    if (v < 0) {
        const char* e = std::getenv("CIPC_FACTOR_CAP");
        v = e ? std::max(10, std::atoi(e)) : 1000;
    }
    return v;
}

static int pcgSolve64(Ctx& c) {
    reservePcg(c);
    computeDinv(c);
    bool learned = prepareLearned(c);
    int n3 = 3 * c.nv;
    int flag = 0;
    double rel = 0;
    // the pipelined recurrences are asked for no more than 1e-8 relative
    // (their attainable accuracy); tighter tolerances are reached by the
    // corrections below
    int it = runPcgPersistent<double, double>(c, c.valD, c.dynBD, c.rhs.p, c.sol.p, c.r.p, c.z.p, c.p.p, c.Ap.p,
                                              pcgClassic() ? c.pcgTol : std::max(c.pcgTol, 1e-8),
                                              learned ? std::min(c.pcgMaxIter, factorCap()) : c.pcgMaxIter, flag, rel, learned);
    // the true FP64 residual decides every solve; corrections restart from
    // the current iterate (residual replacement) with the textbook
    // recurrences, block-Jacobi taking over from a rejected factor
    double rhs2 = deviceDot(c, c.rhs, c.rhs, n3);
    double thr = std::max(c.pcgTol * c.pcgTol * rhs2, 2.2250738585072014e-308);
    double tr2 = trueResidual2(c);
    if (debugPcg()) std::fprintf(stderr, "[pcg] fp64 it %d flag %d true rr/b2 %.3e factor %d\n", it, flag, tr2 / rhs2, (int)learned);
    if (learned && (flag != 1 || !(tr2 < thr))) {
        c.mpFallbacks++;
        learned = false;
    }
    c.corrX.reserve(n3); c.corrR.reserve(n3);
    for (int k = 0; k < 8 && !(tr2 < thr) && it < c.pcgMaxIter; ++k) {
        int f2 = 0;
        int it2 = runPcgPersistent<double, double>(c, c.valD, c.dynBD, c.r.p, c.corrX.p, c.corrR.p, c.z.p, c.p.p, c.Ap.p,
                                                   0.5 * std::sqrt(thr / tr2), c.pcgMaxIter - it, f2, rel, learned, true);
        it += it2;
        launch(accumulateKernelD, vecBlocks(c.nv + 1), VB, 0, c.s, n3, (const double*)c.corrX.p, c.sol.p);
        tr2 = trueResidual2(c);
        if (debugPcg()) std::fprintf(stderr, "[pcg] fp64 correction it %d flag %d true rr/b2 %.3e\n", it2, f2, tr2 / rhs2);
    }
    c.lastPcgIters = it;
    c.lastPcgRelRes = rhs2 > 0 ? std::sqrt(tr2 / rhs2) : 0.0;
    c.pcgItersTotal += it;
    if (!(tr2 < thr) && rhs2 > 0) throw std::runtime_error("GPU PCG did not converge within " + std::to_string(c.pcgMaxIter) + " iterations");
    return it;
}

// r = b - A sol in FP64 (FP32 blocks promoted), bF = (float) r; returns |r|^2
static double mixedResidual(Ctx& c, float* bF) {
    int nv = c.nv, n3 = 3 * nv;
    double* part = c.red.p + 3 * MAXPART;
    spmv<float>(c, c.valF, c.dynBF, c.sol.p, c.Ap.p);
    int nb = vecBlocks(nv);
    launch(residualKernel, nb, VB, 0, c.s, n3, c.rhs.p, c.Ap.p, c.r.p, bF, part);
    return deviceSum(c, part, nb);
}

// FP32 inner PCG + FP64 iterative refinement on the true residual, starting
// from the current c.sol.  Returns false when a factor preconditioner was
// rejected (inner solve over its cap, or the true residual not reached).
static bool refineMixed(Ctx& c, bool learned, double thr, double rhs2, int& total, double& rr) {
    int nv = c.nv, n3 = 3 * nv;
    float* bF = c.DinvF.p;  // FP32 copy of the current residual (right-hand side of the correction)
    int vb = vecBlocks(nv + 1);
    const double innerTol = 1e-3;
    double prevRR = 1e308;
    rr = mixedResidual(c, bF);
    // The pipelined kernel's recurrences stagnate with FP32 vectors on these
    // systems (measured), so with it the corrections run FP64 vectors over
    // the FP32 blocks below; the FP32-vector inner loop serves the classic
    // kernel.
    const int outerMax = pcgClassic() ? 40 : 0;
    for (int outer = 0; outer < outerMax && !(rr < thr); ++outer) {
        if (!(rr < 0.25 * prevRR) && outer > 2) break;  // refinement stagnates: finish in FP64 below
        prevRR = rr;
        int budget = c.pcgMaxIter - total;
        if (budget <= 0) break;
        int cap = learned ? std::min(budget, factorCap()) : budget;
        int flag = 0;
        double rel = 0;
        int it = runPcgPersistent<float, float>(c, c.valF, c.dynBF, bF, c.xF.p, c.rF.p, c.zF.p, c.pF.p, c.ApF.p,
                                                std::max(innerTol, 0.5 * std::sqrt(thr / rr)), cap, flag, rel, learned);
        total += it;
        launch(accumulateKernel, vb, VB, 0, c.s, n3, c.xF.p, c.sol.p);
        rr = mixedResidual(c, bF);
        if (debugPcg()) std::fprintf(stderr, "[pcg] mixed outer %d inner it %d flag %d rel %.3e -> rr/b2 %.3e learned %d\n", outer, it, flag, rel, rr / rhs2,
                                     (int)learned);
        if (learned && flag != 1) return false;
    }
    // FP64-vector PCG on the true residual (FP32 blocks promoted), repeated
    // as residual replacement until the true FP64 residual passes; the
    // repeats use the textbook recurrences, free of pipelining drift
    c.corrX.reserve(n3); c.corrR.reserve(n3);
    for (int k = 0; k < 8 && !(rr < thr) && total < c.pcgMaxIter; ++k) {
        int budget = c.pcgMaxIter - total;
        int flag = 0;
        double rel = 0;
        double tol = 0.5 * std::sqrt(thr / rr);
        if (k == 0 && !pcgClassic()) tol = std::max(tol, 1e-8);
        int it = runPcgPersistent<float, double>(c, c.valF, c.dynBF, c.r.p, c.corrX.p, c.corrR.p, c.z.p, c.p.p, c.Ap.p, tol,
                                                 learned ? std::min(budget, factorCap()) : budget, flag, rel, learned, k > 0);
        total += it;
        launch(accumulateKernelD, vb, VB, 0, c.s, n3, c.corrX.p, c.sol.p);
        rr = mixedResidual(c, bF);
        if (debugPcg()) std::fprintf(stderr, "[pcg] mixed FP64-vector run it %d flag %d -> rr/b2 %.3e learned %d\n", it, flag, rr / rhs2, (int)learned);
        if (learned && flag != 1) return false;
    }
    return !learned || rr < thr;
}

static int pcgSolveMixed(Ctx& c, bool learned) {
    int nv = c.nv;
    int n3 = 3 * nv;
    c.rF.reserve(n3); c.zF.reserve(n3); c.pF.reserve(n3); c.ApF.reserve(n3); c.xF.reserve(n3); c.DinvF.reserve(n3);
    launch(zeroKernel, vecBlocks(nv + 1), VB, 0, c.s, n3, c.sol.p);
    double rhs2 = deviceDot(c, c.rhs, c.rhs, n3);
    c.lastPcgIters = 0;
    if (rhs2 == 0.0) { c.lastPcgRelRes = 0; return 0; }
    double thr = std::max(c.pcgTol * c.pcgTol * rhs2, 2.2250738585072014e-308);
    int total = 0;
    double rr = rhs2;
    if (!refineMixed(c, learned, thr, rhs2, total, rr)) {
        // the factor was rejected (cap or true FP64 residual): block-Jacobi
        // continues the refinement from the current iterate
        c.mpFallbacks++;
        if (debugPcg()) std::fprintf(stderr, "[pcg] factor rejected after %d iterations (rr/b2 %.3e): block-Jacobi\n", total, rr / rhs2);
        refineMixed(c, false, thr, rhs2, total, rr);
    }
    if (!(rr < thr)) throw std::runtime_error("GPU PCG did not converge within " + std::to_string(c.pcgMaxIter) + " iterations");
    c.lastPcgIters = total;
    c.lastPcgRelRes = std::sqrt(rr / rhs2);
    c.pcgItersTotal += total;
    return total;
}

static int pcgSolveMixed(Ctx& c) {
    reservePcg(c);
    computeDinv(c);
    bool learned = prepareLearned(c);
    return pcgSolveMixed(c, learned);
}

__global__ void roundBlocksKernel(size_t n, const double* src, float* dst) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) dst[i] = (float)src[i];
}

void roundBlocks(Ctx& c, size_t n, const double* src, float* dst) {
    launch(roundBlocksKernel, (int)std::max<size_t>(1, std::min<size_t>((n + VB - 1) / VB, 148 * 8)), VB, 0, c.s, n, src, dst);
    CIPC_CUDA(cudaGetLastError());
}

void lendPcg(Ctx& c, DevSlab& slab) {
    const size_t nv = c.nv, n3 = 3 * nv;
    for (DBuf<double>* d : {&c.rhs, &c.sol, &c.r, &c.z, &c.p, &c.Ap, &c.corrX, &c.corrR}) slab.lend(*d, n3);
    slab.lend(c.Dinv, 9 * nv);
    slab.lend(c.red, 4 * PMAX + 16);
    slab.lend(c.scal, 16);
    slab.lend(c.counters, 16);
    slab.lend(c.rF, n3);
    if (c.mixed)
        for (DBuf<float>* d : {&c.zF, &c.pF, &c.ApF, &c.xF, &c.DinvF}) slab.lend(*d, n3);
    slab.lend(c.pcgParts, 6 * (size_t)PIPE_PMAX);
    slab.lend(c.pcgBar, BAR_WORDS);
    int dev = 0, sms = 0;
    CIPC_CUDA(cudaGetDevice(&dev));
    CIPC_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    const bool single = nv <= (size_t)sms * ROWS_PER_BLOCK, rows = !single && !rowsSuitTiles(c);
    if (single || rows) {
        slab.lend(c.pcgPipe, 6 * n3 + 6);
    } else {
        // more rows than a single-pass launch of one block per SM can hold
        const size_t tiles = (nv + 7) / 8;
        slab.lend(c.sellA.tile, tiles + 1);
        slab.lend(c.sellA.col, 32 * (size_t)c.sellA.steps);
        slab.lend(c.sellA.val, 288 * (c.mixed ? sizeof(float) : sizeof(double)) * (size_t)c.sellA.steps);
        slab.lend(c.pcgGather, 16 * nv);
    }
}

int pcgSolve(Ctx& c) { return c.mixed ? pcgSolveMixed(c) : pcgSolve64(c); }

}  // namespace cipc

// ---------------------------------------------------------------------------
// Allocation-free stand-alone PCG.
//
// For callers that must not allocate device memory: code running where
// cudaMalloc is forbidden or unwanted, e.g. a host whose device memory is
// owned by its own allocator (a framework's caching allocator, a pre-sized
// arena) or a loop that must not pay allocation latency.  The caller passes
// device pointers for the matrix, right-hand side and solution; every scratch
// vector lives in the file-scope array below.  The array is sized for at
// most CIPC_NOALLOC_MAX_ROWS block rows (NOALLOC_DOUBLES doubles: 8,008,064
// bytes, 7.6 MiB) and every GPU that loads this library keeps it until the
// process exits.  All calls share it and it keeps the last call's contents,
// so calls that overlap on the GPU (two streams, two host threads) race;
// serialise them.
// ---------------------------------------------------------------------------
namespace {
constexpr int NOALLOC_MAX_ROWS = 32768;
constexpr int NOALLOC_PARTS = 3 * 512;
// r, z, p, Ap (3 per row each), Dinv and a zero diagonal term (9 per row
// each), partial sums, scalars, then int storage (flag words, diagonal slots).
constexpr size_t NOALLOC_VEC = 3 * (size_t)NOALLOC_MAX_ROWS;
constexpr size_t NOALLOC_DOUBLES = 4 * NOALLOC_VEC + 18 * (size_t)NOALLOC_MAX_ROWS + NOALLOC_PARTS + 16 + (NOALLOC_MAX_ROWS + 64) / 2;
static_assert(NOALLOC_DOUBLES * sizeof(double) == 8008064, "the documented scratch size");
}  // namespace

static __device__ __align__(256) double g_noallocScratch[NOALLOC_DOUBLES];

namespace {
double* g_noallocAddr[256] = {nullptr};  // device address of the scratch, per device id

// Checks the caller's block-CSR structure while locating the diagonal blocks:
// row pointers non-negative and non-decreasing, column indices in range, and
// exactly one diagonal block per row (an SPD matrix has a nonsingular
// diagonal block in every row; the block-Jacobi inverse needs it).  A failure
// sets a bit of *bad; the caller then reads no block.
__global__ void noallocDiagKernel(int nv, const int* rowPtr, const int* colIdx, int* diagSlot, double* zeroDiag, int* bad) {
    CIPC_KERNEL_LOOP(r, nv) {
        const int b = rowPtr[r], e = rowPtr[r + 1];
        int s = -1, nd = 0;
        if (b < 0 || e < b) {
            atomicOr(bad, 1);
        } else {
            for (int k = b; k < e; ++k) {
                const int cl = colIdx[k];
                if (cl < 0 || cl >= nv) { atomicOr(bad, 2); break; }
                if (cl == r) { s = k; ++nd; }
            }
            if (nd != 1) atomicOr(bad, 4);
        }
        diagSlot[r] = s;
        for (int q = 0; q < 9; ++q) zeroDiag[9 * r + q] = 0.0;
    }
}
}  // namespace

extern "C" int cipc_gpu_pcg_bsr_noalloc(int nv, const int* rowPtr, const int* colIdx, const double* vals, const double* rhs, double* sol,
                                        double relativeTolerance, int maximumIterations, void* stream, int* iterations, double* relResidual) {
    using namespace cipc;
    if (nv <= 0 || !rowPtr || !colIdx || !vals || !rhs || !sol) return CIPC_ERR_INVALID_ARGUMENT;
    if (nv > NOALLOC_MAX_ROWS) return CIPC_ERR_INVALID_ARGUMENT;
    if (!(relativeTolerance > 0) || maximumIterations <= 0) return CIPC_ERR_INVALID_ARGUMENT;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 256) return CIPC_ERR_CUDA;
    if (!g_noallocAddr[dev]) {
        // first call on this device: resolve the array's device address with
        // this device current (the host symbol itself is not a device address)
        void* p = nullptr;
        if (cudaGetSymbolAddress(&p, g_noallocScratch) != cudaSuccess || !p) return CIPC_ERR_CUDA;
        g_noallocAddr[dev] = static_cast<double*>(p);
    }
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    double* base = g_noallocAddr[dev];
    double* r = base;
    double* z = r + NOALLOC_VEC;
    double* p = z + NOALLOC_VEC;
    double* Ap = p + NOALLOC_VEC;
    double* Dinv = Ap + NOALLOC_VEC;
    double* zeroDiag = Dinv + 9 * (size_t)NOALLOC_MAX_ROWS;
    double* parts = zeroDiag + 9 * (size_t)NOALLOC_MAX_ROWS;
    double* scal = parts + NOALLOC_PARTS;
    int* ints = reinterpret_cast<int*>(scal + 16);
    int* flag = ints;
    int* bad = ints + 1;
    int* diagSlot = ints + 64;
    unsigned* bar = reinterpret_cast<unsigned*>(ints + 32);
    int vb = vecBlocks(nv);
    // the structure check runs (and is read back) before any kernel reads a
    // block through the caller's column indices
    int hbad = 0;
    if (cudaMemsetAsync(ints, 0, 64 * sizeof(int), s) != cudaSuccess) return CIPC_ERR_CUDA;
    launch(noallocDiagKernel, vb, VB, 0, s, nv, rowPtr, colIdx, diagSlot, zeroDiag, bad);
    if (cudaGetLastError() != cudaSuccess) return CIPC_ERR_CUDA;
    if (cudaMemcpyAsync(&hbad, bad, sizeof(int), cudaMemcpyDeviceToHost, s) != cudaSuccess) return CIPC_ERR_CUDA;
    if (cudaStreamSynchronize(s) != cudaSuccess) return CIPC_ERR_CUDA;
    if (hbad) return CIPC_ERR_INVALID_ARGUMENT;
    launch(dinvKernel<double>, vb, VB, 0, s, nv, diagSlot, vals, (const int*)nullptr, (const int*)nullptr, (const int*)nullptr,
           (const double*)nullptr, zeroDiag, Dinv);
    if (cudaGetLastError() != cudaSuccess) return CIPC_ERR_CUDA;
    // The textbook recurrences in one cooperative launch, its rows spread over
    // one block per SM while 512 threads hold them.  Bound by the two grid
    // barriers of an iteration: a call on 5,003 rows (96 iterations) takes 1.32 ms
    // on a B200, and took 2.35 with four launches per iteration and a wait
    // every 16.
    int smCount = 0, perSM = 0;
    if (cudaDeviceGetAttribute(&smCount, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return CIPC_ERR_CUDA;
    const int threads = std::min(PB, std::max(32, ((nv * GROUP + smCount - 1) / smCount + 31) / 32 * 32));
    const void* fn = (const void*)pcgPersistentKernel<double, double, false>;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&perSM, fn, threads, 0) != cudaSuccess) return CIPC_ERR_CUDA;
    const int grid = std::max(1, std::min({(nv * GROUP + threads - 1) / threads, perSM * smCount, NOALLOC_PARTS / 3}));
    PcgArgs<double, double> a{};
    a.nv = nv; a.rowPtr = rowPtr; a.col = colIdx; a.val = vals;
    a.diagExtra = zeroDiag; a.Dinv = Dinv; a.b = rhs; a.x = sol; a.r = r; a.z = z; a.p = p; a.Ap = Ap;
    a.partA = parts; a.partB = parts + NOALLOC_PARTS / 3; a.partC = parts + 2 * (NOALLOC_PARTS / 3);
    a.scal = scal; a.flag = flag; a.bar = bar;
    a.tol = relativeTolerance; a.maxIter = maximumIterations;
    void* args[] = {&a};
    ++g_kernelLaunches;
    if (cudaLaunchCooperativeKernel(fn, dim3(grid), dim3(threads), args, 0, s) != cudaSuccess) return CIPC_ERR_CUDA;
    int hflag = 0;
    double hs[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    if (cudaMemcpyAsync(&hflag, flag, sizeof(int), cudaMemcpyDeviceToHost, s) != cudaSuccess) return CIPC_ERR_CUDA;
    if (cudaMemcpyAsync(hs, scal, 8 * sizeof(double), cudaMemcpyDeviceToHost, s) != cudaSuccess) return CIPC_ERR_CUDA;
    if (cudaStreamSynchronize(s) != cudaSuccess) return CIPC_ERR_CUDA;
    if (hflag == 3) return CIPC_ERR_CUDA;  // a grid barrier timed out
    if (iterations) *iterations = (int)hs[4];
    if (relResidual) *relResidual = hs[6] > 0 ? std::sqrt(hs[3] / hs[6]) : 0.0;
    return hflag == 1 ? CIPC_OK : CIPC_ERR_NOT_CONVERGED;
}
