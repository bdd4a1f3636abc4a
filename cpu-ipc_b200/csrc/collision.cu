// Broad phase and step bounds on the GPU.
//
// * LBVH build, faces and edges by the same launches: primitive boxes and scene
//   box -> 30-bit Morton keys with the primitive id in the low word -> one radix
//   sort -> Karras internal nodes -> bottom-up boxes (arrival flags).  Topology
//   follows CPULinearBVH::build, CPU IPC/LBVH.cpp:163-250.
// * Active sets: a warp walks the tree for 32 queries with one shared stack, by
//   the inclusive overlaps(gap) test (LBVH.cpp:157-161), applies the collider /
//   incidence filters of SpatialHash::calculateActivateSet
//   (CPU IPC/CollisionBroadPhase.cpp:765-1059) and emits candidate pairs; one
//   thread per candidate classifies it and emits 64-bit pair keys.  Keys are
//   radix-sorted together, so every list comes out in the
//   reference's order (query ascending, then primitive ascending); PP/PE
//   duplicates are merged by sort + run-length encoding, the job of the
//   reference's std::map.
// * Partial CCD, full (swept) CCD, ground bound, CFL bound and the
//   edge-triangle intersection test (IPCSolver.cpp:476-542, 943-990;
//   ContactMechanics.cpp:3704-3867; FeasibleStep.cpp:8-40).
#include "../../include/cipc_gpu.h"
#include "cipc_internal.h"
#include "geometry.cuh"

#include <cooperative_groups.h>
#include <cub/cub.cuh>
#include <thrust/iterator/counting_iterator.h>

#include <algorithm>
#include <cstdlib>

namespace cipc {

namespace cg = cooperative_groups;

namespace {

constexpr int TB = 128;
inline int blocksFor(int n, int tb = TB) { return std::max(1, std::min((n + tb - 1) / tb, 148 * 32)); }

__device__ __forceinline__ void boxInit(double lo[3], double hi[3]) {
    for (int k = 0; k < 3; ++k) { lo[k] = 1.7976931348623157e308; hi[k] = -1.7976931348623157e308; }
}
__device__ __forceinline__ void boxAdd(double lo[3], double hi[3], d3 p) {
    lo[0] = fmin(lo[0], p.x); lo[1] = fmin(lo[1], p.y); lo[2] = fmin(lo[2], p.z);
    hi[0] = fmax(hi[0], p.x); hi[1] = fmax(hi[1], p.y); hi[2] = fmax(hi[2], p.z);
}
// (query lo, hi).overlaps(node lo, hi, gap), inclusive.
__device__ __forceinline__ bool overlaps(const double* qlo, const double* qhi, const double* nlo, const double* nhi, double gap) {
    return !((nlo[0] - qhi[0] > gap) || (nlo[1] - qhi[1] > gap) || (nlo[2] - qhi[2] > gap) || (qlo[0] - nhi[0] > gap) ||
             (qlo[1] - nhi[1] > gap) || (qlo[2] - nhi[2] > gap));
}

// Swept point box: combine(p) then combine(p - step * d).
__device__ __forceinline__ void sweptAdd(double lo[3], double hi[3], d3 p, d3 d, double step) {
    boxAdd(lo, hi, p);
    boxAdd(lo, hi, p - step * d);
}

// The face and the edge tree are built by the same launches (blockIdx.y 0 and
// 1): a build is a chain of small kernels, each a few microseconds of latency,
// and one radix sort serves both key sets.
struct TreeBuild {
    int n, verts;          // primitives, vertices per primitive (3 faces, 2 edges)
    const int* prim;       // vertex indices
    double *plo, *phi;     // primitive boxes
    double* part;          // 6 per block of the box kernel
    uint64_t* keys;        // unsorted Morton keys
    const uint64_t* sorted;
    int* nbig;
    int4* links;           // internal nodes: left, right, parent, the other end of the node's leaf range
    int *leafParent, *leafPrim, *flags;
    double *lo, *hi;
    float* rec;
};
struct TreePair {
    TreeBuild t[2];
};

// Primitive boxes at x, or swept from x to x - step d, and each block's box of
// its primitives (min and max do not depend on the order).
__global__ void primBoxKernel(TreePair pair, const double* x, const double* d, double stepVal, const double* stepPtr, int swept) {
    const TreeBuild& t = pair.t[blockIdx.y];
    const double step = stepPtr ? *stepPtr : stepVal;
    double bl[3], bh[3];
    boxInit(bl, bh);
    CIPC_KERNEL_LOOP(f, t.n) {
        double l[3], h[3];
        boxInit(l, h);
        for (int k = 0; k < t.verts; ++k) {
            const int v = t.prim[t.verts * f + k];
            if (swept) sweptAdd(l, h, ld3(x, v), ld3(d, v), step);
            else boxAdd(l, h, ld3(x, v));
        }
        for (int k = 0; k < 3; ++k) {
            t.plo[3 * f + k] = l[k];
            t.phi[3 * f + k] = h[k];
            bl[k] = fmin(bl[k], l[k]);
            bh[k] = fmax(bh[k], h[k]);
        }
    }
    for (int k = 0; k < 3; ++k) {
        bl[k] = blockReduce(bl[k], MinOp(), 1.7976931348623157e308);
        __syncthreads();
        bh[k] = blockReduce(bh[k], MaxOp(), -1.7976931348623157e308);
        __syncthreads();
        if (threadIdx.x == 0) { t.part[6 * blockIdx.x + k] = bl[k]; t.part[6 * blockIdx.x + 3 + k] = bh[k]; }
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) *t.nbig = 0;
}

__device__ __forceinline__ uint32_t expandBits(uint32_t v) {
    v = (v * 0x00010001u) & 0xFF0000FFu;
    v = (v * 0x00000101u) & 0x0F00F00Fu;
    v = (v * 0x00000011u) & 0xC30C30C3u;
    v = (v * 0x00000005u) & 0x49249249u;
    return v;
}
__device__ __forceinline__ uint32_t quantize(double v) {
    v = fmax(0.0, fmin(v * 1024.0, 1023.0));
    return (uint32_t)v;
}

// Morton keys (30-bit code << 32 | index).  A primitive whose box spans
// more than bigExtent along an axis (the walls of a container, a fast swept
// primitive) gets bit 62 instead: the sort moves it past the others, the
// tree is built over the rest, and every query tests the few large ones
// directly - a large box would otherwise widen all its ancestors' boxes and
// draw every query down their paths.  *nbig counts them.
// Every block first reduces the box kernel's nbPart partials to the scene box.
// The edges' keys carry bit 63: one sort puts them behind the faces'.
__global__ void mortonKernel(TreePair pair, int nbPart, double bigExtent) {
    const TreeBuild& t = pair.t[blockIdx.y];
    __shared__ double scene[6];
    {
        double l[3], h[3];
        boxInit(l, h);
        for (int i = threadIdx.x; i < nbPart; i += blockDim.x)
            for (int k = 0; k < 3; ++k) { l[k] = fmin(l[k], t.part[6 * i + k]); h[k] = fmax(h[k], t.part[6 * i + 3 + k]); }
        for (int k = 0; k < 3; ++k) {
            l[k] = blockReduce(l[k], MinOp(), 1.7976931348623157e308);
            __syncthreads();
            h[k] = blockReduce(h[k], MaxOp(), -1.7976931348623157e308);
            __syncthreads();
            if (threadIdx.x == 0) { scene[k] = l[k]; scene[3 + k] = h[k]; }
        }
        __syncthreads();
    }
    const uint64_t tag = (uint64_t)blockIdx.y << 63;
    const double *lo = t.plo, *hi = t.phi;
    CIPC_KERNEL_LOOP(i, t.n) {
        bool big = false;
        for (int k = 0; k < 3; ++k) big = big || (hi[3 * i + k] - lo[3 * i + k] > bigExtent);
        if (big) {
            atomicAdd(t.nbig, 1);
            t.keys[i] = tag | (1ull << 62) | (uint32_t)i;
            continue;
        }
        double c[3], q[3];
        for (int k = 0; k < 3; ++k) {
            c[k] = 0.5 * (lo[3 * i + k] + hi[3 * i + k]);
            double ext = scene[3 + k] - scene[k];
            double off = c[k] - scene[k];
            q[k] = ext > 0.0 ? off / ext : 0.0;
        }
        uint32_t code = (expandBits(quantize(q[0])) << 2) | (expandBits(quantize(q[1])) << 1) | expandBits(quantize(q[2]));
        t.keys[i] = tag | ((uint64_t)code << 32) | (uint32_t)i;
    }
}

__device__ __forceinline__ int prefixLen(const uint64_t* k, int n, int a, int b) {
    if (b < 0 || b >= n) return -1;
    uint64_t x = k[a] ^ k[b];
    return x == 0 ? 64 : __clzll(x);
}

// Internal nodes (topology as CPULinearBVH::build) and the leaves' primitives.
__global__ void karrasKernel(TreePair pair) {
    const TreeBuild& t = pair.t[blockIdx.y];
    const uint64_t* keys = t.sorted;
    const int n = t.n - *t.nbig;  // leaves of the tree (the large primitives stay out)
    CIPC_KERNEL_LOOP(in, n) {
        t.leafPrim[in] = (int)(keys[in] & 0xffffffffu);
        if (in == 0) {
            if (n > 1) t.links[0].z = -1;
            else t.leafParent[0] = -1;
        }
        if (in == n - 1) continue;
        int first, last, other;
        if (in == 0) { first = 0; last = n - 1; other = last; }
        else {
            int lp = prefixLen(keys, n, in, in - 1), rp = prefixLen(keys, n, in, in + 1);
            int dir = rp > lp ? 1 : -1;
            int minp = min(lp, rp);
            int maxLen = 2;
            while (prefixLen(keys, n, in, in + dir * maxLen) > minp) maxLen <<= 1;
            int len = 0;
            for (int step = maxLen >> 1; step > 0; step >>= 1)
                if (prefixLen(keys, n, in, in + dir * (len + step)) > minp) len += step;
            other = in + dir * len;
            first = min(in, other); last = max(in, other);
        }
        int split;
        uint64_t fc = keys[first], lc = keys[last];
        if (fc == lc) split = (first + last) >> 1;
        else {
            int common = __clzll(fc ^ lc);
            split = first;
            unsigned step = (unsigned)(last - first);
            do {
                step = (step + 1) >> 1;
                int cand = split + (int)step;
                if (cand < last && __clzll(fc ^ keys[cand]) > common) split = cand;
            } while (step > 1);
        }
        const bool leafL = split == first, leafR = split + 1 == last;
        const int l = leafL ? split + n - 1 : split, r = leafR ? split + n : split + 1;
        t.links[in].x = l;
        t.links[in].y = r;
        t.links[in].w = other;
        if (leafL) t.leafParent[split] = in; else t.links[l].z = in;
        if (leafR) t.leafParent[split + 1] = in; else t.links[r].z = in;
        t.flags[in] = 0;
    }
}

__device__ __forceinline__ int atomAddAcqRel(int* p, int v) {
    int old;
    asm volatile("atom.add.acq_rel.gpu.s32 %0, [%1], %2;" : "=r"(old) : "l"(p), "r"(v) : "memory");
    return old;
}

// Bottom-up boxes: the second child to arrive at a node combines both child
// boxes and goes on with the node's.  It also writes the node's traversal record:
// the boxes of both children rounded outward to FP32 (lo down, hi up) and the
// children's node indices, 64 bytes, so that one load tests both children.
//
// Bound: the chain of arrivals up the tree, each a release, an atomic and the
// sibling's box through L2 (about 2.5 us; 42 us for 50-70k leaves).  A block owns
// REFIT consecutive leaves, and a node whose leaf range lies among them (half the
// levels and more) is combined through shared memory; only the rest meets in
// global memory, by acquire-release atomics: they publish the box this thread
// wrote for the child it came from and, for the second arrival, make the
// sibling's box visible.
constexpr int REFIT = 256;
__global__ void __launch_bounds__(REFIT) refitKernel(TreePair pair) {
    const TreeBuild& t = pair.t[blockIdx.y];
    __shared__ double sbox[REFIT][2][6];
    __shared__ int sflag[REFIT];
    const int n = t.n - *t.nbig;
    for (int base = blockIdx.x * REFIT; base < n; base += gridDim.x * REFIT) {
        __syncthreads();  // the previous leaves' boxes are done with
        sflag[threadIdx.x] = 0;
        __syncthreads();
        const int s = base + (int)threadIdx.x, top = min(base + REFIT, n);
        if (s >= n) continue;
        const int prim = t.leafPrim[s];
        double b[6];
        for (int k = 0; k < 3; ++k) { b[k] = t.plo[3 * prim + k]; b[3 + k] = t.phi[3 * prim + k]; }
        int node = s + n - 1, p = t.leafParent[s];
        for (int k = 0; k < 3; ++k) { t.lo[3 * (size_t)node + k] = b[k]; t.hi[3 * (size_t)node + k] = b[3 + k]; }
        for (int guard = 0; guard < 64 && p >= 0; ++guard) {
            const int4 link = t.links[p];  // left, right, parent, other end of the range
            const int side = link.x == node ? 0 : 1;
            double o[6];
            if (min(p, link.w) >= base && max(p, link.w) < top) {
                double(*slot)[6] = sbox[p - base];
                for (int k = 0; k < 6; ++k) slot[side][k] = b[k];
                __threadfence_block();
                if (atomicAdd(&sflag[p - base], 1) == 0) break;
                __threadfence_block();
                for (int k = 0; k < 6; ++k) o[k] = reinterpret_cast<volatile double*>(slot[1 - side])[k];
            } else {
                if (atomAddAcqRel(&t.flags[p], 1) == 0) break;
                const size_t sib = side == 0 ? link.y : link.x;
                for (int k = 0; k < 3; ++k) { o[k] = __ldcg(&t.lo[3 * sib + k]); o[3 + k] = __ldcg(&t.hi[3 * sib + k]); }
            }
            float r[16];
            for (int k = 0; k < 3; ++k) {
                const double l0 = side == 0 ? b[k] : o[k], l1 = side == 0 ? o[k] : b[k];
                const double h0 = side == 0 ? b[3 + k] : o[3 + k], h1 = side == 0 ? o[3 + k] : b[3 + k];
                r[k] = __double2float_rd(l0); r[3 + k] = __double2float_ru(h0);
                r[6 + k] = __double2float_rd(l1); r[9 + k] = __double2float_ru(h1);
                b[k] = fmin(l0, l1);
                b[3 + k] = fmax(h0, h1);
                t.lo[3 * (size_t)p + k] = b[k];
                t.hi[3 * (size_t)p + k] = b[3 + k];
            }
            r[12] = __int_as_float(link.x);
            r[13] = __int_as_float(link.y);
            r[14] = r[15] = 0.f;
            float4* out = reinterpret_cast<float4*>(t.rec) + 4 * (size_t)p;
            for (int k = 0; k < 4; ++k) out[k] = make_float4(r[4 * k], r[4 * k + 1], r[4 * k + 2], r[4 * k + 3]);
            node = p;
            p = link.z;
        }
    }
}

struct BvhView {
    static constexpr bool kSplitsBig = true;  // large primitives are kept out of the tree (see warpQueries)
    double bigExtent;  // a box wider than this along an axis is large
    int nAll;         // primitives; the tree holds nAll - *nbig of them
    const int* nbig;  // primitives kept out of the tree (their keys sort last)
    const uint64_t* keys;
    const int4* links;  // left, right, parent (internal nodes)
    const int *leafParent, *leafPrim;
    const double *lo, *hi;
    const double *plo, *phi;  // primitive boxes
    const float4* rec;
    int walkCap;  // entries a warp's stack may hold (<= WALK_CAP)
};
constexpr int WALK_CAP = 1024;
// CIPC_WALK_STACK: a smaller stack (a small value exercises the subtree walks)
int walkCap() {
    static int v = -1;
    if (v < 0) {
        const char* e = std::getenv("CIPC_WALK_STACK");
        v = e ? std::min(WALK_CAP, std::max(32, std::atoi(e))) : WALK_CAP;
    }
    return v;
}
BvhView view(const DevBvh& t) {
    return BvhView{t.bigExtent, t.n, t.bigCount, t.keys, t.links, t.leafParent, t.leafPrim, t.lo, t.hi, t.primLo, t.primHi,
                   reinterpret_cast<const float4*>(t.rec.p), walkCap()};
}

__device__ __forceinline__ bool isLargeBox(const double* lo, const double* hi, double ext) {
    return (hi[0] - lo[0] > ext) || (hi[1] - lo[1] > ext) || (hi[2] - lo[2] > ext);
}

// Walk of one warp's 32 queries over the tree.  One thread per query walks its
// own path, so a warp lasts as long as its query with the most nodes, at one
// memory latency per node (cloth drape 128: 1.7 ms for the edge-edge walk, a few
// queries with some thousand nodes each).  Here the warp keeps one stack of
// (node, query) pairs in shared memory and every lane pops any of them, so the
// lanes stay busy until the warp's common work is done.  The boxes of an
// internal node's children come from its 64-byte record and are tested in FP32
// against the query box grown by the gap and rounded outward: it contains every
// leaf that passes the FP64 test, which alone decides what is reported.  The
// stack is popped from its end, which keeps it near 32 times the depth; children
// that do not fit are walked by the lane itself (walkSubtree).  f(query slot,
// primitive) is called by the lane that met the leaf.  Sets, energy, intersection test and step bounds of the 128 x 128 cloth
// on its cube: 5.81 -> 3.61 ms; of 27 cubes of 12 cells: 4.49 -> 3.65 ms (B200).
constexpr int WALK_WARPS = TB / 32;
constexpr int WALK_SLOT_SHIFT = 27;  // entries: node index in the low bits (a tree has far fewer than 2^27 nodes), query slot above
struct WalkSmem {
    unsigned stack[WALK_CAP];
    float lo[3][32], hi[3][32];     // grown by the gap, outward
    double dlo[3][32], dhi[3][32];  // the query boxes
};

__device__ __forceinline__ bool overlapsF(const WalkSmem& sm, int s, float lx, float ly, float lz, float hx, float hy, float hz) {
    return !((lx > sm.hi[0][s]) || (ly > sm.hi[1][s]) || (lz > sm.hi[2][s]) || (sm.lo[0][s] > hx) || (sm.lo[1][s] > hy) || (sm.lo[2][s] > hz));
}
__device__ __forceinline__ bool overlapsLeaf(const BvhView& t, const WalkSmem& sm, int s, int node, double gap) {
    const double qlo[3] = {sm.dlo[0][s], sm.dlo[1][s], sm.dlo[2][s]}, qhi[3] = {sm.dhi[0][s], sm.dhi[1][s], sm.dhi[2][s]};
    return overlaps(qlo, qhi, t.lo + 3 * (size_t)node, t.hi + 3 * (size_t)node, gap);
}

// the leaves under an internal node, depth first; back up along the parents
template <class F>
__device__ __noinline__ void walkSubtree(const BvhView& t, const WalkSmem& sm, int s, int root, int n, double gap, int* status, F& f) {
    const int firstLeaf = n - 1;
    int cur = t.links[root].x;
    for (int visits = 0;; ++visits) {
        if (visits > 4 * n) { raiseStatus(status, CIPC_ST_STACK_OVERFLOW); return; }
        if (overlapsLeaf(t, sm, s, cur, gap)) {
            if (cur < firstLeaf) { cur = t.links[cur].x; continue; }
            f(s, t.leafPrim[cur - firstLeaf]);
        }
        int p = cur < firstLeaf ? t.links[cur].z : t.leafParent[cur - firstLeaf];
        while (cur != t.links[p].x) {  // both of p's children are done
            if (p == root) return;
            cur = p;
            p = t.links[cur].z;
        }
        cur = t.links[p].y;
    }
}

template <class F>
__device__ __forceinline__ void warpWalk(const BvhView& t, int n, WalkSmem& sm, bool active, const double* qlo, const double* qhi, double gap,
                                         int* status, F& f) {
    const int lane = threadIdx.x & 31, firstLeaf = n - 1;
    const unsigned below = (1u << lane) - 1u;
    if (n <= 0) return;
    __syncwarp();  // the previous queries' boxes are no longer read
    for (int k = 0; k < 3; ++k) {
        sm.dlo[k][lane] = qlo[k];
        sm.dhi[k][lane] = qhi[k];
        sm.lo[k][lane] = __double2float_rd(__dadd_rd(qlo[k], -gap));
        sm.hi[k][lane] = __double2float_ru(__dadd_ru(qhi[k], gap));
    }
    active = active && overlaps(qlo, qhi, t.lo, t.hi, gap);  // the root (node 0)
    if (n == 1) {
        if (active) f(lane, t.leafPrim[0]);
        return;
    }
    const unsigned start = __ballot_sync(0xffffffffu, active);
    if (active) sm.stack[__popc(start & below)] = (unsigned)lane << WALK_SLOT_SHIFT;
    int size = __popc(start);
    __syncwarp();
    while (size > 0) {
        const int take = min(size, 32);
        bool in0 = false, in1 = false, leaf0 = false, leaf1 = false;
        int s = 0, c0 = 0, c1 = 0;
        if (lane < take) {
            const unsigned e = sm.stack[size - take + lane];
            s = (int)(e >> WALK_SLOT_SHIFT);
            const float4* r = t.rec + 4 * (size_t)(e & ((1u << WALK_SLOT_SHIFT) - 1u));
            const float4 a = r[0], b = r[1], cc = r[2], d = r[3];
            c0 = __float_as_int(d.x); c1 = __float_as_int(d.y);
            in0 = overlapsF(sm, s, a.x, a.y, a.z, a.w, b.x, b.y);
            in1 = overlapsF(sm, s, b.z, b.w, cc.x, cc.y, cc.z, cc.w);
            leaf0 = in0 && c0 >= firstLeaf;
            leaf1 = in1 && c1 >= firstLeaf;
            in0 = in0 && !leaf0;
            in1 = in1 && !leaf1;
        }
        size -= take;
        const unsigned b0 = __ballot_sync(0xffffffffu, in0), b1 = __ballot_sync(0xffffffffu, in1);
        const int pushed = __popc(b0) + __popc(b1);
        if (size + pushed <= t.walkCap) {
            if (in0) sm.stack[size + __popc(b0 & below)] = ((unsigned)s << WALK_SLOT_SHIFT) | (unsigned)c0;
            if (in1) sm.stack[size + __popc(b0) + __popc(b1 & below)] = ((unsigned)s << WALK_SLOT_SHIFT) | (unsigned)c1;
            size += pushed;
        } else {
            if (in0) walkSubtree(t, sm, s, c0, n, gap, status, f);
            if (in1) walkSubtree(t, sm, s, c1, n, gap, status, f);
        }
        if (leaf0 && overlapsLeaf(t, sm, s, c0, gap)) f(s, t.leafPrim[c0 - firstLeaf]);
        if (leaf1 && overlapsLeaf(t, sm, s, c1, gap)) f(s, t.leafPrim[c1 - firstLeaf]);
        __syncwarp();
    }
}

// The 32 queries first + lane of a warp (every lane calls): f(query, prim,
// fromLargeList).  For queries over the tree's own primitive set (edges against
// edges, largeQuery may be true) a large query does not walk the tree; it meets
// only the large primitives.  Its pairs with the tree's primitives are reported
// from their side, through their own loop over the large primitives, which
// therefore sees every large primitive whatever the indices.
template <class F>
__device__ __forceinline__ void warpQueries(const BvhView& t, WalkSmem& sm, int first, bool active, const double* qlo, const double* qhi, double gap,
                                            bool largeQuery, int* status, F f) {
    if (t.nAll <= 0) return;
    const int nb = *t.nbig, n = t.nAll - nb;
    auto g = [&](int s, int p) { f(first + s, p, false); };
    warpWalk(t, n, sm, active && !largeQuery, qlo, qhi, gap, status, g);
    if (!active) return;
    const int query = first + (int)(threadIdx.x & 31);
    for (int b = 0; b < nb; ++b) {
        const int p = (int)(t.keys[n + b] & 0xffffffffu);
        if (overlaps(qlo, qhi, t.plo + 3 * p, t.phi + 3 * p, gap)) f(query, p, true);
    }
}

// ---------------------------------------------------------------------------
// Spatial-hash backend (the reference's SpatialHash, CollisionBroadPhase.cpp:
// 11-763, as an A/B alternative to the LBVH): every primitive box is entered
// in the cubic cells of edge `h` (the mean surface edge length, as the
// reference's sh.build(mesh, averageEdgeLenth)) that it touches, as
// (cell key, primitive) pairs sorted by key.  A query visits the cells of its
// box grown by the gap (and one cell more on each side, against rounding),
// finds each cell's run by binary search, and reports a primitive only in the
// lowest cell it shares with the query, after the same inclusive FP64 box
// test as the LBVH walk - so both backends report the same set.  Primitives
// touching more than HASH_MAX_CELLS cells are kept in a list that every query
// tests; a query touching more than HASH_MAX_QUERY cells tests all
// primitives.
// ---------------------------------------------------------------------------
constexpr int HASH_MAX_CELLS = 64;
constexpr long long HASH_MAX_QUERY = 4096;
constexpr int HASH_BIAS = 1 << 20;  // cell coordinates are offset into [0, 2^21)

struct HashView {
    static constexpr bool kSplitsBig = false;
    double bigExtent;
    int n, pairs;
    double inv;
    const uint64_t* key;
    const int* prim;
    const int* big;
    const int* nbig;
    const double *plo, *phi;
};

__device__ __forceinline__ int hashCell(double v, double inv) {
    const double c = floor(v * inv) + (double)HASH_BIAS;
    return (int)fmin(fmax(c, 0.0), (double)(2 * HASH_BIAS - 1));
}
__device__ __forceinline__ uint64_t hashKeyOf(int ix, int iy, int iz) {
    return ((uint64_t)ix << 42) | ((uint64_t)iy << 21) | (uint64_t)iz;
}

template <class F>
__device__ __forceinline__ void traverse(const HashView& t, const double* qlo, const double* qhi, double gap, int* status, F f) {
    if (t.n <= 0) return;
    int lo[3], hi[3];
    long long cells = 1;
    for (int k = 0; k < 3; ++k) {
        lo[k] = max(hashCell(qlo[k] - gap, t.inv) - 1, 0);
        hi[k] = min(hashCell(qhi[k] + gap, t.inv) + 1, 2 * HASH_BIAS - 1);
        cells *= (long long)(hi[k] - lo[k] + 1);
    }
    if (cells > HASH_MAX_QUERY) {  // a large query box: test every primitive
        for (int p = 0; p < t.n; ++p)
            if (overlaps(qlo, qhi, t.plo + 3 * p, t.phi + 3 * p, gap)) f(p);
        return;
    }
    for (int iz = lo[2]; iz <= hi[2]; ++iz)
        for (int iy = lo[1]; iy <= hi[1]; ++iy)
            for (int ix = lo[0]; ix <= hi[0]; ++ix) {
                const uint64_t key = hashKeyOf(ix, iy, iz);
                int a = 0, b = t.pairs;  // first pair with a key >= key
                while (a < b) {
                    const int m = (a + b) >> 1;
                    if (t.key[m] < key) a = m + 1;
                    else b = m;
                }
                for (int k = a; k < t.pairs && t.key[k] == key; ++k) {
                    const int p = t.prim[k];
                    const double* pl = t.plo + 3 * p;
                    // the lowest cell the primitive shares with the query
                    if (max(hashCell(pl[0], t.inv), lo[0]) != ix || max(hashCell(pl[1], t.inv), lo[1]) != iy ||
                        max(hashCell(pl[2], t.inv), lo[2]) != iz)
                        continue;
                    if (overlaps(qlo, qhi, pl, t.phi + 3 * p, gap)) f(p);
                }
            }
    const int nb = *t.nbig;
    for (int b = 0; b < nb; ++b) {
        const int p = t.big[b];
        if (overlaps(qlo, qhi, t.plo + 3 * p, t.phi + 3 * p, gap)) f(p);
    }
}

template <class F>
__device__ __forceinline__ void warpQueries(const HashView& t, WalkSmem&, int first, bool active, const double* qlo, const double* qhi, double gap, bool,
                                            int* status, F f) {
    const int query = first + (int)(threadIdx.x & 31);
    if (active) traverse(t, qlo, qhi, gap, status, [&](int p) { f(query, p, false); });
}

// Loop of the query kernels: first is the warp's first query, uniform across
// the warp (every lane takes part in a walk), query the lane's own.
#define CIPC_WARP_QUERIES(first, query, n)                                                                                      \
    for (int first = (blockIdx.x * TB + (threadIdx.x & ~31)), query = first + (int)(threadIdx.x & 31); first < (n);              \
         first += gridDim.x * TB, query += gridDim.x * TB)

__global__ void hashCountKernel(int n, const double* plo, const double* phi, double inv, int* count, int* bigFlag) {
    CIPC_KERNEL_LOOP(p, n) {
        long long cells = 1;
        for (int k = 0; k < 3; ++k) cells *= (long long)(hashCell(phi[3 * p + k], inv) - hashCell(plo[3 * p + k], inv) + 1);
        const bool big = cells > HASH_MAX_CELLS;
        count[p] = big ? 0 : (int)cells;
        bigFlag[p] = big ? 1 : 0;
    }
}

__global__ void hashEmitKernel(int n, const double* plo, const double* phi, double inv, const int* offset, const int* count, uint64_t* key, int* prim) {
    CIPC_KERNEL_LOOP(p, n) {
        if (count[p] == 0) continue;
        int lo[3], hi[3];
        for (int k = 0; k < 3; ++k) { lo[k] = hashCell(plo[3 * p + k], inv); hi[k] = hashCell(phi[3 * p + k], inv); }
        int o = offset[p];
        for (int iz = lo[2]; iz <= hi[2]; ++iz)
            for (int iy = lo[1]; iy <= hi[1]; ++iy)
                for (int ix = lo[0]; ix <= hi[0]; ++ix) { key[o] = hashKeyOf(ix, iy, iz); prim[o] = p; ++o; }
    }
}

__device__ __forceinline__ bool isCollider(int t) { return t >= 2; }

// Packed PP/PE key: lexicographic order of (c0 = -v-1, c1, c2) with c3 = -1.
constexpr uint64_t M21 = (1ull << 21) - 1;
__device__ __forceinline__ uint64_t ppeKey(int c0, int c1, int c2) {
    uint64_t v = (uint64_t)(-c0 - 1);
    return ((M21 - v) << 42) | ((uint64_t)c1 << 21) | (uint64_t)(c2 + 1);
}

// Appends a key to a list: the lanes of a warp that emit at the same point
// take one atomic for all of them (the leader reserves the group's slots and
// broadcasts the base).  The list is sorted afterwards, so the order of the
// slots does not matter.
struct Emit {
    uint64_t* buf;
    int cap;
    int* counter;
    __device__ void operator()(uint64_t k, int* status) const {
        cg::coalesced_group g = cg::coalesced_threads();
        int base = 0;
        if (g.thread_rank() == 0) base = atomicAdd(counter, (int)g.size());
        const int i = g.shfl(base, 0) + (int)g.thread_rank();
        if (i < cap) buf[i] = k;
        else raiseStatus(status, CIPC_ST_CAPACITY);
    }
};

// Active sets in two kernels per kind, so that the distance classification
// runs one thread per candidate instead of inside the divergent tree walk:
// the walk emits every candidate pair (the partial-CCD set), then one thread
// per stored candidate classifies it and emits the contact keys.  The sets
// are sorted afterwards, so the order of emission does not matter.
template <class View>
__global__ void activePTKernel(int nsv, const int* surfVerts, const int* faces, const int* btype, const double* x, View tree, double sq, Emit ccd,
                               int* status) {
    __shared__ WalkSmem sm[WALK_WARPS];
    CIPC_WARP_QUERIES(first, query, nsv) {
        const bool active = query < nsv;
        const d3 p = ld3(x, surfVerts[active ? query : 0]);
        const double lo[3] = {p.x, p.y, p.z};
        warpQueries(tree, sm[threadIdx.x >> 5], first, active, lo, lo, sq, false, status, [&](int svI, int sfI, bool) {
            const int vI = surfVerts[svI];
            int f0 = faces[3 * sfI], f1 = faces[3 * sfI + 1], f2 = faces[3 * sfI + 2];
            if (isCollider(btype[vI]) && isCollider(btype[f0]) && isCollider(btype[f1]) && isCollider(btype[f2])) return;
            if (vI == f0 || vI == f1 || vI == f2) return;
            ccd(((uint64_t)svI << 32) | (uint32_t)sfI, status);
        });
    }
}

// the point-triangle candidates (svI << 32 | sfI) stored by activePTKernel
__global__ void activePTClassKernel(const uint64_t* cand, const int* count, int cap, const int* surfVerts, const int* faces, const double* x,
                                    double Hhat, Emit ptk, Emit ppe, int* status) {
    const int n = min(*count, cap);
    CIPC_KERNEL_LOOP(k, n) {
        const uint64_t key = cand[k];
        const int svI = (int)(key >> 32), sfI = (int)(key & 0xffffffffu);
        const int vI = surfVerts[svI];
        const int f0 = faces[3 * sfI], f1 = faces[3 * sfI + 1], f2 = faces[3 * sfI + 2];
        const d3 p = ld3(x, vI), a = ld3(x, f0), b = ld3(x, f1), c = ld3(x, f2);
        double d;
        switch (dTypePT(p, a, b, c)) {
        case 0: d = dPP(p, a); if (d < Hhat) ppe(ppeKey(-vI - 1, f0, -1), status); break;
        case 1: d = dPP(p, b); if (d < Hhat) ppe(ppeKey(-vI - 1, f1, -1), status); break;
        case 2: d = dPP(p, c); if (d < Hhat) ppe(ppeKey(-vI - 1, f2, -1), status); break;
        case 3: d = dPE(p, a, b); if (d < Hhat) ppe(ppeKey(-vI - 1, f0, f1), status); break;
        case 4: d = dPE(p, b, c); if (d < Hhat) ppe(ppeKey(-vI - 1, f1, f2), status); break;
        case 5: d = dPE(p, c, a); if (d < Hhat) ppe(ppeKey(-vI - 1, f2, f0), status); break;
        default: d = dPT(p, a, b, c); if (d < Hhat) ptk(key, status); break;
        }
    }
}

template <class View>
__global__ void activeEEKernel(int ne, const int* edges, const int* btype, const double* x, View tree, double sq, Emit ccd, int* status) {
    __shared__ WalkSmem sm[WALK_WARPS];
    CIPC_WARP_QUERIES(first, query, ne) {
        const bool active = query < ne;
        double lo[3], hi[3];
        boxInit(lo, hi);
        if (active) {
            boxAdd(lo, hi, ld3(x, edges[2 * query]));
            boxAdd(lo, hi, ld3(x, edges[2 * query + 1]));
        }
        const bool large = View::kSplitsBig && active && isLargeBox(lo, hi, tree.bigExtent);
        // the pair (eI, eJ), eI < eJ, as the reference forms it
        auto pair = [&](int eI, int eJ) {
            int e0 = edges[2 * eI], e1 = edges[2 * eI + 1];
            int g0 = edges[2 * eJ], g1 = edges[2 * eJ + 1];
            if (isCollider(btype[e0]) && isCollider(btype[e1]) && isCollider(btype[g0]) && isCollider(btype[g1])) return;
            if (e0 == g0 || e0 == g1 || e1 == g0 || e1 == g1) return;
            ccd(((uint64_t)eI << 32) | (uint32_t)eJ, status);
        };
        warpQueries(tree, sm[threadIdx.x >> 5], first, active, lo, hi, sq, large, status, [&](int self, int other, bool fromLarge) {
            // a pair is handled once: by its lower index, except that a small
            // edge handles its pairs with the large ones either way (the large
            // list is walked by the query's own lane, whose flag this is)
            if (!fromLarge || large) {
                if (other > self) pair(self, other);
            } else if (other != self) {
                if (other > self) pair(self, other);
                else pair(other, self);
            }
        });
    }
}

// the edge-edge candidates (eI << 32 | eJ) stored by activeEEKernel,
// classified as the reference does with eI's points first
__global__ void activeEEClassKernel(const uint64_t* cand, const int* count, int cap, const int* edges, const double* x, const double* rest,
                                    double Hhat, Emit eek, Emit moll, Emit ppe, int* status) {
    const int n = min(*count, cap);
    CIPC_KERNEL_LOOP(k, n) {
        const uint64_t key = cand[k];
        const int eI = (int)(key >> 32), eJ = (int)(key & 0xffffffffu);
        const int e0 = edges[2 * eI], e1 = edges[2 * eI + 1];
        const int g0 = edges[2 * eJ], g1 = edges[2 * eJ + 1];
        const d3 p0 = ld3(x, e0), p1 = ld3(x, e1), q0 = ld3(x, g0), q1 = ld3(x, g1);
        const int t = dTypeEE(p0, p1, q0, q1);
        const double cs = crossSqNormEE(p0, p1, q0, q1);
        const double ex = 1e-3 * sqn(ld3(rest, e0) - ld3(rest, e1)) * sqn(ld3(rest, g0) - ld3(rest, g1));
        const bool mol = cs < ex;
        double d;
        int c0 = 0, c1 = 0, c2 = -1;
        switch (t) {
        case 0: d = dPP(p0, q0); c0 = -e0 - 1; c1 = g0; break;
        case 1: d = dPP(p0, q1); c0 = -e0 - 1; c1 = g1; break;
        case 2: d = dPE(p0, q0, q1); c0 = -e0 - 1; c1 = g0; c2 = g1; break;
        case 3: d = dPP(p1, q0); c0 = -e1 - 1; c1 = g0; break;
        case 4: d = dPP(p1, q1); c0 = -e1 - 1; c1 = g1; break;
        case 5: d = dPE(p1, q0, q1); c0 = -e1 - 1; c1 = g0; c2 = g1; break;
        case 6: d = dPE(q0, p0, p1); c0 = -g0 - 1; c1 = e0; c2 = e1; break;
        case 7: d = dPE(q1, p0, p1); c0 = -g1 - 1; c1 = e0; c2 = e1; break;
        default: d = dEE(p0, p1, q0, q1); break;
        }
        if (!(d < Hhat)) continue;
        if (mol) moll(((uint64_t)eI << 34) | ((uint64_t)eJ << 4) | (uint64_t)t, status);
        else if (t == 8) eek(key, status);
        else ppe(ppeKey(c0, c1, c2), status);
    }
}

// The six lists of an active-set pass (candidate pairs and contacts of both
// kinds, mollified pairs, PP/PE contacts) are sorted at once: a sort of some
// ten thousand keys is a dozen launches of 3-9 us each, whatever it sorts.  Each
// key is packed to the bits its indices need, below its list's number.
struct SetLists {
    uint64_t* key[6];  // PT candidates, PT, PP/PE, EE candidates, EE, mollified
    int end[6];        // where the list ends in the common array
    int faceBits, edgeBits, vertBits, tagShift;
};
__device__ __forceinline__ int listOf(const SetLists& s, int i) {
    int l = 0;
    while (i >= s.end[l]) ++l;
    return l;
}
__global__ void packSetsKernel(SetLists s, uint64_t* out) {
    CIPC_KERNEL_LOOP(i, s.end[5]) {
        const int l = listOf(s, i);
        const uint64_t k = s.key[l][i - (l ? s.end[l - 1] : 0)];
        uint64_t v;
        if (l == 2) {  // (M21 - vertex, c1, c2 + 1), the order of the fields kept
            const uint64_t m = (1ull << s.vertBits) - 1;
            v = ((m - (M21 - (k >> 42))) << (2 * s.vertBits)) | (((k >> 21) & M21) << s.vertBits) | (k & M21);
        } else if (l == 5) {
            v = ((k >> 34) << (s.edgeBits + 4)) | (k & ((1ull << 34) - 1));
        } else {
            v = ((k >> 32) << (l < 2 ? s.faceBits : s.edgeBits)) | (k & 0xffffffffu);
        }
        out[i] = ((uint64_t)l << s.tagShift) | v;
    }
}
__global__ void unpackSetsKernel(SetLists s, const uint64_t* sorted) {
    CIPC_KERNEL_LOOP(i, s.end[5]) {
        const int l = listOf(s, i);
        const uint64_t v = sorted[i] & ((1ull << s.tagShift) - 1);
        uint64_t k;
        if (l == 2) {
            const uint64_t m = (1ull << s.vertBits) - 1;
            k = ((M21 - (m - (v >> (2 * s.vertBits)))) << 42) | (((v >> s.vertBits) & m) << 21) | (v & m);
        } else if (l == 5) {
            k = ((v >> (s.edgeBits + 4)) << 34) | (v & ((1ull << (s.edgeBits + 4)) - 1));
        } else {
            const int b = l < 2 ? s.faceBits : s.edgeBits;
            k = ((v >> b) << 32) | (v & ((1ull << b) - 1));
        }
        s.key[l][i - (l ? s.end[l - 1] : 0)] = k;
    }
}

__global__ void decodeSelfKernel(int nPT, int nEE, int nPPE, const uint64_t* kPT, const uint64_t* kEE, const uint64_t* uniq, const int* counts,
                                 const int* surfVerts, const int* faces, const int* edges, int* out) {
    int n = nPT + nEE + nPPE;
    CIPC_KERNEL_LOOP(i, n) {
        int c[4];
        if (i < nPT) {
            int svI = (int)(kPT[i] >> 32), sfI = (int)(kPT[i] & 0xffffffffu);
            c[0] = -surfVerts[svI] - 1; c[1] = faces[3 * sfI]; c[2] = faces[3 * sfI + 1]; c[3] = faces[3 * sfI + 2];
        } else if (i < nPT + nEE) {
            uint64_t k = kEE[i - nPT];
            int eI = (int)(k >> 32), eJ = (int)(k & 0xffffffffu);
            c[0] = edges[2 * eI]; c[1] = edges[2 * eI + 1]; c[2] = edges[2 * eJ]; c[3] = edges[2 * eJ + 1];
        } else {
            int j = i - nPT - nEE;
            uint64_t k = uniq[j];
            int v = (int)(M21 - (k >> 42));
            c[0] = -v - 1; c[1] = (int)((k >> 21) & M21); c[2] = (int)(k & M21) - 1; c[3] = -counts[j];
        }
        for (int q = 0; q < 4; ++q) out[4 * i + q] = c[q];
    }
}

__global__ void decodeMollKernel(int n, const uint64_t* k, const int* edges, int* selfEE, int* eeIe) {
    CIPC_KERNEL_LOOP(i, n) {
        uint64_t key = k[i];
        int eI = (int)(key >> 34), eJ = (int)((key >> 4) & ((1u << 30) - 1)), t = (int)(key & 15);
        int e0 = edges[2 * eI], e1 = edges[2 * eI + 1], g0 = edges[2 * eJ], g1 = edges[2 * eJ + 1];
        int c[4] = {0, 0, -1, -1};
        switch (t) {
        case 0: c[0] = -e0 - 1; c[1] = g0; break;
        case 1: c[0] = -e0 - 1; c[1] = g1; break;
        case 2: c[0] = -e0 - 1; c[1] = g0; c[2] = g1; break;
        case 3: c[0] = -e1 - 1; c[1] = g0; break;
        case 4: c[0] = -e1 - 1; c[1] = g1; break;
        case 5: c[0] = -e1 - 1; c[1] = g0; c[2] = g1; break;
        case 6: c[0] = -g0 - 1; c[1] = e0; c[2] = e1; break;
        case 7: c[0] = -g1 - 1; c[1] = e0; c[2] = e1; break;
        default: c[0] = e0; c[1] = e1; c[2] = g0; c[3] = g1; break;
        }
        for (int q = 0; q < 4; ++q) selfEE[4 * i + q] = c[q];
        eeIe[2 * i] = t == 8 ? -1 : eI;
        eeIe[2 * i + 1] = t == 8 ? -1 : eJ;
    }
}

__global__ void groundFlagKernel(int nsv, const int* surfVerts, const double* x, double nx, double ny, double nz, double D, double Hhat, int* flags) {
    CIPC_KERNEL_LOOP(i, nsv) {
        d3 p = ld3(x, surfVerts[i]);
        double dist = nx * p.x + ny * p.y + nz * p.z - D;
        flags[i] = dist * dist < Hhat ? 1 : 0;
    }
}

// ---- step bounds ----
__global__ void groundBoundKernel(int nsv, const int* surfVerts, const double* x, const double* dir, double nx, double ny, double nz, double D,
                                  double slack, double* out) {
    CIPC_KERNEL_LOOP(i, nsv) {
        int v = surfVerts[i];
        d3 p = ld3(x, v), d = ld3(dir, v);
        double r = 1.0;
        double nm = nx * -d.x + ny * -d.y + nz * -d.z;
        if (nm < 0.0) {
            double dist = nx * p.x + ny * p.y + nz * p.z - D;
            double cand = -dist / nm * slack;
            if (cand >= 0.0) r = cand;
        }
        out[i] = r;
    }
}

__global__ void surfMoveKernel(int nsv, const int* surfVerts, const double* dir, double* out) {
    CIPC_KERNEL_LOOP(i, nsv) out[i] = sqrt(sqn(ld3(dir, surfVerts[i])));
}

__global__ void partialCCDKernel(int nPT, int nEE, const uint64_t* ccdPT, const uint64_t* ccdEE, const int* surfVerts, const int* faces,
                                 const int* edges, const double* x, const double* dir, double eta, double* out, int* status) {
    CIPC_KERNEL_LOOP(i, nPT + nEE) {
        double a;
        if (i < nPT) {
            int svI = (int)(ccdPT[i] >> 32), sfI = (int)(ccdPT[i] & 0xffffffffu);
            int p = surfVerts[svI], f0 = faces[3 * sfI], f1 = faces[3 * sfI + 1], f2 = faces[3 * sfI + 2];
            a = pointTriangleCCD(ld3(x, p), ld3(x, f0), ld3(x, f1), ld3(x, f2), -ld3(dir, p), -ld3(dir, f0), -ld3(dir, f1), -ld3(dir, f2), eta, status);
        } else {
            uint64_t k = ccdEE[i - nPT];
            int eI = (int)(k >> 32), eJ = (int)(k & 0xffffffffu);
            int a0 = edges[2 * eI], a1 = edges[2 * eI + 1], b0 = edges[2 * eJ], b1 = edges[2 * eJ + 1];
            a = edgeEdgeCCD(ld3(x, a0), ld3(x, a1), ld3(x, b0), ld3(x, b1), -ld3(dir, a0), -ld3(dir, a1), -ld3(dir, b0), -ld3(dir, b1), eta, status);
        }
        out[i] = a;
    }
}

// Full point-triangle CCD in two kernels (as the edge-edge one below): the
// walk of each surface vertex's swept box emits (vertex, face) pairs that do
// not share a vertex and are not all colliders, then one thread per pair
// runs the additive CCD.
template <class View>
__global__ void fullPTPairsKernel(int nsv, const int* surfVerts, const int* faces, const int* btype, const double* x, const double* dir,
                                  double stepVal, const double* stepPtr, View tree, int2* pairs, int cap, int* count, int* status) {
    __shared__ WalkSmem sm[WALK_WARPS];
    const double step = stepPtr ? *stepPtr : stepVal;
    CIPC_WARP_QUERIES(first, query, nsv) {
        const bool active = query < nsv;
        const int own = surfVerts[active ? query : 0];
        double lo[3], hi[3];
        boxInit(lo, hi);
        sweptAdd(lo, hi, ld3(x, own), ld3(dir, own), step);
        warpQueries(tree, sm[threadIdx.x >> 5], first, active, lo, hi, 0.0, false, status, [&](int svI, int sfI, bool) {
            const int vI = surfVerts[svI];
            const int f0 = faces[3 * sfI], f1 = faces[3 * sfI + 1], f2 = faces[3 * sfI + 2];
            if (isCollider(btype[vI]) && isCollider(btype[f0]) && isCollider(btype[f1]) && isCollider(btype[f2])) return;
            if (vI == f0 || vI == f1 || vI == f2) return;
            cg::coalesced_group g = cg::coalesced_threads();
            int base = 0;
            if (g.thread_rank() == 0) base = atomicAdd(count, (int)g.size());
            const int i = g.shfl(base, 0) + (int)g.thread_rank();
            if (i < cap) pairs[i] = make_int2(vI, sfI);
        });
    }
}

__global__ void fullPTAccdKernel(const int2* pairs, const int* count, int cap, const int* faces, const double* x, const double* dir, double eta,
                                 double* outMin, int* status) {
    const int n = min(*count, cap);
    double best = 1.0;
    CIPC_KERNEL_LOOP(k, n) {
        const int2 pr = pairs[k];
        const int vI = pr.x, f0 = faces[3 * pr.y], f1 = faces[3 * pr.y + 1], f2 = faces[3 * pr.y + 2];
        best = fmin(pointTriangleCCD(ld3(x, vI), ld3(x, f0), ld3(x, f1), ld3(x, f2), -ld3(dir, vI), -ld3(dir, f0), -ld3(dir, f1), -ld3(dir, f2), eta,
                                     status),
                    best);
    }
    best = blockReduce(best, MinOp(), 1.0);
    if (threadIdx.x == 0) atomicMin(reinterpret_cast<unsigned long long*>(outMin), (unsigned long long)__double_as_longlong(best));
}

// Full edge-edge CCD in two kernels, so that the additive CCD runs one
// thread per candidate pair instead of inside the divergent tree walk.  The
// walk emits (query eJ, candidate eI > eJ) as the reference forms its pairs
// (Self_largestFeasibleStepSize_CCD): no two colliders, no shared vertex, and
// swept boxes at the entry step that overlap.  Pairs past `cap` are counted
// but not stored; the caller grows the buffer and runs again.
template <class View>
__global__ void fullEEPairsKernel(int ne, const int* edges, const int* btype, const double* x, const double* dir, const double* treeBoxLo,
                                  const double* treeBoxHi, double eeStepVal, const double* eeStepPtr, View tree, int2* pairs, int cap, int* count,
                                  int* status) {
    __shared__ WalkSmem sm[WALK_WARPS];
    const double eeStep = eeStepPtr ? *eeStepPtr : eeStepVal;
    CIPC_WARP_QUERIES(first, query, ne) {
        const bool active = query < ne;
        const int own = active ? query : 0;
        double qlo[3], qhi[3];
        for (int k = 0; k < 3; ++k) { qlo[k] = treeBoxLo[3 * own + k]; qhi[k] = treeBoxHi[3 * own + k]; }
        const bool large = View::kSplitsBig && active && isLargeBox(qlo, qhi, tree.bigExtent);
        auto pair = [&](int eJ, int eI) {
            int g0 = edges[2 * eJ], g1 = edges[2 * eJ + 1];
            int e0 = edges[2 * eI], e1 = edges[2 * eI + 1];
            if (isCollider(btype[e0]) && isCollider(btype[e1]) && isCollider(btype[g0]) && isCollider(btype[g1])) return;
            if (e0 == g0 || e0 == g1 || e1 == g0 || e1 == g1) return;
            double blo[3], bhi[3], clo[3], chi[3];
            boxInit(blo, bhi);
            sweptAdd(blo, bhi, ld3(x, g0), ld3(dir, g0), eeStep);
            sweptAdd(blo, bhi, ld3(x, g1), ld3(dir, g1), eeStep);
            boxInit(clo, chi);
            sweptAdd(clo, chi, ld3(x, e0), ld3(dir, e0), eeStep);
            sweptAdd(clo, chi, ld3(x, e1), ld3(dir, e1), eeStep);
            if (!overlaps(blo, bhi, clo, chi, 0.0)) return;
            cg::coalesced_group g = cg::coalesced_threads();
            int base = 0;
            if (g.thread_rank() == 0) base = atomicAdd(count, (int)g.size());
            const int i = g.shfl(base, 0) + (int)g.thread_rank();
            if (i < cap) pairs[i] = make_int2(eJ, eI);
        };
        warpQueries(tree, sm[threadIdx.x >> 5], first, active, qlo, qhi, 0.0, large, status, [&](int self, int other, bool fromLarge) {
            if (!fromLarge || large) {
                if (other > self) pair(self, other);
            } else if (other != self) {
                if (other > self) pair(self, other);
                else pair(other, self);
            }
        });
    }
}

// The additive CCD of every stored pair (eI's points first, as the
// reference calls it); the minimum of 1 and every time of impact goes into
// *outMin by an atomic minimum on the bit pattern (non-negative doubles order
// as their bits), so the result does not depend on the order of the pairs.
__global__ void fullEEAccdKernel(const int2* pairs, const int* count, int cap, const int* edges, const double* x, const double* dir, double eta,
                                 double* outMin, int* status) {
    const int n = min(*count, cap);
    double best = 1.0;
    CIPC_KERNEL_LOOP(k, n) {
        const int2 pr = pairs[k];
        const int g0 = edges[2 * pr.x], g1 = edges[2 * pr.x + 1];
        const int e0 = edges[2 * pr.y], e1 = edges[2 * pr.y + 1];
        const d3 q0 = ld3(x, g0), q1 = ld3(x, g1), dq0 = ld3(dir, g0), dq1 = ld3(dir, g1);
        const d3 p0 = ld3(x, e0), p1 = ld3(x, e1), dp0 = ld3(dir, e0), dp1 = ld3(dir, e1);
        best = fmin(edgeEdgeCCD(p0, p1, q0, q1, -dp0, -dp1, -dq0, -dq1, eta, status), best);
    }
    best = blockReduce(best, MinOp(), 1.0);
    if (threadIdx.x == 0) atomicMin(reinterpret_cast<unsigned long long*>(outMin), (unsigned long long)__double_as_longlong(best));
}

__global__ void setDoubleKernel(double* p, double v) { *p = v; }
__global__ void copyCountKernel(const int* count, double* out) { *out = (double)*count; }

// The segment-triangle test of one (face, edge) pair (the filters of
// checkEdgeTriIntersectionIfAny, IPCSolver.cpp:514-542).
__device__ __forceinline__ bool faceEdgeHit(const int* faces, const int* edges, const int* btype, const double* x, int f, int e, double coplanarTol) {
    int f0 = faces[3 * f], f1 = faces[3 * f + 1], f2 = faces[3 * f + 2];
    int e0 = edges[2 * e], e1 = edges[2 * e + 1];
    if (e0 == f0 || e0 == f1 || e0 == f2 || e1 == f0 || e1 == f1 || e1 == f2) return false;
    if (isCollider(btype[e0]) && isCollider(btype[e1]) && isCollider(btype[f0]) && isCollider(btype[f1]) && isCollider(btype[f2])) return false;
    return segTriIntersect(ld3(x, e0), ld3(x, e1), ld3(x, f0), ld3(x, f1), ld3(x, f2), coplanarTol);
}

// Faces against the edge tree.  A large face (one the face tree keeps out of
// its tree) meets only the edge tree's large edges here; its pairs with the
// other edges are tested by largeFaceKernel from the edges' side.
// Intersection test in two kernels, as the full CCD: each face's walk over
// the edge tree emits its candidate (face, edge) pairs, then one thread per
// pair runs the segment-triangle test (faceEdgeHit) and raises the flag.
template <class View>
__global__ void intersectPairsKernel(int nsf, const int* faces, const double* x, View tree, int2* pairs, int cap, int* count, int* status) {
    __shared__ WalkSmem sm[WALK_WARPS];
    CIPC_WARP_QUERIES(first, query, nsf) {
        const bool active = query < nsf;
        double lo[3], hi[3];
        boxInit(lo, hi);
        if (active)
            for (int k = 0; k < 3; ++k) boxAdd(lo, hi, ld3(x, faces[3 * query + k]));
        const bool large = View::kSplitsBig && active && isLargeBox(lo, hi, tree.bigExtent);
        warpQueries(tree, sm[threadIdx.x >> 5], first, active, lo, hi, 0.0, large, status, [&](int f, int e, bool) {
            cg::coalesced_group g = cg::coalesced_threads();
            int base = 0;
            if (g.thread_rank() == 0) base = atomicAdd(count, (int)g.size());
            const int i = g.shfl(base, 0) + (int)g.thread_rank();
            if (i < cap) pairs[i] = make_int2(f, e);
        });
    }
}

__global__ void intersectTestKernel(const int2* pairs, const int* count, int cap, const int* faces, const int* edges, const int* btype,
                                    const double* x, double coplanarTol, int* flag) {
    const int n = min(*count, cap);
    bool hit = false;
    CIPC_KERNEL_LOOP(k, n) {
        const int2 pr = pairs[k];
        if (!hit && faceEdgeHit(faces, edges, btype, x, pr.x, pr.y, coplanarTol)) hit = true;
    }
    if (hit) atomicOr(flag, 1);
}

// The edges that are not large (the edge tree's own) against the large faces
// of the face tree (the last *nbig keys of its sorted order).
__global__ void largeFaceKernel(int ne, const int* faces, const int* edges, const int* btype, const double* x, BvhView faceTree, BvhView edgeTree,
                                double coplanarTol, int* flag) {
    const int nbf = *faceTree.nbig;
    if (nbf == 0) return;
    const int nf = faceTree.nAll - nbf;
    CIPC_KERNEL_LOOP(e, ne) {
        const double* elo = edgeTree.plo + 3 * e;
        const double* ehi = edgeTree.phi + 3 * e;
        if (isLargeBox(elo, ehi, edgeTree.bigExtent)) continue;  // met by the large faces' own queries
        bool hit = false;
        for (int b = 0; b < nbf && !hit; ++b) {
            const int f = (int)(faceTree.keys[nf + b] & 0xffffffffu);
            if (overlaps(faceTree.plo + 3 * f, faceTree.phi + 3 * f, elo, ehi, 0.0) && faceEdgeHit(faces, edges, btype, x, f, e, coplanarTol)) hit = true;
        }
        if (hit) atomicOr(flag, 1);
    }
}

__global__ void groundIntersectKernel(int n, const int* ground, const double* x, double nx, double ny, double nz, double D, int* flag) {
    CIPC_KERNEL_LOOP(i, n) {
        d3 p = ld3(x, ground[i]);
        double dist = nx * p.x + ny * p.y + nz * p.z - D;
        if (dist * dist <= 0.0) atomicOr(flag, 1);
    }
}

// Radix sort of n 64-bit keys on bits [0, endBit), in place
void sortKeys(Ctx& c, uint64_t* keys, int n, int endBit) {
    if (n <= 1) return;
    c.kTmp.reserve(n);
    size_t bytes = 0;
    CIPC_CUDA(cub::DeviceRadixSort::SortKeys(nullptr, bytes, keys, c.kTmp.p, n, 0, endBit, c.s));
    c.sortTmp.reserve(bytes + 16);
    CIPC_CUDA(cub::DeviceRadixSort::SortKeys(c.sortTmp.p, bytes, keys, c.kTmp.p, n, 0, endBit, c.s));
    CIPC_CUDA(cudaMemcpyAsync(keys, c.kTmp.p, sizeof(uint64_t) * n, cudaMemcpyDeviceToDevice, c.s));
}
// CIPC_SETS_APART=1: sort the active sets' lists one by one, as in scenes too large for the joint sort
bool sortSetsApart() {
    static int v = -1;
    if (v < 0) { const char* e = std::getenv("CIPC_SETS_APART"); v = (e && *e == '1') ? 1 : 0; }
    return v == 1;
}

// bits needed for the values 0 .. m - 1
int bitsFor(int m) {
    int b = 1;
    while (b < 31 && (1 << b) < m) ++b;
    return b;
}

}  // namespace

// The spatial-hash tables of one primitive set from its boxes (primLo/Hi).
void buildHash(Ctx& c, DevBvh& t, int n) {
    t.n = n;
    t.hashPairs = 0;
    t.hashBig.reserve(std::max(1, n)); t.hashBigFlag.reserve(std::max(1, n));
    t.hashCount.reserve(std::max(1, n)); t.hashOffset.reserve(std::max(1, n));
    c.counters.reserve(16);
    if (n <= 0) return;
    const double inv = 1.0 / c.P.avgEdge;
    launch(hashCountKernel, blocksFor(n), TB, 0, c.s, n, t.primLo, t.primHi, inv, t.hashCount, t.hashBigFlag);
    size_t bytes = 0;
    cub::DeviceScan::ExclusiveSum(nullptr, bytes, t.hashCount.p, t.hashOffset.p, n, c.s);
    size_t b2 = 0;
    cub::DeviceSelect::Flagged(nullptr, b2, thrust::counting_iterator<int>(0), t.hashBigFlag.p, t.hashBig.p, c.counters.p + 11, n, c.s);
    t.hashTmp.reserve(std::max(bytes, b2) + 16);
    CIPC_CUDA(cub::DeviceScan::ExclusiveSum(t.hashTmp.p, bytes, t.hashCount.p, t.hashOffset.p, n, c.s));
    int last[2];
    CIPC_CUDA(cudaMemcpyAsync(&last[0], t.hashOffset.p + n - 1, sizeof(int), cudaMemcpyDeviceToHost, c.s));
    CIPC_CUDA(cudaMemcpyAsync(&last[1], t.hashCount.p + n - 1, sizeof(int), cudaMemcpyDeviceToHost, c.s));
    hostSync(c);
    const int pairs = last[0] + last[1];
    t.hashPairs = pairs;
    t.hashKey.reserve(std::max(1, pairs)); t.hashKeyAlt.reserve(std::max(1, pairs));
    t.hashPrim.reserve(std::max(1, pairs)); t.hashPrimAlt.reserve(std::max(1, pairs));
    launch(hashEmitKernel, blocksFor(n), TB, 0, c.s, n, t.primLo, t.primHi, inv, (const int*)t.hashOffset, (const int*)t.hashCount, t.hashKeyAlt,
           t.hashPrimAlt);
    if (pairs > 0) {
        size_t b3 = 0;
        cub::DeviceRadixSort::SortPairs(nullptr, b3, t.hashKeyAlt.p, t.hashKey.p, t.hashPrimAlt.p, t.hashPrim.p, pairs, 0, 63, c.s);
        t.hashTmp.reserve(b3 + 16);
        CIPC_CUDA(cub::DeviceRadixSort::SortPairs(t.hashTmp.p, b3, t.hashKeyAlt.p, t.hashKey.p, t.hashPrimAlt.p, t.hashPrim.p, pairs, 0, 63, c.s));
    }
    // the primitives too large for the cells (their ids in order)
    thrust::counting_iterator<int> ids(0);
    size_t b4 = 0;
    cub::DeviceSelect::Flagged(nullptr, b4, ids, t.hashBigFlag.p, t.hashBig.p, c.counters.p + (&t == &c.edgeTree ? 14 : 11), n, c.s);
    t.hashTmp.reserve(b4 + 16);
    CIPC_CUDA(cub::DeviceSelect::Flagged(t.hashTmp.p, b4, ids, t.hashBigFlag.p, t.hashBig.p, c.counters.p + (&t == &c.edgeTree ? 14 : 11), n,
                                         c.s));
    CIPC_CUDA(cudaGetLastError());
}

HashView hview(Ctx& c, const DevBvh& t) {
    return HashView{t.bigExtent, t.n, t.hashPairs, 1.0 / c.P.avgEdge, t.hashKey, t.hashPrim, t.hashBig, c.counters.p + (&t == &c.edgeTree ? 14 : 11),
                    t.primLo, t.primHi};
}

// Both trees over the primitive boxes at x, or swept from x to x - step * d
// (step read from *stepPtr on the device when it is given).
static void buildTrees(Ctx& c, const double* x, const double* d, double step, bool swept, const double* stepPtr) {
    TreePair pair{};
    const int total = c.nsf + c.nse;
    c.treeKeys.reserve(std::max(1, total));
    c.treeSorted.reserve(std::max(1, total));
    c.treeBig.reserve(2);
    // one share of the boxes per block; the same count for both trees, whose
    // Morton kernel reduces the partials
    const int nbBox = std::max(1, std::min(148, (std::max(c.nsf, c.nse) + 255) / 256));
    const bool hash = c.broadPhase == CIPC_BROAD_PHASE_SPATIAL_HASH;
    for (int k = 0; k < 2; ++k) {
        DevBvh& t = k == 0 ? c.faceTree : c.edgeTree;
        const int n = k == 0 ? c.nsf : c.nse, nn = std::max(1, 2 * n - 1);
        t.n = n;
        t.bigExtent = 0.1 * std::sqrt(c.P.bboxDiag2);
        t.primLo.reserve(3 * (size_t)std::max(1, n)); t.primHi.reserve(3 * (size_t)std::max(1, n));
        t.boxPart.reserve(6 * (size_t)nbBox);
        if (!hash) {
            t.links.reserve(std::max(1, n)); t.leafParent.reserve(std::max(1, n)); t.leafPrim.reserve(std::max(1, n)); t.flags.reserve(std::max(1, n));
            t.lo.reserve(3 * (size_t)nn); t.hi.reserve(3 * (size_t)nn);
            t.rec.reserve(16 * (size_t)std::max(1, n - 1));
        }
        t.keys = c.treeSorted.p + (k == 0 ? 0 : c.nsf);
        t.bigCount = c.treeBig.p + k;
        pair.t[k] = TreeBuild{n, k == 0 ? 3 : 2, k == 0 ? c.faces.p : c.edges.p, t.primLo, t.primHi, t.boxPart, c.treeKeys.p + (k == 0 ? 0 : c.nsf),
                              t.keys, t.bigCount, t.links, t.leafParent, t.leafPrim, t.flags, t.lo, t.hi, t.rec};
    }
    launch(primBoxKernel, dim3(nbBox, 2), 256, 0, c.s, pair, x, d, step, stepPtr, swept ? 1 : 0);
    if (hash) {
        buildHash(c, c.faceTree, c.nsf);
        buildHash(c, c.edgeTree, c.nse);
        return;
    }
    const int most = std::max(1, std::max(c.nsf, c.nse));
    launch(mortonKernel, dim3(std::min(blocksFor(most), 148 * 2), 2), TB, 0, c.s, pair, nbBox, c.faceTree.bigExtent);
    // keys are (tree << 63 | code << 32) | index (bit 62: kept out of the tree),
    // written in index order: a stable sort on bits 32-63 gives the order of a
    // sort on the whole key
    if (total > 0) {
        size_t bytes = 0;
        CIPC_CUDA(cub::DeviceRadixSort::SortKeys(nullptr, bytes, c.treeKeys.p, c.treeSorted.p, total, 32, 64, c.s));
        c.sortTmp.reserve(bytes + 16);
        CIPC_CUDA(cub::DeviceRadixSort::SortKeys(c.sortTmp.p, bytes, c.treeKeys.p, c.treeSorted.p, total, 32, 64, c.s));
    }
    launch(karrasKernel, dim3(blocksFor(most), 2), TB, 0, c.s, pair);
    launch(refitKernel, dim3(std::max(1, std::min((most + REFIT - 1) / REFIT, 148 * 8)), 2), REFIT, 0, c.s, pair);
    CIPC_CUDA(cudaGetLastError());
}

// Calls k(view) with the selected backend's view of tree t.
template <class K>
void withView(Ctx& c, const DevBvh& t, K k) {
    if (c.broadPhase == CIPC_BROAD_PHASE_SPATIAL_HASH) k(hview(c, t));
    else k(view(t));
}

static void buildStaticTrees(Ctx& c) { buildTrees(c, c.x, c.x, 0.0, false, nullptr); }

// Ground::calculateActivateSet: the surface vertices within dHat of the
// ground, in order, into c.ground; their count lands in counters[15] (read
// back by the caller).
void groundActiveSetLaunch(Ctx& c) {
    c.ground.reserve(std::max(1, c.nsv));
    c.counts.reserve(std::max(1, c.nsv) + 1);
    c.counters.reserve(16);
    if (c.nsv == 0) {
        CIPC_CUDA(cudaMemsetAsync(c.counters.p + 15, 0, sizeof(int), c.s));
        return;
    }
    launch(groundFlagKernel, blocksFor(c.nsv), TB, 0, c.s, c.nsv, c.surfVerts, c.x, c.P.groundN[0], c.P.groundN[1], c.P.groundN[2], c.P.groundD,
                                                       c.P.Hhat, c.counts);
    size_t bytes = 0;
    cub::DeviceSelect::Flagged(nullptr, bytes, c.surfVerts.p, c.counts.p, c.ground.p, c.counters.p + 15, c.nsv, c.s);
    c.groundTmp.reserve(bytes + 16);
    CIPC_CUDA(cub::DeviceSelect::Flagged(c.groundTmp.p, bytes, c.surfVerts.p, c.counts.p, c.ground.p, c.counters.p + 15, c.nsv, c.s));
}

void groundActiveSet(Ctx& c) {
    groundActiveSetLaunch(c);
    int n = 0;
    CIPC_CUDA(cudaMemcpyAsync(&n, c.counters.p + 15, sizeof(int), cudaMemcpyDeviceToHost, c.s));
    hostSync(c);
    c.nGround = n;
}

// SpatialHash::calculateActivateSet with the LBVH backend, then
// Ground::calculateActivateSet (IPCSolver.cpp:544-556).
void buildCollisionSets(Ctx& c, bool rehash) {
    if (c.P.useBarrier) {
        if (rehash) buildStaticTrees(c);
        double sq = sqrt(c.P.Hhat);
        int caps[6] = {(int)std::max<size_t>(c.ccdPT.cap, 1024), (int)std::max<size_t>(c.kPT.cap, 1024), (int)std::max<size_t>(c.kPPE.cap, 1024),
                       (int)std::max<size_t>(c.ccdEE.cap, 1024), (int)std::max<size_t>(c.kEE.cap, 1024), (int)std::max<size_t>(c.kMoll.cap, 1024)};
        int cnt[6];
        int stWord = 0;
        bool fits = false;
        for (int attempt = 0; attempt < 4; ++attempt) {
            c.ccdPT.reserve(caps[0]); c.kPT.reserve(caps[1]); c.kPPE.reserve(caps[2]);
            c.ccdEE.reserve(caps[3]); c.kEE.reserve(caps[4]); c.kMoll.reserve(caps[5]);
            c.counters.reserve(16);
            CIPC_CUDA(cudaMemsetAsync(c.counters.p, 0, 8 * sizeof(int), c.s));
            Emit eCcdPT{c.ccdPT, caps[0], c.counters.p + 0}, ePT{c.kPT, caps[1], c.counters.p + 1}, ePPE{c.kPPE, caps[2], c.counters.p + 2};
            Emit eCcdEE{c.ccdEE, caps[3], c.counters.p + 3}, eEE{c.kEE, caps[4], c.counters.p + 4}, eMoll{c.kMoll, caps[5], c.counters.p + 5};
            profBegin(c, PROF_ACTIVE);
            if (c.nsv) {
                withView(c, c.faceTree, [&](auto v) {
                    launch(activePTKernel<decltype(v)>, blocksFor(c.nsv), TB, 0, c.s, c.nsv, c.surfVerts, c.faces, c.btype, c.x, v, sq, eCcdPT, c.status);
                });
                launch(activePTClassKernel, 148 * 8, TB, 0, c.s, (const uint64_t*)c.ccdPT.p, (const int*)c.counters.p + 0, caps[0], c.surfVerts, c.faces,
                       c.x, c.P.Hhat, ePT, ePPE, c.status);
            }
            if (c.nse) {
                withView(c, c.edgeTree, [&](auto v) {
                    launch(activeEEKernel<decltype(v)>, blocksFor(c.nse), TB, 0, c.s, c.nse, c.edges, c.btype, c.x, v, sq, eCcdEE, c.status);
                });
                launch(activeEEClassKernel, 148 * 8, TB, 0, c.s, (const uint64_t*)c.ccdEE.p, (const int*)c.counters.p + 3, caps[3], c.edges, c.x, c.rest,
                       c.P.Hhat, eEE, eMoll, ePPE, c.status);
            }
            profEnd(c, PROF_ACTIVE);
            CIPC_CUDA(cudaGetLastError());
            CIPC_CUDA(cudaMemcpyAsync(cnt, c.counters.p, 6 * sizeof(int), cudaMemcpyDeviceToHost, c.s));
            CIPC_CUDA(cudaMemcpyAsync(&stWord, c.status.p, sizeof(int), cudaMemcpyDeviceToHost, c.s));
            hostSync(c);
            fits = true;
            for (int k = 0; k < 6; ++k)
                if (cnt[k] > caps[k]) { caps[k] = cnt[k] + cnt[k] / 2 + 1024; fits = false; }
            if (fits || attempt == 3) break;
            int st = 0;  // clear the capacity bit before retrying (only when another attempt follows)
            CIPC_CUDA(cudaMemcpyAsync(c.status.p, &st, sizeof(int), cudaMemcpyHostToDevice, c.s));
        }
        if (stWord) checkStatus(c, "active set");
        // the counts size the sorts and decodes below: never past what the
        // last launch could write
        if (!fits) throw std::runtime_error("active-set candidate counts exceed their buffers after four attempts");
        c.nCcdPT = cnt[0]; c.nPT = cnt[1]; c.nPPERaw = cnt[2]; c.nCcdEE = cnt[3]; c.nEE = cnt[4]; c.nMoll = cnt[5];
        {
            SetLists lists{};
            uint64_t* keys[6] = {c.ccdPT.p, c.kPT.p, c.kPPE.p, c.ccdEE.p, c.kEE.p, c.kMoll.p};
            long long n = 0;
            for (int k = 0; k < 6; ++k) {
                lists.key[k] = keys[k];
                n += cnt[k];
                lists.end[k] = (int)n;
            }
            // PP/PE fields hold up to nv (c2 + 1); edge pairs of the mollified list 4 type bits
            lists.faceBits = bitsFor(c.nsf); lists.edgeBits = bitsFor(c.nse); lists.vertBits = bitsFor(c.nv + 1);
            lists.tagShift = std::max(std::max(bitsFor(c.nsv) + lists.faceBits, 2 * lists.edgeBits + 4), 3 * lists.vertBits);
            if (lists.tagShift > 61 || n > 0x7fffffff || sortSetsApart()) {
                // over 2^20 vertices three vertex fields and the list's number do not
                // fit 64 bits; the lists together may hold more keys than one alone can
                const int endBit[6] = {32 + bitsFor(c.nsv), 32 + bitsFor(c.nsv), 63, 32 + bitsFor(c.nse), 32 + bitsFor(c.nse),
                                       std::min(64, 34 + bitsFor(c.nse))};
                for (int k = 0; k < 6; ++k) sortKeys(c, keys[k], cnt[k], endBit[k]);
            } else if (n > 1) {
                c.kTmp.reserve(2 * (size_t)n);
                uint64_t *in = c.kTmp.p, *out = c.kTmp.p + n;
                launch(packSetsKernel, blocksFor((int)n), TB, 0, c.s, lists, in);
                size_t bytes = 0;
                CIPC_CUDA(cub::DeviceRadixSort::SortKeys(nullptr, bytes, in, out, (int)n, 0, lists.tagShift + 3, c.s));
                c.sortTmp.reserve(bytes + 16);
                CIPC_CUDA(cub::DeviceRadixSort::SortKeys(c.sortTmp.p, bytes, in, out, (int)n, 0, lists.tagShift + 3, c.s));
                launch(unpackSetsKernel, blocksFor((int)n), TB, 0, c.s, lists, (const uint64_t*)out);
            }
        }
        // merge PP/PE duplicates (multiplicity)
        int nu = 0;
        c.uniq.reserve(std::max(cnt[2], 1));
        c.runs.reserve(std::max(cnt[2], 1));
        if (cnt[2] > 0) {
            size_t bytes = 0;
            cub::DeviceRunLengthEncode::Encode(nullptr, bytes, c.kPPE.p, c.uniq.p, c.runs.p, c.counters.p + 6, cnt[2], c.s);
            c.sortTmp.reserve(bytes + 16);
            CIPC_CUDA(cub::DeviceRunLengthEncode::Encode(c.sortTmp.p, bytes, c.kPPE.p, c.uniq.p, c.runs.p, c.counters.p + 6, cnt[2], c.s));
        } else {
            CIPC_CUDA(cudaMemsetAsync(c.counters.p + 6, 0, sizeof(int), c.s));
        }
        // the ground set is selected meanwhile; both counts come back at once
        groundActiveSetLaunch(c);
        {
            int h[10];
            CIPC_CUDA(cudaMemcpyAsync(h, c.counters.p + 6, 10 * sizeof(int), cudaMemcpyDeviceToHost, c.s));
            hostSync(c);
            nu = h[0];
            c.nGround = h[9];
        }
        c.nPPE = nu;
        c.nSelf = c.nPT + c.nEE + c.nPPE;
        c.selfActive.reserve(4 * std::max(c.nSelf, 1));
        if (c.nSelf)
            launch(decodeSelfKernel, blocksFor(c.nSelf), TB, 0, c.s, c.nPT, c.nEE, c.nPPE, c.kPT, c.kEE, c.uniq, c.runs, c.surfVerts, c.faces, c.edges,
                                                                 c.selfActive);
        c.selfEE.reserve(4 * std::max(c.nMoll, 1));
        c.eeIe.reserve(2 * std::max(c.nMoll, 1));
        if (c.nMoll) launch(decodeMollKernel, blocksFor(c.nMoll), TB, 0, c.s, c.nMoll, c.kMoll, c.edges, c.selfEE, c.eeIe);
        CIPC_CUDA(cudaGetLastError());
    } else {
        groundActiveSet(c);
    }
}

// the candidate-pair buffer shared by the intersection test and the full CCD
static int ccdPairsReserve(Ctx& c);

bool isIntersected(Ctx& c) {
    c.counters.reserve(16);
    CIPC_CUDA(cudaMemsetAsync(c.counters.p + 7, 0, sizeof(int), c.s));
    if (c.nGround)
        launch(groundIntersectKernel, blocksFor(c.nGround), TB, 0, c.s, c.nGround, c.ground, c.x, c.P.groundN[0], c.P.groundN[1], c.P.groundN[2],
                                                                   c.P.groundD, c.counters.p + 7);
    if (c.nse && c.nsf && c.broadPhase == CIPC_BROAD_PHASE_LBVH)
        launch(largeFaceKernel, blocksFor(c.nse), TB, 0, c.s, c.nse, c.faces, c.edges, c.btype, c.x, view(c.faceTree), view(c.edgeTree), c.coplanarTol,
               c.counters.p + 7);
    for (;;) {
        int cap = 0;
        if (c.nsf) {
            cap = ccdPairsReserve(c);
            CIPC_CUDA(cudaMemsetAsync(c.ccdPairCount.p, 0, sizeof(int), c.s));
            withView(c, c.edgeTree, [&](auto v) {
                launch(intersectPairsKernel<decltype(v)>, blocksFor(c.nsf), TB, 0, c.s, c.nsf, c.faces, c.x, v, c.ccdPairs.p, cap, c.ccdPairCount.p,
                       c.status);
            });
            launch(intersectTestKernel, 148 * 8, TB, 0, c.s, (const int2*)c.ccdPairs.p, (const int*)c.ccdPairCount.p, cap, c.faces, c.edges, c.btype,
                   c.x, c.coplanarTol, c.counters.p + 7);
        }
        int h[3] = {0, 0, 0};
        CIPC_CUDA(cudaMemcpyAsync(&h[0], c.counters.p + 7, sizeof(int), cudaMemcpyDeviceToHost, c.s));
        CIPC_CUDA(cudaMemcpyAsync(&h[1], c.status.p, sizeof(int), cudaMemcpyDeviceToHost, c.s));
        if (c.nsf) CIPC_CUDA(cudaMemcpyAsync(&h[2], c.ccdPairCount.p, sizeof(int), cudaMemcpyDeviceToHost, c.s));
        hostSync(c);
        if (h[1]) checkStatus(c, "intersection test");
        // a hit among the stored pairs stands; otherwise every pair must have been tested
        if (h[0] != 0 || h[2] <= cap) return h[0] != 0;
        c.ccdPairs.reserve((size_t)h[2]);
    }
}

// Rebuild the static trees at the current positions (sh.build in the line search).
void rebuildTrees(Ctx& c) { buildStaticTrees(c); }

double groundStepBound(Ctx& c) {
    if (c.nsv == 0) return 1.0;
    c.energyBuf.reserve(std::max(c.nsv, 1));
    launch(groundBoundKernel, blocksFor(c.nsv), TB, 0, c.s, c.nsv, c.surfVerts, c.x, c.dir, c.P.groundN[0], c.P.groundN[1], c.P.groundN[2], c.P.groundD,
                                                        0.8, c.energyBuf);
    return deviceMin(c, c.energyBuf, c.nsv, 1e308);
}

double partialCCD(Ctx& c, double alpha) {
    int n = c.nCcdPT + c.nCcdEE;
    if (n == 0) return alpha;
    c.energyBuf.reserve(n);
    launch(partialCCDKernel, blocksFor(n), TB, 0, c.s, c.nCcdPT, c.nCcdEE, c.ccdPT, c.ccdEE, c.surfVerts, c.faces, c.edges, c.x, c.dir, 1.0 - 0.8,
                                                  c.energyBuf, c.status);
    double mn = deviceMin(c, c.energyBuf, n, 1e308);
    checkStatus(c, "partial CCD");
    return std::min(alpha, mn);
}

double cflBound(Ctx& c) {
    if (c.nsv == 0) return 1.0;
    c.energyBuf.reserve(c.nsv);
    launch(surfMoveKernel, blocksFor(c.nsv), TB, 0, c.s, c.nsv, c.surfVerts, c.dir, c.energyBuf);
    double mx = std::max(0.0, deviceMax(c, c.energyBuf, c.nsv));
    return mx > 0.0 ? sqrt(c.P.Hhat) / (mx * 2.0) : 1.0;
}

// The full edge-edge CCD over the swept edge tree (built with the entry
// step stepVal, or *stepPtr when given): candidate pairs, then one thread per
// pair; min(1, every time of impact) into the device scalar *outMin.  The
// pair count stays on the device (ccdPairCount): a caller that finds it above
// the buffer's capacity grows the buffer and runs again.
// First size of the pair buffer: 8 pairs per query, or CIPC_CCD_PAIRS_INITIAL
// pairs (a small value exercises the grow-and-rerun path).
static size_t ccdPairsInitial(const Ctx& c) {
    static long long v = -2;
    if (v == -2) { const char* e = std::getenv("CIPC_CCD_PAIRS_INITIAL"); v = e ? std::atoll(e) : -1; }
    return v > 0 ? (size_t)v : std::max<size_t>(1024, 8 * (size_t)std::max(c.nse, c.nsv));
}
static int ccdPairsReserve(Ctx& c) {
    c.ccdPairCount.reserve(2);
    c.ccdPairs.reserve(ccdPairsInitial(c));
    return (int)std::min<size_t>(c.ccdPairs.cap, 0x7fffffff);
}
static void fullEEDevice(Ctx& c, const double* d, double stepVal, const double* stepPtr, double* outMin) {
    const int cap = ccdPairsReserve(c);
    CIPC_CUDA(cudaMemsetAsync(c.ccdPairCount.p + 1, 0, sizeof(int), c.s));
    launch(setDoubleKernel, 1, 1, 0, c.s, outMin, 1.0);
    withView(c, c.edgeTree, [&](auto v) {
        launch(fullEEPairsKernel<decltype(v)>, blocksFor(c.nse), TB, 0, c.s, c.nse, c.edges, c.btype, c.x, d, c.edgeTree.primLo, c.edgeTree.primHi,
               stepVal, stepPtr, v, c.ccdPairs.p, cap, c.ccdPairCount.p + 1, c.status);
    });
    launch(fullEEAccdKernel, 148 * 8, TB, 0, c.s, (const int2*)c.ccdPairs.p, (const int*)c.ccdPairCount.p + 1, cap, c.edges, c.x, d, 1.0 - 0.8,
           outMin, c.status);
}
// The same for the point-triangle pairs (surface vertices against the swept
// face tree), count in ccdPairCount[0].
static void fullPTDevice(Ctx& c, const double* d, double stepVal, const double* stepPtr, double* outMin) {
    const int cap = ccdPairsReserve(c);
    CIPC_CUDA(cudaMemsetAsync(c.ccdPairCount.p, 0, sizeof(int), c.s));
    launch(setDoubleKernel, 1, 1, 0, c.s, outMin, 1.0);
    withView(c, c.faceTree, [&](auto v) {
        launch(fullPTPairsKernel<decltype(v)>, blocksFor(c.nsv), TB, 0, c.s, c.nsv, c.surfVerts, c.faces, c.btype, c.x, d, stepVal, stepPtr, v,
               c.ccdPairs.p, cap, c.ccdPairCount.p, c.status);
    });
    launch(fullPTAccdKernel, 148 * 8, TB, 0, c.s, (const int2*)c.ccdPairs.p, (const int*)c.ccdPairCount.p, cap, c.faces, c.x, d, 1.0 - 0.8, outMin,
           c.status);
}

// Swept build with the entry step, then Self_largestFeasibleStepSize_CCD.
double fullCCDDir(Ctx& c, const double* d, double alpha) {
    double step = alpha;
    buildTrees(c, c.x, d, step, true, nullptr);
    c.stepScal.reserve(16);
    double* sm = c.stepScal.p + 12;  // [12] minimum, [13] pair count
    // one pass (point-triangle or edge-edge) with the host's entry step; a
    // pair buffer that was too small is grown and the pass runs again
    auto pass = [&](bool pt) {
        for (;;) {
            profBegin(c, PROF_FULLCCD);
            if (pt) fullPTDevice(c, d, step, nullptr, sm);
            else fullEEDevice(c, d, step, nullptr, sm);
            profEnd(c, PROF_FULLCCD);
            launch(copyCountKernel, 1, 1, 0, c.s, (const int*)c.ccdPairCount.p + (pt ? 0 : 1), sm + 1);
            double h[2];
            CIPC_CUDA(cudaMemcpyAsync(h, sm, sizeof(h), cudaMemcpyDeviceToHost, c.s));
            hostSync(c);
            if (h[1] <= (double)c.ccdPairs.cap) { step = std::min(step, h[0]); return; }
            c.ccdPairs.reserve((size_t)h[1]);
        }
    };
    if (c.nsv) pass(true);
    if (c.nse) pass(false);
    checkStatus(c, "full CCD");
    return step;
}

double fullCCD(Ctx& c, double alpha) { return fullCCDDir(c, c.dir, alpha); }

namespace {
// Scalars of the chained step bounds (stepBoundsDevice), one thread each.
// s: 0 ground min, 1 partial-CCD min, 2 max surface move, 3 entry step,
// 4 full point-triangle min, 5 edge-edge entry step, 6 full edge-edge min,
// 7 merged step, 8 status word, 9 and 10 point-triangle and edge-edge
// CCD pair counts.
__global__ void stepEntryKernel(double* s, int nsv) {
    double a = nsv ? s[0] : 1.0;
    a = fmin(1.0, a);
    if (a <= 0) a = 1;
    s[3] = a;
    s[5] = a;
}
__global__ void stepEeEntryKernel(double* s) { s[5] = fmin(s[3], s[4]); }
__global__ void stepMergeKernel(double* s, int nsv, int nse, int nPartial, int barrier, double sqrtHhat, const int* status) {
    const double alpha = s[3];
    double a = alpha;
    if (barrier) {
        const double partial = nPartial ? fmin(alpha, s[1]) : alpha;
        const double mx = nsv ? fmax(0.0, s[2]) : 0.0;
        const double aCFL = mx > 0.0 ? sqrtHhat / (mx * 2.0) : 1.0;
        double full = alpha;
        if (nsv) full = fmin(full, s[4]);
        if (nse) full = fmin(full, s[6]);
        a = fmin(a, aCFL);
        if (partial > 2.0 * aCFL) {
            a = fmin(partial, full);
            a = fmax(a, aCFL);
        }
        s[1] = partial; s[2] = aCFL; s[6] = full;
    }
    s[7] = a;
    s[8] = (double)*status;
}
}  // namespace

// The step bound of one Newton iteration (IPCSolver.cpp:943-990) without
// host round trips between its stages: the ground bound gives the entry step,
// the partial CCD, CFL bound and the swept full CCD (entry step read on the
// device, the edge-edge pass starting from the point-triangle result) write
// device scalars, and one kernel applies the merge rule.  One read-back.
double stepBoundsDevice(Ctx& c) {
    c.stepScal.reserve(16);
    double* s = c.stepScal.p;
    const int nPartial = c.nCcdPT + c.nCcdEE;
    c.energyBuf.reserve(std::max(std::max(std::max(c.nsv, c.nse), nPartial), 1));
    if (c.nsv) {
        launch(groundBoundKernel, blocksFor(c.nsv), TB, 0, c.s, c.nsv, c.surfVerts, c.x, c.dir, c.P.groundN[0], c.P.groundN[1], c.P.groundN[2],
               c.P.groundD, 0.8, c.energyBuf);
        deviceMinTo(c, c.energyBuf, c.nsv, s + 0);
    }
    launch(stepEntryKernel, 1, 1, 0, c.s, s, c.nsv);
    if (c.P.useBarrier) {
        if (nPartial) {
            launch(partialCCDKernel, blocksFor(nPartial), TB, 0, c.s, c.nCcdPT, c.nCcdEE, c.ccdPT, c.ccdEE, c.surfVerts, c.faces, c.edges, c.x, c.dir,
                   1.0 - 0.8, c.energyBuf, c.status);
            deviceMinTo(c, c.energyBuf, nPartial, s + 1);
        }
        if (c.nsv) {
            launch(surfMoveKernel, blocksFor(c.nsv), TB, 0, c.s, c.nsv, c.surfVerts, c.dir, c.energyBuf);
            deviceMaxTo(c, c.energyBuf, c.nsv, s + 2);
        }
        buildTrees(c, c.x, c.dir, 0.0, true, s + 3);
        ccdPairsReserve(c);
        CIPC_CUDA(cudaMemsetAsync(c.ccdPairCount.p, 0, 2 * sizeof(int), c.s));
        if (c.nsv) {
            profBegin(c, PROF_FULLCCD);
            fullPTDevice(c, c.dir, 0.0, s + 3, s + 4);
            profEnd(c, PROF_FULLCCD);
            launch(stepEeEntryKernel, 1, 1, 0, c.s, s);
        }
        if (c.nse) {
            profBegin(c, PROF_FULLCCD);
            fullEEDevice(c, c.dir, 0.0, s + 5, s + 6);
            profEnd(c, PROF_FULLCCD);
        }
        launch(copyCountKernel, 1, 1, 0, c.s, (const int*)c.ccdPairCount.p, s + 9);
        launch(copyCountKernel, 1, 1, 0, c.s, (const int*)c.ccdPairCount.p + 1, s + 10);
    }
    launch(stepMergeKernel, 1, 1, 0, c.s, s, c.nsv, c.nse, nPartial, c.P.useBarrier ? 1 : 0, std::sqrt(c.P.Hhat), (const int*)c.status.p);
    CIPC_CUDA(cudaGetLastError());
    double h[11];
    CIPC_CUDA(cudaMemcpyAsync(h, s, sizeof(h), cudaMemcpyDeviceToHost, c.s));
    hostSync(c);
    if (h[8] != 0.0) checkStatus(c, "step bounds");
    const double pairs = std::max(h[9], h[10]);
    if (c.P.useBarrier && pairs > (double)c.ccdPairs.cap) {
        // more CCD candidates than the pair buffer holds: grow it and
        // recompute the bounds (every input is unchanged)
        c.ccdPairs.reserve((size_t)pairs);
        return stepBoundsDevice(c);
    }
    return h[7];
}


// Additive CCD on a batch of independent candidate pairs (the per-pair time
// of impact of Self_largestFeasibleStepSize, ContactMechanics.cpp:3704-3752,
// AdditiveCCD.cpp:221-329): kind 0 point-triangle (point, t0, t1, t2), kind 1
// edge-edge (a0, a1, b0, b1); 12 positions and 12 displacements per pair.
namespace {
__global__ void accdBatchKernel(int n, const int* kind, const double* p, const double* d, double eta, double* toi, int* status) {
    CIPC_KERNEL_LOOP(k, n) {
        const double* q = p + 12 * (size_t)k;
        const double* m = d + 12 * (size_t)k;
        d3 x[4], v[4];
        for (int a = 0; a < 4; ++a) {
            x[a] = mk(q[3 * a], q[3 * a + 1], q[3 * a + 2]);
            v[a] = mk(m[3 * a], m[3 * a + 1], m[3 * a + 2]);
        }
        toi[k] = kind[k] == 0 ? pointTriangleCCD(x[0], x[1], x[2], x[3], v[0], v[1], v[2], v[3], eta, status)
                              : edgeEdgeCCD(x[0], x[1], x[2], x[3], v[0], v[1], v[2], v[3], eta, status);
    }
}
}  // namespace

void accdBatch(int n, const int* kind, const double* p, const double* d, double eta, double* toi) {
    DevSlab slab;
    DBuf<int> dk, st;
    DBuf<double> dp, dd, dt;
    slab.lendAll([&](DevSlab& s) {
        s.lend(dp, 12 * (size_t)n);
        s.lend(dd, 12 * (size_t)n);
        s.lend(dt, n);
        s.lend(dk, n);
        s.lend(st, 1);
    });
    CIPC_CUDA(cudaMemcpy(dk.p, kind, sizeof(int) * n, cudaMemcpyHostToDevice));
    CIPC_CUDA(cudaMemcpy(dp.p, p, sizeof(double) * 12 * (size_t)n, cudaMemcpyHostToDevice));
    CIPC_CUDA(cudaMemcpy(dd.p, d, sizeof(double) * 12 * (size_t)n, cudaMemcpyHostToDevice));
    CIPC_CUDA(cudaMemset(st.p, 0, sizeof(int)));
    launch(accdBatchKernel, blocksFor(n), TB, 0, (cudaStream_t)0, n, (const int*)dk.p, (const double*)dp.p, (const double*)dd.p, eta,
           dt.p, st.p);
    CIPC_CUDA(cudaGetLastError());
    int hs = 0;
    CIPC_CUDA(cudaMemcpy(toi, dt.p, sizeof(double) * n, cudaMemcpyDeviceToHost));
    CIPC_CUDA(cudaMemcpy(&hs, st.p, sizeof(int), cudaMemcpyDeviceToHost));
    if (hs & CIPC_ST_CCD_CAP) throw std::runtime_error("a pair reached the CCD iteration cap");
}

}  // namespace cipc
