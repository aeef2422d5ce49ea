// bvh_gpu.cu - binned-SAH BVH build on the device, with the split rules of the host builder
// (bvh_build.cpp: 32 bins over the centroid bounds, the same SAH sweep and leaf tests, median
// split when no axis can be binned), and the four-child collapse.  Replaces Embree's BVH build
// inside World::freeze / rtcCommit (src/RayTracing/World.h:543-550).
//
// Three phases, with the counts they hand on kept on the device (the host waits once per few
// levels, once after the subtrees and once after the collapse):
//  * levels over the nodes of more than kMid triangles: bins, split, partition (with the children's
//    boxes), one launch each; a warp takes a run of positions and collects in shared memory and
//    registers, with one set of global atomics per node it meets;
//  * the subtrees of at most kMid triangles, one block each, level by level in shared memory, one
//    warp per node;
//  * the four-child collapse, one launch per level, nodes in breadth-first order.
// Min/max are exact in any order, so every split decision is the host's; only the median fallback
// (no binnable axis) splits by array order, which may differ.
#include <cuda_runtime.h>

#include <algorithm>
#include <chrono>
#include <cstring>
#include <functional>
#include <string>
#include <vector>

#include "bvh_build.h"
#include "tr_internal.h"

namespace trh {
using tri::CudaError;
namespace {

constexpr int kBins = 32;
constexpr uint32_t kMid = 512;          // subtrees finished by one block
constexpr int kMidThreads = 128;
constexpr float kBig = 3.4e38f;
constexpr uint32_t kWarpRun = 128;      // positions per warp in the level kernels
constexpr uint32_t kMaxLevels = 64;     // four-child levels (twice what the traversal stack takes)
constexpr unsigned kAll = 0xffffffffu;

// floats as unsigned integers of the same order, so min / max reduce with integer operations
__device__ __forceinline__ uint32_t key_of(float f) {
    const uint32_t u = __float_as_uint(f);
    return u ^ ((uint32_t)((int32_t)u >> 31) | 0x80000000u);
}
__device__ __forceinline__ float of_key(uint32_t k) {
    return __uint_as_float(k ^ ((uint32_t)((int32_t)~k >> 31) | 0x80000000u));
}
__device__ __forceinline__ int bin_of(float c, float lo, float scale) {
    const int b = (int)((c - lo) * scale);
    return b < 0 ? 0 : (b >= kBins ? kBins - 1 : b);
}
__device__ __forceinline__ float area(const float* lo, const float* hi) {
    const float dx = hi[0] - lo[0], dy = hi[1] - lo[1], dz = hi[2] - lo[2];
    if (dx < 0.f) return 0.f;
    return 2.f * (dx * dy + dy * dz + dz * dx);
}
// a triangle's centroid, the centre of its box
__device__ __forceinline__ float centre(float lo, float hi) { return 0.5f * (lo + hi); }

struct Box { float lo[3], hi[3]; };
__device__ __forceinline__ void clear(Box& b) {
#pragma unroll
    for (int k = 0; k < 3; ++k) { b.lo[k] = kBig; b.hi[k] = -kBig; }
}
__device__ __forceinline__ void grow(Box& b, float4 lo, float4 hi) {
    b.lo[0] = fminf(b.lo[0], lo.x); b.lo[1] = fminf(b.lo[1], lo.y); b.lo[2] = fminf(b.lo[2], lo.z);
    b.hi[0] = fmaxf(b.hi[0], hi.x); b.hi[1] = fmaxf(b.hi[1], hi.y); b.hi[2] = fmaxf(b.hi[2], hi.z);
}
// the box over all lanes, in every lane
__device__ __forceinline__ void warp_union(Box& b) {
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        b.lo[k] = of_key(__reduce_min_sync(kAll, key_of(b.lo[k])));
        b.hi[k] = of_key(__reduce_max_sync(kAll, key_of(b.hi[k])));
    }
}

enum { kNodes = 0, kError = 1, kDepth = 2, kNumMid = 3, kActive = 4 /* two, by level parity */, kLeaves = 6,
       kVertex = 8 /* six keys: vertex box */, kLevel = 16 /* four-child nodes per level */, kCounters = kLevel + kMaxLevels + 2 };

struct Dev {
    float4 *plo, *phi;                 // per triangle id: bounds
    uint32_t* ids[2];                  // per position (ping-pong): triangle id
    int32_t* pn[2];                    // per position: active node of the level, -1 when done
    uint4* act[2];                     // active nodes: first, count, out index, depth
    uint32_t* nc[2];                   // per active node, by level parity: keys of its box and centroid box (12)
    uint32_t* bb;                      // per active node: bins [3][7][kBins]: box keys, count
    int32_t* d_ax;                     // split axis, -1: median split by position
    int32_t* d_split;                  // last bin of the left child
    uint32_t* d_nl;                    // triangles of the left child
    float2* d_scale;                   // centroid box's lower end and kBins / its extent on the axis
    int32_t* d_child;                  // [2] next-level active index per child, -1 when at most kMid
    uint2* cursor;                     // next free position of the left and right child
    uint4* mid;                        // subtree roots: first, count, out index, depth
    BinNode* nodes;
    uint32_t* counters;
    uint32_t max_leaf;
};

__device__ __forceinline__ uint32_t empty_key(int k) { return k % 6 < 3 ? 0xffffffffu : 0u; }

// Triangle and vertex boxes, the input check, the root's box and centroid box.
__global__ void __launch_bounds__(256) k_prims(const float* __restrict__ v, uint32_t nv, const uint32_t* __restrict__ t,
                                               uint32_t nt, Dev d) {
    Box nb, cb, vb;
    clear(nb); clear(cb); clear(vb);
    bool any_bad = false;
    const uint32_t stride = gridDim.x * blockDim.x, i0 = blockIdx.x * blockDim.x + threadIdx.x;
    for (uint32_t i = i0; i < nt; i += stride) {
        float lo[3] = {kBig, kBig, kBig}, hi[3] = {-kBig, -kBig, -kBig};
        bool bad = false;
        for (int j = 0; j < 3 && !bad; ++j) {
            const uint32_t vi = t[3 * (size_t)i + j];
            if (vi >= nv) { bad = true; break; }
            for (int k = 0; k < 3; ++k) {
                const float p = v[3 * (size_t)vi + k];
                if (!isfinite(p)) bad = true;
                lo[k] = fminf(lo[k], p);
                hi[k] = fmaxf(hi[k], p);
            }
        }
        any_bad = any_bad || bad;
        const float4 l = make_float4(lo[0], lo[1], lo[2], 0.f), h = make_float4(hi[0], hi[1], hi[2], 0.f);
        d.plo[i] = l;
        d.phi[i] = h;
        d.ids[0][i] = i;
        d.pn[0][i] = 0;
        grow(nb, l, h);
        const float4 c = make_float4(centre(l.x, h.x), centre(l.y, h.y), centre(l.z, h.z), 0.f);
        grow(cb, c, c);
    }
    for (uint32_t i = i0; i < nv; i += stride) {
        const float4 p = make_float4(v[3 * (size_t)i], v[3 * (size_t)i + 1], v[3 * (size_t)i + 2], 0.f);
        grow(vb, p, p);
    }
    if (any_bad) atomicOr(&d.counters[kError], 1u);
    // the three boxes over the block, then one set of atomics
    __shared__ uint32_t keys[18];
    if (threadIdx.x < 18) keys[threadIdx.x] = empty_key((int)(threadIdx.x % 6u));
    __syncthreads();
    warp_union(nb); warp_union(cb); warp_union(vb);
    if ((threadIdx.x & 31u) == 0) {
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            atomicMin(&keys[k], key_of(nb.lo[k])); atomicMax(&keys[3 + k], key_of(nb.hi[k]));
            atomicMin(&keys[6 + k], key_of(cb.lo[k])); atomicMax(&keys[9 + k], key_of(cb.hi[k]));
            atomicMin(&keys[12 + k], key_of(vb.lo[k])); atomicMax(&keys[15 + k], key_of(vb.hi[k]));
        }
    }
    __syncthreads();
    if (threadIdx.x < 18) {
        uint32_t* to = threadIdx.x < 12 ? d.nc[0] + threadIdx.x : d.counters + kVertex + threadIdx.x - 12;
        if (threadIdx.x % 6u < 3) atomicMin(to, keys[threadIdx.x]);
        else atomicMax(to, keys[threadIdx.x]);
    }
}

// Empty accumulators for `na` nodes, and the root as the first node.
__global__ void k_start(Dev d, uint32_t na, uint32_t nt) {
    const uint32_t stride = gridDim.x * blockDim.x, i0 = blockIdx.x * blockDim.x + threadIdx.x;
    for (uint32_t i = i0; i < na * 12u; i += stride) { d.nc[0][i] = empty_key((int)(i % 6u)); d.nc[1][i] = empty_key((int)(i % 6u)); }
    for (uint32_t i = i0; i < na * 21u * kBins; i += stride) {
        const uint32_t f = (i / kBins) % 7u;
        d.bb[i] = f < 3u ? 0xffffffffu : 0u;
    }
    for (uint32_t i = i0; i < (uint32_t)kCounters; i += stride) {
        uint32_t c = 0;
        if (i == kNodes) c = 1;
        if (i == kActive) c = nt > kMid ? 1u : 0u;
        if (i == kNumMid) c = nt > kMid ? 0u : 1u;
        if (i >= kVertex && i < kVertex + 3) c = 0xffffffffu;
        if (i == kLevel) c = 1;
        d.counters[i] = c;
    }
    if (i0 == 0) (nt > kMid ? d.act[0] : d.mid)[0] = make_uint4(0, nt, 0, 0);
}

// A warp's bins in shared memory, [axis][box keys, count][bin], and one lane's view of them: bin
// `lane` of the three axes.
constexpr uint32_t kBinWords = 21u * kBins;
struct LaneBins { Box box[3]; uint32_t count[3]; };
__device__ __forceinline__ void clear_bins(uint32_t* bins, uint32_t lane) {
#pragma unroll
    for (uint32_t k = 0; k < 21u; ++k) bins[k * kBins + lane] = k % 7u < 3u ? 0xffffffffu : 0u;
}
// one triangle per calling lane into bin b of axis a
__device__ __forceinline__ void add(uint32_t* bins, uint32_t a, uint32_t b, const uint32_t* lo, const uint32_t* hi) {
    uint32_t* at = bins + 7u * a * kBins + b;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        atomicMin(at + k * kBins, lo[k]);
        atomicMax(at + (3 + k) * kBins, hi[k]);
    }
    atomicAdd(at + 6 * kBins, 1u);
}
__device__ __forceinline__ LaneBins lane_bins(const uint32_t* bins, uint32_t lane) {
    LaneBins B;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        clear(B.box[a]);
        B.count[a] = bins[(7 * a + 6) * kBins + lane];
        if (B.count[a]) {
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                B.box[a].lo[k] = of_key(bins[(7 * a + k) * kBins + lane]);
                B.box[a].hi[k] = of_key(bins[(7 * a + 3 + k) * kBins + lane]);
            }
        }
    }
    return B;
}

// The SAH sweep over a warp's bins: the cheapest split in (axis, bin) order, as the host's strict
// comparison picks it.  The right-hand and left-hand boxes and counts are suffix and prefix scans
// over the lanes (min / max and integer sums: exact).  usable: axes with a centroid extent.
struct Split { float cost; int axis, bin; uint32_t left; };
__device__ __forceinline__ Split sweep(const LaneBins& B, uint32_t usable, int lane) {
    float best = 3.4e38f;
    int bidx = 0x7fffffff;                             // axis * kBins + bin of the best split
    uint32_t lcnt_at[3];
#pragma unroll
    for (int ax = 0; ax < 3; ++ax) {
        lcnt_at[ax] = 0;
        if (!((usable >> ax) & 1u)) continue;
        Box r = B.box[ax], l = B.box[ax];
        uint32_t rc = B.count[ax], lc = rc;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            Box t;
#pragma unroll
            for (int k = 0; k < 3; ++k) {              // suffix: bins lane .. 31
                t.lo[k] = __shfl_down_sync(kAll, r.lo[k], off);
                t.hi[k] = __shfl_down_sync(kAll, r.hi[k], off);
            }
            uint32_t tc = __shfl_down_sync(kAll, rc, off);
            if (lane + off < 32) {
#pragma unroll
                for (int k = 0; k < 3; ++k) { r.lo[k] = fminf(r.lo[k], t.lo[k]); r.hi[k] = fmaxf(r.hi[k], t.hi[k]); }
                rc += tc;
            }
#pragma unroll
            for (int k = 0; k < 3; ++k) {              // prefix: bins 0 .. lane
                t.lo[k] = __shfl_up_sync(kAll, l.lo[k], off);
                t.hi[k] = __shfl_up_sync(kAll, l.hi[k], off);
            }
            tc = __shfl_up_sync(kAll, lc, off);
            if (lane >= off) {
#pragma unroll
                for (int k = 0; k < 3; ++k) { l.lo[k] = fminf(l.lo[k], t.lo[k]); l.hi[k] = fmaxf(l.hi[k], t.hi[k]); }
                lc += tc;
            }
        }
        // split after bin `lane`: left = bins 0..lane, right = bins lane+1..31
        const float ra_next = __shfl_down_sync(kAll, area(r.lo, r.hi), 1);
        const uint32_t rc_next = __shfl_down_sync(kAll, rc, 1);
        lcnt_at[ax] = lc;
        if (lane < kBins - 1 && lc != 0 && rc_next != 0) {
            const float cost = area(l.lo, l.hi) * (float)lc + ra_next * (float)rc_next;
            if (cost < best) { best = cost; bidx = ax * kBins + lane; }
        }
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        const float ob = __shfl_xor_sync(kAll, best, off);
        const int oi = __shfl_xor_sync(kAll, bidx, off);
        if (ob < best || (ob == best && oi < bidx)) { best = ob; bidx = oi; }
    }
    Split s{best, -1, -1, 0};
    if (bidx != 0x7fffffff) { s.axis = bidx / kBins; s.bin = bidx % kBins; }
#pragma unroll
    for (int ax = 0; ax < 3; ++ax) {
        const uint32_t v = __shfl_sync(kAll, lcnt_at[ax], s.bin < 0 ? 0 : s.bin);
        if (ax == s.axis) s.left = v;
    }
    return s;
}

// Bins of every active node.  A warp adds its run's triangles to bins of its own in shared memory (a
// lane per triangle, integer min / max: lanes meet only in the same bin) and those to the node's when
// the node changes: 18 us per level of 328 k triangles (with each lane scanning the run for its own bin in
// registers 33 us, with bins shared by a block and float atomics 58 us).
__global__ void __launch_bounds__(256) k_bin(Dev d, int cur, uint32_t nt) {
    if (blockIdx.x == 0 && threadIdx.x == 0) d.counters[kActive + (cur ^ 1)] = 0u;   // counted by this level's k_split
    if (d.counters[kActive + cur] == 0u) return;
    __shared__ uint32_t all_bins[8][kBinWords];
    const uint32_t lane = threadIdx.x & 31u;
    uint32_t* bins = all_bins[threadIdx.x >> 5];
    const uint32_t p0 = ((blockIdx.x * blockDim.x + threadIdx.x) >> 5) * kWarpRun, p1 = min(nt, p0 + kWarpRun);
    clear_bins(bins, lane);
    __syncwarp();
    int32_t node = -1;
    auto flush = [&]() {
        __syncwarp();
        uint32_t* bb = d.bb + (size_t)node * kBinWords + lane;
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            const uint32_t c = bins[(7 * a + 6) * kBins + lane];
            if (c) {
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    atomicMin(bb + (7 * a + k) * kBins, bins[(7 * a + k) * kBins + lane]);
                    atomicMax(bb + (7 * a + 3 + k) * kBins, bins[(7 * a + 3 + k) * kBins + lane]);
                }
                atomicAdd(bb + (7 * a + 6) * kBins, c);
            }
        }
        __syncwarp();
        clear_bins(bins, lane);
        __syncwarp();
    };
    for (uint32_t b = p0; b < p1; b += 32u) {
        const uint32_t i = b + lane;
        const int32_t n = i < p1 ? d.pn[cur][i] : -1;
        uint32_t lo[3], hi[3], at[3];
        bool use[3] = {false, false, false};
        if (n >= 0) {
            const uint32_t id = d.ids[cur][i];
            const float4 l = d.plo[id], h = d.phi[id];
            const float c[3] = {centre(l.x, h.x), centre(l.y, h.y), centre(l.z, h.z)};
            lo[0] = key_of(l.x); lo[1] = key_of(l.y); lo[2] = key_of(l.z);
            hi[0] = key_of(h.x); hi[1] = key_of(h.y); hi[2] = key_of(h.z);
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                const float clo = of_key(d.nc[cur][12 * n + 6 + a]), ext = of_key(d.nc[cur][12 * n + 9 + a]) - clo;
                use[a] = ext > 0.f;
                at[a] = use[a] ? (uint32_t)bin_of(c[a], clo, (float)kBins / ext) : 0u;
            }
        }
        unsigned left = __ballot_sync(kAll, n >= 0);
        while (left) {
            const int32_t m = __shfl_sync(kAll, n, __ffs(left) - 1);
            if (m != node && node >= 0) flush();
            node = m;
            if (n == m) {
#pragma unroll
                for (uint32_t a = 0; a < 3; ++a)
                    if (use[a]) add(bins, a, at[a], lo, hi);
            }
            left &= ~__ballot_sync(kAll, n == m);
        }
    }
    if (node >= 0) flush();
}

// schedule a child: a next-level active node, or a subtree for one block; returns its active index or -1
__device__ __forceinline__ int32_t schedule(Dev& d, int nxt, uint32_t first, uint32_t count, uint32_t out,
                                            uint32_t depth) {
    if (count <= kMid) {
        d.mid[atomicAdd(&d.counters[kNumMid], 1u)] = make_uint4(first, count, out, depth);
        return -1;
    }
    const uint32_t k = atomicAdd(&d.counters[kActive + nxt], 1u);
    d.act[nxt][k] = make_uint4(first, count, out, depth);
    return (int32_t)k;
}

// One warp per active node: its split and the scheduling of the children (more than kMid
// triangles: no leaf test).  The node's bins and the next level's box slots are left empty.
__global__ void __launch_bounds__(128) k_split(Dev d, int cur) {
    const uint32_t n = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = (int)(threadIdx.x & 31u);
    if (n >= d.counters[kActive + cur]) return;        // whole warps leave together
    const uint4 A = d.act[cur][n];
    const uint32_t first = A.x, count = A.y;
    const uint32_t* nc = d.nc[cur] + 12 * n;
    uint32_t* bb = d.bb + (size_t)n * kBinWords;
    uint32_t usable = 0;
#pragma unroll
    for (int a = 0; a < 3; ++a)
        if (of_key(nc[9 + a]) - of_key(nc[6 + a]) > 0.f) usable |= 1u << a;
    const LaneBins B = lane_bins(bb, (uint32_t)lane);
    clear_bins(bb, (uint32_t)lane);
    if (lane < 24) d.nc[cur ^ 1][24 * n + lane] = empty_key(lane);
    const Split s = sweep(B, usable, lane);
    if (lane != 0) return;
    const uint32_t nl = s.axis < 0 ? count / 2 : s.left;    // median split by position without a SAH split
    const uint32_t base = atomicAdd(&d.counters[kNodes], 2u);
    BinNode& o = d.nodes[A.z];
    for (int k = 0; k < 3; ++k) { o.lo[k] = of_key(nc[k]); o.hi[k] = of_key(nc[3 + k]); }
    o.left = (int32_t)base;
    o.right = (int32_t)base + 1;
    o.first = 0;
    o.count = 0;
    o.n_tris = count;
    atomicMax(&d.counters[kDepth], A.w + 1u);
    d.d_ax[n] = s.axis;
    d.d_split[n] = s.bin;
    d.d_nl[n] = nl;
    if (s.axis >= 0) {
        const float lo = of_key(nc[6 + s.axis]);
        d.d_scale[n] = make_float2(lo, (float)kBins / (of_key(nc[9 + s.axis]) - lo));
    }
    d.cursor[n] = make_uint2(first, first + nl);
    d.d_child[2 * n] = schedule(d, cur ^ 1, first, nl, base, A.w + 1u);
    d.d_child[2 * n + 1] = schedule(d, cur ^ 1, first + nl, count - nl, base + 1, A.w + 1u);
}

// Triangles into their child's range (order within a child is arbitrary: min/max and counts do not
// depend on it), and the boxes and centroid boxes of the children that go on to the next level;
// finished positions are carried over unchanged.  A warp whose run lies in one node reduces the boxes and
// takes its slots of each child with one set of atomics, else the lanes do so one by one and per 32
// positions.
__global__ void __launch_bounds__(256) k_partition(Dev d, int cur, uint32_t nt) {
    constexpr int kIt = (int)(kWarpRun / 32u);
    const unsigned lane = threadIdx.x & 31u;
    unsigned lt;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(lt));
    const uint32_t p0 = ((blockIdx.x * blockDim.x + threadIdx.x) >> 5) * kWarpRun;
    int32_t node[kIt];
    uint32_t id[kIt];
    unsigned right = 0, move = 0;                     // bit k: position p0 + 32 k + lane goes right / is moved
    Box nb[2], cb[2];                                 // of the lane's triangles, by side
    clear(nb[0]); clear(nb[1]); clear(cb[0]); clear(cb[1]);
    bool same = true;
    int32_t first_node = 0;
#pragma unroll
    for (int k = 0; k < kIt; ++k) {
        const uint32_t i = p0 + 32u * k + lane;
        node[k] = i < nt ? d.pn[cur][i] : -1;
        id[k] = i < nt ? d.ids[cur][i] : 0u;
        if (k == 0) first_node = __shfl_sync(kAll, node[0], 0);
        same = same && node[k] == first_node;
    }
    const bool one = __all_sync(kAll, same && first_node >= 0);      // the whole run in one node
    auto add_box = [&](int32_t child, const Box& n, const Box& c) {
        uint32_t* to = d.nc[cur ^ 1] + 12 * child;
#pragma unroll
        for (int e = 0; e < 3; ++e) {
            atomicMin(to + e, key_of(n.lo[e])); atomicMax(to + 3 + e, key_of(n.hi[e]));
            atomicMin(to + 6 + e, key_of(c.lo[e])); atomicMax(to + 9 + e, key_of(c.hi[e]));
        }
    };
#pragma unroll
    for (int k = 0; k < kIt; ++k) {
        const int32_t n = node[k];
        if (n < 0) continue;
        const int32_t ax = d.d_ax[n];
        const float4 lo = d.plo[id[k]], hi = d.phi[id[k]];
        const float4 c = make_float4(centre(lo.x, hi.x), centre(lo.y, hi.y), centre(lo.z, hi.z), 0.f);
        bool r;
        if (ax < 0) {
            r = p0 + 32u * k + lane - d.act[cur][n].x >= d.d_nl[n];
        } else {
            const float2 sc = d.d_scale[n];
            r = bin_of(ax == 0 ? c.x : ax == 1 ? c.y : c.z, sc.x, sc.y) > d.d_split[n];
            move |= 1u << k;
        }
        if (r) right |= 1u << k;
        if (one) {
            if (r) { grow(nb[1], lo, hi); grow(cb[1], c, c); }
            else { grow(nb[0], lo, hi); grow(cb[0], c, c); }
        } else if (d.d_child[2 * n + (r ? 1 : 0)] >= 0) {
            Box b1, b2;
            clear(b1); clear(b2);
            grow(b1, lo, hi);
            grow(b2, c, c);
            add_box(d.d_child[2 * n + (r ? 1 : 0)], b1, b2);
        }
    }
    if (one) {
#pragma unroll
        for (int side = 0; side < 2; ++side) {
            const int32_t child = d.d_child[2 * first_node + side];
            if (child < 0) continue;                  // warp uniform
            warp_union(nb[side]);
            warp_union(cb[side]);
            if (lane == 0) add_box(child, nb[side], cb[side]);
        }
    }
    const bool run = __all_sync(kAll, same && move == (1u << kIt) - 1u);
    uint32_t at_l = 0, at_r = 0;
    if (run) {
        uint32_t nr = 0;
#pragma unroll
        for (int k = 0; k < kIt; ++k) nr += (uint32_t)__popc(__ballot_sync(kAll, (right >> k) & 1u));
        if (lane == 0) at_l = atomicAdd(&d.cursor[first_node].x, kWarpRun - nr);
        if (lane == 1) at_r = atomicAdd(&d.cursor[first_node].y, nr);
        at_l = __shfl_sync(kAll, at_l, 0);
        at_r = __shfl_sync(kAll, at_r, 1);
    }
#pragma unroll
    for (int k = 0; k < kIt; ++k) {
        const uint32_t i = p0 + 32u * k + lane;
        const uint32_t side = (right >> k) & 1u;
        const unsigned mr = __ballot_sync(kAll, side);
        uint32_t pos = i;
        if (run) {
            pos = side ? at_r + __popc(mr & lt) : at_l + __popc(~mr & lt);
            at_r += __popc(mr);
            at_l += 32u - __popc(mr);
        } else {
            const int32_t key = (move >> k) & 1u ? 2 * node[k] + (int32_t)side : -1;
            const unsigned grp = __match_any_sync(kAll, key);
            const int leader = __ffs(grp) - 1;
            uint32_t base = 0;
            if (key >= 0 && (int)lane == leader)
                base = atomicAdd(side ? &d.cursor[node[k]].y : &d.cursor[node[k]].x, (uint32_t)__popc(grp));
            base = __shfl_sync(kAll, base, leader);
            if (key >= 0) pos = base + (uint32_t)__popc(grp & lt);
        }
        if (i < nt) {
            d.ids[cur ^ 1][pos] = id[k];
            d.pn[cur ^ 1][pos] = node[k] < 0 ? -1 : d.d_child[2 * node[k] + side];
        }
    }
}

// One block per subtree of at most kMid triangles, down to the leaves (written where the subtree's
// triangle positions are): its nodes level by level, 8 or 16 lanes per node of at most as many
// triangles, one warp per larger node.  Bound by min / max issue and the latency of a node's steps: 328 k
// triangles take 251 us (363 us with the bins scanned by their lanes, 420 us with a warp sweep per
// node of 9 to 16 too, 507 us with a warp per node and leaf).
struct MidItem { uint16_t first, count; uint32_t out; };
// Nodes of at most G triangles, one per G lanes of the warp (lane t of a group: its node's triangle t);
// `on`: the lane's group has a node.  Every triangle's bin is a split candidate on each axis; the lanes
// of a group each evaluate their triangle's.  Reorders the node's triangles in perm and returns the
// size of its left child, 0 for a leaf; nb: the node's box.
template <int G>
__device__ __forceinline__ uint32_t small_node(bool on, uint32_t f, uint32_t cnt, uint32_t max_leaf, const float4* slo,
                                               const float4* shi, float* bins_of, uint16_t* perm, Box& nb) {
    const int lane = (int)(threadIdx.x & 31u);
    const uint32_t t = (uint32_t)lane & (G - 1u);
    cnt = on ? cnt : 0u;
    const bool have = t < cnt;
    const uint32_t j = have ? perm[f + t] : 0u;
    Box cb;
    clear(nb); clear(cb);
    float ce[3] = {0.f, 0.f, 0.f};
    if (have) {
        const float4 lo = slo[j], hi = shi[j];
        grow(nb, lo, hi);
        ce[0] = centre(lo.x, hi.x); ce[1] = centre(lo.y, hi.y); ce[2] = centre(lo.z, hi.z);
        const float4 p = make_float4(ce[0], ce[1], ce[2], 0.f);
        grow(cb, p, p);
    }
#pragma unroll
    for (int off = G / 2; off > 0; off >>= 1) {
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            nb.lo[k] = fminf(nb.lo[k], __shfl_xor_sync(kAll, nb.lo[k], off));
            nb.hi[k] = fmaxf(nb.hi[k], __shfl_xor_sync(kAll, nb.hi[k], off));
        }
    }
    const bool tiny = cnt <= 2u && cnt <= max_leaf;
    const uint32_t most = __reduce_max_sync(kAll, tiny ? 0u : cnt);
    if (most == 0u) return 0;
#pragma unroll
    for (int off = G / 2; off > 0; off >>= 1) {
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            cb.lo[k] = fminf(cb.lo[k], __shfl_xor_sync(kAll, cb.lo[k], off));
            cb.hi[k] = fmaxf(cb.hi[k], __shfl_xor_sync(kAll, cb.hi[k], off));
        }
    }
    uint32_t usable = 0, bins = 0;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const float ext = cb.hi[a] - cb.lo[a];
        if (ext > 0.f) {
            usable |= 1u << a;
            bins |= (uint32_t)bin_of(ce[a], cb.lo[a], (float)kBins / ext) << (5 * a);
        }
    }
    if (have) bins_of[4u * j] = __uint_as_float(bins);
    __syncwarp();
    Box l[3], r[3];
    uint32_t nl[3] = {0, 0, 0};
#pragma unroll
    for (int a = 0; a < 3; ++a) { clear(l[a]); clear(r[a]); }
    for (uint32_t i = 0; i < most; ++i) {
        if (i >= cnt) continue;
        const uint32_t k = perm[f + i];
        const float4 lo = slo[k], hi = shi[k];
        const uint32_t ob = __float_as_uint(lo.w);
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            if ((ob & (31u << (5 * a))) <= (bins & (31u << (5 * a)))) { grow(l[a], lo, hi); ++nl[a]; }
            else grow(r[a], lo, hi);
        }
    }
    float best = 3.4e38f;
    uint32_t key = 0xffffffffu;                       // axis, bin, size of the left child of the best split
    if (have) {
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            if (!((usable >> a) & 1u) || nl[a] == cnt) continue;
            const float cost = area(l[a].lo, l[a].hi) * (float)nl[a] + area(r[a].lo, r[a].hi) * (float)(cnt - nl[a]);
            if (cost < best) { best = cost; key = ((uint32_t)a << 16) | (((bins >> (5 * a)) & 31u) << 8) | nl[a]; }
        }
    }
#pragma unroll
    for (int off = G / 2; off > 0; off >>= 1) {
        const float ob = __shfl_xor_sync(kAll, best, off);
        const uint32_t ok = __shfl_xor_sync(kAll, key, off);
        if (ob < best || (ob == best && ok < key)) { best = ob; key = ok; }
    }
    bool leaf = tiny;
    if (!leaf && cnt <= max_leaf) {
        const float a = area(nb.lo, nb.hi);
        leaf = key == 0xffffffffu || best + a >= a * (float)cnt;
    }
    const bool median = key == 0xffffffffu;           // split by position without a SAH split
    const uint32_t ax = key >> 16, left = median ? cnt / 2 : key & 255u;
    const bool right = have && !median && ((bins >> (5 * ax)) & 31u) > ((key >> 8) & 255u);
    const unsigned gm = (G == 32 ? kAll : (1u << (G & 31)) - 1u) << (lane & ~(G - 1)), lt = (1u << lane) - 1u;
    const unsigned mr = __ballot_sync(kAll, right) & gm, ml = __ballot_sync(kAll, have && !right) & gm;
    if (have && !leaf && !median) perm[f + (right ? left + __popc(mr & lt) : __popc(ml & lt))] = (uint16_t)j;
    return leaf ? 0u : left;
}

__global__ void __launch_bounds__(kMidThreads) k_mid(Dev d, int cur, uint32_t* __restrict__ order) {
    __shared__ float4 slo[kMid], shi[kMid];          // w: packed bins, triangle id
    __shared__ uint16_t perm[kMid], tmp[kMid];
    __shared__ MidItem q[2][kMid];
    __shared__ uint32_t qn[2], next_node, max_depth;
    __shared__ uint32_t all_bins[kMidThreads / 32][kBinWords];
    if (blockIdx.x >= d.counters[kNumMid]) return;
    const uint4 S = d.mid[blockIdx.x];
    const uint32_t n = S.y;
    const int lane = (int)(threadIdx.x & 31u);
    const uint32_t warp = threadIdx.x >> 5, nwarps = kMidThreads / 32;
    for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) {
        const uint32_t id = d.ids[cur][S.x + i];
        slo[i] = d.plo[id];
        float4 hi = d.phi[id];
        hi.w = __uint_as_float(id);
        shi[i] = hi;
        perm[i] = (uint16_t)i;
    }
    if (threadIdx.x == 0) {
        q[0][0] = MidItem{0, (uint16_t)n, S.z};
        qn[0] = 1;
        qn[1] = 0;
        next_node = n > 1 ? atomicAdd(&d.counters[kNodes], 2u * n - 2u) : 0u;   // a subtree's nodes beside its root
        max_depth = 0;
    }
    __syncthreads();
    for (uint32_t level = 0;; ++level) {
        const int c = (int)(level & 1u);
        const uint32_t items = qn[c];
        if (items == 0) break;
        // node o of triangles [f, f + cnt): a leaf, or an inner node with nl triangles on the left
        auto set_leaf = [&](BinNode& o, const Box& nb, uint32_t f, uint32_t cnt) {
            float4* p = reinterpret_cast<float4*>(&o);
            p[0] = make_float4(nb.lo[0], nb.lo[1], nb.lo[2], __int_as_float(-1));
            p[1] = make_float4(nb.hi[0], nb.hi[1], nb.hi[2], __int_as_float(-1));
            reinterpret_cast<uint4*>(p)[2] = make_uint4(S.x + f, cnt, cnt, 0u);
        };
        auto set_inner = [&](BinNode& o, const Box& nb, uint32_t f, uint32_t cnt, uint32_t nl) {
            const uint32_t ob = atomicAdd(&next_node, 2u);
            float4* p = reinterpret_cast<float4*>(&o);
            p[0] = make_float4(nb.lo[0], nb.lo[1], nb.lo[2], __int_as_float((int)ob));
            p[1] = make_float4(nb.hi[0], nb.hi[1], nb.hi[2], __int_as_float((int)ob + 1));
            reinterpret_cast<uint4*>(p)[2] = make_uint4(0u, 0u, cnt, 0u);
            const uint32_t k = atomicAdd(&qn[c ^ 1], 2u);
            q[c ^ 1][k] = MidItem{(uint16_t)f, (uint16_t)nl, ob};
            q[c ^ 1][k + 1] = MidItem{(uint16_t)(f + nl), (uint16_t)(cnt - nl), ob + 1};
            max_depth = level + 1;                      // the same value from every node of the level
        };
        for (uint32_t it0 = 0; it0 < items; it0 += 4u * nwarps) {
            const uint32_t mine = it0 + (uint32_t)(lane >> 3) * nwarps + warp;    // the lane group's item
            MidItem m{0, 0, 0};
            if (mine < items) m = q[c][mine];
            float* bins = &slo[0].w;
            if (__any_sync(kAll, m.count != 0 && m.count <= 8u)) {
                const bool on = m.count != 0 && m.count <= 8u;
                Box nb;
                const uint32_t nl = small_node<8>(on, m.first, m.count, d.max_leaf, slo, shi, bins, perm, nb);
                if (on && (lane & 7) == 0) {
                    BinNode& o = d.nodes[m.out];
                    if (nl) set_inner(o, nb, m.first, m.count, nl);
                    else set_leaf(o, nb, m.first, m.count);
                }
            }
            // nodes of 9 to 16 triangles, two of the warp's four at a time
            unsigned pair = __ballot_sync(kAll, m.count > 8u && m.count <= 16u && (lane & 7) == 0);
            while (pair) {
                const int s0 = __ffs(pair) - 1;
                pair &= pair - 1u;
                const int s1 = pair ? __ffs(pair) - 1 : -1;
                pair &= pair ? pair - 1u : 0u;
                const int src = lane < 16 ? s0 : s1;
                const uint32_t f = __shfl_sync(kAll, (uint32_t)m.first, src < 0 ? 0 : src);
                const uint32_t cnt = __shfl_sync(kAll, (uint32_t)m.count, src < 0 ? 0 : src);
                const uint32_t to = __shfl_sync(kAll, m.out, src < 0 ? 0 : src);
                Box nb;
                const uint32_t nl = small_node<16>(src >= 0, f, cnt, d.max_leaf, slo, shi, bins, perm, nb);
                if (src >= 0 && (lane & 15) == 0) set_inner(d.nodes[to], nb, f, cnt, nl);
            }
            // the larger nodes of the warp's four, one after the other
            for (unsigned big = __ballot_sync(kAll, m.count > 16u && (lane & 7) == 0); big; big &= big - 1u) {
                const int src = __ffs(big) - 1;
                const uint32_t f = __shfl_sync(kAll, (uint32_t)m.first, src), cnt = __shfl_sync(kAll, (uint32_t)m.count, src);
                BinNode& o = d.nodes[__shfl_sync(kAll, m.out, src)];
                Box nb, cb;
                clear(nb); clear(cb);
                for (uint32_t i = f + lane; i < f + cnt; i += 32u) {
                    const uint32_t j = perm[i];
                    const float4 lo = slo[j], hi = shi[j];
                    grow(nb, lo, hi);
                    const float4 ce = make_float4(centre(lo.x, hi.x), centre(lo.y, hi.y), centre(lo.z, hi.z), 0.f);
                    grow(cb, ce, ce);
                }
                warp_union(nb);
                warp_union(cb);
                float scale[3];
                uint32_t usable = 0;
#pragma unroll
                for (int a = 0; a < 3; ++a) {
                    const float ext = cb.hi[a] - cb.lo[a];
                    scale[a] = ext > 0.f ? (float)kBins / ext : 0.f;
                    usable |= ext > 0.f ? 1u << a : 0u;
                }
                // the triangles' packed bins (beside their boxes) and the warp's bins of them
                uint32_t* wb = all_bins[warp];
                clear_bins(wb, (uint32_t)lane);
                __syncwarp();
                for (uint32_t i = f + lane; i < f + cnt; i += 32u) {
                    const uint32_t j = perm[i];
                    const float4 lo = slo[j], hi = shi[j];
                    const float ce[3] = {centre(lo.x, hi.x), centre(lo.y, hi.y), centre(lo.z, hi.z)};
                    const uint32_t kl[3] = {key_of(lo.x), key_of(lo.y), key_of(lo.z)}, kh[3] = {key_of(hi.x), key_of(hi.y), key_of(hi.z)};
                    uint32_t bins = 0;
#pragma unroll
                    for (uint32_t a = 0; a < 3; ++a)
                        if ((usable >> a) & 1u) {
                            const uint32_t bin = (uint32_t)bin_of(ce[a], cb.lo[a], scale[a]);
                            bins |= bin << (5 * a);
                            add(wb, a, bin, kl, kh);
                        }
                    slo[j].w = __uint_as_float(bins);
                }
                __syncwarp();
                const LaneBins B = lane_bins(wb, (uint32_t)lane);
                const Split s = sweep(B, usable, lane);
                uint32_t nl = cnt / 2;                   // median split by position without a SAH split
                if (s.axis >= 0) {
                    nl = s.left;
                    uint32_t a = f, b = f + nl;
                    for (uint32_t i0 = f; i0 < f + cnt; i0 += 32u) {
                        const uint32_t i = i0 + lane;
                        const bool in = i < f + cnt;
                        const uint32_t j = in ? perm[i] : 0u;
                        const bool right = in && (int)((__float_as_uint(slo[j].w) >> (5 * s.axis)) & 31u) > s.bin;
                        const unsigned ml = __ballot_sync(kAll, in && !right), mr = __ballot_sync(kAll, right);
                        const unsigned lt = (1u << lane) - 1u;
                        if (in) tmp[right ? b + __popc(mr & lt) : a + __popc(ml & lt)] = (uint16_t)j;
                        a += __popc(ml);
                        b += __popc(mr);
                    }
                    __syncwarp();
                    for (uint32_t i = f + lane; i < f + cnt; i += 32u) perm[i] = tmp[i];
                }
                if (lane == 0) set_inner(o, nb, f, cnt, nl);
            }
        }
        __syncthreads();
        if (threadIdx.x == 0) qn[c] = 0;
        __syncthreads();
    }
    for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) order[S.x + i] = __float_as_uint(shi[perm[i]].w);
    if (threadIdx.x == 0) atomicMax(&d.counters[kDepth], S.w + max_depth);
}

// ---- four-child collapse (the rules of finish_bvh in bvh_build.cpp) ----

// Level L of the four-child tree: each root picks its children (the binary children, then the
// interior child of largest area, the first on ties, is opened while there are fewer than four),
// gives the interior ones their places in the next level and writes its node (boxes one ulp
// outward).  q holds the roots' binary indices at their four-child indices, breadth first; the
// leaves' triangles stay in the builder's order.
__global__ void __launch_bounds__(128) k_collapse(const BinNode* __restrict__ nodes, uint32_t* q, uint32_t* counters,
                                                  uint32_t level, DevNode* __restrict__ out) {
    const uint32_t n = counters[kLevel + level];
    uint32_t lo = 0;
    for (uint32_t k = 0; k < level; ++k) lo += counters[kLevel + k];
    const uint32_t next = lo + n;
    const int lane = (int)(threadIdx.x & 31u);
    for (uint32_t i0 = blockIdx.x * blockDim.x; i0 < n; i0 += gridDim.x * blockDim.x) {     // warp-uniform
        const uint32_t i = i0 + threadIdx.x;
        const bool on = i < n;
        const BinNode root = nodes[q[lo + (on ? i : 0u)]];
        int32_t c[4] = {root.left, root.right, -1, -1};
        BinNode b[4];
        b[0] = nodes[c[0]];
        b[1] = nodes[c[1]];
        int k = 2;
        while (k < 4) {
            int best = -1;
            float ba = -1.0f;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                if (j >= k || b[j].left < 0) continue;
                const float a = area(b[j].lo, b[j].hi);
                if (a > ba) { ba = a; best = j; }
            }
            if (best < 0) break;
            int32_t l = -1, r = -1;
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (j == best) { l = b[j].left; r = b[j].right; }
#pragma unroll
            for (int j = 3; j >= 1; --j)
                if (j > best + 1) { c[j] = c[j - 1]; b[j] = b[j - 1]; }
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                if (j == best) { c[j] = l; b[j] = nodes[l]; }
                if (j == best + 1) { c[j] = r; b[j] = nodes[r]; }
            }
            ++k;
        }
        DevNode g;
        uint32_t inner = 0, leaves = 0;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            if (j < k && b[j].left >= 0) ++inner;
            if (j < k && b[j].left < 0) ++leaves;
        }
        if (!on) inner = leaves = 0;
        // places in the next level: one atomic per warp
        uint32_t incl = inner;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const uint32_t v = __shfl_up_sync(kAll, incl, off);
            if (lane >= off) incl += v;
        }
        leaves = __reduce_add_sync(kAll, leaves);
        uint32_t base = 0;
        if (lane == 31 && incl) base = atomicAdd(&counters[kLevel + level + 1], incl);
        if (lane == 0 && leaves) atomicAdd(&counters[kLeaves], leaves);
        uint32_t at = next + __shfl_sync(kAll, base, 31) + incl - inner;
        if (!on) continue;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            if (j >= k) {
                for (int e = 0; e < 3; ++e) g.plane[e][j][0] = g.plane[e][j][1] = 3.402823466e+38f;
                g.child[j] = ~(int32_t)0;           // leaf of 0 triangles: never entered
                continue;
            }
#pragma unroll
            for (int e = 0; e < 3; ++e) {
                float l = b[j].lo[e], h = b[j].hi[e];
                if (l <= h) { l = nextafterf(l, -INFINITY); h = nextafterf(h, INFINITY); }
                g.plane[e][j][0] = l;
                g.plane[e][j][1] = h;
            }
            if (b[j].left >= 0) {
                g.child[j] = (int32_t)at;
                q[at] = (uint32_t)c[j];
                ++at;
            } else {
                g.child[j] = ~(int32_t)((b[j].first << 3) | b[j].count);
            }
        }
        g.pad[0] = g.pad[1] = g.pad[2] = g.pad[3] = 0;
        const float4* src = reinterpret_cast<const float4*>(&g);
        float4* dst = reinterpret_cast<float4*>(out + lo + i);
#pragma unroll
        for (int e = 0; e < 8; ++e) dst[e] = src[e];
    }
}

}  // namespace

// Builds the four-child BVH of device-resident vertices [nv][3] and triangles [nt][3]; returns
// false when the input is invalid (out-of-range index or non-finite vertex: the caller's host
// builder reports which).  Throws tri::CudaError on CUDA failures.
bool build_bvh_device(const float* d_v, uint32_t nv, const uint32_t* d_t, uint32_t nt, uint32_t max_leaf,
                      cudaStream_t s, const std::function<DevNode*(size_t)>& alloc_nodes, uint32_t* d_order,
                      DeviceBvh& out) {
    const auto t0 = std::chrono::steady_clock::now();
    if (nt == 0 || nt >= (1u << 28)) return false;
    if (max_leaf < 1 || max_leaf > 7) max_leaf = 4;
    const uint32_t amax = nt / (kMid + 1) + 2;        // active nodes of a level (> kMid triangles each)
    // one scratch block, returned to the pool in stream order
    Dev d{};
    d.max_leaf = max_leaf;
    uint32_t* q = nullptr;
    DevNode* dn = nullptr;
    auto carve = [&](char* base) {
        size_t at = 0;
        auto take = [&](auto*& p, size_t count) {
            using T = std::remove_reference_t<decltype(*p)>;
            p = reinterpret_cast<T*>(reinterpret_cast<uintptr_t>(base) + at);
            at = (at + count * sizeof(T) + 255) & ~size_t(255);
        };
        take(d.plo, nt); take(d.phi, nt);
        for (int b = 0; b < 2; ++b) { take(d.ids[b], nt); take(d.pn[b], nt); take(d.act[b], amax); take(d.nc[b], 24 * (size_t)amax); }
        take(d.bb, (size_t)amax * 21 * kBins);
        take(d.d_ax, amax); take(d.d_split, amax); take(d.d_nl, amax); take(d.d_scale, amax);
        take(d.d_child, 2 * (size_t)amax); take(d.cursor, amax);
        take(d.mid, (size_t)nt + 1);                  // disjoint and not empty
        take(d.nodes, 2 * (size_t)nt);
        take(d.counters, (size_t)kCounters);
        take(q, nt);
        take(dn, nt);
        return at;
    };
    int dev = 0, sms = 1;
    TR_CUDA(cudaGetDevice(&dev));
    TR_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    void* block = nullptr;
    TR_CUDA(tri::pool_malloc(&block, carve(nullptr), s));
    struct Free { void* p; cudaStream_t s; ~Free() { tri::pool_free_after(p, s); } } release{block, s};
    carve(static_cast<char*>(block));

    uint32_t h[kCounters];
    auto read = [&]() {
        TR_CUDA(cudaMemcpyAsync(h, d.counters, sizeof(h), cudaMemcpyDeviceToHost, s));
        TR_CUDA(cudaStreamSynchronize(s));
    };
    k_start<<<std::max(1u, std::min(592u, (amax * 21u * kBins + 255) / 256)), 256, 0, s>>>(d, amax, nt);
    k_prims<<<std::max(1u, std::min(4u * (uint32_t)sms, (std::max(nt, nv) + 255) / 256)), 256, 0, s>>>(d_v, nv, d_t, nt, d);
    TR_CUDA(cudaGetLastError());
    const uint32_t run_blocks = (nt + kWarpRun * 8u - 1u) / (kWarpRun * 8u);
    int cur = 0;
    uint32_t level = 0;
    // the first wait after the levels that halving takes, later ones every three levels
    uint32_t ahead = 1;
    while (nt > kMid && (nt >> ahead) > kMid) ++ahead;
    for (bool more = nt > kMid; more;) {
        for (uint32_t k = 0; k < ahead; ++k, ++level) {
            const uint32_t na = level < 28 ? std::min(amax, 1u << level) : amax;
            k_bin<<<run_blocks, 256, 0, s>>>(d, cur, nt);
            k_split<<<(na + 3) / 4, 128, 0, s>>>(d, cur);                    // one warp per active node
            k_partition<<<run_blocks, 256, 0, s>>>(d, cur, nt);
            cur ^= 1;
        }
        TR_CUDA(cudaGetLastError());
        read();
        if (h[kError]) return false;                  // invalid input
        more = h[kActive + cur] != 0;
        ahead = 3;
    }
    if (nt <= kMid) h[kNumMid] = 1;
    k_mid<<<h[kNumMid], kMidThreads, 0, s>>>(d, cur, d_order);
    TR_CUDA(cudaGetLastError());
    // the collapse of as many levels as a balanced tree has, then a few at a time
    uint32_t done = 0;
    ahead = 2;
    while ((1ull << (2 * ahead)) < nt) ++ahead;
    ahead = std::min(ahead + 2u, kMaxLevels);
    TR_CUDA(cudaMemsetAsync(q, 0, sizeof(uint32_t), s));
    BinNode top;
    TR_CUDA(cudaMemcpyAsync(&top, d.nodes, sizeof(top), cudaMemcpyDeviceToHost, s));
    read();
    if (h[kError]) return false;
    if (top.left < 0) return false;                 // a one-leaf scene: the host builder takes it
    for (;;) {
        for (uint32_t k = 0; k < ahead; ++k, ++done)
            k_collapse<<<std::max(1u, std::min(1184u, (uint32_t)std::min<uint64_t>(nt, 1ull << std::min(30u, 2 * done)) / 128u + 1u)), 128, 0, s>>>(
                d.nodes, q, d.counters, done, dn);
        TR_CUDA(cudaGetLastError());
        read();
        if (h[kLevel + done] == 0 || done + 4 > kMaxLevels) break;
        ahead = 4;
    }
    uint32_t n4 = 0, levels = 0;
    for (uint32_t k = 0; k < done && h[kLevel + k]; ++k) { n4 += h[kLevel + k]; ++levels; }
    if (h[kLevel + done]) levels = kMaxLevels;      // deeper than any traversal stack
    DevNode* dst = alloc_nodes(n4);
    TR_CUDA(cudaMemcpyAsync(dst, dn, (size_t)n4 * sizeof(DevNode), cudaMemcpyDeviceToDevice, s));
    out.nodes = n4;
    out.depth = levels;
    out.stack = 3 * out.depth + 1;
    out.binary_depth = h[kDepth];
    out.leaves = h[kLeaves];
    for (int k = 0; k < 6; ++k) {
        const uint32_t key = h[kVertex + k];
        const uint32_t u = key ^ ((uint32_t)((int32_t)~key >> 31) | 0x80000000u);
        float f;
        std::memcpy(&f, &u, 4);
        (k < 3 ? out.vlo : out.vhi)[k % 3] = f;
    }
    out.build_ms = std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count();
    return true;
}

}  // namespace trh
