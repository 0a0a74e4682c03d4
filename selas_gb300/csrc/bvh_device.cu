// Device SAH BVH builder: the 8-wide quantised layout of bvh_build.cpp built on the GPU.
//
// Same method as the host builder (binned SAH after Wald 2007, 32 bins per axis, leaves of at most 3 triangles by
// default (1..8 selectable), median splits beyond depth 40, greedy collapse to 8 children by largest surface area,
// octant slot assignment and outward 8-bit child-box quantisation after Ylitie, Karras and Laine 2017), in four
// launches:
//   1. k_records: one thread per triangle: leaf record, bounds, scene box and centroid box;
//   2. k_top (cooperative): subtrees of more than kSmall triangles, one level at a time: chunks of triangles are
//      binned into block-local bins, one warp per subtree picks the split, chunks are partitioned;
//   3. k_small: subtrees of at most kSmall triangles, one block each with the triangles' boxes in shared memory, one
//      level at a time: a warp bins a part of more than 16 triangles, 16 or 8 lanes sweep smaller ones exactly
//      (every centroid is a candidate plane);
//   4. k_collapse (cooperative): collapse and quantisation one level at a time, eight lanes per 8-wide node.
// Node slots follow the host builder's layout (a subtree of n triangles occupies slots [s, s + 2n - 1),
// left child at s + 1, right child at s + 2 * n_left), so the tree needs no slot allocation.  Traversal
// results do not depend on the tree (order-independent closest-hit rule, outward-rounded boxes).
//
// The build is bound by latency (dependent levels) and by the number of instructions per tree node, not by memory.
// Before, one warp per subtree of 1,024 triangles, depth first, took 3.4 ms whatever the scene's size, a thread per
// 8-wide node 0.07 ms a level, every level a round trip to the host, and the host made the leaf records.  Whole
// commits now take (then): 22 triangles 0.15 (0.81) ms, 163,842 1.7 (9.6), 655,362 3.2 (18.5), 5,242,882 14.5 (109),
// of which the upload and these kernels 0.15 (0.54), 1.7 (6.8), 3.1 (8.9), 14.4 (28.5).
#include <algorithm>
#include <chrono>
#include <cmath>
#include <cstring>
#include <type_traits>

#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include "sel_internal.h"

namespace sel {

namespace {

namespace cg = cooperative_groups;

constexpr int kBinsD = 32;
constexpr int kBinWords = 3 * kBinsD * 7;  // per bin: box lo, hi as ordered ints, count
constexpr uint32_t kMaxLeafLimit = kMaxLeafRecords;  // leaves beyond a node's 32 records move one level down
constexpr int kMedianDepthD = 40;
constexpr uint32_t kSmall = 1024;   // subtrees at or below this many triangles are built by one block
constexpr uint32_t kChunk = 2048;   // triangles a block bins or partitions at a time (256 threads x 8)
constexpr int kSmallWarps = 8;
constexpr uint32_t kErrTooDeep = 1u, kErrNonFinite = 2u, kErrIndex = 4u;

__device__ __forceinline__ int f2o(float f) {  // float -> int with the same order
    const int i = __float_as_int(f);
    return i >= 0 ? i : i ^ 0x7fffffff;
}
__device__ __forceinline__ float o2f(int i) { return __int_as_float(i >= 0 ? i : i ^ 0x7fffffff); }

__device__ __forceinline__ float box_area(float3 lo, float3 hi) {
    if (lo.x > hi.x) return 0.0f;
    const float dx = hi.x - lo.x, dy = hi.y - lo.y, dz = hi.z - lo.z;
    return 2.0f * (dx * dy + dy * dz + dz * dx);
}
__device__ __forceinline__ float comp(const float4& v, int axis) { return axis == 0 ? v.x : (axis == 1 ? v.y : v.z); }
__device__ __forceinline__ float centre(const float4& l, const float4& h, int axis) {
    return 0.5f * (comp(l, axis) + comp(h, axis));
}
__device__ __forceinline__ int bin_of(float c, float lo, float k) {
    int b = int((c - lo) * k);
    return b < 0 ? 0 : (b > kBinsD - 1 ? kBinsD - 1 : b);
}
__device__ __forceinline__ float bin_scale(float ext) { return ext > 0.0f ? float(kBinsD) * (1.0f - 1e-6f) / ext : 0.0f; }

// A mesh's arrays in HBM and its first triangle in the scene.
struct MeshDev {
    const float* vertices;
    const uint32_t* indices;
    uint32_t first, vertex_count, geom, kind;
};

// A subtree of more than kSmall triangles.
struct TopTask {
    uint32_t first, count, slot, depth;
    uint32_t chunk0, pad[3];  // its first chunk in the level's chunk list
    int box[6], cbox[6];      // bounds of the boxes and of the centroids (ordered ints)
    uint32_t axis, bin, left_count, by_position;  // the split
    uint32_t cursor[2];                           // triangles moved left / right so far
    uint32_t child[2];                            // their tasks in the next level's list (all ones: small)
};

struct Counters {
    uint32_t tasks[2], chunks[2], small, depth, err, pad;
    int box[6], cbox[6];
    uint32_t wide, tris, levels, pad2;
};

struct Build {
    const MeshDev* meshes;
    uint32_t mesh_count;
    float4* soup;            // leaf records in input order, 3 x float4 (TriRecord)
    float4* lo[2];           // per triangle: box lo, w = input index bits; partitions ping-pong
    float4* hi[2];
    uint32_t* idx;           // triangle order of the leaves
    float4* nlo;             // binary nodes: box lo, w = left slot bits (leaf: all ones)
    float4* nhi;             // box hi, w = right slot bits
    uint2* nrange;           // first, count (count > 0: leaf)
    TopTask* tasks[2];
    int* bins;               // per task of the level
    uint32_t* chunk_task[2]; // task of each chunk of the level
    uint4* small;            // first, count, slot, depth | buffer << 31
    Counters* ctr;
    uint32_t n, max_leaf;
};

// ---------------------------------------------------------------------------------------------------
// 1. Leaf records and bounds.
// ---------------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(256) k_records(Build B) {
    float v[12];
    for (int k = 0; k < 12; ++k) v[k] = (k % 6) < 3 ? INFINITY : -INFINITY;
    uint32_t err = 0;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < B.n; i += gridDim.x * blockDim.x) {
        uint32_t m = 0, top = B.mesh_count;  // the last mesh whose first triangle is at or below i
        while (top - m > 1) {
            const uint32_t mid = (m + top) >> 1;
            if (B.meshes[mid].first <= i) m = mid;
            else top = mid;
        }
        const MeshDev& M = B.meshes[m];
        const uint32_t t = i - M.first;
        float p[3][3];
        for (int k = 0; k < 3; ++k) {
            uint32_t vi = M.indices[3 * size_t(t) + k];
            if (vi >= M.vertex_count) {
                err |= kErrIndex;
                vi = 0;
            }
            for (int a = 0; a < 3; ++a) {
                p[k][a] = M.vertices[3 * size_t(vi) + a];
                if (!isfinite(p[k][a])) err |= kErrNonFinite;
            }
        }
        float4* rec = B.soup + size_t(i) * 3;
        rec[0] = make_float4(p[0][0], p[0][1], p[0][2], __uint_as_float(t));
        rec[1] = make_float4(p[1][0], p[1][1], p[1][2], __uint_as_float(M.geom));
        rec[2] = make_float4(p[2][0], p[2][1], p[2][2], __uint_as_float(M.kind));
        float l[3], h[3];
        for (int a = 0; a < 3; ++a) {
            l[a] = fminf(fminf(p[0][a], p[1][a]), p[2][a]);
            h[a] = fmaxf(fmaxf(p[0][a], p[1][a]), p[2][a]);
            const float c = 0.5f * (l[a] + h[a]);
            v[a] = fminf(v[a], l[a]);
            v[3 + a] = fmaxf(v[3 + a], h[a]);
            v[6 + a] = fminf(v[6 + a], c);
            v[9 + a] = fmaxf(v[9 + a], c);
        }
        B.lo[0][i] = make_float4(l[0], l[1], l[2], __uint_as_float(i));
        B.hi[0][i] = make_float4(h[0], h[1], h[2], 0.0f);
    }
    if (err) atomicOr(&B.ctr->err, err);
    for (int k = 0; k < 12; ++k) {
        const int o = (k % 6) < 3 ? __reduce_min_sync(0xffffffffu, f2o(v[k])) : __reduce_max_sync(0xffffffffu, f2o(v[k]));
        int* dst = k < 6 ? &B.ctr->box[k] : &B.ctr->cbox[k - 6];
        if ((threadIdx.x & 31) == 0) {
            if ((k % 6) < 3) atomicMin(dst, o);
            else atomicMax(dst, o);
        }
    }
}

// ---------------------------------------------------------------------------------------------------
// 2. Subtrees of more than kSmall triangles, level by level.
// ---------------------------------------------------------------------------------------------------

// SAH over the 32 bins of one axis, lane b = bin b: the cost of splitting after bin b (infinite where a side is
// empty) and the triangles left of it.
__device__ __forceinline__ void sah_sweep(const int* bins, int lane, float& cost, uint32_t& nleft) {
    const int* b = bins + lane * 7;
    float lo[3] = {o2f(b[0]), o2f(b[1]), o2f(b[2])}, hi[3] = {o2f(b[3]), o2f(b[4]), o2f(b[5])};
    const uint32_t c = uint32_t(b[6]);
    // inclusive prefix (left side of the split after this bin)
    float plo[3] = {lo[0], lo[1], lo[2]}, phi[3] = {hi[0], hi[1], hi[2]};
    uint32_t pc = c;
    // inclusive suffix
    float slo[3] = {lo[0], lo[1], lo[2]}, shi[3] = {hi[0], hi[1], hi[2]};
    uint32_t sc = c;
    for (int o = 1; o < 32; o <<= 1) {
        float t;
        for (int a = 0; a < 3; ++a) {
            t = __shfl_up_sync(0xffffffffu, plo[a], o); if (lane >= o) plo[a] = fminf(plo[a], t);
            t = __shfl_up_sync(0xffffffffu, phi[a], o); if (lane >= o) phi[a] = fmaxf(phi[a], t);
            t = __shfl_down_sync(0xffffffffu, slo[a], o); if (lane + o < 32) slo[a] = fminf(slo[a], t);
            t = __shfl_down_sync(0xffffffffu, shi[a], o); if (lane + o < 32) shi[a] = fmaxf(shi[a], t);
        }
        uint32_t u = __shfl_up_sync(0xffffffffu, pc, o); if (lane >= o) pc += u;
        u = __shfl_down_sync(0xffffffffu, sc, o); if (lane + o < 32) sc += u;
    }
    // split after bin `lane`: left = prefix(lane), right = suffix(lane + 1)
    float rlo[3], rhi[3];
    for (int a = 0; a < 3; ++a) {
        rlo[a] = __shfl_down_sync(0xffffffffu, slo[a], 1);
        rhi[a] = __shfl_down_sync(0xffffffffu, shi[a], 1);
    }
    const uint32_t rc = __shfl_down_sync(0xffffffffu, sc, 1);
    cost = INFINITY;
    nleft = pc;
    if (lane < 31 && pc > 0 && rc > 0) {
        const float la = box_area(make_float3(plo[0], plo[1], plo[2]), make_float3(phi[0], phi[1], phi[2]));
        const float ra = box_area(make_float3(rlo[0], rlo[1], rlo[2]), make_float3(rhi[0], rhi[1], rhi[2]));
        cost = la * float(pc) + ra * float(rc);
    }
}

// The best binned split of a part with centroid bounds clo..chi: its axis (-1: none), bin, left count and cost.
__device__ __forceinline__ int best_bin_split(const int* bins, const float* clo, const float* chi, int lane,
                                              uint32_t& bin, uint32_t& nl, float& best) {
    best = INFINITY;
    int best_axis = -1;
    for (int a = 0; a < 3; ++a) {
        if (!(chi[a] > clo[a])) continue;
        float cost;
        uint32_t n_left;
        sah_sweep(bins + a * kBinsD * 7, lane, cost, n_left);
        const int key = f2o(cost);
        const int least = __reduce_min_sync(0xffffffffu, key);
        const int bb = __ffs(__ballot_sync(0xffffffffu, key == least)) - 1;  // ties to the lower bin
        const float bc = o2f(least);
        const uint32_t nlb = __shfl_sync(0xffffffffu, n_left, bb);
        if (bc < best) {
            best = bc;
            best_axis = a;
            bin = uint32_t(bb);
            nl = nlb;
        }
    }
    return best_axis;
}

__device__ __forceinline__ void clear_bins(int* bins, int i0, int step) {
    for (int i = i0; i < kBinWords; i += step) {
        const int w = i % 7;
        bins[i] = w < 3 ? f2o(INFINITY) : (w < 6 ? f2o(-INFINITY) : 0);
    }
}

__device__ __forceinline__ void bin_prim(int* bins, const float4& l, const float4& h, const float* clo, const float* kk) {
    const int lo[3] = {f2o(l.x), f2o(l.y), f2o(l.z)}, hi[3] = {f2o(h.x), f2o(h.y), f2o(h.z)};
    for (int a = 0; a < 3; ++a) {
        int* b = bins + (a * kBinsD + bin_of(centre(l, h, a), clo[a], kk[a])) * 7;
        for (int q = 0; q < 3; ++q) {
            atomicMin(b + q, lo[q]);
            atomicMax(b + 3 + q, hi[q]);
        }
        atomicAdd(b + 6, 1);
    }
}

// Adds a subtree to the next level's list, or to the small ones (one lane).  Returns its task index.
__device__ uint32_t add_task(const Build& B, int next, uint32_t first, uint32_t count, uint32_t slot, uint32_t depth,
                             int buffer) {
    if (count <= kSmall) {
        B.small[atomicAdd(&B.ctr->small, 1u)] = make_uint4(first, count, slot, depth | (uint32_t(buffer) << 31));
        return 0xffffffffu;
    }
    const uint32_t q = atomicAdd(&B.ctr->tasks[next], 1u);
    const uint32_t chunks = (count + kChunk - 1) / kChunk;
    const uint32_t c0 = atomicAdd(&B.ctr->chunks[next], chunks);
    TopTask& t = B.tasks[next][q];
    t.first = first;
    t.count = count;
    t.slot = slot;
    t.depth = depth;
    t.chunk0 = c0;
    for (int k = 0; k < 6; ++k) t.box[k] = t.cbox[k] = k < 3 ? f2o(INFINITY) : f2o(-INFINITY);
    t.cursor[0] = t.cursor[1] = 0;
    for (uint32_t k = 0; k < chunks; ++k) B.chunk_task[next][c0 + k] = q;
    return q;
}

__device__ void split_task(const Build& B, int cur, uint32_t index, int lane) {
    TopTask& t = B.tasks[cur][index];
    const uint32_t count = t.count, depth = t.depth;
    float clo[3], chi[3];
    for (int a = 0; a < 3; ++a) {
        clo[a] = o2f(t.cbox[a]);
        chi[a] = o2f(t.cbox[3 + a]);
    }
    int axis = 0;
    for (int a = 1; a < 3; ++a)
        if (chi[a] - clo[a] > chi[axis] - clo[axis]) axis = a;
    const bool degenerate = !(chi[axis] > clo[axis]);
    const int* bins = B.bins + size_t(index) * kBinWords;
    uint32_t by_position = 1, split_axis = uint32_t(axis), bin = 0, nl = count / 2;
    if (!degenerate && int(depth) < kMedianDepthD) {
        float cost;
        const int a = best_bin_split(bins, clo, chi, lane, bin, nl, cost);
        if (a >= 0) {
            split_axis = uint32_t(a);
            by_position = 0;
        }
    } else if (!degenerate) {
        // object median through the bins of the widest axis: the bin where half of the triangles is reached
        uint32_t incl = uint32_t(bins[(axis * kBinsD + lane) * 7 + 6]);
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t u = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += u;
        }
        const uint32_t ok = __ballot_sync(0xffffffffu, incl >= count / 2 && incl < count);
        if (ok) {
            by_position = 0;
            bin = uint32_t(__ffs(ok) - 1);
            nl = __shfl_sync(0xffffffffu, incl, int(bin));
        }
    }
    if (nl == 0 || nl >= count) {
        by_position = 1;
        nl = count / 2;
    }
    if (lane == 0) {
        t.axis = split_axis;
        t.bin = bin;
        t.left_count = nl;
        t.by_position = by_position;
        const uint32_t left = t.slot + 1, right = t.slot + 2 * nl;
        B.nlo[t.slot] = make_float4(o2f(t.box[0]), o2f(t.box[1]), o2f(t.box[2]), __uint_as_float(left));
        B.nhi[t.slot] = make_float4(o2f(t.box[3]), o2f(t.box[4]), o2f(t.box[5]), __uint_as_float(right));
        B.nrange[t.slot] = make_uint2(t.first, 0);
        const int next = cur ^ 1;  // the triangles move to the other buffer with the level
        t.child[0] = add_task(B, next, t.first, nl, left, depth + 1, next);
        t.child[1] = add_task(B, next, t.first + nl, count - nl, right, depth + 1, next);
    }
}

// Moves a chunk's triangles to their sides in the other buffer and grows the bounds of the children's tasks.
__device__ void partition_chunk(const Build& B, int cur, uint32_t chunk) {
    __shared__ uint32_t warp_left[8], warp_right[8], base_left, base_right;
    __shared__ int child_box[2][12];
    const TopTask& t = B.tasks[cur][B.chunk_task[cur][chunk]];
    const uint32_t begin = (chunk - t.chunk0) * kChunk, end = min(t.count, begin + kChunk);
    const int a = int(t.axis), lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const float clo = o2f(t.cbox[a]), kk = bin_scale(o2f(t.cbox[3 + a]) - clo);
    if (threadIdx.x < 24) child_box[threadIdx.x / 12][threadIdx.x % 12] = (threadIdx.x % 6) < 3 ? f2o(INFINITY) : f2o(-INFINITY);
    float4 l[8], h[8];
    uint32_t left = 0, n_left = 0, n_right = 0;  // bit k: the thread's k-th triangle goes left
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        const uint32_t i = begin + uint32_t(k) * 256u + threadIdx.x;
        if (i >= end) continue;
        l[k] = B.lo[cur][t.first + i];
        h[k] = B.hi[cur][t.first + i];
        const bool go = t.by_position ? i < t.left_count : bin_of(centre(l[k], h[k], a), clo, kk) <= int(t.bin);
        left |= uint32_t(go) << k;
        n_left += go;
        n_right += !go;
    }
    // exclusive offsets of the threads' triangles within the block
    uint32_t il = n_left, ir = n_right;
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t x = __shfl_up_sync(0xffffffffu, il, o), y = __shfl_up_sync(0xffffffffu, ir, o);
        if (lane >= o) {
            il += x;
            ir += y;
        }
    }
    if (lane == 31) {
        warp_left[w] = il;
        warp_right[w] = ir;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t sl = 0, sr = 0;
        for (int k = 0; k < 8; ++k) {
            const uint32_t x = warp_left[k], y = warp_right[k];
            warp_left[k] = sl;
            warp_right[k] = sr;
            sl += x;
            sr += y;
        }
        TopTask& out = B.tasks[cur][B.chunk_task[cur][chunk]];
        base_left = sl ? atomicAdd(&out.cursor[0], sl) : 0u;
        base_right = sr ? atomicAdd(&out.cursor[1], sr) : 0u;
    }
    __syncthreads();
    uint32_t at_left = t.first + base_left + warp_left[w] + il - n_left;
    uint32_t at_right = t.first + t.left_count + base_right + warp_right[w] + ir - n_right;
    int v[2][12];
    for (int c = 0; c < 2; ++c)
        for (int k = 0; k < 12; ++k) v[c][k] = (k % 6) < 3 ? f2o(INFINITY) : f2o(-INFINITY);
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        const uint32_t i = begin + uint32_t(k) * 256u + threadIdx.x;
        if (i >= end) continue;
        const int c = (left >> k) & 1u ? 0 : 1;
        const uint32_t dst = c == 0 ? at_left++ : at_right++;
        B.lo[cur ^ 1][dst] = l[k];
        B.hi[cur ^ 1][dst] = h[k];
        for (int q = 0; q < 3; ++q) {
            const int lo = f2o(comp(l[k], q)), hi = f2o(comp(h[k], q)), ce = f2o(centre(l[k], h[k], q));
            for (int side = 0; side < 2; ++side) {
                if (side != c) continue;
                v[side][q] = min(v[side][q], lo);
                v[side][3 + q] = max(v[side][3 + q], hi);
                v[side][6 + q] = min(v[side][6 + q], ce);
                v[side][9 + q] = max(v[side][9 + q], ce);
            }
        }
    }
    for (int c = 0; c < 2; ++c) {
        if (t.child[c] == 0xffffffffu) continue;  // small subtrees find their bounds themselves
        for (int k = 0; k < 12; ++k) {
            const int r = (k % 6) < 3 ? __reduce_min_sync(0xffffffffu, v[c][k]) : __reduce_max_sync(0xffffffffu, v[c][k]);
            if (lane == 0) {
                if ((k % 6) < 3) atomicMin(&child_box[c][k], r);
                else atomicMax(&child_box[c][k], r);
            }
        }
    }
    __syncthreads();
    if (threadIdx.x < 24) {
        const int c = threadIdx.x / 12, k = threadIdx.x % 12;
        if (t.child[c] != 0xffffffffu) {
            TopTask& child = B.tasks[cur ^ 1][t.child[c]];
            int* dst = k < 6 ? &child.box[k] : &child.cbox[k - 6];
            if ((k % 6) < 3) atomicMin(dst, child_box[c][k]);
            else atomicMax(dst, child_box[c][k]);
        }
    }
    __syncthreads();  // the shared words are the next chunk's
}

__global__ void __launch_bounds__(256, 2) k_top(Build B) {
    if (B.ctr->err) return;  // bad input, found by k_records
    cg::grid_group grid = cg::this_grid();
    __shared__ int bins[kBinWords];
    const int lane = threadIdx.x & 31;
    const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, warps = (gridDim.x * blockDim.x) >> 5;
    if (blockIdx.x == 0 && threadIdx.x == 0) {  // the root
        const uint32_t q = add_task(B, 0, 0, B.n, 0, 0, 0);
        if (q != 0xffffffffu)
            for (int k = 0; k < 6; ++k) {
                B.tasks[0][q].box[k] = B.ctr->box[k];
                B.tasks[0][q].cbox[k] = B.ctr->cbox[k];
            }
    }
    grid.sync();
    for (int cur = 0;; cur ^= 1) {
        const uint32_t ntasks = *(volatile uint32_t*)&B.ctr->tasks[cur];
        const uint32_t nchunks = *(volatile uint32_t*)&B.ctr->chunks[cur];
        if (ntasks == 0) break;
        for (uint32_t t = blockIdx.x; t < ntasks; t += gridDim.x)
            clear_bins(B.bins + size_t(t) * kBinWords, threadIdx.x, 256);
        if (blockIdx.x == 0 && threadIdx.x == 0) B.ctr->tasks[cur ^ 1] = B.ctr->chunks[cur ^ 1] = 0;
        grid.sync();
        for (uint32_t c = blockIdx.x; c < nchunks; c += gridDim.x) {
            const uint32_t index = B.chunk_task[cur][c];
            const TopTask& t = B.tasks[cur][index];
            const uint32_t begin = (c - t.chunk0) * kChunk, end = min(t.count, begin + kChunk);
            float clo[3], kk[3];
            for (int a = 0; a < 3; ++a) {
                clo[a] = o2f(t.cbox[a]);
                kk[a] = bin_scale(o2f(t.cbox[3 + a]) - clo[a]);
            }
            clear_bins(bins, threadIdx.x, 256);
            __syncthreads();
            for (uint32_t i = begin + threadIdx.x; i < end; i += 256)
                bin_prim(bins, B.lo[cur][t.first + i], B.hi[cur][t.first + i], clo, kk);
            __syncthreads();
            int* g = B.bins + size_t(index) * kBinWords;
            for (int i = threadIdx.x; i < kBinWords; i += 256) {
                if (!bins[i - i % 7 + 6]) continue;  // an empty bin
                const int w = i % 7;
                if (w < 3) atomicMin(g + i, bins[i]);
                else if (w < 6) atomicMax(g + i, bins[i]);
                else atomicAdd(g + i, bins[i]);
            }
            __syncthreads();
        }
        grid.sync();
        for (uint32_t t = warp; t < ntasks; t += warps) split_task(B, cur, t, lane);
        grid.sync();
        for (uint32_t c = blockIdx.x; c < nchunks; c += gridDim.x) partition_chunk(B, cur, c);
        grid.sync();
    }
}

// ---------------------------------------------------------------------------------------------------
// 3. Subtrees of at most kSmall triangles, one block each.
// ---------------------------------------------------------------------------------------------------

// A part of the subtree: first and count within the block's order array, depth, node slot.
__device__ __forceinline__ uint2 pack_part(uint32_t first, uint32_t count, uint32_t depth, uint32_t slot) {
    return make_uint2(first | (count << 10) | (depth << 21), slot);
}

constexpr uint32_t kBigParts = kSmall / 17 + 1, kMidParts = kSmall / 9 + 1, kTinyParts = kSmall / 2;

struct SmallShared {
    float box[6][kSmall];            // lo x y z, hi x y z of triangle k
    uint32_t tri[kSmall];            // its input index
    uint16_t order[2][kSmall];       // order and partition scratch
    int bins[kSmallWarps][kBinWords];
    uint2 big[2][kBigParts], mid[2][kMidParts], tiny[2][kTinyParts];
    uint32_t counts[2][3];
};

__device__ __forceinline__ void write_node(const Build& B, uint32_t slot, const float* v, uint32_t left, uint32_t right,
                                           uint32_t first, uint32_t leaf_count) {
    B.nlo[slot] = make_float4(v[0], v[1], v[2], __uint_as_float(left));
    B.nhi[slot] = make_float4(v[3], v[4], v[5], __uint_as_float(right));
    B.nrange[slot] = make_uint2(first, leaf_count);
}

__device__ __forceinline__ void add_part(SmallShared& S, int next, uint32_t first, uint32_t count, uint32_t depth,
                                         uint32_t slot) {
    if (count < 2) return;  // single triangles became leaves as they were partitioned
    const int kind = count > 16 ? 0 : (count > 8 ? 1 : 2);
    const uint32_t q = atomicAdd(&S.counts[next][kind], 1u);
    uint2* list = kind == 0 ? S.big[next] : (kind == 1 ? S.mid[next] : S.tiny[next]);
    list[q] = pack_part(first, count, depth, slot);
}

// A part of more than 16 triangles by one warp: binned SAH, stable partition.
__device__ void split_big(const Build& B, SmallShared& S, int* bins, int next, uint2 part, uint32_t global_first) {
    const uint32_t first = part.x & 1023u, count = (part.x >> 10) & 2047u, depth = part.x >> 21, slot = part.y;
    const uint32_t lane = threadIdx.x & 31u;
    float v[12];
    for (int k = 0; k < 12; ++k) v[k] = (k % 6) < 3 ? INFINITY : -INFINITY;
    for (uint32_t i = lane; i < count; i += 32) {
        const uint32_t p = S.order[0][first + i];
        for (int a = 0; a < 3; ++a) {
            const float l = S.box[a][p], h = S.box[3 + a][p], c = 0.5f * (l + h);
            v[a] = fminf(v[a], l);
            v[3 + a] = fmaxf(v[3 + a], h);
            v[6 + a] = fminf(v[6 + a], c);
            v[9 + a] = fmaxf(v[9 + a], c);
        }
    }
    for (int k = 0; k < 12; ++k) {
        const int o = f2o(v[k]);
        v[k] = o2f((k % 6) < 3 ? __reduce_min_sync(0xffffffffu, o) : __reduce_max_sync(0xffffffffu, o));
    }
    int axis = 0;
    for (int a = 1; a < 3; ++a)
        if (v[9 + a] - v[6 + a] > v[9 + axis] - v[6 + axis]) axis = a;
    const bool degenerate = !(v[9 + axis] > v[6 + axis]);
    uint32_t nl = count / 2, bin = 0;
    bool by_position = true;
    if (!degenerate && int(depth) < kMedianDepthD) {
        clear_bins(bins, int(lane), 32);
        __syncwarp();
        float kk[3];
        for (int a = 0; a < 3; ++a) kk[a] = bin_scale(v[9 + a] - v[6 + a]);
        for (uint32_t i = lane; i < count; i += 32) {
            const uint32_t p = S.order[0][first + i];
            bin_prim(bins, make_float4(S.box[0][p], S.box[1][p], S.box[2][p], 0.0f),
                     make_float4(S.box[3][p], S.box[4][p], S.box[5][p], 0.0f), v + 6, kk);
        }
        __syncwarp();
        float cost;
        const int a = best_bin_split(bins, v + 6, v + 9, int(lane), bin, nl, cost);
        if (a >= 0 && nl > 0 && nl < count) {
            axis = a;
            by_position = false;
        }
        __syncwarp();
    }
    if (by_position) nl = count / 2;
    const float lo = v[6 + axis], k = bin_scale(v[9 + axis] - v[6 + axis]);
    const uint32_t left = slot + 1, right = slot + 2 * nl, below = (1u << lane) - 1u;
    uint32_t lcount = 0, rcount = 0;
    for (uint32_t base = 0; base < count; base += 32) {
        const uint32_t i = base + lane;
        uint32_t p = 0;
        bool go = false;
        if (i < count) {
            p = S.order[0][first + i];
            go = by_position ? i < nl : bin_of(0.5f * (S.box[axis][p] + S.box[3 + axis][p]), lo, k) <= int(bin);
        }
        const uint32_t lm = __ballot_sync(0xffffffffu, i < count && go), rm = __ballot_sync(0xffffffffu, i < count && !go);
        if (i < count) {
            S.order[1][go ? first + lcount + __popc(lm & below) : first + nl + rcount + __popc(rm & below)] = uint16_t(p);
            if ((go ? nl : count - nl) == 1) {  // a leaf of one triangle
                const float b[6] = {S.box[0][p], S.box[1][p], S.box[2][p], S.box[3][p], S.box[4][p], S.box[5][p]};
                write_node(B, go ? left : right, b, ~0u, ~0u, global_first + (go ? first : first + nl), 1);
            }
        }
        lcount += __popc(lm);
        rcount += __popc(rm);
    }
    __syncwarp();
    for (uint32_t i = lane; i < count; i += 32) S.order[0][first + i] = S.order[1][first + i];
    if (lane == 0) {
        write_node(B, slot, v, left, right, global_first + first, 0);
        add_part(S, next, first, nl, depth + 1, left);
        add_part(S, next, first + nl, count - nl, depth + 1, right);
    }
}

// A part of at most G triangles by G lanes (an aligned group): exact SAH over every centroid plane of every axis,
// lane i's candidates being the planes through its triangle's centroid.
template <int G>
__device__ void split_group(const Build& B, SmallShared& S, int next, uint2 part, uint32_t global_first) {
    const uint32_t lane = threadIdx.x & 31u, gl = lane & uint32_t(G - 1), g0 = lane & ~uint32_t(G - 1);
    const uint32_t mask = (G == 32 ? 0xffffffffu : ((1u << (G & 31)) - 1u)) << g0;
    const uint32_t first = part.x & 1023u, count = (part.x >> 10) & 2047u, depth = part.x >> 21, slot = part.y;
    const bool mine = gl < count;
    const uint32_t p = mine ? S.order[0][first + gl] : 0u;
    float b[6];  // this lane's box; lanes past the part repeat nothing
    for (int k = 0; k < 6; ++k) b[k] = mine ? S.box[k][p] : (k < 3 ? INFINITY : -INFINITY);
    const float c[3] = {0.5f * (b[0] + b[3]), 0.5f * (b[1] + b[4]), 0.5f * (b[2] + b[5])};
    float llo[3][3], lhi[3][3], rlo[3][3], rhi[3][3];  // per candidate axis: left and right boxes
    uint32_t nleft[3] = {0, 0, 0};
    float v[6];
    for (int a = 0; a < 3; ++a)
        for (int q = 0; q < 3; ++q) {
            llo[a][q] = rlo[a][q] = INFINITY;
            lhi[a][q] = rhi[a][q] = -INFINITY;
        }
    for (int q = 0; q < 3; ++q) {
        v[q] = INFINITY;
        v[3 + q] = -INFINITY;
    }
    for (uint32_t j = 0; j < count; ++j) {
        float o[6];
        for (int k = 0; k < 6; ++k) o[k] = __shfl_sync(mask, b[k], int(g0 + j));
        for (int q = 0; q < 3; ++q) {
            v[q] = fminf(v[q], o[q]);
            v[3 + q] = fmaxf(v[3 + q], o[3 + q]);
        }
        for (int a = 0; a < 3; ++a) {
            const bool l = 0.5f * (o[a] + o[3 + a]) <= c[a];
            nleft[a] += l;
            for (int q = 0; q < 3; ++q) {
                llo[a][q] = fminf(llo[a][q], l ? o[q] : INFINITY);
                lhi[a][q] = fmaxf(lhi[a][q], l ? o[3 + q] : -INFINITY);
                rlo[a][q] = fminf(rlo[a][q], l ? INFINITY : o[q]);
                rhi[a][q] = fmaxf(rhi[a][q], l ? -INFINITY : o[3 + q]);
            }
        }
    }
    float cost = INFINITY;
    int axis = -1;
    for (int a = 0; a < 3; ++a) {
        if (!mine || nleft[a] >= count) continue;
        const float la = box_area(make_float3(llo[a][0], llo[a][1], llo[a][2]), make_float3(lhi[a][0], lhi[a][1], lhi[a][2]));
        const float ra = box_area(make_float3(rlo[a][0], rlo[a][1], rlo[a][2]), make_float3(rhi[a][0], rhi[a][1], rhi[a][2]));
        const float x = la * float(nleft[a]) + ra * float(count - nleft[a]);
        if (x < cost) {
            cost = x;
            axis = a;
        }
    }
    const int key = f2o(cost);
    const int least = __reduce_min_sync(mask, key);
    const uint32_t win = __ffs(__ballot_sync(mask, key == least)) - 1;
    axis = __shfl_sync(mask, axis, int(win));
    const float plane = axis < 0 ? 0.0f : (axis == 0 ? c[0] : (axis == 1 ? c[1] : c[2]));
    const float threshold = __shfl_sync(mask, plane, int(win));
    const float best = o2f(least);
    const float area = box_area(make_float3(v[0], v[1], v[2]), make_float3(v[3], v[4], v[5]));
    const bool median = axis < 0 || int(depth) >= kMedianDepthD;
    const bool leaf = count <= B.max_leaf && (median || area + best >= area * float(count));
    if (leaf) {
        if (gl == 0) write_node(B, slot, v, ~0u, ~0u, global_first + first, count);
        return;
    }
    bool go = gl < count / 2;
    if (!median) go = (axis == 0 ? c[0] : (axis == 1 ? c[1] : c[2])) <= threshold;
    const uint32_t lm = (__ballot_sync(mask, mine && go) >> g0), rm = (__ballot_sync(mask, mine && !go) >> g0);
    const uint32_t nl = __popc(lm), below = (1u << gl) - 1u;
    const uint32_t left = slot + 1, right = slot + 2 * nl;
    if (mine) {
        S.order[0][go ? first + __popc(lm & below) : first + nl + __popc(rm & below)] = uint16_t(p);
        if ((go ? nl : count - nl) == 1)
            write_node(B, go ? left : right, b, ~0u, ~0u, global_first + (go ? first : first + nl), 1);
    }
    if (gl == 0) {
        write_node(B, slot, v, left, right, global_first + first, 0);
        add_part(S, next, first, nl, depth + 1, left);
        add_part(S, next, first + nl, count - nl, depth + 1, right);
    }
}

__global__ void __launch_bounds__(32 * kSmallWarps, 2) k_small(Build B) {
    extern __shared__ __align__(16) unsigned char small_shared[];
    SmallShared& S = *reinterpret_cast<SmallShared*>(small_shared);
    if (B.ctr->err) return;
    const uint32_t ntasks = B.ctr->small;
    const uint32_t w = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    for (uint32_t task = blockIdx.x; task < ntasks; task += gridDim.x) {
        const uint4 t = B.small[task];
        const uint32_t first = t.x, count = t.y;
        const int buffer = int(t.w >> 31);
        for (uint32_t i = threadIdx.x; i < count; i += blockDim.x) {
            const float4 l = B.lo[buffer][first + i], h = B.hi[buffer][first + i];
            S.box[0][i] = l.x; S.box[1][i] = l.y; S.box[2][i] = l.z;
            S.box[3][i] = h.x; S.box[4][i] = h.y; S.box[5][i] = h.z;
            S.tri[i] = __float_as_uint(l.w);
            S.order[0][i] = uint16_t(i);
        }
        if (threadIdx.x < 6) S.counts[threadIdx.x / 3][threadIdx.x % 3] = 0;
        __syncthreads();
        if (threadIdx.x == 0) {
            if (count == 1) {
                const float b[6] = {S.box[0][0], S.box[1][0], S.box[2][0], S.box[3][0], S.box[4][0], S.box[5][0]};
                write_node(B, t.z, b, ~0u, ~0u, first, 1);
            }
            add_part(S, 0, 0, count, t.w & 0x7fffffffu, t.z);
        }
        __syncthreads();
        for (int cur = 0;; cur ^= 1) {
            const uint32_t nb = S.counts[cur][0], nm = S.counts[cur][1], nt = S.counts[cur][2];
            if (nb + nm + nt == 0) break;
            for (uint32_t k = w; k < nb; k += kSmallWarps) split_big(B, S, S.bins[w], cur ^ 1, S.big[cur][k], first);
            for (uint32_t k = 2 * w; k < nm; k += 2 * kSmallWarps)
                if (k + (lane >> 4) < nm) split_group<16>(B, S, cur ^ 1, S.mid[cur][k + (lane >> 4)], first);
            for (uint32_t k = 4 * w; k < nt; k += 4 * kSmallWarps)
                if (k + (lane >> 3) < nt) split_group<8>(B, S, cur ^ 1, S.tiny[cur][k + (lane >> 3)], first);
            __syncthreads();
            if (threadIdx.x < 3) S.counts[cur][threadIdx.x] = 0;
            __syncthreads();
        }
        for (uint32_t i = threadIdx.x; i < count; i += blockDim.x) B.idx[first + i] = S.tri[S.order[0][i]];
        __syncthreads();
    }
}

// ---------------------------------------------------------------------------------------------------
// 4. Collapse to 8-wide nodes and quantisation, one level at a time, eight lanes per node.
// ---------------------------------------------------------------------------------------------------
struct Collapse {
    int* binary;        // binary node of each 8-wide node; -(node + 2): a demoted leaf, alone in a node of its own
    WideNode* nodes;
    float4* tris;
    uint32_t max_wide;
};

// Outward 8-bit quantisation of the child boxes on one axis (the host builder's rule, in double precision), lane s
// the child in slot s: the node's origin and exponent, this child's planes.
__device__ __forceinline__ void quantise_axis(uint32_t mask, bool present, float clo, float chi, float& origin, int& exponent,
                                              uint32_t& qlo, uint32_t& qhi) {
    const float nlo = o2f(__reduce_min_sync(mask, f2o(present ? clo : INFINITY)));
    const float nhi = o2f(__reduce_max_sync(mask, f2o(present ? chi : -INFINITY)));
    const double ext = double(nhi) - double(nlo);
    const double mag = fmax(fabs(double(nlo)), fabs(double(nhi)));
    const double min_q = fmax(mag * (1.0 / 1048576.0), ldexp(1.0, -60));
    const double least = fmax(ext / 250.0, min_q);
    // 2^e >= least: the exponent frexp returns for a positive normal number
    int e = int((__double2hiint(least) >> 20) & 0x7ff) - 1022;
    for (int guard = 0; guard < 2100; ++guard, ++e) {
        const double scale = __hiloint2double((e + 1023) << 20, 0), inv = __hiloint2double((1023 - e) << 20, 0);
        float p = float(double(nlo) - scale);
        if (double(p) > double(nlo) - scale) p = nextafterf(p, -INFINITY);
        bool ok = true;
        double lo = 255.0, hi = 0.0;
        if (present) {
            lo = floor((double(clo) - p) * inv) - 1.0;
            hi = ceil((double(chi) - p) * inv) + 1.0;
            while (lo > 0.0 && double(p) + lo * scale > double(clo) - 0.5 * scale) lo -= 1.0;
            while (double(p) + hi * scale < double(chi) + 0.5 * scale) hi += 1.0;
            ok = !(lo < 0.0 || hi > 255.0 || double(p) + lo * scale > double(clo) - 0.5 * scale);
        }
        if (__all_sync(mask, ok)) {
            origin = p;
            exponent = e;
            qlo = uint32_t(lo);
            qhi = uint32_t(hi);
            return;
        }
    }
    origin = nlo;
    exponent = 127;
    qlo = present ? 0u : 255u;
    qhi = present ? 255u : 0u;
}

// One 8-wide node by an aligned group of eight lanes, lane k first a child, then a slot.
__device__ void collapse_node(const Build& B, const Collapse& C, uint32_t wide) {
    const uint32_t lane = threadIdx.x & 31u, k = lane & 7u, g0 = lane & 24u, mask = 0xffu << g0;
    const int entry = C.binary[wide];
    const int root = entry <= -2 ? -entry - 2 : entry;
    // children: the root's two (or the root itself, a leaf), then the largest internal one opened until there are 8
    int child = -1;
    float4 l = make_float4(0, 0, 0, 0), h = l;
    uint2 range = make_uint2(0, 0);
    auto load = [&](int node) {
        child = node;
        l = B.nlo[node];
        h = B.nhi[node];
        range = B.nrange[node];
    };
    auto open_key = [&]() -> int {  // area of an internal child as an ordered int; -1: not to be opened
        return child >= 0 && range.y == 0
                   ? __float_as_int(fmaxf(box_area(make_float3(l.x, l.y, l.z), make_float3(h.x, h.y, h.z)), 0.0f))
                   : -1;
    };
    uint32_t nc = 1;
    if (k == 0) load(root);
    for (;;) {
        const int key = open_key();
        const int most = __reduce_max_sync(mask, key);
        if (most < 0 || nc >= 8 || (entry <= -2)) break;
        const uint32_t w = __ffs(__ballot_sync(mask, key == most)) - 1;
        const int left = __shfl_sync(mask, int(__float_as_uint(l.w)), int(w));
        const int right = __shfl_sync(mask, int(__float_as_uint(h.w)), int(w));
        if (lane == w) load(left);
        if (k == nc) load(right);
        ++nc;
    }
    // slots by octant direction (the host builder's rule): the cheapest (child, slot) pair of those left, ties in
    // (child, slot) order
    const bool real = child >= 0;
    const float blo[3] = {l.x, l.y, l.z}, bhi[3] = {h.x, h.y, h.z};
    float off[3];
    for (int a = 0; a < 3; ++a) {
        const float nlo = o2f(__reduce_min_sync(mask, f2o(real ? blo[a] : INFINITY)));
        const float nhi = o2f(__reduce_max_sync(mask, f2o(real ? bhi[a] : -INFINITY)));
        off[a] = 0.5f * (blo[a] + bhi[a]) - 0.5f * (nlo + nhi);
    }
    uint32_t taken = 0, my_slot = 0xffu;
    for (uint32_t round = 0; round < nc; ++round) {
        float best = INFINITY;
        uint32_t bs = 8;
        if (real && my_slot == 0xffu)
            for (uint32_t s = 0; s < 8; ++s) {
                if ((taken >> s) & 1u) continue;
                const float d = (s & 4u ? off[0] : -off[0]) + (s & 2u ? off[1] : -off[1]) + (s & 1u ? off[2] : -off[2]);
                if (-d < best) {
                    best = -d;
                    bs = s;
                }
            }
        const int key = f2o(__fadd_rn(best, 0.0f));
        const int least = __reduce_min_sync(mask, key);
        const uint32_t who = __ballot_sync(mask, bs < 8 && key == least);
        if (!who) break;
        const uint32_t w = __ffs(who) - 1;
        const uint32_t s = __shfl_sync(mask, bs, int(w));
        if (lane == w) my_slot = s;
        taken |= 1u << s;
    }
    // lane s takes the child of slot s
    uint32_t from = 0xffu;
    for (uint32_t j = 0; j < 8; ++j)
        if (__shfl_sync(mask, my_slot, int(g0 + j)) == k) from = j;
    const int src = int(g0 + (from < 8 ? from : 0u));
    const int sc = __shfl_sync(mask, child, src);
    const uint32_t rx = __shfl_sync(mask, range.x, src), ry = __shfl_sync(mask, range.y, src);
    float slo[3], shi[3];
    for (int a = 0; a < 3; ++a) {
        slo[a] = __shfl_sync(mask, blo[a], src);
        shi[a] = __shfl_sync(mask, bhi[a], src);
    }
    const bool present = from < 8;
    bool leaf = present && ry > 0;
    // A node's leaf children hold 32 records at most (the traversal's record mask).  With leaves of more than
    // 4 triangles eight of them can hold more: the largest leaf (the lowest slot among equals) then becomes an
    // internal child, a node of its own one level down whose single slot is that leaf, until the rest fit.
    bool demoted = false;
    for (int guard = 0; guard < 8; ++guard) {
        const uint32_t total = __reduce_add_sync(mask, leaf ? ry : 0u);
        if (total <= kMaxNodeRecords) break;
        const uint32_t big = __reduce_max_sync(mask, leaf ? ry : 0u);
        const uint32_t w = __ffs(__ballot_sync(mask, leaf && ry == big)) - 1;
        if (lane == w) {
            leaf = false;
            demoted = true;
        }
    }
    const bool inner = present && !leaf;
    const uint32_t inner_mask = (__ballot_sync(mask, inner) >> g0) & 0xffu;
    // records of the leaf slots, in slot order
    uint32_t incl = leaf ? ry : 0u;
    for (int o = 1; o < 8; o <<= 1) {
        const uint32_t x = __shfl_up_sync(mask, incl, o, 8);
        if (int(k) >= o) incl += x;
    }
    const uint32_t records = __shfl_sync(mask, incl, int(g0 + 7u)), offset = incl - (leaf ? ry : 0u);
    uint32_t child_base = 0, tri_base = 0;
    if (k == 0) {
        child_base = atomicAdd(&B.ctr->wide, __popc(inner_mask));
        tri_base = atomicAdd(&B.ctr->tris, records);
    }
    child_base = __shfl_sync(mask, child_base, int(g0));
    tri_base = __shfl_sync(mask, tri_base, int(g0));
    unsigned char* node = reinterpret_cast<unsigned char*>(C.nodes + wide);
    for (int a = 0; a < 3; ++a) {
        float p;
        int e;
        uint32_t qlo, qhi;
        quantise_axis(mask, present, slo[a], shi[a], p, e, qlo, qhi);
        if (k == 0) {
            reinterpret_cast<float*>(node)[a] = p;
            node[12 + a] = uint8_t(e + 127);
        }
        node[32 + 8 * a + k] = uint8_t(qlo);
        node[56 + 8 * a + k] = uint8_t(qhi);
    }
    if (k == 0) {
        node[15] = uint8_t(inner_mask);
        reinterpret_cast<uint32_t*>(node)[4] = child_base;
        reinterpret_cast<uint32_t*>(node)[5] = tri_base;
    }
    node[24 + k] = uint8_t(leaf ? ((ry - 1u) << 5) | offset : kLeafNone);
    if (inner) {
        const uint32_t at = child_base + __popc(inner_mask & ((1u << k) - 1u));
        if (at < C.max_wide) C.binary[at] = demoted ? -(sc + 2) : sc;
    }
    if (leaf)
        for (uint32_t j = 0; j < ry; ++j) {
            const uint32_t at = tri_base + offset + j;
            if (at >= B.n) break;  // reported as lost triangles
            const float4* rec = B.soup + size_t(B.idx[rx + j]) * 3;
            float4* dst = C.tris + size_t(at) * 3;
            dst[0] = rec[0];
            dst[1] = rec[1];
            dst[2] = rec[2];
        }
}

__global__ void __launch_bounds__(256, 2) k_collapse(Build B, Collapse C) {
    if (B.ctr->err) return;  // set before this launch, or by the last level of it
    cg::grid_group grid = cg::this_grid();
    const uint32_t group = (blockIdx.x * blockDim.x + threadIdx.x) >> 3, groups = (gridDim.x * blockDim.x) >> 3;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        C.binary[0] = 0;
        B.ctr->wide = 1;
        B.ctr->tris = 0;
    }
    grid.sync();
    uint32_t begin = 0;
    for (uint32_t level = 1;; ++level) {
        const uint32_t end = min(*(volatile uint32_t*)&B.ctr->wide, C.max_wide);
        if (begin >= end) break;
        if (level > uint32_t(kWideStack)) {
            if (blockIdx.x == 0 && threadIdx.x == 0) atomicOr(&B.ctr->err, kErrTooDeep);
            break;
        }
        if (blockIdx.x == 0 && threadIdx.x == 0) B.ctr->levels = level;
        grid.sync();  // every thread has read the level's end
        for (uint32_t i = begin + group; i < end; i += groups) collapse_node(B, C, i);
        begin = end;
        grid.sync();
    }
}

}  // namespace

std::string build_wide_device(const std::vector<MeshInput>& meshes, uint32_t max_leaf, DeviceBuild& out) {
    if (max_leaf < 1 || max_leaf > kMaxLeafLimit) return "leaf size must lie in 1..8";
    size_t total = 0, vertex_total = 0;
    for (const MeshInput& m : meshes) {
        total += m.indices.size() / 3;
        vertex_total += m.vertices.size();
    }
    if (total == 0) return "scene has no triangles";
    if (total > (size_t(1) << 30)) return "too many triangles";
    const uint32_t n = uint32_t(total);
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const auto t0 = std::chrono::steady_clock::now();

    // 8-wide nodes: each has at least two slots except the single-leaf nodes of demoted leaves (at most one per
    // five triangles, as only a leaf of five or more is demoted), so at most n + n / 5 + 1 of them
    const size_t max_wide = max_leaf > 4 ? size_t(n) + n / 5 + 1 : n;
    const size_t max_top = size_t(n) / kSmall + 2;         // subtrees of more than kSmall triangles in one level
    const size_t max_chunks = size_t(n) / kChunk + max_top;
    Build B;
    Collapse C;
    std::memset(&B, 0, sizeof(B));
    std::memset(&C, 0, sizeof(C));
    B.n = n;
    B.max_leaf = max_leaf;
    B.mesh_count = uint32_t(meshes.size());
    C.max_wide = uint32_t(max_wide);
    float* vertices = nullptr;
    uint32_t* indices = nullptr;
    MeshDev* mesh_table = nullptr;
    // What is copied to the GPU lies in memory that lives until the stream is synchronised below, on every way out;
    // the host's allocations come before the GPU's, so that one that fails leaves nothing behind.
    constexpr size_t kDirectBytes = 64 * 1024;
    std::vector<MeshDev> table;
    std::vector<uint32_t> packed;  // small meshes: vertices (as bits) and indices, in the order of their places
    size_t small_words = 0;
    for (const MeshInput& m : meshes)
        for (const size_t words : {m.vertices.size(), m.indices.size()})
            if (words * 4 < kDirectBytes) small_words += words;
    table.reserve(meshes.size());
    packed.reserve(small_words);
    const uint4 root = make_uint4(0, n, 0, 0);
    Counters ctr;
    std::memset(&ctr, 0, sizeof(ctr));
    ctr.small = n > kSmall ? 0u : 1u;  // the scene is one small subtree
    for (int k = 0; k < 6; ++k) {
        // +-infinity as ordered ints
        ctr.box[k] = ctr.cbox[k] = k < 3 ? 0x7f800000 : int(0xff800000u ^ 0x7fffffffu);
    }
    // one scratch block for everything but the result: sized on the first walk, carved on the second
    size_t scratch_bytes = 0;
    char* scratch = nullptr;
    for (int walk = 0; walk < 2; ++walk) {
        size_t at = 0;
        auto take = [&](auto*& p, size_t count) {
            using T = std::remove_reference_t<decltype(*p)>;
            if (walk) p = reinterpret_cast<T*>(scratch + at);
            at += (sizeof(T) * std::max<size_t>(count, 1) + 255) & ~size_t(255);
        };
        take(B.ctr, 1);
        take(mesh_table, meshes.size());
        take(vertices, vertex_total);
        take(indices, 3 * total);
        take(B.soup, size_t(n) * 3);
        for (int k = 0; k < 2; ++k) {
            take(B.lo[k], n);
            take(B.hi[k], n);
            take(B.tasks[k], max_top);
            take(B.chunk_task[k], max_chunks);
        }
        take(B.idx, n);
        take(B.nlo, 2 * size_t(n));
        take(B.nhi, 2 * size_t(n));
        take(B.nrange, 2 * size_t(n));
        take(B.bins, max_top * kBinWords);
        take(B.small, size_t(n));
        take(C.binary, max_wide);
        take(C.nodes, max_wide);
        if (!walk) {
            scratch_bytes = at;
            const cudaError_t e = cudaMalloc(&scratch, scratch_bytes);
            if (e != cudaSuccess) return std::string("device BVH build: ") + cudaGetErrorString(e);
        }
    }
    B.meshes = mesh_table;
    cudaStream_t s = nullptr;
    cudaError_t e = cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking);
    if (e == cudaSuccess) e = cudaMalloc(&C.tris, sizeof(TriRecord) * size_t(n));

    // the meshes' arrays: large ones are copied from where they lie, small ones gathered into one copy
    size_t vat = 0, iat = 0;
    uint32_t first = 0;
    for (const MeshInput& m : meshes) {
        MeshDev d;
        d.vertices = vertices + vat;
        d.indices = indices + iat;
        d.first = first;
        d.vertex_count = uint32_t(m.vertices.size() / 3);
        d.geom = m.geomID;
        d.kind = m.quads ? kTriQuadHalf : (m.curves ? kTriCurve : kTriPlain);
        if (!m.indices.empty()) table.push_back(d);
        vat += m.vertices.size();
        iat += m.indices.size();
        first += uint32_t(m.indices.size() / 3);
    }
    auto upload = [&](void* dst, auto array_of) {  // runs of small arrays together
        char* run = static_cast<char*>(dst);
        auto flush = [&]() {
            if (!packed.empty() && e == cudaSuccess)
                e = cudaMemcpyAsync(run, packed.data(), packed.size() * 4, cudaMemcpyHostToDevice, s);
            if (!packed.empty() && e == cudaSuccess) e = cudaStreamSynchronize(s);  // packed is refilled
            run += packed.size() * 4;
            packed.clear();
        };
        for (const MeshInput& m : meshes) {
            const auto& a = array_of(m);
            const size_t bytes = a.size() * 4;
            if (bytes < kDirectBytes) {
                const uint32_t* w = reinterpret_cast<const uint32_t*>(a.data());
                packed.insert(packed.end(), w, w + a.size());
                continue;
            }
            flush();
            if (e == cudaSuccess) e = cudaMemcpyAsync(run, a.data(), bytes, cudaMemcpyHostToDevice, s);
            run += bytes;
        }
        flush();
    };
    upload(vertices, [](const MeshInput& m) -> const std::vector<float>& { return m.vertices; });
    upload(indices, [](const MeshInput& m) -> const std::vector<uint32_t>& { return m.indices; });
    B.mesh_count = uint32_t(table.size());
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(mesh_table, table.data(), sizeof(MeshDev) * table.size(), cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess) e = cudaMemcpyAsync(B.ctr, &ctr, sizeof(ctr), cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess) {
        const int records_grid = int(std::min<size_t>((size_t(n) + 255) / 256, size_t(sms) * 8));
        k_records<<<records_grid, 256, 0, s>>>(B);
        void* top_args[] = {&B};
        void* collapse_args[] = {&B, &C};
        // as many blocks as run at once, fewer for small scenes (a grid barrier costs less)
        auto cooperative = [&](const void* kernel, size_t work, void** args) {
            int per_sm = 0;
            e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, 256, 0);
            const size_t most = size_t(sms) * size_t(std::max(per_sm, 1));
            const unsigned blocks = unsigned(std::min(most, std::max<size_t>(work, 1)));
            if (e == cudaSuccess) e = cudaLaunchCooperativeKernel(kernel, dim3(blocks), dim3(256), args, 0, s);
        };
        if (n > kSmall) cooperative(reinterpret_cast<const void*>(&k_top), (size_t(n) + kChunk - 1) / kChunk, top_args);
        else e = cudaMemcpyAsync(B.small, &root, sizeof(root), cudaMemcpyHostToDevice, s);
        if (e == cudaSuccess)
            e = cudaFuncSetAttribute(k_small, cudaFuncAttributeMaxDynamicSharedMemorySize, int(sizeof(SmallShared)));
        if (e == cudaSuccess) {
            const int small_grid = int(std::min<size_t>((size_t(n) + 63) / 64, size_t(sms) * 16));
            k_small<<<small_grid, 32 * kSmallWarps, sizeof(SmallShared), s>>>(B);
            e = cudaGetLastError();
        }
        if (e == cudaSuccess)
            cooperative(reinterpret_cast<const void*>(&k_collapse), (size_t(n) + 127) / 128, collapse_args);
    }
    if (e == cudaSuccess) e = cudaMemcpyAsync(&ctr, B.ctr, sizeof(ctr), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    std::string err;
    if (e == cudaSuccess) {
        if (ctr.err & kErrIndex) err = "triangle index out of range";
        else if (ctr.err & kErrNonFinite) err = "non-finite vertex";
        else if (ctr.err & kErrTooDeep) err = "8-wide BVH deeper than the traversal stack";
        else if (ctr.tris != n || ctr.wide > max_wide) err = "device BVH build lost triangles";
    }
    WideNode* nodes = nullptr;
    if (e == cudaSuccess && err.empty()) {
        e = cudaMalloc(&nodes, sizeof(WideNode) * size_t(ctr.wide));
        if (e == cudaSuccess)
            e = cudaMemcpyAsync(nodes, C.nodes, sizeof(WideNode) * size_t(ctr.wide), cudaMemcpyDeviceToDevice, s);
        if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    }
    if (s) {
        cudaStreamSynchronize(s);  // after an error copies may still be under way
        cudaStreamDestroy(s);
    }
    cudaFree(scratch);
    if (e != cudaSuccess || !err.empty()) {
        cudaGetLastError();
        if (nodes) cudaFree(nodes);
        if (C.tris) cudaFree(C.tris);
        return err.empty() ? std::string("device BVH build: ") + cudaGetErrorString(e) : err;
    }
    const auto t1 = std::chrono::steady_clock::now();
    out.d_nodes = nodes;
    out.d_tris = C.tris;
    auto o2f_host = [](int i) {
        const int b = i >= 0 ? i : i ^ 0x7fffffff;
        float f;
        std::memcpy(&f, &b, 4);
        return f;
    };
    for (int a = 0; a < 3; ++a) {
        out.lo[a] = o2f_host(ctr.box[a]);
        out.hi[a] = o2f_host(ctr.box[3 + a]);
    }
    out.node_count = ctr.wide;
    out.tri_count = n;
    out.max_depth = ctr.levels;
    out.build_ms = std::chrono::duration<double, std::milli>(t1 - t0).count();
    return "";
}

}  // namespace sel
