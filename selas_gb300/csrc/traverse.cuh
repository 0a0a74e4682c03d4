// Device-side ray queries: watertight ray/triangle test and traversal of the two BVH layouts.
//
// The query contract is the one Embree gives rtcIntersect1 / rtcOccluded1
// (Middleware/embree-latest/include/embree3/rtcore_scene.h:94,118; used by
// Source/Applications/Selas/Source/PathTracer.cpp:71-139).  Intersection follows Woop, Benthin and
// Wald, "Watertight Ray/Triangle Intersection", JCGT 2(1) 2013, with every rounding step written out
// (fmaf / __fmul_rn / __fadd_rn) so that the CPU oracle, written independently with the same rounding
// steps, reproduces t, u, v bit for bit.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include "sel_internal.h"

namespace sel {

constexpr uint32_t kIterationCap = 1u << 22;  // node visits + triangle tests per ray before giving up
constexpr uint32_t kErrIterationCap = 1u;
constexpr uint32_t kErrStackOverflow = 2u;
constexpr float kBoxMargin = 1.0f / 1048576.0f;  // relative widening of the ray interval for box tests
constexpr float kOut = 1.0f / 2097152.0f;        // relative outward widening of a node's plane offsets

__device__ __forceinline__ float pick3(int k, float x, float y, float z) { return k == 0 ? x : (k == 1 ? y : z); }

struct Watertight {
    int kx, ky, kz;
    float sx, sy, sz;
};

// kz = dominant axis of |d| (ties resolved x, then y, then z); kx, ky follow cyclically and are swapped
// when d[kz] < 0 to keep the winding.
__device__ __forceinline__ Watertight watertight_setup(float dx, float dy, float dz) {
    Watertight w;
    const float ax = fabsf(dx), ay = fabsf(dy), az = fabsf(dz);
    w.kz = (ax >= ay && ax >= az) ? 0 : (ay >= az ? 1 : 2);
    w.kx = w.kz == 2 ? 0 : w.kz + 1;
    w.ky = w.kx == 2 ? 0 : w.kx + 1;
    const float dkz = pick3(w.kz, dx, dy, dz);
    if (dkz < 0.0f) { int t = w.kx; w.kx = w.ky; w.ky = t; }
    const float dkx = pick3(w.kx, dx, dy, dz), dky = pick3(w.ky, dx, dy, dz);
    w.sx = __fdiv_rn(dkx, dkz);
    w.sy = __fdiv_rn(dky, dkz);
    w.sz = __frcp_rn(dkz);
    return w;
}

// Returns true and t/u/v when the triangle is hit with tnear <= t <= tfar.
__device__ __forceinline__ bool watertight_intersect(const Watertight& w, float ox, float oy, float oz, const float4& p0,
                                                     const float4& p1, const float4& p2, float tnear, float tfar,
                                                     float& t, float& u, float& v) {
    const float a0 = __fsub_rn(p0.x, ox), a1 = __fsub_rn(p0.y, oy), a2 = __fsub_rn(p0.z, oz);
    const float b0 = __fsub_rn(p1.x, ox), b1 = __fsub_rn(p1.y, oy), b2 = __fsub_rn(p1.z, oz);
    const float c0 = __fsub_rn(p2.x, ox), c1 = __fsub_rn(p2.y, oy), c2 = __fsub_rn(p2.z, oz);
    const float Akz = pick3(w.kz, a0, a1, a2), Bkz = pick3(w.kz, b0, b1, b2), Ckz = pick3(w.kz, c0, c1, c2);
    const float Ax = fmaf(-w.sx, Akz, pick3(w.kx, a0, a1, a2));
    const float Ay = fmaf(-w.sy, Akz, pick3(w.ky, a0, a1, a2));
    const float Bx = fmaf(-w.sx, Bkz, pick3(w.kx, b0, b1, b2));
    const float By = fmaf(-w.sy, Bkz, pick3(w.ky, b0, b1, b2));
    const float Cx = fmaf(-w.sx, Ckz, pick3(w.kx, c0, c1, c2));
    const float Cy = fmaf(-w.sy, Ckz, pick3(w.ky, c0, c1, c2));
    float U = fmaf(Cx, By, -__fmul_rn(Cy, Bx));
    float V = fmaf(Ax, Cy, -__fmul_rn(Ay, Cx));
    float W = fmaf(Bx, Ay, -__fmul_rn(By, Ax));
    if (U == 0.0f || V == 0.0f || W == 0.0f) {
        // Edge case: redo the 2D edge functions exactly (products of floats are exact in double).
        U = (float)__dsub_rn(__dmul_rn((double)Cx, (double)By), __dmul_rn((double)Cy, (double)Bx));
        V = (float)__dsub_rn(__dmul_rn((double)Ax, (double)Cy), __dmul_rn((double)Ay, (double)Cx));
        W = (float)__dsub_rn(__dmul_rn((double)Bx, (double)Ay), __dmul_rn((double)By, (double)Ax));
    }
    if ((U < 0.0f || V < 0.0f || W < 0.0f) && (U > 0.0f || V > 0.0f || W > 0.0f)) return false;
    const float det = __fadd_rn(__fadd_rn(U, V), W);
    if (det == 0.0f) return false;
    const float Az = __fmul_rn(w.sz, Akz), Bz = __fmul_rn(w.sz, Bkz), Cz = __fmul_rn(w.sz, Ckz);
    const float T = fmaf(U, Az, fmaf(V, Bz, __fmul_rn(W, Cz)));
    const float rcp = __frcp_rn(det);
    const float tt = __fmul_rn(T, rcp);
    if (!(tt >= tnear && tt <= tfar)) return false;
    t = tt;
    u = __fmul_rn(V, rcp);
    v = __fmul_rn(W, rcp);
    return true;
}

// Geometric normal (v1 - v0) x (v2 - v0) with explicit rounding.
__device__ __forceinline__ float3 triangle_ng(const float4& p0, const float4& p1, const float4& p2) {
    const float e1x = __fsub_rn(p1.x, p0.x), e1y = __fsub_rn(p1.y, p0.y), e1z = __fsub_rn(p1.z, p0.z);
    const float e2x = __fsub_rn(p2.x, p0.x), e2y = __fsub_rn(p2.y, p0.y), e2z = __fsub_rn(p2.z, p0.z);
    return make_float3(fmaf(e1y, e2z, -__fmul_rn(e1z, e2y)), fmaf(e1z, e2x, -__fmul_rn(e1x, e2z)),
                       fmaf(e1x, e2y, -__fmul_rn(e1y, e2x)));
}

__device__ __forceinline__ float safe_rcp(float d) {
    return __frcp_rn(fabsf(d) > 1e-30f ? d : copysignf(1e-30f, d));
}

struct QueryRay {
    float ox, oy, oz, dx, dy, dz, tnear, tfar;
};

struct QueryHit {
    float t, u, v;
    uint32_t tri;  // index into the triangle array in leaf order (0xffffffff: no hit)
};

__device__ __forceinline__ uint64_t tri_key(const float4& p0, const float4& p1) {
    return (uint64_t(__float_as_uint(p1.w)) << 32) | uint64_t(__float_as_uint(p0.w));
}

// ---------------------------------------------------------------------------------------------------
// 8-wide quantised BVH.  Node groups on the stack are (child_base, hit bits 24..31 | imask bits 0..7);
// hit bit 24 + (slot ^ octant) so that the lowest set bit is the nearest child for this ray octant.
// A ray's traversal is a resumable per-lane state and one step (a node visit or one leaf record), so that
// the lanes of a warp can be refilled with new rays between steps (trace_stream).
// ---------------------------------------------------------------------------------------------------
struct WideState {
    float ox, oy, oz, dx, dy, dz;
    float tnear, tfar;  // tfar shrinks to the closest hit found so far
    float ix, iy, iz;
    Watertight wt;
    uint32_t oct;
    uint2 group;
    int sp;
    uint32_t iters;
    QueryHit hit;  // t is tfar
};

// A thread's traversal stack in shared memory: entry k at mem[k * stride], `depth` entries (the scene's tree
// depth: a descent pushes at most one group a level).  Sizing it to the scene leaves the rest of the SM's 256 KB
// to L1: with 12 entries instead of 24 a thread, 4 M incoherent rays over 5.2 M triangles take 1.81 ms, not 2.68
// (closest hit), and 1.22, not 1.44 (any hit).
struct WideStack {
    uint2* mem;
    int stride;
    int depth;
};

// A ray that no triangle can hit under the watertight test: a non-finite origin or direction component
// (NaN arithmetic rejects every triangle) or a zero direction (no dominant axis).  Traversing it would be
// worse than useless: with NaN slab distances fminf/fmaxf keep the interval bounds and every box is
// entered, so one such ray walks the whole tree.  The traversals return "no hit" for it at once, which is
// what the full walk returns.
__device__ __forceinline__ bool ray_untraceable(const QueryRay& r) {
    const bool finite = isfinite(r.ox) && isfinite(r.oy) && isfinite(r.oz) && isfinite(r.dx) && isfinite(r.dy) &&
                        isfinite(r.dz);
    return !finite || (r.dx == 0.0f && r.dy == 0.0f && r.dz == 0.0f);
}

__device__ __forceinline__ void wide_init(WideState& s, const QueryRay& r) {
    s.ox = r.ox; s.oy = r.oy; s.oz = r.oz;
    s.dx = r.dx; s.dy = r.dy; s.dz = r.dz;
    s.tnear = r.tnear;
    s.tfar = r.tfar;
    s.wt = watertight_setup(r.dx, r.dy, r.dz);
    s.ix = safe_rcp(r.dx); s.iy = safe_rcp(r.dy); s.iz = safe_rcp(r.dz);
    s.oct = (s.ix < 0.0f ? 4u : 0u) | (s.iy < 0.0f ? 2u : 0u) | (s.iz < 0.0f ? 1u : 0u);
    s.group = make_uint2(0u, (1u << (24 + s.oct)) | 1u);
    s.sp = 0;
    s.iters = 0;
    s.hit.tri = 0xffffffffu;
}

// Three-input minimum / maximum (one instruction on sm_100 and later); NaN operands are ignored, as by fminf / fmaxf.
__device__ __forceinline__ float max3_f32(float a, float b, float c) {
    float d;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}
__device__ __forceinline__ float min3_f32(float a, float b, float c) {
    float d;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}

// Packed FP32 pairs (sm_100 and later): two multiply-adds an instruction, each rounded once.
__device__ __forceinline__ uint64_t pack2(float a, float b) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void unpack2(uint64_t r, float& a, float& b) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(r));
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}

// 2^15 + q exactly: 0x4700qq00.
__device__ __forceinline__ float qbyte(uint32_t word, uint32_t byte) {
    return __uint_as_float(__byte_perm(word, 0x47000000u, 0x7404u | (byte << 4)));
}

// Visits the nearest pending node of s.group (which must have one): pushes the rest of the group, tests the
// node's eight child boxes, makes its hit internal children the new group and returns the triangles of its
// hit leaf children as a bit mask over records tbase..tbase+31.  Returns false on stack overflow.
//
// A plane's distance is (2^15 + q) * (scale / d) + (origin - 2^15 * scale / d): one byte permute and one
// multiply-add, the bias folded into the offset.  The offset is widened outward by 2^-21 of its magnitude.  That
// covers every rounding of the distance (three in the node's own distance p, one in the offset, one in the sum) once p
// exceeds 2^17 quanta; nearer, where p and the bias can cancel, at most 0.04 of a quantum is left uncovered, well
// within the half quantum that both builders leave between a child's planes and its box.  So no distance of the ray's
// origin loses what a box holds.  Offsets that overflow turn into infinities and NaN that the minima and maxima ignore:
// their axis then accepts every box.
__device__ __forceinline__ bool wide_visit(WideState& s, const uint4* __restrict__ nodes, const WideStack& stack,
                                           uint32_t& status, uint32_t& tmask, uint32_t& tbase) {
    const int b = __ffs(s.group.y >> 24) - 1;
    s.group.y &= ~(1u << (24 + b));
    const uint32_t slot = uint32_t(b) ^ s.oct;
    const uint32_t idx = s.group.x + __popc(s.group.y & ((1u << slot) - 1u));
    const uint4* np = nodes + size_t(idx) * 5;
    const uint4 n0 = __ldg(np), n1 = __ldg(np + 1), n2 = __ldg(np + 2), n3 = __ldg(np + 3), n4 = __ldg(np + 4);
    if (s.group.y & 0xff000000u) {
        if (s.sp >= stack.depth) { status |= kErrStackOverflow; return false; }
        stack.mem[s.sp * stack.stride] = s.group;
        ++s.sp;
    }
    const float sx = __fmul_rn(__uint_as_float((n0.w << 23) & 0x7f800000u), s.ix);
    const float sy = __fmul_rn(__uint_as_float((n0.w << 15) & 0x7f800000u), s.iy);
    const float sz = __fmul_rn(__uint_as_float((n0.w << 7) & 0x7f800000u), s.iz);
    const float ax = fmaf(-32768.0f, sx, __fmul_rn(__fsub_rn(__uint_as_float(n0.x), s.ox), s.ix));
    const float ay = fmaf(-32768.0f, sy, __fmul_rn(__fsub_rn(__uint_as_float(n0.y), s.oy), s.iy));
    const float az = fmaf(-32768.0f, sz, __fmul_rn(__fsub_rn(__uint_as_float(n0.z), s.oz), s.iz));
    // (near, far) pairs
    const uint64_t sx2 = pack2(sx, sx), sy2 = pack2(sy, sy), sz2 = pack2(sz, sz);
    const uint64_t ax2 = pack2(fmaf(-kOut, fabsf(ax), ax), fmaf(kOut, fabsf(ax), ax));
    const uint64_t ay2 = pack2(fmaf(-kOut, fabsf(ay), ay), fmaf(kOut, fabsf(ay), ay));
    const uint64_t az2 = pack2(fmaf(-kOut, fabsf(az), az), fmaf(kOut, fabsf(az), az));
    const uint32_t imask = n0.w >> 24;
    const float tnear_box = s.tnear - fabsf(s.tnear) * kBoxMargin;
    const float tfar_box = s.tfar + fabsf(s.tfar) * kBoxMargin;
    const bool px = s.ix >= 0.0f, py = s.iy >= 0.0f, pz = s.iz >= 0.0f;
    const uint32_t nx0 = px ? n2.x : n3.z, nx1 = px ? n2.y : n3.w, fx0 = px ? n3.z : n2.x, fx1 = px ? n3.w : n2.y;
    const uint32_t ny0 = py ? n2.z : n4.x, ny1 = py ? n2.w : n4.y, fy0 = py ? n4.x : n2.z, fy1 = py ? n4.y : n2.w;
    const uint32_t nz0 = pz ? n3.x : n4.z, nz1 = pz ? n3.y : n4.w, fz0 = pz ? n4.z : n3.x, fz1 = pz ? n4.w : n3.y;
    uint32_t miss = 0;  // bit c: child c's interval is empty, the sign of its length
#pragma unroll
    for (int c = 7; c >= 0; --c) {
        const uint32_t byte = uint32_t(c & 3);
        float tnx, tny, tnz, tfx, tfy, tfz;
        unpack2(fma2(pack2(qbyte(c < 4 ? nx0 : nx1, byte), qbyte(c < 4 ? fx0 : fx1, byte)), sx2, ax2), tnx, tfx);
        unpack2(fma2(pack2(qbyte(c < 4 ? ny0 : ny1, byte), qbyte(c < 4 ? fy0 : fy1, byte)), sy2, ay2), tny, tfy);
        unpack2(fma2(pack2(qbyte(c < 4 ? nz0 : nz1, byte), qbyte(c < 4 ? fz0 : fz1, byte)), sz2, az2), tnz, tfz);
        const float tmin = fmaxf(max3_f32(tnx, tny, tnz), tnear_box);
        const float tmax = fminf(min3_f32(tfx, tfy, tfz), tfar_box);
        miss = __funnelshift_l(__float_as_uint(__fsub_rn(tmax, tmin)), miss, 1);
    }
    const uint32_t hits = ~miss & 0xffu;
    uint32_t in = hits & imask, t;  // the internal hits, bit c moved to bit c ^ octant
    t = ((in >> 1) ^ in) & ((s.oct & 1u) ? 0x55u : 0u);
    in ^= t ^ (t << 1);
    t = ((in >> 2) ^ in) & ((s.oct & 2u) ? 0x33u : 0u);
    in ^= t ^ (t << 2);
    t = ((in >> 4) ^ in) & ((s.oct & 4u) ? 0x0fu : 0u);
    in ^= t ^ (t << 4);
    for (uint32_t leaf = hits & ~imask; leaf; leaf &= leaf - 1u) {
        const uint32_t meta = __byte_perm(n1.z, n1.w, __ffs(leaf) - 1) & 0xffu;
        if (meta != kLeafNone) tmask |= ((2u << (meta >> 5)) - 1u) << (meta & 31u);
    }
    s.group = make_uint2(n1.x, (in << 24) | imask);
    tbase = n1.y;
    return true;
}

// Tests leaf record ti and keeps it when it is the ray's new closest hit: t < tfar, or t == tfar and a smaller
// (geomID, primID) than the hit so far (whose record is read again then: ties are rare).  Returns whether the
// record is hit.
__device__ __forceinline__ bool wide_test(WideState& s, const float4* __restrict__ tris, uint32_t ti) {
    const float4* tp = tris + size_t(ti) * 3;
    const float4 p0 = __ldg(tp), p1 = __ldg(tp + 1), p2 = __ldg(tp + 2);
    float t, u, v;
    if (!watertight_intersect(s.wt, s.ox, s.oy, s.oz, p0, p1, p2, s.tnear, s.tfar, t, u, v)) return false;
    bool take = t < s.tfar || s.hit.tri == 0xffffffffu;
    if (!take) {
        const float4* bp = tris + size_t(s.hit.tri) * 3;
        take = tri_key(p0, p1) < tri_key(__ldg(bp), __ldg(bp + 1));
    }
    if (take) {
        s.tfar = t;
        s.hit.u = u;
        s.hit.v = v;
        s.hit.tri = ti;
    }
    return true;
}

// The flat traversal of one lane, as trace_stream and trace_packet step it.
struct WideWalk {
    static constexpr bool kAims = false;
    __device__ __forceinline__ bool aiming() const { return false; }
    WideState s;
    uint32_t tmask, tbase;  // leaf records still to test: bit k is record tbase + k

    template <typename Rays>
    __device__ __forceinline__ bool start(const QueryRay& r, const Rays&) {
        wide_init(s, r);
        tmask = 0;
        return !ray_untraceable(r);
    }

    __device__ __forceinline__ bool pending() const { return tmask != 0u; }

    // Visits the nearest pending node (there is one when no leaf record is pending).  False: the ray is given up.
    template <typename Rays>
    __device__ __forceinline__ bool visit(const Rays& rays, const WideStack& stack, uint32_t& status) {
        return wide_visit(s, rays.nodes(), stack, status, tmask, tbase);
    }

    // Tests one pending leaf record.  False: the ray is finished (any-hit: on the first hit).
    template <bool kAnyHit, typename Rays>
    __device__ __forceinline__ bool test(const Rays& rays, const WideStack&, uint32_t&) {
        const uint32_t ti = tbase + uint32_t(__ffs(tmask) - 1);
        tmask &= tmask - 1u;
        return !(wide_test(s, rays.tris(), ti) && kAnyHit);
    }

    // Ends a step: with nothing pending, goes back to the nearest node group.  False: the ray is finished.
    __device__ __forceinline__ bool advance(const WideStack& stack, uint32_t& status) {
        if (++s.iters > kIterationCap) {
            status |= kErrIterationCap;
            return false;
        }
        if (!tmask && !(s.group.y & 0xff000000u)) {
            if (s.sp == 0) return false;
            --s.sp;
            s.group = stack.mem[s.sp * stack.stride];
        }
        return true;
    }
};

// Traces a stream of rays with one warp.  The lanes step together; whenever kRefillLanes of them have finished
// (or all have), these write their results and take the next rays, so the warp neither waits for its longest ray
// nor pays a ray's set-up with few lanes.  A step visits a node in the lanes without pending leaf records, then tests
// one record in the lanes with some (and further ones while at least kTestLanes lanes test): testing all that a visit
// exposed at once would hold the other lanes up.  32 incoherent rays over 5.2 M triangles take 19 visits of 23 lanes
// and 19 record tests of 9 lanes, against 32 visits of 14 lanes and 53 tests of 3 with a packet of 32 rays and all
// records a visit.  The ballots between the phases matter beyond their masks: they bring the lanes back together,
// without them the record tests run twice (2.34 against 1.95 ms, 4 M of those rays, closest hit; 2.41 for the packet
// form).  Kernels of the wavefront (room at 1280 x 720, a bounce): closest hit 1.07 against 1.58 ms, any hit 0.52
// against 0.61.  kRefillLanes 2, 4, 6, 8, 12: 1.90, 1.82, 1.80, 1.81, 1.88 ms; a threshold following the rays' length
// lost everywhere.  kTestLanes 4, 8, 16: closest hit 2.39, 2.20, 2.13 ms, the Cornell box's path tracer (few
// nodes, many records) 24.06, 24.06, 24.31 ms.
// A Rays object gives the warp its rays:
//   bool next(b, e)        the next range of ray indices, warp-uniform, called by the whole warp; false: no more
//   bool begin(i, ray)     a lane's ray i; false: nothing to trace or to write for it
//   void end(i, state)     its result: state.hit (tri 0xffffffff: no hit, else at distance s.tfar)
//   nodes(), tris(), insts()  the lane's scene
constexpr int kRefillLanes = 8;
constexpr int kTestLanes = 16;

template <bool kAnyHit, typename Walk, typename Rays>
__device__ __forceinline__ void trace_stream(Rays& rays, const WideStack& stack, uint32_t& status) {
    const uint32_t below = (1u << (threadIdx.x & 31u)) - 1u;
    uint32_t next = 0, end = 0, id = 0;
    bool busy = false, have = false, more = true;
    Walk w;
    for (;;) {
        const uint32_t idle = __ballot_sync(0xffffffffu, !busy);
        if (idle == 0xffffffffu || (more && __popc(idle) >= kRefillLanes)) {
            if (!busy && have) {
                rays.end(id, w.s);
                have = false;
            }
            if (more && next >= end) more = rays.next(next, end);
            if (more) {
                const uint32_t mine = next + __popc(idle & below);
                next += __popc(idle);
                QueryRay r;
                if (!busy && mine < end && rays.begin(mine, r)) {
                    id = mine;
                    have = true;
                    busy = w.start(r, rays);
                }
            } else if (idle == 0xffffffffu) {
                break;
            }
        }
        if constexpr (Walk::kAims) {
            if (busy && w.aiming()) w.aim();
            __syncwarp();
        }
        if (busy && !w.pending()) busy = w.visit(rays, stack, status);
        uint32_t testing = __ballot_sync(0xffffffffu, busy && w.pending());
        while (testing) {
            if (busy && w.pending()) busy = w.template test<kAnyHit>(rays, stack, status);
            if (__popc(testing) < kTestLanes) break;
            testing = __ballot_sync(0xffffffffu, busy && w.pending());
        }
        if (busy && !w.aiming()) busy = w.advance(stack, status);
    }
}

// Traces one ray of each lane to its end: a node visit, then every leaf record that it exposed.  The lanes of a warp
// whose rays run side by side stay in step that way and share their fetches, and a batch that gives each resident
// warp only a few ranges of rays cannot refill its lanes long enough to gain from trace_stream (query.cu has the
// figures of both).  live: the lane has a ray; its result is in w.s.
template <bool kAnyHit, typename Walk, typename Rays>
__device__ __forceinline__ void trace_packet(const Rays& rays, bool live, const QueryRay& r, Walk& w,
                                             const WideStack& stack, uint32_t& status) {
    bool busy = live && w.start(r, rays);
    while (busy) {
        if constexpr (Walk::kAims) {
            if (w.aiming()) w.aim();
        }
        if (!w.pending()) busy = w.visit(rays, stack, status);
        while (busy && w.pending()) busy = w.template test<kAnyHit>(rays, stack, status);
        if (busy && !w.aiming()) busy = w.advance(stack, status);
    }
}

// The any-hit packet of a flat scene: the warp tests the records that a step exposed together, 32 (ray, record) pairs a
// round, each lane one pair with its owner's ray taken by shuffles.  Rays that part leave most lanes idle otherwise
// (300,000 surface rays over 0.33 M triangles 117 against 122 us, 500,000 camera rays over 10,000 triangles 32 against
// 42).  For closest hits the shuffles and result slots cost what the fuller warps save.  Called by the whole warp; only
// the fact of a hit is reported (s.hit.tri is not the record's index).
__device__ __forceinline__ void trace_packet_any(const uint4* __restrict__ nodes, const float4* __restrict__ tris,
                                                 bool live, const QueryRay& r, WideState& s, const WideStack& stack,
                                                 uint32_t& status) {
    wide_init(s, r);
    bool busy = live && !ray_untraceable(r);
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t axes = uint32_t(s.wt.kx) | (uint32_t(s.wt.ky) << 2) | (uint32_t(s.wt.kz) << 4);
    while (__any_sync(0xffffffffu, busy)) {
        uint32_t tmask = 0, tbase = 0;
        if (busy && !wide_visit(s, nodes, stack, status, tmask, tbase)) {
            busy = false;
            tmask = 0;
        }
        // lane L owns pairs [first, last) of the warp's concatenation: its records in ascending order
        uint32_t last = __popc(tmask);
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, last, o);
            if (lane >= uint32_t(o)) last += y;
        }
        const uint32_t first = last - __popc(tmask), total = __shfl_sync(0xffffffffu, last, 31);
        for (uint32_t base = 0; base < total; base += 32) {
            const uint32_t j = base + lane;
            uint32_t owner = 0;  // the first lane whose last exceeds j
#pragma unroll
            for (uint32_t step = 16; step >= 1; step >>= 1) {
                const uint32_t e = __shfl_sync(0xffffffffu, last, int(owner + step - 1));
                if (e <= j) owner += step;
            }
            const int from = int(owner);
            const uint32_t o_mask = __shfl_sync(0xffffffffu, tmask, from);
            const uint32_t o_base = __shfl_sync(0xffffffffu, tbase, from);
            const uint32_t o_first = __shfl_sync(0xffffffffu, first, from);
            const uint32_t o_axes = __shfl_sync(0xffffffffu, axes, from);
            Watertight w;
            w.kx = int(o_axes & 3u);
            w.ky = int((o_axes >> 2) & 3u);
            w.kz = int((o_axes >> 4) & 3u);
            w.sx = __shfl_sync(0xffffffffu, s.wt.sx, from);
            w.sy = __shfl_sync(0xffffffffu, s.wt.sy, from);
            w.sz = __shfl_sync(0xffffffffu, s.wt.sz, from);
            const float ox = __shfl_sync(0xffffffffu, s.ox, from), oy = __shfl_sync(0xffffffffu, s.oy, from);
            const float oz = __shfl_sync(0xffffffffu, s.oz, from);
            const float tnear = __shfl_sync(0xffffffffu, s.tnear, from);
            const float tfar = __shfl_sync(0xffffffffu, s.tfar, from);
            bool got = false;
            const uint32_t bit = j < total ? __fns(o_mask, 0u, int(j - o_first) + 1) : 0xffffffffu;
            if (bit < 32u) {
                const float4* tp = tris + size_t(o_base + bit) * 3;
                const float4 p0 = __ldg(tp), p1 = __ldg(tp + 1), p2 = __ldg(tp + 2);
                float t, u, v;
                got = watertight_intersect(w, ox, oy, oz, p0, p1, p2, tnear, tfar, t, u, v);
            }
            const uint32_t hits = __ballot_sync(0xffffffffu, got);
            const uint32_t a = first > base ? first : base, b = last < base + 32 ? last : base + 32;  // own pairs
            if (busy && a < b && ((hits >> (a - base)) & (0xffffffffu >> (32u - (b - a))))) {
                s.hit.tri = 0u;
                busy = false;
            }
        }
        if (busy && ++s.iters > kIterationCap) {
            status |= kErrIterationCap;
            busy = false;
        }
        if (busy && !(s.group.y & 0xff000000u)) {
            if (s.sp == 0) {
                busy = false;
            } else {
                --s.sp;
                s.group = stack.mem[s.sp * stack.stride];
            }
        }
    }
}

// Traces one ray with eight lanes: the lanes of an aligned group of eight hold the same ray and stack (each its own
// copy), test one child box each and up to eight leaf records at once.  A lone warp takes about 1,100 cycles for the
// 280 dependent instructions of wide_visit, so batches too short to fill the GPU with one lane per ray wait for
// arithmetic, not memory.  Called by all eight lanes; s.hit is the same in all of them.
template <bool kAnyHit>
__device__ __forceinline__ void trace_group(const uint4* __restrict__ nodes, const float4* __restrict__ tris,
                                            const QueryRay& r, WideState& s, const WideStack& stack,
                                            uint32_t& status) {
    const uint32_t lane = threadIdx.x & 31u, child = lane & 7u, first = lane & 24u;
    const uint32_t group_mask = 0xffu << first;
    wide_init(s, r);
    if (ray_untraceable(r)) return;
    const bool px = s.ix >= 0.0f, py = s.iy >= 0.0f, pz = s.iz >= 0.0f;
    const float tnear_box = s.tnear - fabsf(s.tnear) * kBoxMargin;
    for (;;) {
        const int b = __ffs(s.group.y >> 24) - 1;
        s.group.y &= ~(1u << (24 + b));
        const uint32_t slot = uint32_t(b) ^ s.oct;
        const uint4* np = nodes + size_t(s.group.x + __popc(s.group.y & ((1u << slot) - 1u))) * 5;
        const uint4 n0 = __ldg(np), n1 = __ldg(np + 1), n2 = __ldg(np + 2), n3 = __ldg(np + 3), n4 = __ldg(np + 4);
        if (s.group.y & 0xff000000u) {
            if (s.sp >= stack.depth) { status |= kErrStackOverflow; return; }
            stack.mem[s.sp * stack.stride] = s.group;
            ++s.sp;
        }
        const float sx = __fmul_rn(__uint_as_float((n0.w << 23) & 0x7f800000u), s.ix);
        const float sy = __fmul_rn(__uint_as_float((n0.w << 15) & 0x7f800000u), s.iy);
        const float sz = __fmul_rn(__uint_as_float((n0.w << 7) & 0x7f800000u), s.iz);
        const float ax = __fmul_rn(__fsub_rn(__uint_as_float(n0.x), s.ox), s.ix);
        const float ay = __fmul_rn(__fsub_rn(__uint_as_float(n0.y), s.oy), s.iy);
        const float az = __fmul_rn(__fsub_rn(__uint_as_float(n0.z), s.oz), s.iz);
        auto plane = [&](uint32_t w0, uint32_t w1) { return __uint2float_rn(__byte_perm(w0, w1, child) & 0xffu); };
        const float lx = plane(n2.x, n2.y), hx = plane(n3.z, n3.w);
        const float ly = plane(n2.z, n2.w), hy = plane(n4.x, n4.y);
        const float lz = plane(n3.x, n3.y), hz = plane(n4.z, n4.w);
        const float tnx = fmaf(px ? lx : hx, sx, fmaf(-kOut, fabsf(ax), ax));
        const float tfx = fmaf(px ? hx : lx, sx, fmaf(kOut, fabsf(ax), ax));
        const float tny = fmaf(py ? ly : hy, sy, fmaf(-kOut, fabsf(ay), ay));
        const float tfy = fmaf(py ? hy : ly, sy, fmaf(kOut, fabsf(ay), ay));
        const float tnz = fmaf(pz ? lz : hz, sz, fmaf(-kOut, fabsf(az), az));
        const float tfz = fmaf(pz ? hz : lz, sz, fmaf(kOut, fabsf(az), az));
        const float tfar_box = s.tfar + fabsf(s.tfar) * kBoxMargin;
        const float tmin = fmaxf(max3_f32(tnx, tny, tnz), tnear_box);
        const float tmax = fminf(min3_f32(tfx, tfy, tfz), tfar_box);
        const uint32_t imask = n0.w >> 24;
        const uint32_t meta = __byte_perm(n1.z, n1.w, child) & 0xffu;
        const bool hit = !(tmax < tmin);
        uint32_t in = (__ballot_sync(group_mask, hit) >> first) & imask, t;
        t = ((in >> 1) ^ in) & ((s.oct & 1u) ? 0x55u : 0u);
        in ^= t ^ (t << 1);
        t = ((in >> 2) ^ in) & ((s.oct & 2u) ? 0x33u : 0u);
        in ^= t ^ (t << 2);
        t = ((in >> 4) ^ in) & ((s.oct & 4u) ? 0x0fu : 0u);
        in ^= t ^ (t << 4);
        uint32_t tmask = __reduce_or_sync(
            group_mask, hit && meta != kLeafNone ? ((2u << (meta >> 5)) - 1u) << (meta & 31u) : 0u);
        s.group = make_uint2(n1.x, (in << 24) | imask);
        while (tmask) {  // the eight lowest records, one a lane
            uint32_t m = tmask;
            for (uint32_t k = 0; k < child; ++k) m &= m - 1u;
            const uint32_t last = __shfl_sync(group_mask, m, int(first + 7u));
            tmask = last & (last - 1u);
            float ht = 0.0f, hu = 0.0f, hv = 0.0f;
            uint32_t ti = 0;
            uint64_t key = ~0ull;
            bool got = false;
            if (m) {
                ti = n1.y + uint32_t(__ffs(m) - 1);
                const float4* tp = tris + size_t(ti) * 3;
                const float4 p0 = __ldg(tp), p1 = __ldg(tp + 1), p2 = __ldg(tp + 2);
                got = watertight_intersect(s.wt, s.ox, s.oy, s.oz, p0, p1, p2, s.tnear, s.tfar, ht, hu, hv);
                if (got) key = tri_key(p0, p1);
            }
            const uint32_t any = __ballot_sync(group_mask, got);
            if (!any) continue;
            if (kAnyHit) {
                s.hit.tri = 0u;  // only the fact of a hit is reported
                return;
            }
            // the group's closest: smallest t (-0 as 0), then smallest (geomID, primID)
            const int tb = __float_as_int(__fadd_rn(ht, 0.0f));
            const int ordered = got ? (tb >= 0 ? tb : tb ^ 0x7fffffff) : 0x7fffffff;
            const int least = __reduce_min_sync(group_mask, ordered);
            uint32_t win = __ballot_sync(group_mask, got && ordered == least);
            if (win & (win - 1u)) {
                uint64_t k = got && ordered == least ? key : ~0ull, low = k;
                for (int o = 1; o < 8; o <<= 1) {
                    const uint64_t other = __shfl_xor_sync(group_mask, low, o);
                    low = other < low ? other : low;
                }
                win = __ballot_sync(group_mask, got && ordered == least && k == low);
            }
            const int w = __ffs(win) - 1;
            const float wt = __shfl_sync(group_mask, ht, w), wu = __shfl_sync(group_mask, hu, w);
            const float wv = __shfl_sync(group_mask, hv, w);
            const uint32_t wi = __shfl_sync(group_mask, ti, w);
            const uint64_t wk = __shfl_sync(group_mask, key, w);
            bool take = wt < s.tfar || s.hit.tri == 0xffffffffu;
            if (!take) {
                const float4* bp = tris + size_t(s.hit.tri) * 3;
                take = wk < tri_key(__ldg(bp), __ldg(bp + 1));
            }
            if (take) {
                s.tfar = wt;
                s.hit.u = wu;
                s.hit.v = wv;
                s.hit.tri = wi;
            }
        }
        if (++s.iters > kIterationCap) { status |= kErrIterationCap; return; }
        if (!(s.group.y & 0xff000000u)) {
            if (s.sp == 0) return;
            --s.sp;
            s.group = stack.mem[s.sp * stack.stride];
        }
    }
}

// Queues of at most kGroupWaves rays a group of eight lanes of the launched warps take trace_groups: 58,368 rays on
// 152 SMs, where both forms take the same time (above; 1, 3, 8 rays a group: VCM room passes 13.00, 12.73, 13.23 ms).
constexpr uint32_t kGroupWaves = 3;
__device__ __forceinline__ bool short_queue(uint32_t n) {
    return n <= kGroupWaves * 4u * (gridDim.x * (blockDim.x >> 5));
}

// The rays of a short queue, a group of eight lanes each: the first lane of a group begins and ends its ray.
template <bool kAnyHit, typename Rays>
__device__ __forceinline__ void trace_groups(Rays& rays, uint32_t n, const WideStack& stack, uint32_t& status) {
    const uint32_t lane = threadIdx.x & 31u, first = lane & 24u;
    const uint32_t group_mask = 0xffu << first;
    const uint32_t group = (blockIdx.x * blockDim.x + threadIdx.x) >> 3, groups = (gridDim.x * blockDim.x) >> 3;
    for (uint32_t i = group; i < n; i += groups) {
        QueryRay r{};
        bool live = false;
        if (lane == first) live = rays.begin(i, r);
        if (!__ballot_sync(group_mask, live)) continue;
        float* f = reinterpret_cast<float*>(&r);
#pragma unroll
        for (int k = 0; k < int(sizeof(QueryRay) / sizeof(float)); ++k) f[k] = __shfl_sync(group_mask, f[k], int(first));
        const uint64_t nodes = __shfl_sync(group_mask, reinterpret_cast<uint64_t>(rays.nodes()), int(first));
        const uint64_t tris = __shfl_sync(group_mask, reinterpret_cast<uint64_t>(rays.tris()), int(first));
        WideState s;
        trace_group<kAnyHit>(reinterpret_cast<const uint4*>(nodes), reinterpret_cast<const float4*>(tris), r, s, stack,
                             status);
        if (lane == first) rays.end(i, s);
    }
}

// Ray ranges of a queue of n entries for the persistent kernels: every warp's first range is its own, then warps
// take further ones through an atomic cursor (which starts at 0).  Short queues are spread over all warps, so
// that few lanes of many warps trace them rather than all lanes of a few, and need no atomics.
struct QueueRanges {
    uint32_t n, chunk, first, rest;
    uint32_t* cursor;
    bool started;

    __device__ __forceinline__ QueueRanges(uint32_t count, uint32_t* cur) : n(count), cursor(cur), started(false) {
        const uint32_t warps = gridDim.x * (blockDim.x >> 5);
        const uint32_t warp = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
        chunk = (n + warps - 1) / warps;
        chunk = chunk < 32u ? (chunk ? chunk : 1u) : 32u;
        first = warp * chunk;
        rest = warps * chunk;
    }
    __device__ __forceinline__ bool next(uint32_t& b, uint32_t& e) {
        if (!started) {
            started = true;
            b = first;
        } else {
            if (rest >= n) return false;
            b = 0;
            if ((threadIdx.x & 31u) == 0) b = rest + atomicAdd(cursor, chunk);
            b = __shfl_sync(0xffffffffu, b, 0);
        }
        e = b + chunk < n ? b + chunk : n;
        return b < n;
    }
};

// ---------------------------------------------------------------------------------------------------
// Binary FP32 BVH (the plain GPU path): classic stack traversal, nearer child first.
// `stack` points at this thread's first int entry; entries are `stride` ints apart.
// ---------------------------------------------------------------------------------------------------
template <bool kAnyHit>
__device__ __forceinline__ bool trace_binary(const float4* __restrict__ nodes, const float4* __restrict__ tris,
                                             const QueryRay& r, QueryHit& hit, int* stack, int stride,
                                             uint32_t& status) {
    if (ray_untraceable(r)) {
        hit.tri = 0xffffffffu;
        return false;
    }
    const Watertight wt = watertight_setup(r.dx, r.dy, r.dz);
    const float ix = safe_rcp(r.dx), iy = safe_rcp(r.dy), iz = safe_rcp(r.dz);
    const float oix = __fmul_rn(r.ox, ix), oiy = __fmul_rn(r.oy, iy), oiz = __fmul_rn(r.oz, iz);
    const float tnear_box = r.tnear - fabsf(r.tnear) * kBoxMargin;
    float tfar = r.tfar;
    float tfar_box = tfar + fabsf(tfar) * kBoxMargin;
    uint64_t best_key = ~0ull;
    bool found = false;
    hit.tri = 0xffffffffu;
    const bool nx = ix < 0.0f, ny = iy < 0.0f, nz = iz < 0.0f;

    int node = 0;
    int sp = 0;
    uint32_t iters = 0;
    for (;;) {
        if (++iters > kIterationCap) { status |= kErrIterationCap; break; }
        const float4* np = nodes + size_t(node) * 4;
        const float4 a = __ldg(np), b = __ldg(np + 1), c = __ldg(np + 2);
        const int4 refs = __ldg(reinterpret_cast<const int4*>(np + 3));
        // child 0
        const float t0nx = fmaf(nx ? a.y : a.x, ix, -oix), t0fx = fmaf(nx ? a.x : a.y, ix, -oix);
        const float t0ny = fmaf(ny ? a.w : a.z, iy, -oiy), t0fy = fmaf(ny ? a.z : a.w, iy, -oiy);
        const float t0nz = fmaf(nz ? c.y : c.x, iz, -oiz), t0fz = fmaf(nz ? c.x : c.y, iz, -oiz);
        const float t1nx = fmaf(nx ? b.y : b.x, ix, -oix), t1fx = fmaf(nx ? b.x : b.y, ix, -oix);
        const float t1ny = fmaf(ny ? b.w : b.z, iy, -oiy), t1fy = fmaf(ny ? b.z : b.w, iy, -oiy);
        const float t1nz = fmaf(nz ? c.w : c.z, iz, -oiz), t1fz = fmaf(nz ? c.z : c.w, iz, -oiz);
        const float tmin0 = fmaxf(fmaxf(t0nx, t0ny), fmaxf(t0nz, tnear_box));
        const float tmax0 = fminf(fminf(t0fx, t0fy), fminf(t0fz, tfar_box));
        const float tmin1 = fmaxf(fmaxf(t1nx, t1ny), fmaxf(t1nz, tnear_box));
        const float tmax1 = fminf(fminf(t1fx, t1fy), fminf(t1fz, tfar_box));
        bool h0 = tmin0 <= tmax0 && refs.z >= 0;
        bool h1 = tmin1 <= tmax1 && refs.w >= 0;
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            const bool hk = k == 0 ? h0 : h1;
            const int cnt = k == 0 ? refs.z : refs.w;
            if (!hk || cnt <= 0) continue;
            const int first = k == 0 ? refs.x : refs.y;
            for (int i = 0; i < cnt; ++i) {
                const float4* tp = tris + size_t(first + i) * 3;
                const float4 p0 = __ldg(tp), p1 = __ldg(tp + 1), p2 = __ldg(tp + 2);
                float t, u, v;
                if (watertight_intersect(wt, r.ox, r.oy, r.oz, p0, p1, p2, r.tnear, tfar, t, u, v)) {
                    if (kAnyHit) {
                        hit.t = t; hit.u = u; hit.v = v; hit.tri = uint32_t(first + i);
                        return true;
                    }
                    const uint64_t key = tri_key(p0, p1);
                    if (t < tfar || key < best_key) {
                        tfar = t;
                        tfar_box = tfar + fabsf(tfar) * kBoxMargin;
                        best_key = key;
                        hit.t = t; hit.u = u; hit.v = v; hit.tri = uint32_t(first + i);
                        found = true;
                    }
                }
            }
            if (k == 0) h0 = false; else h1 = false;
        }
        if (h0 && h1) {
            const bool first0 = tmin0 <= tmin1;
            if (sp >= kBinaryStack) { status |= kErrStackOverflow; break; }
            stack[sp * stride] = first0 ? refs.y : refs.x;
            ++sp;
            node = first0 ? refs.x : refs.y;
        } else if (h0) {
            node = refs.x;
        } else if (h1) {
            node = refs.y;
        } else {
            if (sp == 0) break;
            --sp;
            node = stack[sp * stride];
        }
    }
    return found;
}

}  // namespace sel
