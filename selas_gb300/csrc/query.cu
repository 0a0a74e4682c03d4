// Ray-query kernels over SelRay / SelRayHit records (Embree's RTCRay / RTCRayHit layouts) and their launchers.  A ray
// is traced by one lane or, in small batches, by eight; each thread keeps its traversal stack in shared memory.
#include "query.h"

#include <type_traits>

#include "hitref.cuh"
#include "instance.cuh"
#include "radix.cuh"
#include "scan.cuh"
#include "traverse.cuh"

namespace sel {

namespace {

constexpr int kQueryBlock = 128;  // the binary layout's blocks

__device__ __forceinline__ QueryRay load_ray(const float4* rp) {
    const float4 a = rp[0], b = rp[1], c = rp[2];
    QueryRay r;
    r.ox = a.x; r.oy = a.y; r.oz = a.z; r.tnear = a.w;
    r.dx = b.x; r.dy = b.y; r.dz = b.z;
    r.tfar = c.x;
    return r;
}

// The hit as Embree reports it.  A quad's triangles are stored as records 2q (v0, v1, v3) and 2q + 1
// (v2, v3, v1) with kind kTriQuadHalf: primID is q and the second triangle's (u', v') become (1 - u', 1 - v')
// (RTC_GEOMETRY_TYPE_QUAD.3embree3); Ng is the hit triangle's.
__device__ __forceinline__ void embree_hit(const float4& p0, const float4& p2, float& u, float& v, uint32_t& prim) {
    prim = __float_as_uint(p0.w);
    if (__float_as_uint(p2.w) == kTriQuadHalf) {
        if (prim & 1u) {
            u = __fsub_rn(1.0f, u);
            v = __fsub_rn(1.0f, v);
        }
        prim >>= 1;
    }
}

__device__ __forceinline__ void store_hit(SelRayHit* rh, const float4* __restrict__ tris, const QueryHit& h) {
    const float4* tp = tris + size_t(h.tri) * 3;
    const float4 p0 = __ldg(tp), p1 = __ldg(tp + 1), p2 = __ldg(tp + 2);
    const float3 ng = triangle_ng(p0, p1, p2);
    float u = h.u, v = h.v;
    uint32_t prim;
    embree_hit(p0, p2, u, v, prim);
    float* base = reinterpret_cast<float*>(rh);
    base[8] = h.t;  // ray.tfar
    float4* hp = reinterpret_cast<float4*>(base + 12);
    hp[0] = make_float4(ng.x, ng.y, ng.z, u);
    hp[1] = make_float4(v, __uint_as_float(prim), p1.w, __uint_as_float(SEL_INVALID_GEOMETRY_ID));
    reinterpret_cast<uint32_t*>(base)[20] = SEL_INVALID_GEOMETRY_ID;
}

__device__ __forceinline__ void store_hit_instanced(SelRayHit* rh, const InstHit& h) {
    const float4* tp = h.tris + size_t(h.tri) * 3;
    const float4 p0 = __ldg(tp), p1 = __ldg(tp + 1), p2 = __ldg(tp + 2);
    // object space of the hit mesh (a curve segment's from the ray, curve.cuh)
    float3 ng;
    if (__float_as_uint(p2.w) == kTriCurve) {
        const float* ray = reinterpret_cast<const float*>(rh);
        ng = record_ng(tp, p0, p1, p2, h.rec[0], h.rec[1], make_float3(ray[0], ray[1], ray[2]),
                       make_float3(ray[4], ray[5], ray[6]), h.t, h.u);
    } else {
        ng = triangle_ng(p0, p1, p2);
    }
    float u = h.u, v = h.v;
    uint32_t prim;
    embree_hit(p0, p2, u, v, prim);
    float* base = reinterpret_cast<float*>(rh);
    base[8] = h.t;
    float4* hp = reinterpret_cast<float4*>(base + 12);
    hp[0] = make_float4(ng.x, ng.y, ng.z, u);
    hp[1] = make_float4(v, __uint_as_float(prim), p1.w, __uint_as_float(h.inst[0]));
    reinterpret_cast<uint32_t*>(base)[20] = h.inst[1];
}

// ---------------------------------------------------------------------------------------------------
// 8-wide traversal.  Blocks are one warp; 64 registers let 32 of them run on an SM.  Which form a batch takes follows
// its size, in rays for each warp that runs at once, and, where the size does not settle it, a look at the warp's own
// rays (side_by_side).  Device times in us over 10 k | 0.33 M | 5.2 M triangles; "surface" rays bounce off random
// points, "camera" rays are a frame's in pixel order.
//   Eight lanes a ray (trace_group) up to kGroupRays, and to kSideGroupRays for rays side by side.  Against packets:
//     24,000 surface   closest  32 | 53 | 70 against 34 | 59 | 77   any  27 | 39 | 54 against 28 | 46 | 62
//     45,000 surface   closest  43 | 74 | 94 against 36 | 66 | 90   any  36 | 51 | 74 against 31 | 47 | 74
//     58,368 camera    closest  22 | 38 | 62 against 26 | 52 | 77   any  19 | 29 | 48 against 23 | 36 | 64
//     90,000 camera    closest  26 | 46 | 88 against 28 | 54 | 106  any  22 | 36 | 55 against 20 | 44 | 60
//     116,736 camera   closest  32 | 54 | 94 against 29 | 52 | 101  any  28 | 37 | 62 against 22 | 38 | 62
//   (from 34,500 to 45,000 surface rays the packets gain on seven scenes of up to 0.5 M triangles, 1.05 times in the
//   middle; over 1.2 and 2.4 M triangles the groups lead up to kLargeGroupRays, 39,500 rays closest hit 82 and 74
//   against 77 and 90, any hit 60 and 65 against 72 and 76, and over 5.2 M neither does, 92 and 72 against 91 and 69).
//   A lane a ray, side by side to the end (trace_packet), up to kPacketRays, and at any size for rays side by side.
//   Against streams:
//     90,000 surface   closest  41 | 73 | 117 against 47 | 93 | 131        any  34 | 52 | 97 against 43 | 67 | 119
//     300,000 surface  closest  88 | 138 | 253 against 96 | 145 | 257      any  74 | 117 | 213 against 82 | 126 | 210
//     500,000 surface  closest  137 | 200 | 379 against 140 | 206 | 350    any  114 | 162 | 279 against 117 | 163 | 282
//     4.2 M surface    closest  960 | 1404 | 2598 against 890 | 1210 | 2048
//                      any  794 | 1103 | 1844 against 720 | 940 | 1470
//     1 M camera       closest  52 | 113 | 273 against 73 | 145 | 272      any  40 | 86 | 164 against 58 | 105 | 192
//   Streams of rays (trace_stream) otherwise, and, over more than a million triangles, for closest hits of more than
//   kLargeLookRays whatever the rays: there both forms trace camera rays alike (2 M 372 against 370 us, 4.2 M
//   from four places 511 | 533 | 560 | 595 against 515 | 553 | 555 | 580) and parting rays are spared the look.
// Scenes with instances: streams, but for kInstStreamRays to 32 rays a warp, where rays that part are packets (40,000
// random rays, closest hit over 20 | 500 | 2000 instances 46 | 92 | 174 against 45 | 99 | 181, any hit 36 | 73 | 114
// against 41 | 84 | 125; camera rays, which meet different instances from lane to lane, stay streams: 170 against 156
// us as packets over 500 instances, and 4 M of them 3.0 against 2.6 ms).  Scenes with curves stay streams, one segment
// a step (40,000 random rays over 22,000 segments 2.2 ms, as packets 3.5).
//
// Records in host memory, traced in place (far): the link carries every look, so eight looks at a record cost more than
// any form (45,000 camera rays, closest hit over 0.33 M triangles: a call of 161 us with them, 66 as groups, 82 as
// packets). Groups up to kFarGroupRays (58,368 rays surface, packets against groups: closest 78 | 107 | 131 against 73
// | 95 | 144, any 60 | 71 | 105 against 60 | 75 | 105; camera 64 | 93 | 117 against 60 | 79 | 93, any 50 | 63 | 87
// against 36 | 44 | 65), then packets; closest hits are streams, without a look, from kFarPacketRays on (300,000 camera
// rays 303 | 321 | 329 against 315 | 326 | 343 us as packets, surface 238 | 277 | 357 against 233 | 276 | 372).
//
// A stream's warp starts with its block's records, block index k standing for records [32 k, 32 k + 32).  A warp whose
// lanes run out of rays takes over the block index of a block that has not started (cluster launch control) and
// refills its finished lanes from it, so a batch of any size is balanced without a work counter in
// memory, on any number of streams at once and under graph capture.  The next index is requested while the
// warp still traces the last, which hides the answer's latency.  An atomic counter in place of the block indices
// measured 3 % faster (4 M incoherent rays over 5.2 M triangles, closest hit 1.81 against 1.87 ms) but would have to
// be allocated and zeroed by every call.
// 64 registers, 32 warps per SM: with 36 (56 registers) closest hit takes 1.89 against 1.81 ms and any hit 1.34
// against 1.22, with 40 (48 registers) 2.08 and 1.46.
// ---------------------------------------------------------------------------------------------------
constexpr uint32_t kWarpsPerSm = 32, kInstWarpsPerSm = 16;
template <bool kAnyHit>
constexpr uint32_t kGroupRays = kAnyHit ? 7 : 8;
constexpr uint32_t kLargeGroupRays = 9, kLargeLookRays = 256, kLargeScene = 1u << 20;  // triangles
constexpr uint32_t kSideGroupRays = 20, kPacketRays = 64, kInstStreamRays = 2, kFarGroupRays = 12, kFarPacketRays = 32;
constexpr uint32_t kErrClaimTimeout = 32u;  // the answer to a work request never came

__device__ __forceinline__ uint32_t shared_address(const void* p) { return uint32_t(__cvta_generic_to_shared(p)); }

// The ranges of records a warp traces.
struct RecordRanges {
    uint32_t n, status;
    bool claim, started;     // claim: takes over blocks that have not started
    uint32_t phase;
    uint32_t answer, barrier;  // shared memory: 16-byte answer, its mbarrier

    __device__ __forceinline__ explicit RecordRanges(uint32_t count)
        : n(count), status(0), claim(false), started(false), phase(0), answer(0), barrier(0) {}

    __device__ __forceinline__ void take_over(const uint4* ans, const uint64_t* bar) {
        claim = true;
        answer = shared_address(ans);
        barrier = shared_address(bar);
        if ((threadIdx.x & 31u) == 0) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(barrier) : "memory");
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        }
        __syncwarp();
        request();
    }

    __device__ __forceinline__ void request() {
        if ((threadIdx.x & 31u) != 0) return;
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // the last answer was read
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], 16;" ::"r"(barrier) : "memory");
        asm volatile("clusterlaunchcontrol.try_cancel.async.shared::cta.mbarrier::complete_tx::bytes.b128 [%0], [%1];"
                     ::"r"(answer), "r"(barrier) : "memory");
    }

    // The whole warp: waits for the answer; true and a block index when a block was taken over.  After a refusal
    // no further request is made (there is nothing left to take).
    __device__ __forceinline__ bool claimed(uint32_t& block) {
        uint32_t done = 0;
        for (uint32_t k = 0; k < (1u << 20) && !done; ++k)
            asm volatile("{\n\t.reg .pred p;\n\t"
                         "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
                         "selp.u32 %0, 1, 0, p;\n\t}"
                         : "=r"(done) : "r"(barrier), "r"(phase) : "memory");
        if (!done) {
            status |= kErrClaimTimeout;
            return false;
        }
        phase ^= 1u;
        uint32_t got = 0;
        asm volatile("{\n\t.reg .b128 a;\n\t.reg .pred p;\n\t.reg .b64 lo, hi;\n\t"
                     "ld.shared.v2.b64 {lo, hi}, [%2];\n\tmov.b128 a, {lo, hi};\n\t"
                     "clusterlaunchcontrol.query_cancel.is_canceled.pred.b128 p, a;\n\t"
                     "selp.u32 %0, 1, 0, p;\n\tmov.u32 %1, 0;\n\t"
                     "@p clusterlaunchcontrol.query_cancel.get_first_ctaid::x.b32.b128 %1, a;\n\t}"
                     : "=r"(got), "=r"(block) : "r"(answer) : "memory");
        __syncwarp();
        return got != 0;
    }

    __device__ __forceinline__ bool next(uint32_t& b, uint32_t& e) {
        uint32_t block = blockIdx.x;
        if (started) {
            if (!claim) return false;
            if (!claimed(block)) {
                claim = false;
                return false;
            }
            request();
        }
        started = true;
        b = block * 32u;
        e = n - b < 32u ? n : b + 32u;
        return true;
    }
};

template <bool kAnyHit, bool kInst>
struct RecordRays : RecordRanges {
    const uint4* node_array;
    const float4* tri_array;
    const InstanceRecord* inst_array;
    float4* recs;
    uint32_t record_float4s;
    const uint32_t* order;  // null: records in their own order

    using RecordRanges::RecordRanges;

    __device__ __forceinline__ const uint4* nodes() const { return node_array; }
    __device__ __forceinline__ const float4* tris() const { return tri_array; }
    __device__ __forceinline__ const InstanceRecord* insts() const { return inst_array; }
    __device__ __forceinline__ float4* record(uint32_t i) const {
        return recs + size_t(order ? order[i] : i) * record_float4s;
    }
    __device__ __forceinline__ bool begin(uint32_t i, QueryRay& r) const {
        r = load_ray(record(i));
        return true;
    }
    __device__ __forceinline__ void end(uint32_t i, WideState& s) const {
        if (s.hit.tri == 0xffffffffu) return;
        float4* rec = record(i);
        if constexpr (kAnyHit) {
            reinterpret_cast<float*>(rec)[8] = -__int_as_float(0x7f800000);
        } else {
            s.hit.t = s.tfar;
            store_hit(reinterpret_cast<SelRayHit*>(rec), tri_array, s.hit);
        }
    }
    __device__ __forceinline__ void end(uint32_t i, InstState& s) const {
        if (s.hit.tri == 0xffffffffu) return;
        float4* rec = record(i);
        if constexpr (kAnyHit) reinterpret_cast<float*>(rec)[8] = -__int_as_float(0x7f800000);
        else store_hit_instanced(reinterpret_cast<SelRayHit*>(rec), s.hit);
    }
};

struct QueryArgs {
    const uint4* nodes;
    const float4* tris;
    const InstanceRecord* insts;
    float4* rays;
    uint32_t record_float4s, n;
    const uint32_t* order;  // with ctl: the records' order, used when ctl[0] is non-zero
    const uint32_t* ctl;
    int stack_depth;
    uint32_t claim;         // streams take over blocks that have not started
    float reach2;           // side_by_side: the square of the distance between neighbours' origins
    uint32_t* err;
};

template <bool kAnyHit, bool kInst>
__device__ __forceinline__ RecordRays<kAnyHit, kInst> query_records(const QueryArgs& a) {
    RecordRays<kAnyHit, kInst> rays(a.n);
    rays.node_array = a.nodes;
    rays.tri_array = a.tris;
    rays.inst_array = a.insts;
    rays.recs = a.rays;
    rays.record_float4s = a.record_float4s;
    rays.order = a.ctl && a.ctl[0] ? a.order : nullptr;
    return rays;
}

// Whether a warp's rays (lanes 0 .. count - 1) run side by side: three of four neighbours start within a thirty-second
// of the scene's diagonal of one another and point within about 2.5 degrees of one another.
__device__ __forceinline__ bool side_by_side(const QueryRay& r, uint32_t count, float reach2) {
    float v[6] = {r.ox, r.oy, r.oz, r.dx, r.dy, r.dz}, w[6];
#pragma unroll
    for (int k = 0; k < 6; ++k) w[k] = __shfl_down_sync(0xffffffffu, v[k], 1);
    const float ex = w[0] - v[0], ey = w[1] - v[1], ez = w[2] - v[2];
    const float d = v[3] * w[3] + v[4] * w[4] + v[5] * w[5];
    const float nn = (v[3] * v[3] + v[4] * v[4] + v[5] * v[5]) * (w[3] * w[3] + w[4] * w[4] + w[5] * w[5]);
    const bool close = (threadIdx.x & 31u) + 1 < count && ex * ex + ey * ey + ez * ez <= reach2 && nn > 0.0f &&
                       d > 0.0f && d * d > 0.998f * nn;
    return 4 * __popc(__ballot_sync(0xffffffffu, close)) >= 3 * int(count - 1);
}

// The rays of records [base, base + 32), a lane each; count of them exist.
template <bool kAnyHit, bool kInst>
struct Packet {
    QueryRay r;
    uint32_t base, count;
    __device__ __forceinline__ Packet(const RecordRays<kAnyHit, kInst>& rays, uint32_t first)
        : r{}, base(first), count(rays.n - first < 32u ? rays.n - first : 32u) {
        if (threadIdx.x < count) rays.begin(base + threadIdx.x, r);
    }
    __device__ __forceinline__ void trace(const RecordRays<kAnyHit, kInst>& rays, const WideStack& stack,
                                          uint32_t& status) const {
        const bool live = threadIdx.x < count;
        if constexpr (kAnyHit && !kInst) {
            WideState s;
            trace_packet_any(rays.nodes(), rays.tris(), live, r, s, stack, status);
            if (live) rays.end(base + threadIdx.x, s);
        } else {
            std::conditional_t<kInst, InstWalk, WideWalk> w;
            trace_packet<kAnyHit>(rays, live, r, w, stack, status);
            if (live) rays.end(base + threadIdx.x, w.s);
        }
    }
};

extern __shared__ uint2 query_stack[];

__device__ __forceinline__ WideStack warp_stack(const QueryArgs& a) {
    return WideStack{query_stack + threadIdx.x, 32, a.stack_depth};
}

// kLook: a warp looks at its block's rays; flat scenes' rays that run side by side are traced as a packet, instanced
// scenes' rays that do not.
template <bool kAnyHit, bool kInst, bool kLook>
__device__ __forceinline__ void query_warp(const QueryArgs& a) {
    __shared__ __align__(16) uint4 answer;
    __shared__ __align__(8) uint64_t barrier;
    RecordRays<kAnyHit, kInst> rays = query_records<kAnyHit, kInst>(a);
    uint32_t status = 0;
    bool stream = true;
    if constexpr (kLook) {
        const Packet<kAnyHit, kInst> packet(rays, blockIdx.x * 32u);
        stream = side_by_side(packet.r, packet.count, a.reach2) == kInst;
        if (!stream) packet.trace(rays, warp_stack(a), status);
    }
    if (stream) {
        if (a.claim) rays.take_over(&answer, &barrier);
        trace_stream<kAnyHit, std::conditional_t<kInst, InstWalk, WideWalk>>(rays, warp_stack(a), status);
        status |= rays.status;
    }
    if (status) atomicOr(a.err, status);
}

template <bool kAnyHit, bool kLook>
__global__ void __launch_bounds__(32, kWarpsPerSm) k_query_wide(const __grid_constant__ QueryArgs a) {
    query_warp<kAnyHit, false, kLook>(a);
}

// Scenes with instances or curves: 16 warps per SM (the walk's state takes up to 128 registers).
template <bool kAnyHit, bool kLook>
__global__ void __launch_bounds__(32, kInstWarpsPerSm) k_query_instanced(const __grid_constant__ QueryArgs a) {
    query_warp<kAnyHit, true, kLook>(a);
}

template <bool kAnyHit>
__global__ void __launch_bounds__(32, kWarpsPerSm) k_query_packet(const __grid_constant__ QueryArgs a) {
    const RecordRays<kAnyHit, false> rays = query_records<kAnyHit, false>(a);
    uint32_t status = 0;
    Packet<kAnyHit, false>(rays, blockIdx.x * 32u).trace(rays, warp_stack(a), status);
    if (status) atomicOr(a.err, status);
}

// Four rays a one-warp block, eight lanes each.  kLook: the eight blocks of 32 records look at these records' rays
// (whose origins and directions no query writes) and, unless they run side by side, leave them to the first of the
// eight.  The first blocks of all records come before the others, which mostly find nothing to do when the rays part.
template <bool kAnyHit, bool kLook>
__global__ void __launch_bounds__(32, kWarpsPerSm) k_query_groups(const __grid_constant__ QueryArgs a) {
    RecordRays<kAnyHit, false> rays = query_records<kAnyHit, false>(a);
    uint32_t status = 0, first = blockIdx.x * 4u;
    QueryRay r;
    if constexpr (kLook) {
        const uint32_t ranges = (a.n + 31u) / 32u;
        const uint32_t range = blockIdx.x < ranges ? blockIdx.x : (blockIdx.x - ranges) / 7u;
        first = range * 32u + (blockIdx.x < ranges ? 0u : 4u + (blockIdx.x - ranges) % 7u * 4u);
        const Packet<kAnyHit, false> packet(rays, range * 32u);
        if (!side_by_side(packet.r, packet.count, a.reach2)) {
            if (blockIdx.x >= ranges) return;
            packet.trace(rays, warp_stack(a), status);
            if (status) atomicOr(a.err, status);
            return;
        }
        const float* f = reinterpret_cast<const float*>(&packet.r);
        float* mine = reinterpret_cast<float*>(&r);
#pragma unroll
        for (int k = 0; k < int(sizeof(QueryRay) / sizeof(float)); ++k)
            mine[k] = __shfl_sync(0xffffffffu, f[k], int((first & 31u) + (threadIdx.x >> 3)));
    }
    const uint32_t i = first + (threadIdx.x >> 3);
    if (i >= a.n) return;
    WideState s;
    if (!kLook) rays.begin(i, r);
    trace_group<kAnyHit>(rays.nodes(), rays.tris(), r, s, warp_stack(a), status);
    if ((threadIdx.x & 7u) == 0) rays.end(i, s);
    if (status) atomicOr(a.err, status);
}

template <bool kAnyHit>
cudaError_t launch_wide(const DeviceBvh& bvh, float4* d_rays, uint32_t record_float4s, uint32_t n,
                        const uint32_t* order, const uint32_t* ctl, uint32_t* d_err, cudaStream_t s, bool far) {
    const bool inst = bvh.insts != nullptr;
    const uint32_t blocks = (n + 31u) / 32u;
    const uint32_t resident = uint32_t(bvh.sm_count) * (inst ? kInstWarpsPerSm : kWarpsPerSm);
    QueryArgs a;
    a.nodes = static_cast<const uint4*>(bvh.nodes);
    a.tris = bvh.tris;
    a.insts = bvh.insts;
    a.rays = d_rays;
    a.record_float4s = record_float4s;
    a.n = n;
    a.order = order;
    a.ctl = ctl;
    a.stack_depth = bvh.stack_depth;
    a.claim = n > 32u * resident ? 1u : 0u;  // a batch whose blocks all run at once leaves none to take over
    float diagonal2 = 0.0f;
    for (int k = 0; k < 3; ++k) diagonal2 += (bvh.hi[k] - bvh.lo[k]) * (bvh.hi[k] - bvh.lo[k]);
    a.reach2 = diagonal2 / 1024.0f;
    a.err = d_err;
    const size_t stack_bytes = size_t(bvh.stack_depth) * 32 * sizeof(uint2);
    const auto up_to = [&](uint32_t rays) { return n <= rays * resident; };
    if (inst) {
        const bool streams = far || bvh.curves || a.claim || up_to(kInstStreamRays);
        if (streams) k_query_instanced<kAnyHit, false><<<blocks, 32, stack_bytes, s>>>(a);
        else k_query_instanced<kAnyHit, true><<<blocks, 32, stack_bytes, s>>>(a);
    } else if (up_to(far ? kFarGroupRays : bvh.tri_count > kLargeScene ? kLargeGroupRays : kGroupRays<kAnyHit>)) {
        k_query_groups<kAnyHit, false><<<(n + 3u) / 4u, 32, stack_bytes, s>>>(a);
    } else if (!far && up_to(kSideGroupRays)) {
        k_query_groups<kAnyHit, true><<<8 * blocks, 32, stack_bytes, s>>>(a);
    } else if (up_to(far && !kAnyHit ? kFarPacketRays : kPacketRays)) {
        k_query_packet<kAnyHit><<<blocks, 32, stack_bytes, s>>>(a);
    } else {
        if constexpr (!kAnyHit) {
            if (far || (bvh.tri_count > kLargeScene && !up_to(kLargeLookRays))) {
                k_query_wide<false, false><<<blocks, 32, stack_bytes, s>>>(a);
                return cudaGetLastError();
            }
        }
        k_query_wide<kAnyHit, true><<<blocks, 32, stack_bytes, s>>>(a);
    }
    return cudaGetLastError();
}

// ---------------------------------------------------------------------------------------------------
// Ray order.  A large batch of incoherent rays in HBM is traced in the order of a 24-bit key (the direction's
// octant above a 21-bit Morton code of the origin in the scene bounds), so that the rays of a warp start near
// one another and fetch the same nodes and triangles: a stable radix sort of (key, index) pairs, then the query
// kernel reads ray order[i] and writes its hit in place.  Results do not depend on the order.  A batch whose
// sampled neighbouring rays run nearly parallel (camera rays in pixel order) is coherent already: k_order_gate
// sets the count to sort to 0 and the sort and the indirection drop out on the device, without a host round trip.
// ---------------------------------------------------------------------------------------------------
constexpr uint32_t kOrderMin = 1u << 20;  // smaller batches keep their order
constexpr int kGatePairs = 1024;

__global__ void __launch_bounds__(256) k_order_gate(const float4* rays, uint32_t record_float4s, uint32_t n,
                                                    uint32_t* ctl) {
    __shared__ uint32_t close;
    if (threadIdx.x == 0) close = 0;
    __syncthreads();
    uint32_t c = 0;
    for (int k = 0; k < kGatePairs / 256; ++k) {
        const size_t i = size_t(threadIdx.x * (kGatePairs / 256) + k) * (n - 2) / (kGatePairs - 1);
        const float4 a = rays[i * record_float4s + 1], b = rays[(i + 1) * record_float4s + 1];
        const float d = a.x * b.x + a.y * b.y + a.z * b.z;
        const float nn = (a.x * a.x + a.y * a.y + a.z * a.z) * (b.x * b.x + b.y * b.y + b.z * b.z);
        if (nn > 0.0f && d > 0.0f && d * d > 0.998f * nn) ++c;  // within about 2.5 degrees
    }
    atomicAdd(&close, c);
    __syncthreads();
    if (threadIdx.x == 0) ctl[0] = 2 * close > uint32_t(kGatePairs) ? 0u : n;
}

__device__ __forceinline__ uint32_t spread7(uint32_t x) {  // bits 0..6 of x to bits 0, 3, .., 18
    x &= 0x7fu;
    x = (x | (x << 8)) & 0x0000f00fu;
    x = (x | (x << 4)) & 0x000c30c3u;
    x = (x | (x << 2)) & 0x00249249u;
    return x;
}

__global__ void __launch_bounds__(256) k_order_keys(const float4* rays, uint32_t record_float4s, const uint32_t* ctl,
                                                    float3 lo, float3 scale, uint32_t* keys, uint32_t* order) {
    const uint32_t n = ctl[0];
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const float4 o = rays[size_t(i) * record_float4s], d = rays[size_t(i) * record_float4s + 1];
        const uint32_t qx = uint32_t(fminf(fmaxf((o.x - lo.x) * scale.x, 0.0f), 127.0f));
        const uint32_t qy = uint32_t(fminf(fmaxf((o.y - lo.y) * scale.y, 0.0f), 127.0f));
        const uint32_t qz = uint32_t(fminf(fmaxf((o.z - lo.z) * scale.z, 0.0f), 127.0f));
        const uint32_t oct = (d.x < 0.0f ? 4u : 0u) | (d.y < 0.0f ? 2u : 0u) | (d.z < 0.0f ? 1u : 0u);
        keys[i] = (oct << 21) | (spread7(qx) << 2) | (spread7(qy) << 1) | spread7(qz);
        order[i] = i;
    }
}

// Gate, keys, three radix passes and the ordered traversal on stream s, with stream-ordered scratch.
template <bool kAnyHit>
cudaError_t launch_query_ordered(const DeviceBvh& bvh, float4* d_rays, uint32_t record_float4s, uint32_t n,
                                 uint32_t* d_err, cudaStream_t s) {
    const uint32_t ntiles = (n + kSortTile - 1) / kSortTile;
    const size_t hist = size_t(256) * ntiles;
    const size_t words = 4 * size_t(n) + hist + (hist + 1) + scan_scratch_words(hist + 1) + 1;
    uint32_t* mem = nullptr;
    cudaError_t e = bvh.pool ? cudaMallocFromPoolAsync(reinterpret_cast<void**>(&mem), words * 4, bvh.pool, s)
                             : cudaMallocAsync(reinterpret_cast<void**>(&mem), words * 4, s);
    if (e != cudaSuccess) return e;
    uint32_t* keys[2] = {mem, mem + n};
    uint32_t* vals[2] = {mem + 2 * size_t(n), mem + 3 * size_t(n)};
    uint32_t* h = mem + 4 * size_t(n);
    uint32_t* h_off = h + hist;
    uint32_t* scan_tmp = h_off + hist + 1;
    uint32_t* ctl = scan_tmp + scan_scratch_words(hist + 1);
    k_order_gate<<<1, 256, 0, s>>>(d_rays, record_float4s, n, ctl);
    float3 lo, scale;
    const float* b[2] = {bvh.lo, bvh.hi};
    float sc[3];
    for (int a = 0; a < 3; ++a) {
        const float ext = b[1][a] - b[0][a];
        sc[a] = ext > 0.0f ? 128.0f / ext : 0.0f;
    }
    lo = make_float3(bvh.lo[0], bvh.lo[1], bvh.lo[2]);
    scale = make_float3(sc[0], sc[1], sc[2]);
    k_order_keys<<<1024, 256, 0, s>>>(d_rays, record_float4s, ctl, lo, scale, keys[0], vals[0]);
    int in = 0;
    for (int pass = 0; pass < 3; ++pass) {
        k_radix_hist<<<ntiles, 256, 0, s>>>(keys[in], ctl, 8 * pass, h, ntiles);
        scan_exclusive(h, uint32_t(hist), h_off, scan_tmp, s);
        k_radix_scatter<<<ntiles, 256, 0, s>>>(keys[in], vals[in], keys[in ^ 1], vals[in ^ 1], ctl, 8 * pass, h_off,
                                               ntiles);
        in ^= 1;
    }
    e = launch_wide<kAnyHit>(bvh, d_rays, record_float4s, n, vals[in], ctl, d_err, s, false);
    const cudaError_t ef = cudaFreeAsync(mem, s);
    return e != cudaSuccess ? e : ef;
}

// Plain binary FP32 path: one thread per ray, launched over the whole batch.
template <bool kAnyHit>
__global__ void __launch_bounds__(kQueryBlock) k_query_binary(const float4* __restrict__ nodes,
                                                              const float4* __restrict__ tris, float4* rays,
                                                              uint32_t record_float4s, uint32_t n, uint32_t* err) {
    __shared__ int stack_mem[kBinaryStack * kQueryBlock];
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const QueryRay r = load_ray(rays + size_t(i) * record_float4s);
    QueryHit h;
    uint32_t status = 0;
    const bool found = trace_binary<kAnyHit>(nodes, tris, r, h, stack_mem + threadIdx.x, kQueryBlock, status);
    if (status) atomicOr(err, status);
    if (found) {
        if (kAnyHit)
            reinterpret_cast<float*>(rays + size_t(i) * record_float4s)[8] = -__int_as_float(0x7f800000);
        else
            store_hit(reinterpret_cast<SelRayHit*>(rays + size_t(i) * record_float4s), tris, h);
    }
}

template <bool kAnyHit>
cudaError_t launch_query(const DeviceBvh& bvh, float4* d_rays, uint32_t record_float4s, uint32_t n, uint32_t* d_err,
                         cudaStream_t s, bool far = false) {
    if (n == 0) return cudaSuccess;
    if (bvh.insts || bvh.kind == SEL_BVH_WIDE8_Q8)
        return launch_wide<kAnyHit>(bvh, d_rays, record_float4s, n, nullptr, nullptr, d_err, s, far);
    const dim3 grid((n + kQueryBlock - 1) / kQueryBlock);
    k_query_binary<kAnyHit><<<grid, kQueryBlock, 0, s>>>(static_cast<const float4*>(bvh.nodes), bvh.tris, d_rays,
                                                         record_float4s, n, d_err);
    return cudaGetLastError();
}

}  // namespace

cudaError_t launch_intersect(const DeviceBvh& bvh, SelRayHit* d_rays, uint32_t n, uint32_t* d_err, cudaStream_t s) {
    if (bvh.order_rays && n >= kOrderMin && !bvh.insts && bvh.kind == SEL_BVH_WIDE8_Q8)
        return launch_query_ordered<false>(bvh, reinterpret_cast<float4*>(d_rays), sizeof(SelRayHit) / 16, n, d_err, s);
    return launch_query<false>(bvh, reinterpret_cast<float4*>(d_rays), sizeof(SelRayHit) / 16, n, d_err, s);
}

cudaError_t launch_occluded(const DeviceBvh& bvh, SelRay* d_rays, uint32_t n, uint32_t* d_err, cudaStream_t s) {
    if (bvh.order_rays && n >= kOrderMin && !bvh.insts && bvh.kind == SEL_BVH_WIDE8_Q8)
        return launch_query_ordered<true>(bvh, reinterpret_cast<float4*>(d_rays), sizeof(SelRay) / 16, n, d_err, s);
    return launch_query<true>(bvh, reinterpret_cast<float4*>(d_rays), sizeof(SelRay) / 16, n, d_err, s);
}

cudaError_t launch_query_strided(bool any_hit, const DeviceBvh& bvh, void* recs, size_t record_bytes, uint32_t n,
                                 uint32_t* d_err, cudaStream_t s) {
    float4* r = static_cast<float4*>(recs);
    const uint32_t stride = uint32_t(record_bytes / 16);
    return any_hit ? launch_query<true>(bvh, r, stride, n, d_err, s, true)
                   : launch_query<false>(bvh, r, stride, n, d_err, s, true);
}

}  // namespace sel
