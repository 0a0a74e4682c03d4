// Ray-query kernels over SelRay / SelRayHit records (Embree's RTCRay / RTCRayHit layouts) and their
// launchers.  One lane per ray; each thread keeps its traversal stack in shared memory.
#include "query.h"

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
// 8-wide traversal.  Blocks are one warp and block index k stands for records [32 k, 32 k + 32).  A warp whose
// lanes run out of rays takes over the block index of a block that has not started (cluster launch control) and
// refills its finished lanes from it (trace_stream), so a batch of any size is balanced without a work counter in
// memory, on any number of streams at once and under graph capture.  The next index is requested while the
// warp still traces the last, which hides the answer's latency.  An atomic counter in place of the block indices
// measured 3 % faster (4 M incoherent rays over 5.2 M triangles, closest hit 1.81 against 1.87 ms) but would have to
// be allocated and zeroed by every call.
// 64 registers, 32 warps per SM: with 36 (56 registers) closest hit takes 1.89 against 1.81 ms and any hit 1.34
// against 1.22, with 40 (48 registers) 2.08 and 1.46.  Whole calls on that scene, start of a call to its end: closest
// hit 2.92 ms with one thread per ray and a 24-entry stack, 1.95 now; any hit 1.95 and 1.33; camera rays 0.50 and
// 0.45, any hit 0.28 and 0.27.
// ---------------------------------------------------------------------------------------------------
constexpr int kWarpsPerSm = 32;
constexpr uint32_t kErrClaimTimeout = 32u;  // the answer to a work request never came

__device__ __forceinline__ uint32_t shared_address(const void* p) { return uint32_t(__cvta_generic_to_shared(p)); }

// The records a warp traces.  kOrdered: record `order[i]` in place of record i when ctl[0] is non-zero.
struct RecordRanges {
    uint32_t n, status;
    bool claim, started;     // claim: more blocks were launched than run at once
    uint32_t phase;
    uint32_t answer, barrier;  // shared memory: 16-byte answer, its mbarrier

    __device__ __forceinline__ RecordRanges(uint32_t count, bool more_blocks, const uint4* ans, const uint64_t* bar)
        : n(count), status(0), claim(more_blocks), started(false), phase(0), answer(0), barrier(0) {
        if (!claim) return;
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
    uint32_t claim;
    uint32_t* err;
};

template <bool kAnyHit, bool kInst, typename Walk>
__device__ __forceinline__ void query_warp(const QueryArgs& a) {
    extern __shared__ uint2 query_stack[];
    __shared__ __align__(16) uint4 answer;
    __shared__ __align__(8) uint64_t barrier;
    RecordRays<kAnyHit, kInst> rays(a.n, a.claim != 0, &answer, &barrier);
    rays.node_array = a.nodes;
    rays.tri_array = a.tris;
    rays.inst_array = a.insts;
    rays.recs = a.rays;
    rays.record_float4s = a.record_float4s;
    rays.order = a.ctl && a.ctl[0] ? a.order : nullptr;
    uint32_t status = 0;
    trace_stream<kAnyHit, Walk>(rays, WideStack{query_stack + threadIdx.x, 32, a.stack_depth}, status);
    status |= rays.status;
    if (status) atomicOr(a.err, status);
}

template <bool kAnyHit>
__global__ void __launch_bounds__(32, kWarpsPerSm) k_query_wide(const __grid_constant__ QueryArgs a) {
    query_warp<kAnyHit, false, WideWalk>(a);
}

// Scenes with instances or curves: 16 warps per SM (the walk's state takes up to 128 registers).
template <bool kAnyHit>
__global__ void __launch_bounds__(32, 16) k_query_instanced(const __grid_constant__ QueryArgs a) {
    query_warp<kAnyHit, true, InstWalk>(a);
}

// Batches of at most one ray a group of eight lanes: 4 rays a one-warp block.
template <bool kAnyHit>
__global__ void __launch_bounds__(32, kWarpsPerSm) k_query_groups(const __grid_constant__ QueryArgs a) {
    extern __shared__ uint2 query_stack[];
    RecordRays<kAnyHit, false> rays(a.n, false, nullptr, nullptr);
    rays.node_array = a.nodes;
    rays.tri_array = a.tris;
    rays.recs = a.rays;
    rays.record_float4s = a.record_float4s;
    rays.order = nullptr;
    uint32_t status = 0;
    trace_groups<kAnyHit>(rays, a.n, WideStack{query_stack + threadIdx.x, 32, a.stack_depth}, status);
    if (status) atomicOr(a.err, status);
}

template <bool kAnyHit>
cudaError_t launch_wide(const DeviceBvh& bvh, float4* d_rays, uint32_t record_float4s, uint32_t n,
                        const uint32_t* order, const uint32_t* ctl, uint32_t* d_err, cudaStream_t s) {
    const bool inst = bvh.insts != nullptr;
    const uint32_t blocks = (n + 31u) / 32u;
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
    // a batch whose blocks all run at once leaves none to take over
    a.claim = blocks > uint32_t(bvh.sm_count) * (inst ? 16u : uint32_t(kWarpsPerSm)) ? 1u : 0u;
    a.err = d_err;
    const size_t stack_bytes = size_t(bvh.stack_depth) * 32 * sizeof(uint2);
    const uint32_t group_blocks = (n + 3u) / 4u;
    if (inst) k_query_instanced<kAnyHit><<<blocks, 32, stack_bytes, s>>>(a);
    else if (group_blocks <= kGroupWaves * uint32_t(bvh.sm_count) * kWarpsPerSm)
        k_query_groups<kAnyHit><<<group_blocks, 32, stack_bytes, s>>>(a);
    else k_query_wide<kAnyHit><<<blocks, 32, stack_bytes, s>>>(a);
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
    e = launch_wide<kAnyHit>(bvh, d_rays, record_float4s, n, vals[in], ctl, d_err, s);
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
                         cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    if (bvh.insts || bvh.kind == SEL_BVH_WIDE8_Q8)
        return launch_wide<kAnyHit>(bvh, d_rays, record_float4s, n, nullptr, nullptr, d_err, s);
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
    return any_hit ? launch_query<true>(bvh, r, stride, n, d_err, s) : launch_query<false>(bvh, r, stride, n, d_err, s);
}

}  // namespace sel
