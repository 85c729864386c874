// rt_traverse.cuh -- the persistent BVH8 traversal kernel.
//
// Replaces the RT-core traversal behind traceRayEXT of the reference sample
// (vulkan-raytraced-triangle/main.cpp:1047-1052).  Included by rt_trace.cu
// (one structure per launch: the ray-query API and the path tracer) and by
// rt_trace_multi.cu (many scenes per launch: the batched path tracer, where
// each ray carries the index of its scene).
//
// Persistent warps walk a ray array.  A warp refills its idle lanes from a
// global counter (atomic work stealing) whenever at least `refill` of them
// have finished; each lane walks the compressed BVH8 with 16-byte node loads
// and keeps its traversal stack in a shared-memory ring of RING entries whose
// bottom spills to local memory.
//
// Visiting order: internal children in ascending (slot ^ ray octant), the
// remaining siblings pushed as one group; the leaf records met on the way are
// tested in batches (see the triangle queue below).  Closest hit = smallest t,
// ties broken by the smallest triangle index, among the triangles that a walk
// testing each node's records as it visits the node would test: the CPU
// restatement's hit, bit for bit, whatever is tested together.
#pragma once

#include <cuda_runtime.h>

#include "../../include/rtcore.h"
#include "../../include/rtcore_accel.h"
#include "rt_device.cuh"

namespace rtc {
namespace {

constexpr int kTraceThreads = 128;  // block size of the single-structure kernels
// Shared-memory stack entries per ray of the single-structure kernels; deeper
// ones spill to local memory.  With the triangle queue and the rays' hits a
// block takes 15.5 KB, of which this is 8: 16 entries leave node fetches too
// little of the SM's L1 (64 scenes at 16 samples: 4.99 s, 4.36 at 8), and 4
// spill too often (1M soup 1,568 us, 1,558 at 8; 64 instances 820 and 809).
constexpr int kRing = 8;
constexpr uint32_t kAnyBlocksPerSm = 1024u / kTraceThreads;  // resident blocks the any-hit and mixed kernels are bounded for
constexpr int kMaxDepth = 64;       // total stack entries per ray
constexpr uint32_t kNone = 0xffffffffu;
constexpr uint32_t kMinusZero = 0x80000000u;  // the bits of -0; in a record index (below 2^30) the mark of a hit at t = -0
constexpr uint32_t kLate = 0x40000000u;       // in a record index: a hit in whose place an in-order walk may find another
constexpr int32_t kNoLimit = 0x7fffffff;      // as an ordered integer: beyond every distance

struct Hit {
    float t, u, v;
    uint32_t rec;     // leaf-record index of the best triangle
    uint32_t tri;     // build-input triangle index
    uint32_t inst;    // instance index (0 for a bare BLAS)
    bool found;
};

__device__ __forceinline__ uint4 ldg4(const uint4 *p) { return __ldg(p); }

// Traversal view of one bottom-level structure (32 bytes), written on the
// device from the structure's header.  node_count 0 marks a structure whose
// rays all miss (empty, or not a bottom-level structure).
struct TravScene {
    const uint4 *nodes;
    const uint4 *prims;
    uint32_t node_count;
    uint32_t prim_count;
    float slack;  // box_slack of the structure
    uint32_t pad;
};
static_assert(sizeof(TravScene) == 32, "TravScene is read as two 16-byte words");

struct BatchArgs {
    const uint8_t *accel;       // the structure (single-structure kernels)
    const TravScene *scenes;    // per-scene views (multi-scene kernels)
    const uint32_t *ray_scene;  // scene index of each ray (multi-scene kernels)
    uint32_t n_scenes;
    const float4 *rays;      // 2 float4 per ray
    float4 *hits;            // closest: 1 float4 per ray (t, prim bits, u, v)
    rt_hit_ext *hits_ext;    // nullable
    uint8_t *occluded;       // any-hit output
    uint32_t n;
    uint32_t refill;         // refill when at least this many lanes are idle
    uint32_t *counter;
    uint32_t *err;
    const uint32_t *n_dev;   // when set: the ray count, read on the device
    uint32_t out_rec;        // closest hit: write the leaf-record index
    // mixed launches: a second queue of any-hit rays after the closest-hit
    // queue above (rays2[i] is ray n1 + i of the launch; results to occluded)
    const float4 *rays2;
    const uint32_t *ray_scene2;
    const uint32_t *n_dev2;
    uint32_t n2;
};

// ---------------------------------------------------------------------------
// Triangle queue
// ---------------------------------------------------------------------------
// A node visit leaves a lane 0.2-0.3 triangles to test on average, so testing
// them on the spot runs the triangle test with two or three of a warp's 32
// lanes.  Instead each lane appends the leaf records it meets to its warp's
// queue in shared memory (record index and lane) and walks on; once there are
// as many entries as lanes with a ray, the whole warp tests them, one entry per
// lane with the owner's ray read by shuffles, and hands the hits back to their
// owners.  A ray walks a few nodes more because its far limit shrinks a few
// visits later.  A lane keeps its ray until its last entry has been tested.  1M
// soup, 4.15M primary and incoherent rays: 28.6 entries per batch, 18.4 nodes and
// 4.4 triangles per ray against 17.7 and 4.0 when every triangle is tested on the
// spot, 28.1 of 32 lanes walking per node step (2M box, mixed launches: 27.4).  With the box test's instruction count, the
// 64-bit queue entry and the hits' shared-memory minima this took the launch from
// 1.92 to 1.55 ms, the path tracer's 2M-triangle frame of four samples from 25.7
// to 20.4.  What bounds it now: issue slots (79 % busy) and the L1 data path
// (78 %: a node is five 16-byte loads per lane, nearly every one a wavefront of
// its own).
//
// In the order of the CPU restatement a record is tested, and the far limit
// shrunk, before the next node's boxes.  A walk that goes on meanwhile visits
// more, and can only end differently by a triangle X that it tests and the other
// walk does not: one of the boxes above X lets the ray in beyond an earlier
// hit's distance, rounding included, while X's own distance is no greater -- X
// lies on the face of its box where the ray enters, or the ray starts there.
// boxes_may_exceed bounds from X's vertices where those boxes let the ray in.  A
// ray whose best hit has that bound beyond the nearest earlier hit of another
// node (records of one node are tested together in either walk) is set aside --
// its result's place links the lane's rays of that kind -- and its hit confirmed,
// or the ray walked in order, once the lane is done with the others.  For any
// other ray the hit is the other walk's: its far limits are hits no nearer than
// X, so every box above X lets the ray in there too, X is tested, and nothing it
// tests is better.
// (12 coincident copies of 60 axis-parallel triangles, 1M rays: 0 to 3 rays
// differ without this, 2 to 4 of rays that start on the triangles with a window
// of 2^-12 of t in the place of the bound.  The soup's rays take 1.55 ms with
// either, the 2M box's frame 20.37 for 20.43; in the 56-register kernel 8 % more
// with the ray held through the merge instead of read again, in the mixed kernel
// 2 % more with it read again.)
constexpr float kBoxSlack = 0x1p-20f;
constexpr uint32_t kTriQueue = 64;  // entries per warp: below 32 before an append of at most 32
constexpr int kTriDrain = 8;   // lanes waiting for their entries alone before a partial batch is tested

__device__ __forceinline__ float4 xyz_of(const uint4 &q) {
    return make_float4(__uint_as_float(q.x), __uint_as_float(q.y), __uint_as_float(q.z), 0.f);
}

// kBoxSlack times the greatest coordinate of a structure's bounds; infinite where
// a node's quantisation steps (at most 2^RT_QEXP_MAX) may not reach its bounds.
__device__ __forceinline__ float box_slack(const rt_accel_header *h) {
    const float4 lo = *reinterpret_cast<const float4 *>(h->bounds_lo);
    const float4 hi = *reinterpret_cast<const float4 *>(h->bounds_hi);
    const float m = fmaxf(fmax3(fabsf(lo.x), fabsf(lo.y), fabsf(lo.z)), fmax3(fabsf(hi.x), fabsf(hi.y), fabsf(hi.z)));
    return m < 0x1p100f ? kBoxSlack * m : kInf;
}

// kBoxSlack times at least the greatest distance along an axis between a ray's
// origin and anything in the scene.
__device__ __forceinline__ float ray_slack(const float o[3], float scene_slack) {
    return __fmaf_rn(fmax3(fabsf(o[0]), fabsf(o[1]), fabsf(o[2])), kBoxSlack, scene_slack);
}

// A ray's slack and axis order in one word (the slack rounded up, a multiple of
// 64), for the kernels whose lanes walk different structures.
__device__ __forceinline__ uint32_t pack_slack(const Ray &r, const float o[3], float scene_slack) {
    return ((__float_as_uint(ray_slack(o, scene_slack)) & ~63u) + 64u) | r.kxyz;
}

// Whether a box around the triangle of leaf record p, in a node anywhere above
// it, could let the ray in beyond `limit` (a hit's distance); r: origin and
// shear, slack: ray_slack's.
//
// Along axis a such a box's near plane lies no further along the ray than the
// triangle's nearest vertex, and isect_node's distance to it is off by less than
// 6 * 2^-24 D |1 / d_a|, D the greatest distance along an axis between the
// origin and anything in the scene: two roundings of (frame origin - ray origin)
// / d_a, one of the fma, the step exact.  Compared are (nearest vertex - origin
// + slack) / d_z and limit d_a / d_z, d_z the shear's axis, whose own roundings
// stay below 5 * 2^-24 D; the slack is 16 * 2^-24 D.  Products too small to carry
// that accuracy, and limits next to zero, count as exceeded.
__device__ __forceinline__ bool boxes_may_exceed(const Ray &r, float slack, const uint4 *p, float limit) {
    const uint32_t kx = r.kxyz & 3u, kz = (r.kxyz >> 4) & 3u;
    bool exceeds = !(limit >= 0x1p-40f);
#pragma unroll
    for (uint32_t a = 0; a < 3u; ++a) {
        const float s = a == kz ? 1.0f : (a == kx ? r.sx : r.sy);
        const bool neg = ((__float_as_uint(s) ^ __float_as_uint(r.sz)) >> 31) != 0u;
        const float *v = reinterpret_cast<const float *>(p) + a;
        const float v0 = __ldg(v), v1 = __ldg(v + 4), v2 = __ldg(v + 8);
        const float ahead = (neg ? r.o[a] - fmax3(v0, v1, v2) : fmin3(v0, v1, v2) - r.o[a]) + slack;
        const bool within = fabsf(s) >= 0x1p-60f && ahead * fabsf(r.sz) < limit * fabsf(s);
        exceeds = exceeds || !(ahead <= 0.0f || within);
    }
    return exceeds;
}

// With pack_slack's word in the ray.
__device__ __forceinline__ bool boxes_may_exceed(const Ray &r, const uint4 *p, float limit) {
    return boxes_may_exceed(r, __uint_as_float(r.kxyz & ~63u), p, limit);
}

// MIXED: one launch over two queues -- the closest-hit rays (rays, n_dev;
// results to hits) and then the any-hit rays (rays2, n_dev2; results to
// occluded) -- each ray walked exactly as in a launch of its own kind; the
// path tracer traces a depth's shadow rays and the next depth's extension
// rays together, so the two share one launch tail.
// Register budget: the closest-hit single-structure kernel fits nine 128-thread
// blocks per SM (56 registers; at eight blocks and 64 registers the 1M soup's
// rays took 1.74 instead of 1.58 ms); the others keep eight blocks and 64
// registers (mixed, nine blocks: 2M box 21.26 ms per four samples, eight 20.85).
template <bool ANY, bool MULTI, int THREADS, int RING, bool MIXED = false>
__global__ void __launch_bounds__(THREADS, ((MULTI || ANY || MIXED) ? 1024 : 1152) / THREADS) k_trace_blas(const BatchArgs a) {
    static_assert((RING & (RING - 1)) == 0 && RING <= kMaxDepth, "RING is a power of two");
    __shared__ uint2 s_stack[RING][THREADS];
    __shared__ uint2 s_queue[THREADS / 32][kTriQueue];  // leaf record, lane | visits << 5
    // per lane: the triangle test's part of the ray (written once per ray, read
    // by whichever lane tests); the best hit so far -- t as an ordered integer;
    // u, v, leaf record and triangle (kNone: no hit)
    __shared__ float4 s_shear[THREADS];
    __shared__ int32_t s_t[ANY ? 1 : THREADS];
    __shared__ uint4 s_best[ANY ? 1 : THREADS];
    __shared__ uint32_t s_visit[ANY ? 1 : THREADS];  // the node visit of the best hit so far (0: no hit)
    __shared__ int32_t s_prev[ANY ? 1 : THREADS];    // the nearest hit of an earlier visit, as an ordered integer
    static_assert(sizeof(s_stack) + sizeof(s_queue) + sizeof(s_shear) + sizeof(s_t) + sizeof(s_best) + sizeof(s_visit) +
                          sizeof(s_prev) <= 48u * 1024u,
                  "static shared memory");
    const uint4 *nodes = nullptr, *prims = nullptr;
    // A tree walk visits each node at most once: more visits, or a node index
    // past the end, can only come from a corrupt structure.
    uint32_t max_visits = 0;
    bool empty = true;
    const rt_accel_header *hd = reinterpret_cast<const rt_accel_header *>(a.accel);
    if (!MULTI) {
        if (!MIXED && !a.n_dev) pdl_launch();  // a ray query's k_trace_inst
        if (hd->kind != RT_ACCEL_KIND_BLAS) return;  // k_trace_inst handles it
        nodes = reinterpret_cast<const uint4 *>(a.accel + hd->node_offset);
        prims = reinterpret_cast<const uint4 *>(a.accel + hd->prim_offset);
        empty = hd->prim_count == 0;
        max_visits = hd->node_count;
    }
    constexpr uint32_t kFull = 0xffffffffu;
    constexpr bool kFewRegisters = !MULTI && !ANY && !MIXED;
    const int tid = threadIdx.x, lane = tid & 31;
    uint2 *queue = s_queue[tid >> 5];
    const int warp0 = tid & ~31;  // lane 0's thread

    // (one more entry than the stack's: the last ray set aside, this lane's ray)
    uint2 spill[kMaxDepth + 1];
    uint32_t &aside = spill[kMaxDepth].x, &ray_index = spill[kMaxDepth].y;
    aside = kNone;

    if (MULTI) __syncwarp();  // (registers: six scenes 2.98 ms without, 2.91 with it)
    bool have_ray = false, exhausted = false, pending = false;
    Ray r;
    r.o[0] = r.o[1] = r.o[2] = 0.f;
    r.prio = 0u;
    float tmin = 0.f, tbest = 0.f;  // tbest: the ray's far limit, then its best hit
    bool found = false;
    uint32_t node = 0;
    int sp = 0, lo = 0;
    uint32_t visits = 0;
    uint32_t head = 0, tail = 0;  // queue positions tested / appended so far (the same in every lane)
    uint32_t last = ~0u;          // position of this lane's latest entry
    uint32_t error = 0u;          // detail word of an error this lane's ray met
    const uint32_t n1 = a.n_dev ? min(*a.n_dev, a.n) : a.n;
    const uint32_t n_rays = MIXED ? n1 + min(*a.n_dev2, a.n2) : n1;
    bool any_ray = ANY;  // this lane's ray is an any-hit ray
    // Fewer rays than lanes: each warp takes its share of them in as few lanes
    // as that needs, so that the rays' walks do not wait on one another.  So with
    // the path tracer's queues, whose grid is that of the longest; a query's grid
    // has a warp per 32 rays, which leaves up to about a thousand to spread.
    const uint32_t warps = gridDim.x * (THREADS / 32);
    const uint32_t share = n_rays / warps + 1u;
    const uint32_t lanes = share >= 32u ? kFull : (1u << share) - 1u;
    const int refill = (int)min(a.refill, min(share, 32u));

    auto write_hit = [&](uint32_t ray_idx, bool hit, float t, float u, float v, uint32_t rec, uint32_t tri) {
        const float4 out = hit ? make_float4(t, __uint_as_float(a.out_rec ? rec : tri), u, v)
                               : make_float4(kInf, __uint_as_float(kNone), 0.f, 0.f);
        if (MIXED || a.hits) a.hits[ray_idx] = out;
        if (!MULTI && !MIXED && a.hits_ext) {
            rt_hit_ext x;
            x.t = out.x; x.u = out.z; x.v = out.w;
            x.instance_id = hit ? 0u : kNone;
            x.custom_index = 0;
            x.geometry_index = hit ? ldg4(prims + (size_t)rec * 3u + 1).w : 0u;
            x.primitive_id = hit ? ldg4(prims + (size_t)rec * 3u + 2).w : kNone;
            x.sbt_record = x.geometry_index;
            a.hits_ext[ray_idx] = x;
        }
    };
    auto scene_of = [&](uint32_t s) {  // returns the structure's slack
        const uint4 *tv = reinterpret_cast<const uint4 *>(a.scenes + s);
        const uint4 t0 = ldg4(tv), t1 = ldg4(tv + 1);
        nodes = reinterpret_cast<const uint4 *>(((uint64_t)t0.y << 32) | t0.x);
        prims = reinterpret_cast<const uint4 *>(((uint64_t)t0.w << 32) | t0.z);
        max_visits = t1.x;
        empty = t1.x == 0u || t1.y == 0u;
        return __uint_as_float(t1.z);
    };

    for (;;) {
        // ---- lanes whose walk and tests are done: write the result, refill
        const bool waiting = (int)(last - head) >= 0;
        uint32_t done = __ballot_sync(kFull, !pending && !waiting);
        if (done == kFull || (!exhausted && __popc(done & lanes) >= refill)) {
            if (have_ray && !pending && !waiting) {
                have_ray = false;
                const uint32_t ray_idx = ray_index;
                if (error) {
                    report_error(a.err, RT_ERR_BOUNDS, error | ray_idx);
                    error = 0u;
                }
                if (ANY || (MIXED && any_ray)) {
                    if (a.occluded) a.occluded[ray_idx] = found ? 1u : 0u;
                } else {
                    const uint4 best = s_best[tid];
                    if (best.w != kNone && (best.z & kLate)) {
                        const uint32_t rec = best.z & ~(kMinusZero | kLate);
                        a.hits[ray_idx] =
                            make_float4(__uint_as_float(aside), __uint_as_float(rec), ford_inv(s_prev[tid]), tbest);
                        aside = ray_idx;
                    } else {
                        write_hit(ray_idx, best.w != kNone, (best.z & kMinusZero) ? -0.0f : tbest,
                                  __uint_as_float(best.x), __uint_as_float(best.y), best.z & ~kMinusZero, best.w);
                    }
                }
            }
            if (exhausted) break;  // every lane is done
            const uint32_t want = done & lanes;
            const uint32_t cnt = __popc(want);
            uint32_t base = 0;
            if (lane == 0) base = atomicAdd(a.counter, cnt);
            base = __shfl_sync(kFull, base, 0);
            if (base + cnt >= n_rays) exhausted = true;
            uint32_t idx = base + __popc(want & ((1u << lane) - 1u));
            if (((want >> lane) & 1u) && idx < n_rays) {
                const float4 *ray_src = a.rays;
                const uint32_t *scene_src = a.ray_scene;
                if (MIXED) {
                    any_ray = idx >= n1;
                    if (any_ray) {
                        idx -= n1;
                        ray_src = a.rays2;
                        scene_src = a.ray_scene2;
                    }
                }
                float scene_slack = 0.0f;
                if (MULTI) {
                    const uint32_t s = __ldg(scene_src + idx);
                    if (s < a.n_scenes) {
                        scene_slack = scene_of(s);
                    } else {
                        report_error(a.err, RT_ERR_BOUNDS, 0x77000000u | (s & 0xffffffu));
                        empty = true;
                    }
                }
                const float4 r0 = __ldg(ray_src + 2u * idx), r1 = __ldg(ray_src + 2u * idx + 1u);
                const float o[3] = {r0.x, r0.y, r0.z}, d[3] = {r1.x, r1.y, r1.z};
                ray_setup(r, o, d);
                tmin = r0.w;
                tbest = r1.w;
                found = false;
                ray_index = idx;
                const uint32_t order = MULTI ? pack_slack(r, o, scene_slack) : r.kxyz;
                s_shear[tid] = make_float4(r.sx, r.sy, r.sz, __uint_as_float(order));
                if (!ANY) {
                    s_t[tid] = ford(tbest + 0.0f);  // -0 and +0 tie
                    s_best[tid].w = kNone;
                    s_visit[tid] = 0u;
                }
                have_ray = true;
                node = 0;          // start at the root
                visits = 0;
                pending = !empty;  // an empty structure resolves as a miss
                // so does an empty interval or a NaN limit (two forms by what they
                // cost in registers: 2M box 20.56 and 20.84 ms, six scenes 2.96 and 2.91)
                if (MULTI) {
                    pending = pending && tmin <= tbest;
                } else if (!(tmin <= tbest)) {
                    tmin = kInf;
                    tbest = -kInf;
                }
                sp = 0;
                lo = 0;
                last = head - 1u;
            }
            done = __ballot_sync(kFull, !pending && !((int)(last - head) >= 0));
            if (done == kFull) continue;
        }
        const int busy = 32 - __popc(done);  // lanes with a walk or tests to go
        // a partial batch once too many of them wait for their entries
        const int walking = __popc(__ballot_sync(kFull, pending));
        const bool drain = walking == 0 || busy - walking >= kTriDrain;

        // ---- one node per lane, then the lane's next node
        // leaf slots met (bits), the record reached in the first of them, and
        // the node's slot bytes and record base
        uint32_t leaves = 0u, nth = 0u, meta_lo = 0u, meta_hi = 0u, pbase = 0u;
        // (errors are noted and reported with the result: no calls in here, and
        // the rare cases -- a spilled stack entry -- are the only branches)
        if (pending && (visits >= max_visits || node >= max_visits)) {
            pending = false;
            error = 0x76000000u;
        }
        if (pending) {
            ++visits;
            const NodeWords nd = load_node(nodes, node);
            const uint32_t hits = isect_node(r, nd, tmin, tbest);
            leaves = hits & ~(nd.w0.w >> 24);
            meta_lo = nd.w1.z;
            meta_hi = nd.w1.w;
            pbase = nd.w1.y;
            uint2 g = child_group(nd, hits);
            const bool pop = !group_left(g) && sp > 0;
            if (pop) {
                --sp;
                g = s_stack[sp & (RING - 1)][tid];
            }
            if (pop && sp < lo) {
                g = spill[sp];
                lo = sp;
            }
            pending = group_left(g);
            node = take_child(g, r.prio);  // (of no group: unused)
            const bool push = pending && group_left(g);
            if (push && sp - lo == RING) {
                spill[lo] = s_stack[lo & (RING - 1)][tid];
                ++lo;
            }
            if (push) {
                s_stack[sp & (RING - 1)][tid] = g;
                ++sp;
            }
            if (sp > kMaxDepth) {
                pending = false;
                error = 0x72000000u;
            }
        }

        // ---- append the leaf records met, test a batch when there is one
        uint32_t m = __ballot_sync(kFull, leaves != 0u);
        while (m != 0u || (drain && tail != head)) {
            // a leaf's meta byte: its record count in unary (bits 5-7; none for
            // an unused slot), then its first record's offset
            if (leaves) {
                const uint32_t meta = __byte_perm(meta_lo, meta_hi, (uint32_t)__ffs((int)leaves) - 1u) & 0xffu;
                last = tail + __popc(m & ((1u << lane) - 1u));
                queue[last & (kTriQueue - 1u)] =
                    make_uint2((meta & 0x20u) ? pbase + (meta & 0x1fu) + nth : kNone, visits << 5 | (uint32_t)lane);
                const bool again = ((meta >> 6 >> nth) & 1u) != 0u;
                nth = again ? nth + 1u : 0u;
                leaves = again ? leaves : leaves & (leaves - 1u);
            }
            tail += __popc(m);
            m = __ballot_sync(kFull, leaves != 0u);
            const int cnt = (int)(tail - head);
            if (cnt >= busy || (m == 0u && drain)) {
                const uint32_t k = min(cnt, 32);
                __syncwarp();
                uint2 e = make_uint2(kNone, (uint32_t)lane);
                if ((uint32_t)lane < k) e = queue[(head + (uint32_t)lane) & (kTriQueue - 1u)];
                const uint32_t rec = e.x, src = e.y & 31u;
                const bool have = rec != kNone;
                __syncwarp();  // read before the next append reuses the slots
                head += k;
                Ray tr;
                tr.o[0] = __shfl_sync(kFull, r.o[0], src);
                tr.o[1] = __shfl_sync(kFull, r.o[1], src);
                tr.o[2] = __shfl_sync(kFull, r.o[2], src);
                const float4 shear = s_shear[warp0 + src];
                tr.sx = shear.x;
                tr.sy = shear.y;
                tr.sz = shear.z;
                tr.kxyz = __float_as_uint(shear.w);
                const float t_lo = __shfl_sync(kFull, tmin, src), t_hi = __shfl_sync(kFull, tbest, src);
                const uint4 *pr = prims;
                if (MULTI)
                    pr = reinterpret_cast<const uint4 *>(
                        __shfl_sync(kFull, (unsigned long long)reinterpret_cast<uintptr_t>(prims), src));
                float t = 0.f, u = 0.f, v = 0.f;
                uint32_t tri = kNone;
                bool hit = false;
                if (have) {
                    const uint4 *p = pr + (size_t)rec * 3u;
                    const uint4 q0 = ldg4(p), q1 = ldg4(p + 1), q2 = ldg4(p + 2);
                    tri = q0.w;
                    hit = isect_tri(tr, xyz_of(q0), xyz_of(q1), xyz_of(q2), t_lo, t_hi, t, u, v);
                }
                if (ANY) {
                    const uint32_t fm = __reduce_or_sync(kFull, hit ? 1u << src : 0u);
                    if ((fm >> lane) & 1u) {
                        found = true;
                        pending = false;
                        leaves = 0u;
                    }
                } else {
                    // the owner's best: least t, then, among the lanes that
                    // reached it, least triangle (an improved t clears the
                    // triangle of the old one)
                    const int32_t key = ford(t + 0.0f);  // -0 and +0 tie
                    int32_t *bt = s_t + warp0 + src;
                    uint4 *best = s_best + warp0 + src;
                    const uint32_t visit = e.y >> 5;
                    const bool hit_too = hit;
                    if (__any_sync(kFull, hit)) {
                        if (hit && atomicMin(bt, key) > key) best->w = kNone;
                        __syncwarp();
                        hit = hit && *bt == key;
                        if (hit) atomicMin(&best->w, tri);
                        __syncwarp();
                        hit = hit && best->w == tri;
                        if (hit) {
                            const uint32_t before = s_visit[warp0 + src];
                            s_visit[warp0 + src] = visit;
                            if (before != visit) s_prev[warp0 + src] = before ? ford(t_hi + 0.0f) : kNoLimit;
                            best->x = __float_as_uint(u);
                            best->y = __float_as_uint(v);
                            best->z = rec | (__float_as_uint(t) == kMinusZero ? kMinusZero : 0u);
                        }
                        __syncwarp();
                        if (hit_too && !hit && visit < s_visit[warp0 + src]) atomicMin(s_prev + warp0 + src, key);
                        __syncwarp();
                        const int32_t prev = hit ? s_prev[warp0 + src] : kNoLimit;
                        if (kFewRegisters) {  // the ray read again, not held through the above
                            if (__any_sync(kFull, prev != kNoLimit)) {
                                Ray again;
                                again.o[0] = __shfl_sync(kFull, r.o[0], src);
                                again.o[1] = __shfl_sync(kFull, r.o[1], src);
                                again.o[2] = __shfl_sync(kFull, r.o[2], src);
                                const float4 sh = s_shear[warp0 + src];
                                again.sx = sh.x;
                                again.sy = sh.y;
                                again.sz = sh.z;
                                again.kxyz = __float_as_uint(sh.w);
                                if (prev != kNoLimit && boxes_may_exceed(again, ray_slack(again.o, box_slack(hd)),
                                                                         pr + (size_t)rec * 3u, ford_inv(prev)))
                                    best->z |= kLate;
                            }
                        } else if (prev != kNoLimit) {
                            const uint4 *p = pr + (size_t)rec * 3u;
                            const float limit = ford_inv(prev);
                            if (MULTI ? boxes_may_exceed(tr, p, limit)
                                      : boxes_may_exceed(tr, ray_slack(tr.o, box_slack(hd)), p, limit))
                                best->z |= kLate;
                        }
                        __syncwarp();
                    }
                    if (MIXED && any_ray) {
                        found = s_best[tid].w != kNone;
                        if (found) {
                            pending = false;
                            leaves = 0u;
                        }
                    } else {
                        tbest = ford_inv(s_t[tid]);
                    }
                }
                if (ANY || MIXED) m = __ballot_sync(kFull, leaves != 0u);  // a ray that is done appends no more
            }
            if (m == 0u) break;
        }
    }

    // ---- the rays set aside, each lane its own (one loop over rays and nodes: the
    // lanes' walks differ).  First whether the boxes above the hit found let the
    // ray in up to the nearest earlier hit: if so a walk in order tests it too.
    // Few boxes hold a given point, so that takes a tenth of a whole walk (23,000
    // of the walls' 1M rays, walked at the end of their warps: the launch took 1,150
    // us by whole walks alone, 1,037 so, 1,083 with every record tested on the
    // spot).  Only where its record is not reached that way the whole walk in order, every
    // record tested as its node is visited.
    if (!ANY) {
        uint32_t idx = kNone, next = aside, at = 0u, seen = 0u;
        uint32_t found_rec = kNone;  // the hit's record, kNone in the whole walk
        int depth = 0;
        bool walking = false;
        Hit h;
        h.t = 0.f; h.u = 0.f; h.v = 0.f; h.rec = kNone; h.tri = kNone;
        Ray w;
        w.prio = 0u;
        float t_lo = 0.f;
        uint2(&stack)[kMaxDepth + 1] = spill;
        for (;;) {
            if (!walking) {
                if (idx != kNone && found_rec != kNone) {
                    found_rec = kNone;
                    t_lo = __ldg(a.rays + 2u * idx).w;
                    h.t = __ldg(a.rays + 2u * idx + 1u).w;
                } else {
                    if (idx != kNone) write_hit(idx, h.tri != kNone, h.t, h.u, h.v, h.rec, h.tri);
                    idx = next;
                    if (idx == kNone) break;
                    const float4 kept = a.hits[idx];
                    next = __float_as_uint(kept.x);
                    found_rec = __float_as_uint(kept.y);
                    if (MULTI) scene_of(__ldg(a.ray_scene + idx));
                    const float4 r0 = __ldg(a.rays + 2u * idx), r1 = __ldg(a.rays + 2u * idx + 1u);
                    const float o[3] = {r0.x, r0.y, r0.z}, d[3] = {r1.x, r1.y, r1.z};
                    ray_setup(w, o, d);
                    h.t = kept.z;
                    t_lo = fmaxf(r0.w, kept.w - fabsf(kept.w) * 0x1p-16f);
                }
                h.tri = kNone;
                at = 0u;
                seen = 0u;
                depth = 0;
            }
            // (what the first walk reported of a corrupt structure is not reported again)
            walking = seen < max_visits && at < max_visits;
            if (!walking) continue;
            ++seen;
            const NodeWords nd = load_node(nodes, at);
            const uint32_t hits = isect_node(w, nd, t_lo, h.t);
            uint32_t recs = leaf_records(nd, hits);
            if (found_rec != kNone) {
                const uint32_t at_bit = found_rec - nd.w1.y;
                recs = at_bit < 24u ? recs & (1u << at_bit) : 0u;
                if (recs) {
                    t_lo = __ldg(a.rays + 2u * idx).w;
                    h.t = __ldg(a.rays + 2u * idx + 1u).w;
                }
            }
            const bool reached = found_rec != kNone && recs != 0u;
            for (; recs; recs &= recs - 1u) {
                const uint32_t rec = nd.w1.y + (uint32_t)__ffs((int)recs) - 1u;
                const uint4 *p = prims + (size_t)rec * 3u;
                const uint4 q0 = ldg4(p), q1 = ldg4(p + 1), q2 = ldg4(p + 2);
                float t, u, v;
                if (!isect_tri(w, xyz_of(q0), xyz_of(q1), xyz_of(q2), t_lo, h.t, t, u, v)) continue;
                if (t < h.t || q0.w < h.tri) {  // (t <= h.t)
                    h.t = t; h.u = u; h.v = v; h.rec = rec; h.tri = q0.w;
                }
            }
            if (reached) {
                found_rec = kNone;
                walking = false;
                continue;
            }
            uint2 g = child_group(nd, hits);
            if (!group_left(g) && depth > 0) g = stack[--depth];
            walking = group_left(g);
            at = take_child(g, w.prio);  // (of no group: unused)
            if (walking && group_left(g)) {
                if (depth < kMaxDepth) stack[depth++] = g;
                else walking = false;
            }
        }
    }
}

}  // namespace
}  // namespace rtc
