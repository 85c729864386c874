// rt_trace.cu -- BVH8 traversal kernels and the ray-tracing pipeline.
//
// Replaces traceRayEXT / vkCmdTraceRaysKHR of the reference sample
// (vulkan-raytraced-triangle/main.cpp:1047-1052 and :1349-1355), which run on
// RT cores inside the driver.  The GB300 has no RT cores, so traversal runs
// on the SMs:
//
//   k_trace_blas (rt_traverse.cuh)  persistent warps over a ray array
//                   with atomic work stealing and a shared-memory stack ring.
//   k_trace_inst    two-level structures (instances): persistent warps as
//                   above, a lane walking an instance's BLAS with its
//                   object-space ray between TLAS steps.
//                   Both kernels are launched; each returns at once when the
//                   structure in the header is not its kind.
//   k_pipeline      the sample's raygen + traceRayEXT + closest-hit / miss +
//                   imageStore, one thread per launch id.
//   k_trace_stats   node visits and triangle tests of a walk in order.
//
// Visiting order: a node's leaf records first, in ascending record order, then
// its internal children in ascending (slot ^ ray octant); remaining siblings
// are pushed as one group (identical in the CPU restatement, whose statistics
// k_trace_stats equals; the persistent kernels test records in batches).  Closest hit =
// smallest t, ties broken by the smallest (instance, triangle) key.
#include <cmath>
#include <cuda.h>
#include <cuda_runtime.h>
#include <sys/mman.h>
#include <unistd.h>

#include "rt_internal.h"
#include "../../include/rtcore_debug.h"
#include "rt_traverse.cuh"

namespace rtc {

namespace {

__device__ __forceinline__ bool key_less(float t, uint64_t key, float bt, uint64_t bkey) {
    return t < bt || (t == bt && key < bkey);
}

// ---------------------------------------------------------------------------
// Simple per-thread traversal (local-memory stack) for the sample pipeline
// (k_pipeline): one thread per pixel, both structure kinds.  Same visiting
// order as the persistent kernels.
// ---------------------------------------------------------------------------

struct LocalStack {
    uint2 e[kMaxDepth];
    int sp;
};

template <bool ANY>
__device__ bool traverse_blas_simple(const uint8_t *accel, Ray &r, float tmin, Hit &h, uint64_t &hkey,
                                     uint32_t inst, uint32_t *err) {
    const rt_accel_header *hd = reinterpret_cast<const rt_accel_header *>(accel);
    if (hd->prim_count == 0) return false;
    const uint4 *nodes = reinterpret_cast<const uint4 *>(accel + hd->node_offset);
    const uint4 *prims = reinterpret_cast<const uint4 *>(accel + hd->prim_offset);
    LocalStack st;
    st.sp = 0;
    uint32_t node = 0;
    bool sheared = false;  // r is set up for boxes, for triangles once it meets one
    // A tree walk visits each node at most once; more visits (or a node
    // index past the end) can only come from a corrupt structure.
    const uint32_t max_visits = hd->node_count;
    for (uint32_t visits = 0;; ++visits) {
        if (visits >= max_visits || node >= max_visits) {
            report_error(err, RT_ERR_BOUNDS, 0x74000000u | node);
            return h.found;
        }
        NodeWords nd = load_node(nodes, node);
        const uint32_t hits = isect_node(r, nd, tmin, h.t);
        uint32_t ph = leaf_records(nd, hits);
        const uint32_t pbase = nd.w1.y;
        while (ph) {
            uint32_t i = __ffs(ph) - 1;
            ph &= ph - 1u;
            const uint4 *rec = prims + (size_t)(pbase + i) * 3u;
            uint4 a = ldg4(rec), b = ldg4(rec + 1), c = ldg4(rec + 2);
            if (!sheared) ray_setup_shear(r);
            sheared = true;
            float t, u, v;
            if (!isect_tri(r, make_float4(__uint_as_float(a.x), __uint_as_float(a.y), __uint_as_float(a.z), 0.f),
                           make_float4(__uint_as_float(b.x), __uint_as_float(b.y), __uint_as_float(b.z), 0.f),
                           make_float4(__uint_as_float(c.x), __uint_as_float(c.y), __uint_as_float(c.z), 0.f),
                           tmin, h.t, t, u, v))
                continue;
            uint64_t key = ((uint64_t)inst << 32) | a.w;
            if (ANY) {
                h.t = t; h.u = u; h.v = v; h.rec = pbase + i; h.tri = a.w; h.inst = inst; h.found = true;
                return true;
            }
            if (key_less(t, key, h.t, hkey)) {
                h.t = t; h.u = u; h.v = v; h.rec = pbase + i; h.tri = a.w; h.inst = inst; h.found = true;
                hkey = key;
            }
        }
        uint2 g = child_group(nd, hits);
        for (;;) {
            if (group_left(g)) {
                node = take_child(g, r.prio);
                if (group_left(g)) {
                    if (st.sp >= kMaxDepth) {
                        report_error(err, RT_ERR_BOUNDS, 0x70000000u);
                        return h.found;
                    }
                    st.e[st.sp++] = g;
                }
                break;
            }
            if (st.sp == 0) return false;
            g = st.e[--st.sp];
        }
    }
}

struct InstRec {
    float w2o[12];
    uint64_t accel_ref;
    uint32_t cim, sof, id;
};

__device__ __forceinline__ InstRec load_inst(const uint4 *prims, uint32_t i) {
    const uint4 *p = prims + (size_t)i * 5u;
    uint4 a = ldg4(p), b = ldg4(p + 1), c = ldg4(p + 2), d = ldg4(p + 3), e = ldg4(p + 4);
    InstRec r;
    r.w2o[0] = __uint_as_float(a.x); r.w2o[1] = __uint_as_float(a.y); r.w2o[2] = __uint_as_float(a.z);
    r.w2o[3] = __uint_as_float(a.w); r.w2o[4] = __uint_as_float(b.x); r.w2o[5] = __uint_as_float(b.y);
    r.w2o[6] = __uint_as_float(b.z); r.w2o[7] = __uint_as_float(b.w); r.w2o[8] = __uint_as_float(c.x);
    r.w2o[9] = __uint_as_float(c.y); r.w2o[10] = __uint_as_float(c.z); r.w2o[11] = __uint_as_float(c.w);
    r.accel_ref = (uint64_t)d.x | ((uint64_t)d.y << 32);
    r.cim = d.z;
    r.sof = d.w;
    r.id = e.x;
    return r;
}

struct HitIds {
    uint32_t custom, sbt_off, geom, prim;
};

// Full closest/any traversal of a top- or bottom-level structure.
template <bool ANY>
__device__ bool trace_ray(const uint8_t *accel, const float o[3], const float d[3], float tmin, float tmax,
                          uint32_t cull_mask, Hit &h, HitIds &ids, uint32_t *err) {
    const rt_accel_header *hd = reinterpret_cast<const rt_accel_header *>(accel);
    h.t = tmax; h.u = 0.f; h.v = 0.f; h.rec = kNone; h.tri = kNone; h.inst = 0; h.found = false;
    ids.custom = 0; ids.sbt_off = 0; ids.geom = 0; ids.prim = 0;
    if (!(tmin <= tmax)) return false;  // an empty interval, a NaN limit
    uint64_t hkey = ~0ull;
    Ray r;
    ray_setup_box(r, o, d);
    const uint8_t *hit_blas = accel;
    if (hd->kind == RT_ACCEL_KIND_BLAS) {
        bool any = traverse_blas_simple<ANY>(accel, r, tmin, h, hkey, 0u, err);
        if (h.found) {
            const uint4 *prims = reinterpret_cast<const uint4 *>(accel + hd->prim_offset);
            ids.geom = ldg4(prims + (size_t)h.rec * 3u + 1).w;
            ids.prim = ldg4(prims + (size_t)h.rec * 3u + 2).w;
        }
        return ANY ? any : h.found;
    }
    if (hd->prim_count == 0) return false;
    const uint4 *nodes = reinterpret_cast<const uint4 *>(accel + hd->node_offset);
    const uint4 *prims = reinterpret_cast<const uint4 *>(accel + hd->prim_offset);
    LocalStack st;
    st.sp = 0;
    uint32_t node = 0;
    bool done = false;
    for (uint32_t visits = 0; !done; ++visits) {
        if (visits >= hd->node_count || node >= hd->node_count) {
            report_error(err, RT_ERR_BOUNDS, 0x75000000u | node);
            break;
        }
        NodeWords nd = load_node(nodes, node);
        const uint32_t hits = isect_node(r, nd, tmin, h.t);
        uint32_t ph = leaf_records(nd, hits);
        const uint32_t pbase = nd.w1.y;
        while (ph && !(ANY && h.found)) {
            uint32_t i = __ffs(ph) - 1;
            ph &= ph - 1u;
            InstRec ir = load_inst(prims, pbase + i);
            if (((ir.cim >> 24) & cull_mask) == 0u || ir.accel_ref == 0u) continue;
            float o2[3], d2[3];
            xform_point(ir.w2o, o, o2);
            xform_vector(ir.w2o, d, d2);
            Ray r2;
            ray_setup_box(r2, o2, d2);
            const uint8_t *blas = reinterpret_cast<const uint8_t *>(ir.accel_ref);
            bool hit = traverse_blas_simple<ANY>(blas, r2, tmin, h, hkey, ir.id, err);
            // instances occur once in a TLAS: a best hit carrying this id
            // was found in this instance's BLAS
            if (h.found && h.inst == ir.id) {
                ids.custom = ir.cim & 0xffffffu;
                ids.sbt_off = ir.sof & 0xffffffu;
                hit_blas = blas;
            }
            if (ANY && hit) break;
        }
        if (ANY && h.found) break;
        uint2 g = child_group(nd, hits);
        for (;;) {
            if (group_left(g)) {
                node = take_child(g, r.prio);
                if (group_left(g)) {
                    if (st.sp >= kMaxDepth) {
                        report_error(err, RT_ERR_BOUNDS, 0x71000000u);
                        done = true;
                        break;
                    }
                    st.e[st.sp++] = g;
                }
                break;
            }
            if (st.sp == 0) { done = true; break; }
            g = st.e[--st.sp];
        }
    }
    if (h.found && hit_blas) {
        const rt_accel_header *bh = reinterpret_cast<const rt_accel_header *>(hit_blas);
        const uint4 *bp = reinterpret_cast<const uint4 *>(hit_blas + bh->prim_offset);
        ids.geom = ldg4(bp + (size_t)h.rec * 3u + 1).w;
        ids.prim = ldg4(bp + (size_t)h.rec * 3u + 2).w;
    }
    return h.found;
}


// Two-level structures (instances), persistent like k_trace_blas, with its
// triangle queue: warps refill idle lanes from the work counter, stacks live
// in a shared-memory ring whose bottom spills to local memory.  At a TLAS node
// a lane saves the internal children on its stack and stops for the node's
// instances; to enter one it saves the instances left and a return entry and
// walks the instance's BLAS with the object-space ray.  When that walk is over
// it takes the world ray back from shared memory and goes on in the TLAS.
// Closest hit = smallest t, ties broken by the smallest (instance, triangle)
// key.  Launched beside k_trace_blas; each kernel returns at once when the
// structure is not its kind.
//
// A lane enters an instance every few nodes, and the entry (80 bytes of
// record, a transformed ray, its divisions) costs more than a node, so lanes
// stop for it and are served together, with those that need a new ray, once a
// quarter of the lanes with a ray (or the refill threshold) have stopped:
// entered on the spot, the entry and the triangle tests ran with a few lanes
// each (10.5 active threads per instruction).  807K rays in 64 instances of
// three meshes: 1,008 -> 810 us (then a fixed 4 / 8 / 16 stopped lanes 863 / 871 /
// 971, a third or an eighth of the lanes 811 / 821).  What bounds it now: issue
// slots, half of them in steps of warps whose last rays (of up to hundreds of
// nodes) are under way.
//
// The answer is that of a walk in order (see boxes_may_exceed): a lane goes on
// in the TLAS, and enters the next instance, with every triangle it has met
// tested, so the TLAS nodes' boxes and an instance's first meet the same far
// limit as there, and only hits within one instance can have come too late for
// its boxes.
constexpr uint32_t kInstGroup = 0x40000000u;   // stack entry: instances of a TLAS node still to walk
constexpr int kInstDepth = 128;                // stack entries per ray (both levels)
constexpr uint32_t kInstBlocksPerSm = 6;       // 80 registers (7 blocks: 72, within 1 %)

// Whether the boxes of an instance's BLAS let the ray in up to `limit` all the
// way down to leaf record `rec`; if so h and ids are that record's hit.
__device__ bool confirm_hit(const uint4 *tprims, const float o[3], const float d[3], float tmin, float tmax, uint32_t rec,
                            uint32_t inst_rec, float limit, Hit &h, HitIds &ids) {
    const InstRec ir = load_inst(tprims, inst_rec);
    const uint8_t *blas = reinterpret_cast<const uint8_t *>(ir.accel_ref);
    const rt_accel_header *bh = reinterpret_cast<const rt_accel_header *>(blas);
    const uint4 *nodes = reinterpret_cast<const uint4 *>(blas + bh->node_offset);
    const uint4 *p = reinterpret_cast<const uint4 *>(blas + bh->prim_offset) + (size_t)rec * 3u;
    const uint32_t count = bh->node_count;
    float o2[3], d2[3];
    xform_point(ir.w2o, o, o2);
    xform_vector(ir.w2o, d, d2);
    Ray r;
    ray_setup(r, o2, d2);
    const uint4 q0 = ldg4(p), q1 = ldg4(p + 1), q2 = ldg4(p + 2);
    if (!isect_tri(r, xyz_of(q0), xyz_of(q1), xyz_of(q2), tmin, tmax, h.t, h.u, h.v)) return false;
    const float t_lo = fmaxf(tmin, h.t - fabsf(h.t) * 0x1p-16f);
    uint2 stack[kMaxDepth];
    int depth = 0;
    uint32_t node = 0u;
    for (uint32_t visits = 0; visits < count && node < count; ++visits) {
        const NodeWords nd = load_node(nodes, node);
        const uint32_t hits = isect_node(r, nd, t_lo, limit), bit = rec - nd.w1.y;
        if (bit < 24u && ((leaf_records(nd, hits) >> bit) & 1u)) {
            h.rec = rec;
            h.tri = q0.w;
            h.inst = ir.id;
            h.found = true;
            ids.custom = ir.cim & 0xffffffu;
            ids.sbt_off = ir.sof & 0xffffffu;
            ids.geom = q1.w;
            ids.prim = q2.w;
            return true;
        }
        uint2 g = child_group(nd, hits);
        if (!group_left(g) && depth > 0) g = stack[--depth];
        if (!group_left(g)) return false;
        node = take_child(g, r.prio);
        if (group_left(g)) {
            if (depth == kMaxDepth) return false;
            stack[depth++] = g;
        }
    }
    return false;
}

template <bool ANY>
__global__ void __launch_bounds__(kTraceThreads, kInstBlocksPerSm) k_trace_inst(const BatchArgs a) {
    pdl_wait();
    const rt_accel_header *hd = reinterpret_cast<const rt_accel_header *>(a.accel);
    if (hd->kind != RT_ACCEL_KIND_TLAS) return;
    const uint4 *tnodes = reinterpret_cast<const uint4 *>(a.accel + hd->node_offset);
    const uint4 *tprims = reinterpret_cast<const uint4 *>(a.accel + hd->prim_offset);
    const uint32_t t_count = hd->node_count;
    const bool t_empty = hd->prim_count == 0;
    __shared__ uint2 s_stack[kRing][kTraceThreads];
    __shared__ uint2 s_queue[kTraceThreads / 32][kTriQueue];  // leaf record, lane | step << 5
    // per lane: the world ray (origin, visiting order; inverse direction, the
    // ray's index); the triangle test's part of the object-space ray of the
    // instance entered last (origin, tmin; shear); the best hit so far -- t as
    // an ordered integer; instance and triangle (~0: no hit); u, v, leaf record
    // and the instance's record
    __shared__ float4 s_world[2][kTraceThreads];
    __shared__ float4 s_object[2][kTraceThreads];
    __shared__ int32_t s_t[ANY ? 1 : kTraceThreads];
    __shared__ unsigned long long s_key[ANY ? 1 : kTraceThreads];
    __shared__ uint4 s_best[ANY ? 1 : kTraceThreads];
    // within the instance: the step (node visit) of the best hit (0: none), the
    // nearest hit of an earlier step, as an ordered integer
    __shared__ uint32_t s_step[ANY ? 1 : kTraceThreads];
    __shared__ int32_t s_prev[ANY ? 1 : kTraceThreads];
    constexpr uint32_t kFull = 0xffffffffu;
    const int tid = threadIdx.x, lane = tid & 31;
    uint2 *queue = s_queue[tid >> 5];
    const int warp0 = tid & ~31;  // lane 0's thread
    // (one more entry than the stack's: the last ray set aside)
    uint2 spill[kInstDepth + 1];
    uint32_t &aside = spill[kInstDepth].x;
    aside = kNone;

    bool have_ray = false, exhausted = false, pending = false, in_blas = false, found = false;
    Ray r;  // the current level's ray
    r.o[0] = r.o[1] = r.o[2] = 0.f;
    r.prio = 0u;
    float tmin = 0.f, tbest = 0.f;  // tbest: the ray's far limit, then its best hit
    const uint4 *nodes = tnodes, *prims = nullptr;  // the current level's nodes; the instance's leaf records
    uint32_t node = 0, visits = 0, count = 0;       // a walk visits each node of a level at most once
    uint32_t inst_id = 0, inst_rec = 0;
    uint2 ig = make_uint2(0u, 0u);  // instances of a TLAS node to enter: the lane is stopped
    int sp = 0, lo = 0, sp_blas = 0;
    uint32_t head = 0, tail = 0;  // queue positions tested / appended so far (the same in every lane)
    uint32_t last = ~0u;          // position of this lane's latest entry
    uint32_t step = 0u;           // node visits of the warp so far
    uint32_t error = 0u;          // detail word of an error this lane's ray met
    const uint32_t n_rays = a.n;
    // fewer rays than lanes: see k_trace_blas (8 / 31 / 129 rays of 64 instances
    // 147 / 249 / 260 us in full warps, 130 / 207 / 244 spread)
    const uint32_t share = n_rays / (gridDim.x * (kTraceThreads / 32)) + 1u;
    const uint32_t lanes = share >= 32u ? kFull : (1u << share) - 1u;
    const int refill = (int)min(a.refill, min(share, 32u));

    auto push = [&](uint2 e) {
        if (sp - lo == kRing) {
            spill[lo] = s_stack[lo & (kRing - 1)][tid];
            ++lo;
        }
        s_stack[sp & (kRing - 1)][tid] = e;
        ++sp;
    };
    auto pop = [&]() {
        --sp;
        uint2 e = s_stack[sp & (kRing - 1)][tid];
        if (sp < lo) {
            e = spill[sp];
            lo = sp;
        }
        return e;
    };
    auto fail = [&](uint32_t detail) {  // the walk ends here
        pending = false;
        ig.y = 0u;
        error = detail;
    };

    auto world_ray = [&]() {  // back to the TLAS
        in_blas = false;
        nodes = tnodes;
        count = t_count;
        const float4 w0 = s_world[0][tid], w1 = s_world[1][tid];
        r.o[0] = w0.x; r.o[1] = w0.y; r.o[2] = w0.z;
        r.prio = __float_as_uint(w0.w);
        r.invd[0] = w1.x; r.invd[1] = w1.y; r.invd[2] = w1.z;
    };

    auto write_hit = [&](uint32_t ray_idx, bool hit, float t, float u, float v, uint32_t inst, uint32_t tri,
                         const HitIds &ids) {
        const float4 out = hit ? make_float4(t, __uint_as_float(tri), u, v)
                               : make_float4(kInf, __uint_as_float(kNone), 0.f, 0.f);
        if (a.hits) a.hits[ray_idx] = out;
        if (a.hits_ext) {
            rt_hit_ext x;
            x.t = out.x; x.u = out.z; x.v = out.w;
            x.instance_id = hit ? inst : kNone;
            x.custom_index = hit ? ids.custom : 0u;
            x.geometry_index = hit ? ids.geom : 0u;
            x.primitive_id = hit ? ids.prim : kNone;
            x.sbt_record = hit ? ids.sbt_off + ids.geom : 0u;
            a.hits_ext[ray_idx] = x;
        }
    };

    for (;;) {
        // ---- stopped lanes whose queued triangles are tested: result and new
        // ray, or the next instance
        const bool waiting = (int)(last - head) >= 0;
        const uint32_t ready =
            __ballot_sync(kFull, !pending && !waiting && (have_ray || (!exhausted && ((lanes >> lane) & 1u))));
        // (the far limit a TLAS node's boxes meet is that of every triangle met
        // before, so that what a walk in order tests there is the same)
        bool can_step = pending && (ANY || in_blas || !waiting);
        uint32_t walking = __ballot_sync(kFull, can_step);
        // stopped lanes to wait for: they stand idle until served
        const int serve = max(1 + __popc(__ballot_sync(kFull, have_ray)) / 4, exhausted ? 0 : refill);
        if (__popc(ready) >= serve || (walking == 0u && tail == head)) {
            if (ready == 0u) break;  // every lane is done
            const bool mine = (ready >> lane) & 1u;
            const bool enter = mine && ig.y != 0u;
            if (mine && have_ray && !enter) {
                have_ray = false;
                const uint32_t ray_idx = __float_as_uint(s_world[1][tid].w);
                if (error) {
                    report_error(a.err, RT_ERR_BOUNDS, error);
                    error = 0u;
                }
                if (ANY) {
                    if (a.occluded) a.occluded[ray_idx] = found ? 1u : 0u;
                } else {
                    const uint4 best = s_best[tid];
                    const unsigned long long key = s_key[tid];
                    const bool hit = key != ~0ull;
                    if (hit && (best.z & kLate)) {
                        const uint32_t rec = best.z & ~(kMinusZero | kLate);
                        a.hits[ray_idx] = make_float4(__uint_as_float(aside), __uint_as_float(rec),
                                                      __uint_as_float(best.w), ford_inv(s_prev[tid]));
                        aside = ray_idx;
                    } else {
                        const uint32_t rec = best.z & ~kMinusZero;
                        HitIds ids;
                        ids.custom = ids.sbt_off = ids.geom = ids.prim = 0u;
                        if (hit && a.hits_ext) {
                            const InstRec ir = load_inst(tprims, best.w);
                            const uint8_t *blas = reinterpret_cast<const uint8_t *>(ir.accel_ref);
                            const rt_accel_header *bh = reinterpret_cast<const rt_accel_header *>(blas);
                            const uint4 *bp = reinterpret_cast<const uint4 *>(blas + bh->prim_offset);
                            ids.custom = ir.cim & 0xffffffu;
                            ids.sbt_off = ir.sof & 0xffffffu;
                            ids.geom = ldg4(bp + (size_t)rec * 3u + 1).w;
                            ids.prim = ldg4(bp + (size_t)rec * 3u + 2).w;
                        }
                        write_hit(ray_idx, hit, (best.z & kMinusZero) ? -0.0f : tbest, __uint_as_float(best.x),
                                  __uint_as_float(best.y), (uint32_t)(key >> 32), (uint32_t)key, ids);
                    }
                }
            }
            float o[3], d[3], slack = 0.0f;
            bool fresh = false, entered = false;
            const uint32_t want = __ballot_sync(kFull, mine && !have_ray) & lanes;
            if (want != 0u && !exhausted) {
                const uint32_t cnt = __popc(want);
                uint32_t first = 0;
                if (lane == 0) first = atomicAdd(a.counter, cnt);
                first = __shfl_sync(kFull, first, 0);
                if (first + cnt >= n_rays) exhausted = true;
                const uint32_t idx = first + __popc(want & ((1u << lane) - 1u));
                if (((want >> lane) & 1u) && idx < n_rays) {
                    const float4 r0 = __ldg(a.rays + 2u * idx), r1 = __ldg(a.rays + 2u * idx + 1u);
                    o[0] = r0.x; o[1] = r0.y; o[2] = r0.z;
                    d[0] = r1.x; d[1] = r1.y; d[2] = r1.z;
                    s_world[1][tid].w = __uint_as_float(idx);
                    tmin = r0.w;
                    tbest = r1.w;
                    found = false;
                    if (!ANY) {
                        s_t[tid] = ford(tbest + 0.0f);  // -0 and +0 tie
                        s_key[tid] = ~0ull;
                    }
                    have_ray = true;
                    in_blas = false;
                    nodes = tnodes;
                    node = 0;
                    visits = 0;
                    count = t_count;
                    pending = !t_empty;
                    if (!(tmin <= tbest)) {  // a miss, a NaN limit too
                        tmin = kInf;
                        tbest = -kInf;
                    }
                    sp = 0;
                    lo = 0;
                    last = head - 1u;
                    fresh = true;
                }
            }
            if (enter) {
                const uint32_t rec = ig.x + (uint32_t)__ffs((int)ig.y) - 1u;
                ig.y &= ig.y - 1u;
                const InstRec ir = load_inst(tprims, rec);
                const uint8_t *blas = reinterpret_cast<const uint8_t *>(ir.accel_ref);
                const rt_accel_header *bh = reinterpret_cast<const rt_accel_header *>(blas);
                if (((ir.cim >> 24) & 0xffu) == 0u || !blas || bh->prim_count == 0u) {
                    // masked out (cull mask 0xFF), without a structure (its box
                    // is empty, but a ray of NaNs enters any) or empty: on to the next
                    // instance, else to what the stack holds
                    if (ig.y == 0u && sp > 0) {
                        uint2 g = pop();
                        if (g.y & kInstGroup) {
                            ig = make_uint2(g.x, g.y & ~kInstGroup);
                        } else {
                            node = take_child(g, r.prio);
                            if (group_left(g)) push(g);
                            pending = true;
                        }
                    }
                } else if (sp + 2 > kInstDepth) {
                    fail(0x71000000u);
                } else {
                    if (ig.y) push(make_uint2(ig.x, ig.y | kInstGroup));
                    ig.y = 0u;
                    push(make_uint2(visits, 0u));  // the TLAS walk's, while the BLAS walk counts its own
                    sp_blas = sp;
                    const float4 w0 = s_world[0][tid];
                    const float4 r1 = __ldg(a.rays + 2u * __float_as_uint(s_world[1][tid].w) + 1u);
                    const float wo[3] = {w0.x, w0.y, w0.z}, wd[3] = {r1.x, r1.y, r1.z};
                    xform_point(ir.w2o, wo, o);
                    xform_vector(ir.w2o, wd, d);
                    in_blas = true;
                    nodes = reinterpret_cast<const uint4 *>(blas + bh->node_offset);
                    prims = reinterpret_cast<const uint4 *>(blas + bh->prim_offset);
                    node = 0;
                    visits = 0;
                    count = bh->node_count;
                    inst_id = ir.id;
                    inst_rec = rec;
                    if (!ANY) {
                        s_step[tid] = 0u;
                        slack = box_slack(bh);
                    }
                    pending = true;
                    entered = true;
                }
            }
            if (fresh || entered) {
                ray_setup(r, o, d);
                if (fresh) {
                    s_world[0][tid] = make_float4(o[0], o[1], o[2], __uint_as_float(r.prio));
                    s_world[1][tid].x = r.invd[0];
                    s_world[1][tid].y = r.invd[1];
                    s_world[1][tid].z = r.invd[2];
                } else {
                    s_object[0][tid] = make_float4(o[0], o[1], o[2], tmin);
                    s_object[1][tid] =
                        make_float4(r.sx, r.sy, r.sz, __uint_as_float(ANY ? r.kxyz : pack_slack(r, o, slack)));
                }
            }
            can_step = pending && (ANY || in_blas || !((int)(last - head) >= 0));
            walking = __ballot_sync(kFull, can_step);
            if (walking == 0u) continue;
        }
        const uint32_t held = __ballot_sync(kFull, !can_step && (int)(last - head) >= 0);
        const int busy = __popc(walking | held);  // lanes whose triangles may be queued
        // a partial batch once stopped lanes wait for it
        const bool drain = walking == 0u || __popc(held) + __popc(ready & ~walking) >= serve;

        // ---- one node per lane, then the lane's next node (see k_trace_blas)
        ++step;
        uint32_t leaves = 0u, nth = 0u, meta_lo = 0u, meta_hi = 0u, pbase = 0u;
        if (can_step && (visits >= count || node >= count)) {
            can_step = false;
            fail((in_blas ? 0x74000000u : 0x75000000u) | (node & 0xffffffu));
        }
        if (can_step) {
            ++visits;
            const NodeWords nd = load_node(nodes, node);
            const uint32_t hits = isect_node(r, nd, tmin, tbest);
            meta_lo = nd.w1.z;
            meta_hi = nd.w1.w;
            pbase = nd.w1.y;
            uint2 g = child_group(nd, hits);
            leaves = hits & ~(nd.w0.w >> 24);
            if (!in_blas) {
                if (leaves) {
                    ig = make_uint2(pbase, leaf_records(nd, hits));
                    leaves = 0u;
                }
                if (ig.y && group_left(g)) {
                    push(g);
                    g.y = 0u;
                }
            }
            const bool next = ig.y == 0u && !group_left(g);
            if (next && in_blas && sp == sp_blas) {
                visits = pop().x;
                world_ray();
            }
            if (next && sp > 0) {
                g = pop();
                if (g.y & kInstGroup) {
                    ig = make_uint2(g.x, g.y & ~kInstGroup);
                    g.y = 0u;
                }
            }
            pending = group_left(g);
            node = take_child(g, r.prio);  // (of no group: unused)
            if (pending && group_left(g)) push(g);
            if (sp > kInstDepth) fail(in_blas ? 0x70000000u : 0x71000000u);
        }

        // ---- append the leaf records met, test a batch when there is one
        uint32_t m = __ballot_sync(kFull, leaves != 0u);
        while (m != 0u || (drain && tail != head)) {
            if (leaves) {
                const uint32_t meta = __byte_perm(meta_lo, meta_hi, (uint32_t)__ffs((int)leaves) - 1u) & 0xffu;
                last = tail + __popc(m & ((1u << lane) - 1u));
                queue[last & (kTriQueue - 1u)] =
                    make_uint2((meta & 0x20u) ? pbase + (meta & 0x1fu) + nth : kNone, step << 5 | (uint32_t)lane);
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
                __syncwarp();  // read before the next append reuses the slots
                head += k;
                const float4 ob = s_object[0][warp0 + src], shear = s_object[1][warp0 + src];
                Ray tr;
                tr.o[0] = ob.x; tr.o[1] = ob.y; tr.o[2] = ob.z;
                tr.sx = shear.x;
                tr.sy = shear.y;
                tr.sz = shear.z;
                tr.kxyz = __float_as_uint(shear.w);
                const float t_hi = __shfl_sync(kFull, tbest, src);
                const uint4 *pr = reinterpret_cast<const uint4 *>(
                    __shfl_sync(kFull, (unsigned long long)reinterpret_cast<uintptr_t>(prims), src));
                const uint32_t inst = ANY ? 0u : __shfl_sync(kFull, inst_id, src);
                const uint32_t irec = ANY ? 0u : __shfl_sync(kFull, inst_rec, src);
                float t = 0.f, u = 0.f, v = 0.f;
                uint32_t tri = kNone;
                bool hit = false;
                if (rec != kNone) {
                    const uint4 *p = pr + (size_t)rec * 3u;
                    const uint4 q0 = ldg4(p), q1 = ldg4(p + 1), q2 = ldg4(p + 2);
                    tri = q0.w;
                    hit = isect_tri(tr, xyz_of(q0), xyz_of(q1), xyz_of(q2), ob.w, t_hi, t, u, v);
                }
                if (ANY) {
                    const uint32_t fm = __reduce_or_sync(kFull, hit ? 1u << src : 0u);
                    if ((fm >> lane) & 1u) {
                        found = true;
                        pending = false;
                        ig.y = 0u;
                        leaves = 0u;
                    }
                    m = __ballot_sync(kFull, leaves != 0u);  // a ray that is done appends no more
                } else {
                    // the owner's best: least t, then, among the lanes that
                    // reached it, least (instance, triangle) (an improved t
                    // clears the key of the old one)
                    const int32_t tk = ford(t + 0.0f);  // -0 and +0 tie
                    const unsigned long long key = (unsigned long long)inst << 32 | tri;
                    int32_t *bt = s_t + warp0 + src;
                    unsigned long long *bk = s_key + warp0 + src;
                    const uint32_t own = e.y >> 5;
                    const bool hit_too = hit;
                    if (__any_sync(kFull, hit)) {
                        if (hit && atomicMin(bt, tk) > tk) *bk = ~0ull;
                        __syncwarp();
                        hit = hit && *bt == tk;
                        if (hit) atomicMin(bk, key);
                        __syncwarp();
                        hit = hit && *bk == key;
                        if (hit) {
                            const uint32_t before = s_step[warp0 + src];
                            s_step[warp0 + src] = own;
                            if (before != own) s_prev[warp0 + src] = before ? ford(t_hi + 0.0f) : kNoLimit;
                            s_best[warp0 + src] =
                                make_uint4(__float_as_uint(u), __float_as_uint(v),
                                           rec | (__float_as_uint(t) == kMinusZero ? kMinusZero : 0u), irec);
                        }
                        __syncwarp();
                        if (hit_too && !hit && own < s_step[warp0 + src]) atomicMin(s_prev + warp0 + src, tk);
                        __syncwarp();
                        if (hit) {  // see boxes_may_exceed
                            const int32_t prev = s_prev[warp0 + src];
                            if (prev != kNoLimit && boxes_may_exceed(tr, pr + (size_t)rec * 3u, ford_inv(prev)))
                                s_best[warp0 + src].z |= kLate;
                        }
                        __syncwarp();
                    }
                    tbest = ford_inv(s_t[tid]);
                }
            }
            if (m == 0u) break;
        }
    }

    // ---- the rays set aside: see k_trace_blas; the hit is confirmed within its
    // instance
    if (!ANY) {
        uint32_t next = kNone;
        for (uint32_t i = aside; i != kNone; i = next) {
            const float4 kept = a.hits[i];
            next = __float_as_uint(kept.x);
            const float4 r0 = __ldg(a.rays + 2u * i), r1 = __ldg(a.rays + 2u * i + 1u);
            const float o[3] = {r0.x, r0.y, r0.z}, d[3] = {r1.x, r1.y, r1.z};
            Hit h;
            HitIds ids;
            if (!confirm_hit(tprims, o, d, r0.w, r1.w, __float_as_uint(kept.y), __float_as_uint(kept.z), kept.w, h, ids))
                trace_ray<false>(a.accel, o, d, r0.w, r1.w, 0xffu, h, ids, a.err);
            write_hit(i, h.found, h.t, h.u, h.v, h.inst, h.tri, ids);
        }
    }
}

// Traversal statistics (rt_trace_stats): node visits and triangle tests of a
// walk in the order of the CPU restatement, which tests a node's triangles as it
// visits the node (the kernels above test some more).  Persistent warps and the
// stack of the kernels above, a kernel per structure kind.  2M rays of the 1M
// soup: closest hits 1,558 us, any hit 1,273 at nine blocks per SM, 1,562 and
// 1,300 at eight (one thread per ray 3,436 and 2,650; both kinds in one kernel
// 1,616 and 1,343); 800K rays in 64 instances: 1,238 and 1,157 at eight, 1,261
// and 1,175 at nine.
constexpr uint32_t stats_blocks_per_sm(bool top) { return top ? 8u : 9u; }

// isect_node under a NaN limit, as the CPU restatement compares: a child is hit
// where tnear <= tfar, so not where either is NaN.
__device__ uint32_t isect_node_nan(const Ray &r, const NodeWords &n, float tmin, float tcur) {
    const float p[3] = {__uint_as_float(n.w0.x), __uint_as_float(n.w0.y), __uint_as_float(n.w0.z)};
    const uint32_t lo[6] = {n.w2.x, n.w2.y, n.w2.z, n.w2.w, n.w3.x, n.w3.y};
    const uint32_t hi[6] = {n.w3.z, n.w3.w, n.w4.x, n.w4.y, n.w4.z, n.w4.w};
    uint32_t hits = 0u;
    for (int s = 0; s < 8; ++s) {
        float tn = tmin, tf = tcur;
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            const float sc = pow2f((int)(int8_t)(n.w0.w >> (8 * a))) * r.invd[a], adj = (p[a] - r.o[a]) * r.invd[a];
            const uint32_t wl = s < 4 ? lo[2 * a] : lo[2 * a + 1], wh = s < 4 ? hi[2 * a] : hi[2 * a + 1];
            const float ql = (float)((wl >> (8 * (s & 3))) & 0xffu), qh = (float)((wh >> (8 * (s & 3))) & 0xffu);
            const bool neg = r.invd[a] < 0.0f;
            tn = fmaxf(tn, __fmaf_rn(neg ? qh : ql, sc, adj));
            tf = fminf(tf, __fmaf_rn(neg ? ql : qh, sc, adj));
        }
        if (tn <= tf * kTfarScale) hits |= 1u << s;
    }
    return hits;
}

template <bool ANY, bool TOP>
__global__ void __launch_bounds__(kTraceThreads, stats_blocks_per_sm(TOP))
k_trace_stats(const uint8_t *accel, const float4 *rays, uint32_t n, uint32_t refill, uint32_t *counter,
              unsigned long long *counters, uint32_t *err) {
    const rt_accel_header *hd = reinterpret_cast<const rt_accel_header *>(accel);
    if (hd->kind != (TOP ? RT_ACCEL_KIND_TLAS : RT_ACCEL_KIND_BLAS)) return;
    const uint4 *tnodes = reinterpret_cast<const uint4 *>(accel + hd->node_offset);
    const uint4 *tprims = reinterpret_cast<const uint4 *>(accel + hd->prim_offset);
    const uint32_t t_count = hd->node_count;
    const bool empty = hd->prim_count == 0;
    __shared__ uint2 s_stack[kRing][kTraceThreads];
    constexpr uint32_t kFull = 0xffffffffu;
    constexpr uint32_t kReturn = 0x80000000u;  // stack entry: back to the TLAS, its visits so far
    const int tid = threadIdx.x, lane = tid & 31;
    bool walking = false, exhausted = false, in_blas = false;
    Ray r;
    r.prio = 0u;
    const uint4 *nodes = tnodes, *prims = tprims;
    uint32_t ray = 0, node = 0, visits = 0, count = 0;
    float tmin = 0.f, tbest = 0.f;
    int sp = 0, lo = 0;
    uint2 spill[kInstDepth + 1];
    unsigned long long n_nodes = 0ull, n_tris = 0ull;

    auto push = [&](uint2 e) {
        if (sp - lo == kRing) {
            spill[lo] = s_stack[lo & (kRing - 1)][tid];
            ++lo;
        }
        s_stack[sp & (kRing - 1)][tid] = e;
        ++sp;
    };
    auto pop = [&]() {
        --sp;
        uint2 e = s_stack[sp & (kRing - 1)][tid];
        if (sp < lo) {
            e = spill[sp];
            lo = sp;
        }
        return e;
    };
    auto load_ray = [&](float (&o)[3], float (&d)[3]) {
        const float4 r0 = __ldg(rays + 2u * ray), r1 = __ldg(rays + 2u * ray + 1u);
        o[0] = r0.x; o[1] = r0.y; o[2] = r0.z;
        d[0] = r1.x; d[1] = r1.y; d[2] = r1.z;
        return make_float2(r0.w, r1.w);
    };
    auto fail = [&](uint32_t detail) {
        report_error(err, RT_ERR_BOUNDS, detail);
        walking = false;
    };

    for (;;) {
        const uint32_t idle = __ballot_sync(kFull, !walking);
        if (idle == kFull && exhausted) break;
        if (!exhausted && (uint32_t)__popc(idle) >= refill) {
            uint32_t first = 0;
            if (lane == 0) first = atomicAdd(counter, (uint32_t)__popc(idle));
            first = __shfl_sync(kFull, first, 0);
            if (first + (uint32_t)__popc(idle) >= n) exhausted = true;
            const uint32_t idx = first + __popc(idle & ((1u << lane) - 1u));
            if (!walking && idx < n && !empty) {
                ray = idx;
                float o[3], d[3];
                const float2 limits = load_ray(o, d);
                ray_setup(r, o, d);
                tmin = limits.x;
                tbest = limits.y;
                walking = true;
                in_blas = !TOP;
                nodes = tnodes;
                prims = tprims;
                count = t_count;
                node = 0;
                visits = 0;
                sp = 0;
                lo = 0;
            }
        }
        if (!walking) continue;
        if (visits >= count || node >= count) {
            fail((in_blas ? 0x74000000u : 0x75000000u) | (node & 0xffffffu));
            continue;
        }
        ++visits;
        ++n_nodes;
        const NodeWords nd = load_node(nodes, node);
        const bool limits = tmin == tmin && tbest == tbest;
        const uint32_t hits = limits ? isect_node(r, nd, tmin, tbest) : isect_node_nan(r, nd, tmin, tbest);
        uint2 g = child_group(nd, hits), ig = make_uint2(nd.w1.y, leaf_records(nd, hits));
        if (!TOP || in_blas) {
            for (; ig.y; ig.y &= ig.y - 1u) {
                const uint4 *p = prims + (size_t)(ig.x + (uint32_t)__ffs((int)ig.y) - 1u) * 3u;
                const uint4 q0 = ldg4(p), q1 = ldg4(p + 1), q2 = ldg4(p + 2);
                ++n_tris;
                float t, u, v;
                if (!isect_tri(r, xyz_of(q0), xyz_of(q1), xyz_of(q2), tmin, tbest, t, u, v)) continue;
                tbest = t;
                if (ANY) {
                    walking = false;
                    break;
                }
            }
            ig.y = 0u;
        }
        // the next node: mostly a child, in a bare BLAS else the stack's top (past
        // the loop below 1,677 -> 1,572 us)
        if (walking && !TOP && !group_left(g) && sp > 0) g = pop();
        if (walking && ig.y == 0u && group_left(g)) {
            node = take_child(g, r.prio);
            if (group_left(g)) {
                if (sp >= kInstDepth) fail(in_blas ? 0x70000000u : 0x71000000u);
                else push(g);
            }
            continue;
        }
        // else an instance of this node, a child, the stack
        while (walking) {
            if (TOP && ig.y) {
                const uint32_t rec = ig.x + (uint32_t)__ffs((int)ig.y) - 1u;
                ig.y &= ig.y - 1u;
                const InstRec ir = load_inst(tprims, rec);
                const uint8_t *blas = reinterpret_cast<const uint8_t *>(ir.accel_ref);
                const rt_accel_header *bh = reinterpret_cast<const rt_accel_header *>(blas);
                if (((ir.cim >> 24) & 0xffu) == 0u || !blas || bh->prim_count == 0u) continue;
                if (sp + 3 > kInstDepth) {
                    fail(0x71000000u);
                    break;
                }
                if (group_left(g)) push(g);
                if (ig.y) push(make_uint2(ig.x, ig.y | kInstGroup));
                push(make_uint2(visits, kReturn));
                float o[3], d[3], o2[3], d2[3];
                load_ray(o, d);
                xform_point(ir.w2o, o, o2);
                xform_vector(ir.w2o, d, d2);
                ray_setup(r, o2, d2);
                in_blas = true;
                nodes = reinterpret_cast<const uint4 *>(blas + bh->node_offset);
                prims = reinterpret_cast<const uint4 *>(blas + bh->prim_offset);
                count = bh->node_count;
                node = 0;
                visits = 0;
                break;
            }
            if (group_left(g)) {
                node = take_child(g, r.prio);
                if (group_left(g)) {
                    if (sp >= kInstDepth) fail(in_blas ? 0x70000000u : 0x71000000u);
                    else push(g);
                }
                break;
            }
            if (sp == 0) {
                walking = false;
                break;
            }
            const uint2 e = pop();
            if (TOP && (e.y & kReturn)) {
                if (sp == 0) {
                    walking = false;
                    break;
                }
                visits = e.x;
                float o[3], d[3];
                load_ray(o, d);
                ray_setup_box(r, o, d);
                in_blas = false;
                nodes = tnodes;
                count = t_count;
            } else if (TOP && (e.y & kInstGroup)) {
                ig = make_uint2(e.x, e.y & ~kInstGroup);
            } else {
                g = e;
            }
        }
    }
    for (int o = 16; o > 0; o >>= 1) {
        n_nodes += __shfl_xor_sync(kFull, n_nodes, o);
        n_tris += __shfl_xor_sync(kFull, n_tris, o);
    }
    if (lane == 0) {
        atomicAdd(counters, n_nodes);
        atomicAdd(counters + 1, n_tris);
    }
}

// ---------------------------------------------------------------------------
// Sample pipeline: raygen + trace + closest-hit/miss + imageStore
// ---------------------------------------------------------------------------

struct PipelineArgs {
    const uint8_t *accel;
    float cam[3];
    float ay, ax;   // aspect_y, aspect_x of the raygen (host-computed)
    uint32_t width, height;
    uint32_t chit, ray_flags, cull_mask, sbt_record_offset, sbt_record_stride;
    float tmin, tmax;
    float miss[3];
    const float *sbt;
    uint32_t sbt_count, sbt_stride;
    float4 *out;
    uint32_t *err;
};

// The sample's raygen (main.cpp:1036-1045), one IEEE operation at a time.
__device__ __forceinline__ void raygen(const PipelineArgs &a, uint32_t x, uint32_t y, float dir[3]) {
    const float sx = (float)x + 0.5f, sy = (float)y + 0.5f;
    const float ndx = (sx / (float)a.width) * 2.0f - 1.0f;
    const float ndy = (sy / (float)a.height) * 2.0f - 1.0f;
    const float p = ndx * a.ax, q = ndy * a.ay;
    dir[0] = (p * 1.0f + q * 0.0f) + 0.0f;
    dir[1] = (p * 0.0f + q * -1.0f) + 0.0f;
    dir[2] = (p * 0.0f + q * 0.0f) + -1.0f;
}

// Six blocks per SM (80 registers).  Two thirds of the issue slots are busy: 590
// instructions per warp with the triangle test's ray setup (divisions) done for
// every level and instance, before a triangle is met, and both kinds of walk in
// one kernel.  1200x800 pixels of the two-instance sample: 22.5 -> 20.5 us (5 or
// 7 blocks per SM the same, 4 22.5).
template <bool ANY>
__global__ void __launch_bounds__(128, 6) k_pipeline(const PipelineArgs a) {
    const uint32_t x = blockIdx.x * 16u + (threadIdx.x & 15u);
    const uint32_t y = blockIdx.y * 8u + (threadIdx.x >> 4);
    if (x >= a.width || y >= a.height) return;
    float dir[3];
    raygen(a, x, y, dir);
    Hit h;
    HitIds ids;
    float c[3];
    trace_ray<ANY>(a.accel, a.cam, dir, a.tmin, a.tmax, a.cull_mask & 0xffu, h, ids, a.err);
    if (!h.found) {
        c[0] = a.miss[0]; c[1] = a.miss[1]; c[2] = a.miss[2];
    } else if (a.ray_flags & RT_RAY_FLAG_SKIP_CLOSEST_HIT) {
        c[0] = c[1] = c[2] = 0.0f;
    } else {
        const uint32_t rec = ids.sbt_off + ids.geom * a.sbt_record_stride + a.sbt_record_offset;
        const bool bary = a.chit == RT_CHIT_BARYCENTRIC ||
                          (a.chit == RT_CHIT_SAMPLE && ids.prim == 1u && h.inst == 1u && ids.custom == 100u &&
                           ids.geom == 1u);
        if (bary) {
            c[0] = (1.0f - h.u) - h.v; c[1] = h.u; c[2] = h.v;
        } else if (rec < a.sbt_count) {
            c[0] = a.sbt[(size_t)rec * a.sbt_stride + 0];
            c[1] = a.sbt[(size_t)rec * a.sbt_stride + 1];
            c[2] = a.sbt[(size_t)rec * a.sbt_stride + 2];
        } else {
            c[0] = c[1] = c[2] = 0.0f;
            report_error(a.err, RT_ERR_BOUNDS, 0x73000000u | rec);
        }
    }
    a.out[(size_t)y * a.width + x] = make_float4(c[0], c[1], c[2], 0.0f);
}

// The raygen's rays alone.
__global__ void __launch_bounds__(128) k_primary_rays(const PipelineArgs a, rt_ray *rays) {
    const uint32_t x = blockIdx.x * 16u + (threadIdx.x & 15u);
    const uint32_t y = blockIdx.y * 8u + (threadIdx.x >> 4);
    if (x >= a.width || y >= a.height) return;
    rt_ray rr;
    raygen(a, x, y, rr.dir);
    rr.org[0] = a.cam[0]; rr.org[1] = a.cam[1]; rr.org[2] = a.cam[2];
    rr.tmin = a.tmin;
    rr.tmax = a.tmax;
    rays[(size_t)y * a.width + x] = rr;
}

// ---------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------

int launch_batch(rt_context *ctx, cudaStream_t st, uint64_t accel, const rt_ray *rays, rt_hit *hits,
                 rt_hit_ext *hits_ext, uint8_t *occ, uint32_t n, bool any) {
    if (n == 0) return RT_OK;
    BatchArgs a{};
    a.accel = reinterpret_cast<const uint8_t *>(accel);
    a.rays = reinterpret_cast<const float4 *>(rays);
    a.hits = reinterpret_cast<float4 *>(hits);
    a.hits_ext = hits_ext;
    a.occluded = occ;
    a.n = n;
    a.refill = ctx->tuning.batch_rays ? ctx->tuning.batch_rays : 4u;
    if (a.refill > 32u) a.refill = 32u;
    a.err = ctx->d_err;
    a.n_dev = nullptr;
    a.out_rec = 0;
    a.counter = acquire_counter(ctx, st);
    if (!a.counter) return set_error(ctx, RT_ERR_CUDA, "work counter reset failed");
    uint32_t per_sm = ctx->tuning.blocks_per_sm ? ctx->tuning.blocks_per_sm : 8u;
    if (any && per_sm > kAnyBlocksPerSm) per_sm = kAnyBlocksPerSm;
    uint32_t blocks = per_sm * (uint32_t)ctx->sm_count;
    uint32_t need = (n + kTraceThreads - 1) / kTraceThreads;
    if (blocks > need) blocks = need;
    // Both kernels are launched; the one that does not match the structure's
    // kind returns immediately.  The second is in place when the first ends (see
    // pdl_enter; 4,097 visibility rays: 26.2 -> 23.8 us).
    uint32_t tl_blocks = kInstBlocksPerSm * (uint32_t)ctx->sm_count;
    if (tl_blocks > need) tl_blocks = need;
    if (any) {
        k_trace_blas<true, false, kTraceThreads, kRing><<<blocks, kTraceThreads, 0, st>>>(a);
        RT_CUDA_CTX(ctx, launch_pdl(k_trace_inst<true>, tl_blocks, kTraceThreads, 0, st, a));
    } else {
        k_trace_blas<false, false, kTraceThreads, kRing><<<blocks, kTraceThreads, 0, st>>>(a);
        RT_CUDA_CTX(ctx, launch_pdl(k_trace_inst<false>, tl_blocks, kTraceThreads, 0, st, a));
    }
    RT_CUDA_CTX(ctx, cudaGetLastError());
    return RT_OK;
}

}  // namespace

// Refill threshold of the path tracer's queue traversals: a warp refills once
// eight of its lanes are idle (2M box, four samples: 21.07 / 20.97 / 21.20 /
// 21.47 ms at 6 / 8 / 10 / 12).  The batch's autotuner chose 8 as well.  The
// ray-query calls keep the context's batch_rays (default 4; 6 is 1 % faster on
// the soup's primary + incoherent rays).
constexpr uint32_t kQueueRefill = 8u;

// Queue-driven BLAS traversal for the wavefront path tracer: the ray count is
// read on the device from *n_dev (at most max_n), the work counter is
// `counter` (zeroed by the caller on the stream), and closest hits carry the
// leaf-record index.  Capturable in a CUDA graph (no host reads, no
// allocation).
int launch_queue_trace(rt_context *ctx, cudaStream_t st, const uint8_t *accel, const void *rays, void *hits,
                       const uint32_t *n_dev, uint32_t max_n, uint32_t *counter) {
    if (max_n == 0) return RT_OK;
    BatchArgs a{};
    a.accel = accel;
    a.rays = static_cast<const float4 *>(rays);
    a.hits = static_cast<float4 *>(hits);
    a.n = max_n;
    a.refill = kQueueRefill;
    a.err = ctx->d_err;
    a.n_dev = n_dev;
    a.out_rec = 1;
    a.counter = counter;
    uint32_t per_sm = ctx->tuning.blocks_per_sm ? ctx->tuning.blocks_per_sm : 8u;
    uint32_t blocks = per_sm * (uint32_t)ctx->sm_count;
    uint32_t need = (max_n + kTraceThreads - 1) / kTraceThreads;
    if (blocks > need) blocks = need;
    k_trace_blas<false, false, kTraceThreads, kRing><<<blocks, kTraceThreads, 0, st>>>(a);
    RT_CUDA_CTX(ctx, cudaGetLastError());
    return RT_OK;
}

// One launch over two queues of at most max_n rays each: closest hits for
// rays/n_dev (leaf-record index out, to hits), then any hits for
// rays2/n_dev2 (to occluded).  Capturable like launch_queue_trace.
int launch_queue_trace_mixed(rt_context *ctx, cudaStream_t st, const uint8_t *accel, const void *rays, void *hits,
                             const uint32_t *n_dev, const void *rays2, uint8_t *occluded, const uint32_t *n_dev2,
                             uint32_t max_n, uint32_t *counter) {
    if (max_n == 0) return RT_OK;
    BatchArgs a{};
    a.accel = accel;
    a.rays = static_cast<const float4 *>(rays);
    a.hits = static_cast<float4 *>(hits);
    a.occluded = occluded;
    a.n = max_n;
    a.n_dev = n_dev;
    a.rays2 = static_cast<const float4 *>(rays2);
    a.n_dev2 = n_dev2;
    a.n2 = max_n;
    a.refill = kQueueRefill;
    a.err = ctx->d_err;
    a.out_rec = 1;
    a.counter = counter;
    uint32_t per_sm = ctx->tuning.blocks_per_sm ? ctx->tuning.blocks_per_sm : 8u;
    if (per_sm > kAnyBlocksPerSm) per_sm = kAnyBlocksPerSm;
    uint32_t blocks = per_sm * (uint32_t)ctx->sm_count;
    const uint32_t need = (uint32_t)(((uint64_t)max_n * 2u + kTraceThreads - 1) / kTraceThreads);
    if (blocks > need) blocks = need;
    k_trace_blas<false, false, kTraceThreads, kRing, true><<<blocks, kTraceThreads, 0, st>>>(a);
    RT_CUDA_CTX(ctx, cudaGetLastError());
    return RT_OK;
}

}  // namespace rtc

using namespace rtc;

extern "C" rt_status rt_trace_closest(rt_context *ctx, rt_stream stream, uint64_t accel, const rt_ray *rays,
                                      rt_hit *hits, rt_hit_ext *hits_ext, uint32_t n) {
    if (!ctx || !accel || (n && (!rays || !hits))) return set_error(ctx, RT_ERR_INVALID_ARG, "rt_trace_closest: null argument");
    return launch_batch(ctx, static_cast<cudaStream_t>(stream), accel, rays, hits, hits_ext, nullptr, n, false);
}

extern "C" rt_status rt_trace_any(rt_context *ctx, rt_stream stream, uint64_t accel, const rt_ray *rays,
                                  uint8_t *occluded, uint32_t n) {
    if (!ctx || !accel || (n && (!rays || !occluded))) return set_error(ctx, RT_ERR_INVALID_ARG, "rt_trace_any: null argument");
    return launch_batch(ctx, static_cast<cudaStream_t>(stream), accel, rays, nullptr, nullptr, occluded, n, true);
}

// ---------------------------------------------------------------------------
// Rays and results staged through the scratch (pageable memory the device
// cannot reach, misaligned buffers, RT_HOST_TRANSFER_STAGED): a ring of four
// device slots; chunk k is
// copied in on the context's copy-in stream once its slot's previous results
// have left, traced on one of three trace streams (round robin), and copied
// out on the copy-out stream.  The copies of neighbouring chunks overlap the
// traversal, and so do consecutive traversals: a launch ends on its slowest
// ray (a grazing primary ray walks hundreds of nodes), and the next chunk's
// launch fills the SMs the finished warps leave.  The first chunk is small
// (2^18 rays) so the pipeline fills quickly; chunks then double up to what a
// slot holds.
// ---------------------------------------------------------------------------

namespace {

constexpr uint32_t kHostChunk = 1u << 20;  // rays per chunk

// The ring's geometry depends on the scratch size only (never on the call's
// ray count or result size), so slot s covers the same bytes in every call
// that passes the same scratch: its events then order all uses of it.
struct HostSlots {
    uint32_t chunk;  // rays per slot
    uint64_t out_offset, slot_bytes;
};

uint64_t slot_bytes_for(uint32_t chunk) { return align_up((uint64_t)chunk * 32u, 256) + align_up((uint64_t)chunk * 16u, 256); }

HostSlots host_slots(uint64_t scratch_bytes) {
    HostSlots h;
    h.slot_bytes = (scratch_bytes / (uint64_t)rt_context::kHostSlots) & ~255ull;
    uint64_t c = h.slot_bytes / 48u;
    if (c > kHostChunk) c = kHostChunk;
    while (c > 0 && slot_bytes_for((uint32_t)c) > h.slot_bytes) --c;
    h.chunk = (uint32_t)c;
    h.out_offset = align_up(c * 32u, 256);
    return h;
}

int host_setup(rt_context *ctx) {
    if (ctx->host_ready) return RT_OK;
    RT_CUDA_CTX(ctx, cudaStreamCreateWithFlags(&ctx->h2d, cudaStreamNonBlocking));
    RT_CUDA_CTX(ctx, cudaStreamCreateWithFlags(&ctx->d2h, cudaStreamNonBlocking));
    for (int k = 0; k < rt_context::kHostTraceStreams; ++k)
        RT_CUDA_CTX(ctx, cudaStreamCreateWithFlags(&ctx->htr[k], cudaStreamNonBlocking));
    RT_CUDA_CTX(ctx, cudaEventCreateWithFlags(&ctx->ev_start, cudaEventDisableTiming));
    for (int s = 0; s < rt_context::kHostSlots; ++s) {
        RT_CUDA_CTX(ctx, cudaEventCreateWithFlags(&ctx->ev_loaded[s], cudaEventDisableTiming));
        RT_CUDA_CTX(ctx, cudaEventCreateWithFlags(&ctx->ev_traced[s], cudaEventDisableTiming));
        RT_CUDA_CTX(ctx, cudaEventCreateWithFlags(&ctx->ev_free[s], cudaEventDisableTiming));
    }
    ctx->host_ready = true;
    return RT_OK;
}

// Whether every page of the host range [p, p + bytes) is mapped in this
// process.  msync with MS_ASYNC writes nothing back; it only fails with ENOMEM
// where part of the range is unmapped (a gap between two allocations, which a
// kernel reading the range in place would fault on).
bool host_range_mapped(const void *p, uint64_t bytes) {
    const long pg = sysconf(_SC_PAGESIZE);
    const uintptr_t page = pg > 0 ? (uintptr_t)pg : 4096u;
    const uintptr_t lo = reinterpret_cast<uintptr_t>(p) & ~(page - 1u);
    const uintptr_t hi = (reinterpret_cast<uintptr_t>(p) + bytes + page - 1u) & ~(page - 1u);
    return msync(reinterpret_cast<void *>(lo), hi - lo, MS_ASYNC) == 0;
}

// Whether [p, p + bytes) lies inside one CUDA allocation (device, managed or
// pinned host memory), from the driver's pointer attributes; false where the
// driver cannot say.
bool one_cuda_allocation(const void *p, uint64_t bytes) {
    static decltype(&cuPointerGetAttribute) get_attr = [] {
        void *f = nullptr;
        cudaDriverEntryPointQueryResult q = cudaDriverEntryPointSymbolNotFound;
        if (cudaGetDriverEntryPointByVersion("cuPointerGetAttribute", &f, 12000, cudaEnableDefault, &q) !=
                cudaSuccess ||
            q != cudaDriverEntryPointSuccess) {
            (void)cudaGetLastError();
            f = nullptr;
        }
        return reinterpret_cast<decltype(&cuPointerGetAttribute)>(f);
    }();
    if (!get_attr) return false;
    CUdeviceptr base = 0;
    size_t size = 0;
    const CUdeviceptr q = (CUdeviceptr)reinterpret_cast<uintptr_t>(p);
    if (get_attr(&base, CU_POINTER_ATTRIBUTE_RANGE_START_ADDR, q) != CUDA_SUCCESS ||
        get_attr(&size, CU_POINTER_ATTRIBUTE_RANGE_SIZE, q) != CUDA_SUCCESS)
        return false;
    return q >= base && q - base + bytes <= size;
}

// True when kernels reach [p, p + bytes) at the same address: pinned or
// registered host memory under unified addressing (cudaHostAlloc,
// cudaHostRegister), device or managed memory, and -- where the device
// accesses pageable memory through the host's page tables (a Grace system's
// NVLink-C2C; `pageable` from the device attributes) -- plain pageable
// memory.  Both ends are checked, and so is what lies between them: a host
// range must be mapped throughout (and, without pageable access, be one
// pinned allocation), a device range must be one allocation.  Anything else
// goes through the staged copies.
bool reachable_in_place(const void *p, uint64_t bytes, bool pageable) {
    if (bytes == 0) return true;
    const uint8_t *b = static_cast<const uint8_t *>(p);
    bool host_side = true, device_side = true;
    for (const uint8_t *q : {b, b + (bytes - 1u)}) {
        cudaPointerAttributes at;
        if (cudaPointerGetAttributes(&at, q) != cudaSuccess) {
            (void)cudaGetLastError();
            return false;
        }
        if (at.type == cudaMemoryTypeHost) {
            if (at.devicePointer != q) return false;
            device_side = false;
        } else if (at.type == cudaMemoryTypeUnregistered) {
            if (!pageable) return false;
            device_side = false;
        } else {
            host_side = false;
        }
    }
    if (host_side) {
        if (!host_range_mapped(p, bytes)) return false;
        return pageable || one_cuda_allocation(p, bytes);
    }
    return device_side && one_cuda_allocation(p, bytes);
}

// Whether the context's device reads and writes pageable host memory
// coherently through the host page tables (queried once).
bool pageable_in_place(rt_context *ctx) {
    if (ctx->pageable_state == 0) {
        int a = 0, b = 0;
        const bool ok = cudaDeviceGetAttribute(&a, cudaDevAttrPageableMemoryAccess, ctx->device) == cudaSuccess &&
                        cudaDeviceGetAttribute(&b, cudaDevAttrPageableMemoryAccessUsesHostPageTables, ctx->device) ==
                            cudaSuccess;
        (void)cudaGetLastError();
        ctx->pageable_state = (ok && a == 1 && b == 1) ? 1 : 2;
    }
    return ctx->pageable_state == 1;
}

int trace_host(rt_context *ctx, cudaStream_t st, uint64_t accel, const rt_ray *hrays, void *hout, uint32_t n,
               bool any, void *scratch, uint64_t scratch_bytes) {
    if (n == 0) return RT_OK;
    const uint32_t out_size = any ? 1u : 16u;
    // Rays and results the kernels reach in place (pinned memory; on a
    // Grace-Blackwell system also pageable memory, through the host page
    // tables): one launch reads the rays and writes the results where they
    // are, over NVLink-C2C.  A ray is read once (32 bytes) and a result
    // written once -- but for a ray set aside, whose result's place is written,
    // read and written again and which is read again, and half of a ray at each
    // instance it enters --, so no staging copy, chunk or ring is needed (4.15M
    // rays of the 1M soup: 1.77 ms pinned, against 2.23 ms staged from pinned
    // and 1.56 ms with rays and hits in HBM; 800K rays in 64 instances 1.13 to
    // 1.20 ms, staged 1.35, in HBM 1.03).
    RT_CUDA_CTX(ctx, cudaSetDevice(ctx->device));
    const bool pageable = pageable_in_place(ctx);
    if (ctx->host_transfer == RT_HOST_TRANSFER_AUTO && (reinterpret_cast<uintptr_t>(hrays) & 15u) == 0 &&
        (any || (reinterpret_cast<uintptr_t>(hout) & 15u) == 0) &&
        reachable_in_place(hrays, (uint64_t)n * 32u, pageable) &&
        reachable_in_place(hout, (uint64_t)n * out_size, pageable))
        return launch_batch(ctx, st, accel, hrays, any ? nullptr : static_cast<rt_hit *>(hout), nullptr,
                            any ? static_cast<uint8_t *>(hout) : nullptr, n, any);
    const HostSlots H = host_slots(scratch_bytes);
    if (H.chunk == 0) return set_error(ctx, RT_ERR_OOM, "rt_trace_*_host: scratch smaller than rt_trace_host_scratch_bytes(1)");
    if (reinterpret_cast<uintptr_t>(scratch) & 255u) return set_error(ctx, RT_ERR_INVALID_ARG, "rt_trace_*_host: scratch must be 256-byte aligned");
    int rc = host_setup(ctx);
    if (rc) return rc;
    if (scratch != ctx->host_scratch || scratch_bytes != ctx->host_scratch_bytes) {
        // another ring: copy in nothing before every earlier copy out is done
        for (int k = 0; k < rt_context::kHostSlots; ++k) RT_CUDA_CTX(ctx, cudaStreamWaitEvent(ctx->h2d, ctx->ev_free[k], 0));
        ctx->host_scratch = scratch;
        ctx->host_scratch_bytes = scratch_bytes;
    }
    uint8_t *S = static_cast<uint8_t *>(scratch);
    // everything of the call starts after the work queued on `stream` so far
    RT_CUDA_CTX(ctx, cudaEventRecord(ctx->ev_start, st));
    RT_CUDA_CTX(ctx, cudaStreamWaitEvent(ctx->h2d, ctx->ev_start, 0));
    for (int k = 0; k < rt_context::kHostTraceStreams; ++k)
        RT_CUDA_CTX(ctx, cudaStreamWaitEvent(ctx->htr[k], ctx->ev_start, 0));
    uint32_t chunk = kHostChunk / 4u < H.chunk ? kHostChunk / 4u : H.chunk;
    int s = 0, k = 0;
    for (uint32_t off = 0, m = 0; off < n; off += m, ++k) {
        m = n - off < chunk ? n - off : chunk;
        chunk = chunk * 2u < H.chunk ? chunk * 2u : H.chunk;
        s = (int)(ctx->slot_next++ % (uint32_t)rt_context::kHostSlots);
        cudaStream_t ts = ctx->htr[k % rt_context::kHostTraceStreams];
        uint8_t *rays_d = S + (uint64_t)s * H.slot_bytes;
        uint8_t *out_d = rays_d + H.out_offset;
        RT_CUDA_CTX(ctx, cudaStreamWaitEvent(ctx->h2d, ctx->ev_free[s], 0));
        // cudaMemcpyDefault: the direction follows from the pointers (unified
        // addressing), so a device or managed buffer handed to the host API
        // copies correctly too
        RT_CUDA_CTX(ctx, cudaMemcpyAsync(rays_d, hrays + off, (size_t)m * 32u, cudaMemcpyDefault, ctx->h2d));
        RT_CUDA_CTX(ctx, cudaEventRecord(ctx->ev_loaded[s], ctx->h2d));
        RT_CUDA_CTX(ctx, cudaStreamWaitEvent(ts, ctx->ev_loaded[s], 0));
        rc = launch_batch(ctx, ts, accel, reinterpret_cast<const rt_ray *>(rays_d),
                          any ? nullptr : reinterpret_cast<rt_hit *>(out_d), nullptr, any ? out_d : nullptr, m, any);
        if (rc) return rc;
        RT_CUDA_CTX(ctx, cudaEventRecord(ctx->ev_traced[s], ts));
        RT_CUDA_CTX(ctx, cudaStreamWaitEvent(ctx->d2h, ctx->ev_traced[s], 0));
        RT_CUDA_CTX(ctx, cudaMemcpyAsync(static_cast<uint8_t *>(hout) + (size_t)off * out_size, out_d,
                                         (size_t)m * out_size, cudaMemcpyDefault, ctx->d2h));
        RT_CUDA_CTX(ctx, cudaEventRecord(ctx->ev_free[s], ctx->d2h));
    }
    // the caller's stream goes on after the last results have left
    RT_CUDA_CTX(ctx, cudaStreamWaitEvent(st, ctx->ev_free[s], 0));
    return RT_OK;
}

}  // namespace

extern "C" rt_status rt_debug_host_in_place(rt_context *ctx, const void *p, uint64_t bytes, int *in_place) {
    if (!ctx || !in_place || (bytes && !p)) return RT_ERR_INVALID_ARG;
    RT_CUDA_CTX(ctx, cudaSetDevice(ctx->device));
    *in_place = reachable_in_place(p, bytes, pageable_in_place(ctx)) ? 1 : 0;
    return RT_OK;
}

extern "C" rt_status rt_set_host_transfer(rt_context *ctx, uint32_t mode) {
    if (!ctx) return RT_ERR_INVALID_ARG;
    if (mode != RT_HOST_TRANSFER_AUTO && mode != RT_HOST_TRANSFER_STAGED)
        return set_error(ctx, RT_ERR_INVALID_ARG, "rt_set_host_transfer: unknown mode");
    ctx->host_transfer = mode;
    return RT_OK;
}

extern "C" rt_status rt_trace_host_scratch_bytes(uint32_t n, int any_hit, uint64_t *bytes) {
    (void)any_hit;  // one ring serves both kinds of call
    if (!bytes) return RT_ERR_INVALID_ARG;
    const uint32_t c = n == 0 ? 1u : (n < kHostChunk ? n : kHostChunk);
    *bytes = slot_bytes_for(c) * (uint64_t)rt_context::kHostSlots;
    return RT_OK;
}

extern "C" rt_status rt_trace_closest_host(rt_context *ctx, rt_stream stream, uint64_t accel, const rt_ray *rays,
                                           rt_hit *hits, uint32_t n, void *scratch, uint64_t scratch_bytes) {
    if (!ctx || !accel || (n && (!rays || !hits || !scratch)))
        return set_error(ctx, RT_ERR_INVALID_ARG, "rt_trace_closest_host: null argument");
    return trace_host(ctx, static_cast<cudaStream_t>(stream), accel, rays, hits, n, false, scratch, scratch_bytes);
}

extern "C" rt_status rt_trace_any_host(rt_context *ctx, rt_stream stream, uint64_t accel, const rt_ray *rays,
                                       uint8_t *occluded, uint32_t n, void *scratch, uint64_t scratch_bytes) {
    if (!ctx || !accel || (n && (!rays || !occluded || !scratch)))
        return set_error(ctx, RT_ERR_INVALID_ARG, "rt_trace_any_host: null argument");
    return trace_host(ctx, static_cast<cudaStream_t>(stream), accel, rays, occluded, n, true, scratch, scratch_bytes);
}

extern "C" rt_status rt_trace_stats(rt_context *ctx, rt_stream stream, uint64_t accel, const rt_ray *rays,
                                    uint32_t n, int any_hit, unsigned long long *counters) {
    if (!ctx || !accel || !counters || (n && !rays)) return set_error(ctx, RT_ERR_INVALID_ARG, "rt_trace_stats: null argument");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    RT_CUDA_CTX(ctx, cudaMemsetAsync(counters, 0, 16, st));
    if (n == 0) return RT_OK;
    uint32_t *counter = acquire_counter(ctx, st);
    if (!counter) return set_error(ctx, RT_ERR_CUDA, "work counter reset failed");
    const uint32_t refill = ctx->tuning.batch_rays ? (ctx->tuning.batch_rays < 32u ? ctx->tuning.batch_rays : 32u) : 4u;
    const uint32_t need = (n + kTraceThreads - 1) / kTraceThreads, sms = (uint32_t)ctx->sm_count;
    const uint8_t *A = reinterpret_cast<const uint8_t *>(accel);
    const float4 *R = reinterpret_cast<const float4 *>(rays);
    // one of the two returns at once, as in launch_batch
    for (const bool top : {false, true}) {
        const auto kernel = top ? (any_hit ? k_trace_stats<true, true> : k_trace_stats<false, true>)
                                : (any_hit ? k_trace_stats<true, false> : k_trace_stats<false, false>);
        const uint32_t most = stats_blocks_per_sm(top) * sms;
        kernel<<<need < most ? need : most, kTraceThreads, 0, st>>>(A, R, n, refill, counter, counters, ctx->d_err);
    }
    RT_CUDA_CTX(ctx, cudaGetLastError());
    return RT_OK;
}

extern "C" rt_status rt_trace_rays(rt_context *ctx, rt_stream stream, const rt_pipeline *p, const rt_sbt *sbt,
                                   uint64_t accel, const rt_camera *camera, float *out, uint32_t width,
                                   uint32_t height, uint32_t depth) {
    if (!ctx || !p || !accel || !camera || !out) return set_error(ctx, RT_ERR_INVALID_ARG, "rt_trace_rays: null argument");
    if (depth != 1u) return set_error(ctx, RT_ERR_UNSUPPORTED, "rt_trace_rays: depth must be 1 (2D storage image)");
    if (width == 0 || height == 0) return RT_OK;
    if (p->chit > RT_CHIT_SBT_COLOR) return set_error(ctx, RT_ERR_INVALID_ARG, "rt_trace_rays: unknown closest-hit program");
    if (p->max_recursion > 1u) return set_error(ctx, RT_ERR_UNSUPPORTED, "rt_trace_rays: recursion depth > 1");
    if (p->sbt_record_stride == 0u && p->chit != RT_CHIT_BARYCENTRIC)
        ; /* stride 0 is legal in Vulkan: every geometry uses the same record */
    PipelineArgs a;
    a.accel = reinterpret_cast<const uint8_t *>(accel);
    a.cam[0] = camera->position[0]; a.cam[1] = camera->position[1]; a.cam[2] = camera->position[2];
    camera_aspects(camera, width, height, &a.ay, &a.ax);
    a.width = width;
    a.height = height;
    a.chit = p->chit;
    a.ray_flags = p->ray_flags;
    a.cull_mask = p->cull_mask;
    a.sbt_record_offset = p->sbt_record_offset;
    a.sbt_record_stride = p->sbt_record_stride;
    a.tmin = p->tmin;
    a.tmax = p->tmax;
    a.miss[0] = p->miss_color[0]; a.miss[1] = p->miss_color[1]; a.miss[2] = p->miss_color[2];
    a.sbt = sbt ? sbt->hit_colors : nullptr;
    a.sbt_count = sbt && sbt->hit_colors ? sbt->hit_record_count : 0u;
    a.sbt_stride = sbt ? (sbt->hit_record_stride < 3u ? 3u : sbt->hit_record_stride) : 3u;
    a.out = reinterpret_cast<float4 *>(out);
    a.err = ctx->d_err;
    dim3 grid((width + 15u) / 16u, (height + 7u) / 8u);
    const auto kernel = (p->ray_flags & RT_RAY_FLAG_TERMINATE_ON_FIRST_HIT) ? k_pipeline<true> : k_pipeline<false>;
    kernel<<<grid, 128, 0, static_cast<cudaStream_t>(stream)>>>(a);
    RT_CUDA_CTX(ctx, cudaGetLastError());
    return RT_OK;
}

extern "C" rt_status rt_generate_primary_rays(rt_context *ctx, rt_stream stream, const rt_camera *camera,
                                              uint32_t width, uint32_t height, float tmin, float tmax,
                                              rt_ray *rays) {
    if (!ctx || !camera || !rays) return set_error(ctx, RT_ERR_INVALID_ARG, "rt_generate_primary_rays: null argument");
    if (width == 0 || height == 0) return RT_OK;
    PipelineArgs a{};
    a.cam[0] = camera->position[0]; a.cam[1] = camera->position[1]; a.cam[2] = camera->position[2];
    camera_aspects(camera, width, height, &a.ay, &a.ax);
    a.width = width;
    a.height = height;
    a.tmin = tmin;
    a.tmax = tmax;
    a.err = ctx->d_err;
    dim3 grid((width + 15u) / 16u, (height + 7u) / 8u);
    k_primary_rays<<<grid, 128, 0, static_cast<cudaStream_t>(stream)>>>(a, rays);
    RT_CUDA_CTX(ctx, cudaGetLastError());
    return RT_OK;
}
