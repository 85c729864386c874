// rt_device.cuh -- device-side arithmetic shared by the build and trace
// kernels of the GB300 ray-tracing core.
//
// Every kernel translation unit is compiled with -fmad=false: a float
// expression is evaluated one IEEE round-to-nearest operation at a time, and
// an FMA is issued only where __fmaf_rn is written.  That is what makes the
// build bit-exact, and the hits bit-identical, against the CPU restatement of
// the same steps.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include "../../include/rtcore.h"
#include "../../include/rtcore_accel.h"

namespace rtc {

constexpr uint32_t kLeafBit = 0x80000000u;
constexpr float kTfarScale = 1.0f + 0x1p-20f;
constexpr float kInf = __builtin_huge_valf();

// ---------------------------------------------------------------------------
// Float helpers
// ---------------------------------------------------------------------------

// Total order on float bits (-0 < +0): min/max under it give the same bits
// whatever the order of a parallel reduction.
__device__ __forceinline__ int32_t ford(float f) {
    int32_t i = __float_as_int(f);
    return i >= 0 ? i : (i ^ 0x7fffffff);
}
__device__ __forceinline__ float ford_inv(int32_t i) {
    return __int_as_float(i >= 0 ? i : (i ^ 0x7fffffff));
}
__device__ __forceinline__ float fmn(float a, float b) { return ford(b) < ford(a) ? b : a; }
__device__ __forceinline__ float fmx(float a, float b) { return ford(b) > ford(a) ? b : a; }
__device__ __forceinline__ float pow2f(int e) { return __int_as_float((e + 127) << 23); }

struct Box {
    float lo[3], hi[3];
};

__device__ __forceinline__ Box box_empty() {
    Box b;
#pragma unroll
    for (int a = 0; a < 3; ++a) { b.lo[a] = kInf; b.hi[a] = -kInf; }
    return b;
}
__device__ __forceinline__ bool box_is_empty(const Box &b) {
    return !(b.lo[0] <= b.hi[0] && b.lo[1] <= b.hi[1] && b.lo[2] <= b.hi[2]);
}
__device__ __forceinline__ Box box_union(const Box &x, const Box &y) {
    Box b;
#pragma unroll
    for (int a = 0; a < 3; ++a) { b.lo[a] = fmn(x.lo[a], y.lo[a]); b.hi[a] = fmx(x.hi[a], y.hi[a]); }
    return b;
}
__device__ __forceinline__ float half_area(const Box &b) {
    if (box_is_empty(b)) return 0.0f;
    float dx = b.hi[0] - b.lo[0], dy = b.hi[1] - b.lo[1], dz = b.hi[2] - b.lo[2];
    return (dx * dy + dy * dz) + dz * dx;
}

// Smallest e with 255 * 2^e >= ext, clamped to [RT_QEXP_MIN, RT_QEXP_MAX].
__device__ __forceinline__ int qexp_for(float ext) {
    if (!(ext > 0.0f)) return RT_QEXP_MIN;
    int biased = (int)((__float_as_uint(ext) >> 23) & 0xffu);
    int e = (biased == 0 ? -127 : biased - 127) - 8;
    if (e < RT_QEXP_MIN) e = RT_QEXP_MIN;
    while (e < RT_QEXP_MAX && 255.0f * pow2f(e) < ext) ++e;
    return e;
}

__device__ __forceinline__ void xform_point(const float m[12], const float p[3], float out[3]) {
#pragma unroll
    for (int r = 0; r < 3; ++r)
        out[r] = ((m[4 * r + 0] * p[0] + m[4 * r + 1] * p[1]) + m[4 * r + 2] * p[2]) + m[4 * r + 3];
}
__device__ __forceinline__ void xform_vector(const float m[12], const float p[3], float out[3]) {
#pragma unroll
    for (int r = 0; r < 3; ++r) out[r] = (m[4 * r + 0] * p[0] + m[4 * r + 1] * p[1]) + m[4 * r + 2] * p[2];
}

// ---------------------------------------------------------------------------
// Ray setup and the watertight triangle test
// (Woop, Benthin, Wald, JCGT 2013)
// ---------------------------------------------------------------------------

struct Ray {
    float o[3];
    float d[3];
    float invd[3];
    float sx, sy, sz;
    uint32_t prio;  // visiting order of a node's slots, see child_priority
    uint32_t kxyz;  // kx | ky << 2 | kz << 4
};

// Children are visited in ascending (slot ^ octant), bit a of the octant set
// where invd[a] < 0.  Byte a of the word holds the slots whose bit a equals the
// octant's, i.e. those that come first as far as axis a decides, so the next of
// a set of slots is found by narrowing it with the z byte, then y, then x.
__device__ __forceinline__ uint32_t child_priority(uint32_t oct) {
    return (0x55u << (oct & 1u)) | (0x3300u << (oct & 2u)) | (0x0f0000u << (oct & 4u));
}
// The octant's bits back from the word.
__device__ __forceinline__ bool prio_neg_x(uint32_t prio) { return (prio & 1u) == 0u; }
__device__ __forceinline__ bool prio_neg_y(uint32_t prio) { return (prio & 0x100u) == 0u; }
__device__ __forceinline__ bool prio_neg_z(uint32_t prio) { return (prio & 0x10000u) == 0u; }

// The first slot of the non-empty set `slots` (bits 0-7) in visiting order, as
// a one-bit mask.
__device__ __forceinline__ uint32_t first_slot(uint32_t slots, uint32_t prio) {
    uint32_t t = slots & (prio >> 16);
    slots = t ? t : slots;
    t = slots & (prio >> 8);
    slots = t ? t : slots;
    t = slots & prio;
    return t ? t : slots;
}

__device__ __forceinline__ float sel3(uint32_t k, float x, float y, float z) {
    return k == 0 ? x : (k == 1 ? y : z);
}

// The box test's part of a ray: all a walk needs until it meets a triangle.
__device__ __forceinline__ void ray_setup_box(Ray &r, const float o[3], const float d[3]) {
    uint32_t oct = 0;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        r.o[a] = o[a];
        r.d[a] = d[a];
        float dd = fabsf(d[a]) < RT_DIR_EPS ? copysignf(RT_DIR_EPS, d[a]) : d[a];
        r.invd[a] = 1.0f / dd;
        oct |= (r.invd[a] < 0.0f ? 1u : 0u) << a;
    }
    r.prio = child_priority(oct);
}

// The triangle test's part, of a ray set up for the box test.
__device__ __forceinline__ void ray_setup_shear(Ray &r) {
    const float *d = r.d;
    float ax = fabsf(d[0]), ay = fabsf(d[1]), az = fabsf(d[2]);
    uint32_t kz = ax >= ay ? (ax >= az ? 0u : 2u) : (ay >= az ? 1u : 2u);
    uint32_t kx = kz == 2u ? 0u : kz + 1u;
    uint32_t ky = kx == 2u ? 0u : kx + 1u;
    float dkz = sel3(kz, d[0], d[1], d[2]);
    if (dkz < 0.0f) { uint32_t t = kx; kx = ky; ky = t; }
    r.kxyz = kx | (ky << 2) | (kz << 4);
    r.sx = sel3(kx, d[0], d[1], d[2]) / dkz;
    r.sy = sel3(ky, d[0], d[1], d[2]) / dkz;
    // the largest component's reciprocal, computed above unless the whole
    // direction is below RT_DIR_EPS
    r.sz = fabsf(dkz) < RT_DIR_EPS ? 1.0f / dkz : sel3(kz, r.invd[0], r.invd[1], r.invd[2]);
}

__device__ __forceinline__ void ray_setup(Ray &r, const float o[3], const float d[3]) {
    ray_setup_box(r, o, d);
    ray_setup_shear(r);
}

// Returns true and (t, u, v) when the triangle is hit with t in [tmin, tmax].
__device__ __forceinline__ bool isect_tri(const Ray &r, float4 v0, float4 v1, float4 v2, float tmin, float tmax,
                                          float &t_out, float &u_out, float &v_out) {
    const uint32_t kx = r.kxyz & 3u, ky = (r.kxyz >> 2) & 3u, kz = (r.kxyz >> 4) & 3u;
    float A0 = v0.x - r.o[0], A1 = v0.y - r.o[1], A2 = v0.z - r.o[2];
    float B0 = v1.x - r.o[0], B1 = v1.y - r.o[1], B2 = v1.z - r.o[2];
    float C0 = v2.x - r.o[0], C1 = v2.y - r.o[1], C2 = v2.z - r.o[2];
    float Akz = sel3(kz, A0, A1, A2), Bkz = sel3(kz, B0, B1, B2), Ckz = sel3(kz, C0, C1, C2);
    float ax = sel3(kx, A0, A1, A2) - r.sx * Akz, ay = sel3(ky, A0, A1, A2) - r.sy * Akz;
    float bx = sel3(kx, B0, B1, B2) - r.sx * Bkz, by = sel3(ky, B0, B1, B2) - r.sy * Bkz;
    float cx = sel3(kx, C0, C1, C2) - r.sx * Ckz, cy = sel3(ky, C0, C1, C2) - r.sy * Ckz;
    float U = cx * by - cy * bx;
    float V = ax * cy - ay * cx;
    float W = bx * ay - by * ax;
    if (U == 0.0f || V == 0.0f || W == 0.0f) {
        U = (float)((double)cx * (double)by - (double)cy * (double)bx);
        V = (float)((double)ax * (double)cy - (double)ay * (double)cx);
        W = (float)((double)bx * (double)ay - (double)by * (double)ax);
    }
    if ((U < 0.0f || V < 0.0f || W < 0.0f) && (U > 0.0f || V > 0.0f || W > 0.0f)) return false;
    float det = (U + V) + W;
    if (det == 0.0f) return false;
    float T = (U * (r.sz * Akz) + V * (r.sz * Bkz)) + W * (r.sz * Ckz);
    float rcp = 1.0f / det;
    float t = T * rcp;
    if (!(t >= tmin && t <= tmax)) return false;
    t_out = t;
    u_out = V * rcp;
    v_out = W * rcp;
    return true;
}

// ---------------------------------------------------------------------------
// Wide node test
// ---------------------------------------------------------------------------

struct NodeWords {
    uint4 w0, w1, w2, w3, w4;
};

__device__ __forceinline__ NodeWords load_node(const uint4 *nodes, uint32_t idx) {
    const uint4 *p = nodes + (size_t)idx * 5u;
    NodeWords n;
    n.w0 = __ldg(p + 0);
    n.w1 = __ldg(p + 1);
    n.w2 = __ldg(p + 2);
    n.w3 = __ldg(p + 3);
    n.w4 = __ldg(p + 4);
    return n;
}

// Three-input min/max (sm_100+ PTX); exact, so equal to two-input chains.
__device__ __forceinline__ float fmin3(float a, float b, float c) {
    float d;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}
__device__ __forceinline__ float fmax3(float a, float b, float c) {
    float d;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}

// Two-wide FP32 arithmetic (PTX .f32x2, sm_100 and later): one instruction
// for two lanes' worth of add or fma, each half rounded exactly as the scalar
// instruction, so the pair equals two scalar results bit for bit.
__device__ __forceinline__ uint64_t f2_pack(float lo, float hi) {
    uint64_t d;
    asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(lo), "f"(hi));
    return d;
}
__device__ __forceinline__ void f2_unpack(uint64_t v, float &lo, float &hi) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ uint64_t f2_add(uint64_t a, uint64_t b) {
    uint64_t d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ uint64_t f2_fma(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
// Bytes b and b + 1 of w as the pair (2^23 + q, 2^23 + q'); adding
// (-2^23, -2^23) leaves the exact byte values.
__device__ __forceinline__ uint64_t qpair_biased(uint32_t w, int b) {
    const uint32_t lo = __byte_perm(w, 0x4B000000u, 0x7540u | (uint32_t)b);
    const uint32_t hi = __byte_perm(w, 0x4B000000u, 0x7541u + (uint32_t)b);
    uint64_t d;
    asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "r"(lo), "r"(hi));
    return d;
}

// Box test of a node's 8 children against [tmin, tcur]: bit s set where the
// box of slot s is hit (an unused slot may show a hit: its meta byte is 0 and
// it is not an internal child, so it leads nowhere).
//
// The kernels that call it are bound by issue slots, so it is laid out for
// instruction count: two neighbouring children share every .f32x2 add and fma
// (plane distance fma(q, scale, adj), each half rounded as the scalar
// instruction).  Their bytes come out of one word, so the pairs form in place;
// pairing the x and y planes of one child instead cost a register move for
// nearly every pair.  A child is missed when tfar * scale - tnear is negative,
// and the eight sign bits are shifted into one mask: the scale goes on by an
// fma with +0, which leaves no -0 whose difference to +0 would carry a sign,
// and an inf - inf carries none either (a hit, as inf <= inf is).  Neither does
// a NaN, which only a NaN limit brings here (min and max pass over a NaN plane):
// callers do not walk with one, as no triangle is hit within it.  Measured on one node per lane: 175 instructions,
// 301 with the planes of one child paired and a mask bit or-ed in per child.
__device__ __forceinline__ uint32_t isect_node(const Ray &r, const NodeWords &n, float tmin, float tcur) {
    const float px = __uint_as_float(n.w0.x), py = __uint_as_float(n.w0.y), pz = __uint_as_float(n.w0.z);
    const int ex = (int)(int8_t)(n.w0.w & 0xffu);
    const int ey = (int)(int8_t)((n.w0.w >> 8) & 0xffu);
    const int ez = (int)(int8_t)((n.w0.w >> 16) & 0xffu);
    const float scx = pow2f(ex) * r.invd[0], scy = pow2f(ey) * r.invd[1], scz = pow2f(ez) * r.invd[2];
    const float adjx = (px - r.o[0]) * r.invd[0];
    const float adjy = (py - r.o[1]) * r.invd[1];
    const float adjz = (pz - r.o[2]) * r.invd[2];
    // qlo/qhi words for slots 0-3 (lo) and 4-7 (hi), per axis
    const uint32_t lox[2] = {n.w2.x, n.w2.y}, loy[2] = {n.w2.z, n.w2.w}, loz[2] = {n.w3.x, n.w3.y};
    const uint32_t hix[2] = {n.w3.z, n.w3.w}, hiy[2] = {n.w4.x, n.w4.y}, hiz[2] = {n.w4.z, n.w4.w};
    const bool nx = prio_neg_x(r.prio), ny = prio_neg_y(r.prio), nz = prio_neg_z(r.prio);
    const uint64_t bias = f2_pack(-8388608.0f, -8388608.0f), far_scale = f2_pack(kTfarScale, kTfarScale);
    const uint64_t zero = f2_pack(0.0f, 0.0f);
    const uint64_t sx = f2_pack(scx, scx), sy = f2_pack(scy, scy), sz = f2_pack(scz, scz);
    const uint64_t ax = f2_pack(adjx, adjx), ay = f2_pack(adjy, adjy), az = f2_pack(adjz, adjz);
    uint32_t miss = 0u;
#pragma unroll
    for (int h = 1; h >= 0; --h) {
        const uint32_t nearx = nx ? hix[h] : lox[h], farx = nx ? lox[h] : hix[h];
        const uint32_t neary = ny ? hiy[h] : loy[h], fary = ny ? loy[h] : hiy[h];
        const uint32_t nearz = nz ? hiz[h] : loz[h], farz = nz ? loz[h] : hiz[h];
#pragma unroll
        for (int b = 2; b >= 0; b -= 2) {
            float nx0, nx1, ny0, ny1, nz0, nz1, fx0, fx1, fy0, fy1, fz0, fz1, d0, d1;
            f2_unpack(f2_fma(f2_add(qpair_biased(nearx, b), bias), sx, ax), nx0, nx1);
            f2_unpack(f2_fma(f2_add(qpair_biased(neary, b), bias), sy, ay), ny0, ny1);
            f2_unpack(f2_fma(f2_add(qpair_biased(nearz, b), bias), sz, az), nz0, nz1);
            f2_unpack(f2_fma(f2_add(qpair_biased(farx, b), bias), sx, ax), fx0, fx1);
            f2_unpack(f2_fma(f2_add(qpair_biased(fary, b), bias), sy, ay), fy0, fy1);
            f2_unpack(f2_fma(f2_add(qpair_biased(farz, b), bias), sz, az), fz0, fz1);
            const float tn0 = fmaxf(fmax3(tmin, nx0, ny0), nz0), tn1 = fmaxf(fmax3(tmin, nx1, ny1), nz1);
            const float tf0 = fminf(fmin3(tcur, fx0, fy0), fz0), tf1 = fminf(fmin3(tcur, fx1, fy1), fz1);
            f2_unpack(f2_add(f2_fma(f2_pack(tf0, tf1), far_scale, zero), f2_pack(-tn0, -tn1)), d0, d1);
            miss = __funnelshift_l(__float_as_uint(d1), miss, 1);
            miss = __funnelshift_l(__float_as_uint(d0), miss, 1);
        }
    }
    return ~miss & 0xffu;
}

// Leaf records of the hit slots, as a mask relative to the node's prim_base (a
// leaf's meta byte: its record count in unary, then its first record's offset).
__device__ __forceinline__ uint32_t leaf_records(const NodeWords &n, uint32_t hits) {
    uint32_t leaf = hits & ~(n.w0.w >> 24), recs = 0u;
    while (leaf) {
        const uint32_t m = __byte_perm(n.w1.z, n.w1.w, (uint32_t)__ffs((int)leaf) - 1u) & 0xffu;
        leaf &= leaf - 1u;
        recs |= (m >> 5) << (m & 31u);
    }
    return recs;
}

// The hit internal children of a node as a traversal group: first child's
// index, hit slots (bits 0-7) and all internal slots (bits 8-15).
__device__ __forceinline__ uint2 child_group(const NodeWords &n, uint32_t hits) {
    const uint32_t inner = n.w0.w >> 24;
    return make_uint2(n.w1.x, (hits & inner) | (inner << 8));
}
__device__ __forceinline__ bool group_left(const uint2 &g) { return (g.y & 0xffu) != 0u; }
// Takes the next child of a group with children left; returns its node.
__device__ __forceinline__ uint32_t take_child(uint2 &g, uint32_t prio) {
    const uint32_t bit = first_slot(g.y & 0xffu, prio);
    g.y ^= bit;
    return g.x + __popc((g.y >> 8) & (bit - 1u));
}

// Programmatic dependent launch between kernels of a chain: each lets the next
// one launch as soon as all of its own blocks run, then waits for the kernel
// before it to complete (its writes visible) before it reads or writes anything
// that kernel does, so a launch's scheduling overlaps the previous kernel's
// tail.  Every thread waits, so a kernel completes after all before it.  What
// the kernel before writes is not read through the read-only path.  Launched
// without the attribute both instructions do nothing.
__device__ __forceinline__ void pdl_launch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_enter() {
    pdl_launch();
    pdl_wait();
}

// Device-side error reporting: the first error code wins.
__device__ __forceinline__ void report_error(uint32_t *err, int code, uint32_t detail) {
    if (err) {
        if (atomicCAS(err, 0u, (uint32_t)(-code)) == 0u) err[1] = detail;
    }
}

}  // namespace rtc
