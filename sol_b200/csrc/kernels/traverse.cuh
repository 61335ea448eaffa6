// BVH2 traversal on the device: the GPU statement of
// TriangleMesh::intersect_closest / intersect_any (src/triangle_mesh.cpp:64-117),
// which SoL runs through bvh v2's SingleRayTraverser.
//
// The traversal is the stack-based "while-while" loop of Aila & Laine
// ("Understanding the Efficiency of Ray Traversal on GPUs", HPG 2009): descend
// inner nodes, pushing the child that waits, until a leaf is reached; then test
// the leaf's triangles (48 bytes, three 128-bit loads) with the shared watertight
// test, so a hit found here is bit-identical to the one the host finds.
//
// Two forms of the box test walk the same hierarchy:
//   exact  (DNode, lower and upper bounds): the host traversal's operations, so
//          children are visited in the host's order and the first of several hits
//          is the host's.  Ray queries for any hit, which return that hit, and the
//          counting kernels use it.
//   packed (DBoxNode, centre and half size): fewer operations, conservative too,
//          in an order that may differ from the host's where two boxes begin at
//          (nearly) equal distances.  The closest hit is the same unless several
//          triangles are hit at exactly the closest distance; a ray that meets
//          that case is traced again in the exact form (closest_exact), and so is
//          one whose direction the packed test does not take (boxes_take).  A
//          shadow ray only asks whether anything is hit, which no order changes.
#pragma once

#include "../core/layout.h"
#include "../core/math.h"

namespace sol_b200 {

struct TraversalCounters {
    uint32_t nodes;
    uint32_t tris;
};

__device__ __forceinline__ float4 ldg4(const void* p) { return __ldg(reinterpret_cast<const float4*>(p)); }

/// Traversal stack in local memory.
struct LocalStack {
    int v[kTraversalStack];
    __device__ __forceinline__ void put(int i, int x) { v[i] = x; }
    __device__ __forceinline__ int get(int i) const { return v[i]; }
};

#ifndef SOL_SHARED_STACK_DEPTH
#define SOL_SHARED_STACK_DEPTH 16
#endif
/// Entries of the traversal stack kept in shared memory by SharedStack.
constexpr int kSharedStackDepth = SOL_SHARED_STACK_DEPTH;

/// Traversal stack whose first kSharedStackDepth entries live in shared memory,
/// laid out entry-major ([entry][thread] for kThreads threads, so a warp's
/// accesses at any mix of depths fall in distinct banks); deeper entries, which
/// few rays reach, go to local memory.  `column` is the thread's first entry:
/// shared_array + threadIdx.x.
template <int kThreads>
struct SharedStack {
    int* column;
    int deep[kTraversalStack - kSharedStackDepth];
    __device__ __forceinline__ void put(int i, int x) {
        if (i < kSharedStackDepth) column[i * kThreads] = x;
        else deep[i - kSharedStackDepth] = x;
    }
    __device__ __forceinline__ int get(int i) const {
        return i < kSharedStackDepth ? column[i * kThreads] : deep[i - kSharedStackDepth];
    }
};

/// SharedStack with the thread stride given at run time (the block size), for
/// kernels launched with several block sizes: `column` = a dynamic shared
/// array of kSharedStackDepth * blockDim.x ints + threadIdx.x.
struct SharedStackDyn {
    int* column;
    int stride;
    int deep[kTraversalStack - kSharedStackDepth];
    __device__ __forceinline__ void put(int i, int x) {
        if (i < kSharedStackDepth) column[i * stride] = x;
        else deep[i - kSharedStackDepth] = x;
    }
    __device__ __forceinline__ int get(int i) const {
        return i < kSharedStackDepth ? column[i * stride] : deep[i - kSharedStackDepth];
    }
};

__device__ __forceinline__ Vec3 tri_vertex(float4 a) { return vec3(a.x, a.y, a.z); }

__device__ __forceinline__ float fminf3(float a, float b, float c) { return fminf(fminf(a, b), c); }
__device__ __forceinline__ float fmaxf3(float a, float b, float c) { return fmaxf(fmaxf(a, b), c); }

/// (lo - o) * id and (hi - o) * id, both planes of a slab in one packed subtract
/// and one packed multiply (sm_100's two-wide FP32 forms, each half rounded as
/// the scalar operation, so the same bits in half the issue slots).  A packed
/// multiply must not feed a packed add here: ptxas contracts that pair into a
/// fused multiply-add whatever -fmad says.
__device__ __forceinline__ void slab_planes(float lo, float hi, float o, float id, float& t_lo, float& t_hi) {
    asm("{\n\t.reg .b64 p, q, r;\n\t"
        "mov.b64 p, {%2, %3};\n\tmov.b64 q, {%4, %4};\n\tmov.b64 r, {%5, %5};\n\t"
        "sub.rn.f32x2 p, p, q;\n\tmul.rn.f32x2 p, p, r;\n\tmov.b64 {%0, %1}, p;\n\t}"
        : "=f"(t_lo), "=f"(t_hi) : "f"(lo), "f"(hi), "f"(o), "f"(id));
}

/// Entry and (widened) exit distances of a ray against both child boxes of a
/// node: a = c0.x and c0.y bounds, b = c1.x and c1.y bounds, c = both z bounds.
/// (bound - org) * (1/dir) takes two correctly rounded operations per plane, so
/// the widened exit distance stays conservative even for grazing rays (the
/// product-with-offset form loses |org / dir| ulps to cancellation).  The
/// traversal kernels are bound by instruction issue at about 9 of 32 lanes per
/// node step, and the 24 scalar subtracts and multiplies were the largest
/// share of a step; packed they are 12 (1M-triangle frame, 64 samples: 50.4 ->
/// 46.6 ms together with the fused index check of Traversal::run).
__device__ __forceinline__ void child_slabs(float4 a, float4 b, float4 c, Vec3 org, Vec3 idir, float tmin,
                                            float tmax, float& n0, float& f0, float& n1, float& f1) {
    float t0lx, t0hx, t0ly, t0hy, t0lz, t0hz, t1lx, t1hx, t1ly, t1hy, t1lz, t1hz;
    slab_planes(a.x, a.y, org.x, idir.x, t0lx, t0hx);
    slab_planes(a.z, a.w, org.y, idir.y, t0ly, t0hy);
    slab_planes(c.x, c.y, org.z, idir.z, t0lz, t0hz);
    slab_planes(b.x, b.y, org.x, idir.x, t1lx, t1hx);
    slab_planes(b.z, b.w, org.y, idir.y, t1ly, t1hy);
    slab_planes(c.z, c.w, org.z, idir.z, t1lz, t1hz);
    n0 = fmaxf3(fminf(t0lx, t0hx), fminf(t0ly, t0hy), fmaxf(fminf(t0lz, t0hz), tmin));
    f0 = fminf3(fmaxf(t0lx, t0hx), fmaxf(t0ly, t0hy), fminf(fmaxf(t0lz, t0hz), tmax)) * kSlabWiden;
    n1 = fmaxf3(fminf(t1lx, t1hx), fminf(t1ly, t1hy), fmaxf(fminf(t1lz, t1hz), tmin));
    f1 = fminf3(fmaxf(t1lx, t1hx), fmaxf(t1ly, t1hy), fminf(fmaxf(t1lz, t1hz), tmax)) * kSlabWiden;
}

/// Two floats as one packed register pair operand.
struct F2 { float a, b; };
__device__ __forceinline__ F2 sub2(F2 x, float y) {
    F2 r;
    asm("{\n\t.reg .b64 p, q;\n\tmov.b64 p, {%2, %3};\n\tmov.b64 q, {%4, %4};\n\tsub.rn.f32x2 p, p, q;\n\t"
        "mov.b64 {%0, %1}, p;\n\t}" : "=f"(r.a), "=f"(r.b) : "f"(x.a), "f"(x.b), "f"(y));
    return r;
}
__device__ __forceinline__ F2 mul2(F2 x, float y) {
    F2 r;
    asm("{\n\t.reg .b64 p, q;\n\tmov.b64 p, {%2, %3};\n\tmov.b64 q, {%4, %4};\n\tmul.rn.f32x2 p, p, q;\n\t"
        "mov.b64 {%0, %1}, p;\n\t}" : "=f"(r.a), "=f"(r.b) : "f"(x.a), "f"(x.b), "f"(y));
    return r;
}
__device__ __forceinline__ F2 fma2(F2 x, float y, F2 z) {
    F2 r;
    asm("{\n\t.reg .b64 p, q, s;\n\tmov.b64 p, {%2, %3};\n\tmov.b64 q, {%4, %4};\n\tmov.b64 s, {%5, %6};\n\t"
        "fma.rn.f32x2 p, p, q, s;\n\tmov.b64 {%0, %1}, p;\n\t}"
        : "=f"(r.a), "=f"(r.b) : "f"(x.a), "f"(x.b), "f"(y), "f"(z.a), "f"(z.b));
    return r;
}

/// child_slabs on a DBoxNode: per axis both children's centre distances
/// (c - o) / d in one packed subtract and multiply, then entry and exit as
/// that distance -+ h |1/d| in two packed fused multiply-adds: 12 packed
/// operations for both boxes, and no minimum or maximum to order the planes
/// (the exact form has 12 of each).  Node steps are issue-bound, so this shows
/// in full: 1M-triangle frame, 64 samples 46.5 -> 43.8 ms, Cornell box 1409 ->
/// 1357 us, 300k closest-hit rays 42.9 -> 39.2 us (with the two 32-byte loads,
/// of which the frame's share is 0.8 ms).
///
/// Conservative: with eps = 2^-24, D = |c - o| / |d| and H = h / |d|, either
/// distance errs by at most (3 D + H + |distance|) eps (subtraction, 1/d and
/// multiplication on the first term, 1/d on the second, the sum's rounding).
/// pack_boxes enlarges h by 16 eps, which covers D <= H; beyond, |distance| <=
/// D + H and half of the exit's widening (13 eps in all) of a distance of at
/// least D - H covers the rest, since 16 + 6.5 (D / H - 1) >= 4 D / H + 2, with
/// at least 2.5 D eps to spare for the triangle test's own rounding.  (The
/// approximate reciprocal errs by 2 eps, which takes 1 D of that; it gained 1 %
/// on the frame.)
__device__ __forceinline__ void child_boxes(float4 x, float4 y, float4 z, Vec3 org, Vec3 idir, float tmin, float tmax,
                                            float& n0, float& f0, float& n1, float& f1) {
    const float ax = fabsf(idir.x), ay = fabsf(idir.y), az = fabsf(idir.z);
    const F2 cx = mul2(sub2(F2{x.x, x.y}, org.x), idir.x), hx{x.z, x.w};
    const F2 cy = mul2(sub2(F2{y.x, y.y}, org.y), idir.y), hy{y.z, y.w};
    const F2 cz = mul2(sub2(F2{z.x, z.y}, org.z), idir.z), hz{z.z, z.w};
    const F2 nx = fma2(hx, -ax, cx), ny = fma2(hy, -ay, cy), nz = fma2(hz, -az, cz);
    const F2 fx = fma2(hx, ax, cx), fy = fma2(hy, ay, cy), fz = fma2(hz, az, cz);
    n0 = fmaxf3(nx.a, ny.a, fmaxf(nz.a, tmin));
    n1 = fmaxf3(nx.b, ny.b, fmaxf(nz.b, tmin));
    f0 = fminf3(fx.a, fy.a, fminf(fz.a, tmax)) * kSlabWiden;
    f1 = fminf3(fx.b, fy.b, fminf(fz.b, tmax)) * kSlabWiden;
}

/// A box node in two 32-byte loads.
__device__ __forceinline__ void load_boxes(const DBoxNode* n, float4& x, float4& y, float4& z, int2& ref) {
    asm("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=f"(x.x), "=f"(x.y), "=f"(x.z), "=f"(x.w), "=f"(y.x), "=f"(y.y), "=f"(y.z), "=f"(y.w) : "l"(n));
    asm("ld.global.nc.v8.b32 {%0, %1, %2, %3, %4, %5, _, _}, [%6 + 32];"
        : "=f"(z.x), "=f"(z.y), "=f"(z.z), "=f"(z.w), "=r"(ref.x), "=r"(ref.y) : "l"(n));
}

/// Set in Traversal::hit when the exact traversal has to find the hit: another
/// triangle was hit at exactly the distance of the closest one (positions in
/// leaf order stay below 2^28), or the direction is none that boxes_take.
constexpr int kRedoBit = 1 << 30;

/// BVH traversal of one ray as a resumable state: start() sets it up, run()
/// advances it.  For kAnyHit the first triangle hit inside (tmin, tmax) is
/// kept; otherwise the closest one, with `tmax` shrunk to its distance.  `hit`
/// is the triangle's position in leaf order, or -1.  A packed traversal
/// (kExact = false) must be followed by resolve().
///
/// A packed any-hit traversal takes the first child first, whichever is nearer:
/// the answer does not depend on the order, and not ordering the children saves
/// more than it costs (frame 47.0 -> 46.2 ms, 24-view batch 9.87 -> 9.49 ms).
///
/// With kYield, run() may return early, after a leaf, when fewer than
/// `min_active` lanes of the warp are still traversing: the caller gives the
/// lanes whose rays are done new rays and calls run() again, which continues
/// exactly where it stopped (dynamic ray fetch; Aila & Laine, "Understanding
/// the Efficiency of Ray Traversal on GPUs", HPG 2009).  Stopping changes
/// nothing in the order nodes and triangles are visited, so the result is the
/// same as an uninterrupted traversal.
///
/// Self-checks: at most `max_steps` steps, node and triangle references checked
/// against the array sizes and the stack against its capacity; a failed check
/// ORs a kFault* bit into `*fault` and ends the traversal with no hit.
template <bool kAnyHit, bool kCount, bool kYield, bool kExact>
struct Traversal {
    Vec3 org, dir, idir;
    RayShear rs;
    float tmin, tmax;
    int node, sp, hit;
    float hu, hv;   // barycentrics of the closest hit (kAnyHit: unused)
    uint32_t steps;

    template <class Stack>
    __device__ __forceinline__ void start(Vec3 o, Vec3 d, float t0, float t1, bool active, Stack& stack) {
        org = o;
        dir = d;
        tmin = t0;
        tmax = t1;
        idir = kExact ? safe_inverse(d) : vec3(1.0f / d.x, 1.0f / d.y, 1.0f / d.z);   // the same where boxes_take(d)
        rs = make_shear(o, d);
        sp = 0;
        hit = -1;
        hu = hv = 0.0f;
        steps = 0;
        node = active ? 0 : kStackSentinel;
        stack.put(sp++, kStackSentinel);
        if (!kExact && active && !boxes_take(d)) {   // nothing to run, resolve() traces the ray
            node = kStackSentinel;
            hit = kRedoBit;
        }
    }

    __device__ __forceinline__ bool fail(unsigned int* fault, unsigned int bit) {
        atomicOr(fault, bit);
        hit = -1;
        node = kStackSentinel;
        return true;
    }

    /// Advances the traversal; true when it has finished.  `exact_nodes` is
    /// used by the exact form, `boxes` by the packed one.
    template <class Stack>
    __device__ __forceinline__ bool run(const DNode* __restrict__ exact_nodes, const DBoxNode* __restrict__ boxes,
                                        const DTri* __restrict__ tris, TraversalCounters& ctr, uint32_t num_nodes,
                                        uint32_t num_tris, uint32_t max_steps, unsigned int* fault, Stack& stack,
                                        int min_active) {
        while (node != kStackSentinel) {
            // Descend inner nodes until a leaf, the end or a reference outside the
            // node array is reached: as unsigned numbers leaf references and the
            // sentinel lie above every node index, so one comparison decides.
            while ((uint32_t)node < num_nodes) {
                if (++steps > max_steps) return fail(fault, kFaultTraversalSteps);
                if (kCount) ctr.nodes++;
                float n0, f0, n1, f1;
                int2 r;
                if (kExact) {
                    const DNode* n = exact_nodes + node;
                    const float4 a = ldg4(n->b0);
                    const float4 b = ldg4(n->b1);
                    const float4 c = ldg4(n->b2);
                    const int4 r4 = __ldg(reinterpret_cast<const int4*>(n->ref));
                    r = make_int2(r4.x, r4.y);
                    child_slabs(a, b, c, org, idir, tmin, tmax, n0, f0, n1, f1);
                } else {
                    float4 x, y, z;
                    load_boxes(boxes + node, x, y, z, r);
                    child_boxes(x, y, z, org, idir, tmin, tmax, n0, f0, n1, f1);
                }
                const bool h0 = n0 <= f0, h1 = n1 <= f1;
                if (h0 && h1) {
                    int near = r.x, far = r.y;
                    if ((kExact || !kAnyHit) && n1 < n0) { near = r.y; far = r.x; }
                    if (sp >= kTraversalStack) return fail(fault, kFaultTraversalSteps);
                    stack.put(sp++, far);
                    node = near;
                } else if (h0) {
                    node = r.x;
                } else if (h1) {
                    node = r.y;
                } else {
                    if (sp <= 0) return fail(fault, kFaultTraversalSteps);
                    node = stack.get(--sp);
                }
            }
            if (node == kStackSentinel) break;
            if (node >= 0) return fail(fault, kFaultNodeIndex);
            // Leaf: ~node = (first << 3) | (count - 1)
            const uint32_t v = ~(uint32_t)node;
            const uint32_t first = v >> 3, count = (v & 7u) + 1u;
            if (first + count > num_tris) return fail(fault, kFaultTriIndex);
            if (++steps > max_steps) return fail(fault, kFaultTraversalSteps);
            for (uint32_t i = first; i < first + count; ++i) {
                const DTri* tp = tris + i;
                const float4 p0 = ldg4(tp->v0), p1 = ldg4(tp->v1), p2 = ldg4(tp->v2);
                if (kCount) ctr.tris++;
                float t, u, w;
                if (kAnyHit || kExact) {
                    if (intersect_triangle(rs, tri_vertex(p0), tri_vertex(p1), tri_vertex(p2), tmin, tmax, &t, &u, &w)) {
                        hit = (int)i;
                        tmax = t;
                        if (kAnyHit) break;
                        hu = u;
                        hv = w;
                    }
                } else if (intersect_triangle_upto(rs, tri_vertex(p0), tri_vertex(p1), tri_vertex(p2), tmin, tmax, &t,
                                                   &u, &w)) {
                    if (t < tmax) {
                        hit = (int)i;
                        tmax = t;
                        hu = u;
                        hv = w;
                    } else if (hit >= 0 && (hit & ~kRedoBit) != (int)i) {
                        // (Without a hit, tmax is the ray's own end, which is no hit; a tree of
                        // one leaf has it as both children of its root.)
                        hit |= kRedoBit;
                    }
                }
            }
            if (kAnyHit && hit >= 0) return true;
            if (sp <= 0) return fail(fault, kFaultTraversalSteps);
            node = stack.get(--sp);
            if (kYield && node != kStackSentinel && __popc(__activemask()) < min_active) return false;
        }
        return true;
    }

    /// After a packed traversal that began with the end `t1`: where kRedoBit is
    /// set, the hit that the exact traversal finds.
    __device__ __forceinline__ void resolve(const SceneView& s, float t1);
};

/// The closest hit of one ray by the exact traversal, out of line: only the few
/// rays with kRedoBit come here.  (Whether there is any hit is the same question
/// for both queries: they part only after the first.)
struct ExactHit { int hit; float t, u, v; };
static __device__ __noinline__ ExactHit closest_exact(const DNode* nodes, const DTri* tris, uint32_t num_nodes,
                                                      uint32_t num_tris, uint32_t max_steps, unsigned int* fault,
                                                      Vec3 org, Vec3 dir, float tmin, float tmax) {
    LocalStack stack;
    TraversalCounters tc{0u, 0u};
    Traversal<false, false, false, true> tr;
    tr.start(org, dir, tmin, tmax, true, stack);
    tr.run(nodes, nullptr, tris, tc, num_nodes, num_tris, max_steps, fault, stack, 0);
    return ExactHit{tr.hit, tr.tmax, tr.hu, tr.hv};
}

template <bool kAnyHit, bool kCount, bool kYield, bool kExact>
__device__ __forceinline__ void Traversal<kAnyHit, kCount, kYield, kExact>::resolve(const SceneView& s, float t1) {
    if (kExact || hit < kRedoBit) return;
    const ExactHit e = closest_exact(s.nodes(), s.tris, s.num_nodes, s.num_tris, s.max_steps, s.fault, org, dir, tmin, t1);
    hit = e.hit;
    tmax = e.t;
    hu = e.u;
    hv = e.v;
}

/// Traverses a scene's BVH for one ray to completion (see Traversal).  Returns
/// the hit triangle's position in leaf order, or -1; `tmax` becomes the hit
/// distance, (u, v) the barycentrics of a closest hit.
template <bool kAnyHit, bool kCount, bool kExact, class Stack>
__device__ __forceinline__ int traverse_uv(const SceneView& s, Vec3 org, Vec3 dir, float tmin, float& tmax, float& u,
                                           float& v, TraversalCounters& ctr, Stack& stack) {
    Traversal<kAnyHit, kCount, false, kExact> tr;
    const float t1 = tmax;
    tr.start(org, dir, tmin, tmax, s.num_tris > 0, stack);
    tr.run(s.nodes(), s.boxes, s.tris, ctr, s.num_nodes, s.num_tris, s.max_steps, s.fault, stack, 0);
    tr.resolve(s, t1);
    tmax = tr.tmax;
    u = tr.hu;
    v = tr.hv;
    return tr.hit;
}

/// Closest hit for the render kernels (the counting ones walk the exact form).
template <bool kCount, class Stack>
__device__ __forceinline__ int traverse_closest_uv(const SceneView& s, Vec3 org, Vec3 dir, float tmin, float& tmax,
                                                   float& u, float& v, TraversalCounters& ctr, Stack& stack) {
    return traverse_uv<false, kCount, kCount>(s, org, dir, tmin, tmax, u, v, ctr, stack);
}

/// Whether a shadow ray is blocked before `tmax`.
template <bool kCount, class Stack>
__device__ __forceinline__ bool occluded(const SceneView& s, Vec3 org, Vec3 dir, float tmin, float tmax,
                                         TraversalCounters& ctr, Stack& stack) {
    float u, v;
    return traverse_uv<true, kCount, kCount>(s, org, dir, tmin, tmax, u, v, ctr, stack) >= 0;
}

}  // namespace sol_b200
