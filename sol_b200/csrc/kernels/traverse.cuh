// BVH2 traversal on the device: the GPU statement of
// TriangleMesh::intersect_closest / intersect_any (src/triangle_mesh.cpp:64-117),
// which SoL runs through bvh v2's SingleRayTraverser.
//
// Layout: every inner node is 64 bytes holding both child boxes, fetched in two
// 256-bit read-only loads; triangles are 48 bytes (three 128-bit loads).  The
// traversal is the stack-based "while-while" loop of Aila & Laine ("Understanding
// the Efficiency of Ray Traversal on GPUs", HPG 2009): descend inner nodes
// nearest-child first, pushing the farther child, until a leaf is reached; then
// test the leaf's triangles.  Box tests compute (bound - origin) / direction and
// widen the exit distance by kSlabWiden so that they are conservative; they are
// the same operations as the host traversal's, so both visit children in the same
// order and resolve equal-distance hits alike.  The triangle test is the shared
// watertight test, so a hit found here is bit-identical to the one the host finds.
// (Boxes stored as centre and half size need 12 fewer operations per node: frame
// 46.1 -> 43.7 ms, Cornell box 1414 -> 1351 us.  But they have to be enlarged for
// their rounding, which changes which boxes count as entered at their faces: with
// coordinates of 1000 and more and a ray offset of 1e-5, up to 0.04 % of the
// bounces then hit the surface that they leave, whose box the host culls.)
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

/// A node in two 32-byte loads (four of 16 bytes: frame 48.0 against 46.1 ms,
/// Cornell box 1465 against 1414 us).
__device__ __forceinline__ void load_node(const DNode* n, float4& a, float4& b, float4& c, int2& ref) {
    asm("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=f"(a.x), "=f"(a.y), "=f"(a.z), "=f"(a.w), "=f"(b.x), "=f"(b.y), "=f"(b.z), "=f"(b.w) : "l"(n));
    asm("ld.global.nc.v8.b32 {%0, %1, %2, %3, %4, %5, _, _}, [%6 + 32];"
        : "=f"(c.x), "=f"(c.y), "=f"(c.z), "=f"(c.w), "=r"(ref.x), "=r"(ref.y) : "l"(n));
}

/// BVH traversal of one ray as a resumable state: start() sets it up, run()
/// advances it.  For kAnyHit the first triangle hit inside (tmin, tmax) is
/// kept; otherwise the closest one, with `tmax` shrunk to its distance.  `hit`
/// is the triangle's position in leaf order, or -1.
///
/// Without kOrdered (any-hit only) the first child is taken first, whichever is
/// nearer.  Which of several hits is found follows the order, whether there is
/// one does not, and not ordering the children saves more than it costs (frame
/// 47.0 -> 46.2 ms, 24-view batch 9.87 -> 9.49 ms).
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
template <bool kAnyHit, bool kCount, bool kYield, bool kOrdered = true>
struct Traversal {
    static_assert(kAnyHit || kOrdered, "a closest hit needs the nearer child first");
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
        idir = safe_inverse(d);
        rs = make_shear(o, d);
        sp = 0;
        hit = -1;
        hu = hv = 0.0f;
        steps = 0;
        node = active ? 0 : kStackSentinel;
        stack.put(sp++, kStackSentinel);
    }

    __device__ __forceinline__ bool fail(unsigned int* fault, unsigned int bit) {
        atomicOr(fault, bit);
        hit = -1;
        node = kStackSentinel;
        return true;
    }

    /// Advances the traversal; true when it has finished.
    template <class Stack>
    __device__ __forceinline__ bool run(const DNode* __restrict__ nodes, const DTri* __restrict__ tris,
                                        TraversalCounters& ctr, uint32_t num_nodes, uint32_t num_tris,
                                        uint32_t max_steps, unsigned int* fault, Stack& stack, int min_active) {
        while (node != kStackSentinel) {
            // Descend inner nodes until a leaf, the end or a reference outside the
            // node array is reached: as unsigned numbers leaf references and the
            // sentinel lie above every node index, so one comparison decides.
            while ((uint32_t)node < num_nodes) {
                if (++steps > max_steps) return fail(fault, kFaultTraversalSteps);
                if (kCount) ctr.nodes++;
                float4 a, b, c;
                int2 r;
                load_node(nodes + node, a, b, c, r);
                float n0, f0, n1, f1;
                child_slabs(a, b, c, org, idir, tmin, tmax, n0, f0, n1, f1);
                const bool h0 = n0 <= f0, h1 = n1 <= f1;
                if (h0 && h1) {
                    int near = r.x, far = r.y;
                    if (kOrdered && n1 < n0) { near = r.y; far = r.x; }
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
                if (intersect_triangle(rs, tri_vertex(p0), tri_vertex(p1), tri_vertex(p2), tmin, tmax, &t, &u, &w)) {
                    hit = (int)i;
                    tmax = t;
                    if (kAnyHit) break;
                    hu = u;
                    hv = w;
                }
            }
            if (kAnyHit && hit >= 0) return true;
            if (sp <= 0) return fail(fault, kFaultTraversalSteps);
            node = stack.get(--sp);
            if (kYield && node != kStackSentinel && __popc(__activemask()) < min_active) return false;
        }
        return true;
    }
};

/// Closest hit of one ray of a scene.  Returns the hit triangle's position in leaf
/// order, or -1; `tmax` becomes the hit distance, (u, v) its barycentrics.
template <bool kCount, class Stack>
__device__ __forceinline__ int traverse_closest_uv(const SceneView& s, Vec3 org, Vec3 dir, float tmin, float& tmax,
                                                   float& u, float& v, TraversalCounters& ctr, Stack& stack) {
    Traversal<false, kCount, false> tr;
    tr.start(org, dir, tmin, tmax, s.num_tris > 0, stack);
    tr.run(s.nodes, s.tris, ctr, s.num_nodes, s.num_tris, s.max_steps, s.fault, stack, 0);
    tmax = tr.tmax;
    u = tr.hu;
    v = tr.hv;
    return tr.hit;
}

/// Whether a shadow ray is blocked before `tmax`.  The counting kernels take the
/// host's order, so that they count what the host visits.
template <bool kCount, class Stack>
__device__ __forceinline__ bool occluded(const SceneView& s, Vec3 org, Vec3 dir, float tmin, float tmax,
                                         TraversalCounters& ctr, Stack& stack) {
    Traversal<true, kCount, false, kCount> tr;
    tr.start(org, dir, tmin, tmax, s.num_tris > 0, stack);
    tr.run(s.nodes, s.tris, ctr, s.num_nodes, s.num_tris, s.max_steps, s.fault, stack, 0);
    return tr.hit >= 0;
}

}  // namespace sol_b200
