// K9: batched closest-hit / any-hit queries, the device side of
// TriangleMesh::intersect_closest and TriangleMesh::intersect_any
// (src/triangle_mesh.cpp:64-117) for raw rays.  One thread per ray; used to
// check hit identities against the host checker and to time traversal alone.
#include <cuda_runtime.h>

#include "kernels.h"
#include "traverse.cuh"

namespace sol_b200 {

namespace {

/// One ray per thread, on the first `lanes` lanes of each warp (a power of two):
/// a batch that the resident warps could hold with fewer lanes is spread over
/// them, since the rays of a warp mostly trace one after another (1,000 closest
/// hits 25.2 -> 20.1 us with the launch; from 8 lanes on the longest ray alone
/// decides, 20,000 take 43 us with 32 as with 8).  64-thread blocks leave the SM as
/// soon as their own longest ray ends.  Occupancies (16 blocks: 64 registers, 24:
/// 40): closest hits of 300k rays 44.7 us against 46.9 at 24 and 49.6 at 32 blocks
/// (4M rays 381, 359, 366), 1.5M shadow rays 123 us against 124 at 16 and 139 at 32;
/// 128-thread blocks 47.0 and 123.
template <bool kAnyHit>
__global__ void __launch_bounds__(kTraceBlock, kAnyHit ? 24 : 16)
trace_rays(SceneView s, const SolGpuRay* __restrict__ rays, uint32_t count, SolGpuHit* __restrict__ hits, uint32_t lanes) {
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t i = (blockIdx.x * (kTraceBlock / 32u) + (threadIdx.x >> 5)) * lanes + lane;
    if (lane >= lanes || i >= count) return;
    const float4 a = __ldg(reinterpret_cast<const float4*>(rays + i));
    const float4 b = __ldg(reinterpret_cast<const float4*>(rays + i) + 1);
    const Vec3 org = vec3(a.x, a.y, a.z), dir = vec3(b.x, b.y, b.z);
    TraversalCounters tc{0u, 0u};
    LocalStack stack;
    Traversal<kAnyHit, false, false> tr;   // in order, so that which of several blockers is reported is the host's choice
    tr.start(org, dir, a.w, b.w, s.num_tris > 0, stack);
    tr.run(s.nodes, s.tris, tc, s.num_nodes, s.num_tris, s.max_steps, s.fault, stack, 0);
    SolGpuHit h;
    h.tri = -1; h.t = 0.0f; h.u = 0.0f; h.v = 0.0f;
    if (tr.hit >= 0) {
        h.tri = (int32_t)__ldg(&s.tris[tr.hit].prim);
        h.t = tr.tmax;
        if (!kAnyHit) { h.u = tr.hu; h.v = tr.hv; }
    }
    hits[i] = h;
}

}  // namespace

cudaError_t launch_trace(const SceneView& s, const SolGpuRay* rays, uint32_t count, bool any_hit,
                         SolGpuHit* hits, int sms, cudaStream_t stream) {
    if (count == 0) return cudaSuccess;
    const uint64_t warps = (uint64_t)sms * 16 * (kTraceBlock / 32);   // resident warps of the closest-hit kernel
    uint32_t lanes = 1;
    while (lanes < 32u && lanes * warps < count) lanes *= 2;
    if (lanes > 4u) lanes = 32;
    const uint32_t per_block = lanes * (kTraceBlock / 32);
    const uint32_t grid = (uint32_t)(((uint64_t)count + per_block - 1) / per_block);
    if (any_hit) trace_rays<true><<<grid, kTraceBlock, 0, stream>>>(s, rays, count, hits, lanes);
    else trace_rays<false><<<grid, kTraceBlock, 0, stream>>>(s, rays, count, hits, lanes);
    return cudaGetLastError();
}

}  // namespace sol_b200
