// Launchers of the adjoint and loss kernels, and the builds of the adjoint
// kernels for large calls (the others are in adjoint_small.cu: the kernels are
// compiled in two units because the compiler does not take all builds in one).
#include <algorithm>

#include "adjoint_kernels.cuh"

namespace sol_b200 {

namespace {

/// Adds the interleaved texel gradients (one float4 per texel of every image,
/// images in arena order) into the planar parameter vector: image k's texel i
/// channel c is parameter `first_texel_param + images[k].offset + c * w * h + i`.
__global__ void __launch_bounds__(256)
gather_texels(const float4* __restrict__ texels4, uint64_t num_texels, const DImage* __restrict__ images,
              uint32_t num_images, uint64_t first_texel_param, float* __restrict__ grad) {
    for (uint64_t q = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; q < num_texels;
         q += (uint64_t)gridDim.x * blockDim.x) {
        uint32_t lo = 0, hi = num_images;
        while (hi - lo > 1) { const uint32_t mid = (lo + hi) >> 1; if (images[mid].offset / 3 <= q) lo = mid; else hi = mid; }
        const DImage img = images[lo];
        const uint64_t i = q - img.offset / 3, plane = (uint64_t)img.width * img.height;
        if (i >= plane) continue;
        const float4 v = texels4[q];
        float* p = grad + first_texel_param + img.offset + i;
        if (v.x != 0.0f) p[0] += v.x;
        if (v.y != 0.0f) p[plane] += v.y;
        if (v.z != 0.0f) p[2 * plane] += v.z;
    }
}

/// K8: L = sum (scale * film - target)^2 and dL/dfilm = 2 scale (scale * film - target).
__global__ void __launch_bounds__(256)
l2_loss(const float* __restrict__ film, const float* __restrict__ target, uint64_t n, float scale,
        float* __restrict__ dl_dfilm, double* __restrict__ loss) {
    double acc = 0.0;
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        const float d = scale * film[i] - target[i];
        acc += (double)d * (double)d;
        if (dl_dfilm) dl_dfilm[i] = 2.0f * scale * d;
    }
    for (int off = 16; off > 0; off >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, off);
    __shared__ double part[8];
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
        double sum = 0.0;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) sum += part[w];
        atomicAdd(loss, sum);
    }
}

}  // namespace

AdjointFn adjoint_fn_full() { return prb_adjoint<kAdjointFullBlocks>; }
FusedFn fused_fn_full() { return fused_forward_adjoint<kFusedFullBlocks>; }

namespace {

AdjointFn adjoint_fn(AdjointBuild build) {
    return build == AdjointBuild::kFull ? adjoint_fn_full() : build == AdjointBuild::kMiddle ? adjoint_fn_middle()
                                                                                            : adjoint_fn_small();
}
FusedFn fused_fn(AdjointBuild build) { return build == AdjointBuild::kSmall ? fused_fn_small() : fused_fn_full(); }

}  // namespace

AdjointBuild adjoint_build(uint64_t paths, uint32_t max_path_len, int sms) {
    const uint64_t vertices = paths * std::min(max_path_len, (uint32_t)kAdjointMaxDepth);
    const uint64_t lanes = (uint64_t)sms * kAdjointSmallBlocks * kAdjointBlock;
    if (vertices <= kAdjointSmallVerticesPerLane * lanes) return AdjointBuild::kSmall;
    return vertices <= kAdjointMiddleVerticesPerLane * lanes ? AdjointBuild::kMiddle : AdjointBuild::kFull;
}

int fused_blocks_per_sm(AdjointBuild build) {
    int n = 0;
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, fused_fn(build), kAdjointBlock, 0) == cudaSuccess ? n : -1;
}

cudaError_t launch_fused_forward_adjoint(const AdjView* views, uint32_t num_views, uint32_t total_items,
                                         const SceneView* scenes, const DConfig& cfg, DeviceCounters* counters,
                                         AdjointBuild build, int grid, cudaStream_t stream) {
    fused_fn(build)<<<grid, kAdjointBlock, 0, stream>>>(views, num_views, total_items, scenes, cfg, counters);
    return cudaGetLastError();
}

int adjoint_blocks_per_sm(AdjointBuild build, uint32_t n_shared) {
    int n = 0;
    const size_t smem = sizeof(float) * (size_t)n_shared;
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, adjoint_fn(build), kAdjointBlock, smem) == cudaSuccess ? n : -1;
}

cudaError_t launch_adjoint(const SceneView& s, const DCamera& cam, const DConfig& cfg, uint64_t sample_index,
                           uint32_t sample_count, uint32_t chunk, uint32_t width, uint32_t height,
                           const float* dl_dfilm, float* grad, uint32_t n_shared, float4* texels4, uint64_t num_texels,
                           uint32_t num_images, uint64_t first_texel_param, DeviceCounters* counters,
                           AdjointBuild build, int grid, cudaStream_t stream) {
    const size_t smem = sizeof(float) * (size_t)n_shared;
    if (texels4 && num_texels) {
        cudaError_t e = cudaMemsetAsync(texels4, 0, sizeof(float4) * num_texels, stream);
        if (e != cudaSuccess) return e;
    }
    const uint64_t warps = (uint64_t)grid * (kAdjointBlock / 32);
    const uint64_t items = (uint64_t)width * height * ((sample_count + chunk - 1) / chunk);
    uint32_t lanes = 1;
    while (lanes < 32u && lanes * warps < items) lanes *= 2;
    adjoint_fn(build)<<<grid, kAdjointBlock, smem, stream>>>(s, cam, cfg, sample_index, sample_count, chunk, width,
                                                              height, dl_dfilm, grad, n_shared,
                                                              num_texels ? texels4 : nullptr, counters, lanes);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess || !texels4 || !num_texels) return e;
    const int blocks = (int)std::min<uint64_t>((num_texels + 255) / 256, 4096);
    gather_texels<<<blocks, 256, 0, stream>>>(texels4, num_texels, s.images, num_images, first_texel_param, grad);
    return cudaGetLastError();
}

cudaError_t launch_l2_loss(const float* film, const float* target, uint64_t n, float scale, float* dl_dfilm,
                           double* loss, int grid, cudaStream_t stream) {
    l2_loss<<<grid, 256, 0, stream>>>(film, target, n, scale, dl_dfilm, loss);
    return cudaGetLastError();
}

}  // namespace sol_b200
