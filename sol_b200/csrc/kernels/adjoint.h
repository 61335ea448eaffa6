// Launchers of the adjoint (K7) and loss (K8) kernels.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "../core/layout.h"

namespace sol_b200 {

constexpr int kAdjointBlock = 128;

/// Builds of the adjoint kernels, by the resident blocks per SM their registers
/// allow.  Records and shading leave little for the traversal at 16 blocks (32
/// registers): a path then takes three times as long as at 4 (128 registers,
/// hardly any spills), which only many paths in flight make up for.  So the
/// build follows the path vertices of the call, counting each path with its
/// length limit, per resident lane of the 4-block build.  Measured, adjoint at
/// 4 / 8 / 16 blocks (us; in brackets the vertices per lane, 4 blocks are taken up
/// to 20, 8 up to 42): textured Cornell, limit 16: 65.5k paths 390 / 518 / 812
/// (14), 73.7k 406 / 562 / 871 (16), 131k 647 / 612 / 908 (28), 197k 977 / 851 / 964
/// (42), 262k 1346 / 1076 / 1072 (55), 1.6M 10256 / 7844 / 6032; textured sphere
/// field, limit 8: 33k 198 / 306 / 557 (3), 131k 213 / 310 / 545 (14), 262k 285 / 407 /
/// 614 (28), 410k 393 / 513 / 760 (43), 819k 542 / 612 / 851 (86), 1.6M 907 / 891 /
/// 1191 (173).  Fused at 4 / 10 blocks: Cornell 65.5k 388 / 593 (14), 86k 526 / 642
/// (18), 131k 697 / 696 (28), 262k 1424 / 1101 (55), 1M 5598 / 4072; spheres 147k
/// 250 / 400 (16), 229k 311 / 479 (24), 492k 478 / 642 (52), 1M 771 / 787 (111), 2.2M
/// 1812 / 1529 (228).  The limit says little about how long paths are, so no line
/// serves both: these are the Cornell box's, whose paths use their limit; the
/// sphere field's shorter paths would stay with the smaller build about four times
/// as long (262k paths take 411 us instead of 285; one build for all took 636).
enum class AdjointBuild { kSmall, kMiddle, kFull };
constexpr int kAdjointSmallBlocks = 4, kAdjointMiddleBlocks = 8, kAdjointFullBlocks = 16;
constexpr int kFusedFullBlocks = 10;   // the fused kernel's build for middle and full calls
constexpr uint64_t kAdjointSmallVerticesPerLane = 20, kAdjointMiddleVerticesPerLane = 42;

/// Longest path the adjoint replays (vertex records per lane).
constexpr int kAdjointMaxDepth = 16;

/// One view of a fused forward + adjoint batch.
struct AdjView {
    DCamera cam;
    uint32_t scene;
    uint32_t width, height;
    uint32_t sample_count;
    uint64_t sample_index;
    float* film;            // forward sums are added into
    const float* target;    // the loss compares (sum / sample_count) with it
    float* grad;            // the scene's parameter gradient, added into
    double* loss;           // added into
    uint32_t item_begin;    // first work item of the view (fused_items per view, in order)
    uint32_t group;         // lanes per pixel (fused_group of sample_count)
};

/// Lanes per pixel of the fused kernel for a view of `spp` samples: the
/// smallest power of two >= spp, at most 32.
inline uint32_t fused_group(uint32_t spp) {
    uint32_t g = 1;
    while (g < spp && g < 32) g <<= 1;
    return g;
}

/// Work items (one warp each) of a width x height view in the fused kernel:
/// 8x4-pixel tiles, 32 / g pixels per item.
inline uint64_t fused_items(uint32_t width, uint32_t height, uint32_t spp) {
    return (uint64_t)((width + 7) / 8) * ((height + 3) / 4) * fused_group(spp);
}

/// Most constant-texture values whose gradients a block gathers in shared memory.
constexpr uint32_t kAdjointMaxSharedParams = 2048;   // 8 KB per block, so 16 blocks fit an SM

/// The build for a call of `paths` paths of at most `max_path_len` vertices.
AdjointBuild adjoint_build(uint64_t paths, uint32_t max_path_len, int sms);
int adjoint_blocks_per_sm(AdjointBuild build, uint32_t n_shared);
int fused_blocks_per_sm(AdjointBuild build);

/// The kernels of each build (adjoint.cu, adjoint_small.cu).
using AdjointFn = void (*)(SceneView, DCamera, DConfig, uint64_t, uint32_t, uint32_t, uint32_t, uint32_t, const float*,
                           float*, uint32_t, float4*, DeviceCounters*, uint32_t);
using FusedFn = void (*)(const AdjView*, uint32_t, uint32_t, const SceneView*, DConfig, DeviceCounters*);
AdjointFn adjoint_fn_small();
AdjointFn adjoint_fn_middle();
AdjointFn adjoint_fn_full();
FusedFn fused_fn_small();
FusedFn fused_fn_full();

/// Forward render + L2-loss adjoint of every view in one persistent launch.
cudaError_t launch_fused_forward_adjoint(const AdjView* views, uint32_t num_views, uint32_t total_items,
                                         const SceneView* scenes, const DConfig& cfg, DeviceCounters* counters,
                                         AdjointBuild build, int grid, cudaStream_t stream);

/// Adds dL/d(parameters) of the paths of samples [sample_index, + sample_count)
/// of every pixel into `grad`, given dL/dfilm (3 planes of width*height).  Each
/// work item replays `chunk` consecutive samples of one pixel; the first
/// `n_shared` parameters (at most kAdjointMaxSharedParams, all of them constant
/// textures) are gathered per block in shared memory.
/// With `texels4` (num_texels float4, one per image texel in arena order) the
/// image-texel gradients are gathered there with vector reductions and added
/// into `grad` afterwards (parameter first_texel_param + image offset + ...).
cudaError_t launch_adjoint(const SceneView& s, const DCamera& cam, const DConfig& cfg, uint64_t sample_index,
                           uint32_t sample_count, uint32_t chunk, uint32_t width, uint32_t height,
                           const float* dl_dfilm, float* grad, uint32_t n_shared, float4* texels4, uint64_t num_texels,
                           uint32_t num_images, uint64_t first_texel_param, DeviceCounters* counters,
                           AdjointBuild build, int grid, cudaStream_t stream);

/// Adds sum (scale * film - target)^2 into *loss and writes dL/dfilm (optional).
cudaError_t launch_l2_loss(const float* film, const float* target, uint64_t n, float scale, float* dl_dfilm,
                           double* loss, int grid, cudaStream_t stream);

}  // namespace sol_b200
