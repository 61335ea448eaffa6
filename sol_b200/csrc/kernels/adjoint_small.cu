// The builds of the adjoint kernels for small and middle-sized calls (see
// AdjointBuild).
#include "adjoint_kernels.cuh"

namespace sol_b200 {

AdjointFn adjoint_fn_small() { return prb_adjoint<kAdjointSmallBlocks>; }
AdjointFn adjoint_fn_middle() { return prb_adjoint<kAdjointMiddleBlocks>; }
FusedFn fused_fn_small() { return fused_forward_adjoint<kAdjointSmallBlocks>; }

}  // namespace sol_b200
