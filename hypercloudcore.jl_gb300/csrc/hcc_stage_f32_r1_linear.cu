// hcc_stage_f32_r1_linear.cu — stage kernels of the linear modules (advection, kinetic relaxation), float arithmetic,
// reconstruction degree 1.
#include "hcc_stage_impl.cuh"
namespace hcc {
const StageOps *stage_ops_f32_r1_linear(int D, int M, int pde) { return lookup_linear<float, 1>(D, M, pde); }
}  // namespace hcc
