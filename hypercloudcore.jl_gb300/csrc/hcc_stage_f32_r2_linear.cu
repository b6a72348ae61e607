// hcc_stage_f32_r2_linear.cu — stage kernels of the linear modules (advection, kinetic relaxation), float arithmetic,
// reconstruction degree 2.
#include "hcc_stage_impl.cuh"
namespace hcc {
const StageOps *stage_ops_f32_r2_linear(int D, int M, int pde) { return lookup_linear<float, 2>(D, M, pde); }
}  // namespace hcc
