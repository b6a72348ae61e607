// hcc_stage_f64_r2_linear.cu — stage kernels of the linear modules (advection, kinetic relaxation), double arithmetic,
// reconstruction degree 2.
#include "hcc_stage_impl.cuh"
namespace hcc {
const StageOps *stage_ops_f64_r2_linear(int D, int M, int pde) { return lookup_linear<double, 2>(D, M, pde); }
}  // namespace hcc
