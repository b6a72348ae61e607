// hcc_stage_f64_r2.cu — stage kernels of the Euler modules, double arithmetic, reconstruction degree 2.
#include "hcc_stage_impl.cuh"
namespace hcc {
const StageOps *stage_ops_f64_r2(int D, int M, int pde) {
    return pde == HCC_PDE_EULER ? lookup_euler<double, 2>(D, M) : stage_ops_f64_r2_linear(D, M, pde);
}
}  // namespace hcc
