// hcc_stage_f64_r1.cu — stage kernels of the Euler modules, double arithmetic, reconstruction degree 1.
#include "hcc_stage_impl.cuh"
namespace hcc {
const StageOps *stage_ops_f64_r1(int D, int M, int pde) {
    return pde == HCC_PDE_EULER ? lookup_euler<double, 1>(D, M) : stage_ops_f64_r1_linear(D, M, pde);
}
}  // namespace hcc
