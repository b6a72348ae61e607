// hcc_stage_f32_r1.cu — stage kernels of the Euler modules, float arithmetic, reconstruction degree 1.
#include "hcc_stage_impl.cuh"
namespace hcc {
const StageOps *stage_ops_f32_r1(int D, int M, int pde) {
    return pde == HCC_PDE_EULER ? lookup_euler<float, 1>(D, M) : stage_ops_f32_r1_linear(D, M, pde);
}
}  // namespace hcc
