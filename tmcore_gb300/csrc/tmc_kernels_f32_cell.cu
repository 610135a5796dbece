// FP32 instantiation of the cell passes (tmc_kernels_f32.cu has the others).
#include "tmc_kernels_impl.cuh"

namespace tmc {
TMC_INSTANTIATE_CELL(float)
}  // namespace tmc
