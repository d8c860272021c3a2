// The pruned transforms of FP32 grids.
#include "fourier_kernels.cuh"

namespace vpbs {

int fourier_attributes_f32(vpbs_handle* h, const FourierPlan& F) { return set_attributes<float>(h, F); }
int fourier_forward_f32(vpbs_handle* h, const void* grid) { return run_forward_t<float>(h, grid); }
int fourier_operator_f32(vpbs_handle* h, const FourierOp& op) { return run_operator_t<float>(h, op); }
int fourier_inverse_f32(vpbs_handle* h, void* grid, bool quad) { return run_inverse_t<float>(h, grid, quad); }

}  // namespace vpbs
