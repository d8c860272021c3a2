// The pruned transforms of FP64 grids.
#include "fourier_kernels.cuh"

namespace vpbs {

int fourier_attributes_f64(vpbs_handle* h, const FourierPlan& F) { return set_attributes<double>(h, F); }
int fourier_forward_f64(vpbs_handle* h, const void* grid) { return run_forward_t<double>(h, grid); }
int fourier_operator_f64(vpbs_handle* h, const FourierOp& op) { return run_operator_t<double>(h, op); }
int fourier_inverse_f64(vpbs_handle* h, void* grid) { return run_inverse_t<double>(h, grid, false); }

}  // namespace vpbs
