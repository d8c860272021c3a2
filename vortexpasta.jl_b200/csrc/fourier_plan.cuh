// Plans of the pruned transforms (fourier.cu) and the entry points of their kernels per grid precision.
#pragma once

#include "fft_lines.cuh"
#include "vpbs_internal.cuh"

namespace vpbs {

constexpr int kFftThreads = 512;  // most threads of a block (register bound of the kernels)
constexpr size_t kFftSmemMost = 200 * 1024;

struct FourierShape {
    int threads = 0;
    size_t smem = 0;
};

struct FourierPlan {
    fft::Plan px, py, pz;
    int LY = 1, LYq = 1, ltxy = 0, ltxz = 0, kx = 0, kxp = 0;
    FourierShape sx, sq, sy, sz;
    size_t twr = 0;  // offset (in complex values) of e^{-2 pi i k / n0} in the tables
};

// fourier_f32.cu, fourier_f64.cu
int fourier_attributes_f32(vpbs_handle* h, const FourierPlan& F);
int fourier_forward_f32(vpbs_handle* h, const void* grid);
int fourier_operator_f32(vpbs_handle* h, const FourierOp& op);
int fourier_inverse_f32(vpbs_handle* h, void* grid, bool quad);
int fourier_attributes_f64(vpbs_handle* h, const FourierPlan& F);
int fourier_forward_f64(vpbs_handle* h, const void* grid);
int fourier_operator_f64(vpbs_handle* h, const FourierOp& op);
int fourier_inverse_f64(vpbs_handle* h, void* grid);

}  // namespace vpbs
