// Pruned 3-D transforms of the long range with the Fourier-space operators in their middle
// (src/BiotSavart/longrange/longrange.jl:102-156, 380-583).
//
// Of the oversampled n0 x n1 x n2 transform only Ns0/2 x Ns1 x Ns2 modes are kept, so each dimension
// is transformed on its own and what the next one does not need is not written:
//   fft_x_forward   real lines -> modes k_x < Ns0/2 (two real values packed as one complex);
//   fft_y_forward   keeps Ns1 of n1 rows;
//   fft_z_operator  z lines of the three components together: forward, deconvolution, Hermitian
//                   zeroing, vorticity coefficients stored, curl / inverse Laplacian, Ewald filter,
//                   type-2 deconvolution, inverse, without leaving shared memory;
//   fft_y_inverse, fft_x_inverse   back, missing modes taken as zero.
// The complex data lives in one buffer [3][n2][n1][kxp] (kxp: Ns0/2 rounded up to the line tile);
// every kernel reads all of a line before it writes any of it, so the passes are in place.
// k_x = Ns0/2 (always zeroed) is never transformed.
//
// Bound: HBM traffic of the passes (2 + 4 / sigma + 4 / sigma^2 grids of real values for one field, 6.4 at sigma =
// 1.5, and the FP64 coefficients; 12 and more for unpruned transforms and an operator pass), then shared-memory
// and issue rate.
// Against cuFFT and the separate operator kernel: 768^3 FP64 59.0 -> 29.3 ms when first measured, 25 since;
// 384^3 FP32, four evaluations, 13.1 -> 5.8 ms; 288^3 FP32 1.39 -> 0.73 ms.
//
// Compiled once per grid precision (fourier_f32.cu, fourier_f64.cu), so that a process loads the kernels of the one
// it uses; plans are made in fourier.cu.
#pragma once

#include <cmath>

#include "fourier_plan.cuh"

namespace vpbs {
namespace {

using fft::Cplx;
using fft::LinesT;
using fft::LinesX;
using fft::Plan;

// ---- x: real <-> half spectrum ----

template <typename T, bool W>
__global__ void __launch_bounds__(kFftThreads, sizeof(T) == 4 && !W ? 2 : 1) fft_x_forward(Plan P, int64_t nl, int LY, int kx, uint32_t mkx, int kxp,
                                                             const typename Cplx<T>::type* __restrict__ in,
                                                             typename Cplx<T>::type* __restrict__ out,
                                                             const typename Cplx<T>::type* __restrict__ tw,
                                                             const typename Cplx<T>::type* __restrict__ twr) {
    using C = typename Cplx<T>::type;
    extern __shared__ __align__(16) unsigned char fft_raw[];
    C* S = reinterpret_cast<C*>(fft_raw);
    const int H = P.n;
    const int64_t l0 = (int64_t)blockIdx.x * LY;
    const int nlines = nl - l0 < LY ? (int)(nl - l0) : LY;
    const LinesX lay{P.len};
    in += l0 * H;
    out += l0 * kxp;
    fft::run_in<-1, W>(S, lay, P.p[0], nlines, [&](int line, int pos) { return in[(int64_t)line * H + pos]; });
    for (int i = 1; i < P.np; ++i) fft::run_mid<-1, W>(S, lay, P.p[i], nlines, tw);
    // z_j = x_2j + i x_2j+1 has Z_k = E_k + i O_k: X_k = E_k + e^{-2 pi i k / n} O_k
    for (int idx = threadIdx.x; idx < nlines * kx; idx += blockDim.x) {
        const int line = fft::fdiv(idx, mkx), k = idx - line * kx;
        const C a = S[lay.at(line, k)];
        const C b = S[lay.at(line, k == 0 ? 0 : H - k)];
        const C e = fft::mk((T)0.5 * (a.x + b.x), (T)0.5 * (a.y - b.y));
        const C o = fft::mk((T)0.5 * (a.y + b.y), (T)-0.5 * (a.x - b.x));
        out[(int64_t)line * kxp + k] = fft::add(e, fft::mul(o, __ldg(twr + k)));
    }
}

// Value pos of the packed transform of a line X of half-spectrum modes:
// Z_k = (X_k + conj X_{H-k}) + i e^{2 pi i k / n} (X_k - conj X_{H-k}); X_k = 0 for k >= kx (kx <= H); the
// imaginary part of X_0 does not enter a real field.
template <typename C>
__device__ __forceinline__ C x_inverse_input(const C* __restrict__ X, int pos, int H, int kx, const C* __restrict__ twr) {
    using T = decltype(C::x);
    C a = fft::mk((T)0, (T)0), b = a;
    if (pos < kx) a = X[pos];
    if (pos == 0) a.y = (T)0;
    const int q = H - pos;
    if (q < kx) b = X[q];
    const C s = fft::mk(a.x + b.x, a.y - b.y), d = fft::mk(a.x - b.x, a.y + b.y);
    const C t = fft::mul_tw<1>(d, __ldg(twr + pos));
    return fft::mk(s.x - t.y, s.y + t.x);
}

template <typename T, bool W>
__global__ void __launch_bounds__(kFftThreads, sizeof(T) == 4 && !W ? 2 : 1) fft_x_inverse(Plan P, int64_t nl, int LY, int kx, int kxp,
                                                             const typename Cplx<T>::type* __restrict__ in,
                                                             typename Cplx<T>::type* __restrict__ out,
                                                             const typename Cplx<T>::type* __restrict__ tw,
                                                             const typename Cplx<T>::type* __restrict__ twr) {
    using C = typename Cplx<T>::type;
    extern __shared__ __align__(16) unsigned char fft_raw[];
    C* S = reinterpret_cast<C*>(fft_raw);
    const int H = P.n;
    const int64_t l0 = (int64_t)blockIdx.x * LY;
    const int nlines = nl - l0 < LY ? (int)(nl - l0) : LY;
    const LinesX lay{P.len};
    in += l0 * kxp;
    out += l0 * H;
    fft::run_in<1, W>(S, lay, P.p[0], nlines, [&](int line, int pos) {
        return x_inverse_input(in + (int64_t)line * kxp, pos, H, kx, twr);
    });
    for (int i = 1; i + 1 < P.np; ++i) fft::run_mid<1, W>(S, lay, P.p[i], nlines, tw);
    fft::run_out<1, W>(S, lay, P.p[P.np - 1], nlines, tw,
                    [&](int line, int pos, C v) { out[(int64_t)line * H + pos] = v; });
}

// fft_x_inverse with the three components of a grid point side by side, out[row][x] = (c0, c1, c2, 0), the
// layout the interpolation of many nodes reads: a block takes whole rows of all components, the last pass
// stays in shared memory and the rows are written from there, 32 bytes a thread.  FP32 grids only.
template <bool W>
__global__ void __launch_bounds__(kFftThreads, W ? 1 : 2) fft_x_inverse_quad(Plan P, int64_t rows, int LY, int kx, int kxp,
                                                                             const float2* __restrict__ in,
                                                                             float4* __restrict__ out,
                                                                             const float2* __restrict__ tw,
                                                                             const float2* __restrict__ twr) {
    extern __shared__ __align__(16) unsigned char fft_raw[];
    float2* S = reinterpret_cast<float2*>(fft_raw);
    const int H = P.n;
    const int64_t r0 = (int64_t)blockIdx.x * LY;
    const int nr = rows - r0 < LY ? (int)(rows - r0) : LY;
    const LinesX lay{P.len};
    fft::run_in<1, W>(S, lay, P.p[0], 3 * nr, [&](int line, int pos) {
        const int c = line >= 2 * nr ? 2 : line >= nr ? 1 : 0;
        return x_inverse_input(in + (c * rows + r0 + (line - c * nr)) * kxp, pos, H, kx, twr);
    });
    for (int i = 1; i < P.np; ++i) fft::run_mid<1, W>(S, lay, P.p[i], 3 * nr, tw);
    out += r0 * 2 * H;
    for (int idx = threadIdx.x; idx < nr * H; idx += blockDim.x) {
        const int row = idx / H, pos = idx - row * H;
        const float2 a = S[lay.at(row, pos)], b = S[lay.at(nr + row, pos)], c = S[lay.at(2 * nr + row, pos)];
        out[2 * idx] = make_float4(a.x, b.x, c.x, 0.0f);
        out[2 * idx + 1] = make_float4(a.y, b.y, c.y, 0.0f);
    }
}

// ---- y: n1 rows <-> the Ns1 kept ones (row = k_y mod Ns1, k_y = -(Ns1/2) .. (Ns1-1)/2) ----

// Row of the kept modes for position pos of the transform, or -1.
__device__ __forceinline__ int kept_row(int pos, int n, int Ns) {
    if (pos < (Ns + 1) / 2) return pos;
    return pos >= n - Ns / 2 ? pos - (n - Ns) : -1;
}

template <typename T, bool W>
__global__ void __launch_bounds__(kFftThreads, sizeof(T) == 4 && !W ? 2 : 1) fft_y_forward(Plan P, int ltx, int Ns, int kxp,
                                                             typename Cplx<T>::type* __restrict__ g,
                                                             const typename Cplx<T>::type* __restrict__ tw) {
    using C = typename Cplx<T>::type;
    extern __shared__ __align__(16) unsigned char fft_raw[];
    C* S = reinterpret_cast<C*>(fft_raw);
    const int n = P.n;
    const LinesT lay{P.len, ltx};
    g += (int64_t)blockIdx.y * n * kxp + ((int64_t)blockIdx.x << ltx);
    fft::run_in<-1, W>(S, lay, P.p[0], 1 << ltx, [&](int line, int pos) { return g[(int64_t)pos * kxp + line]; });
    for (int i = 1; i + 1 < P.np; ++i) fft::run_mid<-1, W>(S, lay, P.p[i], 1 << ltx, tw);
    fft::run_out<-1, W>(S, lay, P.p[P.np - 1], 1 << ltx, tw, [&](int line, int pos, C v) {
        const int row = kept_row(pos, n, Ns);
        if (row >= 0) g[(int64_t)row * kxp + line] = v;
    });
}

template <typename T, bool W>
__global__ void __launch_bounds__(kFftThreads, sizeof(T) == 4 && !W ? 2 : 1) fft_y_inverse(Plan P, int ltx, int Ns, int kxp,
                                                             typename Cplx<T>::type* __restrict__ g,
                                                             const typename Cplx<T>::type* __restrict__ tw) {
    using C = typename Cplx<T>::type;
    extern __shared__ __align__(16) unsigned char fft_raw[];
    C* S = reinterpret_cast<C*>(fft_raw);
    const int n = P.n;
    const LinesT lay{P.len, ltx};
    g += (int64_t)blockIdx.y * n * kxp + ((int64_t)blockIdx.x << ltx);
    fft::run_in<1, W>(S, lay, P.p[0], 1 << ltx, [&](int line, int pos) {
        const int row = kept_row(pos, n, Ns);
        return row >= 0 ? g[(int64_t)row * kxp + line] : fft::mk((T)0, (T)0);
    });
    for (int i = 1; i + 1 < P.np; ++i) fft::run_mid<1, W>(S, lay, P.p[i], 1 << ltx, tw);
    fft::run_out<1, W>(S, lay, P.p[P.np - 1], 1 << ltx, tw,
                    [&](int line, int pos, C v) { g[(int64_t)pos * kxp + line] = v; });
}

// ---- z and the Fourier-space operators ----

struct ZArgs {
    LRSizes S;
    FourierOp op;
    int kx, kxp, ltx;
    double pref, k0x, k0y, k0z, kmax2, kb_beta2, kb_rc2, kb_c;
    int truncate;
    const double *dec0, *dec1, *dec2, *decE0, *decE1, *decE2;
    double2* uhat;
};

// One block: 2^ltx neighbouring k_x at one kept k_y, all z, all three components.  The arithmetic of
// the operators is FP64 in both forms; only the grids are stored in the grid precision.
template <typename T, bool W>
__global__ void __launch_bounds__(kFftThreads, sizeof(T) == 4 && !W ? 2 : 1) fft_z_operator(Plan P, ZArgs A, typename Cplx<T>::type* __restrict__ g,
                                                              const typename Cplx<T>::type* __restrict__ tw) {
    using C = typename Cplx<T>::type;
    extern __shared__ __align__(16) unsigned char fft_raw[];
    C* S = reinterpret_cast<C*>(fft_raw);
    const LRSizes& Z = A.S;
    const int n = P.n, ltx = A.ltx, TX = 1 << ltx, n1 = Z.n[1];
    const int64_t zs = (int64_t)n1 * A.kxp, cs = zs * n;  // strides of z and of the components
    const int x0 = blockIdx.x << ltx, ry = blockIdx.y;
    const LinesT lay{P.len, ltx};
    g += (int64_t)ry * A.kxp + x0;
    auto ptr = [&](int line, int pos) { return g + (line >> ltx) * cs + pos * zs + (line & (TX - 1)); };
    if (A.op.source == FourierOp::GRID) {
        fft::run_in<-1, W>(S, lay, P.p[0], 3 << ltx, [&](int line, int pos) { return *ptr(line, pos); });
        for (int i = 1; i < P.np; ++i) fft::run_mid<-1, W>(S, lay, P.p[i], 3 << ltx, tw);
    }
    const int ky = ry < (Z.Ns[1] + 1) / 2 ? ry : ry - Z.Ns[1];
    const double kyy = A.k0y * ky;
    const bool zero_y = Z.Ns[1] % 2 == 0 && ky == -(Z.Ns[1] / 2);
    for (int idx = threadIdx.x; idx < n << ltx; idx += blockDim.x) {
        const int tx = idx & (TX - 1), pos = idx >> ltx, ix = x0 + tx;
        const int rz = kept_row(pos, n, Z.Ns[2]);
        double2 r[3] = {{0, 0}, {0, 0}, {0, 0}};
        if (rz >= 0 && ix < A.kx) {
            const int kz = rz < (Z.Ns[2] + 1) / 2 ? rz : rz - Z.Ns[2];
            const double kx = A.k0x * ix, kzz = A.k0z * kz;
            const double k2 = kx * kx + kyy * kyy + kzz * kzz;
            const int64_t u = ((int64_t)rz * Z.Ns[1] + ry) * Z.nkx + ix;
            double2 w[3] = {{0, 0}, {0, 0}, {0, 0}};
            if (A.op.source == FourierOp::GRID) {
                const bool live = !zero_y && !(Z.Ns[2] % 2 == 0 && kz == -(Z.Ns[2] / 2)) && !(A.truncate && k2 > A.kmax2);
                if (live) {
                    const double f = A.pref * (A.dec0[ix] * A.dec1[ry] * A.dec2[rz]);
#pragma unroll
                    for (int c = 0; c < 3; ++c) {
                        const C F = S[lay.at(c * TX + tx, pos)];
                        w[c] = make_double2((double)F.x * f, (double)F.y * f);
                    }
                }
                if (A.op.store)
#pragma unroll
                    for (int c = 0; c < 3; ++c) A.uhat[c * Z.nmodes + u] = w[c];
            } else {
#pragma unroll
                for (int c = 0; c < 3; ++c) w[c] = A.uhat[c * Z.nmodes + u];
            }
            double fk;
            if (A.op.ewald) {
                fk = A.decE0[ix] * A.decE1[ry] * A.decE2[rz];
                if (A.kb_beta2 > 0.0) {
                    // Kaiser-Bessel filter (kaiser_bessel.jl:266-278): beta / sinh(beta) sinh(q) / q,
                    // q = sqrt(beta^2 - k^2 rcut^2), zero beyond k = beta / rcut
                    const double sq = A.kb_beta2 - k2 * A.kb_rc2;
                    if (sq > 0.0) {
                        const double q = sqrt(sq);
                        fk *= A.kb_c * sinh(q) / q;
                    } else {
                        fk = 0.0;
                    }
                }
            } else {
                fk = A.dec0[ix] * A.dec1[ry] * A.dec2[rz];
            }
            if (A.op.quantity != FourierOp::VORTICITY) fk *= k2 == 0.0 ? 0.0 : 1.0 / k2;
            if (A.op.quantity == FourierOp::VELOCITY) {
                // i k x w / k^2 ; (i w).x = -w.y, (i w).y = w.x
                r[0] = make_double2(-(kyy * w[2].y - kzz * w[1].y) * fk, (kyy * w[2].x - kzz * w[1].x) * fk);
                r[1] = make_double2(-(kzz * w[0].y - kx * w[2].y) * fk, (kzz * w[0].x - kx * w[2].x) * fk);
                r[2] = make_double2(-(kx * w[1].y - kyy * w[0].y) * fk, (kx * w[1].x - kyy * w[0].x) * fk);
            } else {
#pragma unroll
                for (int c = 0; c < 3; ++c) r[c] = make_double2(w[c].x * fk, w[c].y * fk);
            }
        }
#pragma unroll
        for (int c = 0; c < 3; ++c) S[lay.at(c * TX + tx, pos)] = fft::mk((T)r[c].x, (T)r[c].y);
    }
    __syncthreads();
    for (int i = 0; i + 1 < P.np; ++i) fft::run_mid<1, W>(S, lay, P.p[i], 3 << ltx, tw);
    fft::run_out<1, W>(S, lay, P.p[P.np - 1], 3 << ltx, tw, [&](int line, int pos, C v) { *ptr(line, pos) = v; });
}

// The kernel of grid type T for a plan's width (wide plans are FP32 only).
#define VPBS_FFT_KERNEL(kernel, T, plan) ((plan).wide && sizeof(T) == 4 ? kernel<T, sizeof(T) == 4> : kernel<T, false>)

template <typename T>
int set_attributes(vpbs_handle* h, const FourierPlan& F) {
    const void* k[] = {(const void*)VPBS_FFT_KERNEL(fft_x_forward, T, F.px), (const void*)VPBS_FFT_KERNEL(fft_x_inverse, T, F.px),
                       (const void*)VPBS_FFT_KERNEL(fft_y_forward, T, F.py), (const void*)VPBS_FFT_KERNEL(fft_y_inverse, T, F.py),
                       (const void*)VPBS_FFT_KERNEL(fft_z_operator, T, F.pz), nullptr};
    if constexpr (sizeof(T) == 4)
        k[5] = F.px.wide ? (const void*)fft_x_inverse_quad<true> : (const void*)fft_x_inverse_quad<false>;
    for (const void* f : k) {
        if (!f) continue;
        // the limit, not this plan's size: the attribute belongs to the function, not to the handle
        int rc = check_cuda(h, cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kFftSmemMost),
                            "FFT kernel shared memory");
        if (rc) return rc;
    }
    return 0;
}

template <typename T>
int run_forward_t(vpbs_handle* h, const void* grid) {
    using C = typename Cplx<T>::type;
    const FourierPlan& F = *h->fplan;
    const LRSizes& S = h->lr;
    C* g = (C*)h->grid_c.p;
    const C* tw = (const C*)h->fft_tw.p;
    const int64_t nl = (int64_t)3 * S.n[2] * S.n[1];
    VPBS_FFT_KERNEL(fft_x_forward, T, F.px)<<<(unsigned)((nl + F.LY - 1) / F.LY), F.sx.threads, F.sx.smem, h->stream>>>(
        F.px, nl, F.LY, F.kx, fft::div_magic(F.kx), F.kxp, (const C*)grid, g, tw, tw + F.twr);
    VPBS_FFT_KERNEL(fft_y_forward, T, F.py)<<<dim3(F.kxp >> F.ltxy, 3 * S.n[2]), F.sy.threads, F.sy.smem, h->stream>>>(F.py, F.ltxy, S.Ns[1], F.kxp,
                                                                                              g, tw);
    h->launches += 2;
    return check_cuda(h, cudaGetLastError(), "forward FFT kernels");
}

template <typename T>
int run_operator_t(vpbs_handle* h, const FourierOp& op) {
    using C = typename Cplx<T>::type;
    const FourierPlan& F = *h->fplan;
    const LRSizes& S = h->lr;
    const vpbs_params& P = h->P;
    ZArgs A;
    A.S = S;
    A.op = op;
    A.kx = F.kx;
    A.kxp = F.kxp;
    A.ltx = F.ltxz;
    const bool kb = P.splitting == VPBS_SPLITTING_KAISER_BESSEL;
    double kmax = INFINITY;
    for (int d = 0; d < 3; ++d) kmax = std::fmin(kmax, 2.0 * kPi * ((P.Ns[d] - 1) / 2) / P.L[d]);
    A.pref = P.Gamma / (P.L[0] * P.L[1] * P.L[2]);
    A.k0x = 2.0 * kPi / P.L[0];
    A.k0y = 2.0 * kPi / P.L[1];
    A.k0z = 2.0 * kPi / P.L[2];
    A.kmax2 = kmax * kmax;
    A.kb_beta2 = kb ? P.kb_beta * P.kb_beta : 0.0;
    A.kb_rc2 = P.rcut * P.rcut;
    A.kb_c = kb ? P.kb_beta / std::sinh(P.kb_beta) : 0.0;
    A.truncate = P.truncate_spherical;
    const double* t = (const double*)h->decx.p;
    A.dec0 = t;
    A.dec1 = A.dec0 + S.nkx;
    A.dec2 = A.dec1 + S.Ns[1];
    A.decE0 = A.dec2 + S.Ns[2];
    A.decE1 = A.decE0 + S.nkx;
    A.decE2 = A.decE1 + S.Ns[1];
    A.uhat = (double2*)h->uhat.p;
    VPBS_FFT_KERNEL(fft_z_operator, T, F.pz)<<<dim3(F.kxp >> F.ltxz, S.Ns[1]), F.sz.threads, F.sz.smem, h->stream>>>(
        F.pz, A, (C*)h->grid_c.p, (const C*)h->fft_tw.p);
    h->launches++;
    return check_cuda(h, cudaGetLastError(), "Fourier kernel");
}

template <typename T>
int run_inverse_t(vpbs_handle* h, void* grid, bool quad) {
    using C = typename Cplx<T>::type;
    const FourierPlan& F = *h->fplan;
    const LRSizes& S = h->lr;
    C* g = (C*)h->grid_c.p;
    const C* tw = (const C*)h->fft_tw.p;
    const int64_t nl = (int64_t)3 * S.n[2] * S.n[1];
    VPBS_FFT_KERNEL(fft_y_inverse, T, F.py)<<<dim3(F.kxp >> F.ltxy, 3 * S.n[2]), F.sy.threads, F.sy.smem, h->stream>>>(F.py, F.ltxy, S.Ns[1], F.kxp,
                                                                                              g, tw);
    if constexpr (sizeof(T) == 4) {
        if (quad) {
            const int64_t rows = (int64_t)S.n[2] * S.n[1];
            auto* kern = F.px.wide ? fft_x_inverse_quad<true> : fft_x_inverse_quad<false>;
            kern<<<(unsigned)((rows + F.LYq - 1) / F.LYq), F.sq.threads, F.sq.smem, h->stream>>>(
                F.px, rows, F.LYq, F.kx, F.kxp, g, (float4*)grid, tw, tw + F.twr);
            h->launches += 2;
            return check_cuda(h, cudaGetLastError(), "inverse FFT kernels");
        }
    }
    VPBS_FFT_KERNEL(fft_x_inverse, T, F.px)<<<(unsigned)((nl + F.LY - 1) / F.LY), F.sx.threads, F.sx.smem, h->stream>>>(
        F.px, nl, F.LY, F.kx, F.kxp, g, (C*)grid, tw, tw + F.twr);
    h->launches += 2;
    return check_cuda(h, cudaGetLastError(), "inverse FFT kernels");
}

}  // namespace
}  // namespace vpbs
