// C ABI of libvpbs.so: handle life cycle, parameter validation, host <-> device staging and
// the compute_on_nodes! orchestration (src/BiotSavart/BiotSavart.jl:395-612).
#include <cmath>
#include <cstring>
#include <algorithm>
#include <new>
#include <string>
#include <atomic>
#include <condition_variable>
#include <functional>
#include <memory>
#include <mutex>
#include <thread>
#include <vector>

#include <unistd.h>

#include "vpbs_internal.cuh"
#include "periodic.cuh"

namespace {
thread_local std::string g_create_error;
}

namespace vpbs {

// Cells r_cut / M wide in y and z (at least 1 per direction); M > 0 splits each cell into G
// x-slabs, up to 4 while the (2M+1)^3-cell neighbourhood stays within 729 slabs.  M = 0 (the
// naive backend) only orders the points (spatial locality).
CellGrid make_cell_grid(const double L[3], double rcut, int M) {
    CellGrid cg{};
    cg.M = M;
    for (int d = 0; d < 3; ++d)
        cg.nc[d] = M > 0 ? (int)std::floor(L[d] * M / rcut) : (int)std::fmax(1.0, std::floor(L[d] / rcut));
    cg.G = 1;
    if (M > 0) {
        const int W = 2 * M + 1;
        cg.G = std::max(1, std::min(4, 729 / (W * W * W)));
        cg.nc[0] *= cg.G;
    }
    cg.ncell = (int64_t)cg.nc[0] * cg.nc[1] * cg.nc[2];
    return cg;
}

int set_error(vpbs_handle* h, int code, const std::string& msg) {
    if (h) h->err = msg;
    else g_create_error = msg;
    return code;
}

int check_cuda(vpbs_handle* h, cudaError_t e, const char* what) {
    if (e == cudaSuccess) return 0;
    return set_error(h, e == cudaErrorMemoryAllocation ? VPBS_ERR_OOM : VPBS_ERR_CUDA,
                     std::string("CUDA error in ") + what + ": " + cudaGetErrorString(e));
}

int ensure(vpbs_handle* h, DevBuf& b, size_t bytes, const char* what) {
    if (bytes == 0) bytes = 8;
    if (b.bytes >= bytes) return 0;
    if (b.p) cudaFree(b.p);
    b.p = nullptr;
    b.bytes = 0;
    cudaError_t e = cudaMalloc(&b.p, bytes);
    if (e != cudaSuccess) {
        b.p = nullptr;
        return set_error(h, VPBS_ERR_OOM, std::string("device allocation of ") + std::to_string(bytes) + " bytes failed (" +
                                              what + "): " + cudaGetErrorString(e));
    }
    b.bytes = bytes;
    return 0;
}

int ensure_pinned(vpbs_handle* h, void** buf, size_t* cap, size_t bytes) {
    if (*cap >= bytes) return 0;
    if (*buf) cudaFreeHost(*buf);
    *buf = nullptr;
    *cap = 0;
    cudaError_t e = cudaHostAlloc(buf, bytes, cudaHostAllocPortable);
    if (e != cudaSuccess) {
        *buf = nullptr;
        return set_error(h, VPBS_ERR_OOM, std::string("pinned host allocation failed: ") + cudaGetErrorString(e));
    }
    *cap = bytes;
    return 0;
}

int ensure_status(vpbs_handle* h) {
    if (h->status_host) return 0;
    void* p = nullptr;
    cudaError_t e = cudaHostAlloc(&p, sizeof(int), cudaHostAllocMapped | cudaHostAllocPortable);
    if (e != cudaSuccess) return set_error(h, VPBS_ERR_OOM, std::string("mapped status word: ") + cudaGetErrorString(e));
    *(volatile int*)p = 0;
    void* d = nullptr;
    e = cudaHostGetDevicePointer(&d, p, 0);
    if (e != cudaSuccess) {
        cudaFreeHost(p);
        return set_error(h, VPBS_ERR_CUDA, std::string("mapped status word: ") + cudaGetErrorString(e));
    }
    h->status_host = (int*)p;
    h->status_dev = (int*)d;
    return 0;
}

int check_status(vpbs_handle* h) {
    if (h->status_host && *(volatile int*)h->status_host) {
        *(volatile int*)h->status_host = 0;
        return set_error(h, VPBS_ERR_TIMEOUT,
                         "a bounded device-side wait gave up (tensor-core spreading); the results of that evaluation are "
                         "not valid");
    }
    return 0;
}

static void free_buf(DevBuf& b) {
    if (b.p) cudaFree(b.p);
    b.p = nullptr;
    b.bytes = 0;
}

static int activate(vpbs_handle* h) { return check_cuda(h, cudaSetDevice(h->device), "cudaSetDevice"); }

// Allocate point-data and output buffers for Np nodes.
static int alloc_points(vpbs_handle* h, int64_t Np) {
    const int64_t Nq = Np * h->K.nquad;
    int rc;
    if ((rc = ensure(h, h->nodes, sizeof(double) * 3 * Np, "nodes"))) return rc;
    if ((rc = ensure(h, h->idx_prev, sizeof(int32_t) * Np, "node_idx_prev"))) return rc;
    if ((rc = ensure(h, h->d1, sizeof(double) * 3 * Np, "derivatives"))) return rc;
    if ((rc = ensure(h, h->d2, sizeof(double) * 3 * Np, "derivatives"))) return rc;
    if ((rc = ensure(h, h->dm, sizeof(double) * Np, "subsegment lengths"))) return rc;
    if ((rc = ensure(h, h->dp, sizeof(double) * Np, "subsegment lengths"))) return rc;
    if ((rc = ensure(h, h->points, sizeof(double) * 3 * Nq, "points"))) return rc;
    if ((rc = ensure(h, h->charges, sizeof(double) * 3 * Nq, "charges"))) return rc;
    if ((rc = ensure(h, h->li_vel, sizeof(double) * 3 * Np, "local integrals"))) return rc;
    if ((rc = ensure(h, h->li_psi, sizeof(double) * 3 * Np, "local integrals"))) return rc;
    if ((rc = ensure(h, h->vel, sizeof(double) * 3 * Np, "velocity"))) return rc;
    if ((rc = ensure(h, h->psi, sizeof(double) * 3 * Np, "streamfunction"))) return rc;
    h->Np = Np;
    h->Nq = Nq;
    return 0;
}

int process_point_charges(vpbs_handle* h) {
    // process_point_charges! of both backends: cell lists (cell_lists.jl:117-127); the long-range
    // rescaling to [0, 2 pi) (longrange.jl:409-471) is folded into the NUFFT kernels.
    int rc = build_cell_lists(h);
    if (rc) return rc;
    h->have_points = true;
    h->have_uhat = false;
    return 0;
}

}  // namespace vpbs

using namespace vpbs;

// Both pair weights in extended precision: of the Kaiser-Bessel series S over x = (xmax / rcut) r, or the Gaussian ones
// where there is none.
static WeightsL pair_weights_l(const KBSeries& S, double xmax) {
    if (S.f.empty()) return gaussian_weights_l;
    return [&S, xmax](long double x, const long double* h, int n, long double* a, long double* g) {
        for (int i = 0; i < n; ++i) kb_weights_series_l(S, (x + h[i]) * S.rcut / xmax, &a[i], &g[i]);
    };
}

extern "C" {

const char* vpbs_last_error(const vpbs_handle* h) { return h ? h->err.c_str() : g_create_error.c_str(); }

int vpbs_create(const vpbs_params* params, vpbs_handle** out) {
    if (!params || !out) return set_error(nullptr, VPBS_ERR_ARG, "null argument to vpbs_create");
    *out = nullptr;
    const vpbs_params& P = *params;
    if (!(P.a > 0) || !std::isfinite(P.Gamma))
        return set_error(nullptr, VPBS_ERR_PARAMS, "vortex core size `a` must be positive and `Gamma` finite");
    if (P.nquad < 1 || P.nquad > kMaxQuad)
        return set_error(nullptr, VPBS_ERR_PARAMS, "nquad must be in 1:16");
    if (P.nquad_near < 0 || P.nquad_near > kMaxQuad)
        return set_error(nullptr, VPBS_ERR_PARAMS, "nquad_near must be in 0:16");
    if (P.lia_segment_fraction > 1.0)
        return set_error(nullptr, VPBS_ERR_PARAMS, "lia_segment_fraction must be in (0, 1]");
    if (P.precision != VPBS_PRECISION_FP64 && P.precision != VPBS_PRECISION_MIXED)
        return set_error(nullptr, VPBS_ERR_PARAMS, "precision must be VPBS_PRECISION_FP64 or VPBS_PRECISION_MIXED");
    if (P.splitting != VPBS_SPLITTING_GAUSSIAN && P.splitting != VPBS_SPLITTING_KAISER_BESSEL)
        return set_error(nullptr, VPBS_ERR_PARAMS, "splitting must be VPBS_SPLITTING_GAUSSIAN or VPBS_SPLITTING_KAISER_BESSEL");
    const bool kb = P.splitting == VPBS_SPLITTING_KAISER_BESSEL;
    if (kb && !(P.kb_beta > 0 && std::isfinite(P.kb_beta)))
        return set_error(nullptr, VPBS_ERR_PARAMS, "KaiserBesselSplitting: beta must be positive and finite");
    if (kb && !(P.kb_rtol > 0 && P.kb_rtol < 1))
        return set_error(nullptr, VPBS_ERR_PARAMS, "KaiserBesselSplitting: rtol must be in (0, 1)");
    const bool open = !kb && !(P.alpha > 0);
    if (P.precision == VPBS_PRECISION_MIXED && open)
        return set_error(nullptr, VPBS_ERR_PARAMS, "the mixed-precision form needs Ewald splitting (alpha > 0)");
    KParams K{};
    K.Gamma = P.Gamma;
    K.a = P.a;
    K.Delta = P.Delta;
    K.kb = kb ? 1 : 0;
    // scale of the weight-table variable x = alpha r (the Gaussian alpha, or the table scale of
    // the Kaiser-Bessel weights)
    K.alpha = open ? 0.0 : (kb ? (P.rcut > 0 ? kb_table_xmax(P.kb_beta) / P.rcut : 0.0) : P.alpha);
    K.open_domain = open ? 1 : 0;
    K.nquad = P.nquad;
    K.nquad_near = P.nquad_near > 0 ? P.nquad_near : P.nquad;
    for (int q = 0; q < P.nquad; ++q) { K.qz[q] = P.quad_zeta[q]; K.qw[q] = P.quad_w[q]; }
    for (int q = 0; q < K.nquad_near; ++q) {
        K.qnz[q] = P.nquad_near > 0 ? P.quad_near_zeta[q] : P.quad_zeta[q];
        K.qnw[q] = P.nquad_near > 0 ? P.quad_near_w[q] : P.quad_w[q];
    }
    K.lia_fraction = P.lia_segment_fraction > 0 ? P.lia_segment_fraction : 0.0;
    // The mixed form always uses the explicit-erf bookkeeping internally (mathematically the same
    // result): pairs on the two local segments are left out of the FP32 pair sum and their
    // long-range part is removed in FP64, so no near-singular pair is ever summed in FP32.
    K.avoid_explicit_erf = P.precision == VPBS_PRECISION_MIXED ? 0 : P.avoid_explicit_erf;
    CellGrid cg{};
    if (open) {
        for (int d = 0; d < 3; ++d) { K.L[d] = 0.0; K.Lh[d] = 0.0; }
        K.rcut = INFINITY;
        K.rcut2 = INFINITY;
        if (!P.avoid_explicit_erf)
            return set_error(nullptr, VPBS_ERR_PARAMS, "avoid_explicit_erf = false requires Ewald splitting");
    } else {
        for (int d = 0; d < 3; ++d) {
            if (!(P.L[d] > 0)) return set_error(nullptr, VPBS_ERR_PARAMS, "periods L must be positive");
            K.L[d] = P.L[d];
            K.Lh[d] = P.L[d] / 2;
        }
        if (!(P.rcut > 0)) return set_error(nullptr, VPBS_ERR_PARAMS, "cutoff distance rcut must be positive");
        const double Lmin = std::fmin(P.L[0], std::fmin(P.L[1], P.L[2]));
        const int M = P.nsubdiv;  // 0 selects the naive (all pairs) short-range backend
        if (M < 0) return set_error(nullptr, VPBS_ERR_PARAMS, "nsubdiv must be >= 0");
        // params.jl:99-106, CellLists.jl:135-147 and naive.jl:8-16
        const double rmax = M > 0 ? (double)M / (2.0 * M + 1.0) * Lmin : 0.5 * Lmin;
        if (P.rcut > rmax)
            return set_error(nullptr, VPBS_ERR_PARAMS,
                             "cutoff distance `rcut = " + std::to_string(P.rcut) + "` is larger than that allowed by the " +
                                 (M > 0 ? "CellListsBackend{" + std::to_string(M) + "} backend (rcut <= M / (2M + 1) * L)"
                                        : std::string("NaiveShortRangeBackend backend (rcut <= L / 2)")));
        if (!(2 * P.rcut <= Lmin))
            return set_error(nullptr, VPBS_ERR_PARAMS, "cutoff distance `rcut` is too large. It must be less than half the cell unit size `L` in each direction");
        K.rcut = P.rcut;
        K.rcut2 = P.rcut * P.rcut;
        cg = make_cell_grid(P.L, P.rcut, M);
        for (int d = 0; d < 3; ++d)
            if (M > 0 && cg.nc[d] < 2 * M + 1 + (d == 0 ? (cg.G - 1) * (2 * M + 1) : 0))
                return set_error(nullptr, VPBS_ERR_PARAMS, "cell lists: the cut-off distance r_cut is too large for periodic padding");
        if (cg.ncell > (int64_t)1 << 30) return set_error(nullptr, VPBS_ERR_PARAMS, "too many cells (rcut too small)");
        if (!(P.sigma > 1.0)) return set_error(nullptr, VPBS_ERR_PARAMS, "NUFFT oversampling factor sigma must be > 1");
        if (P.m < 1 || P.m > kMaxHalfSupport) return set_error(nullptr, VPBS_ERR_PARAMS, "NUFFT half support m must be in 1:8");
        if (P.nufft_kernel != VPBS_NUFFT_ES && P.nufft_kernel != VPBS_NUFFT_KAISER_BESSEL)
            return set_error(nullptr, VPBS_ERR_PARAMS, "nufft_kernel must be VPBS_NUFFT_ES or VPBS_NUFFT_KAISER_BESSEL");
        for (int d = 0; d < 3; ++d) {
            if (P.Ns[d] < 2) return set_error(nullptr, VPBS_ERR_PARAMS, "Ns must be >= 2 in each direction");
            if (vpbs_fft_size(P.Ns[d], P.sigma) < 2 * P.m)
                return set_error(nullptr, VPBS_ERR_PARAMS, "oversampled grid smaller than the NUFFT kernel support");
        }
    }
    vpbs_handle* h = new (std::nothrow) vpbs_handle();
    if (!h) return set_error(nullptr, VPBS_ERR_OOM, "host allocation failed");
    h->P = P;
    h->K = K;
    h->cg = cg;
    h->device = P.device;
    int rc = activate(h);
    if (!rc) rc = check_cuda(h, cudaStreamCreateWithFlags(&h->own_stream, cudaStreamNonBlocking), "cudaStreamCreate");
    if (!rc) rc = check_cuda(h, cudaEventCreateWithFlags(&h->h2d_done, cudaEventDisableTiming), "cudaEventCreate");
    if (!rc) rc = check_cuda(h, cudaStreamCreateWithFlags(&h->aux_stream, cudaStreamNonBlocking), "cudaStreamCreate");
    for (cudaEvent_t* e : {&h->ev_fork, &h->ev_short, &h->ev_long})
        if (!rc) rc = check_cuda(h, cudaEventCreateWithFlags(e, cudaEventDisableTiming), "cudaEventCreate");
    for (int k = 0; k < kStageEvents && !rc; ++k)
        rc = check_cuda(h, cudaEventCreateWithFlags(&h->stage_ev[k], cudaEventDisableTiming), "cudaEventCreate");
    h->stream = h->own_stream;
    if (!rc && !open) rc = longrange_init(h);
    if (!rc && !open) {
        // Ewald weight tables over x = alpha r in [0, alpha rcut]: erfc-based for the Gaussian,
        // fitted to the truncated Chebyshev series for the Kaiser-Bessel kernel
        int ntab = 0;
        std::vector<double> tab;
        KBSeries S;
        if (kb) {
            S = kb_series(P.kb_beta, P.rcut, P.kb_rtol);
            if (S.f.empty()) rc = set_error(h, VPBS_ERR_PARAMS, "KaiserBesselSplitting: Chebyshev series did not converge");
            kb_table_host(S, &ntab, nullptr);
            tab.resize((size_t)2 * ntab * kEwaldNC);
            if (!rc) kb_table_host(S, &ntab, tab.data());
        } else {
            const double xmax = P.alpha * P.rcut;
            ewald_table_host(xmax, &ntab, nullptr);
            tab.resize((size_t)2 * ntab * kEwaldNC);
            ewald_table_host(xmax, &ntab, tab.data());
        }
        // FP32 copy: the leading kEwaldNCf coefficients of each interval, stored after the FP64 table
        std::vector<float> tabf((size_t)2 * ntab * kEwaldNCf);
        for (size_t k = 0; k < (size_t)2 * ntab; ++k)
            for (int n = 0; n < kEwaldNCf; ++n) tabf[k * kEwaldNCf + n] = (float)tab[k * kEwaldNC + n];
        // interleaved copy (erfc coefficient, g coefficient) per degree, stored after the FP32 table
        std::vector<double> tab2((size_t)2 * ntab * kEwaldNC);
        for (size_t k = 0; k < (size_t)ntab; ++k)
            for (int n = 0; n < kEwaldNC; ++n) {
                tab2[2 * (k * kEwaldNC + n)] = tab[k * kEwaldNC + n];
                tab2[2 * (k * kEwaldNC + n) + 1] = tab[(ntab + k) * kEwaldNC + n];
            }
        // FP32 cubic tables of the mixed form's pair kernel, stored after the interleaved table
        const double xmax_c = kb ? kb_table_xmax(P.kb_beta) : P.alpha * P.rcut;
        const int ntab_c = f32_table_size(xmax_c);
        std::vector<float4> tabc((size_t)2 * ntab_c);
        f32_table_host(tab.data(), ntab, xmax_c, tabc.data());
        const size_t bytes_d = sizeof(double) * tab.size(), bytes_f = sizeof(float) * tabf.size();
        const size_t off_c = (2 * bytes_d + bytes_f + 15) / 16 * 16, bytes_c = sizeof(float4) * tabc.size();
        // FP64 tables of the FP64 pair kernel, stored after the FP32 cubic ones (16-byte multiples)
        // unless the FP32 one serves this handle
        const bool f32_pairs = P.precision == VPBS_PRECISION_MIXED && P.nsubdiv > 0 && ntab_c <= kF32TabMax;
        const int ntab_s = f32_pairs ? 0 : tab_s_size(xmax_c);
        std::vector<double> tabs((size_t)2 * ntab_s * kTabSNC);
        if (ntab_s) tab_s_host(pair_weights_l(S, xmax_c), xmax_c, tabs.data());
        const size_t off_s = off_c + bytes_c, bytes_s = sizeof(double) * tabs.size();
        if (!rc) rc = ensure(h, h->ewald_tab, off_s + bytes_s, "Ewald tables");
        if (!rc && ntab_s)
            rc = check_cuda(h, cudaMemcpy((char*)h->ewald_tab.p + off_s, tabs.data(), bytes_s, cudaMemcpyHostToDevice),
                            "copy Ewald tables");
        if (!rc)
            rc = check_cuda(h, cudaMemcpy((char*)h->ewald_tab.p + off_c, tabc.data(), bytes_c, cudaMemcpyHostToDevice),
                            "copy Ewald tables");
        if (!rc)
            rc = check_cuda(h, cudaMemcpy((char*)h->ewald_tab.p + bytes_d + bytes_f, tab2.data(), bytes_d,
                                          cudaMemcpyHostToDevice), "copy Ewald tables");
        if (!rc)
            rc = check_cuda(h, cudaMemcpy(h->ewald_tab.p, tab.data(), bytes_d, cudaMemcpyHostToDevice), "copy Ewald tables");
        if (!rc)
            rc = check_cuda(h, cudaMemcpy((char*)h->ewald_tab.p + bytes_d, tabf.data(), bytes_f, cudaMemcpyHostToDevice),
                            "copy Ewald tables");
        h->K.ewald_tab = (const double*)h->ewald_tab.p;
        h->K.ewald_tab_f = (const float*)((const char*)h->ewald_tab.p + bytes_d);
        h->K.ewald_tab2 = (const double2*)((const char*)h->ewald_tab.p + bytes_d + bytes_f);
        h->K.ewald_ntab = ntab;
        h->K.tab_c = (const float4*)((const char*)h->ewald_tab.p + off_c);
        h->K.ntab_c = ntab_c;
        h->K.tab_s = (const double*)((const char*)h->ewald_tab.p + off_s);
        h->K.ntab_s = ntab_s;
        // streamfunction factor of a uniform background vorticity (BiotSavart.jl:255-286): 1 / (4 alpha^2)
        // for the Gaussian splitting (gaussian.jl:241); int_0^rcut r^2 f(r) dr / 2 for the Kaiser-Bessel one
        // (kaiser_bessel.jl:160-165, 280), with f(r) = beta / (rcut sinh beta) I0(beta sqrt(1 - r^2 / rcut^2)),
        // by 64-point Gauss-Legendre quadrature (the integrand is analytic in r^2)
        if (kb) {
            std::vector<double> gx, gw;
            gauss_legendre(64, gx, gw);
            double acc = 0.0;
            const double rc_ = P.rcut, b_ = P.kb_beta;
            for (int q = 0; q < 64; ++q) {
                const double z = 0.5 * (gx[q] + 1.0), w = 0.5 * gw[q], r = z * rc_, u = r / rc_;
                const double f = b_ / (rc_ * std::sinh(b_)) * std::cyl_bessel_i(0.0, b_ * std::sqrt(std::fmax(0.0, 1.0 - u * u)));
                acc += w * rc_ * r * r * f;
            }
            h->bg_factor = acc / 2.0;
        } else {
            h->bg_factor = 1.0 / (4.0 * P.alpha * P.alpha);
        }
    }
    if (rc) {
        g_create_error = h->err;
        vpbs_destroy(h);
        return rc;
    }
    *out = h;
    return 0;
}

int vpbs_destroy(vpbs_handle* h) {
    if (!h) return 0;
    cudaSetDevice(h->device);
    if (h->stream) cudaStreamSynchronize(h->stream);
    longrange_free(h);
    DevBuf* bufs[] = {&h->nodes_in, &h->offsets, &h->fil_of_node, &h->knots, &h->coefs, &h->dcoef1, &h->dcoef2,
                      &h->spline_scratch, &h->nodes, &h->idx_prev, &h->d1, &h->d2, &h->dm, &h->dp, &h->points,
                      &h->charges, &h->li_vel, &h->li_psi, &h->src_cell, &h->cell_start, &h->cell_counts, &h->src_sorted,
                      &h->src_seg, &h->src_f32, &h->dst_order, &h->counters,
                      &h->grid_r, &h->grid_c, &h->grid_c2, &h->uhat, &h->decx, &h->decy, &h->decz, &h->nodes_lr,
                      &h->vel, &h->psi, &h->spread_bin, &h->spread_counts, &h->spread_start, &h->binned,
                      &h->spread_foot, &h->tc_counts, &h->tc_start, &h->tc_rec, &h->peer_in, &h->ewald_tab, &h->scan_tmp, &h->scan_tmp_lr, &h->rk_vs, &h->rk_tmp,
                      &h->aos_out, &h->fil_off, &h->fft_tw, &h->grid64};
    for (DevBuf* b : bufs) free_buf(*b);
    if (h->pin_in) cudaFreeHost(h->pin_in);
    if (h->status_host) cudaFreeHost(h->status_host);
    if (h->xfer_done) cudaEventDestroy(h->xfer_done);
    if (h->pin_out) cudaFreeHost(h->pin_out);
    if (h->h2d_done) cudaEventDestroy(h->h2d_done);
    if (h->aux_stream) cudaStreamSynchronize(h->aux_stream);
    for (int k = 0; k < kStageEvents; ++k)
        if (h->stage_ev[k]) cudaEventDestroy(h->stage_ev[k]);
    for (cudaEvent_t e : {h->ev_fork, h->ev_short, h->ev_long})
        if (e) cudaEventDestroy(e);
    if (h->aux_stream) cudaStreamDestroy(h->aux_stream);
    if (h->tev[0][0][0])
        for (int s = 0; s < ST_COUNT; ++s)
            for (int k = 0; k < 4; ++k)
                for (int e = 0; e < 2; ++e) cudaEventDestroy(h->tev[s][k][e]);
    if (h->own_stream) cudaStreamDestroy(h->own_stream);
    delete h;
    return 0;
}

int vpbs_set_stream(vpbs_handle* h, void* stream) {
    if (!h) return VPBS_ERR_ARG;
    h->stream = stream ? (cudaStream_t)stream : h->own_stream;
    return 0;
}

}  // extern "C"

namespace vpbs {

// Copies `n` blocks (dst[k] <- src[k], bytes[k]) with up to 8 host threads (large inputs only):
// the staging of filament lists into and out of pinned memory is bound by host memory copies.
// Host copy threads: a pool created on first use (and again in a forked child, whose parent's threads
// do not exist there; the old pool is left alone), running the pieces of one job at a time with the
// calling thread taking part.  Each job has its own counters, so a thread still leaving an old job never
// takes a piece of the next one.
namespace copy_threads {
struct CopyJob {
    std::function<void(int64_t)> fn;
    int64_t n = 0;
    std::atomic<int64_t> next{0}, done{0};
    std::mutex m;
    std::condition_variable cv;
};

struct CopyPool {
    std::mutex submit, m;
    std::condition_variable cv;
    std::shared_ptr<CopyJob> job;
    uint64_t gen = 0;
    pid_t pid;
    explicit CopyPool(int nthreads) : pid(getpid()) {
        for (int i = 0; i < nthreads; ++i) std::thread([this] { loop(); }).detach();
    }
    static void work(CopyJob& j) {
        int64_t i;
        while ((i = j.next.fetch_add(1)) < j.n) {
            j.fn(i);
            if (j.done.fetch_add(1) + 1 == j.n) {
                std::lock_guard<std::mutex> lk(j.m);
                j.cv.notify_all();
            }
        }
    }
    void loop() {
        uint64_t seen = 0;
        for (;;) {
            std::shared_ptr<CopyJob> j;
            {
                std::unique_lock<std::mutex> lk(m);
                cv.wait(lk, [&] { return gen != seen; });
                seen = gen;
                j = job;
            }
            if (j) work(*j);
        }
    }
    void run(int64_t n, std::function<void(int64_t)> fn) {
        std::lock_guard<std::mutex> one(submit);
        auto j = std::make_shared<CopyJob>();
        j->fn = std::move(fn);
        j->n = n;
        {
            std::lock_guard<std::mutex> lk(m);
            job = j;
            ++gen;
        }
        cv.notify_all();
        work(*j);
        std::unique_lock<std::mutex> lk(j->m);
        j->cv.wait(lk, [&] { return j->done.load() == j->n; });
    }
};

CopyPool& copy_pool() {
    static std::mutex mu;
    static CopyPool* pool = nullptr;
    std::lock_guard<std::mutex> lk(mu);
    if (!pool || pool->pid != getpid()) {
        const unsigned hw = std::max(1u, std::thread::hardware_concurrency());
        pool = new CopyPool((int)std::min(7u, hw > 1 ? hw - 1 : 1u));  // lives until the process ends
    }
    return *pool;
}
}  // namespace copy_threads

// Host copies of n blocks, split into pieces of about 1 MB run on the copy pool (blocks below 2 MB
// in total are copied by the calling thread).
static void parallel_copies(int64_t n, void* const* dst, const void* const* src, const size_t* bytes) {
    constexpr size_t kPiece = (size_t)1 << 20;
    size_t total = 0;
    for (int64_t k = 0; k < n; ++k) total += bytes[k];
    if (total < 2 * kPiece) {
        for (int64_t k = 0; k < n; ++k) std::memcpy(dst[k], src[k], bytes[k]);
        return;
    }
    struct Piece {
        char* d;
        const char* s;
        size_t b;
    };
    std::vector<Piece> pieces;
    for (int64_t k = 0; k < n; ++k) {  // large blocks split into pieces
        if (bytes[k] >= kPiece) {
            for (size_t o = 0; o < bytes[k]; o += kPiece)
                pieces.push_back({(char*)dst[k] + o, (const char*)src[k] + o, std::min(kPiece, bytes[k] - o)});
        } else {
            pieces.push_back({(char*)dst[k], (const char*)src[k], bytes[k]});
        }
    }
    // merge runs of small pieces so that each job item copies about kPiece bytes
    std::vector<std::pair<size_t, size_t>> items;  // [first piece, end piece)
    for (size_t i = 0; i < pieces.size();) {
        size_t j = i, acc = 0;
        while (j < pieces.size() && (j == i || acc + pieces[j].b <= kPiece)) acc += pieces[j++].b;
        items.push_back({i, j});
        i = j;
    }
    copy_threads::copy_pool().run((int64_t)items.size(), [&](int64_t it) {
        for (size_t p = items[it].first; p < items[it].second; ++p) std::memcpy(pieces[p].d, pieces[p].s, pieces[p].b);
    });
}

// Shared tail of the filament entry points: offsets (host) are staged in pin_in[0..), the nodes
// either already sit in pin_in after the offsets (host input) or in device memory (d_nodes).
static int set_filaments_staged(vpbs_handle* h, int64_t nfil, const int64_t* offsets, const double* d_nodes) {
    int rc;
    const int64_t Np = offsets[nfil];
    const size_t bytes_off = sizeof(int64_t) * (nfil + 1);
    if ((rc = check_cuda(h, cudaMemcpyAsync(h->offsets.p, h->pin_in, bytes_off, cudaMemcpyHostToDevice, h->stream),
                         "H2D offsets")))
        return rc;
    if (!d_nodes) {
        if ((rc = check_cuda(h, cudaMemcpyAsync(h->nodes_in.p, (char*)h->pin_in + bytes_off, sizeof(double) * 3 * Np,
                                                cudaMemcpyHostToDevice, h->stream), "H2D nodes")))
            return rc;
        d_nodes = (const double*)h->nodes_in.p;
    }
    if ((rc = check_cuda(h, cudaEventRecord(h->h2d_done, h->stream), "event record"))) return rc;
    if (h->have_fil_offsets && h->nfil_off != nfil)
        return set_error(h, VPBS_ERR_ARG, "end-to-end offsets were set for " + std::to_string(h->nfil_off) +
                                              " filaments, not " + std::to_string(nfil));
    h->nfil = nfil;
    h->host_offsets.assign(offsets, offsets + nfil + 1);
    int64_t nmax = 0;
    for (int64_t f = 0; f < nfil; ++f) nmax = std::max<int64_t>(nmax, offsets[f + 1] - offsets[f]);
    h->nmax = nmax;
    h->have_filaments = true;
    if ((rc = geometry_from_filaments(h, nfil, (const int64_t*)h->offsets.p, d_nodes, nmax))) return rc;
    h->li_valid = h->K.lia_fraction > 0;
    return process_point_charges(h);
}

// Checks, allocation and pinned staging common to both filament entry points; on success the
// offsets are in pin_in and room for 3 Np host doubles follows them when host_nodes.
static int prepare_filaments(vpbs_handle* h, int64_t nfil, const int64_t* offsets, bool host_nodes) {
    if (offsets[0] != 0) return set_error(h, VPBS_ERR_ARG, "offsets[0] must be 0");
    for (int64_t f = 0; f < nfil; ++f)
        if (offsets[f + 1] - offsets[f] < 5)
            return set_error(h, VPBS_ERR_ARG, "each filament needs at least 5 nodes (quintic splines)");
    const int64_t Np = offsets[nfil];
    if (Np * h->K.nquad >= ((int64_t)1 << 31)) return set_error(h, VPBS_ERR_ARG, "too many quadrature points");
    int rc;
    if ((rc = activate(h))) return rc;
    if ((rc = alloc_points(h, Np))) return rc;
    if ((rc = ensure(h, h->offsets, sizeof(int64_t) * (nfil + 1), "offsets"))) return rc;
    const size_t bytes_off = sizeof(int64_t) * (nfil + 1);
    const size_t bytes_nodes = host_nodes ? sizeof(double) * 3 * Np : 0;
    if (host_nodes && (rc = ensure(h, h->nodes_in, bytes_nodes, "input nodes"))) return rc;
    if ((rc = check_cuda(h, cudaEventSynchronize(h->h2d_done), "event sync"))) return rc;
    if ((rc = ensure_pinned(h, &h->pin_in, &h->pin_in_bytes, bytes_off + bytes_nodes))) return rc;
    if (offsets != (const int64_t*)h->pin_in) std::memcpy(h->pin_in, offsets, bytes_off);
    return 0;
}

}  // namespace vpbs

extern "C" {

int vpbs_set_filaments(vpbs_handle* h, int64_t nfil, const int64_t* offsets, const double* nodes_xyz, int32_t on_device) {
    if (!h) return VPBS_ERR_ARG;
    if (nfil < 1 || !offsets || !nodes_xyz) return set_error(h, VPBS_ERR_ARG, "vpbs_set_filaments: bad arguments");
    int rc;
    if ((rc = prepare_filaments(h, nfil, offsets, !on_device))) return rc;
    if (on_device) return set_filaments_staged(h, nfil, offsets, nodes_xyz);
    // pinned staging in chunks: the host copy of chunk k overlaps the transfer of chunk k-1
    const size_t bytes_off = sizeof(int64_t) * (nfil + 1);
    const size_t total = sizeof(double) * 3 * offsets[nfil];
    const size_t chunk = std::max<size_t>(kStageChunk, (total / kStageEvents + 7) & ~(size_t)7);
    char* pin = (char*)h->pin_in + bytes_off;
    for (size_t o = 0; o < total; o += chunk) {
        const size_t n = std::min(chunk, total - o);
        const void* src[1] = {(const char*)nodes_xyz + o};
        void* dst[1] = {pin + o};
        parallel_copies(1, dst, src, &n);
        if ((rc = check_cuda(h, cudaMemcpyAsync((char*)h->nodes_in.p + o, pin + o, n, cudaMemcpyHostToDevice, h->stream),
                             "H2D nodes")))
            return rc;
    }
    return set_filaments_staged(h, nfil, offsets, (const double*)h->nodes_in.p);
}

int vpbs_set_filament_offsets(vpbs_handle* h, int64_t nfil, const double* offsets_xyz) {
    if (!h) return VPBS_ERR_ARG;
    if (nfil < 0 || (nfil > 0 && !offsets_xyz)) return set_error(h, VPBS_ERR_ARG, "vpbs_set_filament_offsets: bad arguments");
    int rc;
    if ((rc = activate(h))) return rc;
    double sum[3] = {0.0, 0.0, 0.0};
    bool any = false;
    for (int64_t f = 0; f < nfil; ++f)
        for (int d = 0; d < 3; ++d) {
            const double v = offsets_xyz[3 * f + d];
            if (!std::isfinite(v)) return set_error(h, VPBS_ERR_ARG, "vpbs_set_filament_offsets: non-finite offset");
            any = any || v != 0.0;
            sum[d] += v;
        }
    // the geometry kernels of earlier calls may still read the previous offsets
    if ((rc = check_cuda(h, cudaStreamSynchronize(h->stream), "stream sync"))) return rc;
    if (any) {
        if ((rc = ensure(h, h->fil_off, sizeof(double) * 3 * nfil, "filament offsets"))) return rc;
        if ((rc = check_cuda(h, cudaMemcpy(h->fil_off.p, offsets_xyz, sizeof(double) * 3 * nfil, cudaMemcpyHostToDevice),
                             "H2D filament offsets")))
            return rc;
    }
    h->have_fil_offsets = any;
    h->nfil_off = nfil;
    for (int d = 0; d < 3; ++d) h->offset_sum[d] = any ? sum[d] : 0.0;
    return 0;
}

int vpbs_stage_filaments(vpbs_handle* h, int64_t nfil, int64_t Np, int64_t** offsets, double** nodes) {
    if (!h) return VPBS_ERR_ARG;
    if (nfil < 1 || Np < 0 || !offsets || !nodes) return set_error(h, VPBS_ERR_ARG, "vpbs_stage_filaments: bad arguments");
    int rc;
    if ((rc = activate(h))) return rc;
    if ((rc = check_cuda(h, cudaEventSynchronize(h->h2d_done), "event sync"))) return rc;
    const size_t bytes_off = sizeof(int64_t) * (nfil + 1);
    if ((rc = ensure_pinned(h, &h->pin_in, &h->pin_in_bytes, bytes_off + sizeof(double) * 3 * Np))) return rc;
    *offsets = (int64_t*)h->pin_in;
    *nodes = (double*)((char*)h->pin_in + bytes_off);
    return 0;
}

int vpbs_set_staged_filaments(vpbs_handle* h, int64_t nfil) {
    if (!h) return VPBS_ERR_ARG;
    if (nfil < 1 || !h->pin_in) return set_error(h, VPBS_ERR_STATE, "vpbs_set_staged_filaments: nothing staged");
    const int64_t* offsets = (const int64_t*)h->pin_in;
    if ((size_t)(sizeof(int64_t) * (nfil + 1)) > h->pin_in_bytes ||
        sizeof(int64_t) * (nfil + 1) + sizeof(double) * 3 * (size_t)std::max<int64_t>(offsets[nfil], 0) > h->pin_in_bytes)
        return set_error(h, VPBS_ERR_ARG, "vpbs_set_staged_filaments: staged sizes exceed the staging buffer");
    int rc;
    if ((rc = prepare_filaments(h, nfil, offsets, true))) return rc;
    return set_filaments_staged(h, nfil, offsets, nullptr);
}

int vpbs_set_filament_list(vpbs_handle* h, int64_t nfil, const double* const* nodes, const int64_t* counts) {
    if (!h) return VPBS_ERR_ARG;
    if (nfil < 1 || !nodes || !counts) return set_error(h, VPBS_ERR_ARG, "vpbs_set_filament_list: bad arguments");
    std::vector<int64_t> offsets(nfil + 1, 0);
    for (int64_t f = 0; f < nfil; ++f) {
        if (!nodes[f]) return set_error(h, VPBS_ERR_ARG, "vpbs_set_filament_list: null filament");
        offsets[f + 1] = offsets[f] + counts[f];
    }
    int rc;
    if ((rc = prepare_filaments(h, nfil, offsets.data(), true))) return rc;
    double* base = (double*)((char*)h->pin_in + sizeof(int64_t) * (nfil + 1));
    std::vector<void*> dst(nfil);
    std::vector<const void*> src(nfil);
    std::vector<size_t> bytes(nfil);
    for (int64_t f = 0; f < nfil; ++f) {
        dst[f] = base + 3 * offsets[f];
        src[f] = nodes[f];
        bytes[f] = sizeof(double) * 3 * counts[f];
    }
    parallel_copies(nfil, dst.data(), src.data(), bytes.data());
    return set_filaments_staged(h, nfil, offsets.data(), nullptr);
}

int vpbs_set_points(vpbs_handle* h, int64_t Np, vpbs_cvec3 nodes, const int32_t* node_idx_prev, vpbs_cvec3 deriv1,
                    vpbs_cvec3 deriv2, const double* delta_minus, const double* delta_plus, vpbs_cvec3 points,
                    vpbs_cvec3 charges) {
    if (!h) return VPBS_ERR_ARG;
    if (Np < 1 || !node_idx_prev || !delta_minus || !delta_plus || !nodes.x || !nodes.y || !nodes.z || !deriv1.x ||
        !deriv1.y || !deriv1.z || !deriv2.x || !deriv2.y || !deriv2.z || !points.x || !points.y || !points.z ||
        !charges.x || !charges.y || !charges.z)
        return set_error(h, VPBS_ERR_ARG, "vpbs_set_points: null pointer or empty point data");
    if (Np * h->K.nquad >= ((int64_t)1 << 31)) return set_error(h, VPBS_ERR_ARG, "too many quadrature points");
    int rc;
    if ((rc = activate(h))) return rc;
    if ((rc = alloc_points(h, Np))) return rc;
    const int64_t Nq = h->Nq;
    const size_t nd = sizeof(double);
    // layout of the staging buffer: 3Np nodes | 3Np d1 | 3Np d2 | Np dm | Np dp | 3Nq points | 3Nq charges | Np idx
    const size_t total = nd * (11 * Np + 6 * Nq) + sizeof(int32_t) * Np;
    if ((rc = check_cuda(h, cudaEventSynchronize(h->h2d_done), "event sync"))) return rc;
    if ((rc = ensure_pinned(h, &h->pin_in, &h->pin_in_bytes, total))) return rc;
    double* s = (double*)h->pin_in;
    const double* vsrc[] = {nodes.x, nodes.y, nodes.z, deriv1.x, deriv1.y, deriv1.z, deriv2.x, deriv2.y, deriv2.z,
                            delta_minus, delta_plus};
    for (int k = 0; k < 11; ++k) std::memcpy(s + k * Np, vsrc[k], nd * Np);
    const double* qsrc[] = {points.x, points.y, points.z, charges.x, charges.y, charges.z};
    for (int k = 0; k < 6; ++k) std::memcpy(s + 11 * Np + k * Nq, qsrc[k], nd * Nq);
    int32_t* sidx = (int32_t*)(s + 11 * Np + 6 * Nq);
    for (int64_t i = 0; i < Np; ++i) {
        int32_t v = node_idx_prev[i] - 1;  // reference indices are 1-based
        if (v < 0 || v >= Np) return set_error(h, VPBS_ERR_ARG, "node_idx_prev out of range");
        sidx[i] = v;
    }
    struct { void* dst; const void* src; size_t n; } cp[] = {
        {h->nodes.p, s, nd * 3 * Np},          {h->d1.p, s + 3 * Np, nd * 3 * Np},
        {h->d2.p, s + 6 * Np, nd * 3 * Np},    {h->dm.p, s + 9 * Np, nd * Np},
        {h->dp.p, s + 10 * Np, nd * Np},       {h->points.p, s + 11 * Np, nd * 3 * Nq},
        {h->charges.p, s + 11 * Np + 3 * Nq, nd * 3 * Nq}, {h->idx_prev.p, sidx, sizeof(int32_t) * Np}};
    for (auto& c : cp)
        if ((rc = check_cuda(h, cudaMemcpyAsync(c.dst, c.src, c.n, cudaMemcpyHostToDevice, h->stream), "H2D point data")))
            return rc;
    if ((rc = check_cuda(h, cudaEventRecord(h->h2d_done, h->stream), "event record"))) return rc;
    h->dm_pending = false;
    h->li_valid = false;  // add_local_integrals! stays with the caller in the point-data contract
    h->have_filaments = false;  // point data without a filament layout: no time stepping
    return process_point_charges(h);
}

int vpbs_compute(vpbs_handle* h, int32_t fields, int32_t lia_mode, int32_t shortrange, int32_t longrange,
                 double integration_cutoff) {
    if (!h) return VPBS_ERR_ARG;
    if (fields < 1 || fields > 3) return set_error(h, VPBS_ERR_ARG, "fields must be VELOCITY and/or STREAMFUNCTION");
    if (lia_mode < 0 || lia_mode > 2) return set_error(h, VPBS_ERR_ARG, "bad LIA mode");
    if (!h->have_points) return set_error(h, VPBS_ERR_STATE, "no point data: call vpbs_set_filaments or vpbs_set_points first");
    int rc;
    if ((rc = activate(h))) return rc;
    const int64_t Np = h->Np;
    // the local term is the first to write the outputs; without the short range they start from zero
    if ((fields & VPBS_VELOCITY) && !shortrange)
        if ((rc = check_cuda(h, cudaMemsetAsync(h->vel.p, 0, sizeof(double) * 3 * Np, h->stream), "memset"))) return rc;
    if ((fields & VPBS_STREAMFUNCTION) && !shortrange)
        if ((rc = check_cuda(h, cudaMemsetAsync(h->psi.p, 0, sizeof(double) * 3 * Np, h->stream), "memset"))) return rc;
    const bool with_long = longrange && lia_mode != VPBS_LIA_ONLY && !h->K.open_domain;
    // The long range (spread, FFTs, Fourier operators) runs on the auxiliary stream while the
    // short range runs on the main stream; only the long-range interpolation, which adds into
    // the same outputs, waits for the short range.  The main stream then joins.  With stage
    // timing on, everything runs in order on the main stream so that each stage is timed alone.
    cudaStream_t main = h->stream;
    const bool fork = with_long && !h->timing;
    if (fork) {
        if ((rc = check_cuda(h, cudaEventRecord(h->ev_fork, main), "fork"))) return rc;
        if ((rc = check_cuda(h, cudaStreamWaitEvent(h->aux_stream, h->ev_fork, 0), "fork"))) return rc;
    }
    if (shortrange) {
        const bool pairs = lia_mode != VPBS_LIA_ONLY;
        KParams saved = h->K;
        if (!h->li_valid) h->K.lia_fraction = 0.0;
        rc = local_and_self(h, fields, lia_mode, pairs ? 1 : 0, integration_cutoff);
        h->K = saved;
        if (rc) return rc;
        if (pairs)
            if ((rc = pair_interactions(h, fields))) return rc;
    }
    if (with_long && !fork) {
        if ((rc = longrange_compute(h, fields))) return rc;
    } else if (with_long) {
        if ((rc = check_cuda(h, cudaEventRecord(h->ev_short, main), "short done"))) return rc;
        h->stream = h->aux_stream;
        h->interp_wait = h->ev_short;
        rc = longrange_compute(h, fields);
        h->interp_wait = nullptr;
        h->stream = main;
        if (rc) return rc;
        if ((rc = check_cuda(h, cudaEventRecord(h->ev_long, h->aux_stream), "long done"))) return rc;
        if ((rc = check_cuda(h, cudaStreamWaitEvent(main, h->ev_long, 0), "join"))) return rc;
    }
    h->last_fields = fields;
    return 0;
}

}  // extern "C"

namespace vpbs {
__global__ void add_field_kernel(int64_t n, const double* __restrict__ src, double* __restrict__ dst) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) dst[i] += src[i];
}

// SoA [3][Np] -> AoS [Np][3] (the node-order layout of the host output arrays)
__global__ void soa_to_aos_kernel(int64_t Np, const double* __restrict__ src, double* __restrict__ dst) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < 3 * Np) dst[i] = src[(i % 3) * Np + i / 3];
}
}  // namespace vpbs

extern "C" {

int vpbs_add_field(vpbs_handle* dst, vpbs_handle* src, int32_t fields) {
    if (!dst || !src || dst == src) return VPBS_ERR_ARG;
    if (fields < 1 || fields > 3) return set_error(dst, VPBS_ERR_ARG, "fields must be VELOCITY and/or STREAMFUNCTION");
    if (dst->Np != src->Np || dst->Np < 1) return set_error(dst, VPBS_ERR_ARG, "vpbs_add_field: node counts differ");
    if ((dst->last_fields & fields) != fields || (src->last_fields & fields) != fields)
        return set_error(dst, VPBS_ERR_STATE, "vpbs_add_field: field was not computed on both handles");
    int rc;
    // the source's work is done before the destination's stream reads it
    if ((rc = activate(src))) return rc;
    if (!src->xfer_done && (rc = check_cuda(src, cudaEventCreateWithFlags(&src->xfer_done, cudaEventDisableTiming),
                                            "cudaEventCreate")))
        return rc;
    if ((rc = check_cuda(src, cudaEventRecord(src->xfer_done, src->stream), "event record"))) return rc;
    if ((rc = activate(dst))) return rc;
    if ((rc = check_cuda(dst, cudaStreamWaitEvent(dst->stream, src->xfer_done, 0), "stream wait"))) return rc;
    const int64_t n = 3 * dst->Np;
    const size_t bytes = sizeof(double) * n;
    for (int32_t f = VPBS_VELOCITY; f <= VPBS_STREAMFUNCTION; f <<= 1) {
        if (!(fields & f)) continue;
        const double* s = (const double*)(f == VPBS_VELOCITY ? src->vel.p : src->psi.p);
        double* d = (double*)(f == VPBS_VELOCITY ? dst->vel.p : dst->psi.p);
        if (src->device != dst->device) {
            // another GPU: one peer copy into this GPU's memory, then the addition reads local memory
            if ((rc = ensure(dst, dst->peer_in, bytes, "peer field"))) return rc;
            if ((rc = check_cuda(dst, cudaMemcpyPeerAsync(dst->peer_in.p, dst->device, s, src->device, bytes, dst->stream),
                                 "peer copy")))
                return rc;
            s = (const double*)dst->peer_in.p;
        }
        add_field_kernel<<<grid_for(n, 256), 256, 0, dst->stream>>>(n, s, d);
        dst->launches++;
        if ((rc = check_cuda(dst, cudaGetLastError(), "add field kernel"))) return rc;
    }
    return 0;
}

static int fetch_soa(vpbs_handle* h, int32_t field, const double** out) {
    if (field != VPBS_VELOCITY && field != VPBS_STREAMFUNCTION) return set_error(h, VPBS_ERR_ARG, "bad field");
    if (!(h->last_fields & field)) return set_error(h, VPBS_ERR_STATE, "field was not computed");
    int rc;
    if ((rc = activate(h))) return rc;
    const size_t bytes = sizeof(double) * 3 * h->Np;
    if ((rc = ensure_pinned(h, &h->pin_out, &h->pin_out_bytes, bytes))) return rc;
    const void* src = field == VPBS_VELOCITY ? h->vel.p : h->psi.p;
    if ((rc = check_cuda(h, cudaMemcpyAsync(h->pin_out, src, bytes, cudaMemcpyDeviceToHost, h->stream), "D2H"))) return rc;
    if ((rc = check_cuda(h, cudaStreamSynchronize(h->stream), "stream sync"))) return rc;
    if ((rc = check_status(h))) return rc;
    *out = (const double*)h->pin_out;
    return 0;
}

// Device transpose of a computed field to AoS, D2H into pinned memory; returns the pinned copy.
static int fetch_aos(vpbs_handle* h, int32_t field, const double** out) {
    if (field != VPBS_VELOCITY && field != VPBS_STREAMFUNCTION) return set_error(h, VPBS_ERR_ARG, "bad field");
    if (!(h->last_fields & field)) return set_error(h, VPBS_ERR_STATE, "field was not computed");
    int rc;
    if ((rc = activate(h))) return rc;
    const int64_t Np = h->Np;
    const size_t bytes = sizeof(double) * 3 * Np;
    if ((rc = ensure(h, h->aos_out, bytes, "AoS output staging"))) return rc;
    if ((rc = ensure_pinned(h, &h->pin_out, &h->pin_out_bytes, bytes))) return rc;
    soa_to_aos_kernel<<<grid_for(3 * Np, 256), 256, 0, h->stream>>>(
        Np, (const double*)(field == VPBS_VELOCITY ? h->vel.p : h->psi.p), (double*)h->aos_out.p);
    h->launches++;
    if ((rc = check_cuda(h, cudaGetLastError(), "AoS kernel"))) return rc;
    if ((rc = check_cuda(h, cudaMemcpyAsync(h->pin_out, h->aos_out.p, bytes, cudaMemcpyDeviceToHost, h->stream), "D2H")))
        return rc;
    if ((rc = check_cuda(h, cudaStreamSynchronize(h->stream), "stream sync"))) return rc;
    if ((rc = check_status(h))) return rc;
    *out = (const double*)h->pin_out;
    return 0;
}

int vpbs_get(vpbs_handle* h, int32_t field, double* out_xyz, int32_t accumulate) {
    if (!h) return VPBS_ERR_ARG;
    if (!out_xyz) return set_error(h, VPBS_ERR_ARG, "null output");
    if (accumulate) {
        const double* s;
        int rc = fetch_aos(h, field, &s);
        if (rc) return rc;
        const int64_t n = 3 * h->Np;
        for (int64_t i = 0; i < n; ++i) out_xyz[i] += s[i];
        return 0;
    }
    // device transpose, then the transfer in chunks: the host copy of chunk k overlaps the
    // transfer of chunk k+1
    if (field != VPBS_VELOCITY && field != VPBS_STREAMFUNCTION) return set_error(h, VPBS_ERR_ARG, "bad field");
    if (!(h->last_fields & field)) return set_error(h, VPBS_ERR_STATE, "field was not computed");
    int rc;
    if ((rc = activate(h))) return rc;
    const int64_t Np = h->Np;
    const size_t total = sizeof(double) * 3 * Np;
    if ((rc = ensure(h, h->aos_out, total, "AoS output staging"))) return rc;
    if ((rc = ensure_pinned(h, &h->pin_out, &h->pin_out_bytes, total))) return rc;
    soa_to_aos_kernel<<<grid_for(3 * Np, 256), 256, 0, h->stream>>>(
        Np, (const double*)(field == VPBS_VELOCITY ? h->vel.p : h->psi.p), (double*)h->aos_out.p);
    h->launches++;
    if ((rc = check_cuda(h, cudaGetLastError(), "AoS kernel"))) return rc;
    const size_t chunk = std::max<size_t>(kStageChunk, (total / kStageEvents + 7) & ~(size_t)7);
    int nch = 0;
    for (size_t o = 0; o < total; o += chunk, ++nch) {
        const size_t n = std::min(chunk, total - o);
        if ((rc = check_cuda(h, cudaMemcpyAsync((char*)h->pin_out + o, (const char*)h->aos_out.p + o, n,
                                                cudaMemcpyDeviceToHost, h->stream), "D2H")))
            return rc;
        if ((rc = check_cuda(h, cudaEventRecord(h->stage_ev[nch], h->stream), "event record"))) return rc;
    }
    for (int k = 0; k < nch; ++k) {
        const size_t o = (size_t)k * chunk, n = std::min(chunk, total - o);
        if ((rc = check_cuda(h, cudaEventSynchronize(h->stage_ev[k]), "D2H sync"))) return rc;
        const void* src[1] = {(const char*)h->pin_out + o};
        void* dst[1] = {(char*)out_xyz + o};
        parallel_copies(1, dst, src, &n);
    }
    return 0;
}

int vpbs_get_staged(vpbs_handle* h, int32_t field, const double** aos) {
    if (!h) return VPBS_ERR_ARG;
    if (!aos) return set_error(h, VPBS_ERR_ARG, "null output pointer");
    return fetch_aos(h, field, aos);
}

int vpbs_get_filament_list(vpbs_handle* h, int32_t field, double* const* out, int64_t nfil) {
    if (!h) return VPBS_ERR_ARG;
    if (!out) return set_error(h, VPBS_ERR_ARG, "null output list");
    if (!h->have_filaments || nfil != h->nfil || (int64_t)h->host_offsets.size() != nfil + 1)
        return set_error(h, VPBS_ERR_STATE, "output list does not match the filaments of the last vpbs_set_filaments");
    const double* s;
    int rc = fetch_aos(h, field, &s);
    if (rc) return rc;
    std::vector<void*> dst(nfil);
    std::vector<const void*> src(nfil);
    std::vector<size_t> nb(nfil);
    const int64_t* off = h->host_offsets.data();
    for (int64_t f = 0; f < nfil; ++f) {
        if (!out[f]) return set_error(h, VPBS_ERR_ARG, "null filament output");
        dst[f] = out[f];
        src[f] = s + 3 * off[f];
        nb[f] = sizeof(double) * 3 * (off[f + 1] - off[f]);
    }
    parallel_copies(nfil, dst.data(), src.data(), nb.data());
    return 0;
}

int vpbs_get_soa(vpbs_handle* h, int32_t field, vpbs_vec3 out, int32_t accumulate) {
    if (!h) return VPBS_ERR_ARG;
    if (!out.x || !out.y || !out.z) return set_error(h, VPBS_ERR_ARG, "null output");
    const double* s;
    int rc = fetch_soa(h, field, &s);
    if (rc) return rc;
    const int64_t Np = h->Np;
    double* o[3] = {out.x, out.y, out.z};
    for (int d = 0; d < 3; ++d) {
        if (accumulate)
            for (int64_t i = 0; i < Np; ++i) o[d][i] += s[d * Np + i];
        else
            std::memcpy(o[d], s + d * Np, sizeof(double) * Np);
    }
    return 0;
}

int vpbs_device_field(vpbs_handle* h, int32_t field, double** x, double** y, double** z) {
    if (!h || !x || !y || !z) return VPBS_ERR_ARG;
    if (field != VPBS_VELOCITY && field != VPBS_STREAMFUNCTION) return set_error(h, VPBS_ERR_ARG, "bad field");
    double* base = (double*)(field == VPBS_VELOCITY ? h->vel.p : h->psi.p);
    if (!base) return set_error(h, VPBS_ERR_STATE, "no output allocated");
    *x = base;
    *y = base + h->Np;
    *z = base + 2 * h->Np;
    return 0;
}

int vpbs_get_uhat(vpbs_handle* h, double* out, int64_t n_doubles) {
    if (!h || !out) return VPBS_ERR_ARG;
    if (h->K.open_domain) return set_error(h, VPBS_ERR_STATE, "no long-range field with NoSplitting");
    if (n_doubles != 2 * 3 * h->lr.nmodes) return set_error(h, VPBS_ERR_ARG, "wrong output size for uhat");
    if (!h->have_uhat) return set_error(h, VPBS_ERR_STATE, "long-range field not computed yet");
    int rc;
    if ((rc = activate(h))) return rc;
    if ((rc = check_cuda(h, cudaMemcpyAsync(out, h->uhat.p, sizeof(double) * n_doubles, cudaMemcpyDeviceToHost, h->stream), "D2H uhat")))
        return rc;
    if ((rc = check_cuda(h, cudaStreamSynchronize(h->stream), "stream sync"))) return rc;
    return check_status(h);
}

int vpbs_pair_counts(vpbs_handle* h, int64_t* in_range, int64_t* candidates) {
    if (!h || !in_range || !candidates) return VPBS_ERR_ARG;
    if (!h->counters.p) return set_error(h, VPBS_ERR_STATE, "no pair computation yet");
    unsigned long long c[2];
    int rc;
    if ((rc = activate(h))) return rc;
    if ((rc = check_cuda(h, cudaMemcpyAsync(c, h->counters.p, sizeof c, cudaMemcpyDeviceToHost, h->stream), "D2H counters")))
        return rc;
    if ((rc = check_cuda(h, cudaStreamSynchronize(h->stream), "stream sync"))) return rc;
    *in_range = (int64_t)c[0];
    *candidates = (int64_t)c[1];
    return 0;
}

int vpbs_get_pointdata(vpbs_handle* h, int32_t which, void* out, int64_t n_elems) {
    if (!h || !out) return VPBS_ERR_ARG;
    if (!h->have_points) return set_error(h, VPBS_ERR_STATE, "no point data");
    const int64_t Np = h->Np, Nq = h->Nq;
    const void* src = nullptr;
    int64_t n = 0;
    size_t esz = sizeof(double);
    switch (which) {
        case 0: src = h->nodes.p; n = 3 * Np; break;
        case 1: src = h->d1.p; n = 3 * Np; break;
        case 2: src = h->d2.p; n = 3 * Np; break;
        case 3: src = h->dm.p; n = Np; break;
        case 4: src = h->dp.p; n = Np; break;
        case 5: src = h->points.p; n = 3 * Nq; break;
        case 6: src = h->charges.p; n = 3 * Nq; break;
        case 7: src = h->idx_prev.p; n = Np; esz = sizeof(int32_t); break;
        default: return set_error(h, VPBS_ERR_ARG, "bad point-data selector");
    }
    if (n_elems != n) return set_error(h, VPBS_ERR_ARG, "wrong output size for point data");
    int rc;
    if ((rc = activate(h))) return rc;
    if ((rc = check_cuda(h, cudaMemcpyAsync(out, src, esz * n, cudaMemcpyDeviceToHost, h->stream), "D2H point data")))
        return rc;
    return check_cuda(h, cudaStreamSynchronize(h->stream), "stream sync");
}

int64_t vpbs_launch_count(const vpbs_handle* h) { return h ? h->launches : 0; }

int vpbs_ewald_table_eval(double xmax, const double* x, int64_t n, double* erfc_out, double* g_out) {
    if (!x || !erfc_out || !g_out || n < 0 || !(xmax > 0)) return set_error(nullptr, VPBS_ERR_ARG, "bad arguments");
    int K = 0;
    ewald_table_host(xmax, &K, nullptr);
    std::vector<double> tab((size_t)2 * K * kEwaldNC);
    ewald_table_host(xmax, &K, tab.data());
    for (int64_t i = 0; i < n; ++i) {
        if (!(x[i] >= 0.0 && x[i] <= xmax)) return set_error(nullptr, VPBS_ERR_ARG, "x outside [0, xmax]");
        int k = (int)(x[i] * kEwaldInvH);
        k = k < K ? k : K - 1;
        const double t = x[i] - (k + 0.5) * kEwaldH;
        const double* ce = tab.data() + (size_t)k * kEwaldNC;
        const double* cg = tab.data() + (size_t)(K + k) * kEwaldNC;
        double a = ce[kEwaldNC - 1], g = cg[kEwaldNC - 1];
        for (int m = kEwaldNC - 2; m >= 0; --m) {
            a = std::fma(a, t, ce[m]);
            g = std::fma(g, t, cg[m]);
        }
        erfc_out[i] = a;
        g_out[i] = g;
    }
    return 0;
}

int vpbs_stage_timing(vpbs_handle* h, int32_t enable) {
    if (!h) return VPBS_ERR_ARG;
    int rc;
    if ((rc = activate(h))) return rc;
    if (enable && !h->tev[0][0][0]) {
        for (int s = 0; s < ST_COUNT; ++s)
            for (int k = 0; k < 4; ++k)
                for (int e = 0; e < 2; ++e)
                    if ((rc = check_cuda(h, cudaEventCreate(&h->tev[s][k][e]), "cudaEventCreate"))) return rc;
    }
    h->timing = enable != 0;
    for (int s = 0; s < ST_COUNT; ++s) h->tcount[s] = 0;
    return 0;
}

int vpbs_stage_times(vpbs_handle* h, double* ms, int32_t n) {
    if (!h || !ms || n < ST_COUNT) return VPBS_ERR_ARG;
    if (!h->timing) return set_error(h, VPBS_ERR_STATE, "stage timing is not enabled");
    int rc;
    if ((rc = activate(h))) return rc;
    if ((rc = check_cuda(h, cudaStreamSynchronize(h->stream), "stream sync"))) return rc;
    if ((rc = check_status(h))) return rc;
    for (int s = 0; s < ST_COUNT; ++s) {
        double acc = 0.0;
        for (int k = 0; k < h->tcount[s] && k < 4; ++k) {
            float t = 0.f;
            if ((rc = check_cuda(h, cudaEventElapsedTime(&t, h->tev[s][k][0], h->tev[s][k][1]), "event time"))) return rc;
            acc += t;
        }
        ms[s] = acc;
        h->tcount[s] = 0;
    }
    return 0;
}

const char* vpbs_stage_name(int32_t i) {
    static const char* names[ST_COUNT] = {"geometry", "cell_lists", "spread", "fft_forward", "fourier",
                                          "fft_inverse", "interp", "local_self", "pairs"};
    return (i >= 0 && i < ST_COUNT) ? names[i] : nullptr;
}

}  // extern "C"

namespace {
// Independent FMA chains (8 per thread) to measure the CUDA-core FMA throughput.
template <typename T>
__global__ void __launch_bounds__(256) fma_probe_kernel(T* out, int iters, T a, T b) {
    T x[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) x[k] = (T)(threadIdx.x + k) * (T)1e-3;
    for (int it = 0; it < iters; ++it)
#pragma unroll
        for (int k = 0; k < 8; ++k) x[k] = fma(x[k], a, b);
    T s = 0;
#pragma unroll
    for (int k = 0; k < 8; ++k) s += x[k];
    if (s == (T)12345.678) out[threadIdx.x] = s;  // keeps the chains alive
}
}  // namespace

extern "C" int vpbs_fma_throughput(int32_t device, int32_t fp64, double* tflops) {
    if (!tflops) return VPBS_ERR_ARG;
    if (cudaSetDevice(device) != cudaSuccess) return set_error(nullptr, VPBS_ERR_CUDA, "cudaSetDevice failed");
    int nsm = 0;
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, device);
    void* out = nullptr;
    if (cudaMalloc(&out, 4096) != cudaSuccess) return set_error(nullptr, VPBS_ERR_OOM, "probe allocation failed");
    cudaEvent_t e0, e1;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    const int blocks = nsm * 8, iters = fp64 ? 4096 : 16384;
    double best = 0.0;
    for (int rep = 0; rep < 4; ++rep) {
        cudaEventRecord(e0);
        if (fp64) fma_probe_kernel<double><<<blocks, 256>>>((double*)out, iters, 0.999999, 1e-7);
        else fma_probe_kernel<float><<<blocks, 256>>>((float*)out, iters, 0.999999f, 1e-7f);
        cudaEventRecord(e1);
        cudaEventSynchronize(e1);
        float ms = 0.f;
        cudaEventElapsedTime(&ms, e0, e1);
        const double flops = 2.0 * 8.0 * iters * 256.0 * blocks;
        if (rep > 0 && ms > 0) best = fmax(best, flops / (ms * 1e-3) / 1e12);
    }
    cudaError_t err = cudaGetLastError();
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    cudaFree(out);
    if (err != cudaSuccess) return set_error(nullptr, VPBS_ERR_CUDA, cudaGetErrorString(err));
    *tflops = best;
    return 0;
}

extern "C" int vpbs_spread_mode(vpbs_handle* h, int32_t mode) {
    if (!h || mode < 0 || mode > 1) return VPBS_ERR_ARG;
    h->spread_mode = mode;
    return 0;
}

extern "C" int vpbs_f32_weights_eval(int32_t splitting, double alpha, double rcut, double kb_beta, double kb_rtol,
                                     const double* r, int64_t n, float* a, float* g) {
    using namespace vpbs;
    if (!r || !a || !g || n < 0 || !(rcut > 0)) return set_error(nullptr, VPBS_ERR_ARG, "vpbs_f32_weights_eval: bad arguments");
    const bool kb = splitting == VPBS_SPLITTING_KAISER_BESSEL;
    if (!kb && !(alpha > 0)) return set_error(nullptr, VPBS_ERR_ARG, "vpbs_f32_weights_eval: alpha must be positive");
    int ntab = 0;
    std::vector<double> tab;
    double xmax, s;
    if (kb) {
        const KBSeries S = kb_series(kb_beta, rcut, kb_rtol);
        if (S.f.empty()) return set_error(nullptr, VPBS_ERR_PARAMS, "Kaiser-Bessel series did not converge");
        kb_table_host(S, &ntab, nullptr);
        tab.resize((size_t)2 * ntab * kEwaldNC);
        kb_table_host(S, &ntab, tab.data());
        xmax = kb_table_xmax(kb_beta);
    } else {
        xmax = alpha * rcut;
        ewald_table_host(xmax, &ntab, nullptr);
        tab.resize((size_t)2 * ntab * kEwaldNC);
        ewald_table_host(xmax, &ntab, tab.data());
    }
    s = xmax / rcut;
    const int nf = f32_table_size(xmax);
    std::vector<float4> tabc((size_t)2 * nf);
    f32_table_host(tab.data(), ntab, xmax, tabc.data());
    for (int64_t i = 0; i < n; ++i) {
        if (!(r[i] >= 0.0 && r[i] <= rcut)) return set_error(nullptr, VPBS_ERR_ARG, "vpbs_f32_weights_eval: r outside [0, rcut]");
        // the kernel forms x = (r^2 rsqrt(r^2)) alpha in FP32; here x = alpha r rounded to FP32
        f32_table_eval_host(tabc.data(), nf, (float)(s * r[i]), &a[i], &g[i]);
    }
    return 0;
}

extern "C" int vpbs_f64_weights_eval(int32_t splitting, double alpha, double rcut, double kb_beta, double kb_rtol,
                                     const double* r, int64_t n, double* a, double* g) {
    using namespace vpbs;
    if (!r || !a || !g || n < 0 || !(rcut > 0)) return set_error(nullptr, VPBS_ERR_ARG, "vpbs_f64_weights_eval: bad arguments");
    const bool kb = splitting == VPBS_SPLITTING_KAISER_BESSEL;
    if (!kb && !(alpha > 0)) return set_error(nullptr, VPBS_ERR_ARG, "vpbs_f64_weights_eval: alpha must be positive");
    KBSeries S;
    if (kb) {
        S = kb_series(kb_beta, rcut, kb_rtol);
        if (S.f.empty()) return set_error(nullptr, VPBS_ERR_PARAMS, "Kaiser-Bessel series did not converge");
    }
    const double xmax = kb ? kb_table_xmax(kb_beta) : alpha * rcut, s = xmax / rcut;
    const int nf = tab_s_size(xmax);
    std::vector<double2> tab((size_t)nf * kTabSNC);  // both tables (16-byte aligned)
    tab_s_host(pair_weights_l(S, xmax), xmax, (double*)tab.data());
    for (int64_t i = 0; i < n; ++i) {
        if (!(r[i] >= 0.0 && r[i] <= rcut)) return set_error(nullptr, VPBS_ERR_ARG, "vpbs_f64_weights_eval: r outside [0, rcut]");
        tab_s_eval_host((const double*)tab.data(), nf, s * r[i], &a[i], &g[i]);
    }
    return 0;
}

extern "C" int vpbs_host_copies(int64_t n, void* const* dst, const void* const* src, const size_t* bytes) {
    if (n < 0 || (n > 0 && (!dst || !src || !bytes))) return VPBS_ERR_ARG;
    for (int64_t k = 0; k < n; ++k)
        if (bytes[k] && (!dst[k] || !src[k])) return VPBS_ERR_ARG;
    parallel_copies(n, dst, src, bytes);
    return 0;
}

int vpbs_periodic_eval(double L, int32_t nc, const double* x, int64_t n, double* folded, int64_t* cell) {
    using namespace vpbs;
    if (!(L > 0) || nc < 1 || n < 0 || (n > 0 && !x)) return set_error(nullptr, VPBS_ERR_ARG, "vpbs_periodic_eval: bad arguments");
    const int ncs[3] = {nc, 1, 1};
    const double Ls[3] = {L, 1.0, 1.0};
    for (int64_t i = 0; i < n; ++i) {
        const double f = fold(x[i], L, 0);
        if (folded) folded[i] = f;
        if (cell) cell[i] = cell_index(ncs, Ls, f, 0.5, 0.5);
    }
    return 0;
}
