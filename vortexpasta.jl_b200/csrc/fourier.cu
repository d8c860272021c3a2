// Plans of the pruned transforms of the long range (kernels: fourier_kernels.cuh): which sizes take them, the radices
// of every line, the tiles, and the choice of the grid precision.
#include <algorithm>
#include <cmath>
#include <vector>

#include "fourier_plan.cuh"

namespace vpbs {
namespace {

using fft::Cplx;
using fft::Plan;

// Threads a line needs so that a pass of radix R fits its butterflies.
int threads_of(int n, int R, bool wide) {
    const int nb = fft::butterflies(R, wide);
    return (n / R + nb - 1) / nb;
}

// Radices of n with the fewest passes, then the fewest threads a line needs; none if n has one factor.
void plan_search(int n, bool wide, std::vector<int>& cur, std::vector<int>& best, double& cost, int n_all) {
    static const int radices[] = {32, 25, 24, 20, 18, 16, 15, 12, 10, 9, 8, 6, 5, 4, 3, 2};
    if (n == 1) {
        if (cur.size() < 2) return;
        int t = 0;
        for (int R : cur) t = std::max(t, threads_of(n_all, R, wide));
        const double c = 1e4 * (double)cur.size() + t;
        if (c < cost) {
            cost = c;
            best = cur;
        }
        return;
    }
    if ((int)cur.size() >= fft::kMaxPasses) return;
    for (int R : radices)
        if (n % R == 0 && R <= fft::pass_values(wide) && (cur.empty() || R <= cur.back())) {  // largest first
            cur.push_back(R);
            plan_search(n / R, wide, cur, best, cost, n_all);
            cur.pop_back();
        }
}

// The passes of a line of n values; their twiddles are appended to `tab`.
template <typename C>
Plan make_plan(int n, std::vector<C>& tab) {
    using T = decltype(C::x);
    Plan P;
    std::vector<int> cur, best;
    double cost = 1e30;
    plan_search(n, false, cur, best, cost, n);
    if (sizeof(C) == 8) {  // wide where that saves a pass
        std::vector<int> wbest;
        double wcost = 1e30;
        plan_search(n, true, cur, wbest, wcost, n);
        if (wbest.size() < best.size()) {
            best = wbest;
            P.wide = true;
        }
    }
    P.n = n;
    P.np = (int)best.size();
    if (!P.np) return P;
    const int R0 = best[0];
    P.len = n + n / R0;
    int Ns = 1;
    for (int i = 0; i < P.np; ++i) {
        fft::Pass& p = P.p[i];
        p.R = best[i];
        p.Ns = Ns;
        p.nR = n / p.R;
        p.mNs = fft::div_magic((uint32_t)Ns);
        p.mnR = fft::div_magic((uint32_t)p.nR);
        const bool last = i == P.np - 1;
        p.min = i == 0 ? fft::kNoPad : fft::div_magic((uint32_t)R0);
        p.in_stride = i == 0 ? p.nR : p.nR + p.nR / R0;
        p.mout = last ? fft::kNoPad : fft::div_magic((uint32_t)R0);
        p.out_stride = i == 0 ? 1 : last ? Ns : Ns + Ns / R0;
        p.out_q = i == 0 ? p.R + 1 : last ? 0 : Ns * p.R + Ns * p.R / R0;
        p.tw = (int)tab.size();
        for (int r = 1; r < p.R && Ns > 1; ++r)
            for (int k = 0; k < Ns; ++k) {
                const double a = 2.0 * kPi * ((int64_t)r * k % (Ns * p.R)) / (Ns * p.R);
                C w;
                w.x = (T)std::cos(a);
                w.y = (T)-std::sin(a);
                tab.push_back(w);
            }
        Ns *= p.R;
    }
    return P;
}

// Threads that one line needs so that every pass fits its butterflies.
int threads_per_line(const Plan& P) {
    int t = 1;
    for (int i = 0; i < P.np; ++i) t = std::max(t, threads_of(P.n, P.p[i].R, P.wide));
    return t;
}

inline int round32(int t) { return (t + 31) / 32 * 32; }

constexpr size_t kFftSmemGood = 76 * 1024;  // three blocks per SM

// Lines of a tile (a power of two of neighbouring k_x; `group` tiles per block): 64 bytes wide, wider
// while a block would have too few threads, narrower where threads or shared memory run out.
bool tile_shape(const Plan& P, int group, size_t csize, int kx, int* ltx, FourierShape* s) {
    const int tpl = threads_per_line(P);
    int l = csize == 8 ? 3 : 2;
    while ((group * tpl << l) < 96 && (1 << l) < kx && l < 5) ++l;
    auto bytes = [&](int lt) { return csize * P.len * ((size_t)group << lt); };
    while (l > 0 && (round32(group * tpl << l) > kFftThreads || bytes(l) > (l > 1 ? kFftSmemGood : kFftSmemMost))) --l;
    *ltx = l;
    s->threads = round32(group * tpl << l);
    s->smem = bytes(l);
    return s->threads <= kFftThreads && s->smem <= kFftSmemMost;
}

// Plans and twiddle tables of the three dimensions; false where a length has fewer than two factors.
template <typename T>
bool make_plans(const LRSizes& S, FourierPlan& F, std::vector<unsigned char>& tables) {
    using C = typename Cplx<T>::type;
    std::vector<C> tab;
    F.px = make_plan<C>(S.n[0] / 2, tab);
    F.py = make_plan<C>(S.n[1], tab);
    F.pz = make_plan<C>(S.n[2], tab);
    F.twr = tab.size();
    for (int k = 0; k < S.n[0] / 2; ++k) {
        C w;
        w.x = (T)std::cos(2.0 * kPi * k / S.n[0]);
        w.y = (T)-std::sin(2.0 * kPi * k / S.n[0]);
        tab.push_back(w);
    }
    const unsigned char* b = (const unsigned char*)tab.data();
    tables.assign(b, b + sizeof(C) * tab.size());
    return F.px.np >= 2 && F.py.np >= 2 && F.pz.np >= 2;
}

}  // namespace

// The pruned transforms for the sizes in h->lr, or no plan (h->fplan null) where a line has fewer than
// two factors, is longer than 2048, or its tile does not fit a block (z lines of three components above 512 threads:
// 1620, in FP64 also 1944): those sizes use cuFFT.
int fourier_init(vpbs_handle* h) {
    const LRSizes& S = h->lr;
    const bool mixed = h->P.precision == VPBS_PRECISION_MIXED;
    const size_t csize = mixed ? sizeof(float2) : sizeof(double2);
    FourierPlan F;
    F.kx = S.nkx - 1;
    if (S.n[0] % 2 || F.kx < 1 || S.n[0] > 2048 || S.n[1] > 2048 || S.n[2] > 2048) return 0;
    std::vector<unsigned char> tables;
    if (!(mixed ? make_plans<float>(S, F, tables) : make_plans<double>(S, F, tables))) return 0;
    // x: about 256 threads of whole lines
    const int tpl = threads_per_line(F.px);
    if (round32(tpl) > kFftThreads) return 0;
    F.LY = std::max(1, 256 / tpl);
    F.sx.threads = round32(F.LY * tpl);
    F.sx.smem = csize * F.LY * F.px.len;
    F.LYq = std::max(1, F.LY / 3);
    F.sq.threads = round32(3 * F.LYq * tpl);
    F.sq.smem = csize * 3 * F.LYq * F.px.len;
    if (F.sx.smem > kFftSmemMost || F.sq.threads > kFftThreads || F.sq.smem > kFftSmemMost) return 0;
    if (!tile_shape(F.py, 1, csize, F.kx, &F.ltxy, &F.sy) || !tile_shape(F.pz, 3, csize, F.kx, &F.ltxz, &F.sz)) return 0;
    const int tile = 1 << std::max(F.ltxy, F.ltxz);
    F.kxp = (F.kx + tile - 1) / tile * tile;
    if ((int64_t)3 * S.n[2] > 65535 || S.Ns[1] > 65535) return 0;
    int rc = mixed ? fourier_attributes_f32(h, F) : fourier_attributes_f64(h, F);
    if (!rc) rc = ensure(h, h->fft_tw, tables.size(), "FFT tables");
    if (!rc) rc = check_cuda(h, cudaMemcpy(h->fft_tw.p, tables.data(), tables.size(), cudaMemcpyHostToDevice), "copy FFT tables");
    if (!rc) rc = ensure(h, h->grid_c, csize * 3 * S.n[2] * S.n[1] * (size_t)F.kxp, "complex grid");
    // the plane k_x = Ns0/2 of the coefficients is zero and no kernel writes it
    if (!rc) rc = check_cuda(h, cudaMemset(h->uhat.p, 0, sizeof(double2) * 3 * S.nmodes), "memset");
    if (!rc) rc = check_cuda(h, cudaStreamSynchronize(0), "memset");
    if (!rc) h->fplan = new FourierPlan(F);
    return rc;
}

void fourier_free(vpbs_handle* h) {
    delete h->fplan;
    h->fplan = nullptr;
}

int fourier_forward(vpbs_handle* h, const void* grid) {
    return h->P.precision == VPBS_PRECISION_MIXED ? fourier_forward_f32(h, grid) : fourier_forward_f64(h, grid);
}
int fourier_operator(vpbs_handle* h, const FourierOp& op) {
    return h->P.precision == VPBS_PRECISION_MIXED ? fourier_operator_f32(h, op) : fourier_operator_f64(h, op);
}
int fourier_inverse(vpbs_handle* h, void* grid, bool quad) {
    return h->P.precision == VPBS_PRECISION_MIXED ? fourier_inverse_f32(h, grid, quad) : fourier_inverse_f64(h, grid);
}

}  // namespace vpbs
