// One-dimensional FFTs of lines held in shared memory, for the pruned 3-D transforms of the long
// range (fourier_kernels.cuh): Stockham passes of radix 2..32 (FP64: 2..16), any length 2^a 3^b 5^c with at least
// two factors.  A pass reads R values per butterfly (from memory in the first pass, else from shared
// memory), multiplies by the twiddles, transforms in registers and writes R values.  Passes within
// shared memory are in place: every thread keeps its butterflies (32 or 16 values at most) in registers
// across one barrier, so a line takes no second buffer.  The radices are as large as the registers
// allow: two passes (one trip through shared memory) up to n = 32 * 32 in FP32 and 16 * 16 in FP64.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

namespace vpbs {
namespace fft {

constexpr int kMaxPasses = 6;
// Complex values a thread keeps across the barrier of a pass.  The wide form (radices up to 32, FP32
// only) takes 64 registers for them and saves a pass for most n between 256 and 1024; else 16 values are kept.
__host__ __device__ constexpr int pass_values(bool wide) { return wide ? 32 : 16; }

// Butterflies of radix R a thread holds in one in-place pass.
__host__ __device__ constexpr int butterflies(int R, bool wide) { return pass_values(wide) / R; }

struct Pass {
    int R;         // radix
    int Ns;        // product of the earlier radices
    int nR;        // n / R: butterflies per line
    int tw;        // twiddles of this pass: w_{Ns R}^{r k} at table[tw + (r - 1) Ns + k]
    uint32_t mNs, mnR;  // magic numbers of the divisions by Ns and nR
    // Places in shared memory.  Between the passes position p lies at p + p / R0 (R0 the first radix), so
    // that the strided stores spread over the banks; the values before the first and after the last pass
    // lie unpadded.  R0 divides the strides of every later pass, so the R accesses of a butterfly are a
    // base plus r times a constant.
    int in_stride, out_stride, out_q;
    uint32_t min, mout;  // magic numbers of the division by R0 of the base (UINT32_MAX: unpadded)
};

struct Plan {
    int n = 0, np = 0;
    int len = 0;  // places a line takes, padding included
    bool wide = false;
    Pass p[kMaxPasses];
};

// x / d for x < 2^20 and d < 2^12 by a 32-bit multiply-high (m = ceil(2^32 / d); d = 1 has m = 0).
__host__ inline uint32_t div_magic(uint32_t d) { return d <= 1 ? 0u : (uint32_t)(((uint64_t)1 << 32) / d + ((((uint64_t)1 << 32) % d) ? 1 : 0)); }
__device__ __forceinline__ int fdiv(int x, uint32_t m) { return m ? (int)__umulhi((uint32_t)x, m) : x; }
// x + x / R0, or x where the place is not padded
constexpr uint32_t kNoPad = 0xffffffffu;
__device__ __forceinline__ int padded(int x, uint32_t m) { return m == kNoPad ? x : x + fdiv(x, m); }

template <typename T>
struct Cplx;
template <>
struct Cplx<float> { using type = float2; };
template <>
struct Cplx<double> { using type = double2; };

__device__ __forceinline__ float2 mk(float x, float y) { return make_float2(x, y); }
__device__ __forceinline__ double2 mk(double x, double y) { return make_double2(x, y); }
template <typename C>
__device__ __forceinline__ C add(C a, C b) { return mk(a.x + b.x, a.y + b.y); }
template <typename C>
__device__ __forceinline__ C sub(C a, C b) { return mk(a.x - b.x, a.y - b.y); }
template <typename C>
__device__ __forceinline__ C mul(C a, C b) { return mk(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x); }
// a times conj(b) when SIGN > 0 (the tables hold e^{-i t}; the inverse transform needs e^{+i t})
template <int SIGN, typename C>
__device__ __forceinline__ C mul_tw(C a, C b) {
    if (SIGN < 0) return mul(a, b);
    return mk(a.x * b.x + a.y * b.y, a.y * b.x - a.x * b.y);
}
// SIGN i a
template <int SIGN, typename C>
__device__ __forceinline__ C mul_i(C a) {
    return SIGN > 0 ? mk(-a.y, a.x) : mk(a.y, -a.x);
}

// cos and sin of 2 pi m / R at compile time (Taylor series of the angle reduced to [-pi/4, pi/4]).
constexpr double ct_sin(double x) {
    double t = x, s = x;
    for (int k = 1; k < 14; ++k) {
        t *= -x * x / ((2.0 * k) * (2.0 * k + 1.0));
        s += t;
    }
    return s;
}
constexpr double ct_cos(double x) {
    double t = 1.0, s = 1.0;
    for (int k = 1; k < 14; ++k) {
        t *= -x * x / ((2.0 * k - 1.0) * (2.0 * k));
        s += t;
    }
    return s;
}
constexpr double kPiF = 3.14159265358979323846;
// 2 pi m / R = q pi / 2 + x with |x| <= pi / 4
constexpr double unit_cos(int m, int R) {
    m %= R;
    const int q = (8 * m + R) / (2 * R);  // nearest multiple of pi / 2
    const double x = 2.0 * kPiF * (4.0 * m - (double)q * R) / (4.0 * R);
    switch (q & 3) {
        case 0: return ct_cos(x);
        case 1: return -ct_sin(x);
        case 2: return -ct_cos(x);
        default: return ct_sin(x);
    }
}
constexpr double unit_sin(int m, int R) {
    m %= R;
    const int q = (8 * m + R) / (2 * R);
    const double x = 2.0 * kPiF * (4.0 * m - (double)q * R) / (4.0 * R);
    switch (q & 3) {
        case 0: return ct_sin(x);
        case 1: return ct_cos(x);
        case 2: return -ct_sin(x);
        default: return -ct_cos(x);
    }
}
template <int R>
struct Units {
    double c[R], s[R];
    constexpr Units() : c(), s() {
        for (int m = 0; m < R; ++m) {
            c[m] = unit_cos(m, R);
            s[m] = unit_sin(m, R);
        }
    }
};

// a times a constant known to double precision.  FP32 takes it as hi + lo: rounded to FP32 by themselves,
// sqrt(1/2), sqrt(3)/2, cos and sin(pi/8) are all too small, and every value that passes a transform shrinks by
// 2e-8 to 5e-8 (sizes 2^a 3^b; the streamfunction of a 432^3 grid was off by 1.8e-7, with this 0.5e-7).  The
// extra instructions cost the FP32 transforms 2 %.
__device__ __forceinline__ float times(float a, double c) {
    const float hi = (float)c;
    return fmaf(a, hi, a * (float)(c - (double)hi));
}
// a e^{SIGN 2 pi i e / R} in FP32, e (0 < e < R) and R known at compile time
template <int R, int SIGN, typename C>
__device__ __forceinline__ C rotate(C a, int e, double c, double s) {
    using T = decltype(a.x);
    if (4 * e % R == 0) return 4 * e / R == 2 ? mk(-a.x, -a.y) : 4 * e / R == 1 ? mul_i<SIGN>(a) : mul_i<-SIGN>(a);
    if (8 * e % R == 0) {  // c = +-s
        const double f = c < 0 ? -c : c;
        const T u = c < 0 ? -a.x : a.x, v = c < 0 ? -a.y : a.y;
        return (c > 0) == (SIGN * s > 0) ? mk(times(u - v, f), times(u + v, f)) : mk(times(u + v, f), times(v - u, f));
    }
    const T ch = (T)c, sh = (T)(SIGN * s), cl = (T)(c - (double)ch), sl = (T)(SIGN * s - (double)sh);
    return mk(fmaf(a.x, ch, fmaf(-a.y, sh, fmaf(a.x, cl, -a.y * sl))), fmaf(a.x, sh, fmaf(a.y, ch, fmaf(a.x, sl, a.y * cl))));
}

// v <- DFT of v with kernel exp(SIGN 2 pi i n k / R), natural order.
template <int R, int SIGN>
struct Dft;

template <int SIGN>
struct Dft<2, SIGN> {
    template <typename C>
    __device__ __forceinline__ static void run(C (&v)[2]) {
        const C a = v[0], b = v[1];
        v[0] = add(a, b);
        v[1] = sub(a, b);
    }
};

template <int SIGN>
struct Dft<3, SIGN> {
    template <typename C>
    __device__ __forceinline__ static void run(C (&v)[3]) {
        using T = decltype(v[0].x);
        constexpr double h3 = unit_sin(1, 3);
        const C a = add(v[1], v[2]), d = sub(v[1], v[2]);
        const C m = mk(v[0].x - (T)0.5 * a.x, v[0].y - (T)0.5 * a.y);
        C q;
        if constexpr (sizeof(T) == 8) {
            const T f = (T)h3;
            q = mul_i<SIGN>(mk(f * d.x, f * d.y));
        } else {
            q = mul_i<SIGN>(mk(times(d.x, h3), times(d.y, h3)));
        }
        v[0] = add(v[0], a);
        v[1] = add(m, q);
        v[2] = sub(m, q);
    }
};

template <int SIGN>
struct Dft<4, SIGN> {
    template <typename C>
    __device__ __forceinline__ static void run(C (&v)[4]) {
        const C a = add(v[0], v[2]), b = sub(v[0], v[2]), c = add(v[1], v[3]), d = mul_i<SIGN>(sub(v[1], v[3]));
        v[0] = add(a, c);
        v[1] = add(b, d);
        v[2] = sub(a, c);
        v[3] = sub(b, d);
    }
};

template <int SIGN>
struct Dft<5, SIGN> {
    template <typename C>
    __device__ __forceinline__ static void run(C (&v)[5]) {
        using T = decltype(v[0].x);
        constexpr double dc1 = unit_cos(1, 5), dc2 = unit_cos(2, 5), ds1 = unit_sin(1, 5), ds2 = unit_sin(2, 5);
        const T c1 = (T)dc1, c2 = (T)dc2, s1 = (T)ds1, s2 = (T)ds2;
        const C a1 = add(v[1], v[4]), a2 = add(v[2], v[3]), b1 = sub(v[1], v[4]), b2 = sub(v[2], v[3]);
        const C p1 = mk(v[0].x + c1 * a1.x + c2 * a2.x, v[0].y + c1 * a1.y + c2 * a2.y);
        const C p2 = mk(v[0].x + c2 * a1.x + c1 * a2.x, v[0].y + c2 * a1.y + c1 * a2.y);
        const C q1 = mul_i<SIGN>(mk(s1 * b1.x + s2 * b2.x, s1 * b1.y + s2 * b2.y));
        const C q2 = mul_i<SIGN>(mk(s2 * b1.x - s1 * b2.x, s2 * b1.y - s1 * b2.y));
        v[0] = mk(v[0].x + a1.x + a2.x, v[0].y + a1.y + a2.y);
        v[1] = add(p1, q1);
        v[4] = sub(p1, q1);
        v[2] = add(p2, q2);
        v[3] = sub(p2, q2);
    }
};

// R = A B: inner DFTs of length A over n = B n1 + n2, twiddles w_R^{n2 k1}, outer DFTs of length B
// (output k = k1 + A k2).
template <int A, int B, int SIGN>
struct DftAB {
    template <typename C>
    __device__ __forceinline__ static void run(C (&v)[A * B]) {
        using T = decltype(v[0].x);
        constexpr Units<A * B> U;
        C y[B][A];
#pragma unroll
        for (int n2 = 0; n2 < B; ++n2) {
            C t[A];
#pragma unroll
            for (int n1 = 0; n1 < A; ++n1) t[n1] = v[B * n1 + n2];
            Dft<A, SIGN>::run(t);
#pragma unroll
            for (int k1 = 0; k1 < A; ++k1) {
                if (n2 * k1 == 0)
                    y[n2][k1] = t[k1];
                else if constexpr (sizeof(T) == 8)  // plain products: FP64 has no registers for more cases (6 % of the inverse)
                    y[n2][k1] = mul(t[k1], mk((T)U.c[n2 * k1], (T)(SIGN * U.s[n2 * k1])));
                else
                    y[n2][k1] = rotate<A * B, SIGN>(t[k1], n2 * k1, U.c[n2 * k1], U.s[n2 * k1]);
            }
        }
#pragma unroll
        for (int k1 = 0; k1 < A; ++k1) {
            C t[B];
#pragma unroll
            for (int n2 = 0; n2 < B; ++n2) t[n2] = y[n2][k1];
            Dft<B, SIGN>::run(t);
#pragma unroll
            for (int k2 = 0; k2 < B; ++k2) v[k1 + A * k2] = t[k2];
        }
    }
};
template <int SIGN>
struct Dft<6, SIGN> : DftAB<2, 3, SIGN> {};
template <int SIGN>
struct Dft<8, SIGN> : DftAB<2, 4, SIGN> {};
template <int SIGN>
struct Dft<9, SIGN> : DftAB<3, 3, SIGN> {};
template <int SIGN>
struct Dft<10, SIGN> : DftAB<2, 5, SIGN> {};
template <int SIGN>
struct Dft<12, SIGN> : DftAB<3, 4, SIGN> {};
template <int SIGN>
struct Dft<15, SIGN> : DftAB<3, 5, SIGN> {};
template <int SIGN>
struct Dft<16, SIGN> : DftAB<4, 4, SIGN> {};
template <int SIGN>
struct Dft<18, SIGN> : DftAB<3, 6, SIGN> {};
template <int SIGN>
struct Dft<20, SIGN> : DftAB<4, 5, SIGN> {};
template <int SIGN>
struct Dft<24, SIGN> : DftAB<4, 6, SIGN> {};
template <int SIGN>
struct Dft<25, SIGN> : DftAB<5, 5, SIGN> {};
template <int SIGN>
struct Dft<32, SIGN> : DftAB<4, 8, SIGN> {};

// Lines stored one after the other, [line][place]; consecutive threads take consecutive butterflies of
// a line.
struct LinesX {
    int len;
    __device__ __forceinline__ int step() const { return 1; }
    __device__ __forceinline__ void split(int idx, const Pass& P, int& line, int& j) const {
        line = fdiv(idx, P.mnR);
        j = idx - line * P.nR;
    }
    __device__ __forceinline__ int at(int line, int place) const { return line * len + place; }
};

// 2^ltx neighbouring lines interleaved, [group][place][line in group]: consecutive threads take the
// same butterfly of neighbouring lines (the values next to each other in memory).
struct LinesT {
    int len, ltx;
    __device__ __forceinline__ int step() const { return 1 << ltx; }
    __device__ __forceinline__ void split(int idx, const Pass& P, int& line, int& j) const {
        const int tx = idx & ((1 << ltx) - 1), t = idx >> ltx;
        const int g = fdiv(t, P.mnR);
        j = t - g * P.nR;
        line = (g << ltx) + tx;
    }
    __device__ __forceinline__ int at(int line, int place) const {
        return (((line >> ltx) * len + place) << ltx) + (line & ((1 << ltx) - 1));
    }
};

// v[r] *= w^{r k}: neighbouring threads have neighbouring k, so every load is one run of the table.
template <int R, int SIGN, typename C>
__device__ __forceinline__ void twiddle(C (&v)[R], const C* __restrict__ tw, int k, const Pass& P) {
#pragma unroll
    for (int r = 1; r < R; ++r) v[r] = mul_tw<SIGN>(v[r], __ldg(tw + (P.tw + (r - 1) * P.Ns + k)));
}

// First pass (Ns = 1, no twiddles): values from load(line, position), into shared memory.
template <int R, int SIGN, typename C, typename Lay, typename Load>
__device__ __forceinline__ void pass_in(C* S, const Lay& lay, const Pass& P, int nlines, Load load) {
    const int total = nlines * P.nR;
    for (int idx = threadIdx.x; idx < total; idx += blockDim.x) {
        int line, j;
        lay.split(idx, P, line, j);
        C v[R];
#pragma unroll
        for (int r = 0; r < R; ++r) v[r] = load(line, j + r * P.nR);
        Dft<R, SIGN>::run(v);
        C* o = S + lay.at(line, j * P.out_q);
        const int d = lay.step();
#pragma unroll
        for (int r = 0; r < R; ++r) o[r * d] = v[r];
    }
    __syncthreads();
}

// A pass within shared memory (FIRST: Ns = 1, no twiddles); nlines nR <= blockDim butterflies(R).
template <int R, int SIGN, bool WIDE, typename C, typename Lay>
__device__ __forceinline__ void pass_mid(C* S, const Lay& lay, const Pass& P, int nlines, const C* __restrict__ tw) {
    constexpr int NB = butterflies(R, WIDE);
    const int total = nlines * P.nR;
    C v[NB][R];
#pragma unroll
    for (int b = 0; b < NB; ++b) {
        // threads past the end repeat the last butterfly (and do not write it): v is always assigned, so it
        // does not stay live from pass to pass
        const int idx = min((int)(threadIdx.x + b * blockDim.x), total - 1);
        int line, j;
        lay.split(idx, P, line, j);
        const C* in = S + lay.at(line, padded(j, P.min));
        const int d = P.in_stride * lay.step();
#pragma unroll
        for (int r = 0; r < R; ++r) v[b][r] = in[r * d];
        if (P.Ns > 1) twiddle<R, SIGN>(v[b], tw, j - fdiv(j, P.mNs) * P.Ns, P);
        Dft<R, SIGN>::run(v[b]);
    }
    __syncthreads();
#pragma unroll
    for (int b = 0; b < NB; ++b) {
        const int idx = threadIdx.x + b * blockDim.x;
        if (idx < total) {
            int line, j;
            lay.split(idx, P, line, j);
            const int q = fdiv(j, P.mNs), k = j - q * P.Ns;
            C* o = S + lay.at(line, q * P.out_q + padded(k, P.mout));
            const int d = P.out_stride * lay.step();
#pragma unroll
            for (int r = 0; r < R; ++r) o[r * d] = v[b][r];
        }
    }
    __syncthreads();
}

// Last pass (Ns R = n: natural order out): from shared memory to store(line, position, value).
template <int R, int SIGN, typename C, typename Lay, typename Store>
__device__ __forceinline__ void pass_out(const C* S, const Lay& lay, const Pass& P, int nlines,
                                         const C* __restrict__ tw, Store store) {
    const int total = nlines * P.nR;
    for (int idx = threadIdx.x; idx < total; idx += blockDim.x) {
        int line, j;
        lay.split(idx, P, line, j);
        C v[R];
        const C* in = S + lay.at(line, padded(j, P.min));
        const int d = P.in_stride * lay.step();
#pragma unroll
        for (int r = 0; r < R; ++r) v[r] = in[r * d];
        twiddle<R, SIGN>(v, tw, j, P);
        Dft<R, SIGN>::run(v);
#pragma unroll
        for (int r = 0; r < R; ++r) store(line, j + r * P.nR, v[r]);
    }
}

#define VPBS_FFT_RADICES(X) X(2) X(3) X(4) X(5) X(6) X(8) X(9) X(10) X(12) X(15) X(16)
#define VPBS_FFT_RADICES_WIDE(X) X(18) X(20) X(24) X(25) X(32)

template <int SIGN, bool WIDE, typename C, typename Lay, typename Load>
__device__ __forceinline__ void run_in(C* S, const Lay& lay, const Pass& P, int nlines, Load load) {
#define X(r) \
    case r: pass_in<r, SIGN>(S, lay, P, nlines, load); return;
    switch (P.R) { VPBS_FFT_RADICES(X) }
    if constexpr (WIDE) switch (P.R) { VPBS_FFT_RADICES_WIDE(X) }
#undef X
}
template <int SIGN, bool WIDE, typename C, typename Lay>
__device__ __forceinline__ void run_mid(C* S, const Lay& lay, const Pass& P, int nlines, const C* __restrict__ tw) {
#define X(r) \
    case r: pass_mid<r, SIGN, WIDE>(S, lay, P, nlines, tw); return;
    switch (P.R) { VPBS_FFT_RADICES(X) }
    if constexpr (WIDE) switch (P.R) { VPBS_FFT_RADICES_WIDE(X) }
#undef X
}
template <int SIGN, bool WIDE, typename C, typename Lay, typename Store>
__device__ __forceinline__ void run_out(const C* S, const Lay& lay, const Pass& P, int nlines,
                                        const C* __restrict__ tw, Store store) {
#define X(r) \
    case r: pass_out<r, SIGN>(S, lay, P, nlines, tw, store); return;
    switch (P.R) { VPBS_FFT_RADICES(X) }
    if constexpr (WIDE) switch (P.R) { VPBS_FFT_RADICES_WIDE(X) }
#undef X
}

}  // namespace fft
}  // namespace vpbs
