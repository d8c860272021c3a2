// Short-range part of the Ewald split on the device:
//  * local (LIA) term and self-interaction removal, one thread per node
//    (src/BiotSavart/shortrange/local_integrals.jl:4-165);
//  * cell lists as a counting sort of the quadrature points (and of the nodes) by cell
//    (replaces the linked lists of src/CellLists/gpu.jl:28-61 and the destination sort of
//    gpu.jl:183-231);
//  * the pair kernels (src/BiotSavart/shortrange/shortrange.jl:216-273 with the Gaussian
//    weights of splitting/gaussian.jl:273-279): a warp per few nodes that follow one another in
//    cell order, lanes over the contiguous cell-sorted source ranges of the (2M+1)^2
//    neighbour rows, warp-shuffle reduction at the end.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "vpbs_internal.cuh"
#include "periodic.cuh"

namespace vpbs {

// Interval and local coordinate of x in the FP32 cubic tables: k = floor(32 x) (rounded through
// the 1.5 * 2^23 trick, no conversion instruction), t = 32 x - k; k is clamped into [0, nf).
__host__ __device__ __forceinline__ void f32_table_pos(float x, int nf, int* k, float* t) {
    const float u = fmaf(x, kTabCInvH, -0.5f);
#if defined(__CUDA_ARCH__)
    const float y = __fadd_rn(u, 12582912.0f);
    const float kf = __fsub_rn(y, 12582912.0f);
    int kk = __float_as_int(y) - 0x4B400000;
#else
    volatile float yv = u + 12582912.0f;
    const float y = yv;
    volatile float kv = y - 12582912.0f;
    const float kf = kv;
    int kk;
    std::memcpy(&kk, &y, sizeof(int));
    kk -= 0x4B400000;
#endif
    *t = fmaf(x, kTabCInvH, -kf);
    const unsigned top = (unsigned)(nf - 1);
    *k = (int)((unsigned)kk < top ? (unsigned)kk : top);
}

__host__ __device__ __forceinline__ float f32_cubic(float4 c, float t) {
    return fmaf(fmaf(fmaf(c.w, t, c.z), t, c.y), t, c.x);
}

namespace {

__device__ __forceinline__ int64_t cell_of(const CellGrid& cg, const KParams& K, double x, double y, double z) {
    return cell_index(cg.nc, K.L, x, y, z);
}

// Cell of every quadrature point and node and its rank within the cell (atomic counters).  The nodes'
// entries follow the points' in every array; their threads start at a whole warp, so that no warp counts
// both.  dm (if given): delta^- of the nodes, the delta^+ of the previous node.
__global__ void cell_count_kernel(KParams K, CellGrid cg, int64_t Nq, int64_t Np, const double* __restrict__ points,
                                  const double* __restrict__ nodes, int32_t* __restrict__ cell, int32_t* __restrict__ rank,
                                  int32_t* __restrict__ counts, const int32_t* __restrict__ idx_prev,
                                  const double* __restrict__ dp, double* __restrict__ dm) {
    const int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, j0 = (Nq + 31) & ~(int64_t)31;
    if ((j >= Nq && j < j0) || j >= j0 + Np) return;
    const bool node = j >= j0;
    const int64_t k = node ? j - j0 : j, n = node ? Np : Nq, e = node ? Nq + k : k;
    const double* xyz = node ? nodes : points;
    const int32_t c = (int32_t)cell_of(cg, K, xyz[k], xyz[n + k], xyz[2 * n + k]);
    cell[e] = c;
    if (node && dm) dm[k] = dp[idx_prev[k]];
    rank[e] = warp_aggregated_rank(node ? counts + cg.ncell + 1 : counts, c);
}

// Exclusive scan of counts[0..n) into start[0..n] with one CTA of 1024 threads; `sub` is subtracted from
// start[split] on (two arrays scanned as one).
__global__ void __launch_bounds__(1024) scan_kernel(const int32_t* __restrict__ counts, int32_t* __restrict__ start,
                                                    int64_t n, int64_t split, int32_t sub) {
    __shared__ int32_t part[1024];
    const int tid = threadIdx.x;
    const int64_t chunk = (n + 1023) / 1024;
    const int64_t lo = tid * chunk;
    const int64_t hi = lo + chunk < n ? lo + chunk : n;
    int32_t s = 0;
    for (int64_t i = lo; i < hi; ++i) s += counts[i];
    part[tid] = s;
    __syncthreads();
    for (int off = 1; off < 1024; off <<= 1) {
        int32_t v = tid >= off ? part[tid - off] : 0;
        __syncthreads();
        part[tid] += v;
        __syncthreads();
    }
    int32_t acc = part[tid] - s;  // exclusive prefix of this chunk
    for (int64_t i = lo; i < hi; ++i) {
        start[i] = acc - (i >= split ? sub : 0);
        acc += counts[i];
    }
    if (tid == 1023) start[n] = part[1023] - (n >= split ? sub : 0);
}

// Multi-CTA exclusive scan for long count arrays: per-chunk sums, a scan of the sums (with
// scan_kernel), then every chunk scanned in shared memory from its offset.
constexpr int kScanThreads = 1024, kScanPer = 4, kScanChunk = kScanThreads * kScanPer;

__device__ __forceinline__ int warp_incl_scan(int x, int lane) {
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += t;
    }
    return x;
}

__global__ void __launch_bounds__(kScanThreads) scan_partials_kernel(const int32_t* __restrict__ counts, int64_t n,
                                                                    int32_t* __restrict__ part) {
    __shared__ int wt[32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t base = (int64_t)blockIdx.x * kScanChunk + (int64_t)threadIdx.x * kScanPer;
    int s = 0;
#pragma unroll
    for (int k = 0; k < kScanPer; ++k)
        if (base + k < n) s += counts[base + k];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) wt[warp] = s;
    __syncthreads();
    if (warp == 0) {
        int v = wt[lane];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if (lane == 0) part[blockIdx.x] = v;
    }
}

__global__ void __launch_bounds__(kScanThreads) scan_chunks_kernel(const int32_t* __restrict__ counts, int64_t n,
                                                                  const int32_t* __restrict__ part_start,
                                                                  int32_t* __restrict__ start, int64_t split, int32_t sub) {
    __shared__ int wt[32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t base = (int64_t)blockIdx.x * kScanChunk + (int64_t)threadIdx.x * kScanPer;
    int c[kScanPer], s = 0;
#pragma unroll
    for (int k = 0; k < kScanPer; ++k) {
        c[k] = base + k < n ? counts[base + k] : 0;
        s += c[k];
    }
    const int x = warp_incl_scan(s, lane);
    if (lane == 31) wt[warp] = x;
    __syncthreads();
    if (warp == 0) wt[lane] = warp_incl_scan(wt[lane], lane);
    __syncthreads();
    int acc = part_start[blockIdx.x] + (warp > 0 ? wt[warp - 1] : 0) + x - s;
#pragma unroll
    for (int k = 0; k < kScanPer; ++k) {
        if (base + k < n) start[base + k] = acc - (base + k >= split ? sub : 0);
        acc += c[k];
    }
    if (blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) start[n] = part_start[gridDim.x] - (n >= split ? sub : 0);
}

// Scatter the sources into cell order (SoA: x, y, z, qx, qy, qz) and record their segment; list the nodes in
// cell order.
__global__ void scatter_kernel(int64_t Nq, int64_t Np, int nquad, const double* __restrict__ points,
                                       const double* __restrict__ charges, const int32_t* __restrict__ cell,
                                       const int32_t* __restrict__ rank, const int32_t* __restrict__ start,
                                       double* __restrict__ sorted, int32_t* __restrict__ seg,
                                       float4* __restrict__ f32, int f32_parts, const int32_t* __restrict__ dst_start,
                               int32_t* __restrict__ order) {
    int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= Nq + Np) return;
    if (j >= Nq) {
        order[(int64_t)dst_start[cell[j]] + rank[j]] = (int32_t)(j - Nq);
        return;
    }
    const int64_t pos = (int64_t)start[cell[j]] + rank[j];
    double x[3], q[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        x[d] = points[d * Nq + j];
        q[d] = charges[d * Nq + j];
        sorted[d * Nq + pos] = x[d];
        sorted[(3 + d) * Nq + pos] = q[d];
    }
    const int32_t sg = (int32_t)(j / nquad);
    seg[pos] = sg;
    if (f32_parts == 0) return;
    // hi parts and segment | lo parts and charge x | charge y, z
    const float h0 = (float)x[0], h1 = (float)x[1], h2 = (float)x[2];
    f32[pos] = make_float4(h0, h1, h2, __int_as_float(sg));
    if (f32_parts == 2) {
        f32[Nq + pos] = make_float4((float)(x[0] - h0), (float)(x[1] - h1), (float)(x[2] - h2), (float)q[0]);
        reinterpret_cast<float2*>(f32 + 2 * Nq)[pos] = make_float2((float)q[1], (float)q[2]);
    }
}

// Per-lane accumulators in the evaluation precision R; in FP32 they are Kahan-compensated
// (c holds the running compensation), in FP64 plain sums.
template <typename R>
struct PairAcc {
    R v[3], p[3];
    R cv[3], cp[3];
    unsigned long long inr, cand;
};

template <typename R>
__device__ __forceinline__ void acc_add(R& s, R& c, R x) {
    if constexpr (std::is_same<R, float>::value) {
        const R y = x - c;
        const R t = s + y;
        c = (t - s) - y;
        s = t;
    } else {
        s += x;
    }
}

__device__ __forceinline__ void ewald_weights_f(const KParams& K, float x, float& a, float& g) {
    int k = (int)(x * (float)kEwaldInvH);
    k = k < K.ewald_ntab ? k : K.ewald_ntab - 1;
    const float t = x - (k + 0.5f) * (float)kEwaldH;
    const float* ce = K.ewald_tab_f + k * kEwaldNCf;
    const float* cg = K.ewald_tab_f + (K.ewald_ntab + k) * kEwaldNCf;
    a = __ldg(ce + kEwaldNCf - 1);
    g = __ldg(cg + kEwaldNCf - 1);
#pragma unroll
    for (int n = kEwaldNCf - 2; n >= 0; --n) {
        a = fmaf(a, t, __ldg(ce + n));
        g = fmaf(g, t, __ldg(cg + n));
    }
}

// ---- naive pair kernel (periodic, without cell lists) ----
// Per-warp queue of in-range pairs: the separations and source indices of candidates that
// passed the r^2 <= r_cut^2 test are compacted here (ballot + prefix popcount), so that the
// erfc/exp evaluation always runs on 32 live lanes instead of on the ~30% of lanes whose
// candidate happened to be in range.
constexpr int kPairThreads = 256;
constexpr int kQueue = 64;
struct PairQueue {
    double r[3][kQueue];
    int32_t j[kQueue];
};

// Pair integrand of entry k of the queue (short_range_integrand, integrands.jl:2-18).  R is
// the evaluation precision: the separation was formed in FP64 and is cast to R here.
template <bool VEL, bool PSI, typename R>
__device__ __forceinline__ void pair_eval(const KParams& K, const double* __restrict__ src, int64_t Ns,
                                          const PairQueue& Q, int k, PairAcc<R>& acc) {
    const R r0 = (R)Q.r[0][k], r1 = (R)Q.r[1][k], r2 = (R)Q.r[2][k];
    const int64_t j = Q.j[k];
    const R q0 = (R)src[3 * Ns + j], q1 = (R)src[4 * Ns + j], q2 = (R)src[5 * Ns + j];
    R rinv, wa = 1, wg = 1;  // erfc(alpha r) and erfc(alpha r) + 2/sqrt(pi) alpha r exp(-(alpha r)^2)
    if constexpr (std::is_same<R, float>::value) {
        rinv = rsqrtf(r0 * r0 + r1 * r1 + r2 * r2);
        if (K.ewald_ntab > 0) ewald_weights_f(K, (float)K.alpha / rinv, wa, wg);
    } else {
        const double r = sqrt(r0 * r0 + r1 * r1 + r2 * r2);
        rinv = 1.0 / r;
        if (K.ewald_ntab > 0) ewald_weights(K, K.alpha * r, wa, wg);
    }
    if (VEL) {
        const R f = wg * rinv * rinv * rinv;
        acc_add<R>(acc.v[0], acc.cv[0], f * (q1 * r2 - q2 * r1));
        acc_add<R>(acc.v[1], acc.cv[1], f * (q2 * r0 - q0 * r2));
        acc_add<R>(acc.v[2], acc.cv[2], f * (q0 * r1 - q1 * r0));
    }
    if (PSI) {
        const R f = wa * rinv;
        acc_add<R>(acc.p[0], acc.cp[0], f * q0);
        acc_add<R>(acc.p[1], acc.cp[1], f * q1);
        acc_add<R>(acc.p[2], acc.cp[2], f * q2);
    }
}

template <bool VEL, bool PSI, typename R>
__device__ __forceinline__ void pair_range_q(const KParams& K, const double x[3], int64_t i, int32_t iprev,
                                             bool skip_local, const double* __restrict__ src, int64_t Ns,
                                             const int32_t* __restrict__ seg, int64_t b, int64_t e, int lane,
                                             PairAcc<R>& acc, PairQueue& Q, int& qcount) {
    for (int64_t base = b; base < e; base += 32) {
        const int64_t j = base + lane;
        bool inr = false;
        double r0 = 0, r1 = 0, r2 = 0;
        if (j < e && !(skip_local && (seg[j] == i || seg[j] == iprev))) {
            r0 = deper(x[0] - src[j], K.L[0], K.Lh[0], K.open_domain);
            r1 = deper(x[1] - src[Ns + j], K.L[1], K.Lh[1], K.open_domain);
            r2 = deper(x[2] - src[2 * Ns + j], K.L[2], K.Lh[2], K.open_domain);
            acc.cand++;
            inr = r0 * r0 + r1 * r1 + r2 * r2 <= K.rcut2;
        }
        const unsigned m = __ballot_sync(0xffffffffu, inr);
        if (inr) {
            const int pos = qcount + __popc(m & ((1u << lane) - 1u));
            Q.r[0][pos] = r0;
            Q.r[1][pos] = r1;
            Q.r[2][pos] = r2;
            Q.j[pos] = (int32_t)j;
            acc.inr++;
        }
        qcount += __popc(m);
        __syncwarp();
        if (qcount >= 32) {
            pair_eval<VEL, PSI, R>(K, src, Ns, Q, lane, acc);
            __syncwarp();
            const int rest = qcount - 32;
            if (lane < rest) {
                Q.r[0][lane] = Q.r[0][32 + lane];
                Q.r[1][lane] = Q.r[1][32 + lane];
                Q.r[2][lane] = Q.r[2][32 + lane];
                Q.j[lane] = Q.j[32 + lane];
            }
            __syncwarp();
            qcount = rest;
        }
    }
}

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

__device__ __forceinline__ unsigned long long warp_sum_u(unsigned long long v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// All pairs of an open domain (no splitting: the full Biot-Savart integrand, no cut-off).  A CTA takes 128
// nodes and four groups of threads, a thread per node in each, that deal the sources of a tile in shared memory
// out among them (a source is broadcast to a warp).  blockIdx.y takes its share of the sources, so that few nodes
// still fill the device.  The groups' sums are added in their order; the shares' sums go to `part` and the last
// CTA of a block of nodes to arrive (arrive[blockIdx.x], zeroed by the local term's kernel) adds them in the order
// of the shares: the same call gives the same bits each time.  Bound: the FP64 pipe (about 30 instructions per pair).  Against one
// group per CTA and atomic sums, whose order varied: 30,000 nodes 4.74 -> 4.50 ms, 4,014 nodes 0.164 -> 0.168.
constexpr int kOpenNodes = 128;
constexpr int kOpenGroups = 4;
constexpr int kOpenThreads = kOpenNodes * kOpenGroups;
constexpr int kOpenTile = 512;
constexpr int kOpenBlocks = 2;  // CTAs per SM
constexpr int kArrive = 4;      // words of vpbs_handle::counters before the arrivals per block of nodes

template <bool VEL, bool PSI>
__global__ void __launch_bounds__(kOpenThreads, kOpenBlocks) pair_open_kernel(
    int64_t Np, int64_t Ns, int per, double pref, const double* __restrict__ nodes, const double* __restrict__ points,
    const double* __restrict__ charges, double* __restrict__ vel, double* __restrict__ psi, double* __restrict__ part,
    unsigned* __restrict__ arrive, unsigned long long* __restrict__ counters) {
    constexpr int NC = (VEL ? 3 : 0) + (PSI ? 3 : 0);
    __shared__ double2 pxy[kOpenTile], pzq[kOpenTile], qyz[kOpenTile];
    __shared__ double sums[kOpenGroups - 1][NC][kOpenNodes];
    __shared__ bool last;
    __shared__ unsigned sources;  // of this share, those that take part in pairs
    const int local = threadIdx.x % kOpenNodes, group = threadIdx.x / kOpenNodes;
    const int64_t i = (int64_t)blockIdx.x * kOpenNodes + local;
    const int64_t ic = i < Np ? i : Np - 1;
    const double x0 = nodes[ic], x1 = nodes[Np + ic], x2 = nodes[2 * Np + ic];
    const int64_t j0 = (int64_t)blockIdx.y * per, j1 = j0 + per < Ns ? j0 + per : Ns;
    double v0 = 0, v1 = 0, v2 = 0, p0 = 0, p1 = 0, p2 = 0;
    unsigned mine = 0;
    if (threadIdx.x == 0) sources = 0;
    for (int64_t jt = j0; jt < j1; jt += kOpenTile) {
        const int n = j1 - jt < kOpenTile ? (int)(j1 - jt) : kOpenTile;
        __syncthreads();
        for (int t = threadIdx.x; t < n; t += kOpenThreads) {
            const int64_t j = jt + t;
            double s0 = points[j], s1 = points[Ns + j], s2 = points[2 * Ns + j];
            double q0 = charges[j], q1 = charges[Ns + j], q2 = charges[2 * Ns + j];
            if (!(s0 == s0 && s1 == s1 && s2 == s2)) {  // a NaN position takes part in no pair
                s0 = s1 = s2 = 1e100;
                q0 = q1 = q2 = 0.0;
            } else {
                ++mine;
            }
            pxy[t] = make_double2(s0, s1);
            pzq[t] = make_double2(s2, q0);
            qyz[t] = make_double2(q1, q2);
        }
        __syncthreads();
#pragma unroll 4
        for (int t = group; t < n; t += kOpenGroups) {
            const double2 a = pxy[t], b = pzq[t], c = qyz[t];
            const double r0 = x0 - a.x, r1 = x1 - a.y, r2 = x2 - b.x;
            const double rinv = rsqrt(r0 * r0 + r1 * r1 + r2 * r2);
            if (VEL) {
                const double f = rinv * rinv * rinv;
                v0 += f * (c.x * r2 - c.y * r1);
                v1 += f * (c.y * r0 - b.y * r2);
                v2 += f * (b.y * r1 - c.x * r0);
            }
            if (PSI) {
                p0 += rinv * b.y;
                p1 += rinv * c.x;
                p2 += rinv * c.y;
            }
        }
    }
    const int takers = __syncthreads_count(group == 0 && i < Np && x0 == x0 && x1 == x1 && x2 == x2);
    if (mine) atomicAdd(&sources, mine);
    double f[6] = {VEL ? v0 : p0, VEL ? v1 : p1, VEL ? v2 : p2, p0, p1, p2};
    if (group > 0)
#pragma unroll
        for (int c = 0; c < NC; ++c) sums[group - 1][c][local] = f[c];
    __syncthreads();
    if (threadIdx.x == 0) {
        atomicAdd(&counters[0], (unsigned long long)takers * sources);
        if (blockIdx.x == 0 && blockIdx.y == 0) counters[1] = (unsigned long long)Np * (unsigned long long)Ns;
    }
    if (group == 0)
#pragma unroll
        for (int c = 0; c < NC; ++c) {
#pragma unroll
            for (int g = 0; g < kOpenGroups - 1; ++g) f[c] += sums[g][c][local];
            f[c] *= pref;
        }
    if (gridDim.y > 1) {
        if (group == 0) {
            if (i < Np)
#pragma unroll
                for (int c = 0; c < NC; ++c) part[((int64_t)blockIdx.y * NC + c) * Np + i] = f[c];
            __threadfence();
        }
        __syncthreads();
        if (threadIdx.x == 0) last = atomicAdd(&arrive[blockIdx.x], 1u) == gridDim.y - 1;
        __syncthreads();
        if (!last) return;
        __threadfence();
#pragma unroll
        for (int c = 0; c < NC; ++c) f[c] = 0.0;
        if (group == 0)
#pragma unroll 4
            for (unsigned y = 0; y < gridDim.y; ++y)
#pragma unroll
                for (int c = 0; c < NC; ++c) f[c] += __ldcg(&part[((int64_t)y * NC + c) * Np + ic]);
    }
    if (group == 0 && i < Np) {
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            if (VEL) vel[c * Np + i] += f[c];
            if (PSI) psi[c * Np + i] += f[VEL ? 3 + c : c];
        }
    }
}

// One warp per destination node (visited in cell order when cell lists are used).  R = double
// for the plain form, float for the mixed form (separations always formed in FP64).
template <bool VEL, bool PSI, typename R>
__global__ void __launch_bounds__(256) pair_kernel(
    KParams K, CellGrid cg, int64_t Np, int64_t Ns, const int32_t* __restrict__ dst_order,
    const double* __restrict__ nodes, const int32_t* __restrict__ idx_prev, const double* __restrict__ src,
    const int32_t* __restrict__ src_start, const int32_t* __restrict__ seg, int use_cells, int skip_local,
    double* __restrict__ vel, double* __restrict__ psi, unsigned long long* __restrict__ counters) {
    __shared__ PairQueue queues[kPairThreads / 32];
    const int lane = threadIdx.x & 31;
    const int64_t w = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (w >= Np) return;
    PairQueue& Q = queues[threadIdx.x >> 5];
    int qcount = 0;
    const int64_t i = use_cells ? dst_order[w] : w;
    const double x[3] = {nodes[i], nodes[Np + i], nodes[2 * Np + i]};
    const int32_t iprev = idx_prev[i];
    PairAcc<R> acc = {{0, 0, 0}, {0, 0, 0}, {0, 0, 0}, {0, 0, 0}, 0ull, 0ull};
    if (!use_cells) {
        pair_range_q<VEL, PSI, R>(K, x, i, iprev, skip_local, src, Ns, seg, 0, Ns, lane, acc, Q, qcount);
    } else {
        const int M = cg.M;
        const int nc0 = cg.nc[0], nc1 = cg.nc[1], nc2 = cg.nc[2];
        const int cx = cell_coord(x[0], K.L[0], nc0);
        const int cy = cell_coord(x[1], K.L[1], nc1);
        const int cz = cell_coord(x[2], K.L[2], nc2);
        for (int dz = -M; dz <= M; ++dz) {
            int zz = cz + dz;
            zz = zz < 0 ? zz + nc2 : (zz >= nc2 ? zz - nc2 : zz);
            for (int dy = -M; dy <= M; ++dy) {
                int yy = cy + dy;
                yy = yy < 0 ? yy + nc1 : (yy >= nc1 ? yy - nc1 : yy);
                const int64_t base = ((int64_t)zz * nc1 + yy) * nc0;
                const int lo = cx - M * cg.G, hi = cx + M * cg.G;  // M cells = M G slabs in x
                if (lo >= 0 && hi < nc0) {
                    pair_range_q<VEL, PSI, R>(K, x, i, iprev, skip_local, src, Ns, seg, src_start[base + lo],
                                         src_start[base + hi + 1], lane, acc, Q, qcount);
                } else if (lo < 0) {
                    pair_range_q<VEL, PSI, R>(K, x, i, iprev, skip_local, src, Ns, seg, src_start[base + lo + nc0],
                                         src_start[base + nc0], lane, acc, Q, qcount);
                    pair_range_q<VEL, PSI, R>(K, x, i, iprev, skip_local, src, Ns, seg, src_start[base],
                                         src_start[base + hi + 1], lane, acc, Q, qcount);
                } else {
                    pair_range_q<VEL, PSI, R>(K, x, i, iprev, skip_local, src, Ns, seg, src_start[base + lo],
                                         src_start[base + nc0], lane, acc, Q, qcount);
                    pair_range_q<VEL, PSI, R>(K, x, i, iprev, skip_local, src, Ns, seg, src_start[base],
                                         src_start[base + hi - nc0 + 1], lane, acc, Q, qcount);
                }
            }
        }
    }
    if (lane < qcount) pair_eval<VEL, PSI, R>(K, src, Ns, Q, lane, acc);  // queue remainder
    const double pref = K.Gamma / (4.0 * kPi);
    double v0 = 0, v1 = 0, v2 = 0, p0 = 0, p1 = 0, p2 = 0;
    // lane partial sums (compensated in FP32) are reduced across the warp in FP64
    auto lane_total = [](R s, R c) { return (double)s - (double)c; };
    if (VEL) {
        v0 = warp_sum(lane_total(acc.v[0], acc.cv[0]));
        v1 = warp_sum(lane_total(acc.v[1], acc.cv[1]));
        v2 = warp_sum(lane_total(acc.v[2], acc.cv[2]));
    }
    if (PSI) {
        p0 = warp_sum(lane_total(acc.p[0], acc.cp[0]));
        p1 = warp_sum(lane_total(acc.p[1], acc.cp[1]));
        p2 = warp_sum(lane_total(acc.p[2], acc.cp[2]));
    }
    unsigned long long inr = warp_sum_u(acc.inr), cand = warp_sum_u(acc.cand);
    if (lane == 0) {
        if (VEL) { vel[i] += pref * v0; vel[Np + i] += pref * v1; vel[2 * Np + i] += pref * v2; }
        if (PSI) { psi[i] += pref * p0; psi[Np + i] += pref * p1; psi[2 * Np + i] += pref * p2; }
        atomicAdd(&counters[0], inr);
        atomicAdd(&counters[1], cand);
    }
}

// ---- pair kernels over cell lists: common parts ----
constexpr double kScreenMargin = 2e-5;  // of r_cut^2, on top of the rounding of the FP32 places
constexpr size_t kPairSmemMost = 200 * 1024;  // tables of an FP64 pair-kernel CTA

// 1/sqrt(s) in FP64: FP32 hardware estimate refined by two Newton-Raphson steps
// y <- y (3 - s y^2) / 2 (quadratic convergence: ~1e-7 -> ~1e-14 -> rounding level).
__device__ __forceinline__ double rsqrt_nr(double s) {
    double y = (double)rsqrtf((float)s);
    double t = s * y;
    y = y * fma(-0.5 * t, y, 1.5);
    t = s * y;
    y = y * fma(-0.5 * t, y, 1.5);
    return y;
}

// Both Ewald weights from the interleaved table (one 16-byte load per degree).
__device__ __forceinline__ void ewald_weights2(const KParams& K, double x, double& a, double& g) {
    int k = (int)(x * kEwaldInvH);
    k = k < K.ewald_ntab ? k : K.ewald_ntab - 1;
    const double t = x - (k + 0.5) * kEwaldH;
    const double2* c = K.ewald_tab2 + k * kEwaldNC;
    double2 v = __ldg(c + kEwaldNC - 1);
    a = v.x;
    g = v.y;
#pragma unroll
    for (int n = kEwaldNC - 2; n >= 0; --n) {
        v = __ldg(c + n);
        a = fma(a, t, v.x);
        g = fma(g, t, v.y);
    }
}

// Interval and local coordinate of x in the shared-memory tables (intervals centred at k / 128):
// k = round(128 x) by the 1.5 * 2^52 trick, t = 128 x - k in [-1/2, 1/2].
__host__ __device__ __forceinline__ double tab_s_pos(double x, int ntab, int* k) {
    const double y = fma(x, kTabSInvH, 6755399441055744.0);
#if defined(__CUDA_ARCH__)
    const unsigned kk = (unsigned)__double2loint(y);
#else
    uint64_t bits;
    std::memcpy(&bits, &y, sizeof bits);
    const unsigned kk = (unsigned)bits;
#endif
    const unsigned top = (unsigned)(ntab - 1);
    *k = (int)(kk < top ? kk : top);
    return fma(x, kTabSInvH, -(y - 6755399441055744.0));
}

__host__ __device__ __forceinline__ double tab_s_poly(const double* c, double t) {
    const double2* v = reinterpret_cast<const double2*>(c);
    const double2 c0 = v[0], c1 = v[1], c2 = v[2];
    return fma(fma(fma(fma(fma(c2.y, t, c2.x), t, c1.y), t, c1.x), t, c0.y), t, c0.x);
}

// ---- FP32 pair kernel of the mixed form ----
// Every per-pair operation in FP32.  A warp works on its own, without tiles or barriers: it takes D nodes
// that follow one another in cell order, finds the runs of cell-sorted sources within r_cut of their
// bounding box (a lane per row of cells) and reads them, as FP32 hi + lo parts that the cell sort wrote,
// through the L1 cache (neighbouring warps read the same rows).
//  * Each 32 sources are loaded once and screened against the D nodes in turn, two nodes per packed
//    instruction, on the hi parts against r_cut^2 (1 + margin).
//  * The survivors (one in six) go to the warp's queue of that node and are evaluated 32 at a time:
//    separation (x_hi - s_hi) + (x_lo - s_lo) -- the FP64 separation rounded to FP32 within ~2 ulps;
//    periodic images shift the node (its hi + lo parts at x - L, x, x + L are tabulated, each from FP64).
//  * Decision r^2 <= r_cut^2 in FP32, redone in FP64 from the hi + lo parts when r^2 lies within
//    4e-6 r_cut^2 of the cut-off, so the pair set equals the FP64 one; the node's own two segments are
//    left out (the mixed form always takes their long-range part out explicitly).
//  * Weights from cubic tables on 1/32-wide intervals in x = alpha r (FP32, ~3e-8 absolute),
//    interval index without a conversion instruction.
//  * Per-lane FP32 sums over the rows of some kF32Flush evaluations per node, FP32 warp reduction (the D x 3 sums
//    halved from lane half to lane half), FP64 output sums, so that the rounding does not grow with a node's
//    pairs (20,000 a node: streamfunction error 1.3e-7 with one sum per lane, 0.5e-7 so, at the same time;
//    asking after every 32 sources instead of every row costs 3 %).
// blockIdx.y: the rows are dealt to gridDim.y warps where a system has too few nodes to fill the device.
// Bound: issue slots (81 % busy, 10 warp instructions per pair in range; 1M nodes, 155 M pairs: 1.76 ms).
// CTAs that stage tiles of a block's neighbourhood and take a node per warp at a time: 14 instructions per
// pair, a fifth of the time at barriers, 2.89 ms.  D = 4 at 64 registers (32 warps per SM) against D = 8 at
// 80: 2.09 ms, at 128: 2.48, D = 2: 2.18; evaluating a chunk as soon as one lane is in range, unqueued: 2.89.
constexpr float kF32Band = 4e-6f; // relative band around r_cut^2 decided in FP64
constexpr float kF32Far = 1e18f;  // coordinate of an absent node or source (its square is finite)
constexpr int kF32Flush = 16;
constexpr int kF32Warps = 4;
constexpr int kF32Blocks = 8;  // CTAs per SM (64 registers)
// A queue entry: the source's cell-sorted index and above it 2 bits each for its image in x, y and z (0, 1,
// 2: -L, 0, +L).  32-bit entries hold 2^26 sources, larger systems take 64-bit ones.
template <typename E>
constexpr int kIndexBits = sizeof(E) == 4 ? 26 : 32;
template <typename E>
__device__ __forceinline__ uint32_t entry_source(E e) { return (uint32_t)(e & (((E)1 << kIndexBits<E>) - 1)); }
template <typename E>
__device__ __forceinline__ int entry_image(E e, int dim) { return (int)(e >> (kIndexBits<E> + 2 * dim)) & 3; }


__device__ __forceinline__ float rsqrt_fast(float x) {
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// Two FP32 values in one register pair, and the packed operations on them (each half rounded as the
// scalar operation).
using f32x2 = unsigned long long;
__device__ __forceinline__ f32x2 dup2(float a) {
    f32x2 r;
    asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(a));
    return r;
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ float half2f(f32x2 a, int u) { return __uint_as_float((unsigned)(u ? a >> 32 : a)); }

template <typename E>
struct F32Warp {
    float2 x[4][3][3];       // node, dimension, image (-L, 0, +L): hi and lo parts of the node's place
    int2 id[4];              // node and previous node
    ulonglong2 xy2[2];       // hi parts of two nodes in the images of the current row: x, x | y, y
    f32x2 z2[2];
    E queue[4][64];          // per node: screened sources
};

// 32 queued pairs (one a lane; `live` false for lanes past the queue's end) of one node.
template <bool VEL, bool PSI, typename E>
__device__ __forceinline__ void f32_eval(const F32Warp<E>& S, int d, int e, bool live, const float4* __restrict__ srcP,
                                         const float4* __restrict__ srcQ, const float2* __restrict__ srcR,
                                         const float4* __restrict__ tab, float rc2lo, float rc2hi, double rcut2, float alpha,
                                         int nf, float (&v)[3], float (&w)[3], int& ninr) {
    const E entry = S.queue[d][e];
    const uint32_t j = entry_source(entry);
    const float4 p = __ldg(srcP + j), q = __ldg(srcQ + j);
    const float2 qr = __ldg(srcR + j);
    const float2 x0 = S.x[d][0][entry_image(entry, 0)], x1 = S.x[d][1][entry_image(entry, 1)],
                 x2 = S.x[d][2][entry_image(entry, 2)];
    const int2 id = S.id[d];
    const float d0 = (x0.x - p.x) + (x0.y - q.x), d1 = (x1.x - p.y) + (x1.y - q.y), d2 = (x2.x - p.z) + (x2.y - q.z);
    const float s2 = fmaf(d0, d0, fmaf(d1, d1, d2 * d2));
    live = live && __float_as_int(p.w) != id.x && __float_as_int(p.w) != id.y;
    bool ok = live && s2 <= rc2lo;
    const bool near = live && !ok && s2 <= rc2hi;
    if (__any_sync(0xffffffffu, near)) {
        if (near) {  // the FP64 decision on the hi + lo separation (rare)
            const double f0 = ((double)x0.x + (double)x0.y) - ((double)p.x + (double)q.x);
            const double f1 = ((double)x1.x + (double)x1.y) - ((double)p.y + (double)q.y);
            const double f2 = ((double)x2.x + (double)x2.y) - ((double)p.z + (double)q.z);
            ok = f0 * f0 + f1 * f1 + f2 * f2 <= rcut2;
        }
    }
    const float rinv = rsqrt_fast(s2);
    int k;
    float tt;
    f32_table_pos(s2 * rinv * alpha, nf, &k, &tt);
    if (ok) ++ninr;
    if (VEL) {
        const float f = f32_cubic(tab[(PSI ? nf : 0) + k], tt) * (rinv * rinv * rinv);
        const float c0 = fmaf(qr.x, d2, -qr.y * d1), c1 = fmaf(qr.y, d0, -q.w * d2), c2 = fmaf(q.w, d1, -qr.x * d0);
        if (ok) {
            v[0] = fmaf(f, c0, v[0]);
            v[1] = fmaf(f, c1, v[1]);
            v[2] = fmaf(f, c2, v[2]);
        }
    }
    if (PSI) {
        const float f = f32_cubic(tab[k], tt) * rinv;
        if (ok) {
            w[0] = fmaf(f, q.w, w[0]);
            w[1] = fmaf(f, qr.x, w[1]);
            w[2] = fmaf(f, qr.y, w[2]);
        }
    }
}

// Sums of v[n][3] over the warp's lanes, n = D a power of two: lane halves exchange halves of the n
// until a lane holds one of them (number lane / (32 / D)); every lane of its 32 / D has the total.
template <int D, typename T>
__device__ __forceinline__ void group_reduce(T (&v)[D][3], int lane, T (&out)[3]) {
#pragma unroll
    for (int h = D / 2, o = 16; h >= 1; h >>= 1, o >>= 1) {
        const bool up = lane & o;
#pragma unroll
        for (int i = 0; i < h; ++i)
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                const T keep = up ? v[h + i][c] : v[i][c], give = up ? v[i][c] : v[h + i][c];
                v[i][c] = keep + __shfl_xor_sync(0xffffffffu, give, o);
            }
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        T x = v[0][c];
#pragma unroll
        for (int o = 16 / D; o >= 1; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
        out[c] = x;
    }
}

// Sources near a group of nodes of one (y, z) row of cells: row r (of the W^2 around it) as the unwrapped
// slab range [klo, khi] within r_cut of the group's bounding box [lo, hi], the index of its first slab, and
// its periodic image in y and z (0, 1, 2: -L, 0, +L; y + 3 z).
struct RowRange {
    int klo, khi, row, iyz;
};
__device__ __forceinline__ RowRange near_row(const CellGrid& cg, const KParams& K, int r, int gy, int gz,
                                             const float (&lo)[3], const float (&hi)[3], float slack) {
    const int M = cg.M, W = 2 * M + 1, nc0 = cg.nc[0], nc1 = cg.nc[1], nc2 = cg.nc[2];
    RowRange R{0, -1, 0, 0};
    if (r >= W * W) return R;
    const int yu = gy + r % W - M, zu = gz + r / W - M;
    const float h1 = (float)(K.L[1] / nc1), h2 = (float)(K.L[2] / nc2), rc = (float)K.rcut;
    const float ylo = (float)yu * h1, zlo = (float)zu * h2;
    const float ey = fmaxf(fmaxf(ylo - hi[1], lo[1] - (ylo + h1)), 0.0f);
    const float ez = fmaxf(fmaxf(zlo - hi[2], lo[2] - (zlo + h2)), 0.0f);
    const float rest = rc * rc * 1.0001f - ey * ey - ez * ez;
    if (rest >= 0.0f) {
        const float w = sqrtf(rest) + slack;
        const double inv_hx = nc0 / K.L[0];
        R.klo = (int)floor((double)(lo[0] - w) * inv_hx);
        R.khi = (int)floor((double)(hi[0] + w) * inv_hx);
    }
    const int my = yu < 0 ? 0 : (yu >= nc1 ? 2 : 1), mz = zu < 0 ? 0 : (zu >= nc2 ? 2 : 1);
    R.row = ((zu + (1 - mz) * nc2) * nc1 + yu + (1 - my) * nc1) * nc0;
    R.iyz = my + 3 * mz;
    return R;
}

// Bounding box of the lanes with `mine` among the first D, widened by `slack`, on every lane.
template <int D>
__device__ __forceinline__ void group_box(bool mine, const double (&x)[3], float slack, float (&lo)[3], float (&hi)[3]) {
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        lo[d] = mine ? (float)x[d] : kF32Far;
        hi[d] = mine ? (float)x[d] : -kF32Far;
    }
#pragma unroll
    for (int o = 1; o < D; o <<= 1)
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            lo[d] = fminf(lo[d], __shfl_xor_sync(0xffffffffu, lo[d], o));
            hi[d] = fmaxf(hi[d], __shfl_xor_sync(0xffffffffu, hi[d], o));
        }
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        lo[d] = __shfl_sync(0xffffffffu, lo[d], 0) - slack;
        hi[d] = __shfl_sync(0xffffffffu, hi[d], 0) + slack;
    }
}

template <bool VEL, bool PSI, int D, typename E>
__global__ void __launch_bounds__(32 * kF32Warps, sizeof(E) == 4 ? kF32Blocks : 6) pair_f32_kernel(
    KParams K, CellGrid cg, int64_t Np, float rc2s, const int32_t* __restrict__ dst_start,
    const int32_t* __restrict__ dst_order, const double* __restrict__ nodes, const int32_t* __restrict__ idx_prev,
    const float4* __restrict__ srcP, const float4* __restrict__ srcQ, const float2* __restrict__ srcR,
    const int32_t* __restrict__ src_start, double* __restrict__ vel, double* __restrict__ psi,
    unsigned long long* __restrict__ counters) {
    __shared__ F32Warp<E> warps[kF32Warps];
    __shared__ float4 tab[(VEL && PSI ? 2 : 1) * kF32TabMax];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int nf = K.ntab_c;
    for (int k = threadIdx.x; k < (VEL && PSI ? 2 : 1) * nf; k += 32 * kF32Warps) tab[k] = K.tab_c[(VEL && !PSI ? nf : 0) + k];
    __syncthreads();
    F32Warp<E>& S = warps[warp];
    const int64_t first = ((int64_t)blockIdx.x * kF32Warps + warp) * D;
    const int64_t nvalid = dst_start[cg.ncell];  // nodes of the sentinel cell (non-finite) come after these
    if (first >= nvalid) return;
    const int nd = nvalid - first < D ? (int)(nvalid - first) : D;
    const int M = cg.M, nc0 = cg.nc[0], nc1 = cg.nc[1], nc2 = cg.nc[2], W = 2 * M + 1;
    double x[3] = {0.0, 0.0, 0.0};
    int i = -1, cy = 0, cz = 0;
    if (lane < nd) {
        i = dst_order[first + lane];
        S.id[lane] = make_int2(i, idx_prev[i]);
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            x[d] = nodes[d * Np + i];
#pragma unroll
            for (int m = 0; m < 3; ++m) {  // a source image at p + s meets the node at x - s
                const double y = x[d] - (double)(m - 1) * K.L[d];
                const float hi = (float)y;
                S.x[lane][d][m] = make_float2(hi, (float)(y - hi));
            }
        }
        cy = cell_coord(x[1], K.L[1], nc1);
        cz = cell_coord(x[2], K.L[2], nc2);
    }
    const float rc = (float)K.rcut;
    // slack of the row and slab ranges, far above the FP32 rounding of places in the box
    const float slack = 1e-5f * rc + 1e-6f * (float)fmax(K.L[0], fmax(K.L[1], K.L[2]));
    const float rc2lo = (float)(K.rcut2 * (1.0 - (double)kF32Band)), rc2hi = (float)(K.rcut2 * (1.0 + (double)kF32Band));
    const float alpha = (float)K.alpha;
    const unsigned lanelt = (1u << lane) - 1u;
    int ninr = 0;
    unsigned ncand = 0;
    float v[D][3], w[D][3];
    int cnt[D];  // queued pairs per node (warp-uniform)
#pragma unroll
    for (int d = 0; d < D; ++d) {
        cnt[d] = 0;
#pragma unroll
        for (int c = 0; c < 3; ++c) v[d][c] = w[d][c] = 0.0f;
    }
    // the lanes' FP32 sums to the FP64 outputs
    const double pref = K.Gamma / (4.0 * kPi);
    const int slot = lane / (32 / D);
    const int is = __shfl_sync(0xffffffffu, i, slot);
    int nev = 0;  // evaluations since the last flush (warp-uniform)
    auto flush = [&]() {
        float out[3];
        if (VEL) {
            group_reduce<D>(v, lane, out);
            if (lane % (32 / D) == 0 && is >= 0)
                for (int c = 0; c < 3; ++c) atomicAdd(&vel[c * Np + is], pref * (double)out[c]);
        }
        if (PSI) {
            group_reduce<D>(w, lane, out);
            if (lane % (32 / D) == 0 && is >= 0)
                for (int c = 0; c < 3; ++c) atomicAdd(&psi[c * Np + is], pref * (double)out[c]);
        }
#pragma unroll
        for (int d = 0; d < D; ++d)
#pragma unroll
            for (int c = 0; c < 3; ++c) v[d][c] = w[d][c] = 0.0f;
        nev = 0;
    };
    int turn = 0;  // rows seen so far: dealt to the gridDim.y warps of the group in turn
    // the nodes of one (y, z) row of cells within r_cut in x at a time (nearly always all of them)
    for (unsigned todo = __ballot_sync(0xffffffffu, lane < nd); todo;) {
        const int lead = __ffs(todo) - 1;
        const int gy_ = __shfl_sync(0xffffffffu, cy, lead), gz_ = __shfl_sync(0xffffffffu, cz, lead);
        const double xlead = __shfl_sync(0xffffffffu, x[0], lead);
        const bool mine = (todo >> lane & 1) && cy == gy_ && cz == gz_ && fabs(x[0] - xlead) <= K.rcut;
        const unsigned members = __ballot_sync(0xffffffffu, mine);
        todo &= ~members;
        float lo[3], hi[3];
        group_box<D>(mine, x, slack, lo, hi);
        for (int r0 = 0; r0 < W * W; r0 += 32) {  // a lane per row of cells around the nodes' own
        const RowRange R = near_row(cg, K, r0 + lane, gy_, gz_, lo, hi, slack);
        for (int mx = 0; mx < 3; ++mx) {  // images in x: -L, 0, +L
            const int s0 = max(R.klo - (mx - 1) * nc0, 0), s1 = min(R.khi - (mx - 1) * nc0, nc0 - 1);
            int a = 0, b = 0;
            if (s0 <= s1) {
                a = src_start[R.row + s0];
                b = src_start[R.row + s1 + 1];
            }
            for (unsigned rows = __ballot_sync(0xffffffffu, a < b); rows; rows &= rows - 1) {
                const bool skip = turn % (int)gridDim.y != (int)blockIdx.y;  // warp-uniform
                ++turn;
                if (skip) continue;
                const int sl = __ffs(rows) - 1;
                const int ra = __shfl_sync(0xffffffffu, a, sl), rb = __shfl_sync(0xffffffffu, b, sl);
                const int im = __shfl_sync(0xffffffffu, R.iyz, sl), my = im % 3, mz = im / 3;
                __syncwarp();
                if (lane < D) {
                    const float px = mine ? S.x[lane][0][mx].x : kF32Far;
                    float* xy = reinterpret_cast<float*>(S.xy2) + 4 * (lane >> 1) + (lane & 1);
                    xy[0] = px;
                    xy[2] = mine ? S.x[lane][1][my].x : kF32Far;
                    reinterpret_cast<float*>(S.z2)[lane] = mine ? S.x[lane][2][mz].x : kF32Far;
                }
                __syncwarp();
                ncand += (unsigned)(rb - ra) * __popc(members);
                const E code = (E)(mx | my << 2 | mz << 4) << kIndexBits<E>;
                float4 pn = __ldg(srcP + min(ra + lane, rb - 1));
                for (int base = ra; base < rb; base += 32) {
                    const int t = base + lane;
                    float4 p = pn;
                    pn = __ldg(srcP + min(t + 32, rb - 1));
                    if (t >= rb) p.x = -kF32Far;
                    const f32x2 px = dup2(-p.x), py = dup2(-p.y), pz = dup2(-p.z);
                    const E entry = (E)t | code;
#pragma unroll
                    for (int h = 0; h < D / 2; ++h) {
                        const ulonglong2 xy = S.xy2[h];
                        const f32x2 e0 = add2(xy.x, px), e1 = add2(xy.y, py), e2 = add2(S.z2[h], pz);
                        const f32x2 r2 = fma2(e0, e0, fma2(e1, e1, mul2(e2, e2)));
#pragma unroll
                        for (int u = 0; u < 2; ++u) {
                            const int d = 2 * h + u;
                            const bool in = half2f(r2, u) <= rc2s;
                            const unsigned m = __ballot_sync(0xffffffffu, in);
                            if (m == 0) continue;  // warp-uniform
                            if (in) S.queue[d][cnt[d] + __popc(m & lanelt)] = entry;
                            cnt[d] += __popc(m);
                            if (cnt[d] >= 32) {
                                __syncwarp();
                                f32_eval<VEL, PSI, E>(S, d, lane, true, srcP, srcQ, srcR, tab, rc2lo, rc2hi, K.rcut2, alpha, nf, v[d],
                                                   w[d], ninr);
                                ++nev;
                                cnt[d] -= 32;
                                __syncwarp();
                                if (lane < cnt[d]) S.queue[d][lane] = S.queue[d][32 + lane];
                                __syncwarp();
                            }
                        }
                    }
                }
                if (nev >= kF32Flush * D) flush();
            }
        }
        }
    }
    __syncwarp();
#pragma unroll
    for (int d = 0; d < D; ++d)
        if (cnt[d] > 0)  // warp-uniform
            f32_eval<VEL, PSI, E>(S, d, lane < cnt[d] ? lane : 0, lane < cnt[d], srcP, srcQ, srcR, tab, rc2lo, rc2hi, K.rcut2, alpha, nf,
                               v[d], w[d], ninr);
    flush();
    const unsigned long long total = warp_sum_u((unsigned long long)ninr);
    if (lane == 0) {
        atomicAdd(&counters[0], total);
        atomicAdd(&counters[1], (unsigned long long)ncand);
    }
}

// ---- FP64 pair kernel ----
// The same groups, rows, FP32 screen and queues; the evaluation reads the sources' FP64 positions and charges
// (cell-sorted arrays), decides r^2 <= r_cut^2 and evaluates in FP64 (Newton-refined reciprocal square root,
// weights from degree-5 tables in shared memory, one copy per CTA).  SKIP: the node's own two segments left
// out.  Bound: shared-memory and L1 wavefronts of the gathers (per 32 pairs about 30 for the weights' three
// 16-byte loads and 30 for the sources), then the FP64 pipe (17 cycles).  1M nodes, 3.13 G pairs: 27.6 ms (CTAs
// that stage tiles of a block's neighbourhood: 39.5; weight tables a quarter shorter, of 1/96, which leave more L1:
// 26.8); 20k nodes, both fields: 0.205 (0.517).  With those tables, three CTAs per SM of
// 80 registers: 28.7, two of 128: 30.6; both fields in four of 64: 0.217.
constexpr int kF64Warps = 8;
// CTAs per SM: 64 registers for one field (some spilled outside the loops), 80 for both
__host__ __device__ constexpr int f64_blocks(bool both) { return both ? 3 : 4; }

template <int D, typename E>
struct F64Warp {
    double x[D][3][3];      // node, dimension, image (-L, 0, +L)
    int2 id[D];             // node and previous node
    ulonglong2 xy2[D / 2];  // FP32 places of two nodes in the images of the current row: x, x | y, y
    f32x2 z2[D / 2];
    E queue[D][64];
};

template <bool VEL, bool PSI, bool SKIP, int D, typename E>
__device__ __forceinline__ void f64_eval(const KParams& K, const F64Warp<D, E>& S, int d, int e, bool live,
                                         const float4* __restrict__ srcP, const double* __restrict__ src, int64_t Ns,
                                         const double* __restrict__ tab, double (&v)[3], double (&w)[3], int& ninr) {
    const E entry = S.queue[d][e];
    const uint32_t j = entry_source(entry);
    const double* s = src + j;
    const double d0 = S.x[d][0][entry_image(entry, 0)] - __ldg(s);
    const double d1 = S.x[d][1][entry_image(entry, 1)] - __ldg(s + Ns);
    const double d2 = S.x[d][2][entry_image(entry, 2)] - __ldg(s + 2 * Ns);
    const double q0 = __ldg(s + 3 * Ns), q1 = __ldg(s + 4 * Ns), q2 = __ldg(s + 5 * Ns);
    double s2 = d0 * d0 + d1 * d1 + d2 * d2;
    bool ok = live && s2 <= K.rcut2;
    if (SKIP) {
        const int sg = __float_as_int(__ldg(&srcP[j].w));
        const int2 id = S.id[d];
        ok = ok && sg != id.x && sg != id.y;
    }
    if (!ok) s2 = K.rcut2;
    if (ok) ++ninr;
    const double rinv = rsqrt_nr(s2);
    int k;
    const double t = tab_s_pos(K.alpha * (s2 * rinv), K.ntab_s, &k);
    if (VEL) {
        const double f = tab_s_poly(tab + (PSI ? K.ntab_s + k : k) * kTabSNC, t) * rinv * rinv * rinv;
        if (ok) {
            v[0] += f * (q1 * d2 - q2 * d1);
            v[1] += f * (q2 * d0 - q0 * d2);
            v[2] += f * (q0 * d1 - q1 * d0);
        }
    }
    if (PSI) {
        const double f = tab_s_poly(tab + k * kTabSNC, t) * rinv;
        if (ok) {
            w[0] += f * q0;
            w[1] += f * q1;
            w[2] += f * q2;
        }
    }
}

template <bool VEL, bool PSI, bool SKIP, int D, typename E>
__global__ void __launch_bounds__(32 * kF64Warps, f64_blocks(VEL && PSI)) pair_f64_kernel(
    KParams K, CellGrid cg, int64_t Np, float rc2s, const int32_t* __restrict__ dst_start,
    const int32_t* __restrict__ dst_order, const double* __restrict__ nodes, const int32_t* __restrict__ idx_prev,
    const float4* __restrict__ srcP, const double* __restrict__ src, int64_t Ns, const int32_t* __restrict__ src_start,
    double* __restrict__ vel, double* __restrict__ psi,
    unsigned long long* __restrict__ counters) {
    extern __shared__ __align__(16) double tab[];  // weight tables: [weight][interval][kTabSNC]
    __shared__ F64Warp<D, E> warps[kF64Warps];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    {
        constexpr int from = VEL && !PSI ? 1 : 0, nw = VEL && PSI ? 2 : 1;
        const double2* s = reinterpret_cast<const double2*>(K.tab_s + (size_t)from * K.ntab_s * kTabSNC);
        for (int k = threadIdx.x; k < nw * K.ntab_s * kTabSNC / 2; k += 32 * kF64Warps) reinterpret_cast<double2*>(tab)[k] = s[k];
    }
    __syncthreads();
    F64Warp<D, E>& S = warps[warp];
    const int64_t first = ((int64_t)blockIdx.x * kF64Warps + warp) * D;
    const int64_t nvalid = dst_start[cg.ncell];  // nodes of the sentinel cell (non-finite) come after these
    if (first >= nvalid) return;
    const int nd = nvalid - first < D ? (int)(nvalid - first) : D;
    const int M = cg.M, nc0 = cg.nc[0], nc1 = cg.nc[1], nc2 = cg.nc[2], W = 2 * M + 1;
    double x[3] = {0.0, 0.0, 0.0};
    int i = -1, cy = 0, cz = 0;
    if (lane < nd) {
        i = dst_order[first + lane];
        S.id[lane] = make_int2(i, idx_prev[i]);
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            x[d] = nodes[d * Np + i];
#pragma unroll
            for (int m = 0; m < 3; ++m) S.x[lane][d][m] = x[d] - (double)(m - 1) * K.L[d];
        }
        cy = cell_coord(x[1], K.L[1], nc1);
        cz = cell_coord(x[2], K.L[2], nc2);
    }
    const float rc = (float)K.rcut;
    // slack of the row and slab ranges, far above the FP32 rounding of places in the box
    const float slack = 1e-5f * rc + 1e-6f * (float)fmax(K.L[0], fmax(K.L[1], K.L[2]));
    const unsigned lanelt = (1u << lane) - 1u;
    int ninr = 0;
    unsigned ncand = 0;
    double v[D][3], w[D][3];
    int cnt[D];  // queued pairs per node (warp-uniform)
#pragma unroll
    for (int d = 0; d < D; ++d) {
        cnt[d] = 0;
#pragma unroll
        for (int c = 0; c < 3; ++c) v[d][c] = w[d][c] = 0.0;
    }
    int turn = 0;  // rows seen so far: dealt to the gridDim.y warps of the group in turn
    // the nodes of one (y, z) row of cells within r_cut in x at a time (nearly always all of them)
    for (unsigned todo = __ballot_sync(0xffffffffu, lane < nd); todo;) {
        const int lead = __ffs(todo) - 1;
        const int gy_ = __shfl_sync(0xffffffffu, cy, lead), gz_ = __shfl_sync(0xffffffffu, cz, lead);
        const double xlead = __shfl_sync(0xffffffffu, x[0], lead);
        const bool mine = (todo >> lane & 1) && cy == gy_ && cz == gz_ && fabs(x[0] - xlead) <= K.rcut;
        const unsigned members = __ballot_sync(0xffffffffu, mine);
        todo &= ~members;
        float lo[3], hi[3];
        group_box<D>(mine, x, slack, lo, hi);
        for (int r0 = 0; r0 < W * W; r0 += 32) {  // a lane per row of cells around the nodes' own
        const RowRange R = near_row(cg, K, r0 + lane, gy_, gz_, lo, hi, slack);
        for (int mx = 0; mx < 3; ++mx) {  // images in x: -L, 0, +L
            const int s0 = max(R.klo - (mx - 1) * nc0, 0), s1 = min(R.khi - (mx - 1) * nc0, nc0 - 1);
            int a = 0, b = 0;
            if (s0 <= s1) {
                a = src_start[R.row + s0];
                b = src_start[R.row + s1 + 1];
            }
            for (unsigned rows = __ballot_sync(0xffffffffu, a < b); rows; rows &= rows - 1) {
                const bool skip = turn % (int)gridDim.y != (int)blockIdx.y;  // warp-uniform
                ++turn;
                if (skip) continue;
                const int sl = __ffs(rows) - 1;
                const int ra = __shfl_sync(0xffffffffu, a, sl), rb = __shfl_sync(0xffffffffu, b, sl);
                const int im = __shfl_sync(0xffffffffu, R.iyz, sl), my = im % 3, mz = im / 3;
                __syncwarp();
                if (lane < D) {
                    const float px = mine ? (float)S.x[lane][0][mx] : kF32Far;
                    float* xy = reinterpret_cast<float*>(S.xy2) + 4 * (lane >> 1) + (lane & 1);
                    xy[0] = px;
                    xy[2] = mine ? (float)S.x[lane][1][my] : kF32Far;
                    reinterpret_cast<float*>(S.z2)[lane] = mine ? (float)S.x[lane][2][mz] : kF32Far;
                }
                __syncwarp();
                ncand += (unsigned)(rb - ra) * __popc(members);
                const E code = (E)(mx | my << 2 | mz << 4) << kIndexBits<E>;
                float4 pn = __ldg(srcP + min(ra + lane, rb - 1));
                for (int base = ra; base < rb; base += 32) {
                    const int t = base + lane;
                    float4 p = pn;
                    pn = __ldg(srcP + min(t + 32, rb - 1));
                    if (t >= rb) p.x = -kF32Far;
                    const f32x2 px = dup2(-p.x), py = dup2(-p.y), pz = dup2(-p.z);
                    const E entry = (E)t | code;
#pragma unroll
                    for (int h = 0; h < D / 2; ++h) {
                        const ulonglong2 xy = S.xy2[h];
                        const f32x2 e0 = add2(xy.x, px), e1 = add2(xy.y, py), e2 = add2(S.z2[h], pz);
                        const f32x2 r2 = fma2(e0, e0, fma2(e1, e1, mul2(e2, e2)));
#pragma unroll
                        for (int u = 0; u < 2; ++u) {
                            const int d = 2 * h + u;
                            const bool in = half2f(r2, u) <= rc2s;
                            const unsigned m = __ballot_sync(0xffffffffu, in);
                            if (m == 0) continue;  // warp-uniform
                            if (in) S.queue[d][cnt[d] + __popc(m & lanelt)] = entry;
                            cnt[d] += __popc(m);
                            if (cnt[d] >= 32) {
                                __syncwarp();
                                f64_eval<VEL, PSI, SKIP, D, E>(K, S, d, lane, true, srcP, src, Ns, tab, v[d], w[d], ninr);
                                cnt[d] -= 32;
                                __syncwarp();
                                if (lane < cnt[d]) S.queue[d][lane] = S.queue[d][32 + lane];
                                __syncwarp();
                            }
                        }
                    }
                }
            }
        }
        }
    }
    __syncwarp();
#pragma unroll
    for (int d = 0; d < D; ++d)
        if (cnt[d] > 0)  // warp-uniform
            f64_eval<VEL, PSI, SKIP, D, E>(K, S, d, lane < cnt[d] ? lane : 0, lane < cnt[d], srcP, src, Ns, tab, v[d], w[d], ninr);
    const double pref = K.Gamma / (4.0 * kPi);
    const int slot = lane / (32 / D);
    const int is = __shfl_sync(0xffffffffu, i, slot);
    double out[3];
    if (VEL) {
        group_reduce<D>(v, lane, out);
        if (lane % (32 / D) == 0 && is >= 0)
            for (int c = 0; c < 3; ++c) atomicAdd(&vel[c * Np + is], pref * out[c]);
    }
    if (PSI) {
        group_reduce<D>(w, lane, out);
        if (lane % (32 / D) == 0 && is >= 0)
            for (int c = 0; c < 3; ++c) atomicAdd(&psi[c * Np + is], pref * out[c]);
    }
    const unsigned long long total = warp_sum_u((unsigned long long)ninr);
    if (lane == 0) {
        atomicAdd(&counters[0], total);
        atomicAdd(&counters[1], (unsigned long long)ncand);
    }
}

// Local term (the first to write the outputs), self-interaction removal
// and, when lia_segment_fraction is set, the local integrals over the excluded sub-segments.
__global__ void __launch_bounds__(128) local_self_kernel(
    KParams K, int64_t Np, int fields, int do_local, int do_self, int do_li, double rv, double rpsi,
    const double* __restrict__ nodes, const int32_t* __restrict__ idx_prev, const double* __restrict__ d1,
    const double* __restrict__ d2, const double* __restrict__ dm, const double* __restrict__ dp,
    const double* __restrict__ points, const double* __restrict__ charges, const double* __restrict__ li_vel,
    const double* __restrict__ li_psi, double* __restrict__ vel, double* __restrict__ psi, double3 psi_bg,
    unsigned* __restrict__ counters, int ncount) {
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < ncount) counters[i] = 0u;  // of the pair kernel that follows
    if (i >= Np) return;
    const bool want_v = fields & VPBS_VELOCITY, want_p = fields & VPBS_STREAMFUNCTION;
    const double pref = K.Gamma / (4.0 * kPi);
    double v[3] = {0, 0, 0}, p[3] = {0, 0, 0};
    if (do_local) {
        const double delta = sqrt(dm[i] * dp[i]);
        const double s1[3] = {d1[i], d1[Np + i], d1[2 * Np + i]};
        const double s2[3] = {d2[i], d2[Np + i], d2[2 * Np + i]};
        const double mu_inv = 1.0 / sqrt(s1[0] * s1[0] + s1[1] * s1[1] + s1[2] * s1[2]);
        if (want_v) {
            const double f = log(delta / rv) * (mu_inv * mu_inv * mu_inv);
            v[0] = pref * (f * (s1[1] * s2[2] - s1[2] * s2[1]));
            v[1] = pref * (f * (s1[2] * s2[0] - s1[0] * s2[2]));
            v[2] = pref * (f * (s1[0] * s2[1] - s1[1] * s2[0]));
        }
        if (want_p) {
            const double f = 2.0 * log(delta / rpsi) * mu_inv;
            for (int d = 0; d < 3; ++d) p[d] = pref * (f * s1[d]);
        }
    }
    if (do_self) {
        const int64_t Nq = Np * K.nquad;
        const double x[3] = {nodes[i], nodes[Np + i], nodes[2 * Np + i]};
        const int64_t ip = idx_prev[i];
        const bool explicit_erf = !K.avoid_explicit_erf && K.alpha > 0;
        double sv[3] = {0, 0, 0}, sp[3] = {0, 0, 0};
        for (int side = 0; side < 2; ++side) {
            const int64_t base = (side == 0 ? ip : i) * K.nquad;
            for (int q = 0; q < K.nquad; ++q) {
                const int64_t j = base + q;
                double r[3];
                for (int d = 0; d < 3; ++d) r[d] = deper(x[d] - points[d * Nq + j], K.L[d], K.Lh[d], K.open_domain);
                const double rr = sqrt(r[0] * r[0] + r[1] * r[1] + r[2] * r[2]);
                const double rinv = 1.0 / rr;
                const double qc[3] = {charges[j], charges[Nq + j], charges[2 * Nq + j]};
                double fa = 1.0, fb = 0.0;
                if (explicit_erf && K.kb) {
                    // weights_longrange of the Kaiser-Bessel kernel (kaiser_bessel.jl:296-301):
                    // (F(r), r f(r)) = (1 - a, g - a) inside rcut, (1, 0) beyond
                    if (rr < K.rcut) {
                        double wa, wg;
                        ewald_weights2(K, K.alpha * rr, wa, wg);
                        fa = 1.0 - wa;
                        fb = wg - wa;
                    }
                } else if (explicit_erf) {
                    const double ar = K.alpha * rr;
                    fa = erf(ar);
                    fb = 1.1283791670955126 * ar * exp(-(ar * ar));
                }
                if (want_v) {
                    const double f = (fa - fb) * rinv * rinv * rinv;
                    sv[0] += f * (qc[1] * r[2] - qc[2] * r[1]);
                    sv[1] += f * (qc[2] * r[0] - qc[0] * r[2]);
                    sv[2] += f * (qc[0] * r[1] - qc[1] * r[0]);
                }
                if (want_p) {
                    const double f = fa * rinv;
                    for (int d = 0; d < 3; ++d) sp[d] += f * qc[d];
                }
            }
        }
        for (int d = 0; d < 3; ++d) {
            v[d] -= pref * sv[d];
            p[d] -= pref * sp[d];
        }
    }
    if (do_li) {
        for (int d = 0; d < 3; ++d) {
            v[d] += li_vel[d * Np + i];
            p[d] += li_psi[d * Np + i];
        }
    }
    if (want_v)
        for (int d = 0; d < 3; ++d) vel[d * Np + i] = v[d];
    if (want_p) {
        // streamfunction of the uniform background vorticity of unclosed filaments (zero otherwise)
        p[0] += psi_bg.x;
        p[1] += psi_bg.y;
        p[2] += psi_bg.z;
        for (int d = 0; d < 3; ++d) psi[d * Np + i] = p[d];
    }
}

}  // namespace

static bool use_f32_pairs(const vpbs_handle* h);

int build_cell_lists(vpbs_handle* h) {
    if (h->K.open_domain) return 0;
    // Cell size (internal: the pair set does not depend on it).  Where cells r_cut/2 wide would
    // hold fewer than 8 nodes, cells r_cut wide (M = 1) are used instead: the pair search is
    // then bound by per-node overhead, which grows with the (2M+1)^2 rows a node walks (FP32,
    // 1M-node tangle at r_cut = L/45: 1.82 ms with M = 1 against 2.82 with M = 2; FP64, 100k nodes: 0.32 against
    // 0.41; FP32, 20k nodes: even).
    {
        const int Mu = h->P.nsubdiv;
        int M = Mu;
        if (Mu >= 2) {
            const CellGrid c2 = make_cell_grid(h->K.L, h->K.rcut, 2);
            const CellGrid c1 = make_cell_grid(h->K.L, h->K.rcut, 1);
            const double per_cell2 = (double)h->Np * c2.G / (double)c2.ncell;
            if (per_cell2 < 8.0 && c1.nc[0] >= 3 * c1.G && c1.nc[1] >= 3 && c1.nc[2] >= 3) M = 1;
        }
        if (M != h->cg.M) h->cg = make_cell_grid(h->K.L, h->K.rcut, M);
    }
    const int64_t Np = h->Np, Nq = h->Nq, ncell = h->cg.ncell;
    int rc;
    // the nodes' cells, counts and starts follow the points' in the same arrays: one pass and one scan for both
    const int64_t n = Nq + Np, nscan = 2 * (ncell + 1);
    if ((rc = ensure(h, h->src_cell, sizeof(int32_t) * 2 * n, "cells"))) return rc;
    // ncell + 1 cells each: the last one is the sentinel of points with non-finite coordinates
    if ((rc = ensure(h, h->cell_start, sizeof(int32_t) * (nscan + 1), "cell starts"))) return rc;
    if ((rc = ensure(h, h->cell_counts, sizeof(int32_t) * nscan, "cell counts"))) return rc;
    if ((rc = ensure(h, h->src_sorted, sizeof(double) * 6 * Nq, "src_sorted"))) return rc;
    if ((rc = ensure(h, h->src_seg, sizeof(int32_t) * Nq, "src_seg"))) return rc;
    if ((rc = ensure(h, h->dst_order, sizeof(int32_t) * Np, "dst_order"))) return rc;
    // FP32 sources of the pair kernels: the places (screen), and for the mixed form all of them
    const int f32 = use_f32_pairs(h) ? 2 : h->cg.M > 0 ? 1 : 0;
    const size_t f32_size = f32 == 2 ? 2 * sizeof(float4) + sizeof(float2) : f32 ? sizeof(float4) : 0;
    if (f32 && (rc = ensure(h, h->src_f32, f32_size * Nq, "FP32 sources"))) return rc;
    int32_t* cell = (int32_t*)h->src_cell.p;
    int32_t* rank = cell + n;
    int32_t* counts = (int32_t*)h->cell_counts.p;
    h->src_start = (int32_t*)h->cell_start.p;
    h->dst_start = h->src_start + ncell + 1;
    StageScope st(h, ST_CELL_LISTS);
    if ((rc = check_cuda(h, cudaMemsetAsync(counts, 0, sizeof(int32_t) * nscan, h->stream), "memset"))) return rc;
    cell_count_kernel<<<grid_for(n + 32, 256), 256, 0, h->stream>>>(h->K, h->cg, Nq, Np, (const double*)h->points.p,
                                                               (const double*)h->nodes.p, cell, rank, counts,
                                                               (const int32_t*)h->idx_prev.p, (const double*)h->dp.p,
                                                               h->dm_pending ? (double*)h->dm.p : nullptr);
    h->dm_pending = false;
    if ((rc = exclusive_scan(h, counts, h->src_start, nscan, h->scan_tmp, ncell + 1, (int32_t)Nq))) return rc;
    scatter_kernel<<<grid_for(n, 256), 256, 0, h->stream>>>(
        Nq, Np, h->K.nquad, (const double*)h->points.p, (const double*)h->charges.p, cell, rank, h->src_start,
        (double*)h->src_sorted.p, (int32_t*)h->src_seg.p, (float4*)h->src_f32.p, f32, h->dst_start,
        (int32_t*)h->dst_order.p);
    h->launches += 2;  // plus the scan, counted by exclusive_scan
    return check_cuda(h, cudaGetLastError(), "cell list kernels");
}

int ewald_table_size(double xmax) { return (int)std::floor(xmax * kEwaldInvH) + 2; }

// Taylor coefficients of erfc and g(x) = erfc(x) + 2/sqrt(pi) x e^{-x^2} about the centres
// c_k = (k + 1/2)/16.  The derivatives are closed-form:
//   erfc^(n)(c) = (-1)^n 2/sqrt(pi) H_{n-1}(c) e^{-c^2}  (n >= 1, physicists' Hermite H),
//   g^(n)(c) = (1 - n) erfc^(n)(c) - c erfc^(n+1)(c)      (since g = erfc - x erfc').
// With |x - c| <= 1/32 the degree-9 remainder is below 1e-16 for all x >= 0.
void ewald_table_host(double xmax, int* ntab, double* tab) {
    const int K = ewald_table_size(xmax);
    *ntab = K;
    if (!tab) return;
    const double two_over_sqrt_pi = 2.0 / std::sqrt(kPi);
    for (int k = 0; k < K; ++k) {
        const double c = (k + 0.5) * kEwaldH;
        double H[kEwaldNC + 2];
        H[0] = 1.0;
        H[1] = 2.0 * c;
        for (int n = 1; n + 1 < kEwaldNC + 2; ++n) H[n + 1] = 2.0 * c * H[n] - 2.0 * n * H[n - 1];
        const double E = std::exp(-c * c);
        double d[kEwaldNC + 1];  // erfc^(n)(c), n = 0..NC
        d[0] = std::erfc(c);
        for (int n = 1; n <= kEwaldNC; ++n) d[n] = ((n % 2) ? -1.0 : 1.0) * two_over_sqrt_pi * H[n - 1] * E;
        double fact = 1.0;
        for (int n = 0; n < kEwaldNC; ++n) {
            if (n > 0) fact *= n;
            tab[k * kEwaldNC + n] = d[n] / fact;
            tab[(K + k) * kEwaldNC + n] = ((1.0 - n) * d[n] - c * d[n + 1]) / fact;
        }
    }
}

void table_eval_host(const double* tab, int ntab, double x, double* a, double* g) {
    int k = (int)(x * kEwaldInvH);
    k = k < ntab ? (k < 0 ? 0 : k) : ntab - 1;
    const double t = x - (k + 0.5) * kEwaldH;
    const double* ce = tab + (size_t)k * kEwaldNC;
    const double* cg = tab + (size_t)(ntab + k) * kEwaldNC;
    double va = ce[kEwaldNC - 1], vg = cg[kEwaldNC - 1];
    for (int m = kEwaldNC - 2; m >= 0; --m) {
        va = std::fma(va, t, ce[m]);
        vg = std::fma(vg, t, cg[m]);
    }
    *a = va;
    *g = vg;
}

int tab_s_size(double xmax) { return (int)std::floor(xmax * kTabSInvH) + 2; }

// Both weights of the Gaussian splitting in extended precision (gaussian.jl:273-279): Taylor series about x from the
// closed-form derivatives of ewald_table_host, the first term left out below 1e-20 for |h| <= 1/256 (one erfc and one
// exp per interval instead of six: 0.47 ms for the tables of a handle instead of 0.79).
void gaussian_weights_l(long double x, const long double* h, int n, long double* a, long double* g) {
    constexpr int N = 9;
    const long double f = 1.12837916709551257390L * std::exp(-x * x);  // 2 / sqrt(pi) e^{-x^2}
    long double H[N + 1] = {1.0L, 2.0L * x}, d[N + 1] = {std::erfc(x), -f}, fact = 1.0L, ca[N], cg[N];
    for (int k = 1; k < N; ++k) {
        H[k + 1] = 2.0L * x * H[k] - 2.0L * k * H[k - 1];
        d[k + 1] = (k % 2 ? 1.0L : -1.0L) * f * H[k];
    }
    for (int k = 0; k < N; ++k) {
        if (k > 0) fact *= k;
        ca[k] = d[k] / fact;
        cg[k] = ((1.0L - k) * d[k] - x * d[k + 1]) / fact;
    }
    for (int i = 0; i < n; ++i) {
        a[i] = g[i] = 0.0L;
        for (int k = N - 1; k >= 0; --k) {
            a[i] = a[i] * h[i] + ca[k];
            g[i] = g[i] * h[i] + cg[k];
        }
    }
}

// Degree-5 interpolants of both weights on every interval centred at k / 128, through their values at the 6
// Chebyshev points of the interval, in powers of t = 128 x - k.  Largest error over [0, 4],
// Gaussian weights: 1.1e-16 (erfc) and 1.9e-16 (velocity weight), as of the degree-9 tables, root mean squares 2.1e-17
// and 2.9e-17 (2.2e-17, 3.7e-17).  Intervals of 1/96 fitted to values rounded to FP64: 2.2e-16 and 3.7e-16.
void tab_s_host(const WeightsL& weights, double xmax, double* out) {
    constexpr int NC = kTabSNC;
    const int nf = tab_s_size(xmax);
    long double T[NC], A[NC][NC], h[NC];
    for (int j = 0; j < NC; ++j) {
        T[j] = 0.5L * std::cos((2 * j + 1) * 3.14159265358979323846L / (2 * NC));
        h[j] = T[j] / (long double)kTabSInvH;
    }
    // rows of the inverse of the Vandermonde matrix: the Lagrange polynomials in powers of t
    for (int j = 0; j < NC; ++j) {
        long double c[NC] = {1.0L}, den = 1.0L;
        int deg = 0;
        for (int i = 0; i < NC; ++i) {
            if (i == j) continue;
            den *= T[j] - T[i];
            for (int n = ++deg; n > 0; --n) c[n] = c[n - 1] - T[i] * c[n];
            c[0] *= -T[i];
        }
        for (int n = 0; n < NC; ++n) A[j][n] = c[n] / den;
    }
    for (int k = 0; k < nf; ++k) {
        long double cf[2][NC] = {}, a[NC], g[NC];
        weights(k / (long double)kTabSInvH, h, NC, a, g);
        for (int j = 0; j < NC; ++j)
            for (int n = 0; n < NC; ++n) {
                cf[0][n] += A[j][n] * a[j];
                cf[1][n] += A[j][n] * g[j];
            }
        for (int w = 0; w < 2; ++w)
            for (int n = 0; n < NC; ++n) out[((size_t)w * nf + k) * NC + n] = (double)cf[w][n];
    }
}

void tab_s_eval_host(const double* tab, int nf, double x, double* a, double* g) {
    int k;
    const double t = tab_s_pos(x, nf, &k);
    *a = tab_s_poly(tab + (size_t)k * kTabSNC, t);
    *g = tab_s_poly(tab + (size_t)(nf + k) * kTabSNC, t);
}

int f32_table_size(double xmax) { return (int)std::floor(xmax * kTabCInvH) + 2; }

// Cubic interpolants of both weights on every interval [k/32, (k+1)/32], through the values of
// the FP64 table at the 4 Chebyshev points of the interval, in powers of t = 32 x - k (t in
// [0, 1]).  Over [0, xmax] they agree with the FP64 weights to ~3e-8 absolute (the FP32
// rounding of the coefficients), for the Gaussian and the Kaiser-Bessel weights alike.
void f32_table_host(const double* tab, int ntab, double xmax, float4* out) {
    const int nf = f32_table_size(xmax);
    for (int k = 0; k < nf; ++k) {
        double T[4], Va[4], Vg[4];
        for (int j = 0; j < 4; ++j) {
            T[j] = 0.5 + 0.5 * std::cos((2 * j + 1) * kPi / 8.0);
            table_eval_host(tab, ntab, (k + T[j]) / (double)kTabCInvH, &Va[j], &Vg[j]);
        }
        for (int w = 0; w < 2; ++w) {
            // solve the 4x4 Vandermonde system sum_n c_n T_j^n = V_j (Gaussian elimination, pivoting)
            double A[4][5];
            for (int j = 0; j < 4; ++j) {
                double p = 1.0;
                for (int n = 0; n < 4; ++n, p *= T[j]) A[j][n] = p;
                A[j][4] = w == 0 ? Va[j] : Vg[j];
            }
            for (int c = 0; c < 4; ++c) {
                int piv = c;
                for (int r = c + 1; r < 4; ++r)
                    if (std::fabs(A[r][c]) > std::fabs(A[piv][c])) piv = r;
                for (int n = 0; n < 5; ++n) std::swap(A[c][n], A[piv][n]);
                for (int r = c + 1; r < 4; ++r) {
                    const double f = A[r][c] / A[c][c];
                    for (int n = c; n < 5; ++n) A[r][n] -= f * A[c][n];
                }
            }
            double cf[4];
            for (int c = 3; c >= 0; --c) {
                double v = A[c][4];
                for (int n = c + 1; n < 4; ++n) v -= A[c][n] * cf[n];
                cf[c] = v / A[c][c];
            }
            out[(size_t)w * nf + k] = make_float4((float)cf[0], (float)cf[1], (float)cf[2], (float)cf[3]);
        }
    }
}

void f32_table_eval_host(const float4* tabc, int nf, float x, float* a, float* g) {
    int k;
    float t;
    f32_table_pos(x, nf, &k, &t);
    *a = f32_cubic(tabc[k], t);
    *g = f32_cubic(tabc[nf + k], t);
}

int exclusive_scan(vpbs_handle* h, const int32_t* counts, int32_t* start, int64_t n, DevBuf& tmp, int64_t split, int32_t sub) {
    const int64_t nblk = (n + kScanChunk - 1) / kScanChunk;
    if (nblk <= 1) {
        scan_kernel<<<1, 1024, 0, h->stream>>>(counts, start, n, split, sub);
        h->launches++;
        return check_cuda(h, cudaGetLastError(), "scan kernel");
    }
    int rc;
    if ((rc = ensure(h, tmp, sizeof(int32_t) * (2 * nblk + 1), "scan partial sums"))) return rc;
    int32_t* part = (int32_t*)tmp.p;
    int32_t* part_start = part + nblk;
    scan_partials_kernel<<<(unsigned)nblk, kScanThreads, 0, h->stream>>>(counts, n, part);
    scan_kernel<<<1, 1024, 0, h->stream>>>(part, part_start, nblk, INT64_MAX, 0);
    scan_chunks_kernel<<<(unsigned)nblk, kScanThreads, 0, h->stream>>>(counts, n, part_start, start, split, sub);
    h->launches += 3;
    return check_cuda(h, cudaGetLastError(), "scan kernels");
}

// The FP32 pair kernel serves the mixed form with cell lists and weight tables that fit.
static bool use_f32_pairs(const vpbs_handle* h) {
    return h->P.precision == VPBS_PRECISION_MIXED && !h->K.open_domain && !h->K.avoid_explicit_erf && h->K.alpha > 0 &&
           h->cg.M > 0 && h->K.ntab_c > 0 && h->K.ntab_c <= kF32TabMax;
}

// Blocks of nodes and shares of the sources of pair_open_kernel: the fewest shares of at least 128 sources whose CTAs
// fill the last round of those the device holds at a time to 95 % (30,000 nodes: 5 shares, 4.50 ms; one share
// leaves a third of the device idle: 5.76), else those that fill it best.
static unsigned open_blocks(int64_t Np) { return grid_for(Np, kOpenNodes); }
static int64_t open_parts(const vpbs_handle* h) {
    int nsm = 148;
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, h->device);
    const int64_t gx = open_blocks(h->Np), held = kOpenBlocks * (int64_t)nsm;
    const int64_t most = std::max<int64_t>(1, std::min<int64_t>(h->Nq / 128, std::max<int64_t>(held / gx, 16)));
    int64_t best = 1;
    double fill = 0.0;
    for (int64_t parts = 1; parts <= most && fill < 0.95; ++parts) {
        const double f = (double)(gx * parts) / (double)((gx * parts + held - 1) / held * held);
        if (f > fill) {
            fill = f;
            best = parts;
        }
    }
    return best;
}
size_t open_part_bytes(const vpbs_handle* h) {
    const int64_t parts = open_parts(h);
    return parts > 1 ? sizeof(double) * 6 * parts * h->Np : 0;
}

// Adds the pair sums to the outputs; the counters were zeroed by local_and_self.
int pair_interactions(vpbs_handle* h, int fields) {
    const int64_t Np = h->Np, Nq = h->Nq;
    const bool open = h->K.open_domain;
    const int skip_local = (!h->K.avoid_explicit_erf && h->K.alpha > 0) ? 1 : 0;
    if (skip_local && open) return set_error(h, VPBS_ERR_PARAMS, "avoid_explicit_erf=false requires Ewald splitting");
    StageScope st(h, ST_PAIRS);
    const unsigned grid = grid_for(Np, 8);
    const bool v = fields & VPBS_VELOCITY, p = fields & VPBS_STREAMFUNCTION;
    if (open) {
        const unsigned gx = open_blocks(Np);
        const int64_t parts = open_parts(h);
        const int per = (int)((Nq + parts - 1) / parts);
        int rc;  // as large already, after vpbs_set_filaments
        if ((rc = ensure(h, h->spline_scratch, open_part_bytes(h), "partial sums"))) return rc;
        auto launch_open = [&](auto kern) {
            kern<<<dim3(gx, (unsigned)parts), kOpenThreads, 0, h->stream>>>(
                Np, Nq, per, h->K.Gamma / (4.0 * kPi), (const double*)h->nodes.p, (const double*)h->points.p,
                (const double*)h->charges.p, (double*)h->vel.p, (double*)h->psi.p, (double*)h->spline_scratch.p,
                (unsigned*)h->counters.p + kArrive, (unsigned long long*)h->counters.p);
        };
        if (v && p) launch_open(pair_open_kernel<true, true>);
        else if (v) launch_open(pair_open_kernel<true, false>);
        else launch_open(pair_open_kernel<false, true>);
        h->launches++;
        return check_cuda(h, cudaGetLastError(), "open-domain pair kernel");
    }
    const size_t tab_bytes = sizeof(double) * kTabSNC * h->K.ntab_s * (v && p ? 2 : 1);
    if (h->cg.M > 0 && (use_f32_pairs(h) || tab_bytes <= kPairSmemMost)) {
        int nsm = 148;
        cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, h->device);
        const bool f32 = use_f32_pairs(h), big = h->wide_entries || Nq >= (int64_t)1 << kIndexBits<uint32_t>;
        const int Wc = 2 * h->cg.M + 1, D = v && p ? 2 : 4, warps = f32 ? kF32Warps : kF64Warps;
        const unsigned nblk = grid_for(Np, D * warps);
        // a group's rows are shared out where the groups are fewer than the 32 warps an SM holds (1400 nodes,
        // mixed: 25 us with 9 parts)
        const unsigned nparts = (unsigned)std::max(1, std::min(Wc * Wc, (int)((32 * nsm + nblk - 1) / nblk / warps)));
        // screen margin: the FP32 places in the box are rounded to 2^-25 of its size
        const double Lmax = std::fmax(h->K.L[0], std::fmax(h->K.L[1], h->K.L[2]));
        const float rc2s = (float)(h->K.rcut2 * (1.0 + kScreenMargin + 1e-6 * Lmax / h->K.rcut));
        const float4* srcP = (const float4*)h->src_f32.p;
        auto launch_f32 = [&](auto kern) {
            kern<<<dim3(nblk, nparts), 32 * kF32Warps, 0, h->stream>>>(
                h->K, h->cg, Np, rc2s, h->dst_start, (const int32_t*)h->dst_order.p,
                (const double*)h->nodes.p, (const int32_t*)h->idx_prev.p, srcP, srcP + Nq, (const float2*)(srcP + 2 * Nq),
                h->src_start, (double*)h->vel.p, (double*)h->psi.p, (unsigned long long*)h->counters.p);
        };
        auto launch_f64 = [&](auto kern) {
            // the most a table can need, not this handle's: the attribute belongs to the function
            cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kPairSmemMost);
            kern<<<dim3(nblk, nparts), 32 * kF64Warps, tab_bytes, h->stream>>>(
                h->K, h->cg, Np, rc2s, h->dst_start, (const int32_t*)h->dst_order.p,
                (const double*)h->nodes.p, (const int32_t*)h->idx_prev.p, srcP, (const double*)h->src_sorted.p, Nq,
                h->src_start, (double*)h->vel.p, (double*)h->psi.p, (unsigned long long*)h->counters.p);
        };
        auto by_fields = [&](auto entry, auto skip) {
            using E = decltype(entry);
            constexpr bool SK = decltype(skip)::value;
            if (f32) {
                if (v && p) launch_f32(pair_f32_kernel<true, true, 2, E>);
                else if (v) launch_f32(pair_f32_kernel<true, false, 4, E>);
                else launch_f32(pair_f32_kernel<false, true, 4, E>);
            } else {
                if (v && p) launch_f64(pair_f64_kernel<true, true, SK, 2, E>);
                else if (v) launch_f64(pair_f64_kernel<true, false, SK, 4, E>);
                else launch_f64(pair_f64_kernel<false, true, SK, 4, E>);
            }
        };
        if (big && skip_local) by_fields(uint64_t(), std::true_type{});
        else if (big) by_fields(uint64_t(), std::false_type{});
        else if (skip_local) by_fields(uint32_t(), std::true_type{});
        else by_fields(uint32_t(), std::false_type{});
        h->launches++;
        return check_cuda(h, cudaGetLastError(), "pair kernel");
    }
    auto launch = [&](auto kern) {
        kern<<<grid, 256, 0, h->stream>>>(h->K, h->cg, Np, Nq, (const int32_t*)h->dst_order.p, (const double*)h->nodes.p,
                                          (const int32_t*)h->idx_prev.p, (const double*)h->src_sorted.p,
                                          h->src_start, (const int32_t*)h->src_seg.p, h->cg.M == 0 ? 0 : 1,
                                          skip_local, (double*)h->vel.p, (double*)h->psi.p,
                                          (unsigned long long*)h->counters.p);
    };
    if (h->P.precision == VPBS_PRECISION_MIXED) {
        if (v && p) launch(pair_kernel<true, true, float>);
        else if (v) launch(pair_kernel<true, false, float>);
        else launch(pair_kernel<false, true, float>);
    } else {
        if (v && p) launch(pair_kernel<true, true, double>);
        else if (v) launch(pair_kernel<true, false, double>);
        else launch(pair_kernel<false, true, double>);
    }
    h->launches++;
    return check_cuda(h, cudaGetLastError(), "pair kernel");
}

int local_and_self(vpbs_handle* h, int fields, int lia_mode, int with_pairs_self, double integration_cutoff) {
    const KParams& K = h->K;
    double rpsi, rv;
    if (integration_cutoff > 0) {
        rpsi = rv = integration_cutoff;
    } else {
        rpsi = exp(K.Delta - 1.0) * K.a / 2.0;
        rv = rpsi * exp(1.0);
    }
    const int do_local = (lia_mode == VPBS_LIA_TRUE || lia_mode == VPBS_LIA_ONLY) ? 1 : 0;
    const int do_self = with_pairs_self ? 1 : 0;
    const int do_li = (with_pairs_self && K.lia_fraction > 0) ? 1 : 0;
    // background_vorticity_correction! (BiotSavart.jl:255-286), applied with the short range: unclosed
    // filaments whose end-to-end offsets add up to p carry a mean vorticity p Gamma / V, which the
    // long range removes (k = 0 mode); the short-range streamfunction gets that of the compensating
    // uniform background, -(p Gamma / V) C
    double3 bg = make_double3(0.0, 0.0, 0.0);
    if (with_pairs_self && h->have_fil_offsets && !K.open_domain) {
        const double* p = h->offset_sum;
        double dn = 0.0, na = 0.0, nb = 0.0;
        for (int d = 0; d < 3; ++d) {
            dn += p[d] * p[d];
            na += (p[d] + K.L[d]) * (p[d] + K.L[d]);
            nb += K.L[d] * K.L[d];
        }
        // isapprox(p + Ls, Ls) (default rtol sqrt(eps)): no mean vorticity
        if (std::sqrt(dn) > std::sqrt(2.220446049250313e-16) * std::fmax(std::sqrt(na), std::sqrt(nb))) {
            const double f = -(K.Gamma / (K.L[0] * K.L[1] * K.L[2])) * h->bg_factor;
            bg = make_double3(f * p[0], f * p[1], f * p[2]);
        }
    }
    int rc;
    const int ncount = !do_self ? 0 : kArrive + (K.open_domain ? (int)open_blocks(h->Np) : 0);  // fewer than threads
    if (do_self && (rc = ensure(h, h->counters, sizeof(unsigned) * ncount, "counters"))) return rc;
    StageScope st(h, ST_LOCAL_SELF);
    local_self_kernel<<<grid_for(h->Np, 128), 128, 0, h->stream>>>(
        K, h->Np, fields, do_local, do_self, do_li, rv, rpsi, (const double*)h->nodes.p, (const int32_t*)h->idx_prev.p,
        (const double*)h->d1.p, (const double*)h->d2.p, (const double*)h->dm.p, (const double*)h->dp.p,
        (const double*)h->points.p, (const double*)h->charges.p, (const double*)h->li_vel.p,
        (const double*)h->li_psi.p, (double*)h->vel.p, (double*)h->psi.p, bg,
        (unsigned*)h->counters.p, ncount);
    h->launches++;
    return check_cuda(h, cudaGetLastError(), "local term kernel");
}

}  // namespace vpbs
