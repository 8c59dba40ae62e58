// sdot_eval.cu -- evaluation of the entropic semi-discrete dual functional
// and its gradient on B200 (sm_100a).
//
// Replaces SotSolver::evaluate_functional / local_assemble / the value-grad
// lambda / find_nearest_target_points (src/solvers/SotSolver.cc:217-377,
// 769-869, 267-296, 553-570).  One evaluation is two sweeps over the
// (quadrature point, target) pairs plus two small reductions:
//
//   value sweep  (source-centric): per q the reference's max exponent m_q and
//     shifted sum S_q, accumulated online in FP64 with a hand-written exp2
//     (sdot_device.cuh) -> L_q = m_q + log S_q, value and C_global partials.
//   gradient sweep (target-centric, pull): g_j = sum_q w_q nu_j e^{t_qj - L_q}
//     accumulated per target without atomics; exponentials in FP32 ex2 with
//     FP64 accumulation (HYBRID/MIXED) or FP64 (FP64 precision).
//
// Truncation: a (cell, target) pair is a candidate iff
// sqrt_rn(d2(y_j, c_K)) <= r, evaluated as d2 <= s* where s* is the largest
// double with sqrt_rn(s*) <= r (sqrt_rn is monotone, so the two tests are
// identical); d2 is rounded exactly like the reference.  Both sweeps apply
// the same test, after a conservative bounding-sphere cull of whole blocks.
#include <float.h>
#include <math.h>
#include <stdio.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <mutex>
#include <string>
#include <type_traits>

#include "sdot_dense.cuh"
#include "sdot_device.cuh"
#include "sdot_internal.h"
#include "sdot_lattice.cuh"
#include "sdot_lattice_host.h"

namespace sdot {

// ---------------------------------------------------------------------------
// small kernels
// ---------------------------------------------------------------------------

__global__ void k_gather(double *dst, const double *src, const int64_t *perm, int64_t n)
{
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        dst[i] = src[perm[i]];
}

__global__ void k_scatter(double *dst, const double *src, const int64_t *perm, int64_t n)
{
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        dst[perm[i]] = src[i];
}

__global__ void k_axpy(double *x, const double *x0, double a, const double *p, int64_t n)
{
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        x[i] = x0[i] + a * p[i];
}

// Range of the potential, gathered on the way (dst[i] = src[perm[i]]; without
// perm dst is read): max, min and 1 if an entry is not finite, to out and
// out_host.  Four entries per thread and pass, so that their loads overlap;
// the last CTA reduces the CTAs' results.
constexpr int RANGE_THREADS = 256;
constexpr int RANGE_BLOCKS = 148;
__global__ void __launch_bounds__(RANGE_THREADS)
k_psi_range(int64_t n, const double *__restrict__ src, const int64_t *__restrict__ perm, double *__restrict__ dst,
            double *__restrict__ part, unsigned *__restrict__ ticket, double *__restrict__ out,
            double *__restrict__ out_host)
{
    constexpr int U = 4, NW = RANGE_THREADS / 32;
    __shared__ double sh[3][NW];
    double mx = -DBL_MAX, mn = DBL_MAX, bad = 0.0;
    for (int64_t base = blockIdx.x * (int64_t)(RANGE_THREADS * U); base < n;
         base += (int64_t)gridDim.x * (RANGE_THREADS * U)) {
        double a[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int64_t i = base + u * RANGE_THREADS + threadIdx.x;
            a[u] = i < n ? (perm ? src[perm[i]] : dst[i]) : 0.0;
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int64_t i = base + u * RANGE_THREADS + threadIdx.x;
            if (i >= n) continue;
            if (perm) dst[i] = a[u];
            if (!isfinite(a[u])) bad = 1.0;
            mx = a[u] > mx ? a[u] : mx;
            mn = a[u] < mn ? a[u] : mn;
        }
    }
    auto reduce = [&]() {  // over the CTA, to thread 0
        mx = warp_max(mx);
        mn = -warp_max(-mn);
        bad = warp_max(bad);
        const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
        __syncthreads();
        if (l == 0) { sh[0][w] = mx; sh[1][w] = mn; sh[2][w] = bad; }
        __syncthreads();
        if (threadIdx.x == 0)
            for (int i = 1; i < NW; ++i) {
                mx = fmax(mx, sh[0][i]);
                mn = fmin(mn, sh[1][i]);
                bad = fmax(bad, sh[2][i]);
            }
    };
    reduce();
    if (threadIdx.x == 0) {
        part[blockIdx.x * 3 + 0] = mx;
        part[blockIdx.x * 3 + 1] = mn;
        part[blockIdx.x * 3 + 2] = bad;
    }
    if (!last_block(ticket)) return;
    mx = -DBL_MAX;
    mn = DBL_MAX;
    bad = 0.0;
    for (int i = threadIdx.x; i < (int)gridDim.x; i += RANGE_THREADS) {
        mx = fmax(mx, __ldcg(part + i * 3));
        mn = fmin(mn, __ldcg(part + i * 3 + 1));
        bad = fmax(bad, __ldcg(part + i * 3 + 2));
    }
    reduce();
    if (threadIdx.x == 0) {
        out[0] = out_host[0] = mx;
        out[1] = out_host[1] = mn;
        out[2] = out_host[2] = bad;
    }
}

// tpack[j] = {A_j, B_j(DIM), nu_j, y_j(DIM)}: scaled exponent coefficients.
template <int DIM>
__device__ __forceinline__ void target_prep_one(int64_t j, const double *__restrict__ y, const double *__restrict__ nu,
                                                double psi, const EvalArgs &a, double *__restrict__ tpack)
{
    double yt[3], ysq = 0.0;
#pragma unroll
    for (int d = 0; d < DIM; ++d) {
        yt[d] = y[j * DIM + d] - a.o[d];
        ysq += yt[d] * yt[d];
    }
    double *t = tpack + j * TPACK;
    t[0] = a.s * psi - a.halfs * ysq;
#pragma unroll
    for (int d = 0; d < DIM; ++d) t[1 + d] = a.s * yt[d];
    t[1 + DIM] = nu[j];
#pragma unroll
    for (int d = 0; d < DIM; ++d) t[2 + DIM + d] = y[j * DIM + d];
}

// With io, psi is gathered from the caller's array (io->psi) on the way.
template <int DIM>
__global__ void k_target_prep(int64_t nt, const double *__restrict__ y, const double *__restrict__ nu,
                              double *__restrict__ psi, const IoPtrs *__restrict__ io,
                              const int64_t *__restrict__ perm, EvalArgs a, double *__restrict__ tpack)
{
    for (int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; j < nt; j += (int64_t)gridDim.x * blockDim.x) {
        const double p = io ? io->psi[perm[j]] : psi[j];
        if (io) psi[j] = p;
        target_prep_one<DIM>(j, y, nu, p, a, tpack);
    }
}

// Target packing (with the target blocks' largest s psi and the targets' step
// factors, to full precision: a run multiplies up to seven of them) and the lattice
// tiles' shifts in one launch: the first npb CTAs pack the targets, warp <->
// target block, the others take one tile each.
constexpr int LAT_PREP_THREADS = 512;
template <int DIM>
__global__ void __launch_bounds__(LAT_PREP_THREADS)
k_lat_prep(const double *__restrict__ y, const double *__restrict__ nu, double *__restrict__ psi,
           const IoPtrs *__restrict__ io, const int64_t *__restrict__ perm, EvalArgs a, LatArgs L,
           const int64_t *__restrict__ tblk_off, int ntb, int npb, double *__restrict__ tpack,
           double *__restrict__ top, double *__restrict__ shift, double *__restrict__ step)
{
    const double *src = io ? io->psi : nullptr;
    if ((int)blockIdx.x >= npb) {
        lat_shift_block<DIM, LAT_PREP_THREADS>(
            L, a, blockIdx.x - npb, y, [&](int64_t j) { return src ? src[perm[j]] : psi[j]; }, shift);
        return;
    }
    constexpr int NW = LAT_PREP_THREADS / 32;
    const int lane = threadIdx.x & 31;
    for (int b = blockIdx.x * NW + (threadIdx.x >> 5); b < ntb; b += npb * NW) {
        const int64_t j = tblk_off[b] + lane;
        double v = -CUDART_INF;
        if (j < tblk_off[b + 1]) {
            const double p = src ? src[perm[j]] : psi[j];
            if (src) psi[j] = p;
            target_prep_one<DIM>(j, y, nu, p, a, tpack);
            v = a.s * p;
            if (L.runs > 0) {
#pragma unroll
                for (int d = 0; d < DIM; ++d) step[j * DIM + d] = exp2(tpack[j * TPACK + 1 + d] * L.step16[d]);
            }
        }
        v = warp_max(v);
        if (lane == 0) top[b] = v;
    }
}

template <int DIM>
__global__ void __launch_bounds__(LAT_THREADS, 2)
k_lat_value(LatArgs L, EvalArgs a, const double *__restrict__ tpack, const double *__restrict__ shift,
            const double *__restrict__ step, int64_t tslice, int slice0, double *__restrict__ ms)
{
    extern __shared__ __align__(16) unsigned char lat_smem[];
    const int64_t t0 = (slice0 + (int)blockIdx.y) * tslice;
    const int64_t t1 = min(a.nt, t0 + tslice);
    lat_value_block<DIM>(lat_smem, L, a, tpack, shift, step, blockIdx.x, t0, t1,
                         ms + ((int64_t)blockIdx.y * L.ntiles + blockIdx.x) * LAT_TILE);
}

// ms[i] += the n - 1 slices after it, in their order: the sums that
// lat_merge_block forms over the slices, begun where not all of them fit the
// scratch at once.
__global__ void k_lat_fold(int64_t stride, int n, double *__restrict__ ms)
{
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= stride) return;
    double s = ms[i];
    for (int k = 1; k < n; ++k) s += ms[i + k * stride];
    ms[i] = s;
}

template <int DIM>
__global__ void __launch_bounds__(LAT_THREADS)
k_lat_merge(LatArgs L, EvalArgs a, LatBlocks K, int nslice, bool wt, double *__restrict__ ms, const double *__restrict__ shift,
            const double *__restrict__ tpack, const double *__restrict__ rho, const double *__restrict__ jxw, double *__restrict__ Lq,
            double *__restrict__ part)
{
    constexpr int PER = LAT_TILE / LAT_THREADS;
    lat_merge_block<DIM>(L, a, K, blockIdx.x / PER, blockIdx.x % PER, nslice, wt, ms, shift, tpack, rho, jxw, Lq,
                             part + (int64_t)blockIdx.x * 4);
}

template <int DIM>
__global__ void __launch_bounds__(LAT_THREADS, 2)
k_lat_grad(LatArgs L, EvalArgs a, const double *__restrict__ tpack, const double *__restrict__ shift,
           const double *__restrict__ step, const double *__restrict__ wt, int tslice, double *__restrict__ gpart)
{
    extern __shared__ __align__(16) unsigned char lat_smem[];
    const int ta = blockIdx.y * tslice;
    lat_grad_block<DIM>(lat_smem, L, a, tpack, shift, step, wt, blockIdx.x * (int64_t)LAT_GT, ta, min(L.ntiles, ta + tslice),
                        gpart + blockIdx.y * a.nt);
}

// truncated-path layout: component after component (y(3), nu, log2 nu, kappa psi / eps), nt doubles each
template <int DIM>
__global__ void k_target_prep_kd(int64_t nt, const double *__restrict__ y, const double *__restrict__ nu,
                                 const double *__restrict__ psi, EvalArgs a, double *__restrict__ tpack)
{
    for (int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; j < nt; j += (int64_t)gridDim.x * blockDim.x) {
#pragma unroll
        for (int d = 0; d < 3; ++d) tpack[d * nt + j] = d < DIM ? y[j * DIM + d] : 0.0;
        tpack[3 * nt + j] = nu[j];
        tpack[4 * nt + j] = log2(nu[j]);
        tpack[5 * nt + j] = a.s * psi[j];
    }
}

template <int DIM>
__global__ void __launch_bounds__(DENSE_A_THREADS)
k_value_dense(const double *__restrict__ x, const double *__restrict__ rho, const double *__restrict__ jxw,
              const double *__restrict__ tpack, EvalArgs a, double *__restrict__ Lq, double *__restrict__ part)
{
    dense_value_block<DIM>(x, rho, jxw, tpack, a, blockIdx.x, Lq, part + (int64_t)blockIdx.x * 4);
}

template <int DIM>
__global__ void __launch_bounds__(DENSE_A_THREADS)
k_value_dense_slice(const double *__restrict__ x, const double *__restrict__ tpack, EvalArgs a, int64_t tslice,
                    double *__restrict__ ms)
{
    const int64_t t0 = blockIdx.y * tslice;
    const int64_t t1 = min(a.nt, t0 + tslice);
    dense_value_slice<DIM>(x, tpack, a, blockIdx.x, t0, t1, ms + (int64_t)blockIdx.y * 2 * a.nq);
}

constexpr int MERGE_THREADS = DENSE_A_THREADS * DENSE_MERGE_SPLIT;

template <int DIM>
__global__ void __launch_bounds__(MERGE_THREADS)
k_value_dense_merge(const double *__restrict__ x, const double *__restrict__ rho, const double *__restrict__ jxw,
                    const double *__restrict__ ms, int nslice, EvalArgs a, double *__restrict__ Lq,
                    double *__restrict__ part)
{
    dense_value_merge<DIM>(x, rho, jxw, ms, nslice, a, blockIdx.x, Lq, part + (int64_t)blockIdx.x * 4);
}

// Dense value sweep over cells whose points form a TM^DIM tensor grid
// symmetric about the cell centre (point i = i_0 + TM i_1 (+ TM^2 i_2)):
// thread <-> cell, one slice of the targets per blockIdx.y, with the same
// output as k_value_dense_slice (per point: its largest scaled exponent mx
// and the sum relative to it), merged by k_value_dense_merge.  The exponent
// of point q and target j, b_qj = A_j + B_j.(c - o) + sum_d B_jd delta_qd,
// factors per dimension: with G_d = B_jd a_d and the lowest point's
// exponent b_0 = B0 - sum_d G_d, b_qj = b_0 + sum_d i_d h_d G_d (h = 2 for
// TM = 2, 1 for TM = 3), so one exponential 2^((b_0 - M)/16) and one per
// dimension serve the cell's TM^DIM points.  M is a common shift per cell,
// an upper bound of every exponent so far (raised lazily, as in
// lse_update).  The per-point maxima are exact: a target updates them only
// when its upper bound B0 + sum |G_d| reaches the largest lower bound
// B0 - sum |G_d| seen so far, below which it cannot be any point's maximum.
// UNI (every cell has the offsets ua_d): G_d, its factor 2^(H G_d / 16) and
// the sums of G_d and |G_d| depend on the target alone, so they are computed
// once per staged target instead of once per (cell, target), leaving one
// exponential per (cell, target).
struct Spacing {
    double a[3];
};

template <int DIM, int TM, bool UNI>
__global__ void __launch_bounds__(DENSE_A_THREADS)
k_value_dense_tensor(const double *__restrict__ x, const double *__restrict__ tpack, EvalArgs a, int64_t ncells,
                     int64_t tslice, Spacing ua, double *__restrict__ ms)
{
    constexpr int NQ = DIM == 3 ? TM * TM * TM : TM * TM;
    // staged per target: A, B(DIM), nu; UNI adds G(DIM), 2^(H G / 16) (DIM), sum G, sum |G|
    constexpr int TSZ = UNI ? 3 * DIM + 4 : DIM + 2;
    constexpr double H = TM == 2 ? 2.0 : 1.0;
    __shared__ double tab[16];
    __shared__ double stg[DA_CHUNK * TSZ];
    if (threadIdx.x < 16) tab[threadIdx.x] = c_exp2_tab[threadIdx.x];
    const int64_t cell = blockIdx.x * (int64_t)DENSE_A_THREADS + threadIdx.x;
    const bool valid = cell < ncells;
    const int64_t q0 = (valid ? cell : 0) * NQ;
    // cell centre (relative to o) and half spacing per dimension, from the extreme points along d
    double cp[DIM], ah[DIM];
#pragma unroll
    for (int d = 0; d < DIM; ++d) {
        const int stride = d == 0 ? 1 : (d == 1 ? TM : TM * TM);
        const double lo = x[q0 * DIM + d], hi = x[(q0 + (int64_t)(TM - 1) * stride) * DIM + d];
        const double cd = 0.5 * (lo + hi);
        cp[d] = cd - a.o[d];
        ah[d] = hi - cd;
    }
    const int64_t t0 = blockIdx.y * tslice;
    const int64_t t1 = min(a.nt, t0 + tslice);
    double S[NQ], mx[NQ];
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
        S[q] = 0.0;
        mx[q] = -CUDART_INF;
    }
    double M = -CUDART_INF, lbmax = -CUDART_INF;
    for (int64_t c0 = t0; c0 < t1; c0 += DA_CHUNK) {
        const int cn = (int)min((int64_t)DA_CHUNK, t1 - c0);
        __syncthreads();
        if constexpr (UNI) {
            for (int t = threadIdx.x; t < cn; t += DENSE_A_THREADS) {
                const double *src = tpack + (c0 + t) * TPACK;
                double *dst = stg + t * TSZ;
                double sg = 0.0, ag = 0.0;
#pragma unroll
                for (int f = 0; f < DIM + 2; ++f) dst[f] = src[f];
#pragma unroll
                for (int d = 0; d < DIM; ++d) {
                    const double G = src[1 + d] * ua.a[d];
                    dst[DIM + 2 + d] = G;
                    dst[2 * DIM + 2 + d] = exp2_16(H * G, tab);
                    sg += G;
                    ag += fabs(G);
                }
                dst[3 * DIM + 2] = sg;
                dst[3 * DIM + 3] = ag;
            }
        } else {
            for (int i = threadIdx.x; i < cn * TSZ; i += DENSE_A_THREADS) {
                const int t = i / TSZ, f = i - t * TSZ;
                stg[i] = tpack[(c0 + t) * TPACK + f];
            }
        }
        __syncthreads();
        for (int t = 0; t < cn; ++t) {
            const double *tp = stg + t * TSZ;
            double B0 = tp[0], G[DIM], sg = 0.0, ag = 0.0;
#pragma unroll
            for (int d = 0; d < DIM; ++d) {
                B0 = fma(tp[1 + d], cp[d], B0);
                if constexpr (UNI) {
                    G[d] = tp[DIM + 2 + d];
                } else {
                    G[d] = tp[1 + d] * ah[d];
                    sg += G[d];
                    ag += fabs(G[d]);
                }
            }
            if constexpr (UNI) {
                sg = tp[3 * DIM + 2];
                ag = tp[3 * DIM + 3];
            }
            const double ub = B0 + ag;
            if (ub - M > LSE_THR) {   // raise the shift (the first target sets it)
                if (M > -CUDART_INF) {
                    const double sc = exp2_16(M - ub, tab);
#pragma unroll
                    for (int q = 0; q < NQ; ++q) S[q] *= sc;
                }
                M = ub;
            }
            const double P = tp[1 + DIM] * exp2_16(B0 - sg - M, tab);
            double r[DIM];
#pragma unroll
            for (int d = 0; d < DIM; ++d) r[d] = UNI ? tp[2 * DIM + 2 + d] : exp2_16(H * G[d], tab);
#pragma unroll
            for (int i0 = 0; i0 < TM; ++i0) {
                const double f0 = i0 == 0 ? P : (i0 == 1 ? P * r[0] : P * r[0] * r[0]);
#pragma unroll
                for (int i1 = 0; i1 < TM; ++i1) {
                    const double f1 = i1 == 0 ? f0 : (i1 == 1 ? f0 * r[1] : f0 * r[1] * r[1]);
                    if constexpr (DIM == 2) {
                        S[i0 + TM * i1] += f1;
                    } else {
#pragma unroll
                        for (int i2 = 0; i2 < TM; ++i2) {
                            const double f2 = i2 == 0 ? f1 : (i2 == 1 ? f1 * r[2] : f1 * r[2] * r[2]);
                            S[i0 + TM * i1 + TM * TM * i2] += f2;
                        }
                    }
                }
            }
            if (ub >= lbmax) {
                lbmax = fmax(lbmax, B0 - ag);
#pragma unroll
                for (int q = 0; q < NQ; ++q) {
                    double b = B0;
#pragma unroll
                    for (int d = 0; d < DIM; ++d) {
                        const int id = (d == 0 ? q : (d == 1 ? q / TM : q / (TM * TM))) % TM;
                        const double sd = TM == 2 ? (id == 0 ? -1.0 : 1.0) : (double)(id - 1);
                        b = fma(sd, G[d], b);
                    }
                    mx[q] = fmax(mx[q], b);
                }
            }
        }
    }
    if (valid) {
        double *out = ms + (int64_t)blockIdx.y * 2 * a.nq + 2 * q0;
#pragma unroll
        for (int q = 0; q < NQ; ++q) {
            out[2 * q] = mx[q];
            out[2 * q + 1] = (mx[q] == -CUDART_INF) ? 0.0 : S[q] * exp2_16(M - mx[q], tab);
        }
    }
}

// Sum over a tensor-grid cell's points of W_q prod_d r_d^(i_d) (point
// q = i_0 + TM i_1 (+ TM^2 i_2)), by Horner's scheme along each dimension;
// R = f32x2: of two cells.
__device__ __forceinline__ double fma_r(double x, double y, double z) { return fma(x, y, z); }
__device__ __forceinline__ f32x2 fma_r(f32x2 x, f32x2 y, f32x2 z) { return fma2(x, y, z); }

template <int DIM, int TM, typename R>
__device__ __forceinline__ R cell_sum(const R *W, const R *r)
{
    R t2 = R(0);
#pragma unroll
    for (int i2 = (DIM == 3 ? TM - 1 : 0); i2 >= 0; --i2) {
        R t1 = R(0);
#pragma unroll
        for (int i1 = TM - 1; i1 >= 0; --i1) {
            const R *Wr = W + TM * i1 + TM * TM * i2;
            R t0 = Wr[TM - 1];
#pragma unroll
            for (int i0 = TM - 2; i0 >= 0; --i0) t0 = fma_r(t0, r[0], Wr[i0]);
            t1 = (i1 == TM - 1) ? t0 : fma_r(t1, r[1], t0);
        }
        t2 = (DIM == 2 || i2 == TM - 1) ? t1 : fma_r(t2, r[DIM == 3 ? 2 : 0], t1);
    }
    return t2;
}

// Dense gradient sweep over the tensor-grid cells of k_value_dense_tensor:
// thread lane <-> DENSE_B_TT targets, the CTA's slice of cells staged in
// shared memory, DENSE_B_QG groups taking every QG-th staged cell, the
// groups' sums added in group order.  With the cell centre C, the half
// spacing a_d and point offsets delta_qd = (H i_d - 1) a_d,
// |x_q - y|^2 = |C - y|^2 + sum_d (2 delta_qd (C_d - y_d) + delta_qd^2), so a
// (point, target) term is a cell factor times one factor per dimension
// raised to i_d times a per-point weight that does not depend on the target:
//   FP32: 2^(alpha_j + beta_q - c |x_q - y_j|^2)
//       = 2^(alpha_j + bref - c |C - y_j|^2 - sum_d v_d) prod_d 2^(H v_d i_d) W_q,
//         v_d = -2 c a_d (C_d - y_d),  W_q = w_q 2^(beta_q - c |delta_q|^2 - bref);
//   FP64: 2^(u_qj / 16), u_qj = A_j + B_j . (x_q - o) + D_q
//       = 2^((A_j + B_j . (C - o) - sum_d G_d + Dref) / 16) prod_d 2^(H G_d i_d / 16) W_q,
//         G_d = B_jd a_d,  W_q = w_q 2^((D_q - Dref) / 16),
// where bref / Dref is the largest per-point part in the cell (W_q <= w_q).
// One exponential per cell and one per dimension replace TM^DIM.  The
// caller admits the FP32 form only when the factors of a cell span less
// than 2^60 (dense_grad_tensor), so no factor or Horner sum leaves the FP32
// range; the FP64 form inherits the tensor value sweep's bound.
// Non-finite L_q: a cell whose parts are all -inf contributes 0 (as every
// one of its terms does); a +inf part gives a NaN term where the per-point
// form gives +inf (both non-finite, flagged by the finalize).
// UNI (FP64 form, every cell has the offsets ua_d): G_d and its factor
// depend on the target alone and are computed once per target, so one
// exponential per (cell, target) remains.  (The FP32 form measured slower
// with its factors split into cell and target parts: registers.)
// FP32: records hold two cells of a group side by side, one packed
// instruction serves both; every cell's terms and the order of the sums are
// those of one cell at a time (128^2 cells x 16,384 targets: 468 -> 384 us;
// the three ex2 per cell and target alone take 179).
template <int DIM, int TM, bool FP32, bool UNI>
__global__ void __launch_bounds__(DENSE_B_CTA, DENSE_B_PER_SM)
k_grad_dense_tensor(const double *__restrict__ x, const double *__restrict__ w, const double *__restrict__ Lq,
                    const double *__restrict__ tpack, const double *__restrict__ psi, EvalArgs a, int64_t ncells,
                    int64_t cslice, Spacing ua, double *__restrict__ gpart)
{
    constexpr int NQ = DIM == 3 ? TM * TM * TM : TM * TM;
    constexpr int TT = DENSE_B_TT;
    constexpr int QG = DENSE_B_QG;
    constexpr int NTH = DENSE_B_CTA;
    constexpr int GC = NTH / NQ < 64 ? NTH / NQ : 64;  // cells staged at a time: one point per thread
    constexpr int CR = 16;                             // cell record: W (NQ), C (DIM), k (DIM), reference
    static_assert(NQ + 2 * DIM + 1 <= CR, "cell record");
    static_assert(!(UNI && FP32), "per-target factors: FP64 form only");
    constexpr double H = TM == 2 ? 2.0 : 1.0;
    using R = typename std::conditional<FP32, float, double>::type;
    __shared__ double tab[16];
    constexpr int CF = (NQ + 2 * DIM + 2) / 2 * 2;     // FP32: its fields, an even number
    constexpr int GP = GC / QG / 2;                    // FP32: cell pairs of a group
    static_assert(!FP32 || GC % (2 * QG) == 0, "whole cell pairs");
    // FP64: a record per cell; FP32: for each group and pair of its cells, both cells' values of each field
    __shared__ __align__(16) R crec[FP32 ? QG * GP * CF * 2 : GC * CR];
    __shared__ double pb[GC * NQ];
    if (threadIdx.x < 16) tab[threadIdx.x] = c_exp2_tab[threadIdx.x];
    const int tid = threadIdx.x;
    const int lt = tid % DENSE_B_THREADS;
    const int grp = tid / DENSE_B_THREADS;
    const int64_t j0 = blockIdx.x * (int64_t)(DENSE_B_THREADS * TT);
    GradTargets<TT> T;
    grad_targets<DIM, FP32, NTH>(tpack, psi, a, j0, lt, T);
    double acc64[TT];
#pragma unroll
    for (int k = 0; k < TT; ++k) acc64[k] = 0.0;
    // UNI: the per-dimension factors and their exponents' sum, per target
    double rt[TT][DIM], st[TT];
    if constexpr (UNI) {
        __syncthreads();  // tab
#pragma unroll
        for (int k = 0; k < TT; ++k) {
            st[k] = 0.0;
#pragma unroll
            for (int d = 0; d < DIM; ++d) {
                const double G = T.B[k][d] * ua.a[d];
                rt[k][d] = exp2_16(H * G, tab);
                st[k] += G;
            }
        }
    }
    const int64_t ca = blockIdx.y * cslice;
    const int64_t cb = min(ncells, ca + cslice);
    // FP32: the targets' constants in both halves
    f32x2 yn[TT][DIM], al2[TT];
    const f32x2 nc32 = pack2(-(float)a.c32, -(float)a.c32), minus1 = pack2(-1.f, -1.f), two = pack2(2.f, 2.f);
    if (FP32) {
#pragma unroll
        for (int k = 0; k < TT; ++k) {
#pragma unroll
            for (int d = 0; d < DIM; ++d) yn[k][d] = pack2(-T.yt[k][d], -T.yt[k][d]);
            al2[k] = pack2(T.alpha[k], T.alpha[k]);
        }
    }
    for (int64_t c0 = ca; c0 < cb; c0 += GC) {
        const int cn = (int)min((int64_t)GC, cb - c0);
        const int cl = tid / NQ, qi = tid - cl * NQ;
        const bool act = cl < cn;
        const int64_t cq0 = (c0 + (act ? cl : 0)) * NQ;
        // the cell's centre and half spacing from its extreme points along each dimension
        double cen[DIM], ah[DIM];
#pragma unroll
        for (int d = 0; d < DIM; ++d) {
            const int stride = d == 0 ? 1 : (d == 1 ? TM : TM * TM);
            const double lo = x[cq0 * DIM + d], hi = x[(cq0 + (int64_t)(TM - 1) * stride) * DIM + d];
            cen[d] = 0.5 * (lo + hi);
            ah[d] = hi - cen[d];
        }
        __syncthreads();  // the previous cells' records are consumed
        double wq = 0.0;
        if (act) {
            // the part of point q's exponent that does not depend on the target
            const int64_t q = cq0 + qi;
            double part;
            if (FP32) {
                double dsq = 0.0;
#pragma unroll
                for (int d = 0; d < DIM; ++d) {
                    const double dl = x[q * DIM + d] - cen[d];
                    dsq += dl * dl;
                }
                part = -LOG2E * Lq[q] + T.aref - a.c32 * dsq;
            } else {
                double xsq = 0.0;
#pragma unroll
                for (int d = 0; d < DIM; ++d) {
                    const double xt = x[q * DIM + d] - a.o[d];
                    xsq += xt * xt;
                }
                part = -a.halfs * xsq - KAPPA * Lq[q];
            }
            pb[tid] = part;
            wq = w[q];
        }
        __syncthreads();
        if (act) {
            double ref = -CUDART_INF;
#pragma unroll
            for (int u = 0; u < NQ; ++u) ref = fmax(ref, pb[cl * NQ + u]);
            const bool none = ref == -CUDART_INF;  // every term of the cell is 0
            const double own = pb[tid];
            const double Wq = none ? 0.0 : (FP32 ? wq * exp2(own - ref) : wq * exp2_16(own - ref, tab));
            // field f of the cell's record
            auto put = [&](int f, double v) {
                if (FP32) crec[(((cl % QG) * GP + cl / QG / 2) * CF + f) * 2 + (cl / QG & 1)] = (R)v;
                else crec[cl * CR + f] = (R)v;
            };
            put(qi, Wq);
            if (qi == 0) {
#pragma unroll
                for (int d = 0; d < DIM; ++d) {
                    put(NQ + d, FP32 ? cen[d] - T.ob[d] : cen[d] - a.o[d]);
                    put(NQ + DIM + d, FP32 ? -2.0 * a.c32 * ah[d] : ah[d]);
                }
                put(NQ + 2 * DIM, none ? 0.0 : ref);
            }
        } else if (FP32 && cl < cn + QG && cl < GC) {
            // the other half of a group's last pair: a cell of no weight
            float *rec = reinterpret_cast<float *>(crec) + (((cl % QG) * GP + cl / QG / 2) * CF) * 2 + (cl / QG & 1);
            rec[2 * qi] = 0.f;
            if (qi == 0) {
#pragma unroll
                for (int d = 0; d < 2 * DIM; ++d) rec[2 * (NQ + d)] = 0.f;
                rec[2 * (NQ + 2 * DIM)] = -INFINITY;
            }
        }
        __syncthreads();
        if constexpr (FP32) {
            // two cells of the group at a time, one in each half of the packed registers
            const int m = (cn - grp + QG - 1) / QG;
            const f32x2 *rp = reinterpret_cast<const f32x2 *>(crec) + grp * (GP * CF);
            float acc[TT];
#pragma unroll
            for (int k = 0; k < TT; ++k) acc[k] = 0.f;
            for (int p = 0; 2 * p < m; ++p, rp += CF) {
                f32x2 rec[CF];
#pragma unroll
                for (int f = 0; f < CF; f += 2) {
                    const ulonglong2 v = *reinterpret_cast<const ulonglong2 *>(rp + f);
                    rec[f] = v.x;
                    rec[f + 1] = v.y;
                }
#pragma unroll
                for (int k = 0; k < TT; ++k) {
                    f32x2 D2 = 0, sv = 0, r[DIM];
#pragma unroll
                    for (int d = 0; d < DIM; ++d) {
                        const f32x2 dc = add2(rec[NQ + d], yn[k][d]);
                        D2 = d == 0 ? mul2(dc, dc) : fma2(dc, dc, D2);
                        const f32x2 v = mul2(rec[NQ + DIM + d], dc);
                        sv = d == 0 ? v : add2(sv, v);
                        r[d] = ex2_approx2(TM == 2 ? mul2(two, v) : v);
                    }
                    const f32x2 ex = fma2(nc32, D2, add2(al2[k], rec[NQ + 2 * DIM]));
                    const f32x2 P = ex2_approx2(fma2(sv, minus1, ex));
                    float P0, P1, s0, s1;
                    unpack2(P, P0, P1);
                    unpack2(cell_sum<DIM, TM, f32x2>(rec, r), s0, s1);
                    acc[k] = fmaf(P1, s1, fmaf(P0, s0, acc[k]));
                }
                if ((p & 3) == 3) {
#pragma unroll
                    for (int k = 0; k < TT; ++k) { acc64[k] += (double)acc[k]; acc[k] = 0.f; }
                }
            }
#pragma unroll
            for (int k = 0; k < TT; ++k) acc64[k] += (double)acc[k];
        } else {
            for (int cc = grp; cc < cn; cc += QG) {
                const double *rec = crec + cc * CR;
                double Wc[NQ], Cm[DIM], ad[DIM];
#pragma unroll
                for (int u = 0; u < NQ; ++u) Wc[u] = rec[u];
#pragma unroll
                for (int d = 0; d < DIM; ++d) { Cm[d] = rec[NQ + d]; ad[d] = rec[NQ + DIM + d]; }
                const double Dref = rec[NQ + 2 * DIM];
#pragma unroll
                for (int k = 0; k < TT; ++k) {
                    double B0 = T.A[k], sg = 0.0, r[DIM];
#pragma unroll
                    for (int d = 0; d < DIM; ++d) {
                        B0 = fma(T.B[k][d], Cm[d], B0);
                        if constexpr (UNI) {
                            r[d] = rt[k][d];
                        } else {
                            const double G = T.B[k][d] * ad[d];
                            sg += G;
                            r[d] = exp2_16(H * G, tab);
                        }
                    }
                    if constexpr (UNI) sg = st[k];
                    const double P = exp2_16(B0 - sg + Dref, tab);
                    acc64[k] = fma(P, cell_sum<DIM, TM, double>(Wc, r), acc64[k]);
                }
            }
        }
    }
    // the groups' sums, added in group order by group 0
    __shared__ double gsum[(QG - 1) * TT * DENSE_B_THREADS];
    if (grp > 0) {
#pragma unroll
        for (int k = 0; k < TT; ++k) gsum[((grp - 1) * TT + k) * DENSE_B_THREADS + lt] = acc64[k];
    }
    __syncthreads();
    if (grp == 0) {
#pragma unroll
        for (int k = 0; k < TT; ++k) {
            for (int g = 1; g < QG; ++g) acc64[k] += gsum[((g - 1) * TT + k) * DENSE_B_THREADS + lt];
            const int64_t j = j0 + lt + k * DENSE_B_THREADS;
            if (j < a.nt) {
                double gv = acc64[k];
                if (!FP32) gv *= tpack[j * TPACK + 1 + DIM];  // nu_j (FP32 folds it into alpha)
                gpart[blockIdx.y * a.nt + j] = gv;
            }
        }
    }
}

template <int DIM, bool FP32>
__global__ void __launch_bounds__(DENSE_B_CTA, DENSE_B_PER_SM)
k_grad_dense(const double *__restrict__ x, const double *__restrict__ w, const double *__restrict__ Lq,
             const double *__restrict__ tpack, const double *__restrict__ psi, EvalArgs a, int64_t qslice,
             double *__restrict__ gpart)
{
    dense_grad_block<DIM, FP32, DENSE_B_QG>(x, w, Lq, tpack, psi, a, qslice, blockIdx.x, blockIdx.y, gpart);
}

// ---------------------------------------------------------------------------
// finalize: g_j = sum of partials - nu_j, plus the reductions the solver and
// the solver control need (SotSolver.cc:322-327, SotSolver.h:391-442).
// ---------------------------------------------------------------------------

constexpr int FIN_THREADS = 256;
constexpr int FIN_BLOCKS = 148;  // largest grid of k_finalize
constexpr int NRED = 12;  // psinu, l1, linf, comp, l2sq, gp, nonfinite; value, C, skipped, pairs; unused

// Lanes per target of k_finalize for nks slice partials: the smallest
// power of two >= nks, at most 8.
static int fin_parts(int nks)
{
    return nks <= 1 ? 1 : (nks <= 2 ? 2 : (nks <= 4 ? 4 : 8));
}

// Grid of k_finalize for nt targets (FIN_THREADS / parts targets per CTA and pass).
static int fin_blocks(int64_t nt, int parts)
{
    const int64_t per = FIN_THREADS / parts;
    const int64_t g = (nt + per - 1) / per;
    return (int)std::max<int64_t>(1, std::min<int64_t>(FIN_BLOCKS, g));
}

// PARTS consecutive lanes own target j: lane u sums the slice partials
// k = u, u + PARTS, ... in order of k (each lane's loads in flight together),
// and xor exchanges add the lanes' sums in the fixed tree (s0 + s1) + (s2 +
// s3), ...  PARTS = 8, or any power of two PARTS >= nks, gives the sums of
// eight interleaved sums k mod 8 added in the tree ((s0 + s1) + (s2 + s3)) +
// ((s4 + s5) + (s6 + s7)) (the lanes past nks hold zeros).
//
// Each CTA also sums its share of the nval value partials; the last CTA to
// arrive adds the CTAs' results (in order of the CTAs over a fixed tree) and
// writes the evaluation's scalars to scal and to the host.  With io, the
// gradient also goes to the caller's array.  One launch and no copy at the
// end of an evaluation: two kernels, a scatter and a copy engine's transfer
// took 20 us of a 71 us evaluation of 2,304 points x 256 targets.
struct FinArgs {
    int64_t nt;
    int nks;
    const double *gpart, *nu, *psi, *pdir;
    double tol;
    int sub_nu;
    double *grad;
    const IoPtrs *io;
    const int64_t *perm;
    int64_t nval;
    const double *valpart;
    double *redpart;
    unsigned *ticket;
    double *scal, *scal_host;
};

template <int PARTS>
__global__ void __launch_bounds__(FIN_THREADS)
k_finalize(FinArgs f)
{
    constexpr int TPB = FIN_THREADS / PARTS;  // targets per CTA and pass
    constexpr int NW = FIN_THREADS / 32;
    constexpr int NR = 11;
    const int u = threadIdx.x % PARTS;
    const int64_t nt = f.nt;
    const int nks = f.nks;
    const double *gpart = f.gpart;
    // sums: 0 psinu, 1 l1, 4 l2sq, 5 dot_gp, 7 value, 8 C, 9 skipped, 10 pairs; maxima: 2 linf, 3 comp, 6 bad
    double r[NR] = {0, 0, 0, -CUDART_INF, 0, 0, 0, 0, 0, 0, 0};
    double *gout = f.io ? f.io->grad : nullptr;
    for (int64_t base = blockIdx.x * (int64_t)TPB; base < nt; base += (int64_t)gridDim.x * TPB) {
        const int64_t j = base + threadIdx.x / PARTS;
        const bool ok = j < nt;
        double acc = 0.0;
        if (ok) {
            int k = u;
            for (; k + 3 * PARTS < nks; k += 4 * PARTS) {
                const double v0 = gpart[(int64_t)k * nt + j];
                const double v1 = gpart[(int64_t)(k + PARTS) * nt + j];
                const double v2 = gpart[(int64_t)(k + 2 * PARTS) * nt + j];
                const double v3 = gpart[(int64_t)(k + 3 * PARTS) * nt + j];
                acc += v0;
                acc += v1;
                acc += v2;
                acc += v3;
            }
            for (; k < nks; k += PARTS) acc += gpart[(int64_t)k * nt + j];
        }
#pragma unroll
        for (int o = 1; o < PARTS; o <<= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
        if (ok && u == 0) {
            const double s = acc, nuj = f.nu[j], ps = f.psi[j];
            const double g = s - nuj, w = f.sub_nu ? g : s;
            f.grad[j] = w;
            if (gout) gout[f.perm[j]] = w;
            r[0] += ps * nuj;
            const double ag = fabs(g);
            r[1] += ag;
            r[2] = fmax(r[2], ag);
            r[3] = fmax(r[3], ag - nuj * f.tol);
            r[4] += g * g;
            if (f.pdir) r[5] += g * f.pdir[j];
            if (!isfinite(g) || !isfinite(ps)) r[6] = 1.0;
        }
    }
    const double4 *vp = reinterpret_cast<const double4 *>(f.valpart);
    const int64_t per = (f.nval + gridDim.x - 1) / gridDim.x;
    const int64_t v1 = min(f.nval, (blockIdx.x + 1) * per);
#pragma unroll 4
    for (int64_t b = blockIdx.x * per + threadIdx.x; b < v1; b += FIN_THREADS) {
        const double4 t = vp[b];
        r[7] += t.x;
        r[8] += t.y;
        r[9] += t.z;
        r[10] += t.w;
    }
    __shared__ double sh[NR][NW];
    const int wi = threadIdx.x >> 5, lane = threadIdx.x & 31;
    auto is_max = [](int k) { return k == 2 || k == 3 || k == 6; };
    auto reduce = [&]() {  // over the CTA, to warp 0's lane 0
#pragma unroll
        for (int k = 0; k < NR; ++k) r[k] = is_max(k) ? warp_max(r[k]) : warp_sum(r[k]);
        if (lane == 0) {
#pragma unroll
            for (int k = 0; k < NR; ++k) sh[k][wi] = r[k];
        }
        __syncthreads();
        if (wi == 0) {
#pragma unroll
            for (int k = 0; k < NR; ++k) {
                const double t = lane < NW ? sh[k][lane] : (is_max(k) ? -CUDART_INF : 0.0);
                r[k] = is_max(k) ? warp_max(t) : warp_sum(t);
            }
        }
    };
    reduce();
    if (threadIdx.x == 0) {
#pragma unroll
        for (int k = 0; k < NR; ++k) f.redpart[blockIdx.x * NRED + k] = r[k];
    }
    if (!last_block(f.ticket)) return;
#pragma unroll
    for (int k = 0; k < NR; ++k) {
        r[k] = is_max(k) ? -CUDART_INF : 0.0;
        if (threadIdx.x < gridDim.x) r[k] = __ldcg(f.redpart + threadIdx.x * NRED + k);
    }
    static_assert(FIN_BLOCKS <= FIN_THREADS, "one CTA's result per thread");
    reduce();
    if (threadIdx.x == 0) {
        const double value = r[7] - r[0];
        double o[SC_COUNT];
        o[SC_VALUE] = value;
        o[SC_C] = r[8];
        o[SC_DOT_GP] = r[5];
        o[SC_L1] = r[1];
        o[SC_LINF] = fmax(r[2], 0.0);
        o[SC_COMP] = r[3];
        o[SC_L2SQ] = r[4];
        o[SC_PSINU] = r[0];
        o[SC_SKIPPED] = r[9];
        o[SC_NONFINITE] = (r[6] > 0.0 || !isfinite(value)) ? 1.0 : 0.0;
        o[SC_PAIRS] = r[10];
        o[SC_VALSRC] = r[7];
        constexpr int slot[] = {SC_VALUE, SC_C, SC_DOT_GP, SC_L1, SC_LINF, SC_COMP, SC_L2SQ,
                                SC_PSINU, SC_SKIPPED, SC_NONFINITE, SC_PAIRS, SC_VALSRC};
#pragma unroll
        for (int k = 0; k < (int)(sizeof(slot) / sizeof(int)); ++k) {
            f.scal[slot[k]] = o[slot[k]];
            f.scal_host[slot[k]] = o[slot[k]];
        }
    }
}

// k_finalize with fin_parts(nks) lanes per target.
static void launch_finalize(const FinArgs &f, cudaStream_t st)
{
    const int parts = fin_parts(f.nks);
    const int fb = fin_blocks(f.nt, parts);
    auto go = [&](auto kern) { kern<<<fb, FIN_THREADS, 0, st>>>(f); };
    if (parts == 1) go(k_finalize<1>);
    else if (parts == 2) go(k_finalize<2>);
    else if (parts == 4) go(k_finalize<4>);
    else go(k_finalize<8>);
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------

static int grid_for(int64_t n, int threads, int cap = 148 * 8)
{
    int64_t g = (n + threads - 1) / threads;
    if (g < 1) g = 1;
    if (g > cap) g = cap;
    return (int)g;
}

template <int DIM>
static void launch_target_prep(const sdot_ctx *c, const EvalArgs &a, double *psi, const IoPtrs *io, double *tpack)
{
    k_target_prep<DIM><<<grid_for(a.nt, 256), 256, 0, c->stream>>>(a.nt, c->y.p, c->nu.p, psi, io, c->perm.p, a, tpack);
}

void launch_target_prep_dense(sdot_ctx *c, const EvalArgs &a)
{
    if (c->dim == 2) launch_target_prep<2>(c, a, c->psi.p, nullptr, c->tpack.p);
    else launch_target_prep<3>(c, a, c->psi.p, nullptr, c->tpack.p);
}

void k_axpy_launch(cudaStream_t s, double *x, const double *x0, double a, const double *p, int64_t n)
{
    k_axpy<<<grid_for(n, 256), 256, 0, s>>>(x, x0, a, p, n);
}

sdot_status launch_gather(sdot_ctx *c, double *dst, const double *src, int64_t n)
{
    k_gather<<<grid_for(n, 256), 256, 0, c->stream>>>(dst, src, c->perm.p, n);
    c->klaunch[5] += 1;
    return cuda_error(c, cudaGetLastError(), "gather");
}

sdot_status launch_scatter(sdot_ctx *c, double *dst, const double *src, int64_t n)
{
    k_scatter<<<grid_for(n, 256), 256, 0, c->stream>>>(dst, src, c->perm.p, n);
    c->klaunch[5] += 1;
    return cuda_error(c, cudaGetLastError(), "scatter");
}

// largest double s with sqrt_rn(s) <= r (s* = NaN if r is NaN)
double sstar_of(double r)
{
    if (std::isnan(r)) return NAN;
    if (r < 0) return -1.0;
    if (r >= 1.3407807929942596e154) return DBL_MAX;
    double s = r * r;
    while (s > 0 && std::sqrt(s) > r) s = std::nextafter(s, 0.0);
    while (std::sqrt(std::nextafter(s, INFINITY)) <= r) s = std::nextafter(s, INFINITY);
    return s;
}

// SotSolver::compute_distance_threshold (SotSolver.cc:379-429), on the host
// with the same libm calls and operation order as the reference.
double host_threshold(sdot_ctx *c, double maxpsi, double minpsi)
{
    const sdot_solver_params &p = c->prm;
    if (p.threshold_type == SDOT_THRESH_INTEGRAL) {
        double absJ = std::fabs(c->global_functional);
        if (absJ < 1e-10) absJ = 1e-10;
        const double num = p.epsilon * c->C_global;
        const double den = p.tau * absJ;
        const double arg = num / den;
        const double r2 = 2.0 * maxpsi + 2.0 * p.epsilon * std::log(arg);
        const double r = std::sqrt(std::max(0.0, r2));
        return std::max(r, c->covering_radius);
    }
    if (p.threshold_type == SDOT_THRESH_GEOMETRIC) {
        double r0 = c->covering_radius;
        if (!(r0 > 0.0)) {
            double rr = 0.0;
            sdot_compute_covering_radius(c, &rr);
            r0 = rr;
        }
        const double range = maxpsi - minpsi;
        const double mind = c->min_target_density > 0.0 ? c->min_target_density : c->nu_min;
        double fv = std::fabs(c->global_functional);
        if (fv < 1e-10) fv = 1e-10;
        const double log_term = std::log(p.epsilon / (mind * p.tau * fv));
        double r2 = r0 * r0 + 2.0 * range + 2.0 * p.epsilon * log_term;
        if (r2 < r0 * r0) r2 = r0 * r0;
        return std::sqrt(r2);
    }
    const double numin = c->min_target_density > 0.0 ? c->min_target_density : c->nu_min;
    if (numin <= 0 || p.tau <= 0) return DBL_MAX;
    const double r2 = -2.0 * p.epsilon * std::log(p.tau / numin) + 2.0 * maxpsi;
    return std::sqrt(std::max(0.0, r2));
}

// Launch shape of the dense sweeps, shared by every dense evaluation path so
// that they sum in the same order: value-sweep point blocks (one quadrature
// point per thread) and, when those are too few to fill the GPU (fewer than
// four per SM), target slices of the value sweep (about twelve CTAs per SM in
// all, at least 64 targets per slice, at most 16 slices) merged per point;
// gradient target blocks, and q-slices of the gradient sweep (about eight
// CTAs per SM in all, at least 256 points per slice, at most 64 slices).
// With tm > 0 (cells whose points form a tm^dim tensor grid, at most 9
// points) the value sweep runs over cells (k_value_dense_tensor): ncb cell
// blocks x nvs target slices (about six CTAs per SM in all, at least 32
// targets per slice, at most 64 slices), always merged per point.
//
// Sources whose points form a tensor lattice run the lattice sweeps instead
// (lat: sdot_lattice.cuh; the value sweep always, the gradient sweep in FP64):
// ntiles x nvs CTAs of the value sweep (at least 16 targets per slice), and
// target blocks x gts tile groups of the gradient sweep.
struct DenseShape {
    int64_t nval, tb;
    int nks;
    int nvs;          // target slices of the value sweep (1: unsliced)
    int64_t tslice;   // targets per value slice
    int tm;           // > 0: the cell-based tensor value sweep with tm points per dimension
    int64_t ncb;      // its cell blocks
    LatTiling lat;    // cap > 0: the lattice sweeps
    bool lat_grad;    // the gradient sweep too
    int gts;          // tiles per CTA of the lattice gradient sweep (nks groups)
    int slots;        // slices of the lattice value sweep that the partials hold at a time
    // doubles of the value sweep's partials and of the gradient partials
    size_t vpart_need(int64_t nq, int64_t nt, int64_t ntblk) const
    {
        if (lat.cap > 0) return (size_t)lat.ntiles * ((size_t)slots * LAT_TILE + 2) + (size_t)(3 * nt + ntblk);
        return (nvs > 1 || tm > 0) ? (size_t)2 * nvs * nq : 0;
    }
    size_t gpart_need(int64_t nt) const { return (size_t)nks * nt; }
};
// The tensor value sweep applies to the euclidean untruncated evaluation of
// cells whose points form a symmetric tensor grid of at most 9 points, with
// per-dimension factors that stay within 2^100 over the domain.
static int dense_tensor_m(const sdot_ctx *c, double s_scale)
{
    if (c->distance != 0 || c->tensor_m <= 0) return 0;
    const int tm = c->tensor_m;
    const int np = c->dim == 3 ? tm * tm * tm : tm * tm;
    if (np > 9 || c->qpc != np) return 0;
    const double span = (tm == 2 ? 2.0 : 1.0) * s_scale * 0.5 * c->diam * c->tensor_amax * (tm - 1) * c->dim / 16.0;
    return span <= 100.0 ? tm : 0;
}
static DenseShape dense_shape(int64_t nq, int64_t nt, int tm = 0, int64_t ncells = 0)
{
    DenseShape d{};
    const int64_t per = DENSE_A_THREADS;
    d.nval = (nq + per - 1) / per;
    d.nvs = 1;
    if (d.nval < 148 * 4) {
        const int64_t want = (148 * 12 + d.nval - 1) / d.nval;
        const int64_t maxs = std::max<int64_t>(1, nt / 64);
        d.nvs = (int)std::max<int64_t>(1, std::min<int64_t>(16, std::min(want, maxs)));
    }
    d.tslice = (nt + d.nvs - 1) / d.nvs;
    d.tb = (nt + DENSE_B_THREADS * DENSE_B_TT - 1) / (DENSE_B_THREADS * DENSE_B_TT);
    d.nks = dense_grad_slices(nq, nt);
    d.tm = tm;
    if (tm > 0) {
        d.ncb = (ncells + DENSE_A_THREADS - 1) / DENSE_A_THREADS;
        const int64_t want = (148 * 6 + d.ncb - 1) / d.ncb;
        const int64_t maxs = std::max<int64_t>(1, nt / 32);
        d.nvs = (int)std::max<int64_t>(1, std::min<int64_t>(64, std::min(want, maxs)));
        d.tslice = (nt + d.nvs - 1) / d.nvs;
    }
    return d;
}

// dense_shape for an evaluation of the context's problem at eps (every dense
// evaluation path takes its shape from here).
static DenseShape dense_shape_of(const sdot_ctx *c, double eps, bool fp64)
{
    const double s = KAPPA / eps;
    DenseShape d = dense_shape(c->nq, c->nt, dense_tensor_m(c, s), c->ncells);
    if (!c->lat_ok || c->distance != 0) return d;
    double reach[3];
    for (int k = 0; k < 3; ++k)
        reach[k] = std::max(std::fabs(c->tgt_lo[k] - c->origin[k]), std::fabs(c->tgt_hi[k] - c->origin[k]));
    d.lat = lat_tiling(c->lat_n, c->lat_xo, c->lat_X.data(), c->dim, s, reach);
    // The merge takes the points' maxima in one CTA per LAT_THREADS points, and with more targets than it lists at
    // once it goes through their blocks in turn: few points are few CTAs with a long chain each.  Lattice against
    // cell sweeps, us per FP64 evaluation at eps = 1e-2, 1,025 / 3,001 / 10,538 targets: 2D 64^2 points 60 / 85 / 187
    // against 52 / 66 / 110, 96^2 58 / 76 / 153 against 60 / 84 / 175 (hybrid 66 / 86 / 168 against 62 / 84 / 164),
    // 104^2 57 / 76 / 136 against 61 / 90 / 202 (66 / 86 / 157 against 64 / 90 / 188), 192^2 62 / 83 / 161 against
    // 98 / 181 / 507; 3D 24^3 64 / 98 / 247 against 66 / 97 / 208, 26^3 65 / 101 / 249 against 71 / 111 / 254 (hybrid
    // 78 / 110 / 261 against 76 / 111 / 239), 28^3 63 / 102 / 234 against 76 / 120 / 287, 32^3 63 / 96 / 205 against
    // 90 / 148 / 390.
    // (Batches have no such line: their other sweeps go by points without target slices, 1,468 us against 390 for
    // 16^3 points x 10,538 targets alone, and all problems' merges are one launch.)
    constexpr int64_t FEW_2D = 10000, FEW_3D = 18000;
    if (c->nt > LAT_LIST && c->nq < (c->dim == 2 ? FEW_2D : FEW_3D)) d.lat = LatTiling{};
    if (d.lat.cap == 0) return d;
    constexpr int SLOTS = 148 * 2;
    d.nvs = lat_slices(d.lat.ntiles, (c->nt + 15) / 16, SLOTS);
    d.tslice = (c->nt + d.nvs - 1) / d.nvs;
    d.nvs = (int)((c->nt + d.tslice - 1) / d.tslice);
    d.slots = d.nvs;
    d.nval = (int64_t)d.lat.ntiles * (LAT_TILE / LAT_THREADS);
    d.lat_grad = fp64;
    if (fp64) {
        const int g = lat_slices((c->nt + LAT_GT - 1) / LAT_GT, d.lat.ntiles, SLOTS);
        d.gts = (d.lat.ntiles + g - 1) / g;
        d.nks = (d.lat.ntiles + d.gts - 1) / d.gts;
    }
    return d;
}

void dense_sweeps(const sdot_ctx *c, int *sweeps)
{
    const DenseShape d = dense_shape_of(c, c->prm.epsilon, c->precision == SDOT_PREC_FP64);
    const bool lat = d.lat.cap > 0;
    LatArgs L{};
    if (lat) lat_runs(c->lat_period, c->lat_step, c->dim, d.lat, L);
    const int v[SDOT_DENSE_SWEEPS] = {d.lat.cap, d.lat.ntiles, lat && d.lat_grad, L.runs > 0, lat ? 0 : d.tm, d.nvs};
    std::copy(v, v + SDOT_DENSE_SWEEPS, sweeps);
}

size_t dense_gpart_need(const sdot_ctx *c)
{
    if (c->prm.tau > 0 || c->prm.threshold_type != SDOT_THRESH_POINTWISE || !(c->prm.epsilon > 0)) return 0;
    return dense_shape_of(c, c->prm.epsilon, c->precision == SDOT_PREC_FP64).gpart_need(c->nt);
}

static LatArgs lat_args(const sdot_ctx *c, const LatTiling &t)
{
    LatArgs L{};
    L.X = c->lat_buf.p;
    L.q = reinterpret_cast<const int *>(c->lat_buf.p + c->lat_X.size());
    for (int d = 0; d < 3; ++d) {
        L.n[d] = c->lat_n[d];
        L.nt[d] = t.nt[d];
        L.xo[d] = c->lat_xo[d];
    }
    L.cap = t.cap;
    L.ntiles = t.ntiles;
    lat_runs(c->lat_period, c->lat_step, c->dim, t, L);
    return L;
}

template <class K>
static void lat_smem_limit(K k, size_t bytes)
{
    cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
}

// Launches of the lattice sweeps; vpart holds vpart_need doubles (the slices'
// partials, then the tile shifts, the targets' step factors and the target
// blocks' largest s psi).
struct LatScratch {
    double *shift, *step, *top;
    LatScratch(const DenseShape &ds, double *vpart, int64_t nt, int dim)
        : shift(vpart + (size_t)ds.lat.ntiles * ds.slots * LAT_TILE), step(shift + 2 * ds.lat.ntiles), top(step + nt * dim)
    {
    }
};

template <int DIM>
static void launch_lat_prep(const sdot_ctx *c, const DenseShape &ds, double *psi, const IoPtrs *io, const EvalArgs &a,
                            double *tpack, double *vpart, cudaStream_t st)
{
    constexpr int NW = LAT_PREP_THREADS / 32;
    const int npb = (int)std::min<int64_t>((c->ntblk + NW - 1) / NW, 148);
    const LatScratch S(ds, vpart, a.nt, DIM);
    k_lat_prep<DIM><<<(unsigned)(npb + ds.lat.ntiles), LAT_PREP_THREADS, 0, st>>>(
        c->y.p, c->nu.p, psi, io, c->perm.p, a, lat_args(c, ds.lat), c->tblk_off.p, (int)c->ntblk, npb, tpack, S.top, S.shift,
        S.step);
}

template <int DIM>
static void launch_lat_value(const sdot_ctx *c, const DenseShape &ds, const double *tpack, const EvalArgs &a,
                             double *vpart, double *Lq, double *blkpart, cudaStream_t st)
{
    const LatArgs L = lat_args(c, ds.lat);
    const LatScratch S(ds, vpart, a.nt, DIM);
    const LatBlocks K{c->tblk_off.p, nullptr, c->tblk_sph.p, S.top, (int)c->ntblk};
    const size_t smem = sizeof(LatValueSmem<DIM>);
    lat_smem_limit(k_lat_value<DIM>, smem);
    // all slices at once where the partials hold them, else a pass at a time into the slots after the sum so far
    const int64_t stride = (int64_t)L.ntiles * LAT_TILE;
    int held = 0;
    for (int s = 0; s < ds.nvs;) {
        if (held > 1) k_lat_fold<<<(unsigned)(stride / LAT_THREADS), LAT_THREADS, 0, st>>>(stride, held, vpart);
        held = std::min(held, 1);
        const int n = std::min(ds.nvs - s, ds.slots - held);
        k_lat_value<DIM><<<dim3((unsigned)L.ntiles, (unsigned)n), LAT_THREADS, smem, st>>>(
            L, a, tpack, S.shift, S.step, ds.tslice, s, vpart + held * stride);
        s += n;
        held += n;
    }
    k_lat_merge<DIM><<<(unsigned)ds.nval, LAT_THREADS, 0, st>>>(L, a, K, held, ds.lat_grad, vpart, S.shift, tpack,
                                                                c->rho.p, c->jxw.p, Lq, blkpart);
}

template <int DIM>
static void launch_lat_grad(const sdot_ctx *c, const DenseShape &ds, const double *tpack, const EvalArgs &a,
                            double *vpart, double *gpart, cudaStream_t st)
{
    const LatArgs L = lat_args(c, ds.lat);
    const LatScratch S(ds, vpart, a.nt, DIM);
    const size_t smem = sizeof(LatGradSmem<DIM>);
    lat_smem_limit(k_lat_grad<DIM>, smem);
    k_lat_grad<DIM><<<dim3((unsigned)((a.nt + LAT_GT - 1) / LAT_GT), (unsigned)ds.nks), LAT_THREADS, smem, st>>>(
        L, a, tpack, S.shift, S.step, vpart, ds.gts, gpart);
}

template <int DIM>
static void launch_value_dense_tensor(const sdot_ctx *c, const DenseShape &ds, const double *tpack,
                                      const EvalArgs &a, double *ms, cudaStream_t st)
{
    const dim3 grid((unsigned)ds.ncb, (unsigned)ds.nvs);
    Spacing ua;
    for (int d = 0; d < 3; ++d) ua.a[d] = c->tensor_a[d];
    auto go = [&](auto kern) {
        kern<<<grid, DENSE_A_THREADS, 0, st>>>(c->x.p, tpack, a, c->ncells, ds.tslice, ua, ms);
    };
    const bool uni = c->tensor_uniform;
    if constexpr (DIM == 2) {
        if (ds.tm == 3) uni ? go(k_value_dense_tensor<2, 3, true>) : go(k_value_dense_tensor<2, 3, false>);
        else uni ? go(k_value_dense_tensor<2, 2, true>) : go(k_value_dense_tensor<2, 2, false>);
    } else {
        uni ? go(k_value_dense_tensor<3, 2, true>) : go(k_value_dense_tensor<3, 2, false>);
    }
}

// The tensor-cell gradient sweep runs on the tensor value sweep's cells; its
// FP32 form only where a cell's factors span at most 2^60 (their exponents
// vary by H log2(e) / eps |C - y| a_d (TM - 1) per dimension, |C - y| <= diam).
static bool dense_grad_tensor(const sdot_ctx *c, int tm, bool fp32, const EvalArgs &a)
{
    if (tm <= 0) return false;
    if (!fp32) return true;
    const double spread = (tm == 2 ? 2.0 : 1.0) * a.l2e_eps * c->diam * c->tensor_amax * (tm - 1) * c->dim;
    return spread <= 60.0;
}

template <int DIM>
static void launch_grad_dense(const sdot_ctx *c, const DenseShape &ds, bool fp32, const double *Lq,
                              const double *tpack, const double *psi, const EvalArgs &a, double *gpart,
                              cudaStream_t st)
{
    const dim3 g((unsigned)ds.tb, (unsigned)ds.nks);
    if (dense_grad_tensor(c, ds.tm, fp32, a)) {
        const int64_t cs = (c->ncells + ds.nks - 1) / ds.nks;
        Spacing ua;
        for (int d = 0; d < 3; ++d) ua.a[d] = c->tensor_a[d];
        auto go = [&](auto kern) {
            kern<<<g, DENSE_B_CTA, 0, st>>>(c->x.p, c->w.p, Lq, tpack, psi, a, c->ncells, cs, ua, gpart);
        };
        const bool uni = c->tensor_uniform;
        if constexpr (DIM == 2) {
            if (ds.tm == 3) {
                if (fp32) go(k_grad_dense_tensor<2, 3, true, false>);
                else uni ? go(k_grad_dense_tensor<2, 3, false, true>) : go(k_grad_dense_tensor<2, 3, false, false>);
            } else {
                if (fp32) go(k_grad_dense_tensor<2, 2, true, false>);
                else uni ? go(k_grad_dense_tensor<2, 2, false, true>) : go(k_grad_dense_tensor<2, 2, false, false>);
            }
        } else {
            if (fp32) go(k_grad_dense_tensor<3, 2, true, false>);
            else uni ? go(k_grad_dense_tensor<3, 2, false, true>) : go(k_grad_dense_tensor<3, 2, false, false>);
        }
        return;
    }
    const int64_t qslice = (a.nq + ds.nks - 1) / ds.nks;
    if (fp32) k_grad_dense<DIM, true><<<g, DENSE_B_CTA, 0, st>>>(c->x.p, c->w.p, Lq, tpack, psi, a, qslice, gpart);
    else k_grad_dense<DIM, false><<<g, DENSE_B_CTA, 0, st>>>(c->x.p, c->w.p, Lq, tpack, psi, a, qslice, gpart);
}

template <int DIM>
static sdot_status run_eval(sdot_ctx *c, const EvalArgs &a, bool dense, const double *pdir, double tol, bool partial,
                            const IoPtrs *gather, const IoPtrs *scatter)
{
    cudaStream_t st = c->stream;
    const int prec = c->precision;
    auto mark = [&](int i) {
        if (c->profiling) cudaEventRecord(c->pev[i], st);
    };
    mark(0);
    DenseShape ds{};
    if (dense && c->distance == 0) {
        ds = dense_shape_of(c, a.eps, prec == SDOT_PREC_FP64);
        cudaError_t e = c->vpart.alloc(ds.vpart_need(a.nq, a.nt, c->ntblk));
        if (e == cudaSuccess) e = c->gpart.alloc(ds.gpart_need(a.nt));
        if (e == cudaSuccess) e = c->blkpart.alloc((size_t)4 * ds.nval);
        if (e != cudaSuccess) return cuda_error(c, e, "dense sweep partials");
    }
    if (ds.lat.cap > 0) launch_lat_prep<DIM>(c, ds, c->psi.p, gather, a, c->tpack.p, c->vpart.p, st);
    else if (dense) launch_target_prep<DIM>(c, a, c->psi.p, gather, c->tpack.p);
    mark(1);
    int64_t nval = 0;
    int nks = 1;
    if (c->distance == 1) {
        // spherical distance: its own sweeps over every (point, target) pair
        mark(7);
        sdot_status s = run_spherical(c, a, c->current_distance_threshold, &nval);
        if (s != SDOT_OK) return s;
        mark(2);
        mark(3);
        c->klaunch[2] += 1;
        c->klaunch[3] += 1;
    } else if (dense) {
        nval = ds.nval;
        if (ds.lat.cap > 0) {
            launch_lat_value<DIM>(c, ds, c->tpack.p, a, c->vpart.p, c->Lq.p, c->blkpart.p, st);
        } else if (ds.tm > 0) {
            launch_value_dense_tensor<DIM>(c, ds, c->tpack.p, a, c->vpart.p, st);
            k_value_dense_merge<DIM><<<(unsigned)nval, MERGE_THREADS, 0, st>>>(c->x.p, c->rho.p, c->jxw.p, c->vpart.p,
                                                                               ds.nvs, a, c->Lq.p, c->blkpart.p);
        } else if (ds.nvs > 1) {
            k_value_dense_slice<DIM><<<dim3((unsigned)nval, (unsigned)ds.nvs), DENSE_A_THREADS, 0, st>>>(
                c->x.p, c->tpack.p, a, ds.tslice, c->vpart.p);
            k_value_dense_merge<DIM><<<(unsigned)nval, MERGE_THREADS, 0, st>>>(c->x.p, c->rho.p, c->jxw.p, c->vpart.p,
                                                                               ds.nvs, a, c->Lq.p, c->blkpart.p);
        } else {
            k_value_dense<DIM><<<(unsigned)nval, DENSE_A_THREADS, 0, st>>>(c->x.p, c->rho.p, c->jxw.p, c->tpack.p, a,
                                                                           c->Lq.p, c->blkpart.p);
        }
        mark(2);
        // gradient: target blocks x point (or cell) slices
        nks = ds.nks;
        if (ds.lat_grad) launch_lat_grad<DIM>(c, ds, c->tpack.p, a, c->vpart.p, c->gpart.p, st);
        else launch_grad_dense<DIM>(c, ds, prec != SDOT_PREC_FP64, c->Lq.p, c->tpack.p, c->psi.p, a, c->gpart.p, st);
    } else {
        nval = c->nsblk;
        k_target_prep_kd<DIM><<<grid_for(a.nt, 256), 256, 0, st>>>(a.nt, c->y.p, c->nu.p, c->psi.p, a, c->tpack.p);
        sdot_status s = run_trunc(c, a, c->current_distance_threshold);  // records pev 7, 2, 3
        if (s != SDOT_OK) return s;
    }
    if (dense) mark(3);
    FinArgs f{};
    f.nt = a.nt;
    f.nks = nks;
    f.gpart = c->gpart.p;
    f.nu = c->nu.p;
    f.psi = c->psi.p;
    f.pdir = pdir;
    f.tol = tol;
    f.sub_nu = partial ? 0 : 1;
    f.grad = c->grad.p;
    f.io = scatter;
    f.perm = c->perm.p;
    f.nval = nval;
    f.valpart = c->blkpart.p;
    f.redpart = c->redpart.p;
    f.ticket = c->ticket.p;
    f.scal = c->scal.p;
    f.scal_host = c->scal_host;
    launch_finalize(f, st);
    mark(4);
    c->klaunch[1] += 1;
    if (dense && c->distance == 0) {
        c->klaunch[2] += 1;
        c->klaunch[3] += 1;
    }
    c->klaunch[4] += 1;
    return cuda_error(c, cudaGetLastError(), "evaluate launch");
}

// Launch key of the untruncated evaluation's graph: every value its launches
// capture (arguments, sizes, buffer addresses).  Zero-filled before use, so
// that keys compare bytewise.
struct DenseGraphKey {
    EvalArgs a;
    const void *p[20];
    double tol;
    int64_t misc[4];
};

// Replays the context's graph when the key matches it; captures one on the
// second consecutive evaluation with the same key (the first one runs
// eagerly, so every buffer the launches use is allocated before the
// capture); anything else runs eagerly.  A capture that fails turns graphs
// off for the context and runs the evaluation eagerly.
template <class Body>
static sdot_status run_graphed(sdot_ctx *c, const DenseGraphKey &k, Body &&body)
{
    const unsigned char *kb = reinterpret_cast<const unsigned char *>(&k);
    const bool same = c->dg_key.size() == sizeof k && memcmp(c->dg_key.data(), kb, sizeof k) == 0;
    if (same && c->dg_exec) {
        const cudaError_t e = cudaGraphLaunch(c->dg_exec, c->stream);
        if (e != cudaSuccess) return cuda_error(c, e, "evaluation graph launch");
        for (int i = 0; i < 8; ++i) c->klaunch[i] += c->dg_launches[i];
        return SDOT_OK;
    }
    if (c->dg_exec) {
        cudaGraphExecDestroy(c->dg_exec);
        c->dg_exec = nullptr;
    }
    if (!same || !c->dg_armed) {
        c->dg_key.assign(kb, kb + sizeof k);
        c->dg_armed = true;
        return body();
    }
    int64_t before[8];
    memcpy(before, c->klaunch, sizeof before);
    cudaGraph_t g = nullptr;
    cudaError_t e = cudaStreamBeginCapture(c->stream, cudaStreamCaptureModeThreadLocal);
    sdot_status s = SDOT_OK;
    if (e == cudaSuccess) {
        s = body();
        e = cudaStreamEndCapture(c->stream, &g);
        if (s == SDOT_OK && e == cudaSuccess && g) e = cudaGraphInstantiate(&c->dg_exec, g, 0);
        if (g) cudaGraphDestroy(g);
    }
    if (s != SDOT_OK || e != cudaSuccess || !c->dg_exec) {
        cudaGetLastError();
        if (c->dg_exec) cudaGraphExecDestroy(c->dg_exec);
        c->dg_exec = nullptr;
        c->graphs_off = true;
        memcpy(c->klaunch, before, sizeof before);
        return body();
    }
    for (int i = 0; i < 8; ++i) c->dg_launches[i] = c->klaunch[i] - before[i];
    e = cudaGraphLaunch(c->dg_exec, c->stream);
    return e == cudaSuccess ? SDOT_OK : cuda_error(c, e, "evaluation graph launch");
}

sdot_status evaluate_internal(sdot_ctx *c, const double *p_dir, double comp_tol, double *ms_out, bool partial)
{
    EvalPending pend;
    sdot_status s = evaluate_enqueue(c, p_dir, comp_tol, partial, pend);
    if (s != SDOT_OK) return s;
    const cudaError_t e = cudaStreamSynchronize(c->stream);
    if (e != cudaSuccess) return cuda_error(c, e, "evaluate");
    return evaluate_complete(c, pend, ms_out);
}

sdot_status evaluate_enqueue(sdot_ctx *c, const double *p_dir, double comp_tol, bool partial, EvalPending &pend,
                             const IoPtrs *io)
{
    if (c->dim == 0 || c->nq == 0) return set_error(c, SDOT_ESTATE, "source measure not set");
    if (c->nt == 0) return set_error(c, SDOT_ESTATE, "target measure not set");
    const sdot_solver_params &p = c->prm;
    if (c->distance == 1 && p.threshold_type != SDOT_THRESH_POINTWISE)
        return set_error(c, SDOT_EINVAL, "the spherical distance is supported with the pointwise threshold");
    // threshold (host, exact libm), from device max/min of psi
    double r = DBL_MAX;
    const bool may_truncate = (p.threshold_type != SDOT_THRESH_POINTWISE) ||
                              (p.tau > 0 && (c->min_target_density > 0.0 ? c->min_target_density
                                                                          : c->nu_min) > 0);
    if (io && !(*io == c->io_set)) {
        const cudaError_t e = cudaMemcpyAsync(c->io_ptrs.p, io, sizeof *io, cudaMemcpyHostToDevice, c->stream);
        if (e != cudaSuccess) return cuda_error(c, e, "caller arrays");
        c->io_set = *io;
    }
    cudaEventRecord(c->ev0, c->stream);
    const IoPtrs *gather = io ? c->io_ptrs.p : nullptr, *scatter = gather;  // of the evaluation's first and last kernel
    if (may_truncate) {
        if (c->profiling) cudaEventRecord(c->pev[5], c->stream);
        const int64_t blocks = (c->nt + RANGE_THREADS * 4 - 1) / (RANGE_THREADS * 4);
        k_psi_range<<<(unsigned)std::min<int64_t>(RANGE_BLOCKS, blocks), RANGE_THREADS, 0, c->stream>>>(
            c->nt, io ? io->psi : nullptr, io ? c->perm.p : nullptr, c->psi.p, c->redpart.p, c->ticket.p + 1,
            c->scal.p + SC_MAXPSI, c->scal_host + SC_MAXPSI);
        static_assert(SC_MINPSI == SC_MAXPSI + 1 && SC_PSIBAD == SC_MAXPSI + 2, "range slots");
        gather = nullptr;
        if (c->profiling) cudaEventRecord(c->pev[6], c->stream);
        c->klaunch[0] += 1;
        const cudaError_t e = cudaStreamSynchronize(c->stream);
        if (e != cudaSuccess) return cuda_error(c, e, "threshold readback");
        if (c->scal_host[SC_PSIBAD] != 0.0) return set_error(c, SDOT_ENONFINITE, "non-finite potential");
        r = host_threshold(c, c->scal_host[SC_MAXPSI], c->scal_host[SC_MINPSI]);
    } else if (io && c->distance != 0) {
        const sdot_status s = launch_gather(c, c->psi.p, io->psi, c->nt);
        if (s != SDOT_OK) return s;
        gather = nullptr;
    }
    c->current_distance_threshold = r;
    const double sstar = sstar_of(r);
    const bool dense = !(r < c->diam * (1.0 + 1e-12)) || std::isinf(r) ? true : false;
    const bool dense_ok = dense && !std::isnan(r);

    EvalArgs a{};
    a.qpc = c->qpc;
    a.ql = c->ql;
    a.ngroups = c->ngroups;
    a.lse = p.use_log_sum_exp;
    a.nq = c->nq;
    a.ncells = c->ncells;
    a.nunits = c->ncells * a.ngroups;
    a.nt = c->nt;
    a.eps = p.epsilon;
    a.s = KAPPA / p.epsilon;
    a.halfs = 0.5 * a.s;
    for (int d = 0; d < 3; ++d) a.o[d] = c->origin[d];
    a.sstar = sstar;
    a.cull = std::isnan(r) ? 0.0 : std::min(r, 1e300);
    a.c32 = LOG2E / (2.0 * p.epsilon);
    a.l2e_eps = LOG2E / p.epsilon;

    if (!dense_ok && std::isnan(r)) {
        // NaN threshold: the reference's predicate d <= NaN rejects everything
        a.sstar = NAN;
    }
    // everything after the threshold (an untruncated evaluation needs no ψ range)
    auto body = [&]() -> sdot_status {
        return (c->dim == 2) ? run_eval<2>(c, a, dense_ok, p_dir, comp_tol, partial, gather, scatter)
                             : run_eval<3>(c, a, dense_ok, p_dir, comp_tol, partial, gather, scatter);
    };
    // An untruncated euclidean evaluation has no host step between its
    // launches, so it runs as one CUDA graph once its launch key repeats.
    sdot_status s;
    if (!may_truncate && dense_ok && c->distance == 0 && !c->profiling && !c->graphs_off) {
        DenseGraphKey k;
        memset(&k, 0, sizeof k);
        k.a = a;
        const void *ptrs[] = {c->psi.p, c->y.p, c->nu.p, c->x.p, c->rho.p, c->jxw.p, c->w.p, c->tpack.p,
                              c->vpart.p, c->Lq.p, c->blkpart.p, c->gpart.p, c->grad.p, c->redpart.p,
                              c->scal.p, c->scal_host, p_dir, c->io_ptrs.p, c->ticket.p};
        static_assert(sizeof(ptrs) <= sizeof(k.p), "key pointer slots");
        memcpy(k.p, ptrs, sizeof(ptrs));
        k.tol = comp_tol;
        k.misc[0] = c->dim;
        k.misc[1] = c->precision;
        k.misc[2] = (partial ? 1 : 0) + (io ? 2 : 0);
        k.misc[3] = c->geometry_id;
        s = run_graphed(c, k, body);
    } else {
        s = body();
    }
    if (s != SDOT_OK) return s;
    cudaEventRecord(c->ev1, c->stream);
    pend.r = r;
    pend.dense = dense_ok;
    pend.ranged = may_truncate;
    return SDOT_OK;
}

sdot_status evaluate_complete(sdot_ctx *c, const EvalPending &pend, double *ms_out)
{
    const double r = pend.r;
    const bool dense_ok = pend.dense;
    if (ms_out) {
        float ms = 0.f;
        cudaEventElapsedTime(&ms, c->ev0, c->ev1);
        *ms_out = ms;
    }
    if (c->profiling) {
        float t = 0.f;
        if (pend.ranged) {
            cudaEventElapsedTime(&t, c->pev[5], c->pev[6]);
            c->kms[0] += t;
        }
        cudaEventElapsedTime(&t, c->pev[0], c->pev[1]);
        c->kms[1] += t;
        if (dense_ok) {
            cudaEventElapsedTime(&t, c->pev[1], c->pev[2]);
            c->kms[2] += t;
        } else {
            cudaEventElapsedTime(&t, c->pev[1], c->pev[7]);
            c->kms[6] += t;
            cudaEventElapsedTime(&t, c->pev[7], c->pev[2]);
            c->kms[2] += t;
        }
        cudaEventElapsedTime(&t, c->pev[2], c->pev[3]);
        c->kms[3] += t;
        cudaEventElapsedTime(&t, c->pev[3], c->pev[4]);
        c->kms[4] += t;
    }
    c->scal_host[SC_R] = r;
    if (!pend.ranged) {
        // no ψ range was computed (untruncated): the slots say so
        c->scal_host[SC_MAXPSI] = NAN;
        c->scal_host[SC_MINPSI] = NAN;
        c->scal_host[SC_PSIBAD] = 0.0;
    }
    c->global_functional = c->scal_host[SC_VALUE];
    c->C_global = c->scal_host[SC_C];
    if (c->scal_host[SC_NONFINITE] != 0.0) return set_error(c, SDOT_ENONFINITE, "non-finite value or gradient");
    return SDOT_OK;
}

}  // namespace sdot

// ---------------------------------------------------------------------------
// No-allocation dense evaluation (sdot_evaluate_device_noalloc).
//
// The scratch of one untruncated evaluation (gathered psi, gradient, packed
// targets, L_q, gradient partials per q-slice, value / reduction partials,
// scalars) lives in one file-scope device array of NOALLOC_BYTES instead of
// the context's lazily allocated evaluation buffers.  Its device address is
// looked up once per device with cudaGetSymbolAddress and cached for the
// life of the process; a cudaDeviceReset by the host application frees the
// module instance the cached address points into, so no-alloc calls must not
// follow one.  Every scratch word the evaluation reads is written earlier by
// the same evaluation on the same stream (the finalize kernel's arrival
// counter is cleared first): nothing has to start at zero.  The array is
// shared by every context of the process on a device, so calls whose
// executions overlap corrupt each other, but no call after them.
// ---------------------------------------------------------------------------

namespace sdot {

constexpr size_t NOALLOC_BYTES = size_t(8) << 20;  // == SDOT_NOALLOC_SCRATCH_BYTES
constexpr int NOALLOC_MAX_DEVICES = 64;

// (its last words hold the finalize kernel's arrival counter)
static __device__ __align__(256) double g_noalloc_scratch[NOALLOC_BYTES / sizeof(double) + 32];

static double *g_noalloc_ptr[NOALLOC_MAX_DEVICES] = {};
static std::mutex g_noalloc_mu;

// Scratch segments of an evaluation, each rounded up to 256 bytes.
struct NoallocLayout {
    int64_t psi, grad, tpack, Lq, gpart, blkpart, redpart, scal, vpart, total;  // offsets in doubles
    int64_t nval;
    int nks;
    int nvs;
    int64_t tslice;
    DenseShape ds;
};

static NoallocLayout noalloc_layout(const sdot_ctx *c, const DenseShape &ds)
{
    const int64_t nq = c->nq, nt = c->nt;
    auto up = [](int64_t n) { return (n + 31) / 32 * 32; };
    NoallocLayout L{};
    L.ds = ds;
    L.nval = ds.nval;
    L.nks = ds.nks;
    L.nvs = ds.nvs;
    L.tslice = ds.tslice;
    int64_t o = 0;
    L.psi = o;     o += up(nt);
    L.grad = o;    o += up(nt);
    L.tpack = o;   o += up(nt * TPACK);
    L.Lq = o;      o += up(nq);
    L.gpart = o;   o += up((int64_t)L.nks * nt);
    L.blkpart = o; o += up(4 * L.nval);
    L.redpart = o; o += up((int64_t)FIN_BLOCKS * NRED);
    L.scal = o;    o += up(SC_COUNT);
    L.vpart = o;   o += up((int64_t)ds.vpart_need(nq, nt, c->ntblk));
    L.total = o;
    return L;
}

static sdot_status noalloc_scratch(sdot_ctx *c, double **out)
{
    if (c->device < 0 || c->device >= NOALLOC_MAX_DEVICES)
        return set_error(c, SDOT_EINVAL, "no-alloc evaluation: device ordinal out of range");
    std::lock_guard<std::mutex> lk(g_noalloc_mu);
    if (!g_noalloc_ptr[c->device]) {
        double *p = nullptr;
        const cudaError_t e = cudaGetSymbolAddress((void **)&p, g_noalloc_scratch);
        if (e != cudaSuccess) return cuda_error(c, e, "no-alloc evaluation: cudaGetSymbolAddress of the scratch array");
        g_noalloc_ptr[c->device] = p;
    }
    *out = g_noalloc_ptr[c->device];
    return SDOT_OK;
}

template <int DIM>
static void noalloc_launch(sdot_ctx *c, const EvalArgs &a, double *S, unsigned *ticket, const NoallocLayout &L)
{
    cudaStream_t st = c->stream;
    double *psi = S + L.psi, *grad = S + L.grad, *tpack = S + L.tpack, *Lq = S + L.Lq, *gpart = S + L.gpart;
    double *blkpart = S + L.blkpart, *redpart = S + L.redpart, *scal = S + L.scal;
    if (L.ds.lat.cap > 0) launch_lat_prep<DIM>(c, L.ds, psi, nullptr, a, tpack, S + L.vpart, st);
    else launch_target_prep<DIM>(c, a, psi, nullptr, tpack);
    if (L.ds.lat.cap > 0) {
        launch_lat_value<DIM>(c, L.ds, tpack, a, S + L.vpart, Lq, blkpart, st);
    } else if (L.ds.tm > 0) {
        double *vpart = S + L.vpart;
        launch_value_dense_tensor<DIM>(c, L.ds, tpack, a, vpart, st);
        k_value_dense_merge<DIM><<<(unsigned)L.nval, MERGE_THREADS, 0, st>>>(c->x.p, c->rho.p, c->jxw.p, vpart, L.nvs,
                                                                             a, Lq, blkpart);
    } else if (L.nvs > 1) {
        double *vpart = S + L.vpart;
        k_value_dense_slice<DIM><<<dim3((unsigned)L.nval, (unsigned)L.nvs), DENSE_A_THREADS, 0, st>>>(
            c->x.p, tpack, a, L.tslice, vpart);
        k_value_dense_merge<DIM><<<(unsigned)L.nval, MERGE_THREADS, 0, st>>>(c->x.p, c->rho.p, c->jxw.p, vpart, L.nvs,
                                                                             a, Lq, blkpart);
    } else {
        k_value_dense<DIM><<<(unsigned)L.nval, DENSE_A_THREADS, 0, st>>>(c->x.p, c->rho.p, c->jxw.p, tpack, a, Lq,
                                                                          blkpart);
    }
    if (L.ds.lat_grad) launch_lat_grad<DIM>(c, L.ds, tpack, a, S + L.vpart, gpart, st);
    else launch_grad_dense<DIM>(c, L.ds, c->precision != SDOT_PREC_FP64, Lq, tpack, psi, a, gpart, st);
    FinArgs f{};
    f.nt = a.nt;
    f.nks = L.nks;
    f.gpart = gpart;
    f.nu = c->nu.p;
    f.psi = psi;
    f.tol = c->prm.tolerance;
    f.sub_nu = 1;
    f.grad = grad;
    f.perm = c->perm.p;
    f.nval = L.nval;
    f.valpart = blkpart;
    f.redpart = redpart;
    f.ticket = ticket;
    f.scal = scal;
    f.scal_host = c->scal_host;
    launch_finalize(f, st);
}

}  // namespace sdot

extern "C" sdot_status sdot_evaluate_device_noalloc(sdot_ctx *c, const double *psi_dev, double *grad_dev,
                                                    double *value)
{
    using namespace sdot;
    if (!c || !psi_dev || !grad_dev) return SDOT_EINVAL;
    if (c->dim == 0 || c->nq == 0) return set_error(c, SDOT_ESTATE, "source measure not set");
    if (c->nt == 0) return set_error(c, SDOT_ESTATE, "target measure not set");
    const sdot_solver_params &p = c->prm;
    if (p.threshold_type != SDOT_THRESH_POINTWISE || p.tau > 0)
        return set_error(c, SDOT_EINVAL,
                         "no-alloc evaluation covers untruncated problems only (pointwise threshold, tau <= 0)");
    if (c->distance != 0) return set_error(c, SDOT_EINVAL, "no-alloc evaluation covers the euclidean distance only");
    // The launch shape of the allocating path.  Where the lattice sweeps' partials exceed the scratch but the cell
    // or point sweeps' would not, as many target slices at a time as fit (the sums keep their order); only where not
    // even two fit, the cell or point sweeps, which round differently.
    DenseShape ds = dense_shape_of(c, p.epsilon, c->precision == SDOT_PREC_FP64);
    NoallocLayout L = noalloc_layout(c, ds);
    constexpr int64_t CAP = NOALLOC_BYTES / sizeof(double);
    if (L.total > CAP && ds.lat.cap > 0) {
        const int64_t per = (int64_t)ds.lat.ntiles * LAT_TILE;
        ds.slots = (int)(ds.nvs - std::min<int64_t>(ds.nvs, (L.total - CAP + per - 1) / per));
        const NoallocLayout other =
            noalloc_layout(c, dense_shape(c->nq, c->nt, dense_tensor_m(c, KAPPA / p.epsilon), c->ncells));
        L = other.total <= CAP && ds.slots >= 2 ? noalloc_layout(c, ds) : other;
    }
    const size_t need = (size_t)L.total * sizeof(double);
    if (need > NOALLOC_BYTES)
        return set_error(c, SDOT_EINVAL,
                         "no-alloc evaluation needs " + std::to_string(need) + " bytes of scratch; the static limit is " +
                             std::to_string(NOALLOC_BYTES) + " bytes (use sdot_evaluate_device)");
    int prev = -1;
    cudaGetDevice(&prev);
    if (prev != c->device) {
        const cudaError_t e = cudaSetDevice(c->device);
        if (e != cudaSuccess) return cuda_error(c, e, "no-alloc evaluation: set device");
    }
    struct Restore {
        int dev;
        ~Restore() {
            if (dev >= 0) cudaSetDevice(dev);
        }
    } restore{prev != c->device ? prev : -1};
    double *S = nullptr;
    sdot_status s = noalloc_scratch(c, &S);
    if (s != SDOT_OK) return s;

    EvalArgs a{};
    a.qpc = c->qpc;
    a.ql = c->ql;
    a.ngroups = c->ngroups;
    a.lse = p.use_log_sum_exp;
    a.nq = c->nq;
    a.ncells = c->ncells;
    a.nunits = c->ncells * a.ngroups;
    a.nt = c->nt;
    a.eps = p.epsilon;
    a.s = KAPPA / p.epsilon;
    a.halfs = 0.5 * a.s;
    for (int d = 0; d < 3; ++d) a.o[d] = c->origin[d];
    a.sstar = sstar_of(DBL_MAX);
    a.cull = 1e300;
    a.c32 = LOG2E / (2.0 * p.epsilon);
    a.l2e_eps = LOG2E / p.epsilon;

    if ((s = launch_gather(c, S + L.psi, psi_dev, c->nt)) != SDOT_OK) return s;
    unsigned *ticket = reinterpret_cast<unsigned *>(S + NOALLOC_BYTES / sizeof(double));
    // not left to the kernel's own wrap to zero: two overlapping calls of different grids can leave it elsewhere
    cudaError_t e = cudaMemsetAsync(ticket, 0, sizeof *ticket, c->stream);
    if (e != cudaSuccess) return cuda_error(c, e, "no-alloc evaluation");
    if (c->dim == 2) noalloc_launch<2>(c, a, S, ticket, L);
    else noalloc_launch<3>(c, a, S, ticket, L);
    e = cudaGetLastError();
    if (e != cudaSuccess) return cuda_error(c, e, "no-alloc evaluation launch");
    if ((s = launch_scatter(c, grad_dev, S + L.grad, c->nt)) != SDOT_OK) return s;
    // k_finalize writes slots SC_VALUE .. SC_VALSRC of the host's array except the
    // psi range, the psi check and the threshold slots (the untruncated path needs
    // none of them), which are set below.
    e = cudaStreamSynchronize(c->stream);
    if (e != cudaSuccess) return cuda_error(c, e, "no-alloc evaluation");
    c->scal_host[SC_MAXPSI] = NAN;
    c->scal_host[SC_MINPSI] = NAN;
    c->scal_host[SC_PSIBAD] = 0.0;
    c->scal_host[SC_SSTAR] = a.sstar;
    for (int i = SC_VALSRC + 1; i < SC_COUNT; ++i) c->scal_host[i] = 0.0;
    c->klaunch[1] += 1;
    c->klaunch[2] += 1;
    c->klaunch[3] += 1;
    c->klaunch[4] += 1;
    c->current_distance_threshold = DBL_MAX;
    c->scal_host[SC_R] = DBL_MAX;
    c->global_functional = c->scal_host[SC_VALUE];
    c->C_global = c->scal_host[SC_C];
    c->last_pairs = (int64_t)((double)c->nq * (double)c->nt);
    if (value) *value = c->scal_host[SC_VALUE];
    if (c->scal_host[SC_NONFINITE] != 0.0) return set_error(c, SDOT_ENONFINITE, "non-finite value or gradient");
    return SDOT_OK;
}
