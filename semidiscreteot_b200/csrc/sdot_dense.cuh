// sdot_dense.cuh -- per-CTA bodies of the untruncated (dense) value and
// gradient sweeps, shared by the single-problem kernels (sdot_eval.cu) and
// the batched persistent kernels (sdot_batch.cu).
#pragma once

#include <float.h>
#include <limits.h>

#include "sdot_device.cuh"

namespace sdot {

// ---------------------------------------------------------------------------
// value sweep, dense: thread <-> quadrature point, all targets streamed
// through shared memory (broadcast reads).
// ---------------------------------------------------------------------------

constexpr int DA_CHUNK = 256;
constexpr int DA_U = 8;  // targets per step of the sweep

// A point's log-sum-exp under way: S relative to M, the largest exponent mx
// (M <= mx <= M + LSE_THR) and the high word of mx - M (INT_MIN before the
// first finite exponent).
struct LsePoint {
    double M, S, mx;
    int top;
};

// Adds U targets (scaled exponents b, weights nu) to a point's sum.  A new
// maximum is rare and is found by one integer comparison per target: b - M
// and mx - M order as their high words do, and every negative difference has
// a negative high word.  Only then is the maximum compared in FP64, and only
// beyond LSE_THR (or with a NaN difference, which ends at exp2_16's lower
// clamp) is the reference moved: three FP64 comparisons per target cost as
// much as its exponential.  The clamp itself is an unsigned minimum on the
// high word (larger words are more negative numbers).  The U exponentials
// have no branch between them, so their chains overlap.
template <int U>
__device__ __forceinline__ void lse_group(const double *b, const double *nu, LsePoint &P, const double *tab)
{
    double u[U];
    int h = INT_MIN;
#pragma unroll
    for (int i = 0; i < U; ++i) {
        u[i] = b[i] - P.M;
        h = max(h, __double2hiint(u[i]));
    }
    if (h >= P.top) {
        double bm = b[0];
#pragma unroll
        for (int i = 1; i < U; ++i) bm = fmax(bm, b[i]);
        P.mx = fmax(P.mx, bm);
        if (h >= LSE_THR_HI || P.top == INT_MIN) {
            if (bm - P.M > LSE_THR) {
                P.S *= exp2_16(P.M - bm, tab);
                P.M = bm;
            }
#pragma unroll
            for (int i = 0; i < U; ++i) u[i] = b[i] == P.M ? 0.0 : fmax(b[i] - P.M, EXP2_CLAMP);
        }
        P.top = P.mx > -CUDART_INF ? __double2hiint(P.mx - P.M) : INT_MIN;
    }
#pragma unroll
    for (int i = 0; i < U; ++i) {
        const unsigned hi = min((unsigned)__double2hiint(u[i]), (unsigned)CLAMP_HI);
        u[i] = exp2_16_nc(__hiloint2double((int)hi, __double2loint(u[i])), tab);
    }
#pragma unroll
    for (int i = 0; i < U; ++i) P.S = fma(nu[i], u[i], P.S);
}

// One thread's point q of block blk, xt relative to the source's origin, and
// its sum over the targets [t0, t1), staged DA_CHUNK at a time as 16-byte
// aligned records (A, B, nu; the last step is padded with exponents of -inf
// and no weight).  Bound by the FP64 pipe and the shared-memory reads beside
// it: 122,880 points x 1,000 targets (3D) 282 -> 176 us, 0.70e12 pairs/s, 14
// FP64 operations each.  Two points per thread (fewer reads, fewer warps)
// measured 178 to 226 us, 4 or 16 targets per step 196 and 175.
template <int DIM>
struct DensePoint {
    int64_t q;
    double xt[DIM];
    LsePoint P;

    __device__ __forceinline__ void sweep(const double *__restrict__ x, const double *__restrict__ tpack,
                                          const EvalArgs &a, int64_t blk, int64_t t0, int64_t t1, const double *tab)
    {
        constexpr int TS = DIM == 2 ? 4 : 6;
        __shared__ __align__(16) double stg[DA_CHUNK * TS];
        q = blk * DENSE_A_THREADS + threadIdx.x;
#pragma unroll
        for (int d = 0; d < DIM; ++d) xt[d] = (q < a.nq) ? x[q * DIM + d] - a.o[d] : 0.0;
        P = LsePoint{-CUDART_INF, 0.0, -CUDART_INF, INT_MIN};
        for (int64_t c0 = t0; c0 < t1; c0 += DA_CHUNK) {
            const int cn = (int)min((int64_t)DA_CHUNK, t1 - c0);
            const int cu = (cn + DA_U - 1) / DA_U * DA_U;
            __syncthreads();
            for (int i = threadIdx.x; i < cu * TS; i += DENSE_A_THREADS) {
                const int t = i / TS, f = i - t * TS;
                stg[i] = t < cn ? (f < DIM + 2 ? tpack[(c0 + t) * TPACK + f] : 0.0) : (f == 0 ? -CUDART_INF : 0.0);
            }
            __syncthreads();
#pragma unroll 1
            for (int t = 0; t < cu; t += DA_U) {
                double b[DA_U], nu[DA_U];
#pragma unroll
                for (int i = 0; i < DA_U; ++i) {
                    const double2 *tp = reinterpret_cast<const double2 *>(stg + (t + i) * TS);
                    const double2 r0 = tp[0], r1 = tp[1];
                    b[i] = fma(r1.x, xt[1], fma(r0.y, xt[0], r0.x));
                    if (DIM == 3) b[i] = fma(r1.y, xt[DIM - 1], b[i]);
                    nu[i] = DIM == 3 ? tp[DIM - 1].x : r1.y;
                }
                lse_group<DA_U>(b, nu, P, tab);
            }
        }
    }

    // the sum relative to the largest exponent
    __device__ __forceinline__ double sum(const double *tab) const
    {
        return (P.mx == -CUDART_INF) ? 0.0 : P.S * exp2_16(P.M - P.mx, tab);
    }
};

// One CTA's work of the dense value sweep: quadrature points
// [blk * DENSE_A_THREADS, +DENSE_A_THREADS) of one source against all its
// targets; writes L_q and the block's (value, C, skipped, 0) to out4.
// Shared by the single-problem kernel and the batched one.
template <int DIM>
__device__ __forceinline__ void dense_value_block(const double *__restrict__ x, const double *__restrict__ rho,
                                                  const double *__restrict__ jxw, const double *__restrict__ tpack,
                                                  const EvalArgs &a, int64_t blk, double *__restrict__ Lq,
                                                  double *__restrict__ out4)
{
    __shared__ double tab[16];
    if (threadIdx.x < 16) tab[threadIdx.x] = c_exp2_tab[threadIdx.x];
    DensePoint<DIM> D;
    D.sweep(x, tpack, a, blk, 0, a.nt, tab);
    double tv = 0.0, tc = 0.0, ts = 0.0;
    if (D.q < a.nq) {
        double xsq = 0.0;
#pragma unroll
        for (int d = 0; d < DIM; ++d) xsq += D.xt[d] * D.xt[d];
        double L;
        int sk;
        value_epilogue(a, D.P.mx, D.sum(tab), -a.halfs * xsq, rho[D.q], jxw[D.q], tv, tc, L, sk);
        Lq[D.q] = L;
        ts = sk;
    }
    block_partials_at(tv, tc, ts, 0.0, out4);
}

// The same sweep over one slice of the targets [t0, t1), for problems too
// small to fill the GPU with one CTA per point block: per point it writes
// the slice's largest scaled exponent mx and the sum relative to it,
// ms[2 q] = mx, ms[2 q + 1] = sum_j nu_j 2^((b_qj - mx)/16); the merge
// (dense_value_merge) combines the slices in slice order and finishes.
template <int DIM>
__device__ __forceinline__ void dense_value_slice(const double *__restrict__ x, const double *__restrict__ tpack,
                                                  const EvalArgs &a, int64_t blk, int64_t t0, int64_t t1,
                                                  double *__restrict__ ms)
{
    __shared__ double tab[16];
    if (threadIdx.x < 16) tab[threadIdx.x] = c_exp2_tab[threadIdx.x];
    DensePoint<DIM> D;
    D.sweep(x, tpack, a, blk, t0, t1, tab);
    if (D.q < a.nq) {
        ms[2 * D.q] = D.P.mx;
        ms[2 * D.q + 1] = D.sum(tab);
    }
}

// Merge of the target slices of point block blk (slice s of point q at
// ms[s * 2 nq + 2 q ..]) by DENSE_MERGE_SPLIT lanes per point: lane u takes
// the slices s = u, u + SPLIT, ... (their loads in flight together); the
// largest exponent over the slices, each lane's sums rescaled to it and
// added in order of s, the lanes' sums added by xor exchanges in a fixed
// tree; then the epilogue of dense_value_block (L_q, value, C, skipped) and
// the block's partials.  The CTA has DENSE_A_THREADS * SPLIT threads.
constexpr int DENSE_MERGE_SPLIT = 4;

template <int DIM>
__device__ __forceinline__ void dense_value_merge(const double *__restrict__ x, const double *__restrict__ rho,
                                                  const double *__restrict__ jxw, const double *__restrict__ ms,
                                                  int nslice, const EvalArgs &a, int64_t blk,
                                                  double *__restrict__ Lq, double *__restrict__ out4)
{
    constexpr int SP = DENSE_MERGE_SPLIT;
    __shared__ double tab[16];
    if (threadIdx.x < 16) tab[threadIdx.x] = c_exp2_tab[threadIdx.x];
    __syncthreads();
    const int u = threadIdx.x % SP;
    const int64_t q = blk * DENSE_A_THREADS + threadIdx.x / SP;
    const bool ok = q < a.nq;
    const double *mq = ms + 2 * (ok ? q : 0);
    const int64_t st = 2 * a.nq;
    double mx = -CUDART_INF;
    if (ok)
        for (int s = u; s < nslice; s += SP) mx = fmax(mx, mq[s * st]);
#pragma unroll
    for (int o = 1; o < SP; o <<= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    double S = 0.0;
    if (ok && mx > -CUDART_INF)
        for (int s = u; s < nslice; s += SP) {
            const double2 v = *reinterpret_cast<const double2 *>(mq + s * st);
            if (v.x > -CUDART_INF) S += v.y * exp2_16(v.x - mx, tab);
        }
#pragma unroll
    for (int o = 1; o < SP; o <<= 1) S += __shfl_xor_sync(0xffffffffu, S, o);
    double tv = 0.0, tc = 0.0, ts = 0.0;
    if (ok && u == 0) {
        double xsq = 0.0;
#pragma unroll
        for (int d = 0; d < DIM; ++d) {
            const double xt = x[q * DIM + d] - a.o[d];
            xsq += xt * xt;
        }
        const double Cq = -a.halfs * xsq;
        double v, cv, L;
        int sk;
        value_epilogue(a, mx, S, Cq, rho[q], jxw[q], v, cv, L, sk);
        Lq[q] = L;
        tv = v;
        tc = cv;
        ts = sk;
    }
    block_partials_at(tv, tc, ts, 0.0, out4);
}

// ---------------------------------------------------------------------------
// gradient sweep, dense: thread <-> DENSE_B_TT targets, q-slices streamed
// through shared memory (broadcast reads); FP64 partial per (slice, target).
// ---------------------------------------------------------------------------

constexpr int DB_CHUNK = 256;

// Per-target data of one CTA of the gradient sweep: the TT targets j0 + lt +
// k * DENSE_B_THREADS of thread lane lt.  FP32: the CTA's target box centre
// ob and the reference aref = max_j (log2 nu_j + psi_j log2(e) / eps) (block
// reductions over the CTA's NTH threads), each target relative to ob (yt) and
// its exponent offset alpha = log2 nu_j + psi_j log2(e) / eps - aref; FP64:
// A_j and B_j of the packed target.
template <int TT>
struct GradTargets {
    double ob[3] = {0.0, 0.0, 0.0};
    double aref = 0.0;
    float yt[TT][3], alpha[TT];
    double A[TT], B[TT][3];
    bool has[TT];
};

template <int DIM, bool FP32, int NTH, int TT>
__device__ __forceinline__ void grad_targets(const double *__restrict__ tpack, const double *__restrict__ psi,
                                             const EvalArgs &a, int64_t j0, int lt, GradTargets<TT> &T)
{
    const int tid = threadIdx.x;
    if (FP32) {
        double lo[3] = {DBL_MAX, DBL_MAX, DBL_MAX}, hi[3] = {-DBL_MAX, -DBL_MAX, -DBL_MAX};
        double amax = -DBL_MAX;
#pragma unroll
        for (int k = 0; k < TT; ++k) {
            const int64_t j = j0 + lt + k * DENSE_B_THREADS;
            if (j < a.nt) {
                const double *tp = tpack + j * TPACK;
#pragma unroll
                for (int d = 0; d < DIM; ++d) {
                    lo[d] = fmin(lo[d], tp[2 + DIM + d]);
                    hi[d] = fmax(hi[d], tp[2 + DIM + d]);
                }
                const double al = log2(tp[1 + DIM]) + a.l2e_eps * psi[j];
                if (al > amax) amax = al;
            }
        }
        // block reductions (lo/hi/amax) through shared memory
        __shared__ double sred[7][NTH / 32];
        for (int o = 16; o > 0; o >>= 1) {
#pragma unroll
            for (int d = 0; d < DIM; ++d) {
                lo[d] = fmin(lo[d], __shfl_xor_sync(0xffffffffu, lo[d], o));
                hi[d] = fmax(hi[d], __shfl_xor_sync(0xffffffffu, hi[d], o));
            }
            amax = fmax(amax, __shfl_xor_sync(0xffffffffu, amax, o));
        }
        if ((tid & 31) == 0) {
#pragma unroll
            for (int d = 0; d < DIM; ++d) { sred[d][tid >> 5] = lo[d]; sred[3 + d][tid >> 5] = hi[d]; }
            sred[6][tid >> 5] = amax;
        }
        __syncthreads();
        for (int i = 0; i < NTH / 32; ++i) {
#pragma unroll
            for (int d = 0; d < DIM; ++d) { lo[d] = fmin(lo[d], sred[d][i]); hi[d] = fmax(hi[d], sred[3 + d][i]); }
            amax = fmax(amax, sred[6][i]);
        }
#pragma unroll
        for (int d = 0; d < DIM; ++d) T.ob[d] = 0.5 * (lo[d] + hi[d]);
        T.aref = (amax > -DBL_MAX && isfinite(amax)) ? amax : 0.0;
    }
#pragma unroll
    for (int k = 0; k < TT; ++k) {
        const int64_t j = j0 + lt + k * DENSE_B_THREADS;
        T.has[k] = j < a.nt;
        const double *tp = tpack + (T.has[k] ? j : 0) * TPACK;
        if (FP32) {
#pragma unroll
            for (int d = 0; d < 3; ++d) T.yt[k][d] = (d < DIM && T.has[k]) ? (float)(tp[2 + DIM + d] - T.ob[d]) : 0.f;
            T.alpha[k] = T.has[k] ? (float)(log2(tp[1 + DIM]) + a.l2e_eps * psi[j] - T.aref) : -INFINITY;
        } else {
            T.A[k] = tp[0];
#pragma unroll
            for (int d = 0; d < DIM; ++d) T.B[k][d] = tp[1 + d];
        }
    }
}

// One CTA's work of the dense gradient sweep: targets of block tblk against
// quadrature slice ks; writes gpart[ks * nt + j].  Shared by the
// single-problem kernel (QG = DENSE_B_QG) and the batched one (QG = 1).
// The CTA is QG groups of DENSE_B_THREADS threads: thread lt of every group
// holds the same TT targets, group g takes the staged points g, g + QG, ...,
// and the groups' sums are added in group order at the end, so a slice's
// partial does not depend on the scheduling.  FP32: a group's points lie one
// after the other, so that two of them share each packed instruction; the
// sums keep their order, an FP64 addition after every eighth point
// (122,880 points x 1,000 targets, 3D: 72 -> 60 us; the ex2 alone take 34).
template <int DIM, bool FP32, int QG = 1>
__device__ __forceinline__ void dense_grad_block(const double *__restrict__ x, const double *__restrict__ w,
                                                 const double *__restrict__ Lq, const double *__restrict__ tpack,
                                                 const double *__restrict__ psi, const EvalArgs &a, int64_t qslice,
                                                 int64_t tblk, int64_t ks, double *__restrict__ gpart)
{
    constexpr int TT = DENSE_B_TT;
    constexpr int TB = DENSE_B_THREADS * TT;
    constexpr int NTH = DENSE_B_THREADS * QG;          // threads of the CTA
    constexpr int CH = DB_CHUNK * (QG > 1 ? 2 : 1);    // points staged at a time
    __shared__ double tab[16];
    __shared__ __align__(16) double stgd[FP32 ? 1 : CH * (DIM + 2)];
    // FP32: x (DIM), beta, w, each a row of the chunk's points, group after group
    __shared__ __align__(16) float stgf[FP32 ? CH * (DIM + 2) : 1];
    __shared__ double gsum[QG > 1 ? (QG - 1) * TT * DENSE_B_THREADS : 1];
    if (threadIdx.x < 16) tab[threadIdx.x] = c_exp2_tab[threadIdx.x];
    const int tid = threadIdx.x;
    const int lt = tid % DENSE_B_THREADS;  // target lane
    const int grp = tid / DENSE_B_THREADS; // point group
    const int64_t j0 = tblk * TB;
    const int64_t qa = ks * qslice;
    const int64_t qb = min(a.nq, qa + qslice);

    GradTargets<TT> T;
    grad_targets<DIM, FP32, NTH>(tpack, psi, a, j0, lt, T);
    const double *ob = T.ob;
    const double aref = T.aref;
    const auto &A = T.A;
    const auto &B = T.B;
    double acc64[TT];
#pragma unroll
    for (int k = 0; k < TT; ++k) acc64[k] = 0.0;
    // FP32: two points per packed instruction
    f32x2 yn[TT][DIM], al2[TT];
    const f32x2 nc32 = pack2(-(float)a.c32, -(float)a.c32);
    if (FP32) {
#pragma unroll
        for (int k = 0; k < TT; ++k) {
#pragma unroll
            for (int d = 0; d < DIM; ++d) yn[k][d] = pack2(-T.yt[k][d], -T.yt[k][d]);
            al2[k] = pack2(T.alpha[k], T.alpha[k]);
        }
    }
    for (int64_t c0 = qa; c0 < qb; c0 += CH) {
        const int cn = (int)min((int64_t)CH, qb - c0);
        __syncthreads();
        if (FP32) {
            // each group's points in its own order, padded to whole octets with points of no weight
            const int cp = (cn + 8 * QG - 1) / (8 * QG) * (8 * QG);
            for (int i = tid; i < cp; i += NTH) {
                const int64_t q = c0 + i;
                float *v = stgf + (i % QG) * (CH / QG) + i / QG;
#pragma unroll
                for (int d = 0; d < DIM; ++d) v[d * CH] = i < cn ? (float)(x[q * DIM + d] - ob[d]) : 0.f;
                v[DIM * CH] = i < cn ? (float)(-LOG2E * Lq[q] + aref) : -INFINITY;
                v[(DIM + 1) * CH] = i < cn ? (float)w[q] : 0.f;
            }
        } else {
            for (int i = tid; i < cn; i += NTH) {
                const int64_t q = c0 + i;
                double xsq = 0.0;
#pragma unroll
                for (int d = 0; d < DIM; ++d) {
                    const double xt = x[q * DIM + d] - a.o[d];
                    xsq += xt * xt;
                    stgd[i * (DIM + 2) + d] = xt;
                }
                stgd[i * (DIM + 2) + DIM] = -a.halfs * xsq - KAPPA * Lq[q];
                stgd[i * (DIM + 2) + DIM + 1] = w[q];
            }
        }
        __syncthreads();
        if (FP32) {
            const float *v = stgf + grp * (CH / QG);
            const int m = (cn - grp + QG - 1) / QG;  // this group's points
            for (int n = 0; n < m; n += 8) {
                float acc[TT];
#pragma unroll
                for (int k = 0; k < TT; ++k) acc[k] = 0.f;
#pragma unroll
                for (int h = 0; h < 8; h += 4) {
                    ulonglong2 r[DIM + 2];
#pragma unroll
                    for (int f = 0; f < DIM + 2; ++f)
                        r[f] = *reinterpret_cast<const ulonglong2 *>(v + f * CH + n + h);
#pragma unroll
                    for (int k = 0; k < TT; ++k) {
#pragma unroll
                        for (int e = 0; e < 2; ++e) {
                            f32x2 d2 = 0;
#pragma unroll
                            for (int d = 0; d < DIM; ++d) {
                                const f32x2 dd = add2(e ? r[d].y : r[d].x, yn[k][d]);
                                d2 = d == 0 ? mul2(dd, dd) : fma2(dd, dd, d2);
                            }
                            const f32x2 ex = fma2(nc32, d2, add2(al2[k], e ? r[DIM].y : r[DIM].x));
                            float e0, e1, w0, w1;
                            unpack2(ex, e0, e1);
                            unpack2(e ? r[DIM + 1].y : r[DIM + 1].x, w0, w1);
                            acc[k] = fmaf(w0, ex2_approx(e0), acc[k]);
                            acc[k] = fmaf(w1, ex2_approx(e1), acc[k]);
                        }
                    }
                }
#pragma unroll
                for (int k = 0; k < TT; ++k) acc64[k] += (double)acc[k];
            }
        } else {
            for (int t = grp; t < cn; t += QG) {
                const double *v = stgd + t * (DIM + 2);
                const double D = v[DIM], wq = v[DIM + 1];
#pragma unroll
                for (int k = 0; k < TT; ++k) {
                    double u = fma(B[k][0], v[0], A[k] + D);
#pragma unroll
                    for (int d = 1; d < DIM; ++d) u = fma(B[k][d], v[d], u);
                    acc64[k] = fma(wq, exp2_16(u, tab), acc64[k]);
                }
            }
        }
    }
    if (QG > 1) {
        // the groups' sums, added in group order by group 0
        if (grp > 0) {
#pragma unroll
            for (int k = 0; k < TT; ++k) gsum[((grp - 1) * TT + k) * DENSE_B_THREADS + lt] = acc64[k];
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < TT; ++k)
            for (int g = 1; g < QG; ++g) acc64[k] += gsum[((g - 1) * TT + k) * DENSE_B_THREADS + lt];
    }
#pragma unroll
    for (int k = 0; k < TT; ++k) {
        const int64_t j = j0 + lt + k * DENSE_B_THREADS;
        if (grp == 0 && j < a.nt) {
            double g = acc64[k];
            if (!FP32) g *= tpack[j * TPACK + 1 + DIM];  // nu_j (FP32 path folds it into alpha)
            gpart[ks * a.nt + j] = g;
        }
    }
}

}  // namespace sdot
