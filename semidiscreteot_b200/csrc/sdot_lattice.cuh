// sdot_lattice.cuh -- untruncated sweeps over sources whose points form a
// tensor lattice (Gauss points of an axis-aligned structured mesh: every
// combination of per-dimension coordinates is a point).
//
// With the exponent b_qj = A_j + B_j.(x_q - o) (units of 2^(1/16), see
// sdot_internal.h) a (point, target) term is a product of one factor per
// dimension, 2^(B_jd (x_qd - c_d) / 16), about the centre c of a tile of
// lattice points.  The sums of both sweeps are then matrix products:
//   value     S[i] = sum_j (nu_j 2^((B0_j - M) / 16) F0_j[i0]) F1_j[i1] (F2_j[i2]),
//   gradient  g_j  = nu_j sum_i0 E_j F0_j[i0] sum_i1 F1_j[i1] (sum_i2) W[i] F2_j[i2],
// one FP64 multiply-add per (point, target) pair plus the factors, which
// cost one exponential per (tile row, target) instead of one per (cell,
// target) and four multiply-adds per pair (the cell sweeps of sdot_eval.cu).
//
// The products run on the FP64 matrix instruction (m16n8k8).  Its rate is
// the FP64 pipe's (37.1 against 35.2 TFLOP/s measured with either alone), but
// an operand fragment feeds eight times the multiply-adds: register tiles of
// 4 x 4 multiply-adds per thread kept the shared-memory pipe busy 76% and the
// FP64 pipe 52% of the time (0.367 ms for 147,456 points x 16,384 targets).
//
// B0_j = A_j + B_j.(c - o); M = max_j B0_j is the tile's shift, the same for
// every slice of the targets, so the slices' sums add without rescaling.
// The caller admits a tile size only when the factors of a tile span at most
// 2^(+-LAT_BITS): every point's sum is then at least nu 2^-LAT_BITS relative
// to M, and nothing leaves the FP64 range.  exp2_16_full clamps at 2^-1000.
// Only dimension 0's factors, which carry B0 - M, can be that small.  With an
// exponential for each of them a clamped one is multiplied by the other
// dimensions' only: with spans b_d, b in all, it adds at most 2^(b - b_0 - 1000)
// to a sum of at least 2^-b, 300 bits below it.  A run multiplies its clamped
// first factor by up to seven steps too, 2^g: runs are taken where
// g + 2 b - b_0 still leaves LAT_CLAMP_LEFT bits (on a beam whose one run covers a
// tile, g = 2 b_0 = 2 b, up to b = 233; on squares of 64^2-point tiles always),
// and every factor has its own exponential otherwise.
#pragma once

#include "sdot_device.cuh"
#include "sdot_lattice_host.h"

namespace sdot {

constexpr int LAT_THREADS = 256;
constexpr int LAT_TILE = 4096;    // points of a tile: 64 x 64 or 16 x 16 x 16
constexpr int LAT_CK = 32;        // targets of a chunk of the value sweep
constexpr int LAT_GT = 64;        // targets of a CTA of the gradient sweep
constexpr int LAT_MAXRUNS = 32;   // 2D: 2 x period x ceil(64 / (8 period)) <= 24 for periods up to 4
constexpr int LAT_LIST = 1024;    // candidates of a pass over the points' maxima (32 target blocks)
constexpr int LAT_PAD_F = 4;      // row padding of the operands in shared memory: the four rows a fragment
                                  // load touches fall on different banks (row length = 4 mod 16 doubles)

struct LatArgs {
    const double *X;   // lattice coordinates, dimension after dimension
    const int *q;      // point of lattice index i0 + n0 (i1 + n1 i2)
    int n[3], nt[3], xo[3];  // points, tiles and first coordinate per dimension
    int cap;           // points of a tile per dimension
    int ntiles;
    // Factor runs (runs > 0: every dimension has a period): point i + k period
    // is k steps from point i, so a run of LAT_RUN points a period apart takes
    // one exponential and powers of the target's step factor.
    int period[3], runs;     // runs of a target: sum over the dimensions of period x ceil(T / (LAT_RUN period))
    unsigned runs_inv;       // for fast_div by runs
    double step16[3];        // step / 16
};

// Blocks of at most 32 targets (k-d tree leaves): the targets mem[off[b]..]
// (consecutive ones, off[b].., without mem), bounding sphere (4 doubles) and
// largest s psi_j.
struct LatBlocks {
    const int64_t *off;
    const int *mem;
    const double *sph;
    const double *top;
    int n;
};

// D += A B on one warp, A 16 x 8, B 8 x 8, FP64.  Lane 4 g + t holds A[g + 8 (i & 1)][t + 4 (i >> 1)] in a[i],
// B[t + 4 i][g] in b[i] and D[g + 8 (i >> 1)][2 t + (i & 1)] in d[i].
__device__ __forceinline__ void mma_f64(double *d, const double *a, const double *b)
{
    asm("mma.sync.aligned.m16n8k8.row.col.f64.f64.f64.f64 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
        "{%0, %1, %2, %3};"
        : "+d"(d[0]), "+d"(d[1]), "+d"(d[2]), "+d"(d[3])
        : "d"(a[0]), "d"(a[1]), "d"(a[2]), "d"(a[3]), "d"(b[0]), "d"(b[1]));
}

template <int DIM>
struct LatDims {
    static constexpr int T = DIM == 2 ? 64 : 16;   // points per dimension of a full tile
    static constexpr int FD = T * DIM;             // factors per target
    static constexpr int FS = FD + LAT_PAD_F;      // row of one target's factors in shared memory
};

// Run counts of a launch from the lattice's periods and its tiling (host).
inline void lat_runs(const int *period, const double *step, int dim, const LatTiling &t, LatArgs &L)
{
    const int T = dim == 2 ? 64 : 16;
    L.runs = 0;
    const double grow = std::min(2.0 * t.span0, t.slope0 * (LAT_RUN - 1) * step[0]);
    if (!(grow + 2.0 * t.span - t.span0 <= 1000.0 - LAT_CLAMP_LEFT)) return;
    for (int d = 0; d < dim; ++d) {
        const int p = period[d];
        if (p <= 0) {
            L.runs = 0;
            return;
        }
        L.period[d] = p;
        L.step16[d] = step[d] / 16.0;
        L.runs += p * ((T + LAT_RUN * p - 1) / (LAT_RUN * p));
    }
    L.runs_inv = (unsigned)(((1ull << 32) + L.runs - 1) / L.runs);
}

template <int DIM>
struct LatBox {
    int s[DIM], e[DIM];      // first lattice index, points
    double c[DIM], h[DIM];   // centre relative to the origin o, half extent
};

template <int DIM>
__device__ __forceinline__ void lat_box(const LatArgs &L, const EvalArgs &a, int t, LatBox<DIM> &B)
{
#pragma unroll
    for (int d = 0; d < DIM; ++d) {
        const int td = t % L.nt[d];
        t /= L.nt[d];
        B.s[d] = td * L.cap;
        B.e[d] = min(L.cap, L.n[d] - B.s[d]);
        const double lo = L.X[L.xo[d] + B.s[d]], hi = L.X[L.xo[d] + B.s[d] + B.e[d] - 1];
        const double c = 0.5 * (lo + hi);
        B.c[d] = c - a.o[d];
        B.h[d] = hi - c;
    }
}

// Offset of the tile's point ii of dimension d from the tile's centre.
template <int DIM>
__device__ __forceinline__ double lat_delta(const LatArgs &L, const EvalArgs &a, const LatBox<DIM> &B, int d, int ii)
{
    return (L.X[L.xo[d] + B.s[d] + ii] - a.o[d]) - B.c[d];
}

// Run table: dimension and first index of each run.
template <int DIM>
__device__ __forceinline__ void lat_run_table(const LatArgs &L, int2 *run)
{
    const int rr = threadIdx.x;
    if (rr >= L.runs) return;
    int f = rr;
#pragma unroll
    for (int d = 0; d < DIM; ++d) {
        const int p = L.period[d], n = p * ((LatDims<DIM>::T + LAT_RUN * p - 1) / (LAT_RUN * p));
        if (f >= 0 && f < n) run[rr] = make_int2(d, f % p + LAT_RUN * p * (f / p));
        f -= n;
    }
}

// The LAT_RUN factors of a run from the first one and the step factor's
// powers 1, 2 and 4 (products of at most three factors).
__device__ __forceinline__ void lat_run(double f, double r, double r2, double r4, double *o)
{
    o[0] = f;
    o[1] = f * r;
    o[2] = f * r2;
    o[3] = o[1] * r2;
#pragma unroll
    for (int k = 0; k < 4; ++k) o[4 + k] = o[k] * r4;
}

// Shift of tile t over all targets by one CTA: shift[2 t] = M = max_j B0_j,
// shift[2 t + 1] the largest magnitude of a term of an exponent, for the
// rounding of the bounds in lat_merge_block.
template <int DIM, int NTH, class Psi>
__device__ __forceinline__ void lat_shift_block(const LatArgs &L, const EvalArgs &a, int t,
                                                const double *__restrict__ y, Psi &&psi, double *__restrict__ shift)
{
    __shared__ double red[2][NTH / 32];
    LatBox<DIM> B;
    lat_box<DIM>(L, a, t, B);
    double M = -CUDART_INF, mag = 0.0;
#pragma unroll 4
    for (int64_t j = threadIdx.x; j < a.nt; j += NTH) {
        const double sp = a.s * psi(j);
        double ysq = 0.0, b0 = sp, am = fabs(sp);
#pragma unroll
        for (int d = 0; d < DIM; ++d) {
            const double yt = y[j * DIM + d] - a.o[d];
            ysq = fma(yt, yt, ysq);
            b0 = fma(a.s * yt, B.c[d], b0);
            am = fma(a.s * fabs(yt), fabs(B.c[d]) + B.h[d], am);
        }
        M = fmax(M, fma(-a.halfs, ysq, b0));
        mag = fmax(mag, fma(a.halfs, ysq, am));
    }
    M = warp_max(M);
    mag = warp_max(mag);
    if ((threadIdx.x & 31) == 0) {
        red[0][threadIdx.x >> 5] = M;
        red[1][threadIdx.x >> 5] = mag;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int i = 1; i < NTH / 32; ++i) {
            M = fmax(M, red[0][i]);
            mag = fmax(mag, red[1][i]);
        }
        shift[2 * t] = M;
        shift[2 * t + 1] = mag;
    }
}

// Shared memory of the value sweep.
template <int DIM>
struct LatValueSmem {
    double F[2][LAT_CK][LatDims<DIM>::FS];   // factors of two chunks
    double td[3][LAT_CK][2 + 4 * DIM];       // per target of three chunks: B0 - M, B(DIM), nu, step factors' powers
                                             // 1 (DIM), 2 (DIM) and 4 (DIM)
    double tab[16];
    double delta[LatDims<DIM>::FD];          // offsets of the tile's coordinates from its centre
    int2 run[LAT_MAXRUNS];
};

// Value sweep of one tile against the targets [t0, t1): per point the sum
// relative to the tile's shift M, to out[point of the tile].  Chunks of
// LAT_CK targets, double buffered: the threads write chunk k + 1's factors and
// multiply chunk k, and one warp fetches chunk k + 2's targets, so a chunk
// costs one barrier.  A warp owns 32 x 16 points (2D:
// rows i0, columns i1) or two planes i1 (3D: rows i0, columns i2; the A
// operand F0[i0] F1[i1] is formed in registers), as 2 x 2 fragments;
// fragments past the tile's extent are skipped.
template <int DIM>
__device__ __forceinline__ void lat_value_block(unsigned char *smem, const LatArgs &L, const EvalArgs &a,
                                                const double *__restrict__ tpack, const double *__restrict__ shift,
                                                const double *__restrict__ step, int tile, int64_t t0, int64_t t1,
                                                double *__restrict__ out)
{
    constexpr int FD = LatDims<DIM>::FD, FS = LatDims<DIM>::FS, T = LatDims<DIM>::T;
    auto &sm = *reinterpret_cast<LatValueSmem<DIM> *>(smem);
    LatBox<DIM> B;
    lat_box<DIM>(L, a, tile, B);
    const double M = shift[2 * tile];
    const int tid = threadIdx.x, lane = tid & 31, wp = tid >> 5;
    const int g = lane >> 2, t = lane & 3;
    // first row and column of the warp's fragments
    const int row = DIM == 2 ? 32 * (wp & 1) : 0;            // i0
    const int col = DIM == 2 ? 16 * (wp >> 1) : 0;           // 2D: i1, 3D: i2
    const int pl = DIM == 2 ? 0 : 2 * wp;                    // 3D: i1
    bool on[2], onc[2];
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        on[k] = DIM == 2 ? row + 16 * k < B.e[0] : pl + k < B.e[1];
        onc[k] = col + 8 * k < B.e[DIM - 1];
    }
    // factor generation: thread <-> one lattice index of one dimension, every GSth target
    constexpr int GI = DIM == 2 ? 128 : 64;      // threads over the indices
    constexpr int GS = LAT_THREADS / GI;
    const int gi = tid % GI, gj = tid / GI;
    const int gd = gi / T, gii = gi % T;
    const bool gen = gi < FD;
    double gdelta = 0.0;
    if (gen) {
#pragma unroll
        for (int d = 0; d < DIM; ++d)
            if (gd == d && gii < B.e[d]) gdelta = lat_delta<DIM>(L, a, B, d, gii);
    }
    static_assert(LAT_CK == 32, "one warp loads a chunk");
    const int nch = (int)((t1 - t0 + LAT_CK - 1) / LAT_CK);
    // targets of a chunk, by one warp: lane <-> target, fetched to registers and stored after the products
    double pf[2 * DIM + 2];
    auto fetch_chunk = [&](int k) {
        const int64_t j = t0 + (int64_t)k * LAT_CK + lane;
        if (j < t1) {
#pragma unroll
            for (int d = 0; d < DIM + 2; ++d) pf[d] = tpack[j * TPACK + d];
            if (L.runs > 0) {
#pragma unroll
                for (int d = 0; d < DIM; ++d) pf[DIM + 2 + d] = step[j * DIM + d];
            }
        }
    };
    auto store_chunk = [&](int k) {
        if (t0 + (int64_t)k * LAT_CK + lane < t1) {
            double *o = sm.td[k % 3][lane];
            double bb = pf[0];
#pragma unroll
            for (int d = 0; d < DIM; ++d) {
                o[1 + d] = pf[1 + d];
                bb = fma(pf[1 + d], B.c[d], bb);
            }
            o[0] = bb - M;
            o[1 + DIM] = pf[1 + DIM];
            if (L.runs > 0) {
#pragma unroll
                for (int d = 0; d < DIM; ++d) {
                    const double r = pf[DIM + 2 + d], r2 = r * r;
                    o[2 + DIM + d] = r;
                    o[2 + 2 * DIM + d] = r2;
                    o[2 + 3 * DIM + d] = r2 * r2;
                }
            }
        }
    };
    auto gen_chunk = [&](int k) {  // factors, and zeros up to a multiple of the fragments' depth
        const int cn = (int)min((int64_t)LAT_CK, t1 - t0 - (int64_t)k * LAT_CK);
        const int cz = (cn + 7) & ~7;
        if (L.runs > 0) {
            for (int u = tid; u < cz * L.runs; u += LAT_THREADS) {
                const int j = (int)fast_div((unsigned)u, L.runs_inv);
                const int2 rn = sm.run[u - j * L.runs];
                const int d = rn.x, i0 = rn.y;
                const int p = d == 0 ? L.period[0] : (d == 1 ? L.period[1] : L.period[2]);
                double *F = &sm.F[k & 1][j][d * T + i0];
                double o[LAT_RUN];
#pragma unroll
                for (int v = 0; v < LAT_RUN; ++v) o[v] = 0.0;
                if (j < cn) {
                    const double *tp = sm.td[k % 3][j];
                    const double dlt = sm.delta[d * T + i0];
                    double f = exp2_16_full(d == 0 ? fma(tp[1], dlt, tp[0]) : tp[1 + d] * dlt, sm.tab);
                    if (d == 0) f *= tp[1 + DIM];
                    lat_run(f, tp[2 + DIM + d], tp[2 + 2 * DIM + d], tp[2 + 3 * DIM + d], o);
                }
#pragma unroll
                for (int v = 0; v < LAT_RUN; ++v)
                    if (i0 + v * p < T) F[v * p] = o[v];
            }
        } else if (gen) {
            double *F = &sm.F[k & 1][0][gi];
            int j = gj;
            if (gd == 0) {
#pragma unroll 4
                for (; j < cn; j += GS) {
                    const double *tp = sm.td[k % 3][j];
                    F[j * FS] = tp[1 + DIM] * exp2_16_full(fma(tp[1], gdelta, tp[0]), sm.tab);
                }
            } else {
#pragma unroll 4
                for (; j < cn; j += GS) F[j * FS] = exp2_16_full(sm.td[k % 3][j][1 + gd] * gdelta, sm.tab);
            }
            for (; j < cz; j += GS) F[j * FS] = 0.0;
        }
    };
    double S[2][2][4];
#pragma unroll
    for (int i = 0; i < 16; ++i) S[i >> 3][(i >> 2) & 1][i & 3] = 0.0;
    if (tid < 16) sm.tab[tid] = c_exp2_tab[tid];
    if (gen && tid < GI) sm.delta[gi] = gdelta;
    lat_run_table<DIM>(L, sm.run);
    if (wp < 2 && wp < nch) {
        fetch_chunk(wp);
        store_chunk(wp);
    }
    __syncthreads();
    gen_chunk(0);
    const bool mine = (on[0] || on[1]) && onc[0];
    for (int k = 0; k < nch; ++k) {
        __syncthreads();  // chunk k's factors and chunk k + 1's targets are in place; chunk k - 1 is consumed
        const bool loads = k + 2 < nch && wp == (k & 7);
        if (loads) fetch_chunk(k + 2);
        if (k + 1 < nch) gen_chunk(k + 1);
        const int cn = (int)min((int64_t)LAT_CK, t1 - t0 - (int64_t)k * LAT_CK);
        const double *F = &sm.F[k & 1][t][g];
#pragma unroll 2
        for (int j = 0; mine && j < cn; j += 8, F += 8 * FS) {
            double b[2][2];
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                b[c][0] = F[(DIM - 1) * T + col + 8 * c];
                b[c][1] = F[(DIM - 1) * T + col + 8 * c + 4 * FS];
            }
            double f0[4];
            if constexpr (DIM == 3) {
#pragma unroll
                for (int i = 0; i < 4; ++i) f0[i] = F[8 * (i & 1) + 4 * FS * (i >> 1)];
            }
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                if (!on[r]) continue;
                double av[4];
                if constexpr (DIM == 2) {
#pragma unroll
                    for (int i = 0; i < 4; ++i) av[i] = F[row + 16 * r + 8 * (i & 1) + 4 * FS * (i >> 1)];
                } else {
                    const double *F1 = F - g + T + pl + r;
                    const double p0 = F1[0], p1 = F1[4 * FS];
#pragma unroll
                    for (int i = 0; i < 4; ++i) av[i] = f0[i] * (i >> 1 ? p1 : p0);
                }
#pragma unroll
                for (int c = 0; c < 2; ++c)
                    if (onc[c]) mma_f64(S[r][c], av, b[c]);
            }
        }
        if (loads) store_chunk(k + 2);
    }
#pragma unroll
    for (int r = 0; r < 2; ++r)
#pragma unroll
        for (int c = 0; c < 2; ++c)
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int ix[3] = {row + (DIM == 2 ? 16 * r : 0) + g + 8 * (i >> 1),
                                   DIM == 2 ? col + 8 * c + 2 * t + (i & 1) : pl + r, col + 8 * c + 2 * t + (i & 1)};
                bool in = true;
#pragma unroll
                for (int d = 0; d < DIM; ++d) in = in && ix[d] < B.e[d];
                if (in) out[ix[0] + T * ix[1] + (DIM == 3 ? T * T * ix[2] : 0)] = S[r][c][i];
            }
}

// Maxima, merge and epilogue of one box of a tile (16 x 16 or 8 x 8 x 4
// points, LAT_TILE / LAT_THREADS boxes per tile, thread <-> point).
//  * The exact maximum of each point's exponents.  About a centre c of some
//    points, b_qj = b_cj + s (y_j - c).(x_q - c) + (a part that is the same
//    for all targets), so only targets with b_cj + s sum_d |y_jd - c_d| h_d
//    >= lb can be a maximum, lb = the largest b_cj - s sum_d |y_jd - c_d| h_d
//    of any target.  The bound is applied to the box, then by each warp to
//    its own points (8 x 4 or 4 x 4 x 2).  Above LAT_LIST targets the box's
//    candidates come from the target blocks: a block's sphere bounds its
//    targets (with D the least distance of a target to c, at least the box's
//    radius R: psi's largest value and -s D^2 / 2 + s D R); the block of the
//    largest bound gives lb, and only blocks that reach it are opened.
//    Kept out of the value sweep, where a tile's maxima cost more than its
//    sums; a scan of all targets per box took 0.22 ms at 147,456 points x
//    16,384 targets.
//  * The slices' sums added in order of the slices, L_q and the box's
//    (value, C, skipped, 0) partials.  With wt, the gradient sweep's weights
//    w_q / S_q (relative to M; 0 for skipped points and past the tile's
//    extent) replace slice 0's sums.
template <int DIM>
__device__ __forceinline__ void lat_merge_block(const LatArgs &L, const EvalArgs &a, const LatBlocks &K, int tile,
                                                int sub, int nslice, bool wt, double *__restrict__ ms,
                                                const double *__restrict__ shift, const double *__restrict__ tpack,
                                                const double *__restrict__ rho, const double *__restrict__ jxw,
                                                double *__restrict__ Lq, double *__restrict__ out4)
{
    constexpr int T = LatDims<DIM>::T;
    constexpr int NW = LAT_THREADS / 32;
    constexpr int BB = LAT_LIST / 32;   // target blocks opened per pass
    __shared__ double tab[16];
    __shared__ double list[DIM + 1][LAT_LIST];   // b about the tile's centre and B of the box's candidates
    __shared__ int blist[LAT_THREADS];
    __shared__ double redv[NW];
    __shared__ int redi[NW];
    __shared__ int nlist, nblist;
    __shared__ double slb;
    const int tid = threadIdx.x, lane = tid & 31, wp = tid >> 5;
    if (tid < 16) tab[tid] = c_exp2_tab[tid];
    if (tid == 0) nlist = nblist = 0;
    LatBox<DIM> B;
    lat_box<DIM>(L, a, tile, B);
    // first indices of the box and of the warp's points, index of the thread's point in the tile
    int i0[3], w0[3], i[3], ext[3], wext[3];
    if (DIM == 2) {
        i0[0] = 16 * (sub & 3);
        i0[1] = 16 * (sub >> 2);
        i0[2] = 0;
        w0[0] = i0[0] + 8 * (wp & 1);
        w0[1] = i0[1] + 4 * (wp >> 1);
        w0[2] = 0;
        i[0] = w0[0] + (lane & 7);
        i[1] = w0[1] + (lane >> 3);
        i[2] = 0;
        ext[0] = ext[1] = 16;
        wext[0] = 8;
        wext[1] = 4;
        ext[2] = wext[2] = 1;
    } else {
        i0[0] = 8 * (sub & 1);
        i0[1] = 8 * ((sub >> 1) & 1);
        i0[2] = 4 * (sub >> 2);
        w0[0] = i0[0] + 4 * (wp & 1);
        w0[1] = i0[1] + 4 * ((wp >> 1) & 1);
        w0[2] = i0[2] + 2 * (wp >> 2);
        i[0] = w0[0] + (lane & 3);
        i[1] = w0[1] + ((lane >> 2) & 3);
        i[2] = w0[2] + (lane >> 4);
        ext[0] = ext[1] = 8;
        ext[2] = wext[0] = wext[1] = 4;
        wext[2] = 2;
    }
    bool ok = true, any = true, anyw = true;
#pragma unroll
    for (int d = 0; d < DIM; ++d) {
        ok = ok && i[d] < B.e[d];
        any = any && i0[d] < B.e[d];
        anyw = anyw && w0[d] < B.e[d];
    }
    double *p = ms + (int64_t)tile * LAT_TILE + i[0] + T * i[1] + T * T * i[2];
    double tv = 0.0, tc = 0.0, ts = 0.0, W = 0.0;
    __syncthreads();
    if (any) {  // (the box is in the tile: the same for all threads)
        // centre and half extents of the box and of the warp's points: relative to o / to the tile's centre
        double bc[DIM], bh[DIM], wc[DIM], wh[DIM], x[DIM];
#pragma unroll
        for (int d = 0; d < DIM; ++d) {
            auto span = [&](int f, int n, double &c, double &h) {
                const double lo = lat_delta<DIM>(L, a, B, d, min(f, B.e[d] - 1));
                const double hi = lat_delta<DIM>(L, a, B, d, min(f + n, B.e[d]) - 1);
                c = 0.5 * (lo + hi);
                h = hi - c;
            };
            span(i0[d], ext[d], bc[d], bh[d]);
            span(w0[d], wext[d], wc[d], wh[d]);
            bc[d] += B.c[d];
            x[d] = lat_delta<DIM>(L, a, B, d, min(i[d], B.e[d] - 1));
        }
        const double slack = 1e-13 * shift[2 * tile + 1];
        // lower (and, less slack, upper) bound of target j's exponents over the box
        auto target_lb = [&](const double *tp, double &ub) {
            double b = tp[0], ag = 0.0;
#pragma unroll
            for (int d = 0; d < DIM; ++d) {
                b = fma(tp[1 + d], bc[d], b);
                ag = fma(fabs(fma(-a.s, bc[d], tp[1 + d])), bh[d], ag);
            }
            ub = b + ag;
            return b - ag;
        };
        auto push = [&](const double *tp) {
            const int at = atomicAdd(&nlist, 1);
            double bt = tp[0];
#pragma unroll
            for (int d = 0; d < DIM; ++d) {
                bt = fma(tp[1 + d], B.c[d], bt);
                list[1 + d][at] = tp[1 + d];
            }
            list[0][at] = bt;
        };
        // the warp's maxima over the listed candidates
        double mx = -CUDART_INF, lbw = -CUDART_INF;
        auto scan_list = [&]() {
            const int nl = nlist;
            if (!anyw) return;
            auto bound = [&](int k, double &ub) {
                double b = list[0][k], ag = 0.0;
#pragma unroll
                for (int d = 0; d < DIM; ++d) {
                    const double G = list[1 + d][k];
                    b = fma(G, wc[d], b);
                    ag = fma(fabs(fma(-a.s, B.c[d] + wc[d], G)), wh[d], ag);
                }
                ub = b + ag;
                return b - ag;
            };
            double lb = -CUDART_INF, ub;
            for (int k = lane; k < nl; k += 32) lb = fmax(lb, bound(k, ub));
            lbw = fmax(lbw, warp_max(lb));
            for (int k0 = 0; k0 < nl; k0 += 32) {
                bool pass = false;
                if (k0 + lane < nl) {
                    bound(k0 + lane, ub);
                    pass = ub + slack >= lbw - slack;
                }
                unsigned m = __ballot_sync(0xffffffffu, pass);
                while (m) {
                    const int k = k0 + __ffs(m) - 1;
                    m &= m - 1;
                    double b = list[0][k];
#pragma unroll
                    for (int d = 0; d < DIM; ++d) b = fma(list[1 + d][k], x[d], b);
                    mx = fmax(mx, b);
                }
            }
        };
        // the slices' sums, in flight while the maxima are found
        double S = 0.0;
        if (ok) {
            const int64_t st = (int64_t)L.ntiles * LAT_TILE;
            int s = 0;
            for (; s + 16 <= nslice; s += 16) {
                double v[16];
#pragma unroll
                for (int k = 0; k < 16; ++k) v[k] = p[(s + k) * st];
#pragma unroll
                for (int k = 0; k < 16; ++k) S += v[k];
            }
#pragma unroll 4
            for (; s < nslice; ++s) S += p[s * st];
        }
        if (a.nt <= LAT_LIST) {
            constexpr int PER = LAT_LIST / LAT_THREADS;
            double ub[PER], lb = -CUDART_INF;
#pragma unroll
            for (int k = 0; k < PER; ++k) {
                const int64_t j = tid + k * LAT_THREADS;
                ub[k] = -CUDART_INF;
                if (j < a.nt) lb = fmax(lb, target_lb(tpack + j * TPACK, ub[k]));
            }
            lb = warp_max(lb);
            if (lane == 0) redv[wp] = lb;
            __syncthreads();
#pragma unroll
            for (int k = 0; k < NW; ++k) lb = fmax(lb, redv[k]);
            lb -= slack;
#pragma unroll
            for (int k = 0; k < PER; ++k)
                if (ub[k] > -CUDART_INF && ub[k] + slack >= lb) push(tpack + (tid + k * LAT_THREADS) * TPACK);
            __syncthreads();
            scan_list();
        } else {
            double rbox = 0.0, csq = 0.0;
#pragma unroll
            for (int d = 0; d < DIM; ++d) {
                rbox = fma(bh[d], bh[d], rbox);
                csq = fma(bc[d], bc[d], csq);
            }
            rbox = sqrt(rbox);
            auto block_ub = [&](int b) {
                double d2 = 0.0;
#pragma unroll
                for (int d = 0; d < DIM; ++d) {
                    const double t = (K.sph[4 * b + d] - a.o[d]) - bc[d];
                    d2 = fma(t, t, d2);
                }
                const double D = fmax(rbox, sqrt(d2) - K.sph[4 * b + 3]);
                return K.top[b] + a.halfs * (D * (2.0 * rbox - D) + csq) + slack;
            };
            // the block of the largest bound
            double best = -CUDART_INF;
            int bi = 0;
            for (int b = tid; b < K.n; b += LAT_THREADS) {
                const double u = block_ub(b);
                if (u > best) {
                    best = u;
                    bi = b;
                }
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                const double v = __shfl_xor_sync(0xffffffffu, best, o);
                const int w = __shfl_xor_sync(0xffffffffu, bi, o);
                if (v > best) {
                    best = v;
                    bi = w;
                }
            }
            if (lane == 0) {
                redv[wp] = best;
                redi[wp] = bi;
            }
            __syncthreads();
            if (wp == 0) {
                best = redv[0];
                bi = redi[0];
#pragma unroll
                for (int k = 1; k < NW; ++k)
                    if (redv[k] > best) {
                        best = redv[k];
                        bi = redi[k];
                    }
                const int64_t j = K.off[bi] + lane;
                double lb = -CUDART_INF, ub;
                if (j < K.off[bi + 1]) lb = target_lb(tpack + (K.mem ? K.mem[j] : j) * TPACK, ub);
                lb = warp_max(lb);
                if (lane == 0) slb = lb - slack;
            }
            __syncthreads();
            const double lb = slb;
            for (int b0 = 0; b0 < K.n; b0 += LAT_THREADS) {
                if (b0 + tid < K.n && block_ub(b0 + tid) >= lb) blist[atomicAdd(&nblist, 1)] = b0 + tid;
                __syncthreads();
                const int nb = nblist;
                for (int k0 = 0; k0 < nb; k0 += BB) {
#pragma unroll
                    for (int u = 0; u < BB / NW; ++u) {
                        const int k = k0 + wp + u * NW;
                        if (k < nb) {
                            const int64_t j = K.off[blist[k]] + lane;
                            if (j < K.off[blist[k] + 1]) {
                                const double *tp = tpack + (K.mem ? K.mem[j] : j) * TPACK;
                                double ub;
                                target_lb(tp, ub);
                                if (ub + slack >= lb) push(tp);
                            }
                        }
                    }
                    __syncthreads();
                    scan_list();
                    __syncthreads();
                    if (tid == 0) nlist = 0;
                    __syncthreads();
                }
                if (tid == 0) nblist = 0;
                __syncthreads();
            }
        }
        if (ok) {
            int64_t li = B.s[DIM - 1] + i[DIM - 1];
#pragma unroll
            for (int d = DIM - 2; d >= 0; --d) li = li * L.n[d] + B.s[d] + i[d];
            const int64_t q = L.q[li];
            double xsq = 0.0;
#pragma unroll
            for (int d = 0; d < DIM; ++d) {
                const double xt = L.X[L.xo[d] + B.s[d] + i[d]] - a.o[d];
                xsq += xt * xt;
            }
            const double Sref = mx == -CUDART_INF ? 0.0 : S * exp2_16_full(shift[2 * tile] - mx, tab);
            const double r = rho[q], jw = jxw[q];
            double Lv;
            int sk;
            value_epilogue(a, mx, Sref, -a.halfs * xsq, r, jw, tv, tc, Lv, sk);
            Lq[q] = Lv;
            ts = sk;
            W = sk ? 0.0 : r * jw / S;
        }
    }
    if (wt) *p = W;
    block_partials_at(tv, tc, ts, 0.0, out4);
}

template <int DIM>
struct LatGradSmem {
    static constexpr int K = LatDims<DIM>::T;                       // points along the last dimension
    static constexpr int WS = LAT_TILE / K + LAT_PAD_F;             // row of weights at one of them
    static constexpr int FS = LAT_GT + LAT_PAD_F;                   // row of one index's factors
    double W[K][WS];
    double F[LatDims<DIM>::FD][FS];
    double tab[16];
    int2 run[LAT_MAXRUNS];
};

// FP64 gradient sweep of targets [j0, j0 + LAT_GT) over the tiles [ta, tb):
// V = W F_last (rows: 2D i0, 3D i0 and i1; columns: targets) on fragments,
// then V times the remaining factors, summed over the rows; the sums of a
// target are added over lanes and warps in a fixed order at the end.  A warp
// owns 32 rows x 16 targets (2D) or the planes i1 of its parity x 16 targets
// (3D, where F2 and F0 stay in registers).
template <int DIM>
__device__ __forceinline__ void lat_grad_block(unsigned char *smem, const LatArgs &L, const EvalArgs &a,
                                               const double *__restrict__ tpack, const double *__restrict__ shift,
                                               const double *__restrict__ step, const double *__restrict__ wt, int64_t j0, int ta, int tb,
                                               double *__restrict__ gout)
{
    using SM = LatGradSmem<DIM>;
    constexpr int T = LatDims<DIM>::T, ROWS = LAT_TILE / T, FS = SM::FS, WS = SM::WS;
    auto &sm = *reinterpret_cast<SM *>(smem);
    const int tid = threadIdx.x, lane = tid & 31, wp = tid >> 5;
    const int g = lane >> 2, t = lane & 3;
    const int part = DIM == 2 ? wp & 1 : wp >> 2;            // half of the rows (2D) or of the planes (3D)
    const int col = 16 * (DIM == 2 ? wp >> 1 : wp & 3);      // first target of the warp
    const int gj = tid % LAT_GT, gi = tid / LAT_GT;
    if (tid < 16) sm.tab[tid] = c_exp2_tab[tid];
    const double *tp = tpack + min(j0 + gj, a.nt - 1) * TPACK;
    const double A = tp[0];
    double Bj[DIM];
#pragma unroll
    for (int d = 0; d < DIM; ++d) Bj[d] = tp[1 + d];
    double r1[DIM];
    if (L.runs > 0) {
        lat_run_table<DIM>(L, sm.run);
#pragma unroll
        for (int d = 0; d < DIM; ++d) r1[d] = step[min(j0 + gj, a.nt - 1) * DIM + d];
    }
    double acc[2][2] = {{0.0, 0.0}, {0.0, 0.0}};             // [column fragment][column 2 t + e]
    for (int tl = ta; tl < tb; ++tl) {
        LatBox<DIM> B;
        lat_box<DIM>(L, a, tl, B);
        __syncthreads();  // the previous tile is consumed (and the table is in place)
        const double *wsrc = wt + (int64_t)tl * LAT_TILE;
        for (int i = 2 * tid; i < LAT_TILE; i += 2 * LAT_THREADS) {
            const unsigned dst = (unsigned)__cvta_generic_to_shared(&sm.W[i / ROWS][i % ROWS]);
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(wsrc + i) : "memory");
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
        double bb = A - shift[2 * tl];
#pragma unroll
        for (int d = 0; d < DIM; ++d) bb = fma(Bj[d], B.c[d], bb);
        if (L.runs > 0) {
            for (int u = gi; u < L.runs; u += LAT_THREADS / LAT_GT) {
                const int2 rn = sm.run[u];
                const int i0 = rn.y;
#pragma unroll
                for (int d = 0; d < DIM; ++d) {
                    if (rn.x != d) continue;
                    const int p = L.period[d];
                    double o[LAT_RUN];
#pragma unroll
                    for (int v = 0; v < LAT_RUN; ++v) o[v] = 0.0;
                    if (i0 < B.e[d]) {
                        const double dlt = lat_delta<DIM>(L, a, B, d, i0);
                        const double f = d == 0 ? exp2_16_full(fma(Bj[d], dlt, bb), sm.tab) : exp2_16_full(Bj[d] * dlt, sm.tab);
                        const double r2 = r1[d] * r1[d];
                        lat_run(f, r1[d], r2, r2 * r2, o);
                    }
#pragma unroll
                    for (int v = 0; v < LAT_RUN; ++v) {
                        const int i = i0 + v * p;
                        if (i < T) sm.F[d * T + i][gj] = i < B.e[d] ? o[v] : 0.0;
                    }
                }
            }
        } else
#pragma unroll
        for (int d = 0; d < DIM; ++d) {
            const double Bd = Bj[d];
#pragma unroll 4
            for (int i = gi; i < T; i += LAT_THREADS / LAT_GT) {
                double f = 0.0;
                if (i < B.e[d]) {
                    const double dlt = lat_delta<DIM>(L, a, B, d, i);
                    f = d == 0 ? exp2_16_full(fma(Bd, dlt, bb), sm.tab) : exp2_16_full(Bd * dlt, sm.tab);
                }
                sm.F[d * T + i][gj] = f;
            }
        }
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();
        if constexpr (DIM == 2) {
            const int row = 32 * part;
            if (row >= B.e[0]) continue;
            double V[2][2][4];
#pragma unroll
            for (int i = 0; i < 16; ++i) V[i >> 3][(i >> 2) & 1][i & 3] = 0.0;
            const double *Wp = &sm.W[t][row + g];
            const double *Fp = &sm.F[T + t][col + g];
            const int ke = B.e[1];
#pragma unroll 2
            for (int k = 0; k < ke; k += 8, Wp += 8 * WS, Fp += 8 * FS) {
                double b[2][2];
#pragma unroll
                for (int c = 0; c < 2; ++c) {
                    b[c][0] = Fp[8 * c];
                    b[c][1] = Fp[8 * c + 4 * FS];
                }
#pragma unroll
                for (int r = 0; r < 2; ++r) {
                    double av[4];
#pragma unroll
                    for (int i = 0; i < 4; ++i) av[i] = Wp[16 * r + 8 * (i & 1) + 4 * WS * (i >> 1)];
#pragma unroll
                    for (int c = 0; c < 2; ++c) mma_f64(V[r][c], av, b[c]);
                }
            }
#pragma unroll
            for (int r = 0; r < 2; ++r)
#pragma unroll
                for (int h = 0; h < 2; ++h)
#pragma unroll
                    for (int c = 0; c < 2; ++c) {
                        const double2 f = *reinterpret_cast<const double2 *>(
                            &sm.F[row + 16 * r + 8 * h + g][col + 8 * c + 2 * t]);
                        acc[c][0] = fma(f.x, V[r][c][2 * h], acc[c][0]);
                        acc[c][1] = fma(f.y, V[r][c][2 * h + 1], acc[c][1]);
                    }
        } else {
            double b[2][2][2], f0[2][2][2];   // [depth step | row half][column fragment][]
#pragma unroll
            for (int h = 0; h < 2; ++h)
#pragma unroll
                for (int c = 0; c < 2; ++c) {
                    b[h][c][0] = sm.F[2 * T + 8 * h + t][col + 8 * c + g];
                    b[h][c][1] = sm.F[2 * T + 8 * h + t + 4][col + 8 * c + g];
                    const double2 f = *reinterpret_cast<const double2 *>(&sm.F[8 * h + g][col + 8 * c + 2 * t]);
                    f0[h][c][0] = f.x;
                    f0[h][c][1] = f.y;
                }
            for (int pl = part; pl < B.e[1]; pl += 2) {
                double V[2][4];
#pragma unroll
                for (int i = 0; i < 8; ++i) V[i >> 2][i & 3] = 0.0;
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    if (8 * h >= B.e[2]) continue;
                    double av[4];
#pragma unroll
                    for (int i = 0; i < 4; ++i) av[i] = sm.W[8 * h + t + 4 * (i >> 1)][16 * pl + g + 8 * (i & 1)];
#pragma unroll
                    for (int c = 0; c < 2; ++c) mma_f64(V[c], av, b[h][c]);
                }
#pragma unroll
                for (int c = 0; c < 2; ++c) {
                    const double2 f = *reinterpret_cast<const double2 *>(&sm.F[T + pl][col + 8 * c + 2 * t]);
                    acc[c][0] = fma(f.x, fma(f0[1][c][0], V[c][2], f0[0][c][0] * V[c][0]), acc[c][0]);
                    acc[c][1] = fma(f.y, fma(f0[1][c][1], V[c][3], f0[0][c][1] * V[c][1]), acc[c][1]);
                }
            }
        }
    }
#pragma unroll
    for (int o = 4; o < 32; o <<= 1)
#pragma unroll
        for (int c = 0; c < 2; ++c)
#pragma unroll
            for (int e = 0; e < 2; ++e) acc[c][e] += __shfl_xor_sync(0xffffffffu, acc[c][e], o);
    __syncthreads();
    double *red = &sm.W[0][0];  // [2][LAT_GT]
    if (g == 0) {
#pragma unroll
        for (int c = 0; c < 2; ++c)
#pragma unroll
            for (int e = 0; e < 2; ++e) red[part * LAT_GT + col + 8 * c + 2 * t + e] = acc[c][e];
    }
    __syncthreads();
    if (tid < LAT_GT && j0 + tid < a.nt)
        gout[j0 + tid] = (red[tid] + red[LAT_GT + tid]) * tpack[(j0 + tid) * TPACK + 1 + DIM];
    __syncthreads();
}

}  // namespace sdot
