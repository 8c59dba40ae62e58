// sdot_trunc.cu -- truncated evaluation (tau > 0): exact cell-centre candidate
// sets, one fused source-block kernel for both exponential sweeps, and an
// atomic-free reduction of the per-block gradient partials.
//
// Replaces find_nearest_target_points + local_assemble + the WorkStream
// copier (src/solvers/SotSolver.cc:553-570, 769-869, 307-311).
//
// Blocks.  Source cells and targets are ordered by k-d trees built at
// set_source / set_target; a source block is a leaf of <= 8 warp units
// (cell, q-group), a target block a leaf of <= 32 targets.  Each block has a
// bounding sphere (FP64) and a conservative FP32 bounding box.
//
// Per evaluation:
//   1. block-pair lists.  (b, t) is a pair iff the box of b's cell centres is
//      within r of the box of t's targets (FP32, conservatively enlarged;
//      super-blocks by their spheres).  With the blocks' spheres in place of
//      their boxes a third more pairs were listed, staged and reduced.  The
//      forward list (per b, t ascending) is filled from masks; the inverse list
//      (per t, b ascending, with the pairs' forward positions) is its
//      transpose, built on a second stream beside step 2, which does not need
//      it.
//   2. k_fused (CTA <-> source block, warp <-> unit):
//      staging: the targets of the block's pairs, culled per target against
//        the block sphere (|y - c_b| <= r + R_b), compacted in order;
//      exact test: warp of cell K keeps j iff d2(y_j, c_K) <= s*, rounded like
//        the reference (this is the candidate set, bit-exact);
//      value sweep: lane <-> candidate, all q of the unit in registers, FP64
//        online log-sum-exp of b_qj = B0_Kj + G_Kj.delta_q + C'_q, where
//        B0_Kj = kappa (psi_j - d2/2)/eps, G_Kj = kappa (y_j - c_K)/eps,
//        delta_q = x_q - c_K, C'_q = -kappa |delta_q|^2 / (2 eps)
//        (kappa = 16/ln 2; the same expansion as |x_q - y_j|^2 about c_K);
//      gradient sweep: sum over a cell's q of
//        w_q nu_j 2^(E0_Kj + G'_Kj.delta_q + D_q) in FP32 ex2 (or FP64 exp2),
//        E0 and G' formed in FP64 per (cell, target) so every FP32 operand is
//        small; thread <-> staged target for the chunk that is still staged,
//        lane <-> target of a forward entry for the others (tensor-product
//        points; staged again otherwise), over the block's cells in FP64.  The
//        block's partial for each target of each pair is written to the pair's
//        forward position.
//   3. k_grad_reduce (CTA <-> target block): sum of the partials over the
//      pairs in ascending source-block order, lane <-> target.  No atomics;
//      the summation order is fixed, results are bitwise reproducible.
#include <float.h>
#include <math.h>

#include <algorithm>
#include <cmath>
#include <vector>

#include "sdot_device.cuh"
#include "sdot_internal.h"

namespace sdot {

constexpr int FT_WARPS = 8;
constexpr int FT_MAXS = 1024;               // staged targets per chunk
// The tensor-factored sweeps stage at most 936 targets per chunk, so that three
// CTAs share an SM (24 warps; 80 registers): fewer chunks per block, which
// are staged twice but for the last, against occupancy.
constexpr int FT_MAXS_TENSOR = 936;
__host__ __device__ constexpr int fused_cap(int tq) { return tq > 0 ? FT_MAXS_TENSOR : FT_MAXS; }
__host__ __device__ constexpr int fused_min_blocks(int tq) { return tq > 0 ? 3 : 2; }
constexpr int FT_TS = 6;                    // doubles per staged target: y(3), nu, log2 nu, s*psi
constexpr int FT_MAXT = 96;                 // target blocks per chunk
constexpr int FT_MAXQ = 80;                 // quadrature points of one source block
constexpr int SUPER = 32;                   // blocks per super-block of the pair-list hierarchy
constexpr int ORDER_BUCKETS = 256;          // weight classes of the source blocks (the sweeps' order)
constexpr int FT_PREF = 192;                // forward entries of a block prefetched into smem

struct FusedArgs {
    const double *x, *rho, *jxw, *w, *cell_ctr;
    const double *tpk;           // y(3), nu, log2 nu, s*psi of all targets, component after component
    int64_t nt;                  // targets
    const int64_t *sblk_cell;    // source block -> first cell (nsblk + 1)
    const double *sblk_sph;      // FP64 centre(3), radius
    const int64_t *tblk_off;     // target block -> first target (ntblk + 1)
    const int64_t *fwd_off;
    const int *fwd_t;
    double *part;                // partials, 32 per pair, at forward positions minus part_base (FP64 sweeps)
    float *part32;               // the same in FP32 (hybrid sweeps: their rows are FP32 already)
    double *Lq;                  // per q (written by the value sweep)
    double *valpart;             // per source block: value, C, skipped, pairs
    int w_nonneg;                // all w_q >= 0: log2 w_q folded into the FP32 exponent
    const int *order;            // source block of each CTA (null: b0, b0 + 1, ...)
    int b0;                      // first source block of the launch
    int64_t part_base;           // forward position of its first pair
    double cullt;                // per-target cull radius addend (r, enlarged)
};

constexpr int FT_NEAR = 64;                 // candidates per warp and chunk that may hold a point's maximum

// Row: the type of a unit's gradient terms and weights, FP32 in the hybrid
// mode and FP64 in the FP64 mode.
template <int CAP, class Row>
struct FTSmem {
    static constexpr int MAXS = CAP;
    double tab[16];
    double stg[FT_TS][CAP];    // staged targets, structure of arrays (conflict-free lane access)
    double qd[FT_MAXQ][4];        // delta_q (FP64) and C'_q
    double qL[FT_MAXQ];           // L_q of the block
    double qS[FT_MAXQ], qm[FT_MAXQ], qU[FT_MAXQ];  // value sweep, per point: sum relative to U, largest exponent, U
    double uL[FT_WARPS];          // smallest L_q of each unit
    double cellc[FT_WARPS][3];    // centre of each unit's cell
    double uah[FT_WARPS][3];      // tensor path: largest offsets of its points
    __align__(16) float qb[FT_MAXQ][4];  // gradient sweep: delta (3) as float, D_q (+ log2 w_q)
    __align__(16) Row qw[FT_MAXQ];       // gradient sweep: w_q
    __align__(16) Row qtw[FT_MAXQ];      // gradient sweep, tensor path: w_q 2^(D_q)
    unsigned short cand[FT_WARPS][CAP];
    unsigned short dst[CAP];      // (chunk target block, slot) of each staged target
    unsigned keep[FT_MAXT];       // staged slots of each target block of the chunk
    unsigned short near_list[FT_WARPS][FT_NEAR];  // candidates that may hold a point's maximum
    int nnear[FT_WARPS];
    int ecnt[32];                 // survivors per examined forward entry (-1: none)
    int epre[32];                 // staged position of the first survivor of each accepted entry
    int eacc, etot;
    int nstg;
    // tensor path, gradient sweep: centres of the units' cells relative to the block's, and the cells' centre
    // coordinates where there are at most two per dimension (brick), the unit at (i0, i1, i2) of them, the offsets
    float uf[FT_WARPS][3];
    double cs[3][2];
    float csf[3][2], ahf[3];
    int cell_at[8];
    int brick;
    int ent_j0[FT_PREF];           // forward entries of the block: the target block's first target
    unsigned char ent_sz[FT_PREF]; // and its size (prefetched once per block)
};
template <bool FP32B> struct PRow { using T = double; };
template <> struct PRow<true> { using T = float; };

// ---------------------------------------------------------------------------
// block-pair lists
// ---------------------------------------------------------------------------

__device__ __forceinline__ bool pair_test(float4 s, float4 t, float cr)
{
    const float dx = __fsub_rn(s.x, t.x), dy = __fsub_rn(s.y, t.y), dz = __fsub_rn(s.z, t.z);
    const float d2 = __fadd_rn(__fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy)), __fmul_rn(dz, dz));
    const float lim = __fadd_rn(__fadd_rn(cr, s.w), t.w);
    return d2 <= __fmul_rn(lim, lim);
}

// Super-block pairs: sp[si * nts + ti] = 1 iff source super-block si and
// target super-block ti may hold a pair (the same conservative test; a
// super-sphere contains its member spheres, so no block pair is lost).
__global__ void __launch_bounds__(256)
k_super_pairs(const float4 *__restrict__ ssph, int nss, const float4 *__restrict__ tsph, int nts, float cr,
              unsigned char *__restrict__ sp)
{
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= (int64_t)nss * nts) return;
    const int si = (int)(i / nts), ti = (int)(i - (int64_t)si * nts);
    sp[i] = pair_test(ssph[si], tsph[ti], cr) ? 1 : 0;
}

// Warp <-> source super-block: its paired target super-blocks in ascending
// order (shit[si * nts + h]) and their count; hist is cleared.
__global__ void __launch_bounds__(256)
k_super_compact(const unsigned char *__restrict__ sp, int nss, int nts, int *__restrict__ shit,
                int *__restrict__ scount, int *__restrict__ hist)
{
    if (blockIdx.x == 0 && threadIdx.x < ORDER_BUCKETS) hist[threadIdx.x] = 0;
    const int si = (int)((blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5);
    const int lane = threadIdx.x & 31;
    if (si >= nss) return;
    int h = 0;
    for (int t0 = 0; t0 < nts; t0 += 32) {
        const int ti = t0 + lane;
        const bool on = ti < nts && sp[(int64_t)si * nts + ti];
        const unsigned bal = __ballot_sync(0xffffffffu, on);
        const int pos = h + __popc(bal & ((1u << lane) - 1u));
        if (on) shit[(int64_t)si * nts + pos] = ti;
        h += __popc(bal);
    }
    if (lane == 0) scount[si] = h;
}

// Whether two boxes are within cr of each other.
__device__ __forceinline__ bool box_test(float4 slo, float4 shi, float4 tlo, float4 thi, float cr)
{
    const float dx = fmaxf(0.f, fmaxf(tlo.x - shi.x, slo.x - thi.x));
    const float dy = fmaxf(0.f, fmaxf(tlo.y - shi.y, slo.y - thi.y));
    const float dz = fmaxf(0.f, fmaxf(tlo.z - shi.z, slo.z - thi.z));
    return dx * dx + dy * dy + dz * dz <= cr * cr;
}

// Bucket of a source block with c of at most ntb pairs in the order of the
// sweeps, the heaviest blocks first.  Clustered targets make some blocks many
// times the average; started last, they left a quarter of the SM time of a
// launch idle (4,096 blocks x 100,000 targets).
__device__ __forceinline__ int order_bucket(int c, int ntb)
{
    return ORDER_BUCKETS - 1 - min(ORDER_BUCKETS - 1, (int)((int64_t)c * ORDER_BUCKETS / (ntb + 1)));
}

// Warp <-> FM_B consecutive source blocks (of one super-block): for each
// paired target super-block h, the 32-bit mask of its target blocks t with
// box_test(b, t); cnt[b] = total, hist[bucket of b] counts the blocks.
constexpr int FM_B = 4;
__global__ void __launch_bounds__(256)
k_fwd_masks(const float4 *__restrict__ sbox, int nsb, const float4 *__restrict__ tbox, int ntb, int nts, int hmax,
            float cr, const int *__restrict__ shit, const int *__restrict__ scount, unsigned *__restrict__ mask,
            int64_t *__restrict__ cnt, int *__restrict__ hist)
{
    const int b0 = (int)((blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5) * FM_B;
    const int lane = threadIdx.x & 31;
    if (b0 >= nsb) return;
    static_assert(SUPER % FM_B == 0, "the warp's blocks share a super-block");
    float4 slo[FM_B], shi[FM_B];
    int k[FM_B];
#pragma unroll
    for (int i = 0; i < FM_B; ++i) {
        const int b = min(b0 + i, nsb - 1);
        slo[i] = sbox[2 * b];
        shi[i] = sbox[2 * b + 1];
        k[i] = 0;
    }
    const int si = b0 / SUPER;
    const int nh = scount[si];
#pragma unroll 2
    for (int h = 0; h < nh; ++h) {
        const int t = shit[(int64_t)si * nts + h] * SUPER + lane;
        const float4 tlo = tbox[2 * min(t, ntb - 1)], thi = tbox[2 * min(t, ntb - 1) + 1];
#pragma unroll
        for (int i = 0; i < FM_B; ++i) {
            const bool hit = t < ntb && box_test(slo[i], shi[i], tlo, thi, cr);
            const unsigned bal = __ballot_sync(0xffffffffu, hit);
            if (lane == i && b0 + i < nsb) mask[(int64_t)(b0 + i) * hmax + h] = bal;
            k[i] += __popc(bal);
        }
    }
#pragma unroll
    for (int i = 0; i < FM_B; ++i)
        if (lane == i && b0 + i < nsb) {
            cnt[b0 + i] = k[i];
            atomicAdd(&hist[order_bucket(k[i], ntb)], 1);
        }
}

// Forward lists from the masks: fwd_t[fwd_off[b] ..] = paired t, ascending.
// order: the blocks by bucket (hist: the buckets' first positions, advanced).
// Inverse lists are the forward lists transposed (the same pair set by
// construction).
__global__ void __launch_bounds__(256)
k_fwd_fill(int nsb, int nts, int hmax, const int *__restrict__ shit, const int *__restrict__ scount,
           const unsigned *__restrict__ mask, const int64_t *__restrict__ fwd_off, int *__restrict__ fwd_t, int ntb,
           int *__restrict__ hist, int *__restrict__ order)
{
    const int b = (int)((blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5);
    const int lane = threadIdx.x & 31;
    if (b >= nsb) return;
    const int si = b / SUPER;
    const int nh = scount[si];
    int64_t k = fwd_off[b];
    for (int h = 0; h < nh; ++h) {
        const unsigned bal = mask[(int64_t)b * hmax + h];
        if ((bal >> lane) & 1u) fwd_t[k + __popc(bal & ((1u << lane) - 1u))] = shit[(int64_t)si * nts + h] * SUPER + lane;
        k += __popc(bal);
    }
    // (the blocks of a bucket in any order: no result depends on it)
    if (lane == 0) order[atomicAdd(&hist[order_bucket((int)(k - fwd_off[b]), ntb)], 1)] = b;
}

// Warp <-> source block b, lanes over its forward entries: count the pairs of
// each target block (integer atomics, exact totals).
__global__ void __launch_bounds__(256)
k_inv_count(int nsb, const int64_t *__restrict__ fwd_off, const int *__restrict__ fwd_t,
            unsigned long long *__restrict__ cnt)
{
    const int b = (int)((blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5);
    const int lane = threadIdx.x & 31;
    if (b >= nsb) return;
    for (int64_t k = fwd_off[b] + lane; k < fwd_off[b + 1]; k += 32) atomicAdd(&cnt[fwd_t[k]], 1ull);
}

// Scatter each forward pair (b, t) into t's segment of the inverse list, in
// arrival order: tmp_b = b, tmp_k = forward position.  k_inv_order then
// fixes the order.
__global__ void __launch_bounds__(256)
k_inv_scatter(int nsb, const int64_t *__restrict__ fwd_off, const int *__restrict__ fwd_t,
              const int64_t *__restrict__ inv_off, unsigned long long *__restrict__ fill, int *__restrict__ tmp_b,
              int64_t *__restrict__ tmp_k)
{
    const int b = (int)((blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5);
    const int lane = threadIdx.x & 31;
    if (b >= nsb) return;
    for (int64_t k = fwd_off[b] + lane; k < fwd_off[b + 1]; k += 32) {
        const int t = fwd_t[k];
        const int64_t pos = inv_off[t] + (int64_t)atomicAdd(&fill[t], 1ull);
        tmp_b[pos] = b;
        tmp_k[pos] = k;
    }
}

// CTA <-> target block t: order its segment by source block (distinct within
// a segment).  With at most 32 * INV_TILE source blocks: a bitmap of the
// segment's blocks in shared memory, an exclusive scan of its word
// popcounts, and rank(b) = prefix[b / 32] + popc(bits of the word below b).
// Otherwise, up to INV_TILE entries: bitonic sort of (b, entry); longer
// segments: the rank of each entry = the number of entries with a smaller b,
// counted against INV_TILE-entry tiles.  Every way, inv_b[off + rank] = b
// (ascending b, the order the gradient reduction sums in) and
// inv_k[off + rank] = the pair's forward position.
constexpr int INV_TILE = 2048;
constexpr int INV_PER = INV_TILE / 256;
__global__ void __launch_bounds__(256)
k_inv_order(int nsb, const int64_t *__restrict__ inv_off, const int *__restrict__ tmp_b,
            const int64_t *__restrict__ tmp_k, int *__restrict__ inv_b, int64_t *__restrict__ inv_k)
{
    __shared__ int sb[INV_TILE];
    __shared__ short si[INV_TILE];
    __shared__ unsigned bm[INV_TILE];
    __shared__ int pre[INV_TILE];
    __shared__ int wsum[8];
    const int t = blockIdx.x, tid = threadIdx.x, lane = tid & 31, wp = tid >> 5;
    const int64_t off = inv_off[t];
    const int64_t L = inv_off[t + 1] - off;
    const int W = (nsb + 31) >> 5;
    if (W <= INV_TILE) {
        for (int i = tid; i < W; i += 256) bm[i] = 0u;
        __syncthreads();
        for (int64_t i = tid; i < L; i += 256) {
            const int b = tmp_b[off + i];
            atomicOr(&bm[b >> 5], 1u << (b & 31));
        }
        __syncthreads();
        int loc[INV_PER], run = 0;
#pragma unroll
        for (int u = 0; u < INV_PER; ++u) {
            const int w = tid * INV_PER + u;
            loc[u] = run;
            run += w < W ? __popc(bm[w]) : 0;
        }
        int x = run;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += v;
        }
        if (lane == 31) wsum[wp] = x;
        __syncthreads();
        int base = x - run;
        for (int w = 0; w < wp; ++w) base += wsum[w];
#pragma unroll
        for (int u = 0; u < INV_PER; ++u) {
            const int w = tid * INV_PER + u;
            if (w < W) pre[w] = base + loc[u];
        }
        __syncthreads();
        for (int64_t i = tid; i < L; i += 256) {
            const int b = tmp_b[off + i];
            const int r = pre[b >> 5] + __popc(bm[b >> 5] & ((1u << (b & 31)) - 1u));
            inv_b[off + r] = b;
            inv_k[off + r] = tmp_k[off + i];
        }
        return;
    }
    if (L <= INV_TILE) {
        int n = 2;
        while (n < L) n <<= 1;
        for (int i = tid; i < n; i += 256) {
            sb[i] = i < L ? tmp_b[off + i] : 0x7fffffff;
            si[i] = (short)i;
        }
        __syncthreads();
        for (int k = 2; k <= n; k <<= 1) {
            for (int j = k >> 1; j > 0; j >>= 1) {
                for (int i = tid; i < n; i += 256) {
                    const int p = i ^ j;
                    if (p > i) {
                        const int a = sb[i], b = sb[p];
                        if ((a > b) == ((i & k) == 0)) {
                            sb[i] = b;
                            sb[p] = a;
                            const short x = si[i];
                            si[i] = si[p];
                            si[p] = x;
                        }
                    }
                }
                __syncthreads();
            }
        }
        for (int i = tid; i < L; i += 256) {
            inv_b[off + i] = sb[i];
            inv_k[off + i] = tmp_k[off + si[i]];
        }
        return;
    }
    for (int64_t i0 = 0; i0 < L; i0 += INV_TILE) {
        int mine[INV_PER], rank[INV_PER];
#pragma unroll
        for (int u = 0; u < INV_PER; ++u) {
            const int64_t i = i0 + tid + 256 * u;
            mine[u] = i < L ? tmp_b[off + i] : 0x7fffffff;
            rank[u] = 0;
        }
        for (int64_t j0 = 0; j0 < L; j0 += INV_TILE) {
            const int nj = (int)min((int64_t)INV_TILE, L - j0);
            __syncthreads();
            for (int j = tid; j < nj; j += 256) sb[j] = tmp_b[off + j0 + j];
            __syncthreads();
            for (int j = 0; j < nj; ++j) {
                const int v = sb[j];
#pragma unroll
                for (int u = 0; u < INV_PER; ++u) rank[u] += v < mine[u] ? 1 : 0;
            }
        }
#pragma unroll
        for (int u = 0; u < INV_PER; ++u) {
            const int64_t i = i0 + tid + 256 * u;
            if (i < L) {
                inv_b[off + rank[u]] = mine[u];
                inv_k[off + rank[u]] = tmp_k[off + i];
            }
        }
    }
}

// exclusive scan of n counts into off[0..n] (single CTA, order-fixed)
// total_host (may be null): the total, for the host; hist (may be null): bucket
// counts, replaced by the buckets' first positions
__global__ void __launch_bounds__(1024)
k_scan(const int64_t *__restrict__ cnt, int64_t n, int64_t *__restrict__ off, double *__restrict__ total_host,
       int *__restrict__ hist)
{
    // passes of 1,024 x SP counts: each thread loads SP consecutive counts at
    // once (the CTA is bound by load latency), the thread sums are scanned by
    // warp shuffles and warp 0, and a running carry crosses the passes
    // (integer sums: exact in any order)
    constexpr int SP = 8;
    __shared__ long long wsum[32];
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    long long carry = 0;
    for (int64_t t0 = 0; t0 < n; t0 += 1024 * SP) {
        const int64_t base = t0 + (int64_t)tid * SP;
        long long v[SP], tsum = 0;
#pragma unroll
        for (int k = 0; k < SP; ++k) v[k] = base + k < n ? (long long)cnt[base + k] : 0;
#pragma unroll
        for (int k = 0; k < SP; ++k) tsum += v[k];
        long long x = tsum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const long long y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        if (lane == 31) wsum[w] = x;
        __syncthreads();
        if (w == 0) {
            long long z = wsum[lane];
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const long long y = __shfl_up_sync(0xffffffffu, z, o);
                if (lane >= o) z += y;
            }
            wsum[lane] = z;
        }
        __syncthreads();
        long long run = carry + (w > 0 ? wsum[w - 1] : 0) + x - tsum;
#pragma unroll
        for (int k = 0; k < SP; ++k) {
            if (base + k < n) off[base + k] = (int64_t)run;
            run += v[k];
        }
        carry += wsum[31];
        __syncthreads();  // wsum is rewritten by the next pass
    }
    if (tid == 0) {
        off[n] = (int64_t)carry;
        if (total_host) *total_host = (double)carry;
    }
    if (hist && w == 31) {
        constexpr int PER = ORDER_BUCKETS / 32;
        int h[PER], sum = 0;
#pragma unroll
        for (int k = 0; k < PER; ++k) {
            h[k] = hist[lane * PER + k];
            sum += h[k];
        }
        int x = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        x -= sum;
#pragma unroll
        for (int k = 0; k < PER; ++k) {
            hist[lane * PER + k] = x;
            x += h[k];
        }
    }
}

// ---------------------------------------------------------------------------
// fused value + gradient sweeps
// ---------------------------------------------------------------------------

// Stage the targets of the forward pairs [k0, k1) of block b, culled per
// target against the block sphere: each warp takes target blocks (lane <->
// target), counts its survivors with a ballot, and whole target blocks are
// accepted in list order while the staged total fits FT_MAXS.  Returns the
// number of forward entries consumed; staged order = (target block, slot).
template <int DIM, class SM>
__device__ int stage_chunk(SM &sm, const FusedArgs &f, int64_t kb, int64_t k0, int64_t k1, const double *bc,
                           double rcull2)
{
    constexpr int SUB = 4;                       // target blocks per warp per iteration
    constexpr int PER = FT_WARPS * SUB;          // entries examined per iteration
    const int tid = threadIdx.x, lane = tid & 31, wp = tid >> 5;
    int total = 0, nb = 0;
    int64_t k = k0;
    while (k < k1 && nb < FT_MAXT) {
        unsigned bal[SUB];
        int64_t jj[SUB];
#pragma unroll
        for (int s = 0; s < SUB; ++s) {
            const int idx = s * FT_WARPS + wp;
            const int64_t e = k + idx;
            bal[s] = 0u;
            jj[s] = 0;
            int cntv = -1;
            if (e < k1 && nb + idx < FT_MAXT) {
                int sz;
                int64_t j0;
                if (e - kb < FT_PREF) {
                    j0 = sm.ent_j0[e - kb];
                    sz = sm.ent_sz[e - kb];
                } else {
                    const int t = f.fwd_t[e];
                    j0 = f.tblk_off[t];
                    sz = (int)(f.tblk_off[t + 1] - j0);
                }
                jj[s] = j0;
                bool keep = false;
                if (lane < sz) {
                    const double *tp = f.tpk + j0 + lane;
                    double d2 = 0.0;
#pragma unroll
                    for (int d = 0; d < DIM; ++d) {
                        const double q = tp[d * f.nt] - bc[d];
                        d2 += q * q;
                    }
                    keep = d2 <= rcull2;
                }
                bal[s] = __ballot_sync(0xffffffffu, keep);
                cntv = __popc(bal[s]);
            }
            if (lane == 0) sm.ecnt[idx] = cntv;
        }
        __syncthreads();
        // accept entries in list order while they fit: warp 0 scans the PER
        // survivor counts (lane <-> entry), the prefix goes through smem
        if (wp == 0) {
            const int cv = sm.ecnt[lane];
            int incl = cv < 0 ? 0 : cv;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int v = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += v;
            }
            const int excl = incl - (cv < 0 ? 0 : cv);
            const unsigned bad = __ballot_sync(0xffffffffu, cv < 0 || total + incl > SM::MAXS);
            const int na = bad ? __ffs(bad) - 1 : 32;
            sm.epre[lane] = total + excl;
            const int accsum = __shfl_sync(0xffffffffu, incl, na > 0 ? na - 1 : 0);
            if (lane == 0) {
                sm.eacc = na;
                sm.etot = total + (na > 0 ? accsum : 0);
            }
        }
        __syncthreads();
        const int nacc = sm.eacc;
        const int run = nacc > 0 ? sm.etot : total;
#pragma unroll
        for (int s = 0; s < SUB; ++s) {
            const int idx = s * FT_WARPS + wp;
            if (idx < nacc) {
                const int slot = nb + idx;
                const int64_t j0 = jj[s];
                const bool keep = (bal[s] >> lane) & 1u;
                if (keep) {
                    const int pos = sm.epre[idx] + __popc(bal[s] & ((1u << lane) - 1u));
                    sm.dst[pos] = (unsigned short)(slot * TBLK_KD + lane);
                    const double *tp = f.tpk + j0 + lane;
#pragma unroll
                    for (int d = 0; d < FT_TS; ++d) sm.stg[d][pos] = tp[d * f.nt];
                }
                if (lane == 0) sm.keep[slot] = bal[s];
            }
        }
        total = run;
        nb += nacc;
        k += nacc;
        __syncthreads();
        if (nacc < PER) break;  // capacity reached, list exhausted or block limit
    }
    if (tid == 0) sm.nstg = total;
    __syncthreads();
    return nb;
}

// Value-sweep pair loop of one unit over its compacted candidates.
// MODE 0: shift M = per-unit upper bound, exponents provably >= -16000 (no
//         clamp); MODE 1: same with the clamp; MODE 2: per-pair lazy rescale
//         (when the bound could sit more than 2^500 above the true maximum).
// NQ: quadrature points handled (== QL for full units: straight-line code
//     whose NQ exponential chains interleave).
template <int DIM, int QL, int NQ, int MODE, class SM>
__device__ __forceinline__ void value_pairs(const SM &sm, int wp, int lane, int ncand, int qoff, double cc0,
                                            double cc1, double cc2, const EvalArgs &a, double Munit, double *M,
                                            double *S, double *mx)
{
    for (int p = lane; p < ncand; p += 32) {
        const int ti = sm.cand[wp][p];
        const double g0 = sm.stg[0][ti] - cc0, g1 = sm.stg[1][ti] - cc1;
        const double g2 = DIM == 3 ? sm.stg[2][ti] - cc2 : 0.0;
        const double d2 = DIM == 3 ? g0 * g0 + g1 * g1 + g2 * g2 : g0 * g0 + g1 * g1;
        const double B0 = fma(-a.halfs, d2, sm.stg[5][ti]) - (MODE == 2 ? 0.0 : Munit);
        const double G0 = a.s * g0, G1 = a.s * g1, G2 = a.s * g2;
        const double nuj = sm.stg[3][ti];
#pragma unroll
        for (int q = 0; q < NQ; ++q) {
            const double *dq = sm.qd[qoff + q];
            double bb = fma(G0, dq[0], B0);
            bb = fma(G1, dq[1], bb);
            if (DIM == 3) bb = fma(G2, dq[2], bb);
            if (MODE == 2) {
                lse_update(bb, nuj, M[q], S[q], mx[q], sm.tab);
            } else {
                mx[q] = fmax(mx[q], bb);
                S[q] = fma(nuj, MODE == 0 ? exp2_16_nc(bb, sm.tab) : exp2_16(bb, sm.tab), S[q]);
            }
        }
    }
}

// Units with fewer than QL quadrature points (the last q-group of a cell).
template <int DIM, int QL, int MODE, class SM>
__device__ __noinline__ void value_pairs_partial(const SM &sm, int wp, int lane, int ncand, int qoff, int nql,
                                                 double cc0, double cc1, double cc2, const EvalArgs &a, double Munit,
                                                 double *M, double *S, double *mx)
{
    for (int p = lane; p < ncand; p += 32) {
        const int ti = sm.cand[wp][p];
        const double g0 = sm.stg[0][ti] - cc0, g1 = sm.stg[1][ti] - cc1;
        const double g2 = DIM == 3 ? sm.stg[2][ti] - cc2 : 0.0;
        const double d2 = DIM == 3 ? g0 * g0 + g1 * g1 + g2 * g2 : g0 * g0 + g1 * g1;
        const double B0 = fma(-a.halfs, d2, sm.stg[5][ti]) - (MODE == 2 ? 0.0 : Munit);
        const double G0 = a.s * g0, G1 = a.s * g1, G2 = a.s * g2;
        const double nuj = sm.stg[3][ti];
#pragma unroll
        for (int q = 0; q < QL; ++q) {
            if (q < nql) {
                const double *dq = sm.qd[qoff + q];
                double bb = fma(G0, dq[0], B0);
                bb = fma(G1, dq[1], bb);
                if (DIM == 3) bb = fma(G2, dq[2], bb);
                if (MODE == 2) {
                    lse_update(bb, nuj, M[q], S[q], mx[q], sm.tab);
                } else {
                    mx[q] = fmax(mx[q], bb);
                    S[q] = fma(nuj, exp2_16(bb, sm.tab), S[q]);
                }
            }
        }
    }
}

// Exact candidate test of the staged targets for the warp's cell, in-order
// compaction into sm.cand[wp]; returns the count and (through bmax) the
// largest B0_Kj = kappa (psi_j - d2/2)/eps over the candidates.  With TQ > 0
// also (through lb) the largest lower bound B0_Kj - sum_d |G_Kj,d| a_d of a
// candidate's exponents at the cell's points (a: their offsets; gh = s a).
template <int DIM, int TQ, class SM>
__device__ __forceinline__ int compact_candidates(SM &sm, int wp, int lane, int nstg, const double *cc,
                                                  const EvalArgs &a, const double *gh, double &bmax, double &lb)
{
    constexpr int U = 4;  // staged targets per lane in flight (independent distance chains)
    int ncand = 0;
    bmax = -CUDART_INF;
    lb = -CUDART_INF;
    for (int b0 = 0; b0 < nstg; b0 += 32 * U) {
        bool in[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int t = b0 + 32 * u + lane;
            in[u] = false;
            if (t < nstg) {
                const double y[3] = {sm.stg[0][t], sm.stg[1][t], DIM == 3 ? sm.stg[2][t] : 0.0};
                const double d2 = dist2_exact<DIM>(y, cc);
                in[u] = d2 <= a.sstar;
                if (in[u]) {
                    const double B0 = fma(-a.halfs, d2, sm.stg[5][t]);
                    bmax = fmax(bmax, B0);
                    if (TQ > 0) {
                        double l = B0;
#pragma unroll
                        for (int d = 0; d < DIM; ++d) l = fma(-fabs(y[d] - cc[d]), gh[d], l);
                        lb = fmax(lb, l);
                    }
                }
            }
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const unsigned bal = __ballot_sync(0xffffffffu, in[u]);
            if (in[u]) sm.cand[wp][ncand + __popc(bal & ((1u << lane) - 1u))] = (unsigned short)(b0 + 32 * u + lane);
            ncand += __popc(bal);
        }
    }
    bmax = warp_max(bmax);
    if (TQ > 0) lb = warp_max(lb);
    __syncwarp();
    return ncand;
}

// A unit's part of the gradient of one target, sum over the unit's q of
// w_q nu_j e^{t_qj - L_q} at g = y_j - c_K: E0 and G' are formed in FP64 per
// (cell, target) so that every FP32 operand of the hybrid form is small.
// lognu = log2 nu_j, sp = kappa psi_j / eps.
template <int DIM, bool FP32B, class SM>
__device__ __forceinline__ typename PRow<FP32B>::T grad_term(const SM &sm, int w_nonneg, int qoff, int nql,
                                                             const double *g, double lognu, double sp, double Lref,
                                                             const EvalArgs &a)
{
    const double g0 = g[0], g1 = g[1], g2 = DIM == 3 ? g[2] : 0.0;
    const double d2 = DIM == 3 ? g0 * g0 + g1 * g1 + g2 * g2 : g0 * g0 + g1 * g1;
    if constexpr (FP32B) {
        const float sf = (float)(a.s * (1.0 / 16.0));
        const float e0 = (float)(lognu + (fma(-a.halfs, d2, sp) - KAPPA * Lref) * (1.0 / 16.0));
        const float G0 = sf * (float)g0, G1 = sf * (float)g1, G2 = sf * (float)g2;
        float acc0 = 0.f, acc1 = 0.f;
        if (w_nonneg) {
            int q = 0;
            for (; q + 1 < nql; q += 2) {
                const float4 v0 = *reinterpret_cast<const float4 *>(sm.qb[qoff + q]);
                const float4 v1 = *reinterpret_cast<const float4 *>(sm.qb[qoff + q + 1]);
                float ea = fmaf(G0, v0.x, e0 + v0.w), eb = fmaf(G0, v1.x, e0 + v1.w);
                ea = fmaf(G1, v0.y, ea);
                eb = fmaf(G1, v1.y, eb);
                if (DIM == 3) {
                    ea = fmaf(G2, v0.z, ea);
                    eb = fmaf(G2, v1.z, eb);
                }
                acc0 += ex2_approx(ea);
                acc1 += ex2_approx(eb);
            }
            if (q < nql) {
                const float4 v0 = *reinterpret_cast<const float4 *>(sm.qb[qoff + q]);
                float ea = fmaf(G0, v0.x, e0 + v0.w);
                ea = fmaf(G1, v0.y, ea);
                if (DIM == 3) ea = fmaf(G2, v0.z, ea);
                acc0 += ex2_approx(ea);
            }
        } else {
            for (int q = 0; q < nql; ++q) {
                const float *qb = sm.qb[qoff + q];
                float e = fmaf(G0, qb[0], e0 + qb[3]);
                e = fmaf(G1, qb[1], e);
                if (DIM == 3) e = fmaf(G2, qb[2], e);
                acc0 = fmaf(sm.qw[qoff + q], ex2_approx(e), acc0);
            }
        }
        return acc0 + acc1;
    } else {
        const double U0 = 16.0 * lognu + fma(-a.halfs, d2, sp) - KAPPA * Lref;
        const double G0 = a.s * g0, G1 = a.s * g1, G2 = a.s * g2;
        double acc = 0.0;
        for (int q = 0; q < nql; ++q) {
            const double *dq = sm.qd[qoff + q];
            const double L = sm.qL[qoff + q];
            if (!isfinite(L)) continue;
            double u = fma(G0, dq[0], U0 + dq[3] - KAPPA * (L - Lref));
            u = fma(G1, dq[1], u);
            if (DIM == 3) u = fma(G2, dq[2], u);
            acc = fma(sm.qw[qoff + q], exp2_16(u, sm.tab), acc);
        }
        return acc;
    }
}

// Tensor-product points (TM per dimension, symmetric about the cell centre):
// delta_q = (s_0 a_0, s_1 a_1, s_2 a_2) with s_d in {-1, 0, +1}, so
// 2^(b_qj/16) = nu_j 2^(B0_Kj/16) prod_d 2^(s_d G_Kj,d a_d/16) and one
// candidate costs 1 + DIM exponentials and DIM reciprocals for its TM^DIM
// points.  Sums stay relative to Munit (LSE mode only).
template <int TM, int D>
__device__ __forceinline__ constexpr int tstride()
{
    return D == 0 ? 1 : (D == 1 ? TM : TM * TM);
}

// A factor of a product of up to 1 + 2 DIM: exp2_16's 1.5e-13 (always too
// small, 2e-14 on average) would add up over them, so the FP64 mode takes the
// one more term of the polynomial.  Gradients of the FP64 mode against 64
// bits, largest relative error of a target's mass over eight problems: 5e-14
// to 1.5e-13 with an exponential per point, up to 1.8e-13 with exp2_16's
// factors, 1.4e-15 to 3.7e-15 with these; no difference in time (147,456
// points x 10,000 targets in 2D: 187 and 185 us).
template <bool FULL>
__device__ __forceinline__ double exp2_factor(double u, const double *tab)
{
    return FULL ? exp2_16_full(u, tab) : exp2_16(u, tab);
}

// The per-q maximum exponent (the reference's m of the log-sum-exp, which
// C_global depends on) is taken exactly, but only over the candidates that
// can attain it: those whose upper bound B0 + sum_d |G_d| a_d reaches the
// largest lower bound lb of any candidate (relative to Munit here).  They are
// listed (one in 20 to 100 of a cell's candidates) and their exponents taken
// afterwards by near_maxima, lane <-> point, so that the loop keeps no maxima
// in registers.  FULL (the FP64 mode): factors to a few ulp (exp2_factor).
template <int DIM, int TM, int TS, bool FULL, class SM>
__device__ __forceinline__ void value_pairs_tensor(SM &sm, int wp, int lane, int ncand, const double *ah,
                                                   const double *cc, const EvalArgs &a, double Munit, double lb,
                                                   double *S)
{
    for (int p = lane; p < ncand; p += 32) {
        const int ti = sm.cand[wp][p];
        const double g0 = sm.stg[0][ti] - cc[0], g1 = sm.stg[1][ti] - cc[1];
        const double g2 = DIM == 3 ? sm.stg[2][ti] - cc[2] : 0.0;
        const double d2 = DIM == 3 ? g0 * g0 + g1 * g1 + g2 * g2 : g0 * g0 + g1 * g1;
        const double B0 = fma(-a.halfs, d2, sm.stg[5][ti]) - Munit;
        const double G[3] = {a.s * g0, a.s * g1, a.s * g2};
        // per-dimension factors 2^(G_d delta_d): with TS, relative to the lowest
        // point (1, r, r^2 with the shift folded into P); otherwise 2^(-G a), (1), 2^(G a)
        double F[3][TM], ga[3], ub = B0;
        double P;
#pragma unroll
        for (int d = 0; d < DIM; ++d) {
            ga[d] = G[d] * ah[d];
            ub += fabs(ga[d]);
        }
        if (ub >= lb) {
            const int at = atomicAdd(&sm.nnear[wp], 1);
            if (at < FT_NEAR) sm.near_list[wp][at] = (unsigned short)ti;
        }
        if constexpr (TS >= 1) {
            double sga = 0.0;
#pragma unroll
            for (int d = 0; d < DIM; ++d) {
                sga += ga[d];
                const double r = exp2_factor<FULL>(TM == 2 ? 2.0 * ga[d] : ga[d], sm.tab);
                F[d][0] = 1.0;
                F[d][1] = r;
                if (TM == 3) F[d][2] = r * r;
            }
            P = sm.stg[3][ti] * exp2_factor<FULL>(B0 - sga, sm.tab);
        } else {
#pragma unroll
            for (int d = 0; d < DIM; ++d) {
                const double xp = exp2_factor<FULL>(ga[d], sm.tab);
                F[d][0] = __drcp_rn(xp);
                F[d][TM - 1] = xp;
                if (TM == 3) F[d][1] = 1.0;
            }
            P = sm.stg[3][ti] * exp2_factor<FULL>(B0, sm.tab);
        }
#pragma unroll
        for (int i0 = 0; i0 < TM; ++i0) {
            const double t0 = P * F[0][i0];
            if (DIM == 2) {
#pragma unroll
                for (int i1 = 0; i1 < TM; ++i1) S[i0 + TM * i1] = fma(t0, F[1][i1], S[i0 + TM * i1]);
            } else {
#pragma unroll
                for (int i1 = 0; i1 < TM; ++i1) {
                    const double t1 = t0 * F[1][i1];
#pragma unroll
                    for (int i2 = 0; i2 < TM; ++i2) {
                        const int q = i0 + TM * i1 + TM * TM * i2;
                        S[q] = fma(t1, F[2][i2], S[q]);
                    }
                }
            }
        }
    }
}

// Largest exponents (absolute) of the unit's points over the listed
// candidates (all of them where the list overflowed): lanes <-> (point q =
// lane mod NQ, every EP-th candidate), one running maximum per lane.
template <int DIM, int NQ, class SM>
__device__ __forceinline__ void near_maxima(const SM &sm, int wp, int lane, int ncand, int qoff, const double *cc,
                                            const EvalArgs &a, double &mx)
{
    constexpr int EP = 32 / NQ;
    const int q = lane % NQ, sub = lane / NQ;
    const int n = sm.nnear[wp];
    const bool all = n > FT_NEAR;
    const int cnt = all ? ncand : n;
    if (sub >= EP) return;
    const double *dq = sm.qd[qoff + q];
    for (int p = sub; p < cnt; p += EP) {
        const int ti = all ? sm.cand[wp][p] : sm.near_list[wp][p];
        const double g0 = sm.stg[0][ti] - cc[0], g1 = sm.stg[1][ti] - cc[1];
        const double g2 = DIM == 3 ? sm.stg[2][ti] - cc[2] : 0.0;
        const double d2 = DIM == 3 ? g0 * g0 + g1 * g1 + g2 * g2 : g0 * g0 + g1 * g1;
        double bb = fma(a.s * g0, dq[0], fma(-a.halfs, d2, sm.stg[5][ti]));
        bb = fma(a.s * g1, dq[1], bb);
        if (DIM == 3) bb = fma(a.s * g2, dq[2], bb);
        mx = fmax(mx, bb);
    }
}

// Sums over the lanes of the unit's NQ per-lane sums; q's total ends in lane
// q * (32 / 2^ceil(log2 NQ)) for q < 8 (transposed butterflies: each exchange
// halves the sums a lane keeps, NQ + log2 exchanges instead of 5 NQ) and, for
// NQ = 9, the ninth in every lane (last).
template <int NQ>
__device__ __forceinline__ double lane_totals(const double *S, int lane, double &last)
{
    constexpr int H = NQ == 4 ? 2 : 4;   // sums kept after the first exchange
    constexpr int FIRST = 16;
    double s[H];
    const bool b4 = lane & FIRST;
#pragma unroll
    for (int k = 0; k < H; ++k) {
        const double keep = b4 ? S[H + k] : S[k], give = b4 ? S[k] : S[H + k];
        s[k] = keep + __shfl_xor_sync(0xffffffffu, give, FIRST);
    }
    int o = 8;
#pragma unroll
    for (int h = H / 2; h > 0; h >>= 1, o >>= 1) {
        const bool b = lane & o;
#pragma unroll
        for (int k = 0; k < H / 2; ++k) {
            if (k >= h) continue;
            const double keep = b ? s[h + k] : s[k], give = b ? s[k] : s[h + k];
            s[k] = keep + __shfl_xor_sync(0xffffffffu, give, o);
        }
    }
#pragma unroll
    for (int e = NQ == 4 ? 4 : 2; e > 0; e >>= 1) s[0] += __shfl_xor_sync(0xffffffffu, s[0], e);
    last = NQ == 9 ? warp_sum(S[NQ - 1]) : 0.0;
    return s[0];
}

__device__ __forceinline__ float rcp_approx(float x)
{
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// grad_term on tensor-product points: 2^(e0) sum_q W_q prod_d F_d[i_d],
// W_q = w_q 2^(D_q), summed dimension by dimension (Horner order).  The FP64
// form takes the factors relative to the lowest point.
template <int DIM, int TM, int TS, bool FP32B, class SM>
__device__ __forceinline__ typename PRow<FP32B>::T grad_term_tensor(const SM &sm, int qoff, const double *ahd,
                                                                    const double *g, double lognu, double sp,
                                                                    double Lref, const EvalArgs &a)
{
    constexpr int NQ = DIM == 3 ? TM * TM * TM : TM * TM;
    using Row = typename PRow<FP32B>::T;
    Row W[NQ];
#pragma unroll
    for (int q = 0; q < NQ; ++q) W[q] = sm.qtw[qoff + q];
    const double d2 = DIM == 3 ? g[0] * g[0] + g[1] * g[1] + g[2] * g[2] : g[0] * g[0] + g[1] * g[1];
    if constexpr (FP32B) {
        const float sf = (float)(a.s * (1.0 / 16.0));
        float e0 = (float)(lognu + (fma(-a.halfs, d2, sp) - KAPPA * Lref) * (1.0 / 16.0));
        float F[3][TM];
        if constexpr (TS >= 1) {
#pragma unroll
            for (int d = 0; d < DIM; ++d) {
                const float ga = sf * (float)g[d] * (float)ahd[d];
                e0 -= ga;
                const float r = ex2_approx(TM == 2 ? 2.f * ga : ga);
                F[d][0] = 1.f;
                F[d][1] = r;
                if (TM == 3) F[d][2] = r * r;
            }
        } else {
#pragma unroll
            for (int d = 0; d < DIM; ++d) {
                const float xp = ex2_approx(sf * (float)g[d] * (float)ahd[d]);
                F[d][0] = rcp_approx(xp);
                F[d][TM - 1] = xp;
                if (TM == 3) F[d][1] = 1.f;
            }
        }
        float w = 0.f;
        if (DIM == 2) {
#pragma unroll
            for (int i0 = 0; i0 < TM; ++i0) {
                float u = 0.f;
#pragma unroll
                for (int i1 = 0; i1 < TM; ++i1) u = fmaf(W[i0 + TM * i1], F[1][i1], u);
                w = fmaf(u, F[0][i0], w);
            }
        } else {
#pragma unroll
            for (int i0 = 0; i0 < TM; ++i0) {
                float u = 0.f;
#pragma unroll
                for (int i1 = 0; i1 < TM; ++i1) {
                    float v = 0.f;
#pragma unroll
                    for (int i2 = 0; i2 < TM; ++i2) v = fmaf(W[i0 + TM * i1 + TM * TM * i2], F[2][i2], v);
                    u = fmaf(v, F[1][i1], u);
                }
                w = fmaf(u, F[0][i0], w);
            }
        }
        return ex2_approx(e0) * w;
    } else {
        double U = 16.0 * lognu + fma(-a.halfs, d2, sp) - KAPPA * Lref;
        double r[3];
#pragma unroll
        for (int d = 0; d < DIM; ++d) {
            const double ga = a.s * g[d] * ahd[d];
            U -= ga;
            r[d] = exp2_16_full(TM == 2 ? 2.0 * ga : ga, sm.tab);
        }
        double w = 0.0;
#pragma unroll
        for (int i0 = TM - 1; i0 >= 0; --i0) {
            double u = 0.0;
#pragma unroll
            for (int i1 = TM - 1; i1 >= 0; --i1) {
                double v = 0.0;
                if (DIM == 2) {
                    v = W[i0 + TM * i1];
                } else {
#pragma unroll
                    for (int i2 = TM - 1; i2 >= 0; --i2)
                        v = i2 == TM - 1 ? W[i0 + TM * i1 + TM * TM * i2]
                                         : fma(v, r[2], W[i0 + TM * i1 + TM * TM * i2]);
                }
                u = i1 == TM - 1 ? v : fma(u, r[1], v);
            }
            w = i0 == TM - 1 ? u : fma(w, r[0], u);
        }
        return exp2_16_full(U, sm.tab) * w;
    }
}

// A target's gradient terms over the block's units, tensor-product points:
// the exact candidate test (the FP32 squared distance about the block's
// centre decides outside [lo, hi], the FP64 one, rounded like the
// reference's, inside) and grad_term_tensor.  FP32 in 3D is bound by the
// special-function unit (exponentials and conversions between FP32 and
// FP64); where the block's cells have at most two centre coordinates per
// dimension (brick), the target's differences, factors and their conversions
// are taken once per coordinate: 12 per target and 3 per cell instead of 9
// per cell, the same operations on the same operands.
template <int DIM, int TM, bool FP32B, int TS, class SM>
__device__ __forceinline__ double unit_terms(const SM &sm, const double *y, double lognu, double sp, bool on,
                                             bool brick, int nunit, const double *bc, float lo, float hi,
                                             const EvalArgs &a)
{
    constexpr int NQ = DIM == 3 ? TM * TM * TM : TM * TM;
    float z[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) z[d] = d < DIM ? (float)(y[d] - bc[d]) : 0.f;
    double v = 0.0;
    if (brick) {
        if constexpr (DIM == 3 && FP32B && TM == 2) {
            const float sf = (float)(a.s * (1.0 / 16.0));
            double g[3][2];
            float zz[3][2], ga[3][2], Fl[3][2], Fh[3][2];
#pragma unroll
            for (int d = 0; d < 3; ++d)
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    g[d][i] = y[d] - sm.cs[d][i];
                    const float zc = z[d] - sm.csf[d][i];
                    zz[d][i] = zc * zc;
                    ga[d][i] = sf * (float)g[d][i] * sm.ahf[d];
                    if (TS >= 1) {
                        Fl[d][i] = 1.f;
                        Fh[d][i] = ex2_approx(2.f * ga[d][i]);
                    } else {
                        Fh[d][i] = ex2_approx(ga[d][i]);
                        Fl[d][i] = rcp_approx(Fh[d][i]);
                    }
                }
#pragma unroll
            for (int c = 0; c < 8; ++c) {
                const int u = sm.cell_at[c];
                if (u < 0) continue;
                const int i0 = c & 1, i1 = (c >> 1) & 1, i2 = c >> 2;
                const float d2f = zz[2][i2] + (zz[1][i1] + zz[0][i0]);
                bool in = d2f < lo;
                if (!in && !(d2f > hi)) in = dist2_exact<3>(y, sm.cellc[u]) <= a.sstar;
                const double Lref = sm.uL[u];
                if (!in || !on || !isfinite(Lref)) continue;
                float W[8];
#pragma unroll
                for (int q = 0; q < 8; ++q) W[q] = sm.qtw[8 * u + q];
                const double d2 = fma(g[2][i2], g[2][i2], fma(g[1][i1], g[1][i1], g[0][i0] * g[0][i0]));
                float e0 = (float)(lognu + (fma(-a.halfs, d2, sp) - KAPPA * Lref) * (1.0 / 16.0));
                if (TS >= 1) e0 = ((e0 - ga[0][i0]) - ga[1][i1]) - ga[2][i2];
                float w = 0.f;
#pragma unroll
                for (int p0 = 0; p0 < 2; ++p0) {
                    float t1 = 0.f;
#pragma unroll
                    for (int p1 = 0; p1 < 2; ++p1) {
                        const float t2 = fmaf(W[p0 + 2 * p1 + 4], Fh[2][i2], W[p0 + 2 * p1] * Fl[2][i2]);
                        t1 = p1 ? fmaf(t2, Fh[1][i1], t1) : t2 * Fl[1][i1];
                    }
                    w = p0 ? fmaf(t1, Fh[0][i0], w) : t1 * Fl[0][i0];
                }
                v += (double)(ex2_approx(e0) * w);
            }
        }
    } else {
#pragma unroll 1
        for (int u = 0; u < nunit; ++u) {
            const float gx = z[0] - sm.uf[u][0], gy = z[1] - sm.uf[u][1], gz = DIM == 3 ? z[2] - sm.uf[u][2] : 0.f;
            float d2f = fmaf(gy, gy, gx * gx);
            if (DIM == 3) d2f = fmaf(gz, gz, d2f);
            bool in = d2f < lo;
            if (!in && !(d2f > hi)) in = dist2_exact<DIM>(y, sm.cellc[u]) <= a.sstar;
            const double Lref = sm.uL[u];
            if (!in || !on || !isfinite(Lref)) continue;
            const double *cc = sm.cellc[u];
            const double g[3] = {y[0] - cc[0], y[1] - cc[1], DIM == 3 ? y[2] - cc[2] : 0.0};
            v += (double)grad_term_tensor<DIM, TM, TS, FP32B>(sm, u * NQ, sm.uah[u], g, lognu, sp, Lref, a);
        }
    }
    return v;
}

// Gradient sweep of the staged chunk (forward positions k..): thread <->
// staged target, over the block's units in order (the unit terms, FP32 in the
// hybrid mode, added in FP64), and the write of every slot of every pair
// (zeros where a target was not staged).  The exact candidate test is taken
// again per (cell, target) instead of a compacted list per cell: a target's
// data stay in registers over the units and no partial rows go through
// shared memory (rows, their zeroing and their sums, with the lists, were
// two thirds of a re-staged chunk's instructions).
template <int DIM, bool FP32B, int TQ, int TS, class SM>
__device__ __forceinline__ void grad_chunk(SM &sm, const FusedArgs &f, int64_t k, int nt, int nunit,
                                           const EvalArgs &a)
{
    const int tid = threadIdx.x;
    using Row = typename PRow<FP32B>::T;
    const int64_t base = (k - f.part_base) * TBLK_KD;
    Row *out = (FP32B ? reinterpret_cast<Row *>(f.part32) : reinterpret_cast<Row *>(f.part)) + base;
    const int nstg = sm.nstg;
    for (int p = tid; p < nstg; p += FT_WARPS * 32) {
        const double y[3] = {sm.stg[0][p], sm.stg[1][p], DIM == 3 ? sm.stg[2][p] : 0.0};
        const double lognu = sm.stg[4][p], sp = sm.stg[5][p];
        double v = 0.0;
#pragma unroll 2
        for (int u = 0; u < nunit; ++u) {
            const double *cc = sm.cellc[u];
            const double Lref = sm.uL[u];
            const double g[3] = {y[0] - cc[0], y[1] - cc[1], DIM == 3 ? y[2] - cc[2] : 0.0};
            if (dist2_exact<DIM>(y, cc) <= a.sstar && isfinite(Lref)) {
                const int cl = TQ > 0 ? u : u / a.ngroups, qoff = cl * a.qpc + (TQ > 0 ? 0 : (u - cl * a.ngroups) * a.ql);
                Row t;
                if constexpr (TQ > 0)
                    t = grad_term_tensor<DIM, TQ, TS, FP32B>(sm, qoff, sm.uah[u], g, lognu, sp, Lref, a);
                else
                    t = grad_term<DIM, FP32B>(sm, f.w_nonneg, qoff, min(a.ql, (cl + 1) * a.qpc - qoff), g, lognu, sp,
                                              Lref, a);
                v += (double)t;
            }
        }
        out[sm.dst[p]] = (Row)v;
    }
    for (int i = tid; i < nt * TBLK_KD; i += FT_WARPS * 32)
        if (!((sm.keep[i / TBLK_KD] >> (i % TBLK_KD)) & 1u)) out[i] = Row(0);
}

// Gradient sweep of the block's forward entries [k0, k1) whose targets are no
// longer staged: warp <-> entry (target block), lane <-> target, straight from
// the packed targets; every slot of the pair's partial is written.  Staging
// these chunks again took their culling, compaction and barriers a second
// time (2,097,152 points x 100,000 targets, both sweeps: 6,020 -> 5,740 us).
// The last chunk stays with grad_chunk, whose lanes are all within reach of
// the block (direct for it too: 5,907 us, and 10% slower where every block has
// one chunk; the FP32 test and bricks in grad_chunk: no gain).
template <int DIM, int TM, bool FP32B, int TS, class SM>
__device__ __forceinline__ void grad_direct(SM &sm, const FusedArgs &f, int64_t k0, int64_t k1, int nunit,
                                            const double *bc, float lo, float hi, const EvalArgs &a)
{
    const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
    using Row = typename PRow<FP32B>::T;
    Row *out = (FP32B ? reinterpret_cast<Row *>(f.part32) : reinterpret_cast<Row *>(f.part)) +
               (k0 - f.part_base) * TBLK_KD + lane;
    const bool brick = DIM == 3 && FP32B && TM == 2 && sm.brick;
    for (int e = wp; e < (int)(k1 - k0); e += FT_WARPS) {
        int64_t j0;
        int sz;
        if (e < FT_PREF) {
            j0 = sm.ent_j0[e];
            sz = sm.ent_sz[e];
        } else {
            const int t = f.fwd_t[k0 + e];
            j0 = f.tblk_off[t];
            sz = (int)(f.tblk_off[t + 1] - j0);
        }
        const double *tp = f.tpk + j0 + min(lane, sz - 1);
        double y[3] = {0.0, 0.0, 0.0};
#pragma unroll
        for (int d = 0; d < DIM; ++d) y[d] = tp[d * f.nt];
        const double lognu = tp[4 * f.nt], sp = tp[5 * f.nt];
        out[(int64_t)e * TBLK_KD] = (Row)unit_terms<DIM, TM, FP32B, TS>(sm, y, lognu, sp, lane < sz, brick, nunit, bc,
                                                                        lo, hi, a);
    }
}

// One warp's preparation of grad_direct: the units' centres in FP32 and
// whether the block is a brick.
template <int DIM, class SM>
__device__ __forceinline__ void direct_setup(SM &sm, int lane, int nunit, const double *bc)
{
    for (int i = lane; i < nunit * 3; i += 32) sm.uf[i / 3][i % 3] = (float)(sm.cellc[i / 3][i % 3] - bc[i % 3]);
    if (DIM == 2) return;
    // at most two centre coordinates per dimension, each cell at its own place, the same offsets in all?
    const int u = min(lane, nunit - 1);
    bool ok = true;
    int at = 0;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        const double c0 = sm.cellc[0][d], cu = sm.cellc[u][d];
        const unsigned other = __ballot_sync(0xffffffffu, cu != c0);
        const double c1 = other ? sm.cellc[__ffs(other) - 1][d] : c0;
        ok = ok && (cu == c0 || cu == c1) && (float)sm.uah[u][d] == (float)sm.uah[0][d];
        at |= cu == c0 ? 0 : 1 << d;
        if (lane < 2) {
            sm.cs[d][lane] = lane ? c1 : c0;
            sm.csf[d][lane] = (float)((lane ? c1 : c0) - bc[d]);
        }
        if (lane == 2) sm.ahf[d] = (float)sm.uah[0][d];
    }
    if (lane < 8) sm.cell_at[lane] = -1;
    const unsigned same = __match_any_sync(0xffffffffu, lane < nunit ? at : 32 + lane);
    ok = ok && (same & (same - 1)) == 0;
    const bool all = __all_sync(0xffffffffu, ok);
    __syncwarp();
    if (lane < nunit) sm.cell_at[at] = lane;
    if (lane == 0) sm.brick = all;
}

template <int DIM, int QL, bool FP32B, int MODE, int TQ, int TS>
__global__ void __launch_bounds__(FT_WARPS * 32, fused_min_blocks(TQ))
k_fused(FusedArgs f, EvalArgs a)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    using SMem = FTSmem<fused_cap(TQ), typename PRow<FP32B>::T>;
    SMem &sm = *reinterpret_cast<SMem *>(smem_raw);
    const int tid = threadIdx.x, lane = tid & 31, wp = tid >> 5;
    const int b = f.order ? f.order[blockIdx.x] : f.b0 + (int)blockIdx.x;
    if (tid < 16) sm.tab[tid] = c_exp2_tab[tid];
    const int64_t cb0 = f.sblk_cell[b], cb1 = f.sblk_cell[b + 1];
    const int ncell = (int)(cb1 - cb0);
    const int nunit = ncell * a.ngroups;
    const bool valid = wp < nunit;
    const int cl = valid ? wp / a.ngroups : 0;          // cell of this warp (block-local)
    const int grp = valid ? wp - cl * a.ngroups : 0;
    const int qoff = cl * a.qpc + grp * a.ql;           // block-local index of the unit's first q
    const int nql = valid ? min(a.ql, a.qpc - grp * a.ql) : 0;
    const int64_t qblk0 = cb0 * a.qpc;                  // first q of the block
    const int nqb = ncell * a.qpc;
    const double *bs = f.sblk_sph + (int64_t)b * 4;
    const double bc[3] = {bs[0], bs[1], bs[2]};
    const double rc = (f.cullt + bs[3]) * (1.0 + 1e-12) + 1e-300;
    const double rcull2 = rc * rc;
    const int64_t k0 = f.fwd_off[b], k1 = f.fwd_off[b + 1];
    for (int i = tid; i < nunit * 3; i += blockDim.x) {
        const int u = i / 3, d = i - u * 3;
        sm.cellc[u][d] = d < DIM ? f.cell_ctr[(cb0 + u / a.ngroups) * DIM + d] : 0.0;
    }
    for (int i = tid; i < (int)min((int64_t)FT_PREF, k1 - k0); i += blockDim.x) {
        const int t = f.fwd_t[k0 + i];
        const int64_t j0 = f.tblk_off[t];
        sm.ent_j0[i] = (int)j0;
        sm.ent_sz[i] = (unsigned char)(f.tblk_off[t + 1] - j0);
    }
    __syncthreads();
    for (int i = tid; i < nqb; i += blockDim.x) {
        const int c = i / a.qpc;
        double dsq = 0.0;
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            const double dl = d < DIM ? f.x[(qblk0 + i) * DIM + d] - sm.cellc[c * a.ngroups][d] : 0.0;
            sm.qd[i][d] = dl;
            dsq += dl * dl;
        }
        sm.qd[i][3] = -a.halfs * dsq;
    }
    __syncthreads();
    const int wu = valid ? wp : 0;
    const double cc[3] = {sm.cellc[wu][0], sm.cellc[wu][1], sm.cellc[wu][2]};
    // tensor points: the largest offset per dimension, and s times it
    double ah[3] = {0.0, 0.0, 0.0}, gh[3] = {0.0, 0.0, 0.0};
    if constexpr (TQ > 0) {
        ah[0] = sm.qd[qoff + (TQ - 1) * tstride<TQ, 0>()][0];
        ah[1] = sm.qd[qoff + (TQ - 1) * tstride<TQ, 1>()][1];
        if (DIM == 3) ah[2] = sm.qd[qoff + (TQ - 1) * tstride<TQ, 2>()][2];
#pragma unroll
        for (int d = 0; d < DIM; ++d) gh[d] = a.s * ah[d];
        if (valid && lane < 3) sm.uah[wp][lane] = lane == 0 ? ah[0] : (lane == 1 ? ah[1] : ah[2]);
    }
    int tail_off = -1;  // first entry (minus k0) of the value sweep's last chunk, still staged for the gradient sweep
    int tail_nt = 0;

    // ---------------- value sweep ----------------
    {
        // Shift of the online sums.  MODE 0/1: Munit = max_j B0_Kj + s r
        // max_q |delta_q| bounds every exponent of the unit from above
        // (|G_Kj| <= s r for a candidate), so no per-pair rescale is needed;
        // exponents are kept relative to Munit (mx too, on the per-point
        // sweeps) and a chunk that raises the bound rescales S once.  MODE 2
        // keeps a per-q lazy shift M[q].
        constexpr bool TENS = TQ > 0;
        double M[MODE == 2 ? QL : 1], S[QL], mx[TENS ? 1 : QL];
#pragma unroll
        for (int k = 0; k < QL; ++k) S[k] = 0.0;
#pragma unroll
        for (int k = 0; k < (TENS ? 1 : QL); ++k) mx[k] = -CUDART_INF;
#pragma unroll
        for (int k = 0; k < (MODE == 2 ? QL : 1); ++k) M[k] = -CUDART_INF;
        double Munit = -CUDART_INF;
        double dqmax = 0.0;
        for (int q = 0; q < nql; ++q) {
            const double *dq = sm.qd[qoff + q];
            dqmax = fmax(dqmax, dq[0] * dq[0] + dq[1] * dq[1] + dq[2] * dq[2]);
        }
        dqmax = sqrt(dqmax);
        double npairs = 0.0;
        double lb_run = -CUDART_INF;  // largest lower bound of the candidates so far
        const double sr = a.s * a.cull;
        for (int64_t k = k0; k < k1;) {
            const int nt = stage_chunk<DIM>(sm, f, k0, k, k1, bc, rcull2);
            const int nstg = sm.nstg;
            if (valid) {
                double bmax, lb;
                const int ncand = compact_candidates<DIM, TQ>(sm, wp, lane, nstg, cc, a, gh, bmax, lb);
                npairs += (double)ncand * nql;
                if (MODE != 2 && bmax > -CUDART_INF) {
                    const double mnew = bmax + sr * dqmax;
                    if (mnew > Munit) {
                        if (Munit > -CUDART_INF) {
                            const double sc = exp2_16(Munit - mnew, sm.tab);
#pragma unroll
                            for (int q = 0; q < QL; ++q) {
                                S[q] *= sc;
                                if (!TENS) mx[TENS ? 0 : q] += Munit - mnew;
                            }
                        }
                        Munit = mnew;
                    }
                }
                if constexpr (TENS) {
                    if (lb > lb_run) lb_run = lb;
                    if (lane == 0) sm.nnear[wp] = 0;
                    __syncwarp();
                    // the bounds' rounding: a few ulp of the exponents, far below 1e-12 of their range
                    const double lbr = lb_run - Munit;
                    value_pairs_tensor<DIM, TQ, TS, !FP32B>(sm, wp, lane, ncand, ah, cc, a, Munit,
                                                    lbr - 1e-12 * (fabs(lb_run) + fabs(Munit)), S);
                    __syncwarp();
                    near_maxima<DIM, QL>(sm, wp, lane, ncand, qoff, cc, a, mx[0]);
                } else if (nql == QL)
                    value_pairs<DIM, QL, QL, MODE>(sm, wp, lane, ncand, qoff, cc[0], cc[1], cc[2], a, Munit, M, S, mx);
                else
                    value_pairs_partial<DIM, QL, MODE>(sm, wp, lane, ncand, qoff, nql, cc[0], cc[1], cc[2], a, Munit,
                                                       M, S, mx);
            }
            k += nt;
            if (k >= k1) {
                tail_off = (int)(k - nt - k0);  // kept staged for the gradient sweep
                tail_nt = nt;
            } else {
                __syncthreads();  // the next chunk overwrites the staged targets
            }
        }
        // the lanes' sums and maxima of each q, to shared memory
        if (valid) {
            if constexpr (TENS) {
                double last;
                const double tot = lane_totals<QL>(S, lane, last);
                constexpr int EP = 32 / QL;
                double m = mx[0];
#pragma unroll
                for (int e = 1; e < EP; ++e) m = fmax(m, __shfl_down_sync(0xffffffffu, mx[0], e * QL));
                constexpr int LPQ = QL == 4 ? 8 : 4;   // lanes that hold a total
                if (lane % LPQ == 0) sm.qS[qoff + lane / LPQ] = tot;
                if (QL == 9 && lane == 0) sm.qS[qoff + QL - 1] = last;
                if (lane < QL) {
                    sm.qm[qoff + lane] = m;
                    sm.qU[qoff + lane] = Munit;
                }
            } else {
#pragma unroll
                for (int q = 0; q < QL; ++q) {
                    const double mxw = warp_max(mx[TENS ? 0 : q]);
                    // shift of this lane's sum: Munit (exponents relative to it: 0) or the lazy M[q]
                    const double Ml = MODE == 2 ? M[MODE == 2 ? q : 0] : (Munit > -CUDART_INF ? 0.0 : -CUDART_INF);
                    const double sl =
                        (Ml == -CUDART_INF || mxw == -CUDART_INF) ? 0.0 : S[q] * exp2_16(Ml - mxw, sm.tab);
                    const double Sw = warp_sum(sl);
                    if (lane == 0 && q < nql) {
                        const double m = MODE == 2 ? mxw : mxw + Munit;
                        sm.qS[qoff + q] = Sw;
                        sm.qm[qoff + q] = m;
                        sm.qU[qoff + q] = m;   // the sum is relative to the maximum
                    }
                }
            }
        }
        __syncthreads();
        // the points' epilogues, thread <-> point of the block: one or three warps run the logarithms instead of
        // every warp for the eight or nine lanes of its unit
        double tv = 0.0, tcv = 0.0, tsk = 0.0;
        if (tid < nqb) {
            const int64_t qg = qblk0 + tid;
            const double m = sm.qm[tid], U = sm.qU[tid];
            const double Sr =
                (m == -CUDART_INF || U == -CUDART_INF) ? 0.0 : sm.qS[tid] * (TENS ? exp2_factor<!FP32B>(U - m, sm.tab) : 1.0);
            double L;
            int sk;
            value_epilogue(a, m, Sr, sm.qd[tid][3], f.rho[qg], f.jxw[qg], tv, tcv, L, sk);
            f.Lq[qg] = L;
            sm.qL[tid] = L;
            tsk = sk;
        }
        block_partials_at(tv, tcv, tsk, lane == 0 ? npairs : 0.0, f.valpart + (int64_t)b * 4);  // contains __syncthreads
    }

    // ---------------- gradient sweep ----------------
    // per-unit reference L_Kref = min L over the unit's q; per-q data
    if (tid < nqb) {
        const int i = tid, c = i / a.qpc, gr = (i - c * a.qpc) / a.ql;
        const int u0 = c * a.qpc + gr * a.ql, un = min(a.ql, a.qpc - gr * a.ql);
        double Lr = CUDART_INF;
        for (int q = 0; q < un; ++q) Lr = fmin(Lr, sm.qL[u0 + q]);
        if (i == u0) sm.uL[c * a.ngroups + gr] = Lr;
        const double L = sm.qL[i];
        const double D = (!isfinite(Lr) || !isfinite(L)) ? -CUDART_INF
                                                         : (sm.qd[i][3] - KAPPA * (L - Lr)) * (1.0 / 16.0);
        const double wq = f.w[qblk0 + i];
        using Row = typename PRow<FP32B>::T;
        if (FP32B && TQ == 0) {
            sm.qb[i][0] = (float)sm.qd[i][0];
            sm.qb[i][1] = (float)sm.qd[i][1];
            sm.qb[i][2] = (float)sm.qd[i][2];
            sm.qb[i][3] = (float)(f.w_nonneg ? D + log2(wq) : D);  // w_q folded in: p = 2^e directly
        }
        sm.qw[i] = (Row)wq;
        if (TQ > 0) sm.qtw[i] = (Row)(wq * exp2(D));
    }
    __syncthreads();
    // The value sweep's last chunk (the only one when everything fit) is still
    // staged: its gradient comes first, then the earlier entries' (tensor-product
    // points: unstaged; otherwise the earlier chunks are staged again, the same
    // ones: the greedy rule over [k0, k0 + tail_off) ends where the value sweep's
    // did).  Every pair's partial is written once, so the order does not change
    // any sum.
    int64_t kend = k1;
    if (tail_off >= 0) {
        grad_chunk<DIM, FP32B, TQ, TS>(sm, f, k0 + tail_off, tail_nt, nunit, a);
        kend = k0 + tail_off;
    }
    if constexpr (TQ > 0) {
        if (kend == k0) return;
        if (wp == 0) direct_setup<DIM>(sm, lane, nunit, bc);
        __syncthreads();
        // The FP32 squared distance about the block centre is off by less than
        // 1.4e-6 rc^2 (components up to 2 rc, rounded three times).
        grad_direct<DIM, TQ, FP32B, TS>(sm, f, k0, kend, nunit, bc, (float)(a.sstar - 4e-6 * rc * rc),
                                        (float)(a.sstar + 4e-6 * rc * rc), a);
    } else {
        for (int64_t k = k0; k < kend;) {
            __syncthreads();  // the staged targets are consumed
            const int nt = stage_chunk<DIM>(sm, f, k0, k, kend, bc, rcull2);
            grad_chunk<DIM, FP32B, TQ, TS>(sm, f, k, nt, nunit, a);
            k += nt;
        }
    }
}

// gradient of target block t = sum of its pair partials in inverse order
// (ascending source block), lane <-> target.  CTA <-> target block: warp w
// sums entries w, w + 8, ... (the positions of 32 of them fetched at once,
// eight partials in flight: with a position fetched per partial it took 316 us
// for 2.8 million pairs); the 8 warp sums are added in warp order.  Of the pairs at forward positions [k0, k1) only (one
// launch's source blocks; a target's positions ascend), added to gacc after
// the first launch.
template <typename PT>
__global__ void __launch_bounds__(256)
k_grad_reduce(const int64_t *__restrict__ tblk_off, const int64_t *__restrict__ inv_off,
              const int64_t *__restrict__ inv_k, int64_t k0, int64_t k1, int add, const PT *__restrict__ part,
              double *__restrict__ gacc)
{
    __shared__ double ws[8][32];
    const int t = blockIdx.x;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    int64_t p0 = inv_off[t], p1 = inv_off[t + 1];
    if (add || (p1 > p0 && inv_k[p1 - 1] >= k1)) {  // a part of the list: binary searches for its ends
        auto first = [&](int64_t k) {
            int64_t lo = p0, hi = p1;
            while (lo < hi) {
                const int64_t m = (lo + hi) >> 1;
                if (inv_k[m] < k) lo = m + 1;
                else hi = m;
            }
            return lo;
        };
        const int64_t a = first(k0), b = first(k1);
        p0 = a;
        p1 = b;
    }
    double acc = 0.0;
    for (int64_t p = p0 + w; p < p1; p += 256) {
        const int64_t mine = p + 8 * lane < p1 ? inv_k[p + 8 * lane] - k0 : 0;
        const int n = (int)min((int64_t)32, (p1 - p + 7) / 8);
        for (int u0 = 0; u0 < n; u0 += 8) {
            PT v[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                const int64_t k = __shfl_sync(0xffffffffu, mine, u0 + u);
                v[u] = u0 + u < n ? part[k * TBLK_KD + lane] : PT(0);
            }
#pragma unroll
            for (int u = 0; u < 8; ++u)
                if (u0 + u < n) acc += (double)v[u];
        }
    }
    ws[w][lane] = acc;
    __syncthreads();
    if (w == 0) {
        double s = 0.0;
#pragma unroll
        for (int i = 0; i < 8; ++i) s += ws[i][lane];
        const int64_t j = tblk_off[t] + lane;
        if (j < tblk_off[t + 1]) gacc[j] = add ? gacc[j] + s : s;
    }
}

template <int DIM, int QL, bool FP32B, int MODE, int TQ, int TS>
static void launch_fused(sdot_ctx *c, const FusedArgs &f, const EvalArgs &a, size_t smem, int nb)
{
    cudaFuncSetAttribute(k_fused<DIM, QL, FP32B, MODE, TQ, TS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    cudaFuncSetAttribute(k_fused<DIM, QL, FP32B, MODE, TQ, TS>, cudaFuncAttributePreferredSharedMemoryCarveout,
                         (int)cudaSharedmemCarveoutMaxShared);
    k_fused<DIM, QL, FP32B, MODE, TQ, TS><<<(unsigned)nb, FT_WARPS * 32, smem, c->stream>>>(f, a);
}

template <int DIM, int QL, int MODE, int TQ = 0, int TS = 0>
static void dispatch_fused_b(sdot_ctx *c, const FusedArgs &f, const EvalArgs &a, bool fp32b, int nb)
{
    if (fp32b) launch_fused<DIM, QL, true, MODE, TQ, TS>(c, f, a, sizeof(FTSmem<fused_cap(TQ), float>), nb);
    else launch_fused<DIM, QL, false, MODE, TQ, TS>(c, f, a, sizeof(FTSmem<fused_cap(TQ), double>), nb);
}

template <int DIM, int MODE>
static void dispatch_fused_q(sdot_ctx *c, const FusedArgs &f, const EvalArgs &a, bool fp32b, int nb)
{
    // 2D: units of 4 (order 2) or 9 (order 3 and groups of 9); 3D: 8 or 9.
    if constexpr (DIM == 2) {
        if (a.ql <= 4) dispatch_fused_b<DIM, 4, MODE>(c, f, a, fp32b, nb);
        else dispatch_fused_b<DIM, 9, MODE>(c, f, a, fp32b, nb);
    } else {
        if (a.ql <= 8) dispatch_fused_b<DIM, 8, MODE>(c, f, a, fp32b, nb);
        else dispatch_fused_b<DIM, 9, MODE>(c, f, a, fp32b, nb);
    }
}

// MODE selection.  The shift Munit may exceed the true maximum exponent of a
// q by up to 2 s r |delta|max (units of 2^(1/16)); beyond 2^500 the lazy form
// is used.  Exponents u relative to Munit satisfy
// u >= -s (psi_max - psi_min + r^2/2 + 2 r |delta|max); when that is above
// -16000 the clamp of exp2 is provably inactive and dropped.
//
// Tensor form of the sweeps (tensor-product points with an instantiation):
// -1 none (per-point sweeps), 0 symmetric factors 2^(+-G a), 1 factors
// relative to the lowest point.
static int fused_tensor_mode(const sdot_ctx *c, const EvalArgs &a, double psi_range)
{
    const double gap = 2.0 * a.s * a.cull * c->delta_max;
    const double umin = -a.s * (psi_range + 0.5 * a.cull * a.cull + 2.0 * a.cull * c->delta_max);
    // tensor-product points: per-dimension factors 2^(+-G a/16) stay within
    // 2^300 (FP64 value sweep) and 2^40 (FP32 gradient sweep)
    const double fac = a.s * a.cull * c->tensor_amax / 16.0;
    const bool tensor = c->tensor_m > 0 && a.lse && a.ngroups == 1 && fac <= 40.0 && umin > -15000.0 &&
                        gap < 16.0 * 500.0 && a.cull > 1e-12 && a.cull < 1e12;  // (FP32 squared distances)
    const bool shape = (c->dim == 3 && c->tensor_m == 2 && a.ql == 8) ||
                       (c->dim == 2 && c->tensor_m == 3 && a.ql == 9) || (c->dim == 2 && c->tensor_m == 2 && a.ql == 4);
    if (!tensor || !shape) return -1;
    // factors <= 2^8 per dimension: the relative form (no reciprocals, the lowest point's factor 1)
    return fac > 4.0 ? 0 : 1;
}

template <int DIM>
static void dispatch_fused(sdot_ctx *c, const FusedArgs &f, const EvalArgs &a, bool fp32b, int nb, double psi_range,
                           int tmode)
{
    const double gap = 2.0 * a.s * a.cull * c->delta_max;
    const double umin = -a.s * (psi_range + 0.5 * a.cull * a.cull + 2.0 * a.cull * c->delta_max);
    if (gap >= 16.0 * 500.0) {
        dispatch_fused_q<DIM, 2>(c, f, a, fp32b, nb);
        return;
    }
    if (tmode >= 0) {
        if constexpr (DIM == 3) {
            if (tmode == 1) dispatch_fused_b<3, 8, 0, 2, 1>(c, f, a, fp32b, nb);
            else dispatch_fused_b<3, 8, 0, 2, 0>(c, f, a, fp32b, nb);
        } else if (c->tensor_m == 3) {
            if (tmode == 1) dispatch_fused_b<2, 9, 0, 3, 1>(c, f, a, fp32b, nb);
            else dispatch_fused_b<2, 9, 0, 3, 0>(c, f, a, fp32b, nb);
        } else {
            if (tmode == 1) dispatch_fused_b<2, 4, 0, 2, 1>(c, f, a, fp32b, nb);
            else dispatch_fused_b<2, 4, 0, 2, 0>(c, f, a, fp32b, nb);
        }
        return;
    }
    if (umin > -15000.0) dispatch_fused_q<DIM, 0>(c, f, a, fp32b, nb);
    else dispatch_fused_q<DIM, 1>(c, f, a, fp32b, nb);
}

sdot_status run_trunc(sdot_ctx *c, const EvalArgs &a, double r)
{
    cudaStream_t st = c->stream;
    // 1. block-pair structure (conservative FP32 test)
    const float cr = (float)(std::min(r, 1e30) * (1.0 + 1e-6) + 1e-6 * c->coord_scale);
    const int nsb = (int)c->nsblk, ntb = (int)c->ntblk;
    const int nss = (nsb + SUPER - 1) / SUPER, nts = (ntb + SUPER - 1) / SUPER;
    cudaError_t e = c->fwd_cnt.alloc(nsb + 1);
    if (e == cudaSuccess) e = c->fwd_off.alloc(nsb + 1);
    if (e == cudaSuccess) e = c->superpair.alloc((size_t)nss * nts);
    if (e == cudaSuccess) e = c->shit.alloc((size_t)nss * nts);
    if (e == cudaSuccess) e = c->scount.alloc(nss + 1);
    if (e == cudaSuccess) e = c->fwd_hist.alloc(ORDER_BUCKETS);
    if (e == cudaSuccess) e = c->fwd_order.alloc(nsb);
    if (e != cudaSuccess) return cuda_error(c, e, "pair list alloc");
    k_super_pairs<<<(unsigned)(((int64_t)nss * nts + 255) / 256), 256, 0, st>>>(c->ssup_sph32.p, nss, c->tsup_sph32.p,
                                                                             nts, cr, c->superpair.p);
    k_super_compact<<<(unsigned)(((int64_t)nss * 32 + 255) / 256), 256, 0, st>>>(c->superpair.p, nss, nts, c->shit.p,
                                                                              c->scount.p, c->fwd_hist.p);
    // Row length of the per-block pair masks: the most target super-blocks any
    // source super-block pairs with.  Every count is at most nts, so when the
    // nts-wide rows are small (<= 64 MiB) they are used as
    // they are and the counts are not read back (one host round trip fewer).
    int hmax = std::max(1, nts);
    if ((size_t)nsb * (size_t)nts * sizeof(int) > ((size_t)64 << 20)) {
        std::vector<int> sc((size_t)nss);
        e = cudaMemcpyAsync(sc.data(), c->scount.p, nss * sizeof(int), cudaMemcpyDeviceToHost, st);
        if (e == cudaSuccess) e = cudaStreamSynchronize(st);
        if (e != cudaSuccess) return cuda_error(c, e, "pair list count");
        hmax = 1;
        for (int v : sc) hmax = std::max(hmax, v);
    }
    e = c->pmask.alloc((size_t)nsb * hmax);
    if (e != cudaSuccess) return cuda_error(c, e, "pair mask alloc");
    const unsigned gw = (unsigned)(((int64_t)nsb * 32 + 255) / 256);
    const unsigned gm = (unsigned)(((int64_t)((nsb + FM_B - 1) / FM_B) * 32 + 255) / 256);
    k_fwd_masks<<<gm, 256, 0, st>>>(c->sblk_box32.p, nsb, c->tblk_box32.p, ntb, nts, hmax, cr, c->shit.p, c->scount.p,
                                    c->pmask.p, c->fwd_cnt.p, c->fwd_hist.p);
    k_scan<<<1, 1024, 0, st>>>(c->fwd_cnt.p, nsb, c->fwd_off.p, c->scal_host + SC_COVER, c->fwd_hist.p);
    e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) return cuda_error(c, e, "pair list count");
    const int64_t npairs = (int64_t)c->scal_host[SC_COVER];  // (a whole number below 2^53)
    e = c->fwd_t.alloc(npairs + 1);
    if (e == cudaSuccess) e = c->inv_b.alloc(npairs + 1);
    if (e == cudaSuccess) e = c->inv_k.alloc(npairs + 1);
    if (e == cudaSuccess) e = c->inv_tmpb.alloc(npairs + 1);
    if (e == cudaSuccess) e = c->inv_tmpk.alloc(npairs + 1);
    if (e == cudaSuccess) e = c->inv_cnt.alloc(2 * (size_t)(ntb + 1));
    if (e == cudaSuccess) e = c->inv_off.alloc(ntb + 1);
    if (e != cudaSuccess) return cuda_error(c, e, "pair list alloc");
    k_fwd_fill<<<gw, 256, 0, st>>>(nsb, nts, hmax, c->shit.p, c->scount.p, c->pmask.p, c->fwd_off.p, c->fwd_t.p, ntb,
                                   c->fwd_hist.p, c->fwd_order.p);
    c->klaunch[6] += 9;
    if (c->profiling) cudaEventRecord(c->pev[7], st);
    // 2. partial buffer (forward order): all pairs at once under the cap, else groups of source blocks.
    // Partials are FP32 in the hybrid mode (the sweeps' rows are FP32), FP64 otherwise.
    const bool fp32b = c->precision != SDOT_PREC_FP64;
    const size_t pel = fp32b ? sizeof(float) : sizeof(double);
    const int64_t cap_pairs = std::max<int64_t>(1, (int64_t)(c->part_cap_bytes / (TBLK_KD * pel)));
    struct Group {
        int b0, b1;
        int64_t k0, k1;
    };
    std::vector<Group> groups;
    int64_t part_pairs = npairs;
    if (npairs <= cap_pairs) {
        groups.push_back({0, nsb, 0, npairs});
    } else {
        std::vector<int64_t> off((size_t)nsb + 1);
        e = cudaMemcpyAsync(off.data(), c->fwd_off.p, (nsb + 1) * sizeof(int64_t), cudaMemcpyDeviceToHost, st);
        if (e == cudaSuccess) e = cudaStreamSynchronize(st);
        if (e != cudaSuccess) return cuda_error(c, e, "pair list copy");
        part_pairs = 0;
        int b0 = 0;
        while (b0 < nsb) {
            int b1 = b0 + 1;
            while (b1 < nsb && off[b1 + 1] - off[b0] <= cap_pairs) ++b1;
            groups.push_back({b0, b1, off[b0], off[b1]});
            part_pairs = std::max(part_pairs, off[b1] - off[b0]);
            b0 = b1;
        }
    }
    e = c->part.alloc(((size_t)std::max<int64_t>(1, part_pairs) * TBLK_KD * pel + sizeof(double) - 1) / sizeof(double));
    if (e != cudaSuccess) return cuda_error(c, e, "partial buffer alloc");
    // the inverse lists, on the second stream: k_fused needs the forward lists only
    e = cudaEventRecord(c->fork, st);
    if (e == cudaSuccess) e = cudaStreamWaitEvent(c->side, c->fork, 0);
    if (e == cudaSuccess) e = cudaMemsetAsync(c->inv_cnt.p, 0, 2 * (ntb + 1) * sizeof(int64_t), c->side);
    if (e != cudaSuccess) return cuda_error(c, e, "pair list fork");
    unsigned long long *icnt = reinterpret_cast<unsigned long long *>(c->inv_cnt.p), *ifill = icnt + ntb + 1;
    k_inv_count<<<gw, 256, 0, c->side>>>(nsb, c->fwd_off.p, c->fwd_t.p, icnt);
    k_scan<<<1, 1024, 0, c->side>>>(c->inv_cnt.p, ntb, c->inv_off.p, nullptr, nullptr);
    k_inv_scatter<<<gw, 256, 0, c->side>>>(nsb, c->fwd_off.p, c->fwd_t.p, c->inv_off.p, ifill, c->inv_tmpb.p,
                                           c->inv_tmpk.p);
    k_inv_order<<<(unsigned)ntb, 256, 0, c->side>>>(nsb, c->inv_off.p, c->inv_tmpb.p, c->inv_tmpk.p, c->inv_b.p,
                                                    c->inv_k.p);
    e = cudaEventRecord(c->join, c->side);
    if (e != cudaSuccess) return cuda_error(c, e, "pair list join");
    FusedArgs f{};
    f.x = c->x.p; f.rho = c->rho.p; f.jxw = c->jxw.p; f.w = c->w.p; f.cell_ctr = c->cell_ctr.p;
    f.tpk = c->tpack.p; f.nt = c->nt; f.sblk_cell = c->sblk_cell.p; f.sblk_sph = c->sblk_sph.p; f.tblk_off = c->tblk_off.p;
    f.fwd_off = c->fwd_off.p; f.fwd_t = c->fwd_t.p;
    f.part = c->part.p; f.part32 = reinterpret_cast<float *>(c->part.p); f.Lq = c->Lq.p; f.valpart = c->blkpart.p;
    f.cullt = std::isnan(r) ? 0.0 : std::min(r, 1e300);
    f.w_nonneg = c->w_nonneg ? 1 : 0;
    const double prange0 = c->scal_host[SC_MAXPSI] - c->scal_host[SC_MINPSI];
    const double prange = std::isfinite(prange0) ? prange0 : 1e300;
    const int tmode = fused_tensor_mode(c, a, prange);
    for (size_t gi = 0; gi < groups.size(); ++gi) {
        const Group &g = groups[gi];
        f.order = groups.size() == 1 ? c->fwd_order.p : nullptr;
        f.b0 = g.b0;
        f.part_base = g.k0;
        if (c->dim == 2) dispatch_fused<2>(c, f, a, fp32b, g.b1 - g.b0, prange, tmode);
        else dispatch_fused<3>(c, f, a, fp32b, g.b1 - g.b0, prange, tmode);
        if (c->profiling && gi + 1 == groups.size()) cudaEventRecord(c->pev[2], st);
        if (gi == 0) {
            e = cudaStreamWaitEvent(st, c->join, 0);
            if (e != cudaSuccess) return cuda_error(c, e, "pair list join");
        }
        if (fp32b)
            k_grad_reduce<float><<<(unsigned)ntb, 256, 0, st>>>(c->tblk_off.p, c->inv_off.p, c->inv_k.p, g.k0, g.k1,
                                                                gi > 0, f.part32, c->gpart.p);
        else
            k_grad_reduce<double><<<(unsigned)ntb, 256, 0, st>>>(c->tblk_off.p, c->inv_off.p, c->inv_k.p, g.k0, g.k1,
                                                                 gi > 0, c->part.p, c->gpart.p);
        c->klaunch[2] += 1;
        c->klaunch[3] += 1;
    }
    if (c->profiling) cudaEventRecord(c->pev[3], st);
    return cuda_error(c, cudaGetLastError(), "truncated evaluation");
}

}  // namespace sdot
