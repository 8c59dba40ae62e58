// sdot_lattice_host.h -- host side of the lattice sweeps (sdot_lattice.cuh):
// detection of a tensor lattice in a point set, and the tile and slice counts.
#pragma once

#include <math.h>
#include <stdint.h>
#include <string.h>

#include <algorithm>
#include <vector>

namespace sdot {

// A point set that is a tensor lattice: dimension d has n[d] coordinates
// X[xo[d]..], ascending, and q[i0 + n0 (i1 + n1 i2)] is the point at them.
struct Lattice {
    bool ok = false;
    int n[3] = {1, 1, 1}, xo[3] = {0, 0, 0};
    // period[d] > 0: X[i + period] = X[i] + step in dimension d (uniform cells of `period` Gauss points)
    int period[3] = {0, 0, 0};
    double step[3] = {0.0, 0.0, 0.0};
    std::vector<double> X;
    std::vector<int> q;
};
constexpr int LAT_MAXP = 4;   // largest period looked for
constexpr int LAT_RUN = 8;    // points of a factor run

constexpr double LAT_ULPS = 4.0 * 2.220446049250313e-16;

// Finds the lattice, or leaves ok = false.  Coordinates are told apart by
// their bits; where that leaves more coordinates than the lattice can have,
// those within LAT_ULPS of the points' extent are taken as one (meshes that
// map each cell by itself round a shared coordinate in the last bits).  The
// sweeps form the exponents about the source's centre, so their own rounding
// goes by the extent, and so has what merged coordinates and a run's equal
// steps (below) add.  Far from the origin, where coordinates are rounded more
// coarsely than that, a source is a lattice only if its coordinates agree in
// their bits.  Linear in the points; gives up as soon as a dimension has more
// coordinates than MAXN.
inline void find_lattice(const double *x, int64_t n, int dim, Lattice &L)
{
    constexpr int MAXN = 4096, BITS = 13, CAP = 1 << BITS;
    L = Lattice();
    if (n < 4 || n > INT32_MAX) return;
    struct Table {
        uint64_t key[CAP];
        short id[CAP];
    };
    auto bits = [](double v) {
        v = v == 0.0 ? 0.0 : v;
        uint64_t k;
        memcpy(&k, &v, 8);
        return k;
    };
    // coordinate of every point per dimension, numbered in order of appearance (stripes of points that share
    // the previous three points' coordinates, as within a cell, need no search)
    std::vector<double> val[3];
    std::vector<short> num((size_t)n * dim);
    {
        std::vector<Table> table(1);
        Table &t = table[0];
        for (int d = 0; d < dim; ++d) {
            memset(t.id, 0xff, sizeof t.id);
            uint64_t lk[4] = {0, 0, 0, 0};
            short li[4] = {-1, -1, -1, -1};
            int w = 0;
            for (int64_t i = 0; i < n; ++i) {
                const uint64_t k = bits(x[i * dim + d]);
                short id = -1;
                for (int m = 0; m < 4; ++m)
                    if (li[m] >= 0 && lk[m] == k) id = li[m];
                if (id < 0) {
                    uint64_t h = (k * 0x9e3779b97f4a7c15ull) >> (64 - BITS);
                    while (t.id[h] >= 0 && t.key[h] != k) h = (h + 1) & (CAP - 1);
                    id = t.id[h];
                    if (id < 0) {
                        if ((int)val[d].size() >= MAXN) return;
                        id = (short)val[d].size();
                        t.key[h] = k;
                        t.id[h] = id;
                        val[d].push_back(x[i * dim + d]);
                    }
                    lk[w] = k;
                    li[w] = id;
                    w = (w + 1) & 3;
                }
                num[(size_t)i * dim + d] = id;
            }
            // no lattice of n points has this many coordinates in the dimensions seen so far
            double most = 1.0;
            for (int e = 0; e <= d; ++e) most *= (double)val[e].size() / 4.0;
            if (most > (double)n) return;
        }
    }
    std::vector<int> rank[3];
    std::vector<double> coord[3];
    for (int merge = 0; merge < 2; ++merge) {
        int64_t total = 1;
        for (int d = 0; d < dim; ++d) {
            const int m = (int)val[d].size();
            std::vector<int> ord(m);
            for (int i = 0; i < m; ++i) ord[i] = i;
            std::sort(ord.begin(), ord.end(), [&](int a, int b) { return val[d][a] < val[d][b]; });
            const double tol = merge ? LAT_ULPS * (val[d][ord[m - 1]] - val[d][ord[0]]) : -1.0;
            rank[d].assign(m, 0);
            coord[d].clear();
            for (int i = 0; i < m; ++i) {
                const double v = val[d][ord[i]];
                if (coord[d].empty() || v - coord[d].back() > tol) coord[d].push_back(v);
                rank[d][ord[i]] = (int)coord[d].size() - 1;
            }
            total *= (int64_t)coord[d].size();
        }
        if (total == n) break;
        if (merge || total < n) return;
    }
    std::vector<int> q((size_t)n, -1);
    int64_t stride = 1;
    for (int d = 0; d < dim; ++d) {  // ranks to lattice strides
        for (int &r : rank[d]) r = (int)(r * stride);
        stride *= (int64_t)coord[d].size();
    }
    for (int64_t i = 0; i < n; ++i) {
        int64_t li = 0;
        for (int d = 0; d < dim; ++d) li += rank[d][num[(size_t)i * dim + d]];
        if (q[li] >= 0) return;  // two points at one place: no lattice
        q[li] = (int)i;
    }
    int o = 0;
    for (int d = 0; d < dim; ++d) {
        L.n[d] = (int)coord[d].size();
        L.xo[d] = o;
        o += L.n[d];
        L.X.insert(L.X.end(), coord[d].begin(), coord[d].end());
        const std::vector<double> &c = coord[d];
        const double tol = LAT_ULPS * (c.back() - c.front());
        for (int p = 1; p <= LAT_MAXP && L.period[d] == 0 && 2 * p <= L.n[d]; ++p) {
            const int cells = (L.n[d] - 1) / p;
            const double h = (c[cells * p] - c[0]) / cells;
            // every point of every run of LAT_RUN from its first one: the steps' differences add up along a run
            bool same = true;
            for (int i = 0; i + p < L.n[d] && same; ++i)
                for (int k = 1; k < LAT_RUN && i + k * p < L.n[d] && same; ++k)
                    same = fabs(c[i + k * p] - c[i] - k * h) <= tol;
            if (same) {
                L.period[d] = p;
                L.step[d] = h;
            }
        }
    }
    L.q.swap(q);
    L.ok = true;
}

// Tiles of one evaluation: points per dimension of a tile (0: the lattice
// sweeps do not apply) and tile counts.
struct LatTiling {
    int cap = 0, nt[3] = {1, 1, 1}, ntiles = 0;
    double span = 0.0, span0 = 0.0;   // the factors of a tile lie within 2^(+-span), dimension 0's within 2^(+-span0)
    double slope0 = 0.0;              // bits per length of dimension 0's factors
};

// The largest span that the sweeps admit, and the bits between a clamped term
// and the least sum that they leave (sdot_lattice.cuh says why).
constexpr double LAT_BITS = 350.0;
constexpr double LAT_CLAMP_LEFT = 300.0;

constexpr int LAT_CAPS2[2] = {64, 32}, LAT_CAPS3[1] = {16};   // tile sizes (2D, 3D), the largest first

// Tiles of cap points per dimension; false where their padding excludes the
// size.  A tile's work goes by its padded size (64 or 32 points per dimension,
// 16 in 3D); where that would be more than LAT_PAD times the points, the cell
// sweeps (about four multiply-adds per pair against one here, plus a third for
// the factors) are the faster ones.
constexpr double LAT_PAD = 2.5;
inline bool lat_tiles(const int *n, int dim, int cap, LatTiling &t)
{
    int64_t tiles = 1, nq = 1;
    double padded = 1.0;
    for (int d = 0; d < dim; ++d) {
        t.nt[d] = (n[d] + cap - 1) / cap;
        tiles *= t.nt[d];
        nq *= n[d];
        const int rest = n[d] - (t.nt[d] - 1) * cap;
        padded *= (t.nt[d] - 1) * (double)cap + (dim == 2 && rest <= 32 ? 32 : cap);
    }
    if (padded > LAT_PAD * (double)nq || tiles > (1 << 20)) return false;
    t.cap = cap;
    t.ntiles = (int)tiles;
    return true;
}

// Tile size for scaled exponents s = kappa / eps and targets within reach[d]
// of the origin: the largest of 64 and 32 points per dimension (2D) or 16
// (3D) whose factors span at most 2^(+-LAT_BITS).
inline LatTiling lat_tiling(const int *n, const int *xo, const double *X, int dim, double s, const double *reach)
{
    for (int k = 0; k < (dim == 2 ? 2 : 1); ++k) {
        const int cap = dim == 2 ? LAT_CAPS2[k] : LAT_CAPS3[k];
        LatTiling t;
        if (!lat_tiles(n, dim, cap, t)) continue;
        for (int d = 0; d < dim; ++d) {
            double h = 0.0;
            for (int i = 0; i < t.nt[d]; ++i) {
                const int a = i * cap, b = std::min(n[d], a + cap) - 1;
                h = std::max(h, 0.5 * (X[xo[d] + b] - X[xo[d] + a]));
            }
            t.span += s * reach[d] * h / 16.0;
            if (d == 0) t.span0 = t.span;
        }
        t.slope0 = s * reach[0] / 16.0;
        if (t.span <= LAT_BITS) return t;
    }
    return LatTiling();
}

// The fewest and the most tiles that lat_tiling may return at any s and reach (0: never any).
struct LatTileRange {
    int fewest = 0, most = 0;
};
inline LatTileRange lat_tile_range(const int *n, int dim)
{
    LatTileRange r;
    for (int k = 0; k < (dim == 2 ? 2 : 1); ++k) {
        LatTiling t;
        if (!lat_tiles(n, dim, dim == 2 ? LAT_CAPS2[k] : LAT_CAPS3[k], t)) continue;
        r.fewest = r.most == 0 ? t.ntiles : std::min(r.fewest, t.ntiles);
        r.most = std::max(r.most, t.ntiles);
    }
    return r;
}

// Slices of n items (targets, tiles) over `units` independent work items so
// that units x slices CTAs fill whole waves of `slots` resident CTAs: the
// fewest slices that leave less than a tenth of the last wave idle, at most
// maxs.
inline int lat_slices(int64_t units, int64_t maxs, int slots)
{
    if (units <= 0 || maxs <= 1) return 1;
    int best = 1;
    double beff = 0.0;
    for (int64_t w = 1; w <= 8; ++w) {
        const int64_t s = std::min<int64_t>(maxs, w * slots / units);
        if (s < 1) continue;
        const int64_t waves = (units * s + slots - 1) / slots;
        const double eff = (double)(units * s) / (double)(waves * slots);
        if (eff > beff + 1e-9) {
            beff = eff;
            best = (int)s;
        }
        if (beff >= 0.9 || s == maxs) break;
    }
    return best;
}

}  // namespace sdot
