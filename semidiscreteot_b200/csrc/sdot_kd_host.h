// sdot_kd_host.h -- k-d tree order and bounding spheres of point sets (host).
#pragma once

#include <float.h>
#include <math.h>
#include <stdint.h>

#include <algorithm>
#include <cmath>
#include <numeric>
#include <vector>

namespace sdot {

// k-d tree order of n points: recursive split at the balanced position along
// the widest axis until a node holds at most `leaf` points.  Returns the
// point order and the leaf boundaries (DFS order, spatially coherent).
inline void kd_split(const std::vector<double> &pts, int dim, std::vector<int64_t> &idx, int64_t a, int64_t b, int64_t leaf,
              std::vector<int64_t> &bounds)
{
    const int64_t count = b - a;
    if (count <= leaf) {
        bounds.push_back(a);
        return;
    }
    double lo[3] = {DBL_MAX, DBL_MAX, DBL_MAX}, hi[3] = {-DBL_MAX, -DBL_MAX, -DBL_MAX};
    for (int64_t i = a; i < b; ++i)
        for (int d = 0; d < dim; ++d) {
            lo[d] = std::min(lo[d], pts[idx[i] * dim + d]);
            hi[d] = std::max(hi[d], pts[idx[i] * dim + d]);
        }
    int ax = 0;
    for (int d = 1; d < dim; ++d)
        if (hi[d] - lo[d] > hi[ax] - lo[ax]) ax = d;
    const int64_t nleaves = (count + leaf - 1) / leaf;
    const int64_t m = a + (nleaves / 2) * leaf;
    std::nth_element(idx.begin() + a, idx.begin() + m, idx.begin() + b, [&](int64_t u, int64_t v) {
        const double pu = pts[u * dim + ax], pv = pts[v * dim + ax];
        return pu < pv || (pu == pv && u < v);
    });
    kd_split(pts, dim, idx, a, m, leaf, bounds);
    kd_split(pts, dim, idx, m, b, leaf, bounds);
}

inline std::vector<int64_t> kd_order(const std::vector<double> &pts, int dim, int64_t n, int64_t leaf,
                              std::vector<int64_t> &bounds)
{
    std::vector<int64_t> idx(n);
    std::iota(idx.begin(), idx.end(), 0);
    bounds.clear();
    kd_split(pts, dim, idx, 0, n, leaf, bounds);
    bounds.push_back(n);
    return idx;
}

// Bounding sphere (bbox centre, max distance, enlarged by 1e-12 relative).
inline void sphere_of(const double *pts, const std::vector<int64_t> &idx, int dim, double *out)
{
    double lo[3] = {DBL_MAX, DBL_MAX, DBL_MAX}, hi[3] = {-DBL_MAX, -DBL_MAX, -DBL_MAX};
    for (int64_t i : idx)
        for (int d = 0; d < dim; ++d) {
            lo[d] = std::min(lo[d], pts[i * dim + d]);
            hi[d] = std::max(hi[d], pts[i * dim + d]);
        }
    double c[3] = {0, 0, 0};
    for (int d = 0; d < dim; ++d) c[d] = 0.5 * (lo[d] + hi[d]);
    double R = 0.0;
    for (int64_t i : idx) {
        double s = 0.0;
        for (int d = 0; d < dim; ++d) {
            const double t = pts[i * dim + d] - c[d];
            s += t * t;
        }
        R = std::max(R, std::sqrt(s));
    }
    out[0] = c[0];
    out[1] = c[1];
    out[2] = c[2];
    out[3] = R * (1.0 + 1e-12) + 1e-300;
}

}  // namespace sdot
