// sdot_kd_host.h -- k-d tree order and bounding spheres of point sets (host).
#pragma once

#include <float.h>
#include <math.h>
#include <stdint.h>

#include <algorithm>
#include <cmath>
#include <vector>

namespace sdot {

// k-d tree order of n points: recursive split at the balanced position along
// the widest axis until a node holds at most `leaf` points.  Returns the
// point order and the leaf boundaries (DFS order, spatially coherent).  The
// points move with their indices (with an index array alone every comparison is
// two scattered loads: 1.3 to 1.7 times as long at 60,000 to 290,000 points).
template <int DIM>
struct KdPoint {
    double x[DIM];
    int64_t id;
};

template <int DIM>
inline void kd_split(KdPoint<DIM> *p, int64_t a, int64_t b, int64_t leaf, std::vector<int64_t> &bounds)
{
    const int64_t count = b - a;
    if (count <= leaf) {
        bounds.push_back(a);
        return;
    }
    double lo[DIM], hi[DIM];
    for (int d = 0; d < DIM; ++d) lo[d] = hi[d] = p[a].x[d];
    for (int64_t i = a + 1; i < b; ++i)
        for (int d = 0; d < DIM; ++d) {
            lo[d] = std::min(lo[d], p[i].x[d]);
            hi[d] = std::max(hi[d], p[i].x[d]);
        }
    int ax = 0;
    for (int d = 1; d < DIM; ++d)
        if (hi[d] - lo[d] > hi[ax] - lo[ax]) ax = d;
    const int64_t nleaves = (count + leaf - 1) / leaf;
    const int64_t m = a + (nleaves / 2) * leaf;
    std::nth_element(p + a, p + m, p + b, [ax](const KdPoint<DIM> &u, const KdPoint<DIM> &v) {
        return u.x[ax] < v.x[ax] || (u.x[ax] == v.x[ax] && u.id < v.id);
    });
    kd_split<DIM>(p, a, m, leaf, bounds);
    kd_split<DIM>(p, m, b, leaf, bounds);
}

template <int DIM>
inline std::vector<int64_t> kd_order_of(const std::vector<double> &pts, int64_t n, int64_t leaf,
                                        std::vector<int64_t> &bounds)
{
    std::vector<KdPoint<DIM>> p(n);
    for (int64_t i = 0; i < n; ++i) {
        for (int d = 0; d < DIM; ++d) p[i].x[d] = pts[i * DIM + d];
        p[i].id = i;
    }
    bounds.clear();
    kd_split<DIM>(p.data(), 0, n, leaf, bounds);
    bounds.push_back(n);
    std::vector<int64_t> idx(n);
    for (int64_t i = 0; i < n; ++i) idx[i] = p[i].id;
    return idx;
}

inline std::vector<int64_t> kd_order(const std::vector<double> &pts, int dim, int64_t n, int64_t leaf,
                                     std::vector<int64_t> &bounds)
{
    return dim == 2 ? kd_order_of<2>(pts, n, leaf, bounds) : kd_order_of<3>(pts, n, leaf, bounds);
}

// Bounding sphere (bbox centre, max distance, enlarged by 1e-12 relative);
// box (may be null): the bounding box, lo(3) and hi(3), 0 past dim.
inline void sphere_of(const double *pts, const std::vector<int64_t> &idx, int dim, double *out, double *box = nullptr)
{
    double lo[3] = {DBL_MAX, DBL_MAX, DBL_MAX}, hi[3] = {-DBL_MAX, -DBL_MAX, -DBL_MAX};
    for (int64_t i : idx)
        for (int d = 0; d < dim; ++d) {
            lo[d] = std::min(lo[d], pts[i * dim + d]);
            hi[d] = std::max(hi[d], pts[i * dim + d]);
        }
    double c[3] = {0, 0, 0};
    for (int d = 0; d < dim; ++d) c[d] = 0.5 * (lo[d] + hi[d]);
    if (box)
        for (int d = 0; d < 3; ++d) {
            box[d] = d < dim ? lo[d] : 0.0;
            box[3 + d] = d < dim ? hi[d] : 0.0;
        }
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
