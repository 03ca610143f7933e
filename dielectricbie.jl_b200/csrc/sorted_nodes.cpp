// Sort of a geometry's nodes into the order of the direct sums.
#include "sorted_nodes.h"

#include <omp.h>

#include <algorithm>
#include <cmath>
#include <map>
#include <utility>

namespace bie {
namespace {

// Orders idx[0, m) so that consecutive runs of kTB nodes are compact boxes: recursive bisection
// across the longest side, at a multiple of kTB nodes. A tile's own nodes stay in node order. Large
// halves are tasks of the caller's thread team.
void bisect_nodes(const double* pts, int32_t* idx, int64_t m) {
    if (m > kTB) {
        double lo[3] = {INFINITY, INFINITY, INFINITY}, hi[3] = {-INFINITY, -INFINITY, -INFINITY};
        for (int64_t e = 0; e < m; ++e)
            for (int c = 0; c < 3; ++c) {
                lo[c] = std::min(lo[c], pts[3 * (int64_t)idx[e] + c]);
                hi[c] = std::max(hi[c], pts[3 * (int64_t)idx[e] + c]);
            }
        int ax = 0;
        for (int c = 1; c < 3; ++c)
            if (hi[c] - lo[c] > hi[ax] - lo[ax]) ax = c;
        const int64_t half = ((m + kTB - 1) / kTB / 2) * kTB;
        // by coordinate, not-a-numbers last, then by node: a total order for any input
        std::nth_element(idx, idx + half, idx + m, [&](int32_t a, int32_t b) {
            const double p = pts[3 * (int64_t)a + ax], q = pts[3 * (int64_t)b + ax];
            if (p < q || q < p) return p < q;
            const bool pn = std::isnan(p), qn = std::isnan(q);
            return pn == qn ? a < b : qn;
        });
#pragma omp task if (m > 8192)
        bisect_nodes(pts, idx, half);
        bisect_nodes(pts, idx + half, m - half);
    } else {
        std::sort(idx, idx + m);
    }
}

}  // namespace

SortedNodes sort_nodes(const double* pts, const double* nrm, const double* /*w*/, int64_t n) {
    double lo[3] = {INFINITY, INFINITY, INFINITY}, hi[3] = {-INFINITY, -INFINITY, -INFINITY};
    for (int64_t i = 0; i < n; ++i)
        for (int c = 0; c < 3; ++c) {
            lo[c] = std::min(lo[c], pts[3 * i + c]);
            hi[c] = std::max(hi[c], pts[3 * i + c]);
        }
    const double ext = std::max({hi[0] - lo[0], hi[1] - lo[1], hi[2] - lo[2], 0.0});
    // planes (axis, coordinate) of the axis-aligned normals, in the order of their first node
    std::map<std::pair<int, double>, int> plane_id;
    std::vector<std::pair<int, int64_t>> planes;  // axis, nodes
    std::vector<int> of((size_t)n, -1);
    int last = -1;  // nodes come panel by panel: the previous node's plane is the likely one
    std::pair<int, double> last_key(-1, 0.0);
    for (int64_t i = 0; i < n; ++i) {
        const double* m = nrm + 3 * i;
        const int ax = std::fabs(m[0]) == 1.0 && m[1] == 0.0 && m[2] == 0.0   ? 0
                       : std::fabs(m[1]) == 1.0 && m[0] == 0.0 && m[2] == 0.0 ? 1
                       : std::fabs(m[2]) == 1.0 && m[0] == 0.0 && m[1] == 0.0 ? 2
                                                                              : 3;
        if (ax == 3 || !std::isfinite(pts[3 * i + ax])) continue;
        const std::pair<int, double> k(ax, pts[3 * i + ax]);
        if (last < 0 || k != last_key) {
            const auto it = plane_id.emplace(k, (int)planes.size()).first;
            last = it->second;
            last_key = k;
            if (last == (int)planes.size()) planes.push_back({ax, 0});
        }
        of[i] = last;
        ++planes[last].second;
    }
    // group starts, each group padded to whole tiles; the nodes of no (large enough) plane last
    auto padded = [](int64_t m) { return (m + kTB - 1) / kTB * kTB; };
    std::vector<int64_t> at(planes.size() + 1);
    int64_t ns = 0, rest = n;
    for (size_t p = 0; p < planes.size(); ++p) {
        const int64_t m = planes[p].second >= kPlaneMin ? planes[p].second : 0;
        at[p] = ns;
        ns += padded(m);
        rest -= m;
    }
    at.back() = ns;
    ns += padded(rest);
    SortedNodes so;
    so.perm.assign((size_t)ns, -1);
    so.tiles.assign((size_t)(ns / kTB), TileInfo{3, 0, 0, {}, {}});
    for (size_t p = 0; p < planes.size(); ++p) {
        if (planes[p].second < kPlaneMin) continue;
        const int64_t s0 = at[p], s1 = s0 + padded(planes[p].second);
        for (int64_t t = s0 / kTB; t < s1 / kTB; ++t)
            so.tiles[t] = TileInfo{planes[p].first, (int32_t)s0, (int32_t)s1, {}, {}};
    }
    for (int64_t i = 0; i < n; ++i) {
        const bool in_plane = of[i] >= 0 && planes[of[i]].second >= kPlaneMin;
        so.perm[in_plane ? at[of[i]]++ : at.back()++] = (int32_t)i;
    }
    // up to 8 threads, fewer where the caller's OpenMP setting says so (us, one thread and eight: 1,536
    // nodes 40 and 42, 6,144 nodes 350 and 185, 16,224 nodes 1,570 and 530)
#pragma omp parallel num_threads(std::min(8, omp_get_max_threads())) if (n > 2048)
#pragma omp single
    {
        for (size_t p = 0; p < planes.size(); ++p)
            if (planes[p].second >= kPlaneMin) {
                int32_t* idx = &so.perm[at[p] - planes[p].second];
                const int64_t m = planes[p].second;
#pragma omp task firstprivate(idx, m)
                bisect_nodes(pts, idx, m);
            }
        if (rest > 0) bisect_nodes(pts, &so.perm[at.back() - rest], rest);
    }
    int ex = 0;
    if (std::isfinite(ext) && ext > 0.0) std::frexp(ext, &ex);
    const double scale = so.scale = std::ldexp(1.0, -std::max(-300, std::min(300, ex)));
    for (size_t t = 0; t < so.tiles.size(); ++t)
        for (int c = 0; c < 3; ++c) {
            double a = INFINITY, b = -INFINITY;
            for (int64_t e = (int64_t)t * kTB; e < (int64_t)(t + 1) * kTB && so.perm[e] >= 0; ++e) {
                const double x = pts[3 * (int64_t)so.perm[e] + c] * scale;
                a = std::min(a, x);
                b = std::max(b, x);
            }
            so.tiles[t].o[c] = a == b ? a : 0.5 * (a + b);  // exactly the plane's along its axis
            so.tiles[t].h[c] = 0.5 * (b - a);
        }
    return so;
}

}  // namespace bie
