// Node order of the direct sums (host side): coordinate planes together, compact tiles, padding.
#pragma once
#include <cstdint>
#include <vector>

namespace bie {

constexpr int kTB = 128;         // nodes of a tile: targets per CTA of the direct-sum kernels
constexpr int kPlaneMin = 256;   // nodes from which a coordinate plane is kept together
constexpr double kFar = 1.0e18;  // coordinates of padding slots

// Tiles of kTB consecutive slots of the sorted node order (GeomDev). A planar tile's nodes
// share one plane x_axis = const with normals +-e_axis, and that plane's nodes are the slots
// [s0, s1): the kernel n_x . (x - y) / |x - y|^3 of such a target and such a source is exactly
// zero, so the direct sums leave those slots out. axis = 3, s0 = s1 = 0: any other tile. o and h:
// middle and half sides of the tile's bounding box (o is the plane itself along a planar tile's
// axis); o is the origin that the FP32 sums take coordinates relative to.
struct TileInfo {
    int32_t axis, s0, s1;
    double o[3], h[3];
};

// The sorted order of the direct sums (GeomDev): the node of each slot, each tile's plane and origin, and
// the power of two that the positions are scaled by.
struct SortedNodes {
    std::vector<int32_t> perm;
    std::vector<TileInfo> tiles;
    double scale;
};

// Sorts n nodes (positions and normals 3 x n; the order does not depend on the weights).
SortedNodes sort_nodes(const double* pts, const double* nrm, const double* w, int64_t n);

}  // namespace bie
