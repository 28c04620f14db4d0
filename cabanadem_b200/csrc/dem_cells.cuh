// dem_cells.cuh -- cell coordinates and keys of a Grid (dem_internal.cuh), shared by the
// neighbour build (dem_nbr.cu) and the rebuild-every-step loop (dem_refloop.cuh).
#pragma once
#include "dem_internal.cuh"

namespace b200dem {
namespace {

__device__ __forceinline__ unsigned part1by2(unsigned x) {
    x &= 0x3ff;
    x = (x | (x << 16)) & 0x030000FF;
    x = (x | (x << 8)) & 0x0300F00F;
    x = (x | (x << 4)) & 0x030C30C3;
    x = (x | (x << 2)) & 0x09249249;
    return x;
}

__device__ __forceinline__ int cell_key(const Grid &g, int cx, int cy, int cz) {
    if (g.bits > 0)
        return g.base + (int)(part1by2((unsigned)cx) | (part1by2((unsigned)cy) << 1) | (part1by2((unsigned)cz) << 2));
    return g.base + (cz * g.dims[1] + cy) * g.dims[0] + cx;
}

template <typename V4>   // V4: a position with members x, y, z
__device__ __forceinline__ void cell_of(const Grid &g, const V4 &p, int c[3]) {
    const double xs[3] = {p.x, p.y, p.z};
    for (int d = 0; d < 3; ++d) {
        int v = (int)floor((xs[d] - g.lo[d]) * g.inv_cell);
        v = v < 0 ? 0 : (v >= g.dims[d] ? g.dims[d] - 1 : v);
        c[d] = v;
    }
}

}  // namespace
}  // namespace b200dem
