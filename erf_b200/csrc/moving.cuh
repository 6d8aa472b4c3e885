// moving.cuh -- geometry of the moving terrain-following grid, evaluated from
// its nodes ((nz+3) planes of nx*ny, plane k+1 for node level k, periodic
// laterally), shared by the moving-terrain kernels (terrain.cu, moving.cu).
#pragma once
#include "kernels.cuh"

namespace erfb {

__device__ __forceinline__ double mt_time_at(double T, double dt, int tsel) {
    return tsel == 0 ? T : (tsel == 1 ? T + dt / 3.0 : (tsel == 2 ? T + dt / 2.0 : T + dt));
}
// node (i,j,k) of a grid in the znd layout ((nz+3) planes, lateral periodic)
__device__ __forceinline__ double znode(const double* z, const Geo& g, int i, int j, int k) {
    return __ldg(z + (int64_t)(k + 1) * g.sk + (int64_t)wrap(j, g.ny) * g.nx + wrap(i, g.nx));
}
// make_J of one cell from the nodes (Utils/ERF_TerrainMetrics.cpp:583-640);
// k = -1 takes level 0 (the grid's ghost level mirrors the first cell)
__device__ __forceinline__ double mt_detj(const double* z, const Geo& g, int i, int j, int k) {
    if (k < 0) k = 0;
    auto Z = [&](int a, int b, int c) { return znode(z, g, a, b, c); };
    return .25 * g.dzi * (Z(i, j, k + 1) + Z(i + 1, j, k + 1) + Z(i, j + 1, k + 1) + Z(i + 1, j + 1, k + 1)
                          - Z(i, j, k) - Z(i + 1, j, k) - Z(i, j + 1, k) - Z(i + 1, j + 1, k));
}

__device__ __forceinline__ double mt_hzI(const double* z, const Geo& g, int i, int j, int k) {
    return 0.5 * g.dzi * (znode(z, g, i, j, k + 1) + znode(z, g, i, j + 1, k + 1) - znode(z, g, i, j, k) - znode(z, g, i, j + 1, k));
}
__device__ __forceinline__ double mt_hzJ(const double* z, const Geo& g, int i, int j, int k) {
    return 0.5 * g.dzi * (znode(z, g, i, j, k + 1) + znode(z, g, i + 1, j, k + 1) - znode(z, g, i, j, k) - znode(z, g, i + 1, j, k));
}
__device__ __forceinline__ void mt_slopes(const double* z, const Geo& g, int i, int j, int k, double& sx, double& sy) {
    sx = 0.5 * g.dxi * (znode(z, g, i + 1, j + 1, k) + znode(z, g, i + 1, j, k) - znode(z, g, i, j + 1, k) - znode(z, g, i, j, k));
    sy = 0.5 * g.dyi * (znode(z, g, i + 1, j + 1, k) + znode(z, g, i, j + 1, k) - znode(z, g, i + 1, j, k) - znode(z, g, i, j, k));
}
__device__ __forceinline__ double mt_hxI(const double* z, const Geo& g, int i, int j, int k) {
    auto Z = [&](int a, int b, int c) { return znode(z, g, a, b, c); };
    return 0.125 * g.dxi * (Z(i + 1, j, k) + Z(i + 1, j, k + 1) + Z(i + 1, j + 1, k) + Z(i + 1, j + 1, k + 1)
                            - Z(i - 1, j, k) - Z(i - 1, j, k + 1) - Z(i - 1, j + 1, k) - Z(i - 1, j + 1, k + 1));
}
__device__ __forceinline__ double mt_hetaJ(const double* z, const Geo& g, int i, int j, int k) {
    auto Z = [&](int a, int b, int c) { return znode(z, g, a, b, c); };
    return 0.125 * g.dyi * (Z(i, j + 1, k) + Z(i, j + 1, k + 1) + Z(i + 1, j + 1, k) + Z(i + 1, j + 1, k + 1)
                            - Z(i, j - 1, k) - Z(i, j - 1, k + 1) - Z(i + 1, j - 1, k) - Z(i + 1, j - 1, k + 1));
}
// Face-averaged horizontal components at z-face (i,j,k) of x/y-face arrays
// given as accessors (extrapolated to the bottom face).
template <class FU, class FV>
__device__ __forceinline__ void zface_uv(int i, int j, int k, FU ua, FV va, double& u, double& v) {
    if (k == 0) {
        u = 1.5 * (0.5 * (ua(i, j, k) + ua(i + 1, j, k))) - 0.5 * (0.5 * (ua(i, j, k + 1) + ua(i + 1, j, k + 1)));
        v = 1.5 * (0.5 * (va(i, j, k) + va(i, j + 1, k))) - 0.5 * (0.5 * (va(i, j, k + 1) + va(i, j + 1, k + 1)));
    } else {
        u = 0.25 * (ua(i, j, k - 1) + ua(i + 1, j, k - 1) + ua(i, j, k) + ua(i + 1, j, k));
        v = 0.25 * (va(i, j, k - 1) + va(i, j + 1, k - 1) + va(i, j, k) + va(i, j + 1, k));
    }
}
}  // namespace erfb
