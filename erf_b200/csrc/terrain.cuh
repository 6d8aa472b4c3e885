// terrain.cuh -- metric terms and wall-aware accessors of the terrain-following
// grid, shared by the terrain passes (terrain.cu) and the acoustic substeps
// over terrain (ter_fast.cu).
#pragma once
#include "kernels.cuh"
#include "moving.cuh"

namespace erfb {
namespace {

// ---------------------------------------------------------------------------
// Metric terms (Utils/ERF_TerrainMetrics.H:33-395), same operand order.
// ---------------------------------------------------------------------------
__device__ __forceinline__ double Zn(const Params& P, int i, int j, int k) {
    const Geo& g = P.g;
    return __ldg(P.znd + (int64_t)(k + 1) * g.sk + (int64_t)wrap(j, g.ny) * g.nx + wrap(i, g.nx));
}
#define ZN(a, b, c) Zn(P, a, b, c)
__device__ __forceinline__ double detJ_at(const Params& P, int i, int j, int k) {
    const Geo& g = P.g;
    return ld(P.detJ, eidx(g, wrap(i, g.nx), wrap(j, g.ny), clampk(k, g.nz)));
}
__device__ __forceinline__ double hzeta_cc_fn(const Params& P, int i, int j, int k) {
    return 0.25 * P.g.dzi * (ZN(i + 1, j, k + 1) + ZN(i + 1, j + 1, k + 1) + ZN(i, j, k + 1) + ZN(i, j + 1, k + 1)
                             - ZN(i + 1, j, k) - ZN(i + 1, j + 1, k) - ZN(i, j, k) - ZN(i, j + 1, k));
}
__device__ __forceinline__ double hxi_cc_fn(const Params& P, int i, int j, int k) {
    return 0.25 * P.g.dxi * (ZN(i + 1, j, k) + ZN(i + 1, j + 1, k) + ZN(i + 1, j, k + 1) + ZN(i + 1, j + 1, k + 1)
                             - ZN(i, j, k) - ZN(i, j + 1, k) - ZN(i, j, k + 1) - ZN(i, j + 1, k + 1));
}
__device__ __forceinline__ double heta_cc_fn(const Params& P, int i, int j, int k) {
    return 0.25 * P.g.dyi * (ZN(i, j + 1, k) + ZN(i + 1, j + 1, k) + ZN(i, j + 1, k + 1) + ZN(i + 1, j + 1, k + 1)
                             - ZN(i, j, k) - ZN(i + 1, j, k) - ZN(i, j, k + 1) - ZN(i + 1, j, k + 1));
}
// x faces (also ax) and y faces (also ay)
__device__ __forceinline__ double hzeta_I_fn(const Params& P, int i, int j, int k) {
    return 0.5 * P.g.dzi * (ZN(i, j, k + 1) + ZN(i, j + 1, k + 1) - ZN(i, j, k) - ZN(i, j + 1, k));
}
__device__ __forceinline__ double hxi_I_fn(const Params& P, int i, int j, int k) {
    return 0.125 * P.g.dxi * (ZN(i + 1, j, k) + ZN(i + 1, j, k + 1) + ZN(i + 1, j + 1, k) + ZN(i + 1, j + 1, k + 1)
                              - ZN(i - 1, j, k) - ZN(i - 1, j, k + 1) - ZN(i - 1, j + 1, k) - ZN(i - 1, j + 1, k + 1));
}
__device__ __forceinline__ double hzeta_J_fn(const Params& P, int i, int j, int k) {
    return 0.5 * P.g.dzi * (ZN(i, j, k + 1) + ZN(i + 1, j, k + 1) - ZN(i, j, k) - ZN(i + 1, j, k));
}
__device__ __forceinline__ double heta_J_fn(const Params& P, int i, int j, int k) {
    return 0.125 * P.g.dyi * (ZN(i, j + 1, k) + ZN(i, j + 1, k + 1) + ZN(i + 1, j + 1, k) + ZN(i + 1, j + 1, k + 1)
                              - ZN(i, j - 1, k) - ZN(i, j - 1, k + 1) - ZN(i + 1, j - 1, k) - ZN(i + 1, j - 1, k + 1));
}
// z faces
__device__ __forceinline__ double hzeta_K_fn(const Params& P, int i, int j, int k) {
    return 0.125 * P.g.dzi * (ZN(i, j, k + 1) + ZN(i + 1, j, k + 1) + ZN(i, j + 1, k + 1) + ZN(i + 1, j + 1, k + 1)
                              - ZN(i, j, k - 1) - ZN(i + 1, j, k - 1) - ZN(i, j + 1, k - 1) - ZN(i + 1, j + 1, k - 1));
}
__device__ __forceinline__ double hxi_K_fn(const Params& P, int i, int j, int k) {
    return 0.5 * P.g.dxi * (ZN(i + 1, j, k) + ZN(i + 1, j + 1, k) - ZN(i, j, k) - ZN(i, j + 1, k));
}
__device__ __forceinline__ double heta_K_fn(const Params& P, int i, int j, int k) {
    return 0.5 * P.g.dyi * (ZN(i, j + 1, k) + ZN(i + 1, j + 1, k) - ZN(i, j, k) - ZN(i + 1, j, k));
}
// xy edges (EdgeCenterK), xz edges (EdgeCenterJ), yz edges (EdgeCenterI)
__device__ __forceinline__ double hzeta_EK_fn(const Params& P, int i, int j, int k) { return P.g.dzi * (ZN(i, j, k + 1) - ZN(i, j, k)); }
__device__ __forceinline__ double hxi_EK_fn(const Params& P, int i, int j, int k) {
    return 0.25 * P.g.dxi * (ZN(i + 1, j, k) + ZN(i + 1, j, k + 1) - ZN(i - 1, j, k) - ZN(i - 1, j, k + 1));
}
__device__ __forceinline__ double heta_EK_fn(const Params& P, int i, int j, int k) {
    return 0.25 * P.g.dyi * (ZN(i, j + 1, k) + ZN(i, j + 1, k + 1) - ZN(i, j - 1, k) - ZN(i, j - 1, k + 1));
}
__device__ __forceinline__ double hzeta_EJ_fn(const Params& P, int i, int j, int k) {
    return 0.25 * P.g.dzi * (ZN(i, j, k + 1) + ZN(i, j + 1, k + 1) - ZN(i, j, k - 1) - ZN(i, j + 1, k - 1));
}
__device__ __forceinline__ double hxi_EJ_fn(const Params& P, int i, int j, int k) {
    return 0.25 * P.g.dxi * (ZN(i + 1, j + 1, k) + ZN(i + 1, j, k) - ZN(i - 1, j + 1, k) - ZN(i - 1, j, k));
}
__device__ __forceinline__ double heta_EJ_fn(const Params& P, int i, int j, int k) { return P.g.dyi * (ZN(i, j + 1, k) - ZN(i, j, k)); }
__device__ __forceinline__ double hzeta_EI_fn(const Params& P, int i, int j, int k) {
    return 0.25 * P.g.dzi * (ZN(i, j, k + 1) + ZN(i + 1, j, k + 1) - ZN(i, j, k - 1) - ZN(i + 1, j, k - 1));
}
__device__ __forceinline__ double hxi_EI_fn(const Params& P, int i, int j, int k) { return P.g.dxi * (ZN(i + 1, j, k) - ZN(i, j, k)); }
__device__ __forceinline__ double heta_EI_fn(const Params& P, int i, int j, int k) {
    return 0.25 * P.g.dyi * (ZN(i + 1, j + 1, k) + ZN(i, j + 1, k) - ZN(i + 1, j - 1, k) - ZN(i, j - 1, k));
}
// slopes of a z-face (OmegaFromW / WFromOmega, ERF_TerrainMetrics.H:455-520)
__device__ __forceinline__ double zlo_xi_fn(const Params& P, int i, int j, int k) {
    return 0.5 * P.g.dxi * (ZN(i + 1, j + 1, k) + ZN(i + 1, j, k) - ZN(i, j + 1, k) - ZN(i, j, k));
}
__device__ __forceinline__ double zlo_eta_fn(const Params& P, int i, int j, int k) {
    return 0.5 * P.g.dyi * (ZN(i + 1, j + 1, k) + ZN(i, j + 1, k) - ZN(i + 1, j, k) - ZN(i, j, k));
}
#undef ZN

// Static-terrain metric tables: the metric terms the passes read,
// evaluated once per cell / face / edge by the functions above (so bit-identical to
// evaluating them in place) and stored as TER_NMET planes of (nz+1) x ny x
// nx values, k in [0, nz].  A pass reads one value instead of re-deriving it
// from four to eight nodes of z_phys_nd; outside [0, nz] the function runs.
enum { MT_HZETA_I, MT_HZETA_J, MT_HXI_K, MT_HETA_K, MT_HZETA_EK, MT_HZETA_EJ, MT_HZETA_EI,
       MT_ZLO_XI, MT_ZLO_ETA, MT_HZETA_CC, MT_HXI_CC, MT_HETA_CC, MT_HZETA_K, MT_HXI_EK, MT_HETA_EK, MT_HXI_EJ,
       MT_HETA_EJ, MT_HXI_EI, MT_HETA_EI, MT_RXI_I, MT_RETA_J, MT_IJ, MT_COUNT };
static_assert(MT_COUNT == TER_NMET, "metric table count");
__device__ __forceinline__ double mt_at(const Params& P, int q, int i, int j, int k) {
    const Geo& g = P.g;
    return ld(P.met + (int64_t)q * g.nzf, eidx(g, wrap(i, g.nx), wrap(j, g.ny), k));
}
#define ERFB_MT(name, q)                                                           \
    __device__ __forceinline__ double name(const Params& P, int i, int j, int k) { \
        if (k >= 0 && k <= P.g.nz) return mt_at(P, q, i, j, k);                   \
        return name##_fn(P, i, j, k);                                              \
    }
ERFB_MT(hzeta_I, MT_HZETA_I)
ERFB_MT(hzeta_J, MT_HZETA_J)
ERFB_MT(hxi_K, MT_HXI_K)
ERFB_MT(heta_K, MT_HETA_K)
ERFB_MT(hzeta_EK, MT_HZETA_EK)
ERFB_MT(hzeta_EJ, MT_HZETA_EJ)
ERFB_MT(hzeta_EI, MT_HZETA_EI)
ERFB_MT(zlo_xi, MT_ZLO_XI)
ERFB_MT(zlo_eta, MT_ZLO_ETA)
ERFB_MT(hzeta_cc, MT_HZETA_CC)
ERFB_MT(hxi_cc, MT_HXI_CC)
ERFB_MT(heta_cc, MT_HETA_CC)
ERFB_MT(hzeta_K, MT_HZETA_K)
ERFB_MT(hxi_EK, MT_HXI_EK)
ERFB_MT(heta_EK, MT_HETA_EK)
ERFB_MT(hxi_EJ, MT_HXI_EJ)
ERFB_MT(heta_EJ, MT_HETA_EJ)
ERFB_MT(hxi_EI, MT_HXI_EI)
ERFB_MT(heta_EI, MT_HETA_EI)
#undef ERFB_MT
// Quotients of them, k in [0, nz): the slopes h_xi / h_zeta and h_eta / h_zeta
// of the x and y faces and 1 / detJ of the cells (an FP64 division is some
// twenty instructions, and every pass of every substep needs these).
__device__ __forceinline__ double slope_I(const Params& P, int i, int j, int k) { return mt_at(P, MT_RXI_I, i, j, k); }
__device__ __forceinline__ double slope_J(const Params& P, int i, int j, int k) { return mt_at(P, MT_RETA_J, i, j, k); }
__device__ __forceinline__ double inv_detJ(const Params& P, int i, int j, int k) { return mt_at(P, MT_IJ, i, j, clampk(k, P.g.nz)); }

template <class FU, class FV>
__device__ __forceinline__ double omega_from_w(const Params& P, int i, int j, int k, double w, FU ua, FV va) {
    double mx = zlo_xi(P, i, j, k), my = zlo_eta(P, i, j, k), u, v;
    zface_uv(i, j, k, ua, va, u, v);
    return w - mx * u - my * v;
}
template <class FU, class FV>
__device__ __forceinline__ double w_from_omega(const Params& P, int i, int j, int k, double om, FU ua, FV va) {
    double mx = zlo_xi(P, i, j, k), my = zlo_eta(P, i, j, k), u, v;
    zface_uv(i, j, k, ua, va, u, v);
    return om + mx * u + my * v;
}

// qv + qc averaged over two cells (the moist pressure-gradient factor
// 1 + q of ERF_slow_rhs_pre.cpp:594-744 and ERF_fast_rhs_T.cpp:230-300);
// 0 for a dry state.
template <class R>
__device__ __forceinline__ double moist_q(const Params& P, const R* prim, int64_t a, int64_t b) {
    if (!P.moist) return 0.0;
    const int64_t N = P.g.ncell;
    return 0.5 * (double(prim[4 * N + a]) + double(prim[4 * N + b]) + double(prim[5 * N + a]) + double(prim[5 * N + b]));
}

// Base state at (i,j,k), k in [-1, nz].
__device__ __forceinline__ double bs(const double* f, const Geo& g, int i, int j, int k) {
    return __ldg(f + (int64_t)(k + 1) * g.sk + (int64_t)j * g.nx + i);
}

// Horizontal momentum after the M -> V -> M round trip of a boundary fill
// (face (i,j,k) wrapped laterally, k in [0, nz)) and the velocity it gives.
__device__ __forceinline__ double rt_u(const Geo& g, const double* cons, const double* mx, int i, int j, int k) {
    i = wrap(i, g.nx); j = wrap(j, g.ny);
    double rs = cons[cidx(g, i, j, k)] + cons[cidx(g, wrap(i - 1, g.nx), j, k)];
    return (mx[cidx(g, i, j, k)] * 2.0) / rs;
}
__device__ __forceinline__ double rt_v(const Geo& g, const double* cons, const double* my, int i, int j, int k) {
    i = wrap(i, g.nx); j = wrap(j, g.ny);
    double rs = cons[cidx(g, i, j, k)] + cons[cidx(g, i, wrap(j - 1, g.ny), k)];
    return (my[cidx(g, i, j, k)] * 2.0) / rs;
}

// Tangential velocity with its wall ghost (ext_dir 0 or foextrap), lateral
// indices wrapped here.
__device__ __forceinline__ double tvel(const double* f, const Geo& g, int i, int j, int k) {
    i = wrap(i, g.nx); j = wrap(j, g.ny);
    if (k < 0) return g.zlo_noslip ? 0.0 : ld(f, eidx(g, i, j, 0));
    if (k >= g.nz) return g.zhi_noslip ? 0.0 : ld(f, eidx(g, i, j, g.nz - 1));
    return ld(f, eidx(g, i, j, k));
}
// w at z-face k in [0, nz], lateral wrap
__device__ __forceinline__ double wvel(const double* f, const Geo& g, int i, int j, int k) {
    i = wrap(i, g.nx); j = wrap(j, g.ny);
    k = k < 0 ? 0 : (k > g.nz ? g.nz : k);
    return ld(f, eidx(g, i, j, k));
}
// cell-centred value with lateral wrap and foextrap in z
template <class V>
__device__ __forceinline__ double ccw(const V* f, const Geo& g, int i, int j, int k) {
    return double(ld(f, eidx(g, wrap(i, g.nx), wrap(j, g.ny), clampk(k, g.nz))));
}

__device__ __forceinline__ bool cell_ij(const Geo& g, int& i, int& j, int& k) {
    i = blockIdx.x * blockDim.x + threadIdx.x;
    j = blockIdx.y * blockDim.y + threadIdx.y;
    k = blockIdx.z;
    return i < g.nx && j < g.ny && k < g.nz;
}
dim3 ter_block() { return dim3(32, 4, 1); }
dim3 ter_grid(const Geo& g, int nk) { return dim3((g.nx + 31) / 32, (g.ny + 3) / 4, nk); }

}  // namespace
}  // namespace erfb
