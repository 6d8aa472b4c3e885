// moving.cu -- acoustic substeps over moving terrain (erf_fast_rhs_MT,
// TimeIntegration/ERF_fast_rhs_MT.cpp:48-626, with the grid of
// ERF_TI_fast_rhs_fun.H:47-118).  zo / zn: the grids at the substep's old and
// new times, zs: the stage's.
//
// A substep is two kernels: k_mt_h forms the horizontal momenta, and k_mt_col
// does a column's vertical part from the fluxes to the new state in shared
// memory.  The grid of its new time, that grid's detJ and the coefficients of
// its W system depend on the clock and the stage state alone, so they run on
// a second stream ahead of the substep.  Both kernels are bound by the
// latency of their loads (some ninety per cell, two thirds of them L1 or L2
// hits): the stage grid's metric terms come from the stage's tables and detJ
// from the arrays made once per grid, since forming each where it is used
// took forty-eight node loads per face in the right-hand side alone.  A step
// of 20 substeps, FP64: 40x8x79 1.11 ms with the geometry formed at every use
// (3.68 as twelve kernels a substep), 0.84 now; 512x128x79 54.1 (50.9), 39.2.
#include "terrain.cuh"

namespace erfb {
namespace {

// Offsets of the node columns around cell (i, j), and the nodes of a grid (in
// the znd layout: plane k + 1 for level k).
struct NodeCols {
    uint32_t c, x, y, xy, xm, xmy, ym, xym;   // (i,j) (i+1,j) (i,j+1) (i+1,j+1) (i-1,j) (i-1,j+1) (i,j-1) (i+1,j-1)
    uint32_t sk;
    __device__ __forceinline__ NodeCols(const Geo& g, int i, int j) {
        const uint32_t ip = wrap(i + 1, g.nx), im = wrap(i - 1, g.nx);
        const uint32_t r = (uint32_t)g.nx * j, rp = (uint32_t)g.nx * wrap(j + 1, g.ny), rm = (uint32_t)g.nx * wrap(j - 1, g.ny);
        c = r + i; x = r + ip; y = rp + i; xy = rp + ip; xm = r + im; xmy = rp + im; ym = rm + i; xym = rm + ip;
        sk = (uint32_t)g.sk;
    }
    __device__ __forceinline__ double operator()(const double* z, uint32_t col, int k) const {
        return ld(z, col + sk * (uint32_t)(k + 1));
    }
};
// The four nodes around z face (i, j, k): its slopes times horizontal momenta.
struct FaceNodes {
    double n00, n10, n01, n11;
    __device__ __forceinline__ FaceNodes(const NodeCols& n, const double* z, int k)
        : n00(n(z, n.c, k)), n10(n(z, n.x, k)), n01(n(z, n.y, k)), n11(n(z, n.xy, k)) {}
    __device__ __forceinline__ double slopes(const Geo& g, double u, double v) const {
        return 0.5 * g.dxi * (n11 + n10 - n01 - n00) * u + 0.5 * g.dyi * (n11 + n01 - n10 - n00) * v;
    }
};

// Coefficients of the Omega'' system on the substep's old grid, with the
// step's old base density (make_fast_coeffs, ERF_make_fast_coeffs.cpp:
// 110-290): P, Q, and the system eliminated from both walls towards face
// m = nz / 2 as in k_sub_coef (substep.cu).
template <class R>
__global__ void __launch_bounds__(512) k_mt_coef(Params P, double D, const double* __restrict__ r0, const double* __restrict__ dJo, StateBuf Sst,
                          StageAux<R> A, MtCoef<R> c) {
    extern __shared__ __align__(16) double sm[];
    const Geo& g = P.g;
    const int TX = blockDim.x, L = threadIdx.x, w = threadIdx.y, nw = blockDim.y, nz = g.nz, m = nz / 2;
    const int col = blockIdx.x * TX + L;
    const bool ok = col < (int)g.sk;
    const int j = ok ? col / g.nx : 0, i = ok ? col - j * g.nx : 0;
    double* sA = sm;
    double* sB = sA + (nz + 1) * TX;
    double* sC = sB + (nz + 1) * TX;
    const int64_t N = g.ncell, sk = g.sk;
    const double dzi = g.dzi, halfg = P.halfg;
    auto C = [&](int kk) { return eidx(g, i, j, kk); };
    auto th = [&](int kk) { return double(A.prim[C(clampk(kk, nz))]); };
    if (ok) {
        for (int k = w; k <= nz; k += nw) {
            double a = 0.0, b = 1.0, cc = 0.0, p = 0.0, q = 0.0;
            if (k > 0 && k < nz) {
                const Elem f = C(k), fm = f - sk;
                const double dJ = 0.5 * (dJo[f] + dJo[fm]), iJ = 1. / dJ;
                const double pi_c = 0.5 * (double(A.pi[fm]) + double(A.pi[f]));
                p = (-Gamma_ * R_d * dzi * iJ + halfg * R_d * r0[f + sk] / (P.c_v * P.pi0[f + sk] * Sst.cons[N + f])) * pi_c;
                q = (Gamma_ * R_d * dzi * iJ + halfg * R_d * r0[f] / (P.c_v * P.pi0[f] * Sst.cons[N + fm])) * pi_c;
                p = double(R(p));
                q = double(R(q));
                const double tlo = 0.5 * (th(k - 2) + th(k - 1)), tmid = 0.5 * (th(k - 1) + th(k)), thi = 0.5 * (th(k) + th(k + 1));
                a = D * (halfg - q * tlo);
                b = dJ + D * (q - p) * tmid;
                cc = D * (-halfg + p * thi);
            }
            sA[k * TX + L] = a; sB[k * TX + L] = b; sC[k * TX + L] = cc;
            c.P[C(k)] = R(p);
            c.Q[C(k)] = R(q);
        }
    }
    __syncthreads();
    if (ok && w < 2) {
        const bool up = w == 0;
        const int k0 = up ? 0 : nz, dk = up ? 1 : -1, n = up ? m : nz - m;
        double* elim = up ? sA : sC;
        double* keep = up ? sC : sA;
        double gam = 0.0;
        for (int q = 0, k = k0; q < n; ++q, k += dk) {
            const double bet = sB[k * TX + L] - elim[k * TX + L] * gam;
            if (!(fabs(bet) > 1e-300)) atomicOr(P.status, ST_BADSTATE);
            const double inv = 1.0 / bet;
            gam = keep[k * TX + L] * inv;
            sB[k * TX + L] = inv;
            keep[k * TX + L] = gam;
        }
    }
    __syncthreads();
    if (ok) {
        for (int k = w; k <= nz; k += nw) {
            const int s = k * TX + L;
            double inv = sB[s], e, gm;
            if (k == m) {
                const double bet = sB[s] - sA[s] * sC[s - TX] - sC[s] * sA[s + TX];
                if (!(fabs(bet) > 1e-300)) atomicOr(P.status, ST_BADSTATE);
                inv = 1.0 / bet;
                e = sA[s] * inv;
                gm = sC[s] * inv;
            } else {
                e = (k < m ? sA[s] : sC[s]) * inv;
                gm = k < m ? sC[s] : sA[s];
            }
            c.I[C(k)] = R(inv);
            c.E[C(k)] = R(e);
            c.G[C(k)] = R(gm);
        }
    }
}

// x / y momenta of the substep (ERF_fast_rhs_MT.cpp:197-273): h_zeta-weighted
// on the old grid (wx, wy: the fluxes and Omega'' read them), then divided by
// the new grid's h_zeta; d(rho theta) extrapolated with or without the lagged
// correction; the new lag; the averages.
template <class R>
__global__ void k_mt_h(Params P, int step, int lagged, double dtau, double facinv, StateBuf Sprev, StateBuf Sst,
                       StageAux<R> A, const R* __restrict__ Fmx, const R* __restrict__ Fmy, const R* __restrict__ lag_in,
                       R* __restrict__ lag_out, const double* __restrict__ zo, const double* __restrict__ zn,
                       double* __restrict__ wx, double* __restrict__ wy, StateBuf Ssum, R* __restrict__ avx,
                       R* __restrict__ avy) {
    const Geo& g = P.g;
    int i, j, k;
    if (!cell_ij(g, i, j, k)) return;
    const int nz = g.nz, im = wrap(i - 1, g.nx), jm = wrap(j - 1, g.ny);
    const Elem c = eidx(g, i, j, k), cxm = eidx(g, im, j, k), cym = eidx(g, i, jm, k);
    const NodeCols n(g, i, j);
    const double beta_d = 0.1, dxi = g.dxi, dyi = g.dyi, dzi = g.dzi;
    const double* prt = Sprev.cons + g.ncell;
    const double* srt = Sst.cons + g.ncell;
    auto extrap = [&](int ii, int jj, int kk) {
        const Elem e = eidx(g, ii, jj, clampk(kk, nz));
        const double d = ld(prt, e) - ld(srt, e);
        if (step == 0 || !lagged) return d;
        return d + beta_d * (d - double(ld(lag_in, e)));
    };
    if (step == 0 || lagged) at(lag_out, c) = R(ld(prt, c) - ld(srt, c));
    const int km = k == 0 ? 0 : k - 1;   // one-sided in the lowest cell
    const double fz = (k == 0 ? 0.5 : 0.25) * dzi;
    const double ec = extrap(i, j, k), exm = extrap(im, j, k), eym = extrap(i, jm, k);
    const double ecz = extrap(i, j, k + 1) - (k == 0 ? ec : extrap(i, j, km));
    const double pi = double(ld(A.pi, c));
    // h_xi and h_zeta of the x face, h_eta and h_zeta of the y face (mt_hxI, mt_hzI, mt_hetaJ, mt_hzJ of moving.cuh)
    auto hzx = [&](const double* z) { return 0.5 * dzi * (n(z, n.c, k + 1) + n(z, n.y, k + 1) - n(z, n.c, k) - n(z, n.y, k)); };
    auto hzy = [&](const double* z) { return 0.5 * dzi * (n(z, n.c, k + 1) + n(z, n.x, k + 1) - n(z, n.c, k) - n(z, n.x, k)); };
    {
        const double hxi = 0.125 * dxi * (n(zo, n.x, k) + n(zo, n.x, k + 1) + n(zo, n.xy, k) + n(zo, n.xy, k + 1)
                                          - n(zo, n.xm, k) - n(zo, n.xm, k + 1) - n(zo, n.xmy, k) - n(zo, n.xmy, k + 1));
        const double hz = hzx(zo);
        double gp_xi = (ec - exm) * dxi;
        double gp_zeta = fz * (ecz + extrap(im, j, k + 1) - (k == 0 ? exm : extrap(im, j, km)));
        double gpx = hz * gp_xi - hxi * gp_zeta;
        double pi_c = 0.5 * (double(ld(A.pi, cxm)) + pi);
        double mx = hz * at(Sprev.mx, c) + dtau * (-Gamma_ * R_d * pi_c * gpx) + dtau * double(ld(Fmx, c));
        at(wx, c) = mx;
        mx /= hzx(zn);
        at(Ssum.mx, c) = mx;
        at(avx, c) += R(facinv * (mx - ld(Sst.mx, c)));
    }
    {
        const double het = 0.125 * dyi * (n(zo, n.y, k) + n(zo, n.y, k + 1) + n(zo, n.xy, k) + n(zo, n.xy, k + 1)
                                          - n(zo, n.ym, k) - n(zo, n.ym, k + 1) - n(zo, n.xym, k) - n(zo, n.xym, k + 1));
        const double hz = hzy(zo);
        double gp_eta = (ec - eym) * dyi;
        double gp_zeta = fz * (ecz + extrap(i, jm, k + 1) - (k == 0 ? eym : extrap(i, jm, km)));
        double gpy = hz * gp_eta - het * gp_zeta;
        double pi_c = 0.5 * (double(ld(A.pi, cym)) + pi);
        double my = hz * at(Sprev.my, c) + dtau * (-Gamma_ * R_d * pi_c * gpy) + dtau * double(ld(Fmy, c));
        at(wy, c) = my;
        my /= hzy(zn);
        at(Ssum.my, c) = my;
        at(avy, c) += R(facinv * (my - ld(Sst.my, c)));
    }
}

// The vertical part of a column tile (ERF_fast_rhs_MT.cpp:283-600):
//   1  horizontal fluxes of rho and rho theta (the weighted momenta less the
//      stage's on the stage grid), z_t'' (the substep's z_t less the stage's),
//      Omega'' of the previous substep on the old grid.  After the first
//      substep the previous and new states are one, so Omega'' reads the
//      weighted momenta (pmx, pmy), as the reference's aliased arrays do;
//   2  right-hand side of the Omega'' system;
//   3  elimination from both walls and back;
//   4  rho w from Omega'', on the moving ground from Omega = rho (z_t + z_t'');
//   5  vertical fluxes, average contravariant momentum, rho and rho theta
//      detJ-weighted old -> new.
// The M -> V -> M round trip of the fill between substeps is the identity but
// for rounding and is not applied; w on the flat lid is 0 after it.
// P: the stage grid's parameters (its tables and detJ); zo, dJo and zn, dJn: nodes and detJ
// at the substep's old and new times.
template <class R>
__global__ void __launch_bounds__(512) k_mt_col(Params P, double dtau, double beta_1, double beta_2, double facinv, StateBuf Sprev, StateBuf Sst,
                         StageAux<R> A, const R* __restrict__ Fcons, const R* __restrict__ Fmz, MtCoef<R> cf,
                         const double* __restrict__ zo, const double* __restrict__ zn, const double* __restrict__ dJo,
                         const double* __restrict__ dJn, const double* __restrict__ wx, const double* __restrict__ wy,
                         const double* __restrict__ pmx, const double* __restrict__ pmy, R* __restrict__ avz,
                         StateBuf Ssum, int last) {
    extern __shared__ __align__(16) double sm[];
    const Geo& g = P.g;
    const int TX = blockDim.x, L = threadIdx.x, w = threadIdx.y, nw = blockDim.y, nz = g.nz, m = nz / 2;
    const int col = blockIdx.x * TX + L;
    const bool ok = col < (int)g.sk;
    const int j = ok ? col / g.nx : 0, i = ok ? col - j * g.nx : 0;
    const int n1 = (nz + 1) * TX;
    double* sT0 = sm;          // horizontal flux divergences (cells)
    double* sT1 = sT0 + n1;
    double* sO = sT1 + n1;     // Omega'' of the previous substep
    double* sS = sO + n1;      // right-hand side, solution, new Omega''
    double* sN = sS + n1;      // slopes . horizontal momenta: new state, new grid
    double* sT = sN + n1;      //                              stage state and grid
    double* sZ = sT + n1;      // z_t''
    double* sE = sZ + n1;
    double* sG = sE + n1;
    const uint32_t sk = (uint32_t)g.sk;
    const double dzi = g.dzi, halfg = fabs(0.5 * -P.gravity), inv_dt = 1. / dtau;
    const int ip = wrap(i + 1, g.nx), im = wrap(i - 1, g.nx), jp = wrap(j + 1, g.ny), jm = wrap(j - 1, g.ny);
    const NodeCols n(g, i, j);
    const double* srt = Sst.cons + g.ncell;
    const double* hzI = P.met + MT_HZETA_I * g.nzf;
    const double* hzJ = P.met + MT_HZETA_J * g.nzf;
    const R* Ft = Fcons + g.ncell;
    // (the previous state's rho, rho theta and w are the arrays written below: plain loads)
    double* prt = Sprev.cons + g.ncell;
    auto th = [&](int kk) { return double(ld(A.prim, eidx(g, i, j, clampk(kk, nz)))); };
    auto fJ = [&](const double* dJ, Elem f) { return 0.5 * (ld(dJ, f) + ld(dJ, f - sk)); };
    // face-averaged horizontal momenta of an interior z face
    auto ubar = [&](const double* mx, Elem f, Elem fx) { return 0.25 * (ld(mx, f - sk) + ld(mx, fx - sk) + ld(mx, f) + ld(mx, fx)); };
    // ---- 1
    if (ok) {
        for (int k = w; k <= nz; k += nw) {
            const Elem f = eidx(g, i, j, k), fx = eidx(g, ip, j, k), fy = eidx(g, i, jp, k);
            const int s = k * TX + L;
            if (k < nz) {
                const double xl = ld(wx, f) - ld(Sst.mx, f) * ld(hzI, f), xh = ld(wx, fx) - ld(Sst.mx, fx) * ld(hzI, fx);
                const double yl = ld(wy, f) - ld(Sst.my, f) * ld(hzJ, f), yh = ld(wy, fy) - ld(Sst.my, fy) * ld(hzJ, fy);
                auto t2 = [&](Elem e) { return double(ld(A.prim, e)); };
                const double t0 = t2(f);
                sT0[s] = (xh - xl) * g.dxi + (yh - yl) * g.dyi;
                sT1[s] = ((xh * (t0 + t2(fx)) - xl * (t0 + t2(eidx(g, im, j, k)))) * g.dxi +
                          (yh * (t0 + t2(fy)) - yl * (t0 + t2(eidx(g, i, jm, k)))) * g.dyi) * 0.5;
            }
            const FaceNodes N(n, zn, k), O(n, zo, k);
            const double zp = 0.25 * inv_dt * (N.n11 - O.n11 + N.n01 - O.n01 + N.n10 - O.n10 + N.n00 - O.n00) - ld(P.mt_zt, f);
            double an = 0.0, as = 0.0, o = 0.0;
            if (k == nz) o = at(Sprev.mz, f) - ld(Sst.mz, f) - zp;
            else if (k > 0) {
                an = N.slopes(g, ubar(Ssum.mx, f, fx), ubar(Ssum.my, f, fy));
                const double us = ubar(Sst.mx, f, fx), vs = ubar(Sst.my, f, fy);
                as = ld(P.met + MT_ZLO_XI * g.nzf, f) * us + ld(P.met + MT_ZLO_ETA * g.nzf, f) * vs;
                // (Omega'' takes the stage state on the old grid, as the reference does)
                o = ((at(Sprev.mz, f) - O.slopes(g, ubar(pmx, f, fx), ubar(pmy, f, fy))) - (ld(Sst.mz, f) - O.slopes(g, us, vs))) - zp;
            }
            sO[s] = o; sN[s] = an; sT[s] = as; sZ[s] = zp;
            sE[s] = double(ld(cf.E, f));
            sG[s] = double(ld(cf.G, f));
        }
    }
    __syncthreads();
    // ---- 2
    if (ok) {
        for (int k = w; k <= nz; k += nw) {
            const Elem a = eidx(g, i, j, k);
            const int s = k * TX + L;
            double r = 0.0;
            if (k == 0) {
                r = at(Sprev.cons, a) * sZ[s];
            } else if (k < nz) {
                const double Jo = fJ(dJo, a), Jn = fJ(dJn, a), Js = fJ(P.detJ, a);
                const double cp = double(ld(cf.P, a)), cq = double(ld(cf.Q, a));
                const double tlo = 0.5 * (th(k - 2) + th(k - 1)), tmid = 0.5 * (th(k - 1) + th(k)), thi = 0.5 * (th(k) + th(k + 1));
                const Elem b = a - sk;
                double R0t = cp * at(prt, a) * Jo + cq * at(prt, b) * Jo
                             - cp * ld(srt, a) * Js - cq * ld(srt, b) * Js
                             - halfg * (at(Sprev.cons, a) + at(Sprev.cons, b)) * Jo
                             + halfg * (ld(Sst.cons, a) + ld(Sst.cons, b)) * Js;
                double R1t = -halfg * (double(ld(Fcons, a)) + double(ld(Fcons, b))) + (cp * double(ld(Ft, a)) + cq * double(ld(Ft, b)));
                const double Okp1 = sO[s + TX], Ok = sO[s], Okm1 = sO[s - TX];
                R1t += halfg * (beta_1 * dzi * (Okp1 - Okm1) + sT0[s] + sT0[s - TX]);
                R1t += -(cp * (beta_1 * dzi * (Okp1 * thi - Ok * tmid) + sT1[s]) +
                         cq * (beta_1 * dzi * (Ok * tmid - Okm1 * tlo) + sT1[s - TX]));
                r = Jo * at(Sprev.mz, a) - Js * ld(Sst.mz, a) + dtau * (double(ld(Fmz, a)) + R0t + dtau * beta_2 * R1t);
                r += -Jn * sN[s] + Js * sT[s];
            }
            sS[s] = r * double(ld(cf.I, a));
        }
    }
    __syncthreads();
    // ---- 3
    const bool solver = ok && w < 2, up = w == 0;
    if (solver) {
        const int dk = up ? TX : -TX, n = up ? m : nz - m;
        int p = (up ? 0 : nz * TX) + L;
        double s = sS[p];
#pragma unroll 4
        for (int q = 1; q < n; ++q) {
            p += dk;
            s = sS[p] - sE[p] * s;
            sS[p] = s;
        }
    }
    __syncthreads();
    if (solver && up) {
        const int p = m * TX + L;
        sS[p] = sS[p] - sE[p] * sS[p - TX] - sG[p] * sS[p + TX];
    }
    __syncthreads();
    if (solver) {
        const int dk = up ? -TX : TX, n = up ? m : nz - m;
        int p = m * TX + L;
        double s = sS[p];
#pragma unroll 4
        for (int q = 0; q < n; ++q) {
            p += dk;
            s = sS[p] - sG[p] * s;
            sS[p] = s;
        }
    }
    __syncthreads();
    // ---- 4
    if (ok) {
        for (int k = w; k <= nz; k += nw) {
            const Elem a = eidx(g, i, j, k);
            const int s = k * TX + L;
            if (k == nz) {
                at(Ssum.mz, a) = last ? ld(Sst.mz, a) + sS[s] : 0.0;
                continue;
            }
            const double rho_on_face = 0.5 * (at(Sprev.cons, a) + (k > 0 ? at(Sprev.cons, a - sk) : at(Sprev.cons, a)));
            if (k == 0) {   // (the horizontal momenta extrapolated to the ground)
                const Elem fx = eidx(g, ip, j, 0), fy = eidx(g, i, jp, 0);
                auto ground = [&](const double* q, Elem e) {
                    return 1.5 * (0.5 * (ld(q, a) + ld(q, e))) - 0.5 * (0.5 * (ld(q, a + sk) + ld(q, e + sk)));
                };
                at(Ssum.mz, a) = rho_on_face * (ld(P.mt_zt, a) + sZ[s]) +
                                 FaceNodes(n, zn, 0).slopes(g, ground(Ssum.mx, fx), ground(Ssum.my, fy));
                sS[s] = 0.;
                continue;
            }
            const double smz = ld(Sst.mz, a), mz = fJ(dJo, a) * (smz + (sS[s] + (sN[s] - sT[s]))) / fJ(dJn, a);
            at(Ssum.mz, a) = mz;
            sS[s] = (mz - sN[s]) - (smz - sT[s]) - rho_on_face * sZ[s];
        }
    }
    __syncthreads();
    // ---- 5
    if (ok) {
        for (int k = w; k < nz; k += nw) {
            const Elem a = eidx(g, i, j, k);
            const int s = k * TX + L;
            const double zl = beta_2 * sS[s] + beta_1 * sO[s], zh = beta_2 * sS[s + TX] + beta_1 * sO[s + TX];
            at(avz, a) += R(facinv * zl);
            if (k == nz - 1) at(avz, a + sk) += R(facinv * zh);
            const double Jo = ld(dJo, a), Jn = ld(dJn, a);
            const double frho = -(sT0[s] + (zh - zl) * dzi);
            const double tr = Jo * at(Sprev.cons, a) + dtau * (double(ld(Fcons, a)) + frho);
            const double frt = -(sT1[s] + 0.5 * (zh * (th(k) + th(k + 1)) - zl * (th(k) + th(k - 1))) * dzi);
            const double tt = Jo * at(prt, a) + dtau * (double(ld(Ft, a)) + frt);
            at(Ssum.cons, a) = tr / Jn;
            at(Ssum.cons + g.ncell, a) = tt / Jn;
        }
    }
}

// detJ of a grid's cells (make_J): read by the substeps at either end of which the grid stands, and by the
// slow-variable pass
__global__ void k_mt_detj(Params P, const double* __restrict__ z, double* __restrict__ detJ) {
    const Geo& g = P.g;
    int i, j, k;
    if (!cell_ij(g, i, j, k)) return;
    detJ[cidx(g, i, j, k)] = mt_detj(z, g, i, j, k);
}

size_t mt_smem(int nz, int tx, int arrays) { return (size_t)arrays * (nz + 1) * tx * sizeof(double); }
constexpr int MT_COL_ARRAYS = 9, MT_COEF_ARRAYS = 3;
}  // namespace

// Columns per block: 16 (a row of 16 FP64 values is a line) where two blocks
// share an SM, fewer where the plane would leave SMs without a block: the
// levels of a tile are worked in parallel, so a narrow tile is as quick.  A
// single column holds every depth that erf_b200_create takes.
template <class R>
int mt_shape(const Geo& g, int* tx) {
    int dev = 0, nsm = 148, maxopt = 0, persm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    cudaDeviceGetAttribute(&maxopt, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    cudaDeviceGetAttribute(&persm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev);
    int t = 16;
    while (t > 2 && 2 * (mt_smem(g.nz, t, MT_COL_ARRAYS) + 1024) > (size_t)persm) t /= 2;
    while (t > 2 && (g.sk + t - 1) / t < nsm) t /= 2;
    while (t > 1 && mt_smem(g.nz, t, MT_COL_ARRAYS) > (size_t)maxopt) t /= 2;
    *tx = t;
    if (mt_smem(g.nz, t, MT_COL_ARRAYS) > (size_t)maxopt) return 1;
    return cudaFuncSetAttribute(k_mt_coef<R>, cudaFuncAttributeMaxDynamicSharedMemorySize, maxopt) != cudaSuccess ||
           cudaFuncSetAttribute(k_mt_col<R>, cudaFuncAttributeMaxDynamicSharedMemorySize, maxopt) != cudaSuccess;
}
// Threads per block: a row of the tile per level where that is few enough.
static dim3 mt_block(int nz, int tx, int most) {
    int rows = (nz + 1 + 31) / 32 * 32;
    while (rows > 2 && rows * tx > most) rows /= 2;
    return dim3(tx, rows);
}
void launch_mt_detj(const Params& P, cudaStream_t st, const double* z, double* detJ) {
    k_mt_detj<<<dim3((P.g.nx + 31) / 32, (P.g.ny + 3) / 4, P.g.nz), dim3(32, 4), 0, st>>>(P, z, detJ);
}
template <class R>
void launch_mt_coef(const Params& P, cudaStream_t st, int tx, double D, const double* r0, const double* dJo, StateBuf Sst,
                    StageAux<R> A, MtCoef<R> c) {
    k_mt_coef<R><<<(unsigned)((P.g.sk + tx - 1) / tx), mt_block(P.g.nz, tx, 512), mt_smem(P.g.nz, tx, MT_COEF_ARRAYS), st>>>(
        P, D, r0, dJo, Sst, A, c);
}
template <class R>
void launch_mt_fast(const Params& P, cudaStream_t st, int tx, int step, int lagged, double dtau, double beta_s,
                    double facinv, StateBuf Sprev, StateBuf Sst, StageAux<R> A, const R* Fcons, const R* Fmx, const R* Fmy,
                    const R* Fmz, const R* lag_in, R* lag_out, MtCoef<R> c, const double* zo, const double* zn,
                    const double* dJo, const double* dJn, double* wx, double* wy, R* avx, R* avy, R* avz, StateBuf Ssum,
                    int last) {
    const Geo& g = P.g;
    const double beta_1 = 0.5 * (1.0 - beta_s), beta_2 = 0.5 * (1.0 + beta_s);
    k_mt_h<R><<<dim3((g.nx + 31) / 32, (g.ny + 3) / 4, g.nz), dim3(32, 4), 0, st>>>(
        P, step, lagged, dtau, facinv, Sprev, Sst, A, Fmx, Fmy, lag_in, lag_out, zo, zn, wx, wy, Ssum, avx, avy);
    k_mt_col<R><<<(unsigned)((g.sk + tx - 1) / tx), mt_block(g.nz, tx, 512), mt_smem(g.nz, tx, MT_COL_ARRAYS), st>>>(
        P, dtau, beta_1, beta_2, facinv, Sprev, Sst, A, Fcons, Fmz, c, zo, zn, dJo, dJn, wx, wy, step == 0 ? Sprev.mx : wx,
        step == 0 ? Sprev.my : wy, avz, Ssum, last);
}

#define ERFB_MT_INSTANTIATE(R)                                                                                      \
    template int mt_shape<R>(const Geo&, int*);                                                                     \
    template void launch_mt_coef<R>(const Params&, cudaStream_t, int, double, const double*, const double*, StateBuf, \
                                    StageAux<R>, MtCoef<R>);                                                        \
    template void launch_mt_fast<R>(const Params&, cudaStream_t, int, int, int, double, double, double, StateBuf,   \
                                    StateBuf, StageAux<R>, const R*, const R*, const R*, const R*, const R*, R*,    \
                                    MtCoef<R>, const double*, const double*, const double*, const double*, double*, \
                                    double*, R*, R*, R*, StateBuf, int);
ERFB_MT_INSTANTIATE(double)
ERFB_MT_INSTANTIATE(float)
#undef ERFB_MT_INSTANTIATE

}  // namespace erfb
