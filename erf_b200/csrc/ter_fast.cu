// ter_fast.cu -- acoustic substeps over static terrain (erf_fast_rhs_T,
// TimeIntegration/ERF_fast_rhs_T.cpp:130-680, with make_fast_coeffs): the
// stage's coefficients, the horizontal part and the column part of a substep.
#include "terrain.cuh"

namespace erfb {
namespace {

// Coefficients of the Omega'' system (ERF_make_fast_coeffs.cpp:110-290 with
// detJ at the faces and the 3-D base state), eliminated from both walls as in
// k_sub_coef (substep.cu).  256x256x96, FP64: 209 us per stage with a one-sided
// elimination in 32-column tiles, 173 now (on the side stream, under the slow
// passes).
template <class R>
__global__ void __launch_bounds__(512) k_ter_coef(Params P, double D, StateBuf Sst, StageAux<R> A, MtCoef<R> c) {
    extern __shared__ __align__(16) double sm[];
    const Geo& g = P.g;
    const int TX = blockDim.x, L = threadIdx.x, w = threadIdx.y, nw = blockDim.y, nz = g.nz, m = nz / 2;
    const int col = blockIdx.x * TX + L;
    const bool ok = col < (int)g.sk;
    const int j = ok ? col / g.nx : 0, i = ok ? col - j * g.nx : 0;
    double* sA = sm;
    double* sB = sA + (nz + 1) * TX;
    double* sC = sB + (nz + 1) * TX;
    const uint32_t sk = (uint32_t)g.sk;
    const double dzi = g.dzi, halfg = P.halfg;
    const double* srt = Sst.cons + g.ncell;
    auto th = [&](int kk) { return ccw(A.prim, g, i, j, kk); };
    if (ok) {
        for (int k = w; k <= nz; k += nw) {
            const Elem f = eidx(g, i, j, k);
            double a = 0.0, b = 1.0, cc = 0.0, p = 0.0, q = 0.0;
            if (k > 0 && k < nz) {
                const Elem fm = f - sk;
                const double dJ = 0.5 * (detJ_at(P, i, j, k) + detJ_at(P, i, j, k - 1)), iJ = 1. / dJ;
                const double pi_c = 0.5 * (double(ld(A.pi, fm)) + double(ld(A.pi, f)));
                p = (-Gamma_ * R_d * dzi * iJ + halfg * R_d * ld(P.r0, f + sk) / (P.c_v * ld(P.pi0, f + sk) * ld(srt, f))) * pi_c;
                q = (Gamma_ * R_d * dzi * iJ + halfg * R_d * ld(P.r0, f) / (P.c_v * ld(P.pi0, f) * ld(srt, fm))) * pi_c;
                if (P.moist) {
                    const double wet = 1.0 / (1.0 + moist_q(P, A.prim, f, fm));
                    p *= wet;
                    q *= wet;
                }
                p = double(R(p));
                q = double(R(q));
                const double t_1 = th(k - 1), t0 = th(k);
                a = D * (halfg - q * (0.5 * (th(k - 2) + t_1)));
                b = dJ + D * (q - p) * (0.5 * (t_1 + t0));
                cc = D * (-halfg + p * (0.5 * (t0 + th(k + 1))));
            }
            sA[k * TX + L] = a; sB[k * TX + L] = b; sC[k * TX + L] = cc;
            at(c.P, f) = R(p);
            at(c.Q, f) = R(q);
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
            const Elem f = eidx(g, i, j, k);
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
            at(c.I, f) = R(inv);
            at(c.E, f) = R(e);
            at(c.G, f) = R(gm);
        }
    }
}
}  // namespace

// ---------------------------------------------------------------------------
// Acoustic substep with terrain, horizontal part (ERF_fast_rhs_T.cpp:130-320):
// lagged d(rho theta) and its extrapolation, U'' / V'' with the
// terrain-corrected gradient of the extrapolated d(rho theta); the old and
// new increments are kept for the vertical part.
// ---------------------------------------------------------------------------
// After the first substep (of the fused step) the extrapolated d(rho theta)
// comes from the vertical part, which has both substeps' values in hand, and
// in the FP64 form the old increments are the previous substep's new ones:
// nine loads in place of twenty-seven.  In the mixed form the stored
// increments have 24 bits (the vertical part reads those), so that the old
// ones are formed from the FP64 momenta again and the state accumulates in
// FP64.  The M -> V -> M round trip of the fill between substeps is the
// identity but for rounding and is not applied.
template <class R, bool FIRST>
__global__ void k_ter_fast_h(Params P, int step, double dtau, double facinv, StateBuf Sprev, StateBuf Sst, StageAux<R> A,
                             const R* __restrict__ Fmx, const R* __restrict__ Fmy, const R* __restrict__ lag_in,
                             R* __restrict__ lag_out, TerBuf<R> T, R* __restrict__ avx, R* __restrict__ avy,
                             double* outx, double* outy) {
    const Geo& g = P.g;
    int i, j, k;
    if (!cell_ij(g, i, j, k)) return;
    const int nz = g.nz, im = wrap(i - 1, g.nx), jm = wrap(j - 1, g.ny);
    const Elem c = eidx(g, i, j, k), cxm = eidx(g, im, j, k), cym = eidx(g, i, jm, k);
    const double beta_d = 0.1, dxi = g.dxi, dyi = g.dyi;
    const double* prt = Sprev.cons + g.ncell;
    const double* srt = Sst.cons + g.ncell;
    auto extrap = [&](int ii, int jj, int kk) {
        const Elem e = eidx(g, ii, jj, clampk(kk, nz));
        if (!FIRST) return ld(T.ec, e);
        const double drt = ld(prt, e) - ld(srt, e);
        return step == 0 ? drt : drt + beta_d * (drt - double(ld(lag_in, e)));
    };
    if (FIRST && lag_out) at(lag_out, c) = R(ld(prt, c) - ld(srt, c));
    double odu, odv;
    if (FIRST || sizeof(R) < sizeof(double)) {   // (after the first substep Sprev is the array written below)
        odu = at(Sprev.mx, c) - ld(Sst.mx, c);
        odv = at(Sprev.my, c) - ld(Sst.my, c);
        if (FIRST) {
            at(T.odu, c) = R(odu);
            at(T.odv, c) = R(odv);
        }
    } else {
        odu = double(ld(T.odu, c));
        odv = double(ld(T.odv, c));
    }
    const int km = k == 0 ? 0 : k - 1;   // one-sided in the lowest cell
    const double fz = (k == 0 ? 0.5 : 0.25) * g.dzi;
    const double ec = extrap(i, j, k), exm = extrap(im, j, k), eym = extrap(i, jm, k);
    const double ecz = extrap(i, j, k + 1) - extrap(i, j, km);
    double gpx = (ec - exm) * dxi - slope_I(P, i, j, k) * (fz * (ecz + extrap(im, j, k + 1) - extrap(im, j, km)));
    double gpy = (ec - eym) * dyi - slope_J(P, i, j, k) * (fz * (ecz + extrap(i, jm, k + 1) - extrap(i, jm, km)));
    if (P.moist) {
        gpx /= 1.0 + moist_q(P, A.prim, c, cxm);
        gpy /= 1.0 + moist_q(P, A.prim, c, cym);
    }
    const double pc = double(ld(A.pi, c));
    const double fx = -Gamma_ * R_d * (0.5 * (double(ld(A.pi, cxm)) + pc)) * gpx;
    const double fy = -Gamma_ * R_d * (0.5 * (double(ld(A.pi, cym)) + pc)) * gpy;
    const double ndu = odu + dtau * fx + dtau * double(ld(Fmx, c));
    const double ndv = odv + dtau * fy + dtau * double(ld(Fmy, c));
    at(T.ndu, c) = R(ndu);
    at(T.ndv, c) = R(ndv);
    at(avx, c) += R(facinv * ndu);
    at(avy, c) += R(facinv * ndv);
    at(outx, c) = ld(Sst.mx, c) + ndu;
    at(outy, c) = ld(Sst.my, c) + ndv;
}

// ---------------------------------------------------------------------------
// Acoustic substep with terrain, vertical part (ERF_fast_rhs_T.cpp:320-680):
// horizontal rho / rho*theta fluxes through the sloping faces, Omega of the
// previous increments, the detJ-weighted right-hand side of the Omega''
// system, the Thomas sweep on the stage's coefficients, then w'' from
// Omega'', the vertical fluxes, the average contravariant momentum, rho and
// rho*theta (k_ter_fast_vert below).
// ---------------------------------------------------------------------------
namespace {
template <class R>
__device__ __forceinline__ double prev_mz_ter(const Params& P, StateBuf Sprev, int prev_rt, int i, int j, int k) {
    const Geo& g = P.g;
    const int nz = g.nz;
    int64_t f = cidx(g, i, j, k);
    double m = Sprev.mz[f];
    if (prev_rt && (k == 0 || k == nz)) {
        auto U1 = [&](int ii, int jj, int kk) {
            if (kk >= nz) {
                if (g.zhi_noslip) return 0.0;
                kk = nz - 1;
            }
            return rt_u(g, Sprev.cons, Sprev.mx, ii, jj, kk);
        };
        auto V1 = [&](int ii, int jj, int kk) {
            if (kk >= nz) {
                if (g.zhi_noslip) return 0.0;
                kk = nz - 1;
            }
            return rt_v(g, Sprev.cons, Sprev.my, ii, jj, kk);
        };
        int kc = (k == 0) ? 0 : nz - 1;
        double r = Sprev.cons[cidx(g, i, j, kc)];
        double wb = w_from_omega(P, i, j, k, 0.0, U1, V1);
        return (wb * 0.5) * (r + r);
    }
    return m;
}
}  // namespace

// One pass per column tile, the block's warps spread over the levels, the
// column arrays in shared memory, so that the horizontal fluxes, Omega of the
// old increments, the right-hand side and the solution never leave the SM.
// The slopes' part of the new increments is formed once per face (the
// right-hand side and w'' had each read eight increments and two metrics for
// it again); two blocks share an SM, so that one's serial sweep, eliminated
// from both walls, runs under the other's loads.  Bound by the loads in flight
// (thirty-odd values per cell, two thirds of them L2 hits).  256x256x96, FP64:
// 492 us per substep with one 1024-thread block, 460 now.  The momentum of the
// previous substep on the ground and lid faces (w from Omega = 0 of its
// round-tripped u, v) reads neighbouring columns of a state the update
// overwrites in place, so k_ter_fv_bnd forms it first.
template <class R>
__global__ void k_ter_fv_bnd(Params P, StateBuf Sprev, TerBuf<R> T) {
    const Geo& g = P.g;
    const int i = blockIdx.x * blockDim.x + threadIdx.x, j = blockIdx.y * blockDim.y + threadIdx.y;
    if (i >= g.nx || j >= g.ny) return;
    const int64_t col = (int64_t)j * g.nx + i;
    T.bnd[col] = prev_mz_ter<R>(P, Sprev, 1, i, j, 0);
    T.bnd[g.sk + col] = prev_mz_ter<R>(P, Sprev, 1, i, j, g.nz);
}

template <class R>
__global__ void __launch_bounds__(1024) k_ter_fast_vert(Params P, double dtau, double facinv, double beta_1,
                                                        double beta_2, StateBuf Sprev, int prev_rt, StateBuf Sst,
                                                        StageAux<R> A, const R* __restrict__ Fcons,
                                                        const R* __restrict__ Fmz, TerBuf<R> T, MtCoef<R> cf,
                                                        R* __restrict__ avz, double* out_cons, double* out_mz) {
    extern __shared__ __align__(16) double sm[];
    const Geo& g = P.g;
    const int nz = g.nz, TX = blockDim.x, L = threadIdx.x, w0 = threadIdx.y, nw = blockDim.y, m = nz / 2;
    const int col = blockIdx.x * TX + L;   // consecutive columns of the plane, rows running on
    const bool ok = col < (int)g.sk;
    const int j = ok ? col / g.nx : 0, i = ok ? col - j * g.nx : 0;
    const int ip = wrap(i + 1, g.nx), jp = wrap(j + 1, g.ny);
    const int n1 = (nz + 1) * TX;
    double* sT0 = sm;          // horizontal rho flux divergence (cells)
    double* sT1 = sT0 + n1;    // horizontal rho*theta flux divergence (cells)
    double* sO = sT1 + n1;     // Omega of the old increments (faces)
    double* sR = sO + n1;      // right-hand side, then the solution (faces)
    double* sN = sR + n1;      // slopes . new horizontal increments (faces)
    double* sE = sN + n1;
    double* sG = sE + n1;
    const uint32_t sk = (uint32_t)g.sk;
    const double dxi = g.dxi, dyi = g.dyi, dzi = g.dzi, halfg = P.halfg;
    const double* prt = Sprev.cons + g.ncell;
    const double* srt = Sst.cons + g.ncell;
    const R* Ft = Fcons + g.ncell;
    auto th = [&](int ii, int jj, int kk) { return ccw(A.prim, g, ii, jj, kk); };
    auto prev_mz = [&](int k, Elem f) {
        if (prev_rt && (k == 0 || k == nz)) return T.bnd[(k == 0 ? 0 : g.sk) + (int64_t)j * g.nx + i];
        return Sprev.mz[f];
    };
    // ---- phase 1: horizontal fluxes (cells), Omega'' of the old increments, the new increments' part of
    // Omega'' and the coefficients (faces)
    if (ok) {
        for (int k = w0; k <= nz; k += nw) {
            const Elem f = eidx(g, i, j, k), fx = eidx(g, ip, j, k), fy = eidx(g, i, jp, k);
            const int s = k * TX + L;
            double du = 0.0, dup = 0.0, dv = 0.0, dvp = 0.0;
            if (k < nz) {
                du = double(ld(T.ndu, f)); dup = double(ld(T.ndu, fx));
                dv = double(ld(T.ndv, f)); dvp = double(ld(T.ndv, fy));
                const double xl = du * hzeta_I(P, i, j, k), xh = dup * hzeta_I(P, i + 1, j, k);
                const double yl = dv * hzeta_J(P, i, j, k), yh = dvp * hzeta_J(P, i, j + 1, k);
                const double tc = th(i, j, k);
                sT0[s] = (xh - xl) * dxi + (yh - yl) * dyi;
                sT1[s] = ((xh * (tc + th(i + 1, j, k)) - xl * (tc + th(i - 1, j, k))) * dxi +
                          (yh * (tc + th(i, j + 1, k)) - yl * (tc + th(i, j - 1, k))) * dyi) * 0.5;
            }
            double om = 0.0, an = 0.0;
            if (k > 0) {
                om = prev_mz(k, f) - ld(Sst.mz, f);
                if (k < nz) {
                    const double mx = zlo_xi(P, i, j, k), my = zlo_eta(P, i, j, k);
                    an = mx * (0.25 * (double(ld(T.ndu, f - sk)) + double(ld(T.ndu, fx - sk)) + du + dup)) +
                         my * (0.25 * (double(ld(T.ndv, f - sk)) + double(ld(T.ndv, fy - sk)) + dv + dvp));
                    om -= mx * (0.25 * (double(ld(T.odu, f - sk)) + double(ld(T.odu, fx - sk)) + double(ld(T.odu, f)) + double(ld(T.odu, fx)))) +
                          my * (0.25 * (double(ld(T.odv, f - sk)) + double(ld(T.odv, fy - sk)) + double(ld(T.odv, f)) + double(ld(T.odv, fy))));
                }
            }
            sO[s] = om;
            sN[s] = an;
            sE[s] = double(ld(cf.E, f));
            sG[s] = double(ld(cf.G, f));
        }
    }
    __syncthreads();
    // ---- phase 2: the detJ-weighted right-hand side of the Omega'' system (faces)
    if (ok) {
        for (int k = w0; k <= nz; k += nw) {
            const Elem f = eidx(g, i, j, k);
            const int s = k * TX + L;
            double rhs = dtau * double(ld(Fmz, f));
            if (k > 0 && k < nz) {
                const Elem cm = f - sk;
                const double Jk = detJ_at(P, i, j, k), Jkm = detJ_at(P, i, j, k - 1), dJk = 0.5 * (Jk + Jkm);
                const double cPk = double(ld(cf.P, f)), cQk = double(ld(cf.Q, f));
                const double t_2 = th(i, j, k - 2), t_1 = th(i, j, k - 1), t0 = th(i, j, k), t1 = th(i, j, k + 1);
                const double tlo = 0.5 * (t_2 + t_1), tmid = 0.5 * (t_1 + t0), thi = 0.5 * (t0 + t1);
                const double odr_k = Sprev.cons[f] - ld(Sst.cons, f), odr_km = Sprev.cons[cm] - ld(Sst.cons, cm);
                const double odrt_k = prt[f] - ld(srt, f), odrt_km = prt[cm] - ld(srt, cm);
                double R0t = (-halfg * odr_k + cPk * odrt_k) * Jk + (-halfg * odr_km + cQk * odrt_km) * Jkm;
                double R1t = -halfg * (double(ld(Fcons, f)) * Jk + double(ld(Fcons, cm)) * Jkm)
                             + (cPk * double(ld(Ft, f)) * Jk + cQk * double(ld(Ft, cm)) * Jkm);
                const double Okp1 = sO[s + TX], Ok = sO[s], Okm1 = sO[s - TX];
                R1t += halfg * (beta_1 * dzi * (Okp1 - Okm1) + sT0[s] + sT0[s - TX]);
                R1t += -(cPk * (beta_1 * dzi * (Okp1 * thi - Ok * tmid) + sT1[s]) +
                         cQk * (beta_1 * dzi * (Ok * tmid - Okm1 * tlo) + sT1[s - TX]));
                const double odw = prev_mz(k, f) - ld(Sst.mz, f);
                rhs = dJk * (odw - sN[s]) + dtau * (dJk * double(ld(Fmz, f)) + R0t + dtau * beta_2 * R1t);
            }
            sR[s] = rhs * double(ld(cf.I, f));
        }
    }
    __syncthreads();
    // ---- phase 3: elimination from both walls, one warp each, then back
    const bool solver = ok && w0 < 2, up = w0 == 0;
    if (solver) {
        const int dk = up ? TX : -TX, n = up ? m : nz - m;
        int p = (up ? 0 : nz * TX) + L;
        double s = sR[p];
#pragma unroll 8
        for (int q = 1; q < n; ++q) {
            p += dk;
            s = sR[p] - sE[p] * s;
            sR[p] = s;
        }
    }
    __syncthreads();
    if (solver && up) {
        const int p = m * TX + L;
        sR[p] = sR[p] - sE[p] * sR[p - TX] - sG[p] * sR[p + TX];
    }
    __syncthreads();
    if (solver) {
        const int dk = up ? -TX : TX, n = up ? m : nz - m;
        int p = m * TX + L;
        double s = sR[p];
#pragma unroll 8
        for (int q = 0; q < n; ++q) {
            p += dk;
            s = sR[p] - sG[p] * s;
            sR[p] = s;
        }
    }
    __syncthreads();
    // ---- phase 4: w'' from Omega'', vertical fluxes, average Omega, rho and rho*theta
    if (ok) {
        for (int k = w0; k <= nz; k += nw) {
            const Elem c = eidx(g, i, j, k);
            const int s = k * TX + L;
            double mz = ld(Sst.mz, c);
            if (k >= 1 && k <= nz - 1) mz += sR[s] + sN[s];
            out_mz[c] = mz;
            if (k == nz) continue;
            const double zl = beta_2 * sR[s] + beta_1 * sO[s], zh = beta_2 * sR[s + TX] + beta_1 * sO[s + TX];
            avz[c] += R(facinv * zl);
            if (k == nz - 1) avz[c + sk] += R(facinv * zh);
            const double iJ = inv_detJ(P, i, j, k), tc = th(i, j, k);
            const double frho = -(sT0[s] + (zh - zl) * dzi) * iJ;
            const double frt = -(sT1[s] + 0.5 * (zh * (tc + th(i, j, k + 1)) - zl * (tc + th(i, j, k - 1))) * dzi) * iJ;
            const double pt = prt[c];
            out_cons[c] = Sprev.cons[c] + dtau * (double(ld(Fcons, c)) + frho);
            const double nrt = pt + dtau * (double(ld(Ft, c)) + frt);
            out_cons[g.ncell + c] = nrt;
            // the next substep's extrapolation: d + 0.1 (d - previous d) about the stage
            T.ec[c] = (nrt - ld(srt, c)) + 0.1 * (nrt - pt);
        }
    }
}

namespace {
size_t ter_smem(int nz, int tx, int arrays) { return (size_t)arrays * (nz + 1) * tx * sizeof(double); }
constexpr int TER_COL_ARRAYS = 7, TER_COEF_ARRAYS = 3, TER_VERT_THREADS = 512;
}  // namespace

// ec_ready: the previous substep left the extrapolated d(rho theta) and its
// increments (T.odu, T.odv); else both come from Sprev and lag_in.
template <class R>
void launch_ter_fast_h(const Params& P, cudaStream_t st, int step, bool ec_ready, double dtau, double facinv,
                       StateBuf Sprev, StateBuf Sst, StageAux<R> A, const R* Fmx, const R* Fmy, const R* lag_in,
                       R* lag_out, TerBuf<R> T, R* avx, R* avy, double* outx, double* outy) {
    (ec_ready ? k_ter_fast_h<R, false> : k_ter_fast_h<R, true>)<<<ter_grid(P.g, P.g.nz), ter_block(), 0, st>>>(
        P, step, dtau, facinv, Sprev, Sst, A, Fmx, Fmy, lag_in, lag_out, T, avx, avy, outx, outy);
}
template <class R>
void launch_ter_coef(const Params& P, cudaStream_t st, int tx, double D, StateBuf Sst, StageAux<R> A, MtCoef<R> c) {
    k_ter_coef<R><<<(unsigned)((P.g.sk + tx - 1) / tx), dim3(tx, 256 / tx), ter_smem(P.g.nz, tx, TER_COEF_ARRAYS), st>>>(
        P, D, Sst, A, c);
}
template <class R>
void launch_ter_fast_vert(const Params& P, cudaStream_t st, int tx, double dtau, double facinv, double beta_1,
                          double beta_2, StateBuf Sprev, int prev_rt, StateBuf Sst, StageAux<R> A, const R* Fcons,
                          const R* Fmz, TerBuf<R> T, MtCoef<R> c, R* avz, double* out_cons, double* out_mz) {
    if (prev_rt)
        k_ter_fv_bnd<R><<<dim3((P.g.nx + 31) / 32, (P.g.ny + 3) / 4, 1), ter_block(), 0, st>>>(P, Sprev, T);
    k_ter_fast_vert<R><<<(unsigned)((P.g.sk + tx - 1) / tx), dim3(tx, TER_VERT_THREADS / tx),
                         ter_smem(P.g.nz, tx, TER_COL_ARRAYS), st>>>(P, dtau, facinv, beta_1, beta_2, Sprev, prev_rt, Sst,
                                                                     A, Fcons, Fmz, T, c, avz, out_cons, out_mz);
}
// Columns per block: the widest power of two up to 32 of which two blocks
// share an SM (down to 8: narrower rows waste the rest of their lines), or
// that fits at all; 0 if none does.
template <class R>
int ter_vert_shape(int nz, int* tx) {
    int dev = 0, maxopt = 0, persm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&maxopt, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    cudaDeviceGetAttribute(&persm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev);
    int t = 32;
    while (t > 8 && 2 * (ter_smem(nz, t, TER_COL_ARRAYS) + 1024) > (size_t)persm) t /= 2;
    while (t >= 1 && ter_smem(nz, t, TER_COL_ARRAYS) > (size_t)maxopt) t /= 2;
    *tx = t;
    if (t < 1) return 0;
    return cudaFuncSetAttribute(k_ter_fast_vert<R>, cudaFuncAttributeMaxDynamicSharedMemorySize, maxopt) != cudaSuccess ||
           cudaFuncSetAttribute(k_ter_coef<R>, cudaFuncAttributeMaxDynamicSharedMemorySize, maxopt) != cudaSuccess;
}

#define ERFB_TERF_INSTANTIATE(R)                                                                                    \
    template int ter_vert_shape<R>(int, int*);                                                                      \
    template void launch_ter_coef<R>(const Params&, cudaStream_t, int, double, StateBuf, StageAux<R>, MtCoef<R>);   \
    template void launch_ter_fast_h<R>(const Params&, cudaStream_t, int, bool, double, double, StateBuf, StateBuf,  \
                                       StageAux<R>, const R*, const R*, const R*, R*, TerBuf<R>, R*, R*, double*,   \
                                       double*);                                                                    \
    template void launch_ter_fast_vert<R>(const Params&, cudaStream_t, int, double, double, double, double,         \
                                          StateBuf, int, StateBuf, StageAux<R>, const R*, const R*, TerBuf<R>,      \
                                          MtCoef<R>, R*, double*, double*);
ERFB_TERF_INSTANTIATE(double)
ERFB_TERF_INSTANTIATE(float)
#undef ERFB_TERF_INSTANTIATE

}  // namespace erfb
