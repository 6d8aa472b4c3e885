// substep.cu -- the acoustic substep on a flat grid (erf_fast_rhs_N,
// TimeIntegration/ERF_fast_rhs_N.cpp:115-592, with make_fast_coeffs,
// ERF_make_fast_coeffs.cpp:160-290): one kernel per substep and one kernel
// per stage for its coefficients.
//
// Between the substeps of a stage the fast variables are carried as
// deviations from the stage state: d(rho), d(rho theta) in FP64, the momentum
// increments U'', V'', W'' and the extrapolated d(rho theta) in the bulk type
// (the increments are formed in it each substep in any case).  The first
// substep forms the deviations from the old and stage states, the last one
// writes the whole state.  The momentum -> velocity -> momentum round trips
// of the reference's fills between substeps are the identity but for
// rounding and are not applied.
//
// With X = d(rho theta) + dtau b2 G1 and Y = d(rho) + dtau b2 G0 per cell,
// where G0, G1 are the tendencies of rho and rho theta less the fluxes of the
// new U'', V'' and b1 times those of the old W'', the right-hand side of the
// W'' system on face k is
//   W'' + dtau (F_rw + P X_k + Q X_{k-1} - g/2 (Y_k + Y_{k-1})),
// the reference's expression with its terms collected per cell.
//
// Bound: HBM.  A substep forces 31 bulk-sized values per cell (22 read, 9
// written) against 44 of the horizontal and vertical kernels that this one
// replaces (moist bubble 128x128x80, FP64: 45 + 107 us per substep, 105 now).
#include "kernels.cuh"

namespace erfb {
namespace {

// A tile is TX consecutive columns of the plane (rows run on, so that every
// lane has a column whatever nx is); the block's rows share the levels.
struct ColTile {
    int tx, L, w, nw, col, xm, xp, ym, yp;
    bool ok;
    __device__ __forceinline__ ColTile(const Geo& g) {
        tx = blockDim.x; L = threadIdx.x; w = threadIdx.y; nw = blockDim.y;
        col = blockIdx.x * tx + L;
        ok = col < (int)g.sk;
        const int c = ok ? col : 0, j = c / g.nx, i = c - j * g.nx;
        col = c;
        xm = i > 0 ? c - 1 : c + g.nx - 1;
        xp = i < g.nx - 1 ? c + 1 : c - g.nx + 1;
        ym = j > 0 ? c - g.nx : c + (g.ny - 1) * g.nx;
        yp = j < g.ny - 1 ? c + g.nx : c - (g.ny - 1) * g.nx;
    }
};

// Offset of level k.
__device__ __forceinline__ Elem lev(const Geo& g, int k) { return eidx(g, 0, 0, k); }

// The stage's coefficients.  Per x / y face: the factor of the pressure
// gradient of the extrapolated d(rho theta).  Per z face: P and Q, and the
// factors of the W'' system eliminated from both walls towards face m = nz/2
// (each half is a Thomas elimination; the two run side by side, so the
// serial chain is half as long): I = 1 / pivot, E = the eliminated side's
// coefficient times I, G = the other side's times I (back substitution); on
// face m, E and G are the two sides' coefficients times I.
template <class R>
__global__ void k_sub_coef(Params P, double D_d, StateBuf Sst, StageAux<R> A, R* __restrict__ fx, R* __restrict__ fy,
                           R* __restrict__ cE, R* __restrict__ cG, R* __restrict__ cI, R* __restrict__ cP,
                           R* __restrict__ cQ) {
    extern __shared__ __align__(16) unsigned char sm_raw[];
    const Geo& g = P.g;
    const ColTile t(g);
    const int nz = g.nz, TX = t.tx, L = t.L, m = nz / 2;
    R* sA = reinterpret_cast<R*>(sm_raw);
    R* sB = sA + (nz + 1) * TX;
    R* sC = sB + (nz + 1) * TX;
    const int64_t N = g.ncell, sk = g.sk;
    const R D = R(D_d), halfg = R(P.halfg);
    const R* __restrict__ th = A.prim;
    if (t.ok) {
        for (int k = t.w; k < nz; k += t.nw) {
            const Elem o = lev(g, k);
            const R pc = A.pi[o + t.col];
            R gx = R(-Gamma_ * R_d) * (R(0.5) * (A.pi[o + t.xm] + pc)) * R(g.dxi);
            R gy = R(-Gamma_ * R_d) * (R(0.5) * (A.pi[o + t.ym] + pc)) * R(g.dyi);
            R q = R(0), qm = R(0);
            if (P.moist) {
                const R* qv = th + 4 * N;
                const R* qc = th + 5 * N;
                q = qv[o + t.col] + qc[o + t.col];
                gx /= R(1) + R(0.5) * (q + qv[o + t.xm] + qc[o + t.xm]);
                gy /= R(1) + R(0.5) * (q + qv[o + t.ym] + qc[o + t.ym]);
                if (k > 0) qm = qv[o + t.col - sk] + qc[o + t.col - sk];
            }
            fx[o + t.col] = gx;
            fy[o + t.col] = gy;
            if (k == 0) continue;
            const Elem c = o + t.col, cm = c - sk;
            const R pi_c = R(0.5) * (A.pi[cm] + pc);
            R P_ = R(-Gamma_ * R_d * g.dzi + P.halfg * R_d * P.r0[k + 1] / (P.c_v * P.pi0[k + 1] * Sst.cons[N + c]));
            R Q_ = R(Gamma_ * R_d * g.dzi + P.halfg * R_d * P.r0[k] / (P.c_v * P.pi0[k] * Sst.cons[N + cm]));
            P_ *= pi_c;
            Q_ *= pi_c;
            if (P.moist) {
                const R wet = R(1) + R(0.5) * (q + qm);
                P_ /= wet;
                Q_ /= wet;
            }
            const R tc = th[c], tm = th[cm];
            const R tlo = R(0.5) * (th[lev(g, k > 1 ? k - 2 : 0) + t.col] + tm);
            const R thi = R(0.5) * (tc + th[lev(g, k < nz - 1 ? k + 1 : k) + t.col]);
            sA[k * TX + L] = D * (halfg - Q_ * tlo);
            sB[k * TX + L] = R(1) + D * (Q_ - P_) * (R(0.5) * (tm + tc));
            sC[k * TX + L] = D * (-halfg + P_ * thi);
            cP[c] = P_;
            cQ[c] = Q_;
        }
        if (t.w == 0)
            for (int k : {0, nz}) {
                sA[k * TX + L] = R(0); sB[k * TX + L] = R(1); sC[k * TX + L] = R(0);
                const Elem f = lev(g, k) + t.col;
                cP[f] = R(0); cQ[f] = R(0);
            }
    }
    __syncthreads();
    // pivots: sB <- I, and the other side's coefficient times I (sC below m, sA above)
    if (t.ok && t.w < 2) {
        const bool up = t.w == 0;
        const int k0 = up ? 0 : nz, dk = up ? 1 : -1, n = up ? m : nz - m;
        R* elim = up ? sA : sC;
        R* keep = up ? sC : sA;
        R gam = R(0);
        for (int q = 0, k = k0; q < n; ++q, k += dk) {
            const R bet = sB[k * TX + L] - elim[k * TX + L] * gam;
            if (!(fabs(double(bet)) > 1e-300)) atomicOr(P.status, ST_BADSTATE);
            const R inv = R(1) / bet;
            gam = keep[k * TX + L] * inv;
            sB[k * TX + L] = inv;
            keep[k * TX + L] = gam;
        }
    }
    __syncthreads();
    if (t.ok) {
        for (int k = t.w; k <= nz; k += t.nw) {
            const int s = k * TX + L;
            R inv = sB[s], e, gm;
            if (k == m) {
                const R bet = sB[s] - sA[s] * sC[s - TX] - sC[s] * sA[s + TX];
                if (!(fabs(double(bet)) > 1e-300)) atomicOr(P.status, ST_BADSTATE);
                inv = R(1) / bet;
                e = sA[s] * inv;
                gm = sC[s] * inv;
            } else {
                e = (k < m ? sA[s] : sC[s]) * inv;
                gm = k < m ? sC[s] : sA[s];
            }
            const Elem f = lev(g, k) + t.col;
            cI[f] = inv;
            cE[f] = e;
            cG[f] = gm;
        }
    }
}

// One substep.  MODE 0: the deviations are zero (the first stage starts from
// its own state; no pressure gradient there, as in the reference); 1: they
// are old - stage; 2: they are stored.  LAST: the whole state is written.
//
//   phase 1  (cells)  new U'', V'' on the cell's four faces (its neighbours
//                     form the shared ones again: the loads hit L1 / L2 and
//                     cost less than a pass that writes and reads them), the
//                     cell's G0, G1 and X, Y
//   phase 2  (faces)  right-hand side of the W'' system
//   phase 3           elimination from both walls, one warp each, then back
//   phase 4  (cells)  W'', average momenta, rho and rho theta
//
// G0 and G1 are not kept: phase 4 recovers dtau G0 = (Y - d rho) / b2 from Y
// in FP64.  With X, Y in FP64 and three bulk arrays in shared memory, two
// FP64 blocks of 32 columns x 80 levels share an SM and one block's serial
// sweep runs under the other's loads.
template <class R, int MODE, bool LAST>
__global__ void __launch_bounds__(1024) k_substep(Params P, SubArgs<R> a) {
    extern __shared__ __align__(16) unsigned char sm_raw[];
    const Geo& g = P.g;
    const ColTile t(g);
    const int nz = g.nz, TX = t.tx, L = t.L, m = nz / 2;
    double* sX = reinterpret_cast<double*>(sm_raw);
    double* sY = sX + nz * TX;
    R* sS = reinterpret_cast<R*>(sY + nz * TX);
    R* sE = sS + (nz + 1) * TX;
    R* sG = sE + (nz + 1) * TX;
    const uint32_t sk = (uint32_t)g.sk, c0 = t.col;
    const R* th = a.th;
    const R dxi = R(g.dxi), dyi = R(g.dyi), dzi = R(g.dzi);
    const R dtau = R(a.dtau), b1 = R(a.b1), b2 = R(a.b2), c2 = dtau * b2, b1z = b1 * dzi;
    const double* ort = a.old.cons + g.ncell;
    const double* srt = a.st.cons + g.ncell;
    const bool av_init = MODE == 0 || (MODE == 1 && a.av_init), grad = MODE == 2 || (MODE == 1 && a.grad);
    // deviations of cell / face c
    auto dev_rt = [&](Elem c) -> double {
        if (MODE == 0) return 0.0;
        if (MODE == 1) return ld(ort, c) - ld(srt, c);
        return at(a.drt, c);
    };
    auto dev_r = [&](Elem c) -> double {
        if (MODE == 0) return 0.0;
        if (MODE == 1) return ld(a.old.cons, c) - ld(a.st.cons, c);
        return at(a.dr, c);
    };
    auto dev_m = [&](const double* old, const double* st, const R* dev, Elem f) -> R {
        if (MODE == 0) return R(0);
        if (MODE == 1) return R(ld(old, f) - ld(st, f));
        return ld(dev, f);
    };
    auto dev_w = [&](Elem f) -> R { return dev_m(a.old.mz, a.st.mz, a.wi, f); };
    auto ext = [&](Elem c) -> R {   // extrapolated d(rho theta)
        if (MODE == 2) return ld(a.ei, c);
        const R d = R(dev_rt(c));
        return a.lag_in ? d + R(0.1) * (d - ld(a.lag_in, c)) : d;
    };
    // ---- phase 1
    if (t.ok) {
#pragma unroll 1
        for (int k = t.w; k < nz; k += t.nw) {
            const Elem o = lev(g, k), c = o + c0, xm = o + t.xm, xp = o + t.xp, ym = o + t.ym, yp = o + t.yp;
            R xl = ld(a.Fmx, c), xh = ld(a.Fmx, xp), yl = ld(a.Fmy, c), yh = ld(a.Fmy, yp);
            if (grad) {
                const R ec = ext(c);
                xl += ld(a.fx, c) * (ec - ext(xm));
                xh += ld(a.fx, xp) * (ext(xp) - ec);
                yl += ld(a.fy, c) * (ec - ext(ym));
                yh += ld(a.fy, yp) * (ext(yp) - ec);
            }
            xl = dev_m(a.old.mx, a.st.mx, a.ui, c) + dtau * xl;
            xh = dev_m(a.old.mx, a.st.mx, a.ui, xp) + dtau * xh;
            yl = dev_m(a.old.my, a.st.my, a.vi, c) + dtau * yl;
            yh = dev_m(a.old.my, a.st.my, a.vi, yp) + dtau * yh;
            const R tc = ld(th, c);
            const R t0 = (xh - xl) * dxi + (yh - yl) * dyi;
            const R t1 = ((xh * (tc + ld(th, xp)) - xl * (tc + ld(th, xm))) * dxi +
                          (yh * (tc + ld(th, yp)) - yl * (tc + ld(th, ym))) * dyi) * R(0.5);
            R G0 = ld(a.Fr, c) - t0, G1 = ld(a.Ft, c) - t1;
            if (MODE != 0) {
                const R wl = dev_w(c), wh = dev_w(c + sk);
                const R tl = R(0.5) * (tc + ld(th, k > 0 ? c - sk : c));
                const R tu = R(0.5) * (tc + ld(th, k < nz - 1 ? c + sk : c));
                G0 -= b1z * (wh - wl);
                G1 -= b1z * (wh * tu - wl * tl);
            }
            const double dr = dev_r(c), drt = dev_rt(c);
            sY[k * TX + L] = dr + double(c2 * G0);
            sX[k * TX + L] = drt + double(c2 * G1);
            if (MODE == 1 && a.lag_out) at(a.lag_out, c) = R(drt);
            const R ax = av_init ? R(ld(a.st.mx, c)) : at(a.avx, c), ay = av_init ? R(ld(a.st.my, c)) : at(a.avy, c);
            at(a.avx, c) = ax + R(a.facinv) * xl;
            at(a.avy, c) = ay + R(a.facinv) * yl;
            if (LAST) {
                at(a.sum.mx, c) = ld(a.st.mx, c) + double(xl);
                at(a.sum.my, c) = ld(a.st.my, c) + double(yl);
            } else {
                at(a.uo, c) = xl;
                at(a.vo, c) = yl;
            }
        }
    }
    __syncthreads();
    // ---- phase 2
    if (t.ok) {
        const R halfg = R(P.halfg);
#pragma unroll 2
        for (int k = t.w; k <= nz; k += t.nw) {
            const Elem f = lev(g, k) + c0;
            const int s = k * TX + L;
            R r = ld(a.Fmz, f);
            if (k > 0 && k < nz) {
                const R xk = R(sX[s]), xm = R(sX[s - TX]), yk = R(sY[s]), ym = R(sY[s - TX]);
                r += ld(a.cP, f) * xk + ld(a.cQ, f) * xm - halfg * (yk + ym);
            }
            sS[s] = (dev_w(f) + dtau * r) * ld(a.cI, f);
            sE[s] = ld(a.cE, f);
            sG[s] = ld(a.cG, f);
        }
    }
    __syncthreads();
    // ---- phase 3: eight levels at a time, so that their loads are in flight together
    constexpr int CH = 8;
    const bool solver = t.ok && t.w < 2;
    const int up = t.w == 0;
    if (solver) {
        const int dk = up ? TX : -TX, n = up ? m : nz - m;   // faces eliminated: the wall's first
        int p = (up ? 0 : nz * TX) + L;
        R s = sS[p];
        p += dk;
        for (int q = 1; q < n; q += CH) {
            R v[CH], e[CH];
#pragma unroll
            for (int u = 0; u < CH; ++u)
                if (q + u < n) { v[u] = sS[p + u * dk]; e[u] = sE[p + u * dk]; }
#pragma unroll
            for (int u = 0; u < CH; ++u)
                if (q + u < n) { s = v[u] - e[u] * s; sS[p + u * dk] = s; }
            p += CH * dk;
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
        R s = sS[p];
        p += dk;
        for (int q = 0; q < n; q += CH) {
            R v[CH], e[CH];
#pragma unroll
            for (int u = 0; u < CH; ++u)
                if (q + u < n) { v[u] = sS[p + u * dk]; e[u] = sG[p + u * dk]; }
#pragma unroll
            for (int u = 0; u < CH; ++u)
                if (q + u < n) { s = v[u] - e[u] * s; sS[p + u * dk] = s; }
            p += CH * dk;
        }
    }
    __syncthreads();
    // ---- phase 4
    if (t.ok) {
        const double ib2 = 1.0 / a.b2;
#pragma unroll 1
        for (int k = t.w; k < nz; k += t.nw) {
            const Elem c = lev(g, k) + c0;
            const int s = k * TX + L;
            const R sl = sS[s], sh = sS[s + TX];
            const R wl = dev_w(c), wh = dev_w(c + sk);
            const R zl = b2 * sl + b1 * wl;
            auto avz = [&](Elem f, R z) {
                at(a.avz, f) = (av_init ? R(ld(a.st.mz, f)) : at(a.avz, f)) + R(a.facinv) * z;
            };
            avz(c, zl);
            if (k == nz - 1) avz(c + sk, b2 * sh + b1 * wh);
            const R tc = ld(th, c);
            const R tl = R(0.5) * (tc + ld(th, k > 0 ? c - sk : c));
            const R tu = R(0.5) * (tc + ld(th, k < nz - 1 ? c + sk : c));
            const double dr = dev_r(c), drt = dev_rt(c);
            const double nr = dr + ((sY[s] - dr) * ib2 - double(c2 * dzi * (sh - sl)));
            const double nrt = drt + ((sX[s] - drt) * ib2 - double(c2 * dzi * (sh * tu - sl * tl)));
            if (LAST) {
                at(a.sum.cons, c) = ld(a.st.cons, c) + nr;
                at(a.sum.cons + g.ncell, c) = ld(srt, c) + nrt;
                at(a.sum.mz, c) = ld(a.st.mz, c) + double(sl);
                if (k == nz - 1) at(a.sum.mz, c + sk) = ld(a.st.mz, c + sk) + double(sh);
            } else {
                at(a.dr, c) = nr;
                at(a.drt, c) = nrt;
                at(a.eo, c) = R(nrt) + R(0.1) * (R(nrt) - R(drt));
                at(a.wo, c) = sl;
                if (k == nz - 1) at(a.wo, c + sk) = sh;
            }
        }
    }
}

template <class R>
using SubK = void (*)(Params, SubArgs<R>);
template <class R>
SubK<R> sub_kernel(int mode, bool last) {
    if (mode == 0) return last ? k_substep<R, 0, true> : k_substep<R, 0, false>;
    if (mode == 1) return last ? k_substep<R, 1, true> : k_substep<R, 1, false>;
    return last ? k_substep<R, 2, true> : k_substep<R, 2, false>;
}
}  // namespace

template <class R>
size_t sub_smem(int nz, int tx) {
    return (size_t)tx * (2 * (size_t)nz * sizeof(double) + 3 * (size_t)(nz + 1) * sizeof(R));
}
template <class R>
size_t sub_coef_smem(int nz, int tx) {
    return (size_t)3 * (nz + 1) * tx * sizeof(R);
}

// Columns per block: the widest tile of which two blocks share an SM, so that
// one block's serial sweep runs under the other's loads (a row of 8 FP64
// values is two sectors: narrower tiles waste the rest of each line).
template <class R>
SubShape sub_shape(const Geo& g) {
    int dev = 0, nsm = 148, maxopt = 0, persm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    cudaDeviceGetAttribute(&maxopt, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    cudaDeviceGetAttribute(&persm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev);
    SubShape s;
    s.tx = 32;
    while (s.tx > 8 && 2 * (sub_smem<R>(g.nz, s.tx) + 1024) > (size_t)persm) s.tx /= 2;
    while (s.tx > 2 && sub_smem<R>(g.nz, s.tx) > (size_t)maxopt) s.tx /= 2;
    // small planes: narrower tiles while they leave half the SMs without one
    while (s.tx > 8 && 2 * ((g.sk + s.tx - 1) / s.tx) <= nsm) s.tx /= 2;
    // few blocks: all the threads an SM takes; more than one per SM: half each;
    // never more rows than levels
    const int64_t blocks = (g.sk + s.tx - 1) / s.tx;
    s.rows = (blocks <= nsm ? 1024 : 512) / s.tx;
    while (s.rows > 8 && s.rows / 2 > g.nz) s.rows /= 2;
    s.coef_rows = 256 / s.tx;
    return s;
}
// The dynamic shared-memory opt-in is a property of the kernel for the whole
// process, so it is raised to the device maximum for all contexts.
template <class R>
int sub_setup(const Geo& g, const SubShape& s) {
    int dev = 0, maxopt = 0;
    cudaGetDevice(&dev);
    if (cudaDeviceGetAttribute(&maxopt, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess) return 1;
    if (sub_smem<R>(g.nz, s.tx) > (size_t)maxopt || sub_coef_smem<R>(g.nz, s.tx) > (size_t)maxopt) return 1;
    for (int mode = 0; mode < 3; ++mode)
        for (int last = 0; last < 2; ++last)
            if (cudaFuncSetAttribute(sub_kernel<R>(mode, last), cudaFuncAttributeMaxDynamicSharedMemorySize, maxopt) !=
                cudaSuccess)
                return 1;
    return cudaFuncSetAttribute(k_sub_coef<R>, cudaFuncAttributeMaxDynamicSharedMemorySize, maxopt) != cudaSuccess;
}
template <class R>
void launch_sub_coef(const Params& P, cudaStream_t st, const SubShape& s, double D, StateBuf Sst, StageAux<R> A,
                     const SubCoef<R>& c) {
    k_sub_coef<R><<<(unsigned)((P.g.sk + s.tx - 1) / s.tx), dim3(s.tx, s.coef_rows), sub_coef_smem<R>(P.g.nz, s.tx),
                    st>>>(P, D, Sst, A, c.fx, c.fy, c.E, c.G, c.I, c.P, c.Q);
}
template <class R>
void launch_substep(const Params& P, cudaStream_t st, const SubShape& s, int mode, bool last, const SubArgs<R>& a) {
    sub_kernel<R>(mode, last)<<<(unsigned)((P.g.sk + s.tx - 1) / s.tx), dim3(s.tx, s.rows), sub_smem<R>(P.g.nz, s.tx),
                                st>>>(P, a);
}

#define ERFB_SUB_INSTANTIATE(R)                                                                                     \
    template SubShape sub_shape<R>(const Geo&);                                                                     \
    template int sub_setup<R>(const Geo&, const SubShape&);                                                         \
    template void launch_sub_coef<R>(const Params&, cudaStream_t, const SubShape&, double, StateBuf, StageAux<R>,   \
                                     const SubCoef<R>&);                                                            \
    template void launch_substep<R>(const Params&, cudaStream_t, const SubShape&, int, bool, const SubArgs<R>&);
ERFB_SUB_INSTANTIATE(double)
ERFB_SUB_INSTANTIATE(float)
#undef ERFB_SUB_INSTANTIATE

}  // namespace erfb
