// kernels.cu -- dycore kernels for sm_100a.
//
// Each kernel fuses one or more of the reference's AMReX ParallelFor passes
// (file:line cited per kernel).  Lateral neighbours are addressed through
// periodic index wrapping and vertical ghost values through the wall
// conditions, so no separate ghost-fill pass is launched between stages and
// substeps; the reference's momentum<->velocity round trips at every boundary
// fill (BoundaryConditions/ERF_FillIntermediatePatch.cpp:63-67, 224-236) are
// the identity but for rounding (two divisions and an ulp each) and are not
// applied (but by k_ter_step_begin, terrain.cu).
//
// The dycore kernels are templates on R, the type of the bulk arrays (derived
// fields, slow right-hand sides, average momenta, fast coefficients, stresses)
// and of the arithmetic on them: R = double is the plain FP64 form, R = float
// the mixed form.  The prognostic state (conserved variables, momenta,
// between-step velocities), the base state and the equation of state stay
// FP64 in both, and every update of the state is accumulated in FP64.
#include <cfloat>

#include "kernels.cuh"
#include "tiles.cuh"

namespace erfb {

// ---------------------------------------------------------------------------
// Accessors with boundary conditions
// ---------------------------------------------------------------------------
// Tangential velocity at (i,j,k), i,j already wrapped; below/above the walls
// the ghost value is 0 (no-slip, ext_dir) or the nearest interior value
// (slip, foextrap): ERF_BoundaryConditions_xvel.cpp:190-230.
__device__ __forceinline__ double tang(const double* __restrict__ f, const Geo& g, int i, int j, int k) {
    if (k < 0) return g.zlo_noslip ? 0.0 : ld(f, eidx(g, i, j, 0));
    if (k >= g.nz) return g.zhi_noslip ? 0.0 : ld(f, eidx(g, i, j, g.nz - 1));
    return ld(f, eidx(g, i, j, k));
}
// ---------------------------------------------------------------------------
// MOST ground (ABLMost::compute_most_bcs with moeng_flux, implicit MOST,
// BoundaryConditions/ERF_ABLMost.cpp:289-489, ERF_MOSTStress.H:1395-1555):
// the tangential velocity d levels below the ground is the level-0 value plus
// tau / eta * dz * d, with the Moeng stress from the level-0 velocities, the
// step's plane means and u*, and eta the level-0 eddy viscosity averaged to
// the face (floored at 1e-8).  The stage boundary fills impose it, so the
// readers of stage velocities evaluate it where they reach below the ground.
// ---------------------------------------------------------------------------
__device__ __forceinline__ double most_mu(const Params& P, int64_t c) {
    return P.most_mut_f32 ? double(static_cast<const float*>(P.most_mut)[c])
                          : static_cast<const double*>(P.most_mut)[c];
}
__device__ __forceinline__ double most_ghost_u(const Params& P, const double* __restrict__ u,
                                               const double* __restrict__ v, const double* __restrict__ cons, int i,
                                               int j, int d) {
    const Geo& g = P.g;
    const int im = wrap(i - 1, g.nx), jp = wrap(j + 1, g.ny);
    const double velx = u[cidx(g, i, j, 0)];
    const double vely = 0.25 * (v[cidx(g, i, j, 0)] + v[cidx(g, i, jp, 0)] + v[cidx(g, im, j, 0)] + v[cidx(g, im, jp, 0)]);
    const double rho = 0.5 * (cons[cidx(g, im, j, 0)] + cons[cidx(g, i, j, 0)]);
    const double umean = P.most_avg[0];
    double wsp_mean = 0.5 * (P.most_avg[2] + P.most_avg[2]);
    const double ustar = 0.5 * (P.most_avg[3] + P.most_avg[3]);
    const double wsp = sqrt(velx * velx + vely * vely);
    const double num1 = wsp * umean;
    const double num2 = wsp_mean * (velx - umean);
    const double deltaz = P.most_dz * (0 + d);
    wsp_mean = fmax(wsp_mean, 0.1);
    const double stressx = -rho * ustar * ustar * (num1 + num2) / (wsp_mean * wsp_mean);
    double eta = 0.5 * (most_mu(P, cidx(g, im, j, 0)) + most_mu(P, cidx(g, i, j, 0)));
    eta = fmax(eta, 1e-8);
    return velx + stressx / eta * deltaz;
}
__device__ __forceinline__ double most_ghost_v(const Params& P, const double* __restrict__ u,
                                               const double* __restrict__ v, const double* __restrict__ cons, int i,
                                               int j, int d) {
    const Geo& g = P.g;
    const int jm = wrap(j - 1, g.ny), ip = wrap(i + 1, g.nx);
    const double velx = 0.25 * (u[cidx(g, i, j, 0)] + u[cidx(g, ip, j, 0)] + u[cidx(g, i, jm, 0)] + u[cidx(g, ip, jm, 0)]);
    const double vely = v[cidx(g, i, j, 0)];
    const double rho = 0.5 * (cons[cidx(g, i, jm, 0)] + cons[cidx(g, i, j, 0)]);
    const double vmean = P.most_avg[1];
    double wsp_mean = 0.5 * (P.most_avg[2] + P.most_avg[2]);
    const double ustar = 0.5 * (P.most_avg[3] + P.most_avg[3]);
    const double wsp = sqrt(velx * velx + vely * vely);
    const double num1 = wsp * vmean;
    const double num2 = wsp_mean * (vely - vmean);
    const double deltaz = P.most_dz * (0 + d);
    wsp_mean = fmax(wsp_mean, 0.1);
    const double stressy = -rho * ustar * ustar * (num1 + num2) / (wsp_mean * wsp_mean);
    double eta = 0.5 * (most_mu(P, cidx(g, i, jm, 0)) + most_mu(P, cidx(g, i, j, 0)));
    eta = fmax(eta, 1e-8);
    return vely + stressy / eta * deltaz;
}
// Stage velocities with the MOST ghost rule below the ground: the fields a
// stage reader holds (u, v, cons of the stage), none for the other grounds.
struct MostView {
    const double* u;
    const double* v;
    const double* cons;
};
__device__ __forceinline__ double tang_u(const Params& P, const MostView& m, int i, int j, int k) {
    if (k < 0 && P.most) return most_ghost_u(P, m.u, m.v, m.cons, i, j, -k);
    return tang(m.u, P.g, i, j, k);
}
__device__ __forceinline__ double tang_v(const Params& P, const MostView& m, int i, int j, int k) {
    if (k < 0 && P.most) return most_ghost_v(P, m.u, m.v, m.cons, i, j, -k);
    return tang(m.v, P.g, i, j, k);
}


// ---------------------------------------------------------------------------
// Strain-rate components (Diffusion/ERF_ComputeStrain_N.cpp:28-229) with the
// one-sided wall stencils at no-slip walls.  Edge (i,j,k) of an xy/xz/yz edge
// array sits at the low corner of cell (i,j,k).  Velocities are FP64 state;
// the differences are formed in FP64.
// ---------------------------------------------------------------------------
__device__ __forceinline__ double strain12(const double* u, const double* v, const Geo& g, int i, int j, int k) {
    int im = wrap(i - 1, g.nx), jm = wrap(j - 1, g.ny);
    return 0.5 * ((ld(u, eidx(g, i, j, k)) - ld(u, eidx(g, i, jm, k))) * g.dyi +
                  (ld(v, eidx(g, i, j, k)) - ld(v, eidx(g, im, j, k))) * g.dxi);
}
// Stage strain at the ground face of a MOST ground: the centred difference
// with the MOST ghost velocity below
__device__ __forceinline__ double strain13_most(const Params& P, const MostView& m, const double* w, int i, int j) {
    const Geo& g = P.g;
    int im = wrap(i - 1, g.nx);
    double wx = (ld(w, eidx(g, i, j, 0)) - ld(w, eidx(g, im, j, 0))) * g.dxi;
    return 0.5 * ((tang_u(P, m, i, j, 0) - tang_u(P, m, i, j, -1)) * g.dzi + wx);
}
__device__ __forceinline__ double strain23_most(const Params& P, const MostView& m, const double* w, int i, int j) {
    const Geo& g = P.g;
    int jm = wrap(j - 1, g.ny);
    double wy = (ld(w, eidx(g, i, j, 0)) - ld(w, eidx(g, i, jm, 0))) * g.dyi;
    return 0.5 * ((tang_v(P, m, i, j, 0) - tang_v(P, m, i, j, -1)) * g.dzi + wy);
}
__device__ __forceinline__ double strain13(const double* u, const double* w, const Geo& g, int i, int j, int k) {
    int im = wrap(i - 1, g.nx);
    double wx = (ld(w, eidx(g, i, j, k)) - ld(w, eidx(g, im, j, k))) * g.dxi;
    if (k == 0 && g.zlo_noslip)
        return 0.5 * ((-(8. / 3.) * tang(u, g, i, j, k - 1) + 3. * tang(u, g, i, j, k) - (1. / 3.) * tang(u, g, i, j, k + 1)) * g.dzi + wx);
    if (k == g.nz && g.zhi_noslip)
        return 0.5 * (-(-(8. / 3.) * tang(u, g, i, j, k) + 3. * tang(u, g, i, j, k - 1) - (1. / 3.) * tang(u, g, i, j, k - 2)) * g.dzi + wx);
    return 0.5 * ((tang(u, g, i, j, k) - tang(u, g, i, j, k - 1)) * g.dzi + wx);
}
__device__ __forceinline__ double strain23(const double* v, const double* w, const Geo& g, int i, int j, int k) {
    int jm = wrap(j - 1, g.ny);
    double wy = (ld(w, eidx(g, i, j, k)) - ld(w, eidx(g, i, jm, k))) * g.dyi;
    if (k == 0 && g.zlo_noslip)
        return 0.5 * ((-(8. / 3.) * tang(v, g, i, j, k - 1) + 3. * tang(v, g, i, j, k) - (1. / 3.) * tang(v, g, i, j, k + 1)) * g.dzi + wy);
    if (k == g.nz && g.zhi_noslip)
        return 0.5 * (-(-(8. / 3.) * tang(v, g, i, j, k) + 3. * tang(v, g, i, j, k - 1) - (1. / 3.) * tang(v, g, i, j, k - 2)) * g.dzi + wy);
    return 0.5 * ((tang(v, g, i, j, k) - tang(v, g, i, j, k - 1)) * g.dzi + wy);
}

__device__ __forceinline__ bool cell_coords(const Geo& g, int& i, int& j, int& k) {
    i = blockIdx.x * blockDim.x + threadIdx.x;
    j = blockIdx.y * blockDim.y + threadIdx.y;
    k = blockIdx.z;
    return i < g.nx && j < g.ny && k < g.nz;
}

// Whether any pass reads primitive n: KE with Deardorff only, QKE never (no PBL scheme).
__device__ __forceinline__ bool prim_read(const Params& P, int n) {
    return n != ERF_RHOQKE_COMP - 1 && (n != ERF_RHOKE_COMP - 1 || P.les == ERF_LES_DEARDORFF);
}

// Derived stage quantities of one cell: cons_to_prim + pi_stage
// (TimeIntegration/ERF_TI_utils.H:4-45) and p' (ERF_slow_rhs_pre.cpp:337-358),
// evaluated in FP64 from the FP64 state and stored as R.
template <class R>
__device__ __forceinline__ void stage_aux_thermo(const Params& P, double rho, double rt, double ir, double qv, StageAux<R> A,
                                                 int64_t c, int k) {
    A.prim[c] = R(rt * ir);
    const double x = R_d * rt * ip_0, l = log(x);   // of the Exner function, and of p where the air is dry
    A.pi[c] = R(exp(Gamma_ * P.rdOcp * l));
    const double lp = P.moist ? log(x * (1.0 + (R_v / R_d) * qv)) : l;
    A.pp[c] = R(p_0 * exp(Gamma_ * lp) - (P.ter ? P.p0[c + P.g.sk] : P.p0[k + 1]));
    if (!(rt > 0.0) || !(rho > 0.0)) atomicOr(P.status, ST_BADSTATE);
}
template <class R>
__device__ __forceinline__ void stage_aux_cell(const Params& P, const double* __restrict__ cons, StageAux<R> A,
                                               int64_t c, int k) {
    const int64_t N = P.g.ncell;
    const double rho = cons[c], ir = 1.0 / rho;
    for (int n = 1; n < P.nprim; ++n)
        if (prim_read(P, n)) A.prim[n * N + c] = R(cons[(n + 1) * N + c] * ir);
    stage_aux_thermo<R>(P, rho, cons[N + c], ir, P.moist ? cons[5 * N + c] * ir : 0.0, A, c, k);
}

// ---------------------------------------------------------------------------
// Step prologue.  Fuses, for the step's old state:
//   * ComputeStrain_N + ComputeTurbulentViscosityLES (Smagorinsky) from the
//     old velocities (ERF_advance_dycore.cpp:114-223,
//     ERF_ComputeTurbulentViscosity.cpp:85-126; EddyViscosity.H:31-83);
//   * VelocityToMomentum of the old velocities
//     (ERF_advance_dycore.cpp:260-276);
//   * cons_to_prim / pi_stage / p' of the old state.
// ---------------------------------------------------------------------------
template <class R>
__global__ void k_step_begin(Params P, const double* __restrict__ cons, const double* __restrict__ uo,
                             const double* __restrict__ vo, const double* __restrict__ wo, StateBuf S,
                             double* __restrict__ un, double* __restrict__ vn, double* __restrict__ wn,
                             StageAux<R> A, R* __restrict__ mut, TkeBuf<R> tke) {
    const Geo& g = P.g;
    int i, j, k;
    if (!cell_coords(g, i, j, k)) return;
    int im = wrap(i - 1, g.nx), jm = wrap(j - 1, g.ny);
    int64_t c = cidx(g, i, j, k);
    double rho = cons[c];
    {
        double rs = rho + cons[cidx(g, im, j, k)];
        S.mx[c] = (uo[c] * 0.5) * rs; un[c] = uo[c];
    }
    {
        double rs = rho + cons[cidx(g, i, jm, k)];
        S.my[c] = (vo[c] * 0.5) * rs; vn[c] = vo[c];
    }
    if (k == 0) {
        S.mz[c] = 0.0; wn[c] = 0.0;
    } else {
        double rs = rho + cons[cidx(g, i, j, k - 1)];
        S.mz[c] = (wo[c] * 0.5) * rs; wn[c] = wo[c];
    }
    if (k == g.nz - 1) { S.mz[c + g.sk] = 0.0; wn[c + g.sk] = 0.0; }
    // a NaN or infinite velocity in the step's input (the state checks of
    // stage_aux_cell cover rho and rho*theta)
    if (!(fabs(uo[c]) <= DBL_MAX) || !(fabs(vo[c]) <= DBL_MAX) || !(fabs(wo[c]) <= DBL_MAX))
        atomicOr(P.status, ST_NAN);
    stage_aux_cell<R>(P, cons, A, c, k);

    if (P.les == ERF_LES_SMAGORINSKY || P.les == ERF_LES_MLP || P.les == ERF_LES_DEARDORFF) {
        int ip = wrap(i + 1, g.nx), jp = wrap(j + 1, g.ny);
        double s11 = (ld(uo, eidx(g, ip, j, k)) - uo[c]) * g.dxi;
        double s22 = (ld(vo, eidx(g, i, jp, k)) - vo[c]) * g.dyi;
        double s33 = (wo[c + g.sk] - wo[c]) * g.dzi;
        double s12 = 0.25 * (strain12(uo, vo, g, i, j, k) + strain12(uo, vo, g, i, jp, k) +
                             strain12(uo, vo, g, ip, j, k) + strain12(uo, vo, g, ip, jp, k));
        double s13, s23;
        if (P.most && k == 0) {
            // over a MOST ground the ground-face strains are left out and the
            // faces above averaged (ComputeSmnSmn, Diffusion/ERF_EddyViscosity.H:59-77)
            s13 = 0.5 * (strain13(uo, wo, g, i, j, k + 1) + strain13(uo, wo, g, ip, j, k + 1));
            s23 = 0.5 * (strain23(vo, wo, g, i, j, k + 1) + strain23(vo, wo, g, i, jp, k + 1));
        } else {
            s13 = 0.25 * (strain13(uo, wo, g, i, j, k) + strain13(uo, wo, g, i, j, k + 1) +
                          strain13(uo, wo, g, ip, j, k) + strain13(uo, wo, g, ip, j, k + 1));
            s23 = 0.25 * (strain23(vo, wo, g, i, j, k) + strain23(vo, wo, g, i, j, k + 1) +
                          strain23(vo, wo, g, i, jp, k) + strain23(vo, wo, g, i, jp, k + 1));
        }
        double S2 = s11 * s11 + s22 * s22 + s33 * s33 + 2.0 * s12 * s12 + 2.0 * s13 * s13 + 2.0 * s23 * s23;
        if (P.les != ERF_LES_DEARDORFF) {
            mut[c] = R(P.CsDeltaSqr * rho * sqrt(2.0 * S2));
        } else {
            // Deardorff (ERF_ComputeTurbulentViscosity.cpp:129-229, no MOST):
            // SmnSmn for the shear production (formed from the step's
            // velocities, ERF_make_tau_terms.cpp:233-240), K = rho Ck l
            // sqrt(e) with the stratification-limited length, the vertical
            // heat diffusivity (1 + 2 l / Delta) K and the dissipation.
            tke.smn[c] = R(S2);
            const int64_t N = g.ncell;
            const int kp = min(k + 1, g.nz - 1), km = max(k - 1, 0);
            double dtheta_dz;
            if (P.most && k == 0) {
                // one-sided over a MOST ground (ERF_ComputeTurbulentViscosity.cpp:175-188)
                const int64_t c1 = cidx(g, i, j, 1), c2 = cidx(g, i, j, 2);
                dtheta_dz = 0.5 * (-3 * cons[N + c] / cons[c] + 4 * cons[N + c1] / cons[c1] - cons[N + c2] / cons[c2]) * g.dzi;
            } else {
                dtheta_dz = 0.5 * (cons[N + cidx(g, i, j, kp)] / cons[cidx(g, i, j, kp)] -
                                   cons[N + cidx(g, i, j, km)] / cons[cidx(g, i, j, km)]) * g.dzi;
            }
            double E = fmax(cons[2 * N + c] / rho, 0.0);
            double strat = P.g_over_theta0 * dtheta_dz;
            double length;
            if (strat <= 2.220446049250313e-16) {   // DBL_EPSILON
                length = P.Delta;
            } else {
                length = 0.76 * sqrt(E / strat);
                length = fmin(length, P.Delta);
                length = fmax(length, 0.001 * P.Delta);
            }
            double K = rho * P.Ck * length * sqrt(E);
            mut[c] = R(K);
            tke.kthv[c] = R((1. + 2. * length / P.Delta) * K);
            double Ce = ((P.Ce_wall > 0) && (k == 0)) ? P.Ce_wall : 1.9 * P.Ck + P.Ce_lcoeff * length / P.Delta;
            tke.diss[c] = R(rho * Ce * (E * sqrt(E)) / length);
        }
    }
}

// ---------------------------------------------------------------------------
// Stress tensor (erf_make_tau_terms, TimeIntegration/ERF_make_tau_terms.cpp:
// 320-424 with ComputeStress{Cons,Var}Visc_N, Diffusion/ERF_ComputeStress_N.cpp):
// tau_ii at cell centres, tau_12/13/23 on edges.  Strain in FP64 from the
// FP64 velocities, viscosity and stress in R.
// ---------------------------------------------------------------------------
template <class R>
__global__ void k_tau(Params P, const double* __restrict__ cons, const double* __restrict__ u,
                      const double* __restrict__ v, const double* __restrict__ w, const R* __restrict__ mut,
                      R* __restrict__ t11, R* __restrict__ t22, R* __restrict__ t33, R* __restrict__ t12,
                      R* __restrict__ t13, R* __restrict__ t23) {
    const Geo& g = P.g;
    int i, j, k;
    if (!cell_coords(g, i, j, k)) return;
    int im = wrap(i - 1, g.nx), jm = wrap(j - 1, g.ny), ip = wrap(i + 1, g.nx), jp = wrap(j + 1, g.ny);
    const Elem c = eidx(g, i, j, k);
    const R OneThird = R(1. / 3.);
    R s11 = R((ld(u, eidx(g, ip, j, k)) - ld(u, c)) * g.dxi);
    R s22 = R((ld(v, eidx(g, i, jp, k)) - ld(v, c)) * g.dyi);
    R s33 = R((ld(w, c + (uint32_t)g.sk) - ld(w, c)) * g.dzi);
    R er = s11 + s22 + s33;
    const R mu_eff = R(P.mu_eff);
    R base = P.use_consA ? R(cons[c]) * mu_eff : mu_eff;
    R m11 = P.use_turb ? base + R(2) * mut[c] : base;
    t11[c] = -m11 * (s11 - OneThird * er);
    t22[c] = -m11 * (s22 - OneThird * er);
    t33[c] = -m11 * (s33 - OneThird * er);
    auto mu = [&](int ii, int jj, int kk) { return ld(mut, eidx(g, ii, jj, clampk(kk, g.nz))); };
    auto rho = [&](int ii, int jj, int kk) { return R(ld(cons, eidx(g, ii, jj, clampk(kk, g.nz)))); };
    {
        R m = P.use_consA ? R(0.25) * (rho(im, j, k) + rho(i, j, k) + rho(im, jm, k) + rho(i, jm, k)) * mu_eff : mu_eff;
        if (P.use_turb) m = m + R(2) * (R(0.25) * (mu(im, j, k) + mu(i, j, k) + mu(im, jm, k) + mu(i, jm, k)));
        t12[c] = R(strain12(u, v, g, i, j, k)) * -m;
    }
    for (int kk = k; kk <= (k == g.nz - 1 ? g.nz : k); ++kk) {
        const Elem e = eidx(g, i, j, kk);
        R m = P.use_consA ? R(0.25) * (rho(im, j, kk) + rho(i, j, kk) + rho(im, j, kk - 1) + rho(i, j, kk - 1)) * mu_eff : mu_eff;
        if (P.use_turb) m = m + R(2) * (R(0.25) * (mu(im, j, kk) + mu(i, j, kk) + mu(im, j, kk - 1) + mu(i, j, kk - 1)));
        t13[e] = R(strain13(u, w, g, i, j, kk)) * -m;
        R m2 = P.use_consA ? R(0.25) * (rho(i, jm, kk) + rho(i, j, kk) + rho(i, jm, kk - 1) + rho(i, j, kk - 1)) * mu_eff : mu_eff;
        if (P.use_turb) m2 = m2 + R(2) * (R(0.25) * (mu(i, jm, kk) + mu(i, j, kk) + mu(i, jm, kk - 1) + mu(i, j, kk - 1)));
        t23[e] = R(strain23(v, w, g, i, j, kk)) * -m2;
    }
}
// tau_13 / tau_23 on the ground faces of a MOST ground, from the strain with
// the MOST ghost velocities below (run after k_tau, over one plane)
template <class R>
__global__ void k_tau_most_ground(Params P, const double* __restrict__ cons, const double* __restrict__ u,
                                  const double* __restrict__ v, const double* __restrict__ w,
                                  const R* __restrict__ mut, R* __restrict__ t13, R* __restrict__ t23) {
    const Geo& g = P.g;
    const int i = blockIdx.x * blockDim.x + threadIdx.x, j = blockIdx.y * blockDim.y + threadIdx.y;
    if (i >= g.nx || j >= g.ny) return;
    const int im = wrap(i - 1, g.nx), jm = wrap(j - 1, g.ny);
    const R mu_eff = R(P.mu_eff);
    auto mu = [&](int ii, int jj, int kk) { return ld(mut, eidx(g, ii, jj, clampk(kk, g.nz))); };
    auto rho = [&](int ii, int jj, int kk) { return R(ld(cons, eidx(g, ii, jj, clampk(kk, g.nz)))); };
    const MostView mv{u, v, cons};
    const int64_t e = cidx(g, i, j, 0);
    R m = P.use_consA ? R(0.25) * (rho(im, j, 0) + rho(i, j, 0) + rho(im, j, -1) + rho(i, j, -1)) * mu_eff : mu_eff;
    m = m + R(2) * (R(0.25) * (mu(im, j, 0) + mu(i, j, 0) + mu(im, j, -1) + mu(i, j, -1)));
    t13[e] = R(strain13_most(P, mv, w, i, j)) * -m;
    R m2 = P.use_consA ? R(0.25) * (rho(i, jm, 0) + rho(i, j, 0) + rho(i, jm, -1) + rho(i, j, -1)) * mu_eff : mu_eff;
    m2 = m2 + R(2) * (R(0.25) * (mu(i, jm, 0) + mu(i, j, 0) + mu(i, jm, -1) + mu(i, j, -1)));
    t23[e] = R(strain23_most(P, mv, w, i, j)) * -m2;
}

// Stage primitives, Exner function and p' of a state (cons_to_prim,
// ERF_TI_utils.H:4-45), for the per-pass entry points.
template <class R>
__global__ void k_stage_aux(Params P, const double* __restrict__ cons, StageAux<R> A) {
    const Geo& g = P.g;
    int i, j, k;
    if (!cell_coords(g, i, j, k)) return;
    stage_aux_cell<R>(P, cons, A, cidx(g, i, j, k), k);
}

// ---------------------------------------------------------------------------
// Scalar flux helpers
// ---------------------------------------------------------------------------

// Diffusive tendency -div(-rhoAlpha grad phi) (Diffusion/ERF_DiffusionSrcForState_N.cpp:
// 196-667), scalars foextrap at the walls; returns the amount subtracted.
template <class R>
__device__ __forceinline__ R scalar_diff(const Params& P, const double* __restrict__ rhoarr, const R* __restrict__ phi,
                                         const R* __restrict__ mut, double ae_d, double fac_d, int i, int j, int k,
                                         const R* __restrict__ kv = nullptr, R* __restrict__ fz_out = nullptr) {
    const Geo& g = P.g;
    const R ae = R(ae_d), fac = R(fac_d);
    const R dxi = R(g.dxi), dyi = R(g.dyi), dzi = R(g.dzi);
    int im = wrap(i - 1, g.nx), jm = wrap(j - 1, g.ny), ip = wrap(i + 1, g.nx), jp = wrap(j + 1, g.ny);
    auto ph = [&](int ii, int jj, int kk) { return ccz(phi, g, ii, jj, kk); };
    auto rA = [&](int i0, int j0, int k0, int i1, int j1, int k1) {
        R r = P.use_consA ? R(0.5) * (R(ccz(rhoarr, g, i0, j0, k0)) + R(ccz(rhoarr, g, i1, j1, k1))) * ae : ae;
        if (P.use_turb) r += R(0.5) * (ccz(mut, g, i0, j0, k0) * fac + ccz(mut, g, i1, j1, k1) * fac);
        return r;
    };
    // vertical diffusivity: Deardorff's Theta_v when given
    auto rAz = [&](int k0, int k1) {
        if (kv == nullptr) return rA(i, j, k0, i, j, k1);
        R r = P.use_consA ? R(0.5) * (R(ccz(rhoarr, g, i, j, k0)) + R(ccz(rhoarr, g, i, j, k1))) * ae : ae;
        return r + R(0.5) * (ccz(kv, g, i, j, k0) + ccz(kv, g, i, j, k1));
    };
    R fxl = -rA(i, j, k, im, j, k) * (ph(i, j, k) - ph(im, j, k)) * dxi * R(1);
    R fxh = -rA(ip, j, k, i, j, k) * (ph(ip, j, k) - ph(i, j, k)) * dxi * R(1);
    R fyl = -rA(i, j, k, i, jm, k) * (ph(i, j, k) - ph(i, jm, k)) * dyi * R(1);
    R fyh = -rA(i, jp, k, i, j, k) * (ph(i, jp, k) - ph(i, j, k)) * dyi * R(1);
    R fzl = -rAz(k, k - 1) * (ph(i, j, k) - ph(i, j, k - 1)) * dzi;
    R fzh = -rAz(k + 1, k) * (ph(i, j, k + 1) - ph(i, j, k)) * dzi;
    if (fz_out) {   // the z-face fluxes (hfx_z of ERF_DiffusionSrcForState_N.cpp:422-425)
        fz_out[cidx(g, i, j, k)] = fzl;
        if (k == g.nz - 1) fz_out[cidx(g, i, j, k + 1)] = fzh;
    }
    return (fxh - fxl) * dxi * R(1) + (fyh - fyl) * dyi * R(1) + (fzh - fzl) * dzi;
}

// The same from the cell's and its neighbours' values (p[0] the cell; x low,
// high; y low, high; z low, high), for a pass that has them staged.
template <class R>
__device__ __forceinline__ R scalar_diff_vals(const Params& P, const double* __restrict__ rhoarr, const R (&p)[7],
                                              const R* __restrict__ mut, double ae_d, double fac_d, int i, int j, int k) {
    const Geo& g = P.g;
    const R ae = R(ae_d), fac = R(fac_d);
    const uint32_t sk = (uint32_t)g.sk;
    const Elem c = eidx(g, i, j, k);
    const Elem e[6] = {eidx(g, wrap(i - 1, g.nx), j, k), eidx(g, wrap(i + 1, g.nx), j, k), eidx(g, i, wrap(j - 1, g.ny), k),
                           eidx(g, i, wrap(j + 1, g.ny), k), k > 0 ? c - sk : c, k < g.nz - 1 ? c + sk : c};
    const R rc = P.use_consA ? R(ld(rhoarr, c)) : R(0), mc = P.use_turb ? ld(mut, c) * fac : R(0);
    R f[6];
#pragma unroll
    for (int q = 0; q < 6; ++q) {
        R r = P.use_consA ? R(0.5) * (rc + R(ld(rhoarr, e[q]))) * ae : ae;
        if (P.use_turb) r += R(0.5) * (mc + ld(mut, e[q]) * fac);
        f[q] = -r * (q & 1 ? p[q + 1] - p[0] : p[0] - p[q + 1]);
    }
    const R dxi = R(g.dxi), dyi = R(g.dyi), dzi = R(g.dzi);
    return (f[1] - f[0]) * dxi * dxi + (f[3] - f[2]) * dyi * dyi + (f[5] - f[4]) * dzi * dzi;
}

// Horizontal plane averages of rho, theta, qv, qc, qp for buoyancy type 2
// (SourceTerms/ERF_make_buoyancy.cpp:212-249), FP64 sums; also the
// temperature of the mean state of each level.  Each level is split over
// PAVG_PARTS blocks (grid nz x PAVG_PARTS) that write partial sums; the last
// block of a level to finish (counted with an atomic ticket after a memory
// fence) adds the partials in part order and resets the ticket, so the result
// does not depend on which block finishes last.  Buffer layout after the
// 6 nz results: 5 nz PAVG_PARTS partials, then nz tickets (one per double slot).
template <class R>
__global__ void k_plane_avg(Params P, const double* __restrict__ cons, const R* __restrict__ prim,
                            double* __restrict__ avg) {
    const Geo& g = P.g;
    const int k = blockIdx.x, part = blockIdx.y, nz = g.nz;
    const int64_t N = g.ncell;
    double* partial = avg + 6 * nz;
    unsigned int* ticket = reinterpret_cast<unsigned int*>(partial + 5 * nz * PAVG_PARTS);
    double denom = 1.0 / (double)(g.nx * g.ny);
    int nq = P.ncomp - ERF_RHOQ1_COMP;
    const int64_t span = (g.sk + PAVG_PARTS - 1) / PAVG_PARTS;
    const int64_t t0 = part * span, t1 = min(g.sk, t0 + span);
    double acc[5] = {0, 0, 0, 0, 0};
    for (int64_t t = t0 + threadIdx.x; t < t1; t += blockDim.x) {
        int64_t c = g.sk * k + t;
        acc[0] += cons[c] * denom;
        acc[1] += double(prim[c]) * denom;
        if (nq >= 1) acc[2] += double(prim[4 * N + c]) * denom;
        if (nq >= 2) acc[3] += double(prim[5 * N + c]) * denom;
        if (nq >= 3) acc[4] += double(prim[6 * N + c]) * denom;
    }
    __shared__ double sh[5][256];
    __shared__ bool last;
    for (int q = 0; q < 5; ++q) sh[q][threadIdx.x] = acc[q];
    __syncthreads();
    for (int s = blockDim.x / 2; s > 0; s >>= 1) {
        if (threadIdx.x < s)
            for (int q = 0; q < 5; ++q) sh[q][threadIdx.x] += sh[q][threadIdx.x + s];
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        for (int q = 0; q < 5; ++q) partial[(q * nz + k) * PAVG_PARTS + part] = sh[q][0];
        __threadfence();
        last = atomicAdd(&ticket[2 * k], 1u) == PAVG_PARTS - 1;
    }
    __syncthreads();
    if (last && threadIdx.x == 0) {
        __threadfence();
        double m[5];
        for (int q = 0; q < 5; ++q) {
            const volatile double* pq = partial + (q * nz + k) * PAVG_PARTS;
            double sum = 0.0;
            for (int p = 0; p < PAVG_PARTS; ++p) sum += pq[p];
            m[q] = sum;
            avg[q * nz + k] = sum;
        }
        // the plane-mean temperature used by make_buoyancy's type 2
        avg[5 * nz + k] = eos_T(m[0], m[0] * m[1], m[2]);
        ticket[2 * k] = 0u;
    }
}

// Momentum flux helper: vertical stencil of a face velocity (FP64 state) in R
// (ERF_AdvectionSrcForMom_N.H:17-274); away from the walls six loads at
// constant strides.
template <int T, class R>
__device__ __forceinline__ R gatherz_tang(const Geo& g, const double* f, int type, R upw, R frac, int i, int j, int k) {
    R s[6];
    const int w = width_of<T>(type);
    if (k >= w && k + w <= g.nz) {
        const Elem e = eidx(g, i, j, k);
        const uint32_t sk = (uint32_t)g.sk;
#pragma unroll
        for (int m = 0; m < 6; ++m) {
            const int off = m - 3;
            s[m] = (off >= -w && off <= w - 1) ? R(ld(f, e + (uint32_t)off * sk)) : R(0);
        }
    } else {
#pragma unroll
        for (int m = 0; m < 6; ++m) {
            const int off = m - 3;
            s[m] = (off >= -w && off <= w - 1) ? R(tang(f, g, i, j, k + off)) : R(0);
        }
    }
    return interp_of<T, R>(type, s, upw, frac);
}
// The same for the stage's u (comp 0) or v (comp 1) over a MOST ground.
template <int T, class R>
__device__ __forceinline__ R gatherz_most(const Params& P, const MostView& mv, int comp, int type, R upw, R frac, int i,
                                          int j, int k) {
    R s[6];
    const int w = width_of<T>(type);
    for (int m = 0; m < 6; ++m) {
        int off = m - 3;
        s[m] = (off >= -w && off <= w - 1) ? R(comp == 0 ? tang_u(P, mv, i, j, k + off) : tang_v(P, mv, i, j, k + off))
                                           : R(0);
    }
    return interp_of<T, R>(type, s, upw, frac);
}

// ---------------------------------------------------------------------------
// The stage update without acoustic substepping (no_substep_fun,
// TimeIntegration/ERF_TI_no_substep_fun.H:6-150, fixed or no terrain):
// S_sum = S_old + slow_dt * F_slow for rho, rho*theta and the three momenta,
// accumulated in FP64 from the slow right-hand side (type R).  The boundary
// fill that follows in the reference (apply_bcs of S_sum) changes no valid
// value but for rounding.
// ---------------------------------------------------------------------------
template <class R>
__global__ void k_no_substep(Geo g, double slow_dt, StateBuf Sold, const R* __restrict__ Fcons,
                             const R* __restrict__ Fmx, const R* __restrict__ Fmy, const R* __restrict__ Fmz,
                             StateBuf Ssum) {
    int i, j, k;
    if (!cell_coords(g, i, j, k)) return;
    const int64_t N = g.ncell, c = cidx(g, i, j, k);
    Ssum.cons[c] = Sold.cons[c] + slow_dt * (double(Fcons[c]));
    Ssum.cons[N + c] = Sold.cons[N + c] + slow_dt * (double(Fcons[N + c]));
    Ssum.mx[c] = Sold.mx[c] + slow_dt * double(Fmx[c]);
    Ssum.my[c] = Sold.my[c] + slow_dt * double(Fmy[c]);
    Ssum.mz[c] = Sold.mz[c] + slow_dt * double(Fmz[c]);
    if (k == g.nz - 1) Ssum.mz[c + g.sk] = Sold.mz[c + g.sk] + slow_dt * double(Fmz[c + g.sk]);
}

// ---------------------------------------------------------------------------
// Hydrostatic base state, one thread: calc_rho_p Newton integration at cell
// centres (ERF_InputSoundingData.H:176-256, ERF_HSE_utils.H:34-72) and
// erf_enforce_hse (ERF_init1d.cpp:152-260).  FP64, run once at set-up.
// ---------------------------------------------------------------------------
__global__ void k_base_state(int nz, double dz, double g, double rdOcp, const double* __restrict__ th_cc,
                             const double* __restrict__ qv_cc, double th_s, double qv_s, double p_s,
                             double* __restrict__ rho0, double* __restrict__ p0o, double* __restrict__ pi0o,
                             double* __restrict__ th0o) {
    if (blockIdx.x != 0 || threadIdx.x != 0) return;
    const double tol = 1.0e-12;
    const double RdOCp = R_d / Cp_d;
    double pm = p_s;
    double rd = eos_rho_given_theta_p(th_s, p_s, RdOCp, qv_s);
    double zprev = 0.0, qprev = qv_s;
    for (int k = 1; k <= nz; ++k) {
        double z = (k - 1 + 0.5) * dz;
        double th = th_cc[k - 1], qv = qv_cc[k - 1];
        double dzl = z - zprev;
        double rlo = rd * (1. + qprev);
        double C = -pm + 0.5 * rlo * g * dzl;
        double pk = pm;
        double rk = eos_rho_given_theta_p(th, pk, RdOCp, qv);
        double rhi = rk * (1. + qv);
        double F = pk + 0.5 * rhi * g * dzl + C;
        if (fabs(F) > tol) {
            int iter = 0;
            double eps = 1.0e-6, ieps = 1.0e6;
            do {
                double hi = eos_rho_given_theta_p(th, pk + eps, RdOCp, qv);
                double lo = eos_rho_given_theta_p(th, pk - eps, RdOCp, qv);
                double dFdp = 1.0 + 0.25 * ieps * (hi - lo) * g * dzl;
                pk -= F / dFdp;
                rk = eos_rho_given_theta_p(th, pk, RdOCp, qv);
                double rt = rk * (1. + qv);
                F = pk + 0.5 * rt * g * dzl + C;
                ++iter;
            } while (fabs(F) > tol && iter < 30);
        }
        rho0[k] = rk;
        pm = pk; rd = rk; zprev = z; qprev = qv;
    }
    rho0[0] = rho0[1];
    rho0[nz + 1] = rho0[nz];
    double hz = 0.5 * dz;
    p0o[1] = p_0 - hz * rho0[1] * g;
    pi0o[1] = eos_exner_p(p0o[1], rdOcp);
    th0o[1] = eos_rt_given_p(p0o[1]) / rho0[1];
    p0o[0] = p_0 + hz * rho0[1] * g;
    pi0o[0] = eos_exner_p(p0o[0], rdOcp);
    th0o[0] = eos_rt_given_p(p0o[0]) / rho0[0];
    for (int k = 1; k <= nz; ++k) {
        int kk = k + 1;
        double di = 0.5 * (rho0[kk] + rho0[kk - 1]);
        p0o[kk] = p0o[kk - 1] - dz * di * g;
        pi0o[kk] = eos_exner_p(p0o[kk], rdOcp);
        th0o[kk] = eos_rt_given_p(p0o[kk]) / rho0[kk];
    }
}

// ---------------------------------------------------------------------------
// Layout conversion between a caller's Array4 view and the internal arrays.
// kind: 0 cell, 1 x-face, 2 y-face, 3 z-face.  Unpack writes the caller's
// valid region and every ghost cell the view covers (periodic laterally,
// wall conditions vertically).
// ---------------------------------------------------------------------------
__global__ void k_pack(Geo g, erf_b200_fab f, int kind, int ncomp, double* __restrict__ dst) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    int j = blockIdx.y * blockDim.y + threadIdx.y;
    int k = blockIdx.z;
    int nzk = (kind == 3) ? g.nz + 1 : g.nz;
    if (i >= g.nx || j >= g.ny || k >= nzk) return;
    int64_t src0 = (int64_t)(i - f.lo[0]) + (int64_t)(j - f.lo[1]) * f.jstride + (int64_t)(k - f.lo[2]) * f.kstride;
    int64_t per = (kind == 3) ? g.nzf : g.ncell;
    for (int n = 0; n < ncomp; ++n) dst[n * per + cidx(g, i, j, k)] = f.p[src0 + n * f.nstride];
}

__global__ void k_unpack(Geo g, erf_b200_fab f, int kind, int ncomp, const double* __restrict__ src,
                         int tang_lo_zero, int tang_hi_zero, int wall_w) {
    // thread over the caller's whole box
    int64_t nxb = f.hi[0] - f.lo[0] + 1, nyb = f.hi[1] - f.lo[1] + 1;
    int ib = blockIdx.x * blockDim.x + threadIdx.x;
    int jb = blockIdx.y * blockDim.y + threadIdx.y;
    int kb = blockIdx.z;
    if (ib >= nxb || jb >= nyb || kb > f.hi[2] - f.lo[2]) return;
    int i = f.lo[0] + ib, j = f.lo[1] + jb, k = f.lo[2] + kb;
    int64_t dst0 = (int64_t)ib + (int64_t)jb * f.jstride + (int64_t)kb * f.kstride;
    int64_t per = (kind == 3) ? g.nzf : g.ncell;
    int ii = ((i % g.nx) + g.nx) % g.nx, jj = ((j % g.ny) + g.ny) % g.ny;
    for (int n = 0; n < ncomp; ++n) {
        double val;
        if (kind == 3) {
            // beyond the walls 0; on the walls 0 without terrain, the stored
            // value (w from Omega = 0) with terrain
            if (k < 0 || k > g.nz || (!wall_w && (k == 0 || k == g.nz))) val = 0.0;
            else val = src[n * per + cidx(g, ii, jj, k)];
        } else if (k < 0 || k >= g.nz) {
            bool lo = k < 0;
            int ks = lo ? 0 : g.nz - 1;
            bool zero = (kind == 1 || kind == 2) && (lo ? tang_lo_zero : tang_hi_zero);
            val = zero ? 0.0 : src[n * per + cidx(g, ii, jj, ks)];
        } else {
            val = src[n * per + cidx(g, ii, jj, k)];
        }
        f.p[dst0 + n * f.nstride] = val;
    }
}


// The same for a whole state -- the conserved variables and the three face
// velocities -- in one launch each way: a thread moves all of a cell's values,
// so that they are in flight together (eight launches a call otherwise, which
// on a small grid cost as much as its kernels).
__global__ void __launch_bounds__(256) k_pack_state(Geo g, StateFabs f, int ncomp, double* __restrict__ cons,
                                                    double* __restrict__ u, double* __restrict__ v,
                                                    double* __restrict__ w) {
    const int i = blockIdx.x * 32 + threadIdx.x, j = blockIdx.y * 8 + threadIdx.y, k = blockIdx.z;
    if (i >= g.nx || j >= g.ny) return;
    auto src = [&](const erf_b200_fab& a) {
        return a.p + ((i - a.lo[0]) + (j - a.lo[1]) * a.jstride + (k - a.lo[2]) * a.kstride);
    };
    const int64_t c = cidx(g, i, j, k);
    w[c] = *src(f.a[3]);
    if (k >= g.nz) return;
    u[c] = *src(f.a[1]);
    v[c] = *src(f.a[2]);
    const double* p = src(f.a[0]);
    for (int n = 0; n < ncomp; ++n) cons[n * g.ncell + c] = p[n * f.a[0].nstride];
}
// box: the smallest that holds the four views' boxes
__global__ void __launch_bounds__(256) k_unpack_state(Geo g, StateFabs f, int lo0, int lo1, int lo2, int ncomp,
                                                      const double* __restrict__ cons, const double* __restrict__ u,
                                                      const double* __restrict__ v, const double* __restrict__ w,
                                                      int wall_w) {
    const int i = lo0 + (int)(blockIdx.x * 32 + threadIdx.x), j = lo1 + (int)(blockIdx.y * 8 + threadIdx.y);
    const int k = lo2 + (int)blockIdx.z;
    const int ii = (unsigned)i < (unsigned)g.nx ? i : ((i % g.nx) + g.nx) % g.nx;
    const int jj = (unsigned)j < (unsigned)g.ny ? j : ((j % g.ny) + g.ny) % g.ny;
    auto in = [&](const erf_b200_fab& a) {
        return i >= a.lo[0] && i <= a.hi[0] && j >= a.lo[1] && j <= a.hi[1] && k >= a.lo[2] && k <= a.hi[2];
    };
    auto dst = [&](const erf_b200_fab& a) {
        return a.p + ((i - a.lo[0]) + (j - a.lo[1]) * a.jstride + (k - a.lo[2]) * a.kstride);
    };
    const int64_t c = cidx(g, ii, jj, clampk(k, g.nz));
    // tangential velocity beyond a no-slip wall: 0
    const bool zero = (k < 0 && g.zlo_noslip) || (k >= g.nz && g.zhi_noslip);
    if (in(f.a[1])) *dst(f.a[1]) = zero ? 0.0 : u[c];
    if (in(f.a[2])) *dst(f.a[2]) = zero ? 0.0 : v[c];
    if (in(f.a[3]))
        // beyond the walls 0; on the walls 0 without terrain, the stored value
        // (w from Omega = 0) with terrain
        *dst(f.a[3]) = (k < 0 || k > g.nz || (!wall_w && (k == 0 || k == g.nz))) ? 0.0 : w[cidx(g, ii, jj, k)];
    if (in(f.a[0])) {
        double* p = dst(f.a[0]);
        for (int n = 0; n < ncomp; ++n) p[n * f.a[0].nstride] = cons[n * g.ncell + c];
    }
}
void launch_pack_state(const Geo& g, cudaStream_t st, const StateFabs& f, int ncomp, double* cons, double* const* vel) {
    k_pack_state<<<dim3((g.nx + 31) / 32, (g.ny + 7) / 8, g.nz + 1), dim3(32, 8), 0, st>>>(g, f, ncomp, cons, vel[0],
                                                                                            vel[1], vel[2]);
}
void launch_unpack_state(const Geo& g, cudaStream_t st, const StateFabs& f, int ncomp, const double* cons,
                         double* const* vel, int wall_w) {
    int lo[3], hi[3];
    for (int d = 0; d < 3; ++d) {
        lo[d] = f.a[0].lo[d];
        hi[d] = f.a[0].hi[d];
        for (int q = 1; q < 4; ++q) {
            lo[d] = f.a[q].lo[d] < lo[d] ? f.a[q].lo[d] : lo[d];
            hi[d] = f.a[q].hi[d] > hi[d] ? f.a[q].hi[d] : hi[d];
        }
    }
    k_unpack_state<<<dim3((hi[0] - lo[0] + 32) / 32, (hi[1] - lo[1] + 8) / 8, hi[2] - lo[2] + 1), dim3(32, 8), 0, st>>>(
        g, f, lo[0], lo[1], lo[2], ncomp, cons, vel[0], vel[1], vel[2], wall_w);
}

// ---------------------------------------------------------------------------
// Tile layout of k_fast_coef below: a block owns TX
// adjacent columns (i = blockIdx.x*TX + threadIdx.x, j = blockIdx.y) and
// blockDim.y warps split the levels; per-column data live in shared memory as
// [level][column] so a warp touches consecutive banks.
// ---------------------------------------------------------------------------
struct Tile {
    int i, j, lane, w, nw, tx;
    bool ok;
    __device__ Tile(const Geo& g) {
        tx = blockDim.x; lane = threadIdx.x; w = threadIdx.y; nw = blockDim.y;
        i = blockIdx.x * tx + lane; j = blockIdx.y;
        ok = i < g.nx;
    }
};

// ---------------------------------------------------------------------------
// Fast coefficients of one RK stage (make_fast_coeffs,
// TimeIntegration/ERF_make_fast_coeffs.cpp:160-290, no terrain): P and Q
// (divided by 1+q when moist), A, B, C on interior z-faces, Dirichlet rows at
// the walls, then the Thomas forward elimination of B.  Stored per face:
// A, 1/B' (B' at the wall rows, which the reference leaves uninverted),
// C/B', P, Q.  Levels are computed in parallel; the B' recurrence runs in one
// warp from shared memory.  P and Q use the FP64 base and stage state.
// ---------------------------------------------------------------------------
template <class R>
__global__ void k_fast_coef(Params P, double D_d, StateBuf Sst, StageAux<R> A, R* __restrict__ cA,
                            R* __restrict__ cInvB, R* __restrict__ cCB, R* __restrict__ cP, R* __restrict__ cQ) {
    extern __shared__ __align__(16) unsigned char sm_raw[];
    R* sm = reinterpret_cast<R*>(sm_raw);
    const Geo& g = P.g;
    Tile t(g);
    const int nz = g.nz, TX = t.tx;
    R* sA = sm;
    R* sB = sA + (nz + 1) * TX;
    R* sC = sB + (nz + 1) * TX;
    const int64_t N = g.ncell;
    const R D = R(D_d), halfg = R(P.halfg);
    const R* th = A.prim;
    if (t.ok) {
        for (int k = 1 + t.w; k <= nz - 1; k += t.nw) {
            int64_t c = cidx(g, t.i, t.j, k), cm = c - g.sk;
            R pi_c = R(0.5) * (A.pi[cm] + A.pi[c]);
            // with terrain (ERF_make_fast_coeffs.cpp:110-140): the 3-D base
            // state, the acoustic terms over detJ at the face and B = detJ + ...
            double dJk = 1.0, inv_dJk = 1.0, r_hi, r_lo, pi_hi, pi_lo;
            if (P.ter) {
                dJk = 0.5 * (P.detJ[c] + P.detJ[cm]);
                inv_dJk = 1. / dJk;
                r_hi = P.r0[c + g.sk]; r_lo = P.r0[c]; pi_hi = P.pi0[c + g.sk]; pi_lo = P.pi0[c];
            } else {
                r_hi = P.r0[k + 1]; r_lo = P.r0[k]; pi_hi = P.pi0[k + 1]; pi_lo = P.pi0[k];
            }
            R P_ = R(-Gamma_ * R_d * g.dzi * inv_dJk + P.halfg * R_d * r_hi / (P.c_v * pi_hi * Sst.cons[N + c]));
            P_ *= pi_c;
            R Q_ = R(Gamma_ * R_d * g.dzi * inv_dJk + P.halfg * R_d * r_lo / (P.c_v * pi_lo * Sst.cons[N + cm]));
            Q_ *= pi_c;
            if (P.moist) {
                R q = R(0.5) * (th[4 * N + c] + th[4 * N + cm] + th[5 * N + c] + th[5 * N + cm]);
                P_ /= (R(1) + q);
                Q_ /= (R(1) + q);
            }
            R tlo = R(0.5) * (th[cidx(g, t.i, t.j, clampk(k - 2, nz))] + th[cm]);
            R tmid = R(0.5) * (th[cm] + th[c]);
            R thi = R(0.5) * (th[c] + th[cidx(g, t.i, t.j, clampk(k + 1, nz))]);
            R a = D * (halfg - Q_ * tlo);
            R cc = D * (-halfg + P_ * thi);
            R b = R(dJk) + D * (Q_ - P_) * tmid;
            sA[k * TX + t.lane] = a; sB[k * TX + t.lane] = b; sC[k * TX + t.lane] = cc;
            cA[c] = a; cP[c] = P_; cQ[c] = Q_;
        }
        if (t.w == 0) {
            for (int k : {0, nz}) {
                sA[k * TX + t.lane] = R(0); sB[k * TX + t.lane] = R(1); sC[k * TX + t.lane] = R(0);
                int64_t f = cidx(g, t.i, t.j, k);
                cA[f] = R(0); cP[f] = R(0); cQ[f] = R(0);
            }
        }
    }
    __syncthreads();
    if (t.w == 0 && t.ok) {
        R bet = sB[t.lane];
        int64_t f0 = cidx(g, t.i, t.j, 0);
        cInvB[f0] = bet;               // B at the bottom row stays uninverted (== 1)
        cCB[f0] = sC[t.lane] * bet;
        for (int k = 1; k <= nz; ++k) {
            R gam = sC[(k - 1) * TX + t.lane] / bet;
            bet = sB[k * TX + t.lane] - sA[k * TX + t.lane] * gam;
            if (!(fabs(double(bet)) > 1e-300)) atomicOr(P.status, ST_BADSTATE);
            R inv = (k < nz) ? R(1) / bet : bet;
            int64_t f = cidx(g, t.i, t.j, k);
            cInvB[f] = inv;
            cCB[f] = sC[k * TX + t.lane] * inv;
        }
    }
}

// ---------------------------------------------------------------------------
// Scalar and momentum transport on x-y tiles marching up in k.  A block owns
// TTX x TTY columns and `kz` consecutive levels.  At each level every thread
// evaluates the advective flux through its cell's low x and y faces into
// shared memory (the tile's high edge also evaluates the high faces) and
// carries the flux through its top face to the next level, so each face flux
// is evaluated once per block.  All fluxes of one level are staged before a
// single barrier.  `kz` is chosen on the host so that the whole grid is one
// wave of resident blocks.
// Divergence as in AdvectionSrcForScalars (ERF_AdvectionSrcForState.cpp:359-370).
// ---------------------------------------------------------------------------
// Minimum resident blocks per SM requested from the register allocator for
// each tiled kernel (trades instruction-level for warp-level parallelism).
#ifndef ERFB_MINB_CELL
#define ERFB_MINB_CELL 4
#endif
#ifndef ERFB_MINB_MOM
#define ERFB_MINB_MOM 4
#endif
#ifndef ERFB_MINB_POST
#define ERFB_MINB_POST 4
#endif


// ---------------------------------------------------------------------------
// Slow RHS for rho and rho*theta (erf_slow_rhs_pre cell part,
// ERF_slow_rhs_pre.cpp:462-526): AdvectionSrcForRho (also initialises the
// average momenta to the stage mass fluxes, ERF_AdvectionSrcForState.cpp:56-71),
// AdvectionSrcForScalars for theta with the dycore scheme
// (ERF_slow_rhs_pre.cpp:139-142, 469-477), DiffusionSrcForState_N for theta.
// ---------------------------------------------------------------------------
template <class R, int TH, int TV>
__global__ void __launch_bounds__(TTX * TTY, ERFB_MINB_CELL) k_slow_cell(Params P, int kz, StateBuf S, StageAux<R> A,
                                                                         const R* __restrict__ mut,
                                                                         const R* __restrict__ hx,
                                                                         const R* __restrict__ hy,
                                                                         const R* __restrict__ hz, TkeBuf<R> tke,
                                                                         R* __restrict__ Fcons, R* __restrict__ avx,
                                                                         R* __restrict__ avy, R* __restrict__ avz) {
    __shared__ FluxTile<R> sh;
    __shared__ Plane<R> pl;
    const Geo& g = P.g;
    const int i = blockIdx.x * TTX + threadIdx.x, j = blockIdx.y * TTY + threadIdx.y;
    const bool ok = i < g.nx && j < g.ny;
    const int k0 = blockIdx.z * kz, k1 = min(k0 + kz, g.nz);
    const int ip = ok ? wrap(i + 1, g.nx) : 0, jp = ok ? wrap(j + 1, g.ny) : 0;
    R zl = R(0), zh = R(0);
    const TileEdge edge = tile_edge(g);
    const PlaneIdx pidx(g);
    load_plane(g, pidx, pl, A.prim, k0);
    for (int k = k0; k < k1; ++k) {
        plane_wait();
        __syncthreads();
        if (ok)
            tile_put<TH, TV>(g, sh, pl, A.prim, S.mx, S.my, S.mz, P.dyc_h, P.dyc_v, R(P.f_dyc_h), R(P.f_dyc_v), i, j,
                             k, k == k0, zl, zh);
        tile_put_edge<TH>(g, edge, sh, pl, S.mx, S.my, P.dyc_h, R(P.f_dyc_h), k);
        __syncthreads();
        if (k + 1 < k1) load_plane(g, pidx, pl, A.prim, k + 1);   // overlaps the update below
        if (ok) {
            R frt = tile_div(g, sh, zl, zh);
            zl = zh;
            int64_t c = cidx(g, i, j, k);
            if (avx) {   // the per-pass entry wants them; the first substep forms its own
                avx[c] = R(S.mx[c]);
                avy[c] = R(S.my[c]);
                avz[c] = R(S.mz[c]);
                if (k == g.nz - 1) avz[c + g.sk] = R(S.mz[c + g.sk]);
            }
            Fcons[c] = R(-1.0 / 1.0 * ((S.mx[cidx(g, ip, j, k)] - S.mx[c]) * g.dxi +
                                       (S.my[cidx(g, i, jp, k)] - S.my[c]) * g.dyi + (S.mz[c + g.sk] - S.mz[c]) * g.dzi));
            if (P.les == ERF_LES_MLP) {
                // divergence of the learned heat flux rho*q (cell values
                // averaged to faces; no flux through the walls)
                const int im = wrap(i - 1, g.nx), jm = wrap(j - 1, g.ny);
                auto fz = [&](int kk) {
                    if (kk <= 0 || kk >= g.nz) return R(0);
                    return R(0.5) * (hz[cidx(g, i, j, kk - 1)] + hz[cidx(g, i, j, kk)]);
                };
                R fxl = R(0.5) * (hx[cidx(g, im, j, k)] + hx[c]), fxh = R(0.5) * (hx[c] + hx[cidx(g, ip, j, k)]);
                R fyl = R(0.5) * (hy[cidx(g, i, jm, k)] + hy[c]), fyh = R(0.5) * (hy[c] + hy[cidx(g, i, jp, k)]);
                frt -= (fxh - fxl) * R(g.dxi) + (fyh - fyl) * R(g.dyi) + (fz(k + 1) - fz(k)) * R(g.dzi);
            } else if (P.les == ERF_LES_DEARDORFF) {
                frt -= scalar_diff<R>(P, S.cons, A.prim, mut, P.alphaT_eff, P.invPr, i, j, k, tke.kthv, tke.hfz);
            } else if (P.use_diff) {
                frt -= scalar_diff<R>(P, S.cons, A.prim, mut, P.alphaT_eff, P.invPr, i, j, k);
            }
            Fcons[g.ncell + c] = frt;
        }
        // the next level's first barrier orders the reuse of sh
    }
}

// ---------------------------------------------------------------------------
// Slow RHS post + stage finalisation (erf_slow_rhs_post,
// ERF_slow_rhs_post.cpp:228-531, and post_update = apply_bcs(S_new),
// ERF_TI_slow_rhs_fun.H:284-288):
//   * advection (average momenta) and diffusion of the slow scalars
//     (passive scalar with the dry-scalar scheme; moisture with the moist
//     scheme), S_new = S_old + slow_dt * RHS (FP64), moisture clipped at 0;
//   * rho, rho*theta and the momenta copied from the fast solution;
//   * the stage velocities, and (unless last) the next stage's primitive
//     variables, Exner function and p'.
// ---------------------------------------------------------------------------
// Slow variables, in order: the passive scalar, the moisture species, then
// (Deardorff) rho*KE.  A block marches ONE of them up its tile; the rest of
// the stage's end goes to the scalar's blocks (the copies, momenta and
// velocities) and to the vapour's (theta, Exner function and p' of the next
// stage; the scalar's in dry air).  With all variables in one block the
// vertical stencils were loads, L2 hits mostly, on every level (four of six
// levels each on the moist bubble, 262 us per stage at 128x128x80, 200 now); one at a
// time, the column is a window in registers, fed a level ahead along with the
// momenta.  The jobs of a tile are neighbours in the grid, so that what they
// share is read from DRAM once.
template <class R>
struct PostArgs {
    double slow_dt;
    StateBuf old, st, sum, nw;
    StageAux<R> cur, next;
    int make_next;
    const double* keep;   // the state whose rho KE (no Deardorff) and rho QKE go on
    const R* mut;
    TkeBuf<R> tke;
    const R *avx, *avy, *avz;
    double *un, *vn, *wn;
};
template <class R, int TH, int TV>
__device__ __forceinline__ void post_march(const Params& P, const PostArgs<R>& a, FluxTile<R>& sh, Plane<R>& pl, int th,
                                           int tv, R fh, R fv, int q, int nscal, int k0, int k1) {
    const Geo& g = P.g;
    const int64_t N = g.ncell;
    const uint32_t sk = (uint32_t)g.sk;
    const int tx = threadIdx.x, ty = threadIdx.y;
    const int i = blockIdx.x * TTX + tx, j = blockIdx.y * TTY + ty;
    const bool ok = i < g.nx && j < g.ny;
    const int im = ok ? wrap(i - 1, g.nx) : 0, jm = ok ? wrap(j - 1, g.ny) : 0;
    const bool dd = P.les == ERF_LES_DEARDORFF, ke = q >= nscal;
    const int n = q == 0 ? ERF_RHOSCALAR_COMP : (ke ? ERF_RHOKE_COMP : ERF_RHOQ1_COMP + q - 1);
    const bool thermo = P.moist ? n == ERF_RHOQ1_COMP : q == 0;
    const R* __restrict__ phi = a.cur.prim + (int64_t)(n - 1) * N;
    const TileEdge edge = tile_edge(g);
    const PlaneIdx pidx(g);
    constexpr int W = TV < 0 ? 3 : (TV == ERF_ADV_CENTERED_2ND ? 1 : (TV == ERF_ADV_UPWIND_5TH || TV == ERF_ADV_CENTERED_6TH || TV == ERF_ADV_WENO_5 ? 3 : 2));
    const Elem e0 = ok ? eidx(g, i, j, 0) : eidx(g, 0, 0, 0);
    auto lvl = [&](int k) { return ld(phi, e0 + sk * (uint32_t)clampk(k, g.nz)); };
    // win[m]: phi at level f - W + m of the face f whose flux comes next
    R win[2 * W];
    auto zflux = [&](R az) {
        R s[6];
#pragma unroll
        for (int m = 0; m < 6; ++m) s[m] = (m >= 3 - W && m < 3 + W) ? win[m >= 3 - W && m < 3 + W ? m - 3 + W : 0] : R(0);
        return az * interp_of<TV, R>(tv, s, az, fv);
    };
    R zl = R(0), ax = R(0), ay = R(0), az = R(0), top = R(0);
    load_plane(g, pidx, pl, phi, k0);
    if (ok) {
#pragma unroll
        for (int m = 0; m < 2 * W; ++m) win[m] = lvl(k0 - W + m);
        const Elem c = e0 + sk * (uint32_t)k0;
        zl = zflux(ld(a.avz, c));
        ax = ld(a.avx, c); ay = ld(a.avy, c); az = ld(a.avz, c + sk);
        top = lvl(k0 + W);
    }
    for (int k = k0; k < k1; ++k) {
        const Elem c = e0 + sk * (uint32_t)k;
        R zh = R(0), dif = R(0);
        plane_wait();
        __syncthreads();
        if (ok) {
            sh.fx[ty][tx] = plane_flux_x<TH>(pl, ty, tx, ax, th, fh);
            sh.fy[ty][tx] = plane_flux_y<TH>(pl, ty, tx, ay, th, fh);
#pragma unroll
            for (int m = 0; m < 2 * W - 1; ++m) win[m] = win[m + 1];
            win[2 * W - 1] = top;
            zh = zflux(az);
            if (ke || P.use_diff) {
                const int y = ty + PH, x = tx + PH;
                const R pc = pl.v[y][x];
                const R p[7] = {pc, pl.v[y][x - 1], pl.v[y][x + 1], pl.v[y - 1][x], pl.v[y + 1][x],
                                W > 1 ? win[W > 1 ? W - 2 : 0] : lvl(k - 1), W > 1 ? win[W] : lvl(k + 1)};
                dif = scalar_diff_vals<R>(P, a.st.cons, p, a.mut, ke ? 0.0 : P.alphaC_eff, ke ? P.invSigmaK : P.invSc, i, j, k);
            }
        }
        tile_put_edge<TH>(g, edge, sh, pl, a.avx, a.avy, th, fh, k);
        __syncthreads();
        if (k + 1 < k1) load_plane(g, pidx, pl, phi, k + 1);   // arrives during the update below
        if (ok) {
            if (k + 1 < k1) {   // the next level's operands
                ax = ld(a.avx, c + sk); ay = ld(a.avy, c + sk); az = ld(a.avz, c + 2 * sk);
                top = lvl(k + 1 + W);
            }
            R r = tile_div(g, sh, zl, zh);
            zl = zh;
            r -= dif;
            if (ke) {
                // the TKE sources of ERF_DiffusionSrcForState_N.cpp:681-707:
                // buoyancy, shear production, dissipation
                r += R(P.g_over_theta0) * a.tke.hfz[c];
                r += R(2.0) * a.mut[c] * a.tke.smn[c];
                r -= a.tke.diss[c];
            }
            double nv = ld(a.old.cons + n * N, c) + a.slow_dt * double(r);
            if (q > 0) nv = fmax(nv, ke ? 2.220446049250313e-16 : 0.0);
            if (n == 7 && a.nw.rain) a.nw.rain[c] = nv;
            else at(a.nw.cons + n * N, c) = nv;
            const double rho = ld(a.sum.cons, c);
            double ir = 0.0;
            if (a.make_next) {
                ir = 1.0 / rho;
                at(a.next.prim + (n - 1) * N, c) = R(nv * ir);
            }
            if (thermo && a.make_next)
                stage_aux_thermo<R>(P, rho, ld(a.sum.cons + N, c), ir, P.moist ? nv * ir : 0.0, a.next, c, k);
            if (q == 0) {
                at(a.nw.cons, c) = rho;
                at(a.nw.cons + N, c) = ld(a.sum.cons + N, c);
                if (a.keep) {
                    if (!dd) at(a.nw.cons + 2 * N, c) = ld(a.keep + 2 * N, c);
                    at(a.nw.cons + 3 * N, c) = ld(a.keep + 3 * N, c);
                }
                {
                    const double rs = rho + ld(a.sum.cons, eidx(g, im, j, k)), m = ld(a.sum.mx, c);
                    at(a.nw.mx, c) = m; at(a.un, c) = (m * 2.0) / rs;
                }
                {
                    const double rs = rho + ld(a.sum.cons, eidx(g, i, jm, k)), m = ld(a.sum.my, c);
                    at(a.nw.my, c) = m; at(a.vn, c) = (m * 2.0) / rs;
                }
                if (k == 0) {
                    at(a.nw.mz, c) = 0.0; at(a.wn, c) = 0.0;
                } else {
                    const double rs = rho + ld(a.sum.cons, c - sk), m = ld(a.sum.mz, c);
                    at(a.nw.mz, c) = m; at(a.wn, c) = (m * 2.0) / rs;
                }
                if (k == g.nz - 1) { at(a.nw.mz, c + sk) = 0.0; at(a.wn, c + sk) = 0.0; }
            }
        }
        // the next level's first barrier orders the reuse of sh
    }
}
template <class R, int DH, int DV, int MH, int MV>
__global__ void __launch_bounds__(TTX * TTY, ERFB_MINB_POST) k_post(Params P, int kz, PostArgs<R> a) {
    __shared__ FluxTile<R> sh;
    __shared__ Plane<R> pl;
    const int nscal = P.moist ? 1 + (P.ncomp - ERF_RHOQ1_COMP) : 1;
    const int nslow = nscal + (P.les == ERF_LES_DEARDORFF ? 1 : 0);
    const int q = blockIdx.z % nslow, k0 = blockIdx.z / nslow * kz, k1 = min(k0 + kz, P.g.nz);
    if (q == 0 || q >= nscal)   // scalar and KE: dry-scalar schemes
        post_march<R, DH, DV>(P, a, sh, pl, P.dry_h, P.dry_v, R(P.f_dry_h), R(P.f_dry_v), q, nscal, k0, k1);
    else
        post_march<R, MH, MV>(P, a, sh, pl, P.moi_h, P.moi_v, R(P.f_moi_h), R(P.f_moi_v), q, nscal, k0, k1);
}

// Momentum fluxes of AdvectionSrcFor{X,Y,Z}Mom_N (ERF_AdvectionSrcForMom_N.H:
// 17-274).  Each is the flux through the low side of the face's control
// volume in one direction; the high side is the same function one index up.
// The x / y stencils of the face velocity come from the level's staged
// plane: column c0 = tx (low face) or tx + 1 (the tile edge's high face),
// row r0 = ty or ty + 1 likewise.
template <int T, class R, class V>
__device__ __forceinline__ R plane_interp_x(const Plane<V>& p, int ty, int c0, int type, R upw, R frac) {
    R s[6];
    const int w = width_of<T>(type);
#pragma unroll
    for (int m = 0; m < 6; ++m) {
        const int off = m - 3;
        s[m] = (off >= -w && off <= w - 1) ? R(p.v[ty + PH][c0 + m]) : R(0);
    }
    return interp_of<T, R>(type, s, upw, frac);
}
template <int T, class R, class V>
__device__ __forceinline__ R plane_interp_y(const Plane<V>& p, int r0, int tx, int type, R upw, R frac) {
    R s[6];
    const int w = width_of<T>(type);
#pragma unroll
    for (int m = 0; m < 6; ++m) {
        const int off = m - 3;
        s[m] = (off >= -w && off <= w - 1) ? R(p.v[r0 + m][tx + PH]) : R(0);
    }
    return interp_of<T, R>(type, s, upw, frac);
}
template <int HT, class R>
__device__ __forceinline__ R xmom_flux_x(const Params& P, const double* ru, const Plane<double>& pu, int c0, int ty,
                                         int i, int j, int k) {
    const Geo& g = P.g;
    R a = R(0.5) * (R(ld(ru, eidx(g, wrap(i - 1, g.nx), j, k))) + R(ld(ru, eidx(g, i, j, k))));
    return a * plane_interp_x<HT, R>(pu, ty, c0, P.dyc_h, a, R(P.f_dyc_h));
}
template <int HT, class R>
__device__ __forceinline__ R xmom_flux_y(const Params& P, const double* rv, const Plane<double>& pu, int tx, int r0,
                                         int i, int j, int k) {
    const Geo& g = P.g;
    R a = R(0.5) * (R(ld(rv, eidx(g, i, j, k))) + R(ld(rv, eidx(g, wrap(i - 1, g.nx), j, k))));
    return a * plane_interp_y<HT, R>(pu, r0, tx, P.dyc_h, a, R(P.f_dyc_h));
}
template <int VT, class R>
__device__ __forceinline__ R xmom_flux_z(const Params& P, const double* rw, const MostView& mv, int i, int j, int k) {
    const Geo& g = P.g;
    R a = R(0.5) * (R(ld(rw, eidx(g, i, j, k))) + R(ld(rw, eidx(g, wrap(i - 1, g.nx), j, k))));
    if (P.most && k < 3) return a * gatherz_most<VT, R>(P, mv, 0, P.dyc_v, a, R(P.f_dyc_v), i, j, k);
    return a * gatherz_tang<VT, R>(g, mv.u, P.dyc_v, a, R(P.f_dyc_v), i, j, k);
}
template <int HT, class R>
__device__ __forceinline__ R ymom_flux_x(const Params& P, const double* ru, const Plane<double>& pv, int c0, int ty,
                                         int i, int j, int k) {
    const Geo& g = P.g;
    R a = R(0.5) * (R(ld(ru, eidx(g, i, j, k))) + R(ld(ru, eidx(g, i, wrap(j - 1, g.ny), k))));
    return a * plane_interp_x<HT, R>(pv, ty, c0, P.dyc_h, a, R(P.f_dyc_h));
}
template <int HT, class R>
__device__ __forceinline__ R ymom_flux_y(const Params& P, const double* rv, const Plane<double>& pv, int tx, int r0,
                                         int i, int j, int k) {
    const Geo& g = P.g;
    R a = R(0.5) * (R(ld(rv, eidx(g, i, j, k))) + R(ld(rv, eidx(g, i, wrap(j - 1, g.ny), k))));
    return a * plane_interp_y<HT, R>(pv, r0, tx, P.dyc_h, a, R(P.f_dyc_h));
}
template <int VT, class R>
__device__ __forceinline__ R ymom_flux_z(const Params& P, const double* rw, const MostView& mv, int i, int j, int k) {
    const Geo& g = P.g;
    R a = R(0.5) * (R(ld(rw, eidx(g, i, j, k))) + R(ld(rw, eidx(g, i, wrap(j - 1, g.ny), k))));
    if (P.most && k < 3) return a * gatherz_most<VT, R>(P, mv, 1, P.dyc_v, a, R(P.f_dyc_v), i, j, k);
    return a * gatherz_tang<VT, R>(g, mv.v, P.dyc_v, a, R(P.f_dyc_v), i, j, k);
}
template <int HT, class R>
__device__ __forceinline__ R zmom_flux_x(const Params& P, const double* ru, const Plane<double>& pw, int c0, int ty,
                                         int i, int j, int k) {
    const Geo& g = P.g;
    R a = R(0.5) * (R(ld(ru, eidx(g, i, j, k))) + R(ld(ru, eidx(g, i, j, k - 1)))) * R(1);
    return a * plane_interp_x<HT, R>(pw, ty, c0, P.dyc_h, a, R(P.f_dyc_h));
}
template <int HT, class R>
__device__ __forceinline__ R zmom_flux_y(const Params& P, const double* rv, const Plane<double>& pw, int tx, int r0,
                                         int i, int j, int k) {
    const Geo& g = P.g;
    R a = R(0.5) * (R(ld(rv, eidx(g, i, j, k))) + R(ld(rv, eidx(g, i, j, k - 1)))) * R(1);
    return a * plane_interp_y<HT, R>(pw, r0, tx, P.dyc_h, a, R(P.f_dyc_h));
}
// Vertical flux of w between faces kk-1 and kk (the "lo" flux of face kk),
// with the order reduction next to the walls (ERF_AdvectionSrcForMom_N.H:
// 220-265); for kk == nz it is the "hi" flux of the top interior face,
// which the reference takes centred.
template <int VT, class R>
__device__ __forceinline__ R zmom_flux_z(const Params& P, const double* rw, const double* w, int i, int j, int kk) {
    const Geo& g = P.g;
    const int vt = P.dyc_v, lo_z_face = 0, hi_z_face = g.nz;
    const R vf = R(P.f_dyc_v);
    const Elem e0 = eidx(g, i, j, 0);
    auto wz = [&](int q) { return R(ld(w, e0 + (uint32_t)g.sk * (uint32_t)q)); };
    auto all = [&](int q, R upw, R frac, int type) {
        R sv[6];
        bool wide = (type == ERF_ADV_UPWIND_5TH || type == ERF_ADV_CENTERED_6TH);
        sv[0] = wide ? wz(q - 3) : R(0);
        sv[1] = (type == ERF_ADV_CENTERED_2ND) ? R(0) : wz(q - 2);
        sv[2] = wz(q - 1);
        sv[3] = wz(q);
        sv[4] = (type == ERF_ADV_CENTERED_2ND) ? R(0) : wz(q + 1);
        sv[5] = wide ? wz(q + 2) : R(0);
        return interp_all<R>(type, sv, upw, frac);
    };
    auto normal = [&](int q, R upw) {
        R sv[6];
        const int wd = width_of<VT>(vt);
        for (int m = 0; m < 6; ++m) {
            int off = m - 3;
            sv[m] = (off >= -wd && off <= wd - 1) ? wz(q + off) : R(0);
        }
        return interp_of<VT, R>(vt, sv, upw, vf);
    };
    R a = R(0.5) * (R(ld(rw, eidx(g, i, j, kk))) + R(ld(rw, eidx(g, i, j, kk - 1))));
    R iv;
    if (kk == hi_z_face || kk == lo_z_face + 1) iv = all(kk, a, R(0), ERF_ADV_CENTERED_2ND);
    else if (kk == lo_z_face + 2 || kk == hi_z_face - 1) {
        if (vt != ERF_ADV_CENTERED_2ND && vt != ERF_ADV_UPWIND_3RD) iv = all(kk, a, R(0), ERF_ADV_CENTERED_4TH);
        else iv = all(kk, a, vf, vt);
    } else iv = normal(kk, a);
    return a * iv;
}

// ---------------------------------------------------------------------------
// Slow RHS for the three momenta (erf_slow_rhs_pre face part,
// ERF_slow_rhs_pre.cpp:556-744): AdvectionSrcForMom (N), DiffusionSrcForMom_N,
// pressure gradient of p', buoyancy / Coriolis / geostrophic sources
// (make_mom_sources, make_buoyancy).  Same tiles as the scalar transport;
// the three momenta's x/y fluxes of a level are staged before one barrier.
// Buoyancy is evaluated in FP64 from the FP64 state (EOS), the rest in R.
// ---------------------------------------------------------------------------
template <class R, int HT, int VT>
__global__ void __launch_bounds__(TTX * TTY, ERFB_MINB_MOM) k_slow_mom(Params P, int kz, StateBuf S, StageAux<R> A,
                                                                       const double* __restrict__ u,
                                                                       const double* __restrict__ v,
                                                                       const double* __restrict__ w,
                                                                       const R* __restrict__ t11,
                                                                       const R* __restrict__ t22,
                                                                       const R* __restrict__ t33,
                                                                       const R* __restrict__ t12,
                                                                       const R* __restrict__ t13,
                                                                       const R* __restrict__ t23,
                                                                       const double* __restrict__ pavg,
                                                                       R* __restrict__ Fmx, R* __restrict__ Fmy,
                                                                       R* __restrict__ Fmz) {
    __shared__ FluxTile<R> sh[3];
    __shared__ Plane<double> pu, pv, pw;   // face velocities of the level, with halo
    const Geo& g = P.g;
    const int64_t N = g.ncell;
    const int tx = threadIdx.x, ty = threadIdx.y;
    const int i = blockIdx.x * TTX + tx, j = blockIdx.y * TTY + ty;
    const bool ok = i < g.nx && j < g.ny;
    const int k0 = blockIdx.z * kz, k1 = min(k0 + kz, g.nz);
    const int im = ok ? wrap(i - 1, g.nx) : 0, jm = ok ? wrap(j - 1, g.ny) : 0;
    const int ip = ok ? wrap(i + 1, g.nx) : 0, jp = ok ? wrap(j + 1, g.ny) : 0;
    const TileEdge edge = tile_edge(g);
    const PlaneIdx pidx(g);
    const R dxi = R(g.dxi), dyi = R(g.dyi), dzi = R(g.dzi);
    const MostView mv{u, v, S.cons};   // stage velocities (MOST ghosts below a MOST ground)
    const double* ru = S.mx;
    const double* rv = S.my;
    const double* rw = S.mz;
    const double* cd = S.cons;
    const R* prim = A.prim;
    const R* pp = A.pp;
    R zlu = R(0), zhu = R(0), zlv = R(0), zhv = R(0), zlw = R(0), zhw = R(0);
    double t_below = 0.0;   // temperature of the cell below (buoyancy type 2, moist)
    load_plane(g, pidx, pu, u, k0);
    load_plane(g, pidx, pv, v, k0);
    load_plane(g, pidx, pw, w, k0);
    for (int k = k0; k < k1; ++k) {
        const Elem c = ok ? eidx(g, i, j, k) : eidx(g, 0, 0, 0);
        const uint32_t sk = (uint32_t)g.sk;
        const bool zk = ok && k >= 1;   // z-momentum on interior faces only
        plane_wait();
        __syncthreads();
        if (ok) {
            sh[0].fx[ty][tx] = xmom_flux_x<HT, R>(P, ru, pu, tx, ty, i, j, k);
            sh[0].fy[ty][tx] = xmom_flux_y<HT, R>(P, rv, pu, tx, ty, i, j, k);
            if (k == k0) zlu = xmom_flux_z<VT, R>(P, rw, mv, i, j, k);
            zhu = xmom_flux_z<VT, R>(P, rw, mv, i, j, k + 1);
            sh[1].fx[ty][tx] = ymom_flux_x<HT, R>(P, ru, pv, tx, ty, i, j, k);
            sh[1].fy[ty][tx] = ymom_flux_y<HT, R>(P, rv, pv, tx, ty, i, j, k);
            if (k == k0) zlv = ymom_flux_z<VT, R>(P, rw, mv, i, j, k);
            zhv = ymom_flux_z<VT, R>(P, rw, mv, i, j, k + 1);
        }
        if (zk) {
            sh[2].fx[ty][tx] = zmom_flux_x<HT, R>(P, ru, pw, tx, ty, i, j, k);
            sh[2].fy[ty][tx] = zmom_flux_y<HT, R>(P, rv, pw, tx, ty, i, j, k);
            if (k == k0 || k == 1) zlw = zmom_flux_z<VT, R>(P, rw, w, i, j, k);
            zhw = zmom_flux_z<VT, R>(P, rw, w, i, j, k + 1);
        }
        // the tile's high-side halo faces (see TileEdge)
        if (edge.row >= 0) {
            const int r = edge.row, ih = wrap(edge.i0 + edge.nvx, g.nx), jr = edge.j0 + r;
            sh[0].fx[r][edge.nvx] = xmom_flux_x<HT, R>(P, ru, pu, edge.nvx, r, ih, jr, k);
            sh[1].fx[r][edge.nvx] = ymom_flux_x<HT, R>(P, ru, pv, edge.nvx, r, ih, jr, k);
            if (k >= 1) sh[2].fx[r][edge.nvx] = zmom_flux_x<HT, R>(P, ru, pw, edge.nvx, r, ih, jr, k);
        }
        if (edge.col >= 0) {
            const int cc = edge.col, ic = edge.i0 + cc, jh = wrap(edge.j0 + edge.nvy, g.ny);
            sh[0].fy[edge.nvy][cc] = xmom_flux_y<HT, R>(P, rv, pu, cc, edge.nvy, ic, jh, k);
            sh[1].fy[edge.nvy][cc] = ymom_flux_y<HT, R>(P, rv, pv, cc, edge.nvy, ic, jh, k);
            if (k >= 1) sh[2].fy[edge.nvy][cc] = zmom_flux_y<HT, R>(P, rv, pw, cc, edge.nvy, ic, jh, k);
        }
        __syncthreads();
        if (k + 1 < k1) {   // next level's planes arrive during the right-hand sides below
            load_plane(g, pidx, pu, u, k + 1);
            load_plane(g, pidx, pv, v, k + 1);
            load_plane(g, pidx, pw, w, k + 1);
        }
        // ---------------- x-momentum on face i
        if (ok) {
            R rhs = -((sh[0].fx[ty][tx + 1] - sh[0].fx[ty][tx]) * dxi * R(1) +
                      (sh[0].fy[ty + 1][tx] - sh[0].fy[ty][tx]) * dyi * R(1) + (zhu - zlu) * dzi);
            zlu = zhu;
            if (P.use_diff)
                rhs -= ((ld(t11, c) - ld(t11, eidx(g, im, j, k))) * dxi * R(1) + (ld(t12, eidx(g, i, jp, k)) - ld(t12, c)) * dyi * R(1) +
                        (ld(t13, c + sk) - ld(t13, c)) * dzi);
            R gpx = dxi * (ld(pp, c) - ld(pp, eidx(g, im, j, k)));
            gpx *= R(1);
            R q = R(0);
            if (P.moist) q = R(0.5) * (ld(prim + 4 * N, c) + ld(prim + 4 * N, eidx(g, im, j, k)) + ld(prim + 5 * N, c) + ld(prim + 5 * N, eidx(g, im, j, k)));
            R src = R(0);
            if (P.coriolis) {
                R rvl = R(0.25) * (R(ld(rv, eidx(g, i, jp, k))) + R(ld(rv, c)) + R(ld(rv, eidx(g, im, jp, k))) + R(ld(rv, eidx(g, im, j, k))));
                R rwl = R(0.25) * (R(ld(rw, c + sk)) + R(ld(rw, c)) + R(ld(rw, eidx(g, i, jm, k + 1))) + R(ld(rw, eidx(g, i, jm, k))));
                src += R(P.cf) * (rvl * R(P.sinphi) - rwl * R(P.cosphi));
            }
            src += R(0.5) * (R(ld(cd, c)) + R(ld(cd, eidx(g, im, j, k)))) * R(P.geo0);
            rhs += (-gpx - R(0)) / (R(1) + q) + src;
            at(Fmx, c) = rhs;
        }
        // ---------------- y-momentum on face j
        if (ok) {
            R rhs = -((sh[1].fx[ty][tx + 1] - sh[1].fx[ty][tx]) * dxi * R(1) +
                      (sh[1].fy[ty + 1][tx] - sh[1].fy[ty][tx]) * dyi * R(1) + (zhv - zlv) * dzi);
            zlv = zhv;
            if (P.use_diff)
                rhs -= ((ld(t12, eidx(g, ip, j, k)) - ld(t12, c)) * dxi * R(1) + (ld(t22, c) - ld(t22, eidx(g, i, jm, k))) * dyi * R(1) +
                        (ld(t23, c + sk) - ld(t23, c)) * dzi);
            R gpy = dyi * (ld(pp, c) - ld(pp, eidx(g, i, jm, k)));
            gpy *= R(1);
            R q = R(0);
            if (P.moist) q = R(0.5) * (ld(prim + 4 * N, c) + ld(prim + 4 * N, eidx(g, i, jm, k)) + ld(prim + 5 * N, c) + ld(prim + 5 * N, eidx(g, i, jm, k)));
            R src = R(0);
            if (P.coriolis) {
                R rul = R(0.25) * (R(ld(ru, eidx(g, ip, j, k))) + R(ld(ru, c)) + R(ld(ru, eidx(g, ip, jm, k))) + R(ld(ru, eidx(g, i, jm, k))));
                src += -R(P.cf) * rul * R(P.sinphi);
            }
            src += R(0.5) * (R(ld(cd, c)) + R(ld(cd, eidx(g, i, jm, k)))) * R(P.geo1);
            rhs += (-gpy - R(0)) / (R(1) + q) + src;
            at(Fmy, c) = rhs;
        }
        // ---------------- z-momentum on face k
        if (ok && k == 0) at(Fmz, c) = R(0);
        if (zk) {
            R rhs = -((sh[2].fx[ty][tx + 1] - sh[2].fx[ty][tx]) * dxi * R(1) +
                      (sh[2].fy[ty + 1][tx] - sh[2].fy[ty][tx]) * dyi * R(1) + (zhw - zlw) * dzi);
            zlw = zhw;
            if (P.use_diff)
                rhs -= ((ld(t13, eidx(g, ip, j, k)) - ld(t13, c)) * dxi * R(1) + (ld(t23, eidx(g, i, jp, k)) - ld(t23, c)) * dyi * R(1) +
                        (ld(t33, c) - ld(t33, c - sk)) * dzi);
            double b;
            double g2 = -P.gravity;
            if (!P.moist) {
                if (P.buoy_type == 1) {
                    b = g2 * 0.5 * ((ld(cd, c) - P.r0[k + 1]) + (ld(cd, c - sk) - P.r0[k]));
                } else {
                    auto T0 = [&](int kk) {
                        double rt0 = eos_rt_given_p(P.p0[kk + 1]);
                        return (rt0 / P.r0[kk + 1]) / pow(p_0 / P.p0[kk + 1], P.rdOcp);
                    };
                    double t0h = T0(k), th_ = eos_T(ld(cd, c), ld(cd + N, c), 0.0);
                    double t0l = T0(k - 1), tl_ = eos_T(ld(cd, c - sk), ld(cd + N, c - sk), 0.0);
                    double qp_ = (th_ - t0h) / t0h, qm_ = (tl_ - t0l) / t0l;
                    double r0q = 0.5 * (P.r0[k + 1] * qp_ + P.r0[k] * qm_);
                    b = -r0q * g2;
                }
            } else if (P.buoy_type == 1) {
                int nq = P.ncomp - ERF_RHOQ1_COMP;
                double hi = ld(cd, c) + ld(cd + 5 * N, c) + ld(cd + 6 * N, c) - P.r0[k + 1];
                double lo = ld(cd, c - sk) + ld(cd + 5 * N, c - sk) + ld(cd + 6 * N, c - sk) - P.r0[k];
                for (int qo = 2; qo < nq; ++qo) { hi += ld(cd + (5 + qo) * N, c); lo += ld(cd + (5 + qo) * N, c - sk); }
                b = g2 * 0.5 * (hi + lo);
            } else {
                int nq = P.ncomp - ERF_RHOQ1_COMP;
                const double* rd = pavg;
                const double* thd = pavg + g.nz;
                const double* qvd = pavg + 2 * g.nz;
                const double* qcd = pavg + 3 * g.nz;
                const double* qpd = pavg + 4 * g.nz;
                (void)thd;
                double tp1 = pavg[5 * g.nz + k], tm1 = pavg[5 * g.nz + k - 1];
                // cell temperatures: this level's, and the one below carried
                // up the block's column (evaluated once per cell)
                double tp3 = eos_T(ld(cd, c), ld(cd + N, c), ld(cd + 5 * N, c) / ld(cd, c));
                double tm3 = (k == k0 || k == 1) ? eos_T(ld(cd, c - sk), ld(cd + N, c - sk), ld(cd + 5 * N, c - sk) / ld(cd, c - sk))
                                       : t_below;
                t_below = tp3;
                double qvp = nq >= 1 ? ld(prim + 4 * N, c) : 0.0, qvm = nq >= 1 ? ld(prim + 4 * N, c - sk) : 0.0;
                double qcp = nq >= 2 ? ld(prim + 5 * N, c) : 0.0, qcm = nq >= 2 ? ld(prim + 5 * N, c - sk) : 0.0;
                double qpp = nq >= 3 ? ld(prim + 6 * N, c) : 0.0, qpm = nq >= 3 ? ld(prim + 6 * N, c - sk) : 0.0;
                double qplus = 0.61 * (qvp - qvd[k]) - (qcp - qcd[k] + qpp - qpd[k]) + (tp3 - tp1) / tp1 * (1.0 + 0.61 * qvd[k] - qcd[k] - qpd[k]);
                double qminus = 0.61 * (qvm - qvd[k - 1]) - (qcm - qcd[k - 1] + qpm - qpd[k - 1]) + (tm3 - tm1) / tm1 * (1.0 + 0.61 * qvd[k - 1] - qcd[k - 1] - qpd[k - 1]);
                double qavg = 0.5 * (qplus + qminus);
                double r0avg = 0.5 * (rd[k] + rd[k - 1]);
                b = -qavg * r0avg * g2;
            }
            R zsrc = R(b);
            if (P.coriolis) {
                R rul = R(0.25) * (R(ld(ru, eidx(g, ip, j, k))) + R(ld(ru, c)) + R(ld(ru, eidx(g, ip, j, k - 1))) + R(ld(ru, c - sk)));
                zsrc += R(P.cf) * rul * R(P.cosphi);
            }
            zsrc += R(0.5) * (R(ld(cd, c)) + R(ld(cd, c - sk))) * R(P.geo2);
            R gpz = dzi * (ld(pp, c) - ld(pp, c - sk)) / R(1);
            R q = R(0);
            if (P.moist) q = R(0.5) * (ld(prim + 4 * N, c) + ld(prim + 4 * N, c - sk) + ld(prim + 5 * N, c) + ld(prim + 5 * N, c - sk));
            rhs += (zsrc - gpz - R(0)) / (R(1) + q);
            at(Fmz, c) = rhs;
        }
        if (ok && k == g.nz - 1) at(Fmz, c + sk) = R(0);
        // the next level's first barrier orders the reuse of sh
    }
}

// ---------------------------------------------------------------------------
// Host launchers: scheme dispatch, grid sizing and the explicit
// instantiations for the plain (double) and mixed (float) forms.
// ---------------------------------------------------------------------------
namespace {


dim3 cell_block() { return dim3(32, 4, 1); }
dim3 cell_grid(const Geo& g) { return dim3((g.nx + 31) / 32, (g.ny + 3) / 4, g.nz); }

constexpr int U5 = ERF_ADV_UPWIND_5TH, W5 = ERF_ADV_WENO_5;
constexpr int U3 = ERF_ADV_UPWIND_3RD, W3 = ERF_ADV_WENO_3;   // the reference's defaults

template <class R>
using SlowCellK = void (*)(Params, int, StateBuf, StageAux<R>, const R*, const R*, const R*, const R*, TkeBuf<R>, R*, R*,
                           R*, R*);
template <class R>
using SlowMomK = void (*)(Params, int, StateBuf, StageAux<R>, const double*, const double*, const double*, const R*,
                          const R*, const R*, const R*, const R*, const R*, const double*, R*, R*, R*);
template <class R>
using PostK = void (*)(Params, int, PostArgs<R>);

template <class R>
SlowCellK<R> slow_cell_kernel(const Params& P) {
    if (P.dyc_h == U5 && P.dyc_v == U5) return k_slow_cell<R, U5, U5>;
    if (P.dyc_h == U3 && P.dyc_v == U3) return k_slow_cell<R, U3, U3>;
    return k_slow_cell<R, -1, -1>;
}
template <class R>
SlowMomK<R> slow_mom_kernel(const Params& P) {
    if (P.dyc_h == U5 && P.dyc_v == U5) return k_slow_mom<R, U5, U5>;
    if (P.dyc_h == U3 && P.dyc_v == U3) return k_slow_mom<R, U3, U3>;
    return k_slow_mom<R, -1, -1>;
}
int post_jobs(const Params& P) {
    return (P.moist ? 1 + (P.ncomp - ERF_RHOQ1_COMP) : 1) + (P.les == ERF_LES_DEARDORFF ? 1 : 0);
}
template <class R>
PostK<R> post_kernel(const Params& P) {
    const bool dw = P.dry_h == W5 && P.dry_v == W5, du = P.dry_h == U5 && P.dry_v == U5, d3 = P.dry_h == U3 && P.dry_v == U3;
    const bool mw = P.moi_h == W5 && P.moi_v == W5, mu = P.moi_h == U5 && P.moi_v == U5, m3 = P.moi_h == W3 && P.moi_v == W3;
    if (!P.moist) {
        if (dw) return k_post<R, W5, W5, W5, W5>;
        if (du) return k_post<R, U5, U5, W5, W5>;
        if (d3) return k_post<R, U3, U3, W3, W3>;
        return k_post<R, -1, -1, -1, -1>;
    }
    if (mw) {
        if (dw) return k_post<R, W5, W5, W5, W5>;
        if (du) return k_post<R, U5, U5, W5, W5>;
        if (d3) return k_post<R, U3, U3, W5, W5>;
    }
    if (m3) {
        if (dw) return k_post<R, W5, W5, W3, W3>;
        if (du) return k_post<R, U5, U5, W3, W3>;
        if (d3) return k_post<R, U3, U3, W3, W3>;
    }
    if (du && mu) return k_post<R, U5, U5, U5, U5>;
    return k_post<R, -1, -1, -1, -1>;
}

}  // namespace

template <class R>
void tiled_setup(const Params& P, TiledKz* t) {
    t->cell = pick_kz(slow_cell_kernel<R>(P), P.g);
    t->mom = pick_kz(slow_mom_kernel<R>(P), P.g);
    t->post = pick_kz(post_kernel<R>(P), P.g, post_jobs(P));
}

// The dynamic shared-memory opt-in is a property of the kernel for the whole
// process, shared by every context: it is raised to the device maximum (the
// size passed at launch still sets each launch's footprint), so that contexts
// of different sizes never lower it below one another's needs.
template <class R>
int coef_setup(size_t coef_smem) {
    int dev = 0, maxopt = 0;
    cudaGetDevice(&dev);
    if (cudaDeviceGetAttribute(&maxopt, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess) return 1;
    if (coef_smem > (size_t)maxopt) return 1;
    return cudaFuncSetAttribute(k_fast_coef<R>, cudaFuncAttributeMaxDynamicSharedMemorySize, maxopt) != cudaSuccess;
}

template <class R>
void launch_step_begin(const Params& P, cudaStream_t st, const double* cons, const double* uo, const double* vo,
                       const double* wo, StateBuf S, double* un, double* vn, double* wn, StageAux<R> A, R* mut,
                       TkeBuf<R> tke) {
    k_step_begin<R><<<cell_grid(P.g), cell_block(), 0, st>>>(P, cons, uo, vo, wo, S, un, vn, wn, A, mut, tke);
}
template <class R>
void launch_stage_aux(const Params& P, cudaStream_t st, const double* cons, StageAux<R> A) {
    k_stage_aux<R><<<cell_grid(P.g), cell_block(), 0, st>>>(P, cons, A);
}
template <class R>
void launch_tau(const Params& P, cudaStream_t st, const double* cons, const double* u, const double* v,
                const double* w, const R* mut, R* t11, R* t22, R* t33, R* t12, R* t13, R* t23) {
    k_tau<R><<<cell_grid(P.g), cell_block(), 0, st>>>(P, cons, u, v, w, mut, t11, t22, t33, t12, t13, t23);
    if (P.most)   // the validated MOST configurations carry an eddy-viscosity closure
        k_tau_most_ground<R><<<dim3((P.g.nx + 31) / 32, (P.g.ny + 3) / 4), dim3(32, 4), 0, st>>>(P, cons, u, v, w, mut,
                                                                                               t13, t23);
}
template <class R>
void launch_plane_avg(const Params& P, cudaStream_t st, const double* cons, const R* prim, double* avg) {
    k_plane_avg<R><<<dim3(P.g.nz, PAVG_PARTS), 256, 0, st>>>(P, cons, prim, avg);
}
// ABLMost::update_fluxes (BoundaryConditions/ERF_ABLMost.cpp:11-142) on the
// step's old velocities: plane means of u and v on their faces (the periodic
// high face excluded) and of sqrt(uc^2 + vc^2) at the cell centres of level
// most_k (MOSTAverage::compute_plane_averages, ERF_MOSTAverage.cpp:674-940),
// then u* = kappa |U| / ln(z_ref / z0) of the adiabatic surface
// (ERF_MOSTStress.H:89-124).  One block; each thread sums a fixed stride and
// the partial sums are added in a fixed tree, so the result is reproducible.
constexpr int MOST_THREADS = 512;
__global__ void __launch_bounds__(MOST_THREADS) k_most_avg(Params P, const double* __restrict__ u,
                                                           const double* __restrict__ v) {
    __shared__ double red[3][MOST_THREADS];
    const Geo& g = P.g;
    const int k = P.most_k;
    double su = 0.0, sv = 0.0, sm = 0.0;
    for (int64_t q = threadIdx.x; q < g.sk; q += MOST_THREADS) {
        const int i = (int)(q % g.nx), j = (int)(q / g.nx);
        const double uf = u[cidx(g, i, j, k)], vf = v[cidx(g, i, j, k)];
        su += uf;
        sv += vf;
        const double uc = 0.5 * (uf + u[cidx(g, wrap(i + 1, g.nx), j, k)]);
        const double vc = 0.5 * (vf + v[cidx(g, i, wrap(j + 1, g.ny), k)]);
        sm += sqrt(uc * uc + vc * vc + 0.0 * 0.0);
    }
    red[0][threadIdx.x] = su;
    red[1][threadIdx.x] = sv;
    red[2][threadIdx.x] = sm;
    __syncthreads();
    for (int h = MOST_THREADS / 2; h > 0; h >>= 1) {
        if (threadIdx.x < h)
            for (int q = 0; q < 3; ++q) red[q][threadIdx.x] += red[q][threadIdx.x + h];
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        const double denom = 1.0 / (double)g.sk;
        P.most_avg[0] = red[0][0] * denom;
        P.most_avg[1] = red[1][0] * denom;
        P.most_avg[2] = red[2][0] * denom;
        P.most_avg[3] = 0.41 * P.most_avg[2] / log(P.most_zref / P.most_z0);
    }
}
void launch_most_avg(const Params& P, cudaStream_t st, const double* u, const double* v) {
    k_most_avg<<<1, MOST_THREADS, 0, st>>>(P, u, v);
}
template <class R>
void launch_no_substep(const Params& P, cudaStream_t st, double slow_dt, StateBuf Sold, const R* Fcons, const R* Fmx,
                       const R* Fmy, const R* Fmz, StateBuf Ssum) {
    k_no_substep<R><<<cell_grid(P.g), cell_block(), 0, st>>>(P.g, slow_dt, Sold, Fcons, Fmx, Fmy, Fmz, Ssum);
}
template <class R>
void launch_fast_coef(const Params& P, cudaStream_t st, dim3 grid, dim3 block, size_t smem, double D, StateBuf Sst,
                      StageAux<R> A, R* cA, R* cInvB, R* cCB, R* cP, R* cQ) {
    k_fast_coef<R><<<grid, block, smem, st>>>(P, D, Sst, A, cA, cInvB, cCB, cP, cQ);
}
template <class R>
void launch_slow_cell(const Params& P, const TiledKz& t, cudaStream_t st, StateBuf S, StageAux<R> A, const R* mut,
                      const R* hx, const R* hy, const R* hz, TkeBuf<R> tke, R* Fcons, R* avx, R* avy, R* avz) {
    slow_cell_kernel<R>(P)<<<tile_grid(P.g, t.cell), dim3(TTX, TTY, 1), 0, st>>>(P, t.cell, S, A, mut, hx, hy, hz,
                                                                                  tke, Fcons, avx, avy, avz);
}
template <class R>
void launch_slow_mom(const Params& P, const TiledKz& t, cudaStream_t st, StateBuf S, StageAux<R> A, const double* u,
                     const double* v, const double* w, const R* t11, const R* t22, const R* t33, const R* t12,
                     const R* t13, const R* t23, const double* pavg, R* Fmx, R* Fmy, R* Fmz) {
    slow_mom_kernel<R>(P)<<<tile_grid(P.g, t.mom), dim3(TTX, TTY, 1), 0, st>>>(P, t.mom, S, A, u, v, w, t11, t22, t33,
                                                                                t12, t13, t23, pavg, Fmx, Fmy, Fmz);
}
template <class R>
void launch_post(const Params& P, const TiledKz& t, cudaStream_t st, double slow_dt, StateBuf Sold, StateBuf Sst,
                 StateBuf Ssum, StateBuf Snew, StageAux<R> Acur, StageAux<R> Anext, int make_next, const double* keep,
                 const R* mut, TkeBuf<R> tke, const R* avx, const R* avy, const R* avz, double* un, double* vn,
                 double* wn) {
    const PostArgs<R> a{slow_dt, Sold, Sst, Ssum, Snew, Acur, Anext, make_next, keep, mut, tke, avx, avy, avz, un, vn, wn};
    post_kernel<R>(P)<<<tile_grid(P.g, t.post, post_jobs(P)), dim3(TTX, TTY, 1), 0, st>>>(P, t.post, a);
}

#define ERFB_INSTANTIATE(R)                                                                                          \
    template void tiled_setup<R>(const Params&, TiledKz*);                                                           \
    template int coef_setup<R>(size_t);                                                                              \
    template void launch_step_begin<R>(const Params&, cudaStream_t, const double*, const double*, const double*,     \
                                       const double*, StateBuf, double*, double*, double*, StageAux<R>, R*,          \
                                       TkeBuf<R>);                                                                   \
    template void launch_tau<R>(const Params&, cudaStream_t, const double*, const double*, const double*,            \
                                const double*, const R*, R*, R*, R*, R*, R*, R*);                                    \
    template void launch_plane_avg<R>(const Params&, cudaStream_t, const double*, const R*, double*);                \
    template void launch_stage_aux<R>(const Params&, cudaStream_t, const double*, StageAux<R>);                      \
    template void launch_no_substep<R>(const Params&, cudaStream_t, double, StateBuf, const R*, const R*, const R*, \
                                       const R*, StateBuf);                                                          \
    template void launch_fast_coef<R>(const Params&, cudaStream_t, dim3, dim3, size_t, double, StateBuf,             \
                                      StageAux<R>, R*, R*, R*, R*, R*);                                              \
    template void launch_slow_cell<R>(const Params&, const TiledKz&, cudaStream_t, StateBuf, StageAux<R>, const R*,  \
                                      const R*, const R*, const R*, TkeBuf<R>, R*, R*, R*, R*);                      \
    template void launch_slow_mom<R>(const Params&, const TiledKz&, cudaStream_t, StateBuf, StageAux<R>,             \
                                     const double*, const double*, const double*, const R*, const R*, const R*,      \
                                     const R*, const R*, const R*, const double*, R*, R*, R*);                       \
    template void launch_post<R>(const Params&, const TiledKz&, cudaStream_t, double, StateBuf, StateBuf, StateBuf,  \
                                 StateBuf, StageAux<R>, StageAux<R>, int, const double*, const R*, TkeBuf<R>,        \
                                 const R*, const R*, const R*, double*, double*, double*);

ERFB_INSTANTIATE(double)
ERFB_INSTANTIATE(float)
#undef ERFB_INSTANTIATE

}  // namespace erfb
