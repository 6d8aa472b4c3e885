// kessler.cu -- Kessler warm-rain microphysics (Microphysics/Kessler/
// ERF_Kessler.cpp:11-185, ERF_Init_Kessler.cpp:64-99, ERF_Update_Kessler.cpp:
// 14-40), one thread per cell, in place on a view of the conserved variables.
//
// A cell's update reads its neighbours above and below only through the rain
// falling through its faces, so every component but the rain is updated in
// place; the rain is read from one array and written to another (the step
// keeps the two apart anyway, the standalone entries stage it and
// k_kessler_rain puts it back).  A block holds 32 columns x KESS_KB levels:
// each thread evaluates the fall flux through its bottom face and takes its
// top face's from the thread above (the block's top level evaluates its own).
//
// Bound: HBM once the powers are out of the way: 9 values per cell (rain).
// The powers of the fall flux and of evaporation are taken only where there
// is rain, share their logarithms, x^(-1/2) is one rsqrt and evaporation has
// one denominator; the level below comes from the thread below.  The
// saturation chain (one power, one division after another) is what is left.
// Standalone call, 128x128x80: 409 us with one thread per column and a
// staging copy of all components on either side, 66 us now (72 with its own
// quotients per neighbour level and the reference's order of divisions).
#include "kernels.cuh"

namespace erfb {
namespace {

__global__ void __launch_bounds__(32 * KESS_KB) k_kessler(Params P, KessView v, KessLin rin, KessLin rout, double dtn,
                                                          double dzi) {
    __shared__ double sr[KESS_KB + 1][32], sq[KESS_KB + 1][32], sfz[KESS_KB][32];   // [0]: the level below the block
    const Geo& g = P.g;
    const int L = threadIdx.x, col = blockIdx.x * 32 + L, tz = threadIdx.y, k = blockIdx.y * KESS_KB + tz;
    const int nz = g.nz;
    const bool live = col < (int)g.sk && k < nz;
    const int j = live ? col / g.nx : 0, i = live ? col - j * g.nx : 0, kk = live ? k : 0;
    const bool rain = P.kessler_rain;
    const int64_t c = i + j * v.js + kk * v.ks;
    const int64_t r = i + j * rin.js + kk * rin.ks;
    auto flux = [&](double ra, double qa) {
        if (!(qa > 0.0)) return 0.0;
        const double Vt = 36.34 * powxy(ra * 0.001 * qa, 0.1346) * rsqrt(ra * (1.0 / 1.16));
        const double f = ra * Vt * qa;
        return (fabs(f) < 1e-14) ? 0.0 : f;
    };
    const double rho = v.p[c], ir = 1.0 / rho;
    double qp = 0.0, fz_lo = 0.0;
    if (rain) {
        qp = rin.p[r] * ir;
        sr[tz + 1][L] = rho;
        sq[tz + 1][L] = qp;
        if (tz == 0 && live && k > 0) {
            const double rd = v.p[c - v.ks];
            sr[0][L] = rd;
            sq[0][L] = rin.p[r - rin.ks] / rd;
        }
        __syncthreads();
        if (live) fz_lo = k == 0 ? flux(rho, qp) : flux(0.5 * (sr[tz][L] + rho), 0.5 * (sq[tz][L] + qp));
        sfz[tz][L] = fz_lo;
        __syncthreads();
    }
    if (!live) return;
    const double rt = v.p[v.ns + c];
    double theta = rt * ir;
    double qv = v.p[5 * v.ns + c] * ir;
    double qc = v.p[6 * v.ns + c] * ir;
    const double p_pa = eos_p(rt, qv);
    const double tabs = p_pa / (R_d * rho * (1.0 + R_v / R_d * qv));   // eos_T with p formed once
    const double pres = p_pa * 0.01, ip = 1.0 / pres;
    const double fac_cond = lcond / P.c_p;
    const double es = esatw(tabs);
    double qs = Rd_on_Rv * es / fmax(es, pres - es);
    const double dqs = Rd_on_Rv * dtesatw(tabs) * ip;
    const double fac = 1.0 + (L_v / Cp_d) * dqs;
    qc = fmax(0.0, qc);
    if (rain) {
        qv = fmax(0.0, qv);
        qp = fmax(0.0, qp);
        if (qs <= 0.0) qs = 0.0;
    }
    double d_v2c = 0.0, d_c2v = 0.0;
    {
        const double d = fabs(qv - qs) / (1.0 + fac);
        if (qv > qs) d_v2c = fmin(qv, d);
        if (qv < qs && qc > 0.0) d_c2v = fmin(qc, d);
    }
    double d_r2v = 0.0;
    if (rain) {
        double fz_hi;
        if (k == nz - 1) fz_hi = flux(rho, rin.p[r] * ir);
        else if (tz + 1 < KESS_KB) fz_hi = sfz[tz + 1][L];
        else {
            const double ru = v.p[c + v.ks];
            fz_hi = flux(0.5 * (rho + ru), 0.5 * (rin.p[r] * ir + rin.p[r + rin.ks] / ru));
        }
        if (qp > 0.0 && qv < qs) {
            const double l = log(0.001 * rho * qp);
            const double C = 1.6 + 124.9 * exp(0.2046 * l);
            // (1 - qv / qs) / (5.4e5 + 2.55e6 / (p qs)) over one denominator
            d_r2v = 1000.0 * ir * C * exp(0.525 * l) * ((qs - qv) * pres / (5.4e5 * pres * qs + 2.55e6)) * dtn;
            d_r2v = fmin(qp, d_r2v);
        }
        double d_c2r = 0.0;
        if (qc > 0.0) {
            const double auto_r = (qc > 1.e-3) ? 1.e-3 : 0.0;
            const double accrr = qp > 0.0 ? 2.2 * powxy(qp, 0.875) : 0.0;
            d_c2r = fmin(dtn * (accrr * qc + auto_r * (qc - 1.e-3)), qc);
        }
        // over terrain the fall-flux divergence is per unit computational volume
        // (dJinv, ERF_Kessler.cpp:82-97)
        const double dJinv = P.ter ? 1.0 / P.detJ[cidx(g, i, j, k)] : 1.0;
        double dq_sed = dtn * dJinv * ir * (fz_hi - fz_lo) * dzi;
        if (fabs(dq_sed) < 1e-14) dq_sed = 0.0;
        qv += -d_v2c + d_c2v + d_r2v;
        qc += d_v2c - d_c2v - d_c2r;
        qp += dq_sed + d_c2r - d_r2v;
        rout.p[i + j * rout.js + k * rout.ks] = rho * fmax(0.0, qp);
    } else {
        qv += -d_v2c + d_c2v;
        qc += d_v2c - d_c2v;
    }
    theta += theta / tabs * fac_cond * (d_v2c - d_c2v - d_r2v);
    v.p[v.ns + c] = rho * theta;
    v.p[5 * v.ns + c] = rho * fmax(0.0, qv);
    v.p[6 * v.ns + c] = rho * fmax(0.0, qc);
}

// The staged rain back into the caller's view, and every ghost cell that the
// view covers (periodic laterally, the nearest level vertically).
__global__ void k_kessler_rain(Geo g, erf_b200_fab f, int ncomp, int rain, const double* __restrict__ stage) {
    const int nxb = f.hi[0] - f.lo[0] + 1, nyb = f.hi[1] - f.lo[1] + 1;
    const int ib = blockIdx.x * blockDim.x + threadIdx.x, jb = blockIdx.y * blockDim.y + threadIdx.y, kb = blockIdx.z;
    if (ib >= nxb || jb >= nyb || kb > f.hi[2] - f.lo[2]) return;
    const int i = f.lo[0] + ib, j = f.lo[1] + jb, k = f.lo[2] + kb;
    const int ii = ((i % g.nx) + g.nx) % g.nx, jj = ((j % g.ny) + g.ny) % g.ny, kk = clampk(k, g.nz);
    const int64_t dst = ib + jb * f.jstride + kb * f.kstride;
    const int64_t src = (ii - f.lo[0]) + (jj - f.lo[1]) * f.jstride + (kk - f.lo[2]) * f.kstride;
    if (src != dst)
        for (int n = 0; n < ncomp; ++n)
            if (!(rain && n == 7)) f.p[dst + n * f.nstride] = f.p[src + n * f.nstride];
    if (rain) f.p[dst + 7 * f.nstride] = stage[cidx(g, ii, jj, kk)];
}
}  // namespace

void launch_kessler(const Params& P, cudaStream_t st, KessView v, KessLin rin, KessLin rout, double dt, double dz) {
    const dim3 grid((unsigned)((P.g.sk + 31) / 32), (unsigned)((P.g.nz + KESS_KB - 1) / KESS_KB));
    k_kessler<<<grid, dim3(32, KESS_KB), 0, st>>>(P, v, rin, rout, dt, 1.0 / dz);
}

// The microphysics of a caller's view; stage: a cell's worth of doubles (rain only).
cudaError_t launch_kessler_fab(const Params& P, cudaStream_t st, const erf_b200_fab& f, double* stage, double dt,
                               double dz) {
    const Geo& g = P.g;
    KessView v;
    v.p = f.p - f.lo[0] - f.lo[1] * f.jstride - f.lo[2] * f.kstride;
    v.js = f.jstride; v.ks = f.kstride; v.ns = f.nstride;
    const int rain = P.kessler_rain;
    launch_kessler(P, st, v, KessLin{v.p + 7 * v.ns, v.js, v.ks}, KessLin{stage, g.nx, g.sk}, dt, dz);
    const int nxb = f.hi[0] - f.lo[0] + 1, nyb = f.hi[1] - f.lo[1] + 1, nzb = f.hi[2] - f.lo[2] + 1;
    if (cudaError_t e = cudaGetLastError()) return e;
    if (rain || nxb > g.nx || nyb > g.ny || nzb > g.nz)
        k_kessler_rain<<<dim3((nxb + 31) / 32, (nyb + 7) / 8, nzb), dim3(32, 8), 0, st>>>(g, f, P.ncomp, rain, stage);
    return cudaGetLastError();
}

}  // namespace erfb
