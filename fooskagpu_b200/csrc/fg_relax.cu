// Phase relaxation (FP64): partition by saturation temperature, thermal (p, T) equilibrium
// Newton and chemical (p, T, Gibbs) equilibrium Newton, one thread per cell.
// Restates DP/relaxation.cu:4-75, DP/thermRlx.cu:4-235, DP/chemRlx.cu:4-267 on the device;
// the partition is decided per cell in the same kernel instead of atomic-append lists
// (cells are independent, so the result is identical and deterministic).
// Every Newton loop is bounded by the reference's iteration caps (thermItrMax, chemItrMax,
// 50 for the saturation temperature, urf > 0.0005 for step halving).
//
// With a surrogate attached, a chemical cell inside the network's training hull starts from the
// network's equilibrium prediction and takes at most `polishIters` full Newton steps on the
// reference's residuals; it is accepted when every relative residual is within `relTol`,
// otherwise (and outside the hull) the cell takes the reference Newton unchanged.
#include "fg_kernels.cuh"
#include "fg_sg_tc.cuh"

namespace fg {

namespace {

// The Newtons are compiled into several kernels (with and without the surrogate, for few and for many
// cells), whose states agree bitwise: where a product has more than one use, or two products meet in a
// sum, the roundings are written out, so that no instantiation contracts them its own way.

// u^2 + v^2 + w^2
__device__ __forceinline__ double sq_rn(double u, double v, double w) { return fma_rn(w, w, fma_rn(u, u, mul_rn(v, v))); }
// a b - c d
__device__ __forceinline__ double diff_rn(double a, double b, double c, double d) { return fma_rn(a, b, -mul_rn(c, d)); }

// pressure and temperature of phase m at density r and internal energy e (DP/eqos.h); the phase
// constants are precomputed once per launch (RelaxParams)
__device__ __forceinline__ double p_of(const RelaxParams &R, int m, double r, double e) {
    return fma_rn(-R.gm1eta[m], r, fma_rn(mul_rn(R.gm1[m], r), e, -R.gpinf[m]));
}
__device__ __forceinline__ double t_of(const RelaxParams &R, int m, double r, double e) {
    return (p_of(R, m, r, e) + R.pinf[m]) / (R.cvgm1[m] * r);
}

// log10(1 + d) for |d| < kSmallLog by the Taylor series of the logarithm, truncated below 1e-18 of
// the value: the forward differences of the Newton solves change the argument of a logarithm by
// 1e-3 .. 1e-8 of itself, and the series gives that change directly, without the cancellation of
// two logarithms and at a tenth of the cost of the second one
constexpr double kLog10e = 0.43429448190325182765, kSmallLog = 1e-3;
__device__ __forceinline__ double log10_1p(double d, double base = 0.0) {
    const double s = fma_rn(d, fma_rn(d, fma_rn(d, fma_rn(d, fma_rn(d, -1.0 / 6, 1.0 / 5), -1.0 / 4), 1.0 / 3), -1.0 / 2), 1.0);
    return fma_rn(mul_rn(kLog10e, d), s, base);   // base + log10(1 + d)
}

// Newton on the saturation temperature (DP/relaxation.cu:4-38) with the reference's forward
// difference dT = 1e-3 K.  The difference f(T + dT) - f(T) of f = A + B / T + C log10 T comes from the
// series in d = dT / T, so an iteration takes one logarithm and two divisions (partition of the 981 k-tet
// bubble: 66 -> 43 us; of the jet, most of whose cells are below chemLimit and skip it: 122 -> 12 us).
__device__ double sat_temp(const RelaxParams &R, double P, double temp, double urf) {
    const double etaT2 = R.satConst[0] * log10(P) + R.satConst[1];
    const double dT = 1.e-3;
    const double rest = (R.satA + etaT2) * R.satQ + R.satD * log10(P + R.pinf[0]) - log10(P);
    double fun = 1, T = temp;
    for (int itr = 0; fabs(fun) > 1.e-2 && itr < 50; itr++) {
        const double iT = 1.0 / T, d = dT * iT;
        fun = rest + R.satB * iT + R.satC * log10(T);
        double df;
        if (fabs(d) < kSmallLog) {
            // 1 / (T + dT) - 1 / T = -(1 / T) d (1 - d + d^2 - ...)
            df = R.satC * log10_1p(d) - R.satB * iT * d * (1.0 - d * (1.0 - d * (1.0 - d * (1.0 - d * (1.0 - d)))));
        } else {
            df = R.satB / (T + dT) - R.satB * iT + R.satC * (log10(T + dT) - log10(T));
        }
        T = T - urf * fun * dT / df;
    }
    return T;
}

// Thermal (p, T) equilibrium (DP/thermRlx.cu:4-235).  The unknowns are the density r and energy e of
// the minor phase; the primary phase follows from volume and energy.  The two solved phases are
// named minor / primary and mapped to the phases 0 / 1 by selects, so no array is indexed at run
// time.  Divisions are what an iteration costs, and it takes 4 of them (the reference's order of
// operations 23): with s = part_minor / r the primary density is part / (1 - s), so its reciprocal needs
// none; the stepped density is r (1 + 1e-4), so 1 / r and s scale by a constant; and the Newton step is
// solved for in units of the difference steps, so the Jacobian's columns stay differences.
// Bound by the latency of FP64 instructions (their pipe is 33-53 % busy, see the relaxation's profile).  981 k-tet
// bubble (8.6 iterations per cell): 255 us in the reference's order, 159 with shared denominators (11
// divisions), 113 now; 2.0 M-cell jet 241, 145, 116; 128^3 TGV (one iteration) 141, 112, 111.
__device__ int therm_cell(const RelaxParams &R, double *U, int *iters) {
    const double a0 = fmin(fmax(R.avfMin / 100, U[0]), 1 - R.avfMin / 100);
    const double a1 = 1 - a0;
    const double rho0 = U[1] / a0, rho1 = U[2] / a1;
    const double ar0 = mul_rn(a0, rho0), ar1 = mul_rn(a1, rho1);
    const double e0 = U[6] / ar0, e1 = U[7] / ar1;
    const bool m1 = !(a1 > a0);   // the minor phase is phase 1
    const double arm = m1 ? ar1 : ar0, arp = m1 ? ar0 : ar1;
    double r = m1 ? rho1 : rho0, e = m1 ? e1 : e0;
    double enm, enp;
    {
        const double im = 1.0 / add_rn(ar0, ar1);
        const double u = mul_rn(U[3], im), v = mul_rn(U[4], im), w = mul_rn(U[5], im);
        const double de = fma_rn(-0.5, sq_rn(u, v, w),
                                 fma_rn(-mul_rn(ar1, im), e1, fma_rn(U[8], im, -mul_rn(mul_rn(ar0, im), e0))));
        enm = add_rn(e, de);
        enp = add_rn(m1 ? e0 : e1, de);
    }
    const double iarp = 1.0 / arp;
    double br = r, be = e;   // best iterate
    float minRes = 1e9f;
    int aborted = 0;
    for (int itr = 1;; itr++) {
        *iters = itr;
        // residuals at (r, e); i0, i1: reciprocals of Cv (g - 1) rho
        const double ir = 1.0 / r, sh = mul_rn(arm, ir);
        double rp = arp * (1.0 / (1 - sh)), irp = (1 - sh) * iarp;
        const double ep = fma_rn(-iarp, mul_rn(arm, e - enm), enp);
        const double i0 = R.icvgm1[0] * (m1 ? irp : ir), i1 = R.icvgm1[1] * (m1 ? ir : irp);
        double p0 = p_of(R, 0, m1 ? rp : r, m1 ? ep : e), p1 = p_of(R, 1, m1 ? r : rp, m1 ? e : ep);
        const double res0 = p0 - p1, res1 = diff_rn(p0 + R.pinf[0], i0, p1 + R.pinf[1], i1);
        const bool inside = r > 0.0 && rp > 0.0;
        // forward differences in e (same densities), then in r (same energies)
        const double he = mul_rn(1e-4, e), hr = mul_rn(1e-4, r);
        double d01, d11, d00, d10;
        {
            const double eq = add_rn(e, he), epq = fma_rn(-iarp, mul_rn(arm, eq - enm), enp);
            p0 = p_of(R, 0, m1 ? rp : r, m1 ? epq : eq);
            p1 = p_of(R, 1, m1 ? r : rp, m1 ? eq : epq);
            d01 = (p0 - p1) - res0;
            d11 = diff_rn(p0 + R.pinf[0], i0, p1 + R.pinf[1], i1) - res1;
        }
        {
            constexpr double kStep = 1.0 / (1.0 + 1e-4);
            const double rq = add_rn(r, hr), irq = ir * kStep, sq = mul_rn(sh, kStep);
            rp = arp * (1.0 / (1 - sq));
            irp = (1 - sq) * iarp;
            p0 = p_of(R, 0, m1 ? rp : rq, m1 ? ep : e);
            p1 = p_of(R, 1, m1 ? rq : rp, m1 ? e : ep);
            d00 = (p0 - p1) - res0;
            d10 = diff_rn(p0 + R.pinf[0], R.icvgm1[0] * (m1 ? irp : irq), p1 + R.pinf[1], R.icvgm1[1] * (m1 ? irq : irp)) - res1;
        }
        const double det = diff_rn(d00, d11, d10, d01);
        const bool bad = isnan(d00) || isnan(d01) || isnan(d10) || isnan(d11) || det == 0;
        if (!bad && inside) {
            const float chk = sqrt(fma_rn(res0, res0, mul_rn(res1, res1)));
            if (chk < minRes) {
                minRes = chk;
                br = r;
                be = e;
            }
        }
        if (bad || itr > R.thermItrMax) {
            r = br;
            e = be;
            aborted = 1;
            break;
        }
        const double id = R.thermUrf / det;
        r = fma_rn(-hr, mul_rn(id, diff_rn(d11, res0, d01, res1)), r);
        e = fma_rn(-he, mul_rn(id, diff_rn(d00, res1, d10, res0)), e);
        if (!(fabs(res0) > 1.e-2) && !(fabs(res1) > 1.e-2)) break;
    }
    const double rp = arp / (1 - arm / r);
    const double ep = fma_rn(-iarp, mul_rn(arm, e - enm), enp);
    U[0] = fmin(fmax(R.avfMin / 100, ar0 / (m1 ? rp : r)), 1 - R.avfMin / 100);
    U[6] = ar0 * (m1 ? ep : e);
    U[7] = ar1 * (m1 ? e : ep);
    return aborted;
}

// The same Newton in the reference's order of operations, for FP64 runs.  The Newton stops at the absolute residual
// 1e-2 after one more step under-relaxed by thermUrf, so two orders of operations that put a residual on either
// side of it leave states about (1 - thermUrf) 1e-2 apart in pressure: 2.5e-5 of the vortex's p of about 70, where
// FP64 results are otherwise alike to 1e-15.  With the rearranged Newton (and cons2prim_d) 16 FP64 vortex boxes of
// 1,386 to 340,860 cells were 4e-9 to 1.3e-6 off in the norm after 2 to 4 steps.  FP64 runs are what other
// results are checked against, and keep the one order; the roundings are written out, so that every kernel that
// this is compiled into agrees.  20 divisions per iteration: relaxation of the 96^3 TGV 55 us, 51 rearranged.
__device__ int therm_cell_ordered(const RelaxParams &R, double *U, int *iters) {
    const double a0 = fmin(fmax(R.avfMin / 100, U[0]), 1 - R.avfMin / 100);
    const double a1 = 1 - a0;
    const double rho0 = U[1] / a0, rho1 = U[2] / a1;
    const double ar0 = mul_rn(a0, rho0), ar1 = mul_rn(a1, rho1);
    const double e0 = U[6] / ar0, e1 = U[7] / ar1;
    const bool m1 = !(a1 > a0);   // the minor phase is phase 1
    const double arm = m1 ? ar1 : ar0, arp = m1 ? ar0 : ar1;
    double r = m1 ? rho1 : rho0, e = m1 ? e1 : e0;
    double enm, enp;
    {
        const double rm = add_rn(ar0, ar1);
        const double u = U[3] / rm, v = U[4] / rm, w = U[5] / rm;
        const double de = fma_rn(-0.5, sq_rn(u, v, w),
                                 fma_rn(-(ar1 / rm), e1, fma_rn(-(ar0 / rm), e0, U[8] / rm)));
        enm = add_rn(e, de);
        enp = add_rn(m1 ? e0 : e1, de);
    }
    const double iarp = 1 / arp;
    // the primary phase's density and energy, and the residuals, at the minor phase's (r, e)
    auto close = [&](double rq, double eq, double &rp, double &ep) {
        rp = mul_rn(1 / (1 - arm / rq), arp);
        ep = fma_rn(-iarp, mul_rn(arm, eq - enm), enp);
    };
    auto point = [&](double rq, double eq, double &rp, double &d0, double &d1) {
        double ep;
        close(rq, eq, rp, ep);
        const double x0 = m1 ? rp : rq, x1 = m1 ? rq : rp;
        const double p0 = p_of(R, 0, x0, m1 ? ep : eq), p1 = p_of(R, 1, x1, m1 ? eq : ep);
        d0 = p0 - p1;
        d1 = (p0 + R.pinf[0]) / mul_rn(R.cvgm1[0], x0) - (p1 + R.pinf[1]) / mul_rn(R.cvgm1[1], x1);
    };
    double br = r, be = e;   // best iterate
    float minRes = 1e9f;
    int aborted = 0;
    for (int itr = 1;; itr++) {
        *iters = itr;
        double rp, res0, res1, j00, j10, j01, j11;
        point(r, e, rp, res0, res1);
        const double hr = mul_rn(1e-4, r);
        r = add_rn(r, hr);
        point(r, e, rp, j00, j10);
        r = add_rn(r, -hr);   // not always the value it was
        j00 = (j00 - res0) / hr;
        j10 = (j10 - res1) / hr;
        const double he = mul_rn(1e-4, e);
        e = add_rn(e, he);
        point(r, e, rp, j01, j11);
        e = add_rn(e, -he);
        j01 = (j01 - res0) / he;
        j11 = (j11 - res1) / he;
        const double det = diff_rn(j00, j11, j10, j01);
        const bool bad = isnan(j00) || isnan(j01) || isnan(j10) || isnan(j11) || det == 0;
        if (!bad && r > 0.0 && rp > 0.0) {
            const float chk = sqrt(fma_rn(res0, res0, mul_rn(res1, res1)));
            if (chk < minRes) {
                minRes = chk;
                br = r;
                be = e;
            }
        }
        if (bad || itr > R.thermItrMax) {
            r = br;
            e = be;
            aborted = 1;
            break;
        }
        r = fma_rn(-R.thermUrf, fma_rn(j11 / det, res0, mul_rn(-j01 / det, res1)), r);
        e = fma_rn(-R.thermUrf, fma_rn(-j10 / det, res0, mul_rn(j00 / det, res1)), e);
        if (!(fabs(res0) > 1.e-2) && !(fabs(res1) > 1.e-2)) break;
    }
    double rp, ep;
    close(r, e, rp, ep);
    U[0] = fmin(fmax(R.avfMin / 100, ar0 / (m1 ? rp : r)), 1 - R.avfMin / 100);
    U[6] = ar0 * (m1 ? ep : e);
    U[7] = ar1 * (m1 ? e : ep);
    return aborted;
}

// Residuals of the chemical (p, T, Gibbs) equilibrium of a cell with mixture density rm and internal
// energy re per unit volume (DP/chemRlx.cu:4-130), and their forward-difference Jacobian.  The
// unknowns are volume fraction a, density r and energy e of the minor phase (phase 1 if m1).
// The reference's entropy log10(T^g / (p + pinf)^(g - 1)) is evaluated as g log10 T - (g - 1)
// log10(p + pinf), with no powers; the logarithms are taken once, at the base point, and the three
// perturbed points add log10 of the ratio from the series (log10_1p), or logarithms of their own
// where the ratio is not near 1: 4 logarithms an iteration in place of 12 and 16 powers.  A point reuses
// the reciprocals that its step leaves alone, and the Newton step is solved for in units of the difference
// steps: 10 divisions in place of 26.  Bound by FP64 instructions and, on few cells, by the latency of one
// cell's chain of iterations: the relaxation kernel takes 241 us (784 in the reference's order) on a
// 61 x 67 x 59 box with 36 % chemical cells, 79 (331) on 16,096 mixed elements, and 106 (387) on a 64^3 box
// with the surrogate's polish.
struct ChemLog {
    double lT[2], lP[2], lG;   // log10 of T, p + pinf of the phases, and of the gas pressure
};
struct ChemSystem {
    double res[3], dif[3][3];   // residuals; dif[i][q]: change of residual i by step q
    double ap, rp;   // volume fraction and density of the primary phase at the base point
    // the base point: reciprocals of the primary phase's volume fraction and partial density and of r,
    // pressures, temperatures, reciprocals of T and p + pinf, logarithms
    double iap, ipart, ir;
    double p[2], T[2], iT[2], iP[2];
    ChemLog log;
};
__device__ __forceinline__ double chem_gibbs_diff(const RelaxParams &R, const double *T, const ChemLog &l) {
    const double s0 = mul_rn(R.cv[0], diff_rn(R.gam[0], l.lT[0], R.gm1[0], l.lP[0]));
    const double s1 = fma_rn(R.cv[1], diff_rn(R.gam[1], l.lT[1], R.gm1[1], l.lP[1]), fma_rn(R.satConst[0], l.lG, R.satConst[1]));
    return fma_rn(-T[0], s0, fma_rn(R.cp[0], T[0], R.eta[0])) - fma_rn(-T[1], s1, fma_rn(R.cp[1], T[1], R.eta[1]));
}
// the step h[q] of unknown q in the Jacobian
__device__ __forceinline__ double chem_step(double x) { return fabs(x) < 1e-9 ? 1e-10 : mul_rn(1.e-5, x); }
// points from <= q < to: 0 the base point (residuals), 1 .. 3 a, r, e stepped forward (Jacobian columns).
// kWide: the points are unrolled, so that the chains of the three stepped points overlap (same arithmetic,
// more registers).
template <bool kWide>
__device__ __forceinline__ void chem_system(const RelaxParams &R, bool m1, double a, double r, double e, double rm, double re,
                                            int from, int to, ChemSystem &S) {
#pragma unroll(kWide ? 4 : 1)
    for (int q = from; q < to; q++) {
        const double aq = q == 1 ? add_rn(a, chem_step(a)) : a;
        const double rq = q == 2 ? add_rn(r, chem_step(r)) : r;
        const double eq = q == 3 ? add_rn(e, chem_step(e)) : e;
        // a step in a, r or e leaves the reciprocals that do not contain it as they are
        const double ap = 1 - aq, mq = mul_rn(aq, rq), part = add_rn(rm, -mq);
        const double iap = q < 2 ? 1.0 / ap : S.iap;
        const double ipart = q < 3 ? 1.0 / part : S.ipart;
        const double ir = (q & 1) || q > 2 ? S.ir : 1.0 / rq;
        const double rp = part * iap, irp = ap * ipart, ep = mul_rn(fma_rn(-mq, eq, re), ipart);
        const double x0 = m1 ? rp : rq, x1 = m1 ? rq : rp;
        double p[2], T[2];
        p[0] = p_of(R, 0, x0, m1 ? ep : eq);
        p[1] = p_of(R, 1, x1, m1 ? eq : ep);
        T[0] = (p[0] + R.pinf[0]) * (R.icvgm1[0] * (m1 ? irp : ir));
        T[1] = (p[1] + R.pinf[1]) * (R.icvgm1[1] * (m1 ? ir : irp));
        ChemLog l;
        double d0 = 1, d1 = 1, d2 = 1, d3 = 1;   // the base point takes logarithms of its own
        if (q) {
            d0 = (T[0] - S.T[0]) * S.iT[0];
            d1 = (T[1] - S.T[1]) * S.iT[1];
            d2 = (p[0] - S.p[0]) * S.iP[0];
            d3 = (p[1] - S.p[1]) * S.iP[1];
        }
        if (fabs(d0) < kSmallLog && fabs(d1) < kSmallLog && fabs(d2) < kSmallLog && fabs(d3) < kSmallLog) {
            l.lT[0] = log10_1p(d0, S.log.lT[0]);
            l.lT[1] = log10_1p(d1, S.log.lT[1]);
            l.lP[0] = log10_1p(d2, S.log.lP[0]);
            l.lP[1] = log10_1p(d3, S.log.lP[1]);
        } else {
            l.lT[0] = log10(T[0]);
            l.lT[1] = log10(T[1]);
            l.lP[0] = log10(p[0] + R.pinf[0]);
            l.lP[1] = log10(p[1] + R.pinf[1]);
        }
        l.lG = R.pinf[1] == 0.0 ? l.lP[1] : log10(p[1]);
        const double g = chem_gibbs_diff(R, T, l);
        if (q == 0) {
            S.res[0] = p[0] - p[1];
            S.res[1] = T[0] - T[1];
            S.res[2] = g;
            S.ap = ap;
            S.rp = rp;
            S.log = l;
#pragma unroll
            for (int m = 0; m < 2; m++) {
                S.p[m] = p[m];
                S.T[m] = T[m];
                S.iP[m] = 1.0 / (p[m] + R.pinf[m]);
                S.iT[m] = S.iP[m] * (R.cvgm1[m] * (m ? x1 : x0));
            }
            S.iap = iap;
            S.ipart = ipart;
            S.ir = ir;
        } else {
            const double c0 = (p[0] - p[1]) - S.res[0], c1 = (T[0] - T[1]) - S.res[1], c2 = g - S.res[2];
            if (q == 1) { S.dif[0][0] = c0; S.dif[1][0] = c1; S.dif[2][0] = c2; }
            if (q == 2) { S.dif[0][1] = c0; S.dif[1][1] = c1; S.dif[2][1] = c2; }
            if (q == 3) { S.dif[0][2] = c0; S.dif[1][2] = c1; S.dif[2][2] = c2; }
        }
    }
}

// dx = J^-1 res at (a, r, e), by cofactors and in units of the difference steps; the determinant of
// the differences
__device__ __forceinline__ double chem_direction(const ChemSystem &S, double a, double r, double e, double *dx) {
    const double(*j)[3] = S.dif;
    const double c00 = diff_rn(j[1][1], j[2][2], j[1][2], j[2][1]);
    const double c01 = diff_rn(j[1][2], j[2][0], j[1][0], j[2][2]);
    const double c02 = diff_rn(j[1][0], j[2][1], j[1][1], j[2][0]);
    const double det = fma_rn(j[0][0], c00, fma_rn(j[0][1], c01, mul_rn(j[0][2], c02)));
    const double id = 1.0 / det;
    auto row = [&](double h, double x, double y, double z) {
        return mul_rn(mul_rn(h, id), fma_rn(x, S.res[0], fma_rn(y, S.res[1], mul_rn(z, S.res[2]))));
    };
    dx[0] = row(chem_step(a), c00, diff_rn(j[0][2], j[2][1], j[0][1], j[2][2]), diff_rn(j[0][1], j[1][2], j[0][2], j[1][1]));
    dx[1] = row(chem_step(r), c01, diff_rn(j[0][0], j[2][2], j[0][2], j[2][0]), diff_rn(j[0][2], j[1][0], j[0][0], j[1][2]));
    dx[2] = row(chem_step(e), c02, diff_rn(j[0][1], j[2][0], j[0][0], j[2][1]), diff_rn(j[0][0], j[1][1], j[0][1], j[1][0]));
    return det;
}

// relaxed state from the minor phase's (a, r, e): the primary phase closes mass and energy
__device__ __forceinline__ void chem_store(const RelaxParams &R, bool m1, double a, double r, double e, double rm, double re,
                                           double *U) {
    const double mq = mul_rn(a, r), part = add_rn(rm, -mq);
    const double ap = 1 - a, rp = part / ap, ep = fma_rn(-mq, e, re) / part;
    const double x0 = m1 ? ap : a, r0 = m1 ? rp : r, r1 = m1 ? r : rp, e0 = m1 ? ep : e, e1 = m1 ? e : ep;
    const double x1 = m1 ? a : ap;
    U[0] = fmin(fmax(R.avfMin / 100, x0), 1 - R.avfMin / 100);
    U[1] = x0 * r0;
    U[2] = x1 * r1;
    U[6] = x0 * r0 * e0;
    U[7] = x1 * r1 * e1;
    U[9] = x1 * r1;
}

// A step that left the unknown's range is halved until it is back (DP/chemRlx.cu:132-170): volume
// fractions in [0, 1], partial densities in [0, rm].  1 where it stays outside.
__device__ int chem_limit_fraction(const RelaxParams &R, double old, double &x, double dx) {
    float urf = (float)R.chemUrf;
    if (x < 0) { while (x < R.chemLimit && urf > 0.0005f) { urf = urf / 2; x = fma_rn(-(double)urf, dx, old); } }
    if (x > 1) { while (x > 1.0 - R.chemLimit && urf > 0.0005f) { urf = urf / 2; x = fma_rn(-(double)urf, dx, old); } }
    return x < 0 || x > 1;
}
__device__ int chem_limit_density(const RelaxParams &R, double a, double old, double &x, double dx, double rm) {
    float urf = (float)R.chemUrf;
    double ar = a * x;
    if (x < 0) { while (x < 0 && urf > 0.0005f) { urf = urf / 2; x = fma_rn(-(double)urf, dx, old); } }
    if (ar > rm) { while (ar > rm && urf > 0.0005f) { urf = urf / 2; x = fma_rn(-(double)urf, dx, old); ar = a * x; } }
    return x < 0 || ar > rm;
}

// mixture density and internal energy per unit volume of a cell, and the phases it starts from: volume fractions,
// densities and partial densities
struct ChemMix {
    double a0, a1, r0, r1, ar0, ar1, rm, re;
};
__device__ __forceinline__ ChemMix chem_mixture(const RelaxParams &R, const double *U) {
    ChemMix m;
    m.a0 = fmin(fmax(R.avfMin / 100, U[0]), 1 - R.avfMin / 100);
    m.a1 = 1 - m.a0;
    m.r0 = U[1] / m.a0;
    m.r1 = U[2] / m.a1;
    m.ar0 = mul_rn(m.a0, m.r0);
    m.ar1 = mul_rn(m.a1, m.r1);
    m.rm = add_rn(m.ar0, m.ar1);
    const double u = U[3] / m.rm, v = U[4] / m.rm, w = U[5] / m.rm;
    m.re = fma_rn(-mul_rn(0.5, m.rm), sq_rn(u, v, w), U[8]);
    return m;
}

// Chemical equilibrium (DP/chemRlx.cu:4-267): damped Newton from the cell's state
template <bool kWide>
__device__ int chem_cell(const RelaxParams &R, double *U, int *iters) {
    double a, r, e, rm, re;
    bool m1;
    {
        const ChemMix m = chem_mixture(R, U);
        rm = m.rm;
        re = m.re;
        m1 = !(m.a1 > m.a0);
        a = m1 ? m.a1 : m.a0;
        r = m1 ? m.r1 : m.r0;
        e = m1 ? U[7] / m.ar1 : U[6] / m.ar0;
    }
    double ba = a, br = r, be = e;   // best iterate
    float minRes = 1e9f;
    int aborted = 0;
    for (int itr = 1;; itr++) {
        *iters = itr;
        ChemSystem S;
        chem_system<kWide>(R, m1, a, r, e, rm, re, 0, 4, S);
        double dx[3];
        const double det = chem_direction(S, a, r, e, dx);
        int ab = det == 0;
#pragma unroll
        for (int i = 0; i < 3; i++)
#pragma unroll
            for (int j = 0; j < 3; j++) ab |= isnan(S.dif[i][j]);
        if (!ab && a > 0.0 && a < 1.0 && S.ap > 0.0 && S.ap < 1.0 && r > 0.0 && S.rp > 0.0) {
            const float chk = sqrt(fma_rn(S.res[0], S.res[0], fma_rn(S.res[1], S.res[1], mul_rn(S.res[2], S.res[2]))));
            if (chk < minRes) {
                minRes = chk;
                ba = a;
                br = r;
                be = e;
            }
        }
        const double oa = a, orr = r;
        a = fma_rn(-R.chemUrf, dx[0], a);
        ab |= chem_limit_fraction(R, oa, a, dx[0]);
        r = fma_rn(-R.chemUrf, dx[1], r);
        ab |= chem_limit_density(R, a, orr, r, dx[1], rm);
        e = fma_rn(-R.chemUrf, dx[2], e);
        if (ab || itr > R.chemItrMax) {
            a = ba;
            r = br;
            e = be;
            aborted = 1;
            break;
        }
        if (!(fabs(S.res[0]) > 1.e-1) && !(fabs(S.res[1]) > 1.e-1) && !(fabs(S.res[2]) > 1.e-1)) break;
    }
    chem_store(R, m1, a, r, e, rm, re, U);
    return aborted;
}

// Full-step Newton from the surrogate's equilibrium (p, T, alpha) on the residuals of chem_system.
// Returns 1 and writes U when every relative residual is within relTol.
__device__ int chem_polish(const RelaxParams &R, double *U, const float *y, double rm, double re, double relTol, int maxIt,
                           int *iters) {
    const double p = y[0], T = y[1];
    if (!(T > 0) || !(p > -R.pinf[0]) || !(p > -R.pinf[1])) return 0;
    const double rL = (p + R.pinf[0]) / (R.cvgm1[0] * T);
    const double rG = (p + R.pinf[1]) / (R.cvgm1[1] * T);
    double al = (rm - rG) / (rL - rG);   // mass balance at (p, T)
    if (!(al > 0 && al < 1)) al = y[2];
    if (!(al > 0 && al < 1)) return 0;
    const bool m1 = !(1 - al > al);
    double a = m1 ? 1 - al : al, r = m1 ? rG : rL;
    double e = m1 ? (p + R.gpinf[1]) / (R.gm1[1] * rG) + R.eta[1] : (p + R.gpinf[0]) / (R.gm1[0] * rL) + R.eta[0];
    const double sp = fmax(fabs(p), 1.0), sT = T, sg = R.cp[0] * T;
    int ok = 0;
    for (int itr = 0; itr <= maxIt; itr++) {
        ChemSystem S;
        chem_system<false>(R, m1, a, r, e, rm, re, 0, 1, S);
        if (!(a > 0 && a < 1 && r > 0 && S.rp > 0)) break;
        if (fabs(S.res[0]) <= relTol * sp && fabs(S.res[1]) <= relTol * sT && fabs(S.res[2]) <= relTol * sg) {
            ok = 1;
            break;
        }
        if (itr == maxIt) break;
        *iters = itr + 1;
        chem_system<false>(R, m1, a, r, e, rm, re, 1, 4, S);
        double dx[3];
        const double det = chem_direction(S, a, r, e, dx);
        if (!(fabs(det) > 0) || !isfinite(det)) break;
        a -= dx[0];
        r -= dx[1];
        e -= dx[2];
    }
    if (!ok) return 0;
    chem_store(R, m1, a, r, e, rm, re, U);
    return 1;
}

// partitionRelaxation (DP/relaxation.cu:4-75): the cell needs the chemical (Gibbs) solve when its
// liquid temperature is above the saturation temperature at its liquid pressure and its
// volume fraction above chemLimit
__device__ __forceinline__ int needs_chem(const RelaxParams &R, const double *u) {
    const double avf = fmin(fmax(R.avfMin / 100, u[0]), 1 - R.avfMin / 100);
    if (!(avf > R.chemLimit)) return 0;   // whatever its saturation temperature
    const double rho = u[1] / avf;
    const double enr = u[6] / (avf * rho);
    const double tl = t_of(R, 0, rho, enr);
    const double pl = p_of(R, 0, rho, enr);
    return tl > sat_temp(R, pl, tl, R.satTempUrf);
}

}  // namespace

// ---- ordering of the cells for the relaxation: chemical cells first, then thermal cells, each
// in cell order (a deterministic block prefix sum; no atomics), so that every warp of the
// relaxation kernel but one runs a single branch
constexpr int kOrdThreads = 256;

__global__ void k_relax_partition(int n, const double *U, const RelaxParams R, uint8_t *isChem,
                                  int32_t *blockChem) {
    pdl_trigger();
    pdl_wait();
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    int chem = 0;
    if (c < n) {
        double u[NV];
        u[0] = U[c];
        u[1] = U[(size_t)n + c];
        u[6] = U[(size_t)6 * n + c];
        chem = needs_chem(R, u);
        isChem[c] = (uint8_t)chem;
    }
    const int cnt = __syncthreads_count(chem);
    if (threadIdx.x == 0) blockChem[blockIdx.x] = cnt;
}

// exclusive scan of the per-block counts (one block of 1024 threads), total into *total
__global__ void k_relax_scan(const int32_t *cnt, int nb, int32_t *off, int32_t *total) {
    pdl_trigger();
    pdl_wait();
    __shared__ int32_t sh[1024];
    const int t = threadIdx.x;
    const int per = (nb + 1023) / 1024;
    const int lo = min(nb, t * per), hi = min(nb, lo + per);
    int s = 0;
    for (int i = lo; i < hi; i++) s += cnt[i];
    sh[t] = s;
    __syncthreads();
    for (int d = 1; d < 1024; d <<= 1) {
        const int v = (t >= d) ? sh[t - d] : 0;
        __syncthreads();
        sh[t] += v;
        __syncthreads();
    }
    int base = t ? sh[t - 1] : 0;
    for (int i = lo; i < hi; i++) {
        off[i] = base;
        base += cnt[i];
    }
    if (t == 1023) *total = sh[1023];
}

__global__ void k_relax_order(int n, const uint8_t *isChem, const int32_t *blockOff, const int32_t *total,
                              int32_t *order) {
    pdl_trigger();
    pdl_wait();
    __shared__ int32_t warpChem[kOrdThreads / 32];
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int chem = (c < n) ? isChem[c] : 0;
    const unsigned bal = __ballot_sync(0xffffffffu, chem);
    if (lane == 0) warpChem[wid] = __popc(bal);
    __syncthreads();
    int before = 0;   // chemical cells of this block before this warp
    for (int w = 0; w < wid; w++) before += warpChem[w];
    if (c >= n) return;
    const int rankC = before + __popc(bal & ((1u << lane) - 1u));    // chemical cells before c in the block
    const int rankT = (int)threadIdx.x - rankC;                       // thermal cells before c in the block
    const int b = blockIdx.x;
    if (chem) order[blockOff[b] + rankC] = c;
    else order[*total + (b * kOrdThreads - blockOff[b]) + rankT] = c;
}

// surrogate input of the relaxation: chemical cell order[i], i < *nChem
struct InRelax {
    const double *U;
    int n;
    const int32_t *order;
    const int32_t *nChem;
    RelaxParams R;
    __device__ int count() const { return *nChem; }
    __device__ void features(int i, const SurrogateNorm &N, float (&z)[3]) const {
        const int c = order[i];
        double u[NV];
#pragma unroll
        for (int v = 0; v < NV; v++) u[v] = U[(size_t)v * n + c];
        const ChemMix m = chem_mixture(R, u);
        const float f[3] = {(float)m.rm, (float)(m.re / m.rm), (float)(m.ar1 / m.rm)};
#pragma unroll
        for (int k = 0; k < 3; k++) z[k] = (f[k] - N.xMean[k]) / N.xStd[k];
    }
};

// resident blocks asked of the compiler for the thermal-only instantiation (kOrd false): 6 blocks of 128
// threads (80 registers) 114.5 us per relaxation of the 128^3 TGV, 7 blocks 115.7, 8 blocks 117.3
#ifndef FG_THERM_MINBLOCKS
#define FG_THERM_MINBLOCKS 6
#endif
// the same for the chemical-first instantiations (kOrd true: Gibbs and thermal Newton).  Without the
// surrogate, on the box with 36 % chemical cells / the 981 k-tet bubble (almost all thermal): 4 blocks 257 /
// 188 us, 5 blocks 228 / 170, 6 blocks 235 / 160, 8 blocks 254 / 156.  With the surrogate's polish, on the
// 64^3 box: 4 blocks (128 registers) 119 us, 5 blocks 130, 6 blocks 133; the same budget serves
// k_relax_polish, the surrogate's polish as a pass of its own.
#ifndef FG_CHEM_MINBLOCKS
#define FG_CHEM_MINBLOCKS 6
#endif
#ifndef FG_CHEM_SG_MINBLOCKS
#define FG_CHEM_SG_MINBLOCKS 4
#endif

// Chemical-first relaxation of few cells: where every cell has its thread resident at 3 blocks per SM the
// kernel is bound by the longest chain of Gibbs iterations, and takes the unrolled system with
// 157 registers (bitwise the same states).  16,096 mixed elements: 133 -> 100 us; above the limit, where
// 3 blocks cost occupancy, the 73,908-tet bubble went 28 -> 34 us with it.
constexpr int kWideBlocks = 3, kWideCells = 148 * kWideBlocks * 128;

// hullOk[i] of a chemical cell whose polished surrogate solution k_relax_polish accepted
constexpr int32_t kPolished = 2;

// Surrogate pass over the chemical cells (order[0 .. *nChem)), before k_relax: each cell whose
// network input lies inside the training hull (hullOk[i] = 1, k_sg_tc) is polished from the
// network's prediction pred[i]; an accepted cell gets its relaxed state (U and its W record) and
// hullOk[i] = kPolished, and k_relax leaves it alone.  Running the polish in its own kernel keeps
// its register budget off the thermal Newton's.  Grid-stride over the resident blocks.  Counts
// the polish steps (accepted or not) as Newton iterations, the accepted cells and their polish
// steps.  Its results are bitwise those of the polish inside k_relax (same arithmetic per cell).
template <typename T>
__global__ void __launch_bounds__(128, FG_CHEM_SG_MINBLOCKS) k_relax_polish(int n, double *U, T *W, size_t wStride,
                                               const PhysD D, const RelaxParams R, int32_t *counters,
                                               const SurrogateDev S, const int32_t *order, const int32_t *nChem,
                                               const float4 *pred, int32_t *hullOk) {
    pdl_trigger();
    pdl_wait();
    const int m = *nChem;
    // base is the same for every thread of the block: the warp collectives below see full warps
    for (int base = blockIdx.x * blockDim.x; base < m; base += gridDim.x * blockDim.x) {
        const int i = base + threadIdx.x;
        int used = 0, pits = 0;
        if (i < m && hullOk[i]) {
            const int c = order[i];
            double u[NV];
#pragma unroll
            for (int v = 0; v < NV; v++) u[v] = U[(size_t)v * n + c];
            const ChemMix mix = chem_mixture(R, u);
            const float4 p4 = pred[i];
            const float pr[4] = {p4.x, p4.y, p4.z, p4.w};
            used = chem_polish(R, u, pr, mix.rm, mix.re, S.relTol, S.polishIters, &pits);
            if (used) {
                U[(size_t)0 * n + c] = u[0];
                U[(size_t)1 * n + c] = u[1];
                U[(size_t)2 * n + c] = u[2];
                U[(size_t)6 * n + c] = u[6];
                U[(size_t)7 * n + c] = u[7];
                U[(size_t)9 * n + c] = u[9];
                T w[NP];
                cons2prim_d(D, u, w);
                w_store<T>(W, wStride, c, w);
                hullOk[i] = kPolished;
            }
        }
        const unsigned maskS = __ballot_sync(0xffffffffu, used);
        const int itsW = __reduce_add_sync(0xffffffffu, pits);
        const int polW = __reduce_add_sync(0xffffffffu, used ? pits : 0);
        if ((threadIdx.x & 31) == 0) {
            if (itsW) atomicAdd(&counters[3], itsW);
            if (maskS) atomicAdd(&counters[4], __popc(maskS));
            if (polW) atomicAdd(&counters[6], polW);
        }
    }
}

// kSG / kLog: instantiated with the surrogate path / the solve log; the plain instantiation
// carries none of their code (and none of their registers).  kPass (with kSG): the surrogate's
// polish ran before, in k_relax_polish, and the cells it accepted are skipped; otherwise the
// polish runs here.  kOrd: thread i relaxes cell order[i], chemical when i < *nChem
// (k_relax_order); otherwise thread i relaxes cell i, thermally.
template <typename T, bool kSG, bool kLog, bool kOrd, bool kPass = false, bool kWide = false>
__global__ void __launch_bounds__(128, kWide ? kWideBlocks : kOrd ? ((kSG && !kPass) ? FG_CHEM_SG_MINBLOCKS : FG_CHEM_MINBLOCKS)
                                            : FG_THERM_MINBLOCKS) k_relax(int n, double *U, T *W, size_t wStride, const PhysD D, const RelaxParams R,
                                               int32_t *counters, const SurrogateDev S, const RelaxLog Lg,
                                               const int32_t *order, const int32_t *nChem, const float4 *pred,
                                               const int32_t *hullOk) {
    constexpr bool kPolish = kSG && !kPass;   // the polish runs in this kernel
    pdl_trigger();
    pdl_wait();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const bool act = i < n;
    const int c = (kOrd && act) ? order[i] : i;
    int chem = 0, ab = 0, its = 0, used = 0, pits = 0;
    double u[NV];
    double rm = 0, re = 0, ag = 0;
    if (act) {
        // kOrd: cells ordered chemical-first (chemFlag == 1); otherwise every cell is thermal
        // (chemFlag != 1), and the chemical solver is compiled out of this instantiation
        if (kOrd) chem = i < *nChem;
        // relaxed already by the surrogate pass
        if (kSG && kPass && chem) used = hullOk[i] == kPolished;
    }
    if (act && !used) {
#pragma unroll
        for (int v = 0; v < NV; v++) u[v] = U[(size_t)v * n + c];
        if (chem && (kPolish || kLog)) {
            const ChemMix mix = chem_mixture(R, u);
            rm = mix.rm;
            re = mix.re;
            ag = mix.ar1;
        }
        // the network's prediction for this cell (k_sg_tc over the chemical cells) if its input
        // is inside the training hull
        if (kPolish && chem && hullOk[i] != 0) {
            const float4 p4 = pred[i];
            const float pr[4] = {p4.x, p4.y, p4.z, p4.w};
            used = chem_polish(R, u, pr, rm, re, S.relTol, S.polishIters, &pits);
        }
        if (!used) {
            if (kOrd && chem) ab = chem_cell<kWide>(R, u, &its);
            else ab = sizeof(T) == 8 ? therm_cell_ordered(R, u, &its) : therm_cell(R, u, &its);
        }
        if (kLog && chem && !used && !ab) {
            // training sample: (rho, e, Y) before the solve -> (p, T, alpha, Y_eq) after it
            const unsigned long long k = atomicAdd(Lg.count, 1ULL);
            if (k < (unsigned long long)Lg.cap) {
                const double a0 = fmin(fmax(R.avfMin / 100, u[0]), 1 - R.avfMin / 100);
                const double rL = u[1] / a0, eL = u[6] / u[1];
                float *x = Lg.X + k * 3, *y = Lg.Y + k * 4;
                x[0] = (float)rm;
                x[1] = (float)(re / rm);
                x[2] = (float)(ag / rm);
                y[0] = (float)p_of(R, 0, rL, eL);
                y[1] = (float)t_of(R, 0, rL, eL);
                y[2] = (float)a0;
                y[3] = (float)(u[9] / rm);
            }
        }
        its += pits;   // polish steps count as Newton iterations (accepted or not)
        U[(size_t)0 * n + c] = u[0];
        U[(size_t)1 * n + c] = u[1];
        U[(size_t)2 * n + c] = u[2];
        U[(size_t)6 * n + c] = u[6];
        U[(size_t)7 * n + c] = u[7];
        U[(size_t)9 * n + c] = u[9];
        T w[NP];
        cons2prim_d(D, u, w);
        w_store<T>(W, wStride, c, w);
    }
    // warp-aggregated counters (sums of integers: order does not matter)
    const unsigned mask = __ballot_sync(0xffffffffu, act && chem);
    const unsigned maskT = __ballot_sync(0xffffffffu, act && !chem);
    const unsigned maskA = __ballot_sync(0xffffffffu, act && ab);
    // accepted cells and their polish steps: counted here when the polish ran here
    const unsigned maskS = kPolish ? __ballot_sync(0xffffffffu, act && used) : 0u;
    const unsigned maskF = __ballot_sync(0xffffffffu, act && chem && kSG && !used);
    const int itsW = __reduce_add_sync(0xffffffffu, its);
    const int polW = kPolish ? __reduce_add_sync(0xffffffffu, used ? pits : 0) : 0;
    if ((threadIdx.x & 31) == 0) {
        if (maskT) atomicAdd(&counters[0], __popc(maskT));
        if (mask) atomicAdd(&counters[1], __popc(mask));
        if (maskA) atomicAdd(&counters[2], __popc(maskA));
        if (itsW) atomicAdd(&counters[3], itsW);
        if (maskS) atomicAdd(&counters[4], __popc(maskS));
        if (maskF) atomicAdd(&counters[5], __popc(maskF));
        if (polW) atomicAdd(&counters[6], polW);
    }
}

int relax_order_blocks(int n) { return (n + kOrdThreads - 1) / kOrdThreads; }

template <typename T, bool kOrd>
static void launch_relax_k(int n, double *U, T *W, size_t wStride, const PhysD &D, const RelaxParams &R, int32_t *counters,
                           const SurrogateDev &S, const RelaxLog &L, const RelaxOrder *O, cudaStream_t s) {
    const int nb = (n + 127) / 128;
    const bool lg = L.count != nullptr;
    const int32_t *order = O ? O->order : nullptr, *nChem = O ? O->total : nullptr;
    const float4 *pred = O ? O->pred : nullptr;
    const int32_t *hull = O ? O->hullOk : nullptr;
    if constexpr (kOrd) {
        // the surrogate runs only with the chemical-first order; the logged instantiation keeps
        // the polish inside (launch_relax runs no separate pass with the log on)
        if (S.enabled) {
            if (lg)
                launch_pdl(k_relax<T, true, true, kOrd>, nb, 128, 0, s, n, U, W, wStride, D, R, counters, S, L, order, nChem, pred, hull);
            else if (O->polishPass)
                launch_pdl(k_relax<T, true, false, kOrd, true>, nb, 128, 0, s, n, U, W, wStride, D, R, counters, S, L, order, nChem, pred, hull);
            else
                launch_pdl(k_relax<T, true, false, kOrd>, nb, 128, 0, s, n, U, W, wStride, D, R, counters, S, L, order, nChem, pred, hull);
            return;
        }
    }
    if constexpr (kOrd) {
        if (!lg && n <= kWideCells) {
            launch_pdl(k_relax<T, false, false, kOrd, false, true>, nb, 128, 0, s, n, U, W, wStride, D, R, counters, S, L, order,
                       nChem, pred, hull);
            return;
        }
    }
    if (lg)
        launch_pdl(k_relax<T, false, true, kOrd>, nb, 128, 0, s, n, U, W, wStride, D, R, counters, S, L, order, nChem, pred, hull);
    else
        launch_pdl(k_relax<T, false, false, kOrd>, nb, 128, 0, s, n, U, W, wStride, D, R, counters, S, L, order, nChem, pred, hull);
}

template <typename T>
int launch_relax(int n, double *U, T *W, size_t wStride, const PhysD &D, const RelaxParams &R, int32_t *counters,
                 const SurrogateDev &S, const RelaxLog &L, const RelaxOrder &O, cudaStream_t s) {
    if (R.chemFlag != 1) {
        // every cell is thermal: no ordering needed (and no surrogate)
        launch_relax_k<T, false>(n, U, W, wStride, D, R, counters, SurrogateDev{}, L, nullptr, s);
        return 1;
    }
    const int nb = relax_order_blocks(n);
    launch_pdl(k_relax_partition, nb, kOrdThreads, 0, s, n, U, R, O.isChem, O.blockCnt);
    launch_pdl(k_relax_scan, 1, 1024, 0, s, O.blockCnt, nb, O.blockOff, O.total);
    launch_pdl(k_relax_order, nb, kOrdThreads, 0, s, n, O.isChem, O.blockOff, O.total, O.order);
    int k = 4;
    if (S.enabled) {
        // the network on the tensor cores for the chemical cells (order[0 .. nChem)), tiles of 128
        const int tiles = (n + TC_M - 1) / TC_M;
        k_sg_tc<InRelax><<<std::min(tiles, 148 * 4), 128, TC_SMEM, s>>>(S, S.pack, InRelax{U, n, O.order, O.total, R},
                                                                        O.pred, O.hullOk, O.tcErr);
        k++;
        if (O.polishPass && L.count == nullptr) {
            launch_pdl(k_relax_polish<T>, std::min((n + 127) / 128, 148 * FG_CHEM_SG_MINBLOCKS), 128, 0, s,
                n, U, W, wStride, D, R, counters, S, O.order, O.total, O.pred, O.hullOk);
            k++;
        }
    }
    launch_relax_k<T, true>(n, U, W, wStride, D, R, counters, S, L, &O, s);
    return k;
}

template int launch_relax<float>(int, double *, float *, size_t, const PhysD &, const RelaxParams &, int32_t *,
                                 const SurrogateDev &, const RelaxLog &, const RelaxOrder &, cudaStream_t);
template int launch_relax<double>(int, double *, double *, size_t, const PhysD &, const RelaxParams &, int32_t *,
                                  const SurrogateDev &, const RelaxLog &, const RelaxOrder &, cudaStream_t);

}  // namespace fg
