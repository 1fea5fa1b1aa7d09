// uwshcu_fp64_kernel.cuh -- FP64 sm_100a kernel of compute_uwshcu (uwshcu.F90:478-4664), one thread per column.
//
// Included by the uwshcu_fp64_k*.cu translation units, each instantiating the kernel for one
// (level bound, tracer bound) pair so the instantiations compile in parallel; every unit carries its
// own copy of the constant bank.
//
// Each thread owns one column.  The inputs are read directly in the Fortran (mix, k) layout, so a warp
// of 32 consecutive columns issues 32 consecutive 8-byte loads for every level (level-major SoA).
// Read-only inputs stay in global memory (read through the non-coherent path); the profiles the scheme
// updates live in thread-private arrays sized by the template bound KP >= mkx + 1.  The saturation
// table (wv_saturation.F90 estbl) is staged once per block in shared memory, where the data-dependent
// lookups of neighbouring threads do not serialise the way __constant__ reads would.
//
// Numerics: every expression keeps the Fortran evaluation order, the file is built with -fmad=false
// (no FMA contraction) and IEEE division/sqrt, and pow/exp/log/erfc are the routines of uw_math.h,
// which give the same bits on the host and the device; the CPU restatement built with the same
// routines therefore computes the same bits as this kernel.  exnf(p) = (p/p00)**rovcp
// is evaluated once per distinct pressure and passed into conden: conden at p = ps0(k), p0(k), pe,
// prel, plcl or the cloud top recomputes exactly these values in the Fortran, so the result is the
// same bit for bit and the per-call pow disappears from the Newton loop.
//
// Structure relative to the Fortran: the iteration-1 results that the Fortran keeps in *_s arrays
// (uwshcu.F90:4177-4277) are still in this column's profiles when iteration 2 falls back to explicit
// CIN (uwshcu.F90:1891-2011), and only then go to the output slots; the *_o copies of the inputs
// (:1306-1327) are re-read from the input arrays, and the derived profiles are recomputed from them
// with the same operations.  No loop has a data-dependent trip count beyond the fixed Fortran bounds
// (conden 10, qsinvert 10, compute_alpha 10, compute_mumin2 10, compute_ppen 5, findsp 8), and every
// level index the scheme derives (kinv, klcl, klfc, krel, kbup, kpen) comes from a loop over 0..mkx,
// so all array accesses stay inside the column.
#pragma once
#include <cuda_runtime.h>
#include <math.h>
#include "uwshcu_common.cuh"
#include "uw_math.h"
#include "uw_state.cuh"

namespace {

__constant__ UwConst c;
__constant__ double c_estbl[UW_TBL];

// UW_TAPE_ORDER: the adjoint kernel's operations in the order, and with the repetitions, of the Fortran's
// updraft.  A shorter tape would group the additions of its reverse sweep differently, and where a column
// is ill-conditioned the gradient's last bits are large; its values are the same either way.
#ifndef UW_TAPE_ORDER
#define UW_TAPE_ORDER 0
#endif

#define MX(a, b) ((a) > (b) ? (a) : (b))
#define MN(a, b) ((a) < (b) ? (a) : (b))

// estblf (wv_saturation.F90:64-80).  e is clamped to [tmin, tmax] first (a NaN argument ends at
// tmax), so i stays in 1..203 and i+1 inside the 204 filled entries.
__device__ __forceinline__ double estblf(double td, const double* __restrict__ tbl)
{
    double e = MX(MN(td, c.tmax), c.tmin);
    int i = (int)(e - c.tmin) + 1;
    double ai = trunc(e - c.tmin);
    return (c.tmin + ai - e + 1.0) * tbl[i - 1] - (c.tmin + ai - e) * tbl[i];
}

// vqsatd with len = 1 (wv_saturation.F90:482-609) returning es, qs and gam.
__device__ __forceinline__ void qsat3(double t, double p, double& es, double& qs, double& gam,
                                      const double* __restrict__ tbl)
{
    es = estblf(t, tbl);
    qs = c.epsqs * es / (p - c.omeps * es);
    qs = MN(1.0, qs);
    if (qs < 0.0) {
        qs = 1.0;
        es = p;
    }
    double hltalt, desdt;
    if (c.icephs && c.ttrice != 0.0) {
        double tc = t - c.tmelt;
        bool lflg = (tc >= -c.ttrice && tc < 0.0);
        double weight = MN(-tc * c.trinv, 1.0);
        double hlatsb = c.hlatv + weight * c.hlatf;
        double hlatvp = c.hlatv - 2369.0 * tc;
        hltalt = (t < c.tmelt) ? hlatsb : hlatvp;
        double tterm = lflg ? c.pcf[0] + tc * (c.pcf[1] + tc * (c.pcf[2] + tc * (c.pcf[3] + tc * c.pcf[4]))) : 0.0;
        desdt = hltalt * es / (c.rgasv * t * t) + tterm * c.trinv;
    } else {
        double hlatvp = c.hlatv - 2369.0 * (t - c.tmelt);
        double hlatsb = c.icephs ? c.hlatv + c.hlatf : c.hlatv;
        hltalt = (t < c.tmelt) ? hlatsb : hlatvp;
        desdt = hltalt * es / (c.rgasv * t * t);
    }
    gam = hltalt * qs * p * desdt / (c.cpws * es * (p - c.omeps * es));
    if (qs == 1.0) gam = 0.0;
}

// The qs of vqsatd only (what conden and the buoyancy sorting consume).
__device__ __forceinline__ double qsat_qs(double t, double p, const double* __restrict__ tbl)
{
    double es = estblf(t, tbl);
    double qs = c.epsqs * es / (p - c.omeps * es);
    qs = MN(1.0, qs);
    if (qs < 0.0) qs = 1.0;
    return qs;
}

__device__ __forceinline__ double exnf(double p) { return uw_pow(p / c.p00, c.rovcp); }

// conden (uwshcu.F90:4718-4785) with ex = exnf(p) supplied by the caller.  rv0: the saturation humidity
// at (thl ex, p), its first lookup.
__device__ __forceinline__ int conden(double p, double ex, double thl, double qt, double& th, double& qv,
                                      double& ql, double& qi, double& rv0, const double* __restrict__ tbl)
{
    double tc = thl * ex;
    double nu = MX(MN((268.0 - tc) / 20.0, 1.0), 0.0);
    double leff = (1.0 - nu) * c.xlv + nu * c.xls;
    double temps = tc;
    double rvls = qsat_qs(temps, p, tbl);
    rv0 = rvls;
    int id_check = 0;
    if (rvls >= qt) {
        qv = qt;
        ql = 0.0;
        qi = 0.0;
        th = tc / ex;
    } else {
        double qs = rvls;
        // the Fortran's divisions by leff, r and (twice per step) temps go through their
        // correctly rounded reciprocals: the same quotients, bit for bit (uw_div_by)
        const double rleff = 1.0 / leff;
        const double cpl = uw_div_by(c.cp, leff, rleff);
#pragma unroll 1
        for (int it = 0; it < 10; it++) {
            const double rt = 1.0 / temps;
            temps = temps + (uw_div_by((tc - temps) * c.cp, leff, rleff) + qt - rvls) /
                                (cpl + uw_div_by(uw_div_by(uw_div_by(c.ep2 * leff * rvls, c.r, c.rinv), temps, rt), temps, rt));
            qs = qsat_qs(temps, p, tbl);
            rvls = qs;
        }
        double qc = MX(qt - qs, 0.0);
        qv = qt - qc;
        ql = qc * (1.0 - nu);
        qi = nu * qc;
        th = temps / ex;
        id_check = (fabs((temps - (leff / c.cp) * qc) - tc) >= 1.0) ? 1 : 0;
    }
    return id_check;
}

// conden for the fast-FP64 precision mode: the same saturation adjustment with one reciprocal of the
// temperature per Newton step (2 divisions instead of 5), each lane stopping after its first step
// smaller than 1e-10 T.  The Fortran always takes 10 steps; the steps shrink about 100x per
// iteration and fall below 1e-10 T after 5-7, so the result differs from conden by about 1e-12
// relative.  A lane's result depends only on its own column; the warp leaves the loop when every
// lane is done (__all_sync over the lanes active at the call), so the lanes stay together.
__device__ __forceinline__ int conden_fast(double p, double ex, double thl, double qt, double& th, double& qv,
                                           double& ql, double& qi, double& rv0, const double* __restrict__ tbl)
{
    double tc = thl * ex;
    double nu = MX(MN((268.0 - tc) / 20.0, 1.0), 0.0);
    double leff = (1.0 - nu) * c.xlv + nu * c.xls;
    double temps = tc;
    double rvls = qsat_qs(temps, p, tbl);
    rv0 = rvls;
    int id_check = 0;
    if (rvls >= qt) {
        qv = qt;
        ql = 0.0;
        qi = 0.0;
        th = tc / ex;
    } else {
        const double cpl = c.cp / leff;
        const double a2 = c.ep2 * leff / c.r;
        double qs = rvls;
        bool done = false;
#pragma unroll 1
        for (int it = 0; it < 10; it++) {
            if (!done) {
                const double rt = 1.0 / temps;
                const double dT = ((tc - temps) * cpl + qt - rvls) / (cpl + a2 * rvls * rt * rt);
                temps = temps + dT;
                qs = qsat_qs(temps, p, tbl);
                rvls = qs;
                done = fabs(dT) < 1.e-10 * temps;
            }
            if (__all_sync(__activemask(), done)) break;
        }
        double qc = MX(qt - qs, 0.0);
        qv = qt - qc;
        ql = qc * (1.0 - nu);
        qi = nu * qc;
        th = temps / ex;
        id_check = (fabs((temps - (leff / c.cp) * qc) - tc) >= 1.0) ? 1 : 0;
    }
    return id_check;
}

// ---- conden in FP64 (not in the generated kernels) ----
// The same operations as conden above, result for result, where every divisor is a positive number
// between 2^-100 and 2^100; a test per divisor finds the others, and the call is then repeated with conden.
// The kernels spend most of their time in these Newton steps, a chain of dependent FP64 operations with
// three divisions.  Here a division has no slow path to branch around, and the table position needs no
// conversion: a 16-column call takes 6.0 ms, with conden in its place 6.8, 4,096 columns 8.7 and 9.7, 65,536
// columns 11.4 and 12.4, 1,048,576 columns (which wait for memory and instructions) 103.7 and 108.5.

// qsat_qs; ok is cleared where the divisor is out of range.
__device__ __forceinline__ double qsat_qs_f64(double t, double p, bool& ok, const double* __restrict__ tbl)
{
    double e = t;
    if ((unsigned)(__double2hiint(t) - c.tlo) >= (unsigned)c.tnum) e = MX(MN(t, c.tmax), c.tmin);
    // n, ai = trunc(x), 0 <= x < 2^31: the nearest integer in the low word of x + 1.5 2^52, less one if above x
    const double x = e - c.tmin, m = x + 0x1.8p52;
    double ai = m - 0x1.8p52;
    int n = __double2loint(m);
    if (ai > x) {
        ai = ai - 1.0;
        n = n - 1;
    }
    const double w = c.tmin + ai - e;
    const double es = (w + 1.0) * tbl[n] - w * tbl[n + 1];
    const double d = p - c.omeps * es;
    ok = ok && uw_rcp_ok(d);
    double qs = uw_div_by(c.epsqs * es, d, uw_rcp(d));
    if ((unsigned)__double2hiint(qs) >= 0x3ff00000u) {   // not in [0, 1)
        qs = MN(1.0, qs);
        if (qs < 0.0) qs = 1.0;
    }
    return qs;
}

struct CondenOut {
    double th, qv, ql, qi, rv0;
    int id;
};
__device__ __noinline__ CondenOut conden_any(double p, double ex, double thl, double qt, const double* __restrict__ tbl)
{
    CondenOut r;
    r.id = conden(p, ex, thl, qt, r.th, r.qv, r.ql, r.qi, r.rv0, tbl);
    return r;
}
__device__ __forceinline__ CondenOut conden_f64(double p, double ex, double thl, double qt, const double* __restrict__ tbl)
{
    CondenOut r;
    bool ok = true;
    const double tc = thl * ex;
    const double nu = MX(MN(uw_div_by(268.0 - tc, 20.0, 0.05), 1.0), 0.0);
    const double leff = (1.0 - nu) * c.xlv + nu * c.xls;
    double temps = tc;
    double rvls = qsat_qs_f64(temps, p, ok, tbl);
    r.rv0 = rvls;
    r.id = 0;
    if (rvls >= qt) {
        r.qv = qt;
        r.ql = 0.0;
        r.qi = 0.0;
    } else {
        ok = ok && uw_rcp_ok(leff);
        const double rleff = uw_rcp(leff);
        const double cpl = uw_div_by(c.cp, leff, rleff), a2 = c.ep2 * leff;
#pragma unroll 1
        for (int it = 0; it < 10; it++) {
            ok = ok && uw_rcp_ok(temps);
            const double rt = uw_rcp(temps);
            const double num = uw_div_by((tc - temps) * c.cp, leff, rleff) + qt - rvls;
            const double den = cpl + uw_div_by(uw_div_by(uw_div_by(a2 * rvls, c.r, c.rinv), temps, rt), temps, rt);
            ok = ok && uw_rcp_ok(den);
            temps = temps + uw_div_by(num, den, uw_rcp(den));
            rvls = qsat_qs_f64(temps, p, ok, tbl);
        }
        const double qc = MX(qt - rvls, 0.0);
        r.qv = qt - qc;
        r.ql = qc * (1.0 - nu);
        r.qi = nu * qc;
        r.id = (fabs((temps - uw_div_by(leff, c.cp, c.cpinv) * qc) - tc) >= 1.0) ? 1 : 0;
    }
    r.th = temps / ex;
    if (!ok) r = conden_any(p, ex, thl, qt, tbl);
    return r;
}
// ---- end of conden in FP64 ----

// The column code's saturation adjustment: one call for its ~20 sites (inlined at each of them, the stall
// on instruction fetch doubled the run time), with the results by value, in registers (through
// references they went through the stack, a store and a load each around every call).
template <int FAST>
__device__ __noinline__ CondenOut conden_out(double p, double ex, double thl, double qt, const double* __restrict__ tbl)
{
    if (!FAST) return conden_f64(p, ex, thl, qt, tbl);
    CondenOut r;
    r.id = conden_fast(p, ex, thl, qt, r.th, r.qv, r.ql, r.qi, r.rv0, tbl);
    return r;
}
template <int FAST>
__device__ __forceinline__ int conden_call(double p, double ex, double thl, double qt, double& th, double& qv,
                                           double& ql, double& qi, double& rv0, const double* __restrict__ tbl)
{
    const CondenOut r = conden_out<FAST>(p, ex, thl, qt, tbl);
    th = r.th;
    qv = r.qv;
    ql = r.ql;
    qi = r.qi;
    rv0 = r.rv0;
    return r.id;
}

// roots (uwshcu.F90:4787-4829); r1/r2 keep the caller's values on the failure branches.
__device__ __forceinline__ int roots(double a, double b, double cc, double& r1, double& r2)
{
    int status = 0;
    if (a == 0.0) {
        if (b == 0.0) status = 1;
        else r1 = -cc / b;
        r2 = r1;
    } else {
        if (b == 0.0) {
            if (a * cc > 0.0) status = 2;
            else r1 = sqrt(-cc / a);
            r2 = -r1;
        } else {
            if ((b * b - 4.0 * a * cc) < 0.0) {
                status = 3;
            } else {
                double q = -0.5 * (b + copysign(1.0, b) * sqrt(b * b - 4.0 * a * cc));
                r1 = q / a;
                r2 = cc / q;
            }
        }
    }
    return status;
}

// slope (uwshcu.F90:4831-4861); field/p0/sl are 1-based local arrays.
template <int KP>
__device__ __forceinline__ void slope(int mkx, const double* field, const double* p0, double* sl)
{
    double below = (field[2] - field[1]) / (p0[2] - p0[1]);
#pragma unroll 1
    for (int k = 2; k <= mkx; k++) {
        double above = (field[k] - field[k - 1]) / (p0[k] - p0[k - 1]);
        if (above > 0.0) sl[k - 1] = MX(0.0, MN(above, below));
        else sl[k - 1] = MN(0.0, MX(above, below));
        below = above;
    }
    sl[mkx] = sl[mkx - 1];
}

// qsinvert (uwshcu.F90:4863-4929) with exsfc = exnf(psfc).
__device__ __noinline__ double qsinvert(double qt, double thl, double psfc, double exsfc, const double* __restrict__ tbl)
{
    const double psmin = 100.0 * 100.0, dpsmax = 1.0;
    double es, qs, gam;
    double Ti = thl * exsfc;
    qsat3(Ti, psfc, es, qs, gam, tbl);
    double rhi = qt / qs;
    // single exit, fixed trip count: every lane of a warp leaves together
    double result = psmin;
    if (!(rhi <= 0.01)) {
        double TLCL = 55.0 + 1.0 / (1.0 / (Ti - 55.0) - uw_log(rhi) / 2840.0);
        double PiLCL = TLCL / thl;
        double ps = c.p00 * uw_pow(PiLCL, 1.0 / c.rovcp);
        bool done = false;
#pragma unroll 1
        for (int i = 1; i <= 10; i++) {
            if (done) continue;
            double Pis = uw_pow(ps / c.p00, c.rovcp);
            double Ts = thl * Pis;
            qsat3(Ts, ps, es, qs, gam, tbl);
            double err = qt - qs;
            double nu = MX(MN((268.0 - Ts) / 20.0, 1.0), 0.0);
            double leff = (1.0 - nu) * c.xlv + nu * c.xls;
            double dlnqsdT = gam * (c.cp / leff) / qs;
            double dTdPis = thl;
            double dPisdps = c.rovcp * Pis / ps;
            double dlnqsdps = -1.0 / (ps - (1.0 - c.ep2) * es);
            double derrdps = -qs * (dlnqsdT * dTdPis * dPisdps + dlnqsdps);
            double dps = -err / derrdps;
            ps = ps + dps;
            if (ps < 0.0) {
                done = true;
            } else if (fabs(dps) <= dpsmax) {
                result = ps;
                done = true;
            }
        }
    }
    return result;
}

// compute_alpha (uwshcu.F90:4931-4950)
__device__ __noinline__ double compute_alpha(double del_CIN, double ke)
{
    double x0 = 0.0;
#pragma unroll 1
    for (int it = 0; it < 10; it++) {
        double x1 = x0 - (uw_exp(-x0 * ke * del_CIN) - x0) / (-ke * del_CIN * uw_exp(-x0 * ke * del_CIN) - 1.0);
        x0 = x1;
    }
    return x0;
}

// compute_mumin2 (uwshcu.F90:4952-4979)
__device__ __noinline__ double compute_mumin2(double mulcl, double rmaxfrac, double mulow)
{
    double x0 = mulow;
#pragma unroll 1
    for (int it = 0; it < 10; it++) {
        double ex = uw_exp(-(x0 * x0));
        double ef = uw_erfc(x0);
        double exf = ex / ef;
        double t1 = ex / 2.0 / rmaxfrac;
        double t2 = mulcl * 2.5066 / 2.0;
        double f = 0.5 * (exf * exf) - 0.5 * (t1 * t1) - (t2 * t2);
        double fs = (2.0 * (exf * exf)) * (exf / sqrt(3.141592) - x0) + (0.5 * x0 * (ex * ex)) / (rmaxfrac * rmaxfrac);
        double x1 = x0 - f / fs;
        x0 = x1;
    }
    return x0;
}

// compute_ppen (uwshcu.F90:4981-5028); the 1.e-8 at :4998 is a default-real literal.
__device__ __noinline__ double compute_ppen(double wtwb, double D, double bogbot, double bogtop, double rho0j, double dpen)
{
    double x0;
    double SB = (bogtop - bogbot) / dpen;
    double s00 = bogbot / rho0j - D * wtwb;
    if (D * dpen < (double)1.e-8f) {
        if (s00 >= 0.0) x0 = dpen;
        else x0 = MX(0.0, MN(dpen, -0.5 * wtwb / s00));
    } else {
        if (s00 >= 0.0) x0 = dpen;
        else x0 = 0.0;
#pragma unroll 1
        for (int it = 0; it < 5; it++) {
            double f = uw_exp(-2.0 * D * x0) * (wtwb - (bogbot - SB / (2.0 * D)) / (D * rho0j)) +
                       (SB * x0 + bogbot - SB / (2.0 * D)) / (D * rho0j);
            double fs = -2.0 * D * uw_exp(-2.0 * D * x0) * (wtwb - (bogbot - SB / (2.0 * D)) / (D * rho0j)) +
                        (SB) / (D * rho0j);
            if (fs >= 0.0) fs = MX(fs, 1.e-10);
            else fs = MN(fs, -1.e-10);
            double x1 = x0 - f / fs;
            x0 = x1;
        }
    }
    return -MX(0.0, MN(dpen, x0));
}

// single_cin (uwshcu.F90:4704-4715) with the exner values of pbot/ptop supplied.
__device__ __forceinline__ double single_cin(double pbot, double exb, double thv0bot, double ptop, double ext,
                                             double thv0top, double thvubot, double thvutop)
{
    return ((1.0 - thvubot / thv0bot) + (1.0 - thvutop / thv0top)) * (pbot - ptop) /
           (pbot / (c.r * thv0bot * exb) + ptop / (c.r * thv0top * ext));
}

// getbuoy (uwshcu.F90:4672-4702) with the exner values supplied.
__device__ __forceinline__ void getbuoy(double pbot, double exb, double thv0bot, double ptop, double ext,
                                        double thv0top, double thvubot, double thvutop, double& plfc, double& cin)
{
    if (thvubot > thv0bot && thvutop > thv0top) {
        plfc = pbot;
    } else if (thvubot <= thv0bot && thvutop <= thv0top) {
        cin = cin - ((thvubot / thv0bot - 1.0) + (thvutop / thv0top - 1.0)) * (pbot - ptop) /
                        (pbot / (c.r * thv0bot * exb) + ptop / (c.r * thv0top * ext));
    } else if (thvubot > thv0bot && thvutop <= thv0top) {
        double frc = (thvutop / thv0top - 1.0) / ((thvutop / thv0top - 1.0) - (thvubot / thv0bot - 1.0));
        cin = cin - (thvutop / thv0top - 1.0) * ((ptop + frc * (pbot - ptop)) - ptop) /
                        (pbot / (c.r * thv0bot * exb) + ptop / (c.r * thv0top * ext));
    } else {
        double frc = (thvubot / thv0bot - 1.0) / ((thvubot / thv0bot - 1.0) - (thvutop / thv0top - 1.0));
        plfc = pbot - frc * (pbot - ptop);
        cin = cin - (thvubot / thv0bot - 1.0) * (pbot - plfc) /
                        (pbot / (c.r * thv0bot * exb) + ptop / (c.r * thv0top * ext));
    }
}

// fluxbelowinv (uwshcu.F90:5030-5094).  Writes xflx(0:kinv-1); the Fortran zeroes xflx(kinv:mkx)
// too, but the caller only reads 0..kinv-1.
__device__ __forceinline__ void fluxbelowinv(double cbmf, const double* ps0, int kinv, double dt, double xsrc,
                                             double xmean, double xtopin, double xbotin, double* xflx)
{
    double xtop, xbot;
    double dp = ps0[kinv - 1] - ps0[kinv];
    if (fabs(xbotin - xtopin) <= 1.e-13) {
        xbot = xbotin - 1.e-13;
        xtop = xtopin + 1.e-13;
    } else {
        xbot = xbotin;
        xtop = xtopin;
    }
    double xtop_ori = xtop, xbot_ori = xbot;
    double rcbmf = (cbmf * c.g * dt) / dp;
    double rpeff = (xmean - xtop) / (xbot - xtop);
    rpeff = MN(MX(0.0, rpeff), 1.0);
    if (rpeff == 0.0 || rpeff == 1.0) {
        xbot = xmean;
        xtop = xmean;
    }
    double rr = rpeff / rcbmf;
    double pinv = ps0[kinv - 1] - rpeff * dp;
#pragma unroll 1
    for (int k = 0; k <= kinv - 1; k++) xflx[k] = cbmf * (xsrc - xbot) * (ps0[0] - ps0[k]) / (ps0[0] - pinv);
    if (rr <= 1.0) xflx[kinv - 1] = xflx[kinv - 1] - (1.0 - rr) * cbmf * (xtop_ori - xbot_ori);
}

// findsp (uwshcu.F90:5164-5454) for one point; returns the wet-bulb qsp and ORs error bits.
__device__ double findsp_point(double q, double t, double p, unsigned int& errbits, const double* __restrict__ tbl)
{
    const double omeps = 1.0 - c.epsqs, trinv = 1.0 / c.ttrice;
    const double c3 = c.findsp_c3, dttol = 1.e-4, dqtol = 1.e-4, tt0 = 273.15;
    double dtt = 0.0, dq = 0.0, enin, enout = 1.0, tsp, qsp, hltalt = 0.0;
    int doit = 0;
    double tlim = MN(MX(t, 173.0), 373.0);
    double es = estblf(tlim, tbl);
    double denom = p - omeps * es;
    double qs = c.epsqs * es / denom;
    if (p > 5.0 * es && qs > 0.0 && qs < 0.5) {
        qs = MN(c.epsqs * es / denom, 1.0);
        double tc = tlim - tt0;
        double weight = MN(-tc * trinv, 1.0);
        double hlatsb = c.hlatv + weight * c.hlatf;
        double hlatvp = c.hlatv - 2369.0 * tc;
        hltalt = (tlim < tt0) ? hlatsb : hlatvp;
        enin = c.cpws * tlim + hltalt * q;
        double tmp = q - qs;
        double c1 = hltalt * c3;
        double c2 = (tlim + 36.0) * (tlim + 36.0);
        double r1b = c2 / (c2 + c1 * qs);
        double qvd = r1b * tmp;
        tsp = tlim + ((hltalt / c.cpws) * qvd);
        es = estblf(tsp, tbl);
        qsp = MN(c.epsqs * es / (p - omeps * es), 1.0);
    } else {
        doit = 1;
        tsp = tlim;
        qsp = q;
        enin = 1.0;
    }
#pragma unroll 1
    for (int l = 1; l <= 8 && doit == 0; l++) {
#if UW_TAPE_ORDER
        es = estblf(tsp, tbl);
        qs = MN(c.epsqs * es / (p - omeps * es), 1.0);
#else
        qs = qsp;   // es and qsp are those of tsp already
#endif
        double tc = tsp - tt0;
        bool lflg = (tc >= -c.ttrice && tc < 0.0);
        double weight = MN(-tc * trinv, 1.0);
        double hlatsb = c.hlatv + weight * c.hlatf;
        double hlatvp = c.hlatv - 2369.0 * tc;
        hltalt = (tsp < tt0) ? hlatsb : hlatvp;
        double tterm = lflg ? c.pcf[0] + tc * (c.pcf[1] + tc * (c.pcf[2] + tc * (c.pcf[3] + tc * c.pcf[4]))) : 0.0;
        double desdt = hltalt * es / (c.rgasv * tsp * tsp) + tterm * trinv;
        double dqsdt = (c.epsqs + omeps * qs) / (p - omeps * es) * desdt;
        double gg = enin - (c.cpws * tsp + hltalt * qsp);
        double dgdt = -(c.cpws + hltalt * dqsdt);
        double t1 = tsp - gg / dgdt;
        dtt = fabs(t1 - tsp) / t1;
        tsp = MX(t1, c.tmin);
        es = estblf(tsp, tbl);
        double q1 = MN(c.epsqs * es / (p - omeps * es), 1.0);
        dq = fabs(q1 - qsp) / MX(q1, 1.e-12);
        qsp = q1;
        if (dtt < dttol && dq < dqtol) doit = 2;
        enout = c.cpws * tsp + hltalt * qsp;
        if (tsp < 174.16) doit = 4;
    }
    if (doit == 0 && (dtt > dttol || dq > dqtol)) errbits |= UW_ERRBIT_FINDSP;
    if (doit == 2 && fabs((enin - enout) / (enin + enout)) > 1.e-4) errbits |= UW_ERRBIT_ENTHALPY;
    return qsp;
}

}  // namespace

// ------------------------------------------------------------------------------------------------
// The column kernel.  KP bounds the level arrays (mkx + 1 <= KP), NC the tracer count.
//
// MODE selects what a launch does:
//   UW_MODE_ALL      every column 0..iend-1 runs the whole scheme (single pass);
//   UW_MODE_TRIGGER  every column runs up to the end of the iteration-1 closure (uwshcu.F90:2184).
//                    Columns that leave the scheme on the way write their final outputs (the
//                    label-333 zeroes); the others write nothing and get their release level in
//                    A.trig_key, from which the caller builds the worklist, or without A.trig_key
//                    are appended to the worklist `wl` (warp ballot, one atomicAdd per warp);
//   UW_MODE_LIST     runs the whole scheme for the columns wl[0 .. *wl_count), 32 to a warp or fewer
//                    (uw_spread);
//   UW_MODE_LIST1    as UW_MODE_LIST, except that a column taking the implicit-CIN branch of
//                    iteration 2 (uwshcu.F90:1759-1889) stores its state in the hand-off region
//                    A.hand (a free slot permitting) and stops there;
//   UW_MODE_RESUME   continues the hand-off slots order[] from that point to the end.
// The worklist path recomputes the phase-1 part of a convecting column instead of storing it: the
// heavy buoyancy-sorting work then runs in warps made only of convecting columns.  The split at the
// CIN decision drops the columns that end in iteration 1 or take the explicit-CIN branch from the
// warps of iteration 2, and sorts the rest by release level and iteration-1 updraft depth, which predicts
// the iteration-2 depth (lanes whose updraft has stopped wait for the deepest one in their warp).  The
// worklist itself is in order of the release level: lanes that start their updraft at the same level
// access the same rows of their profiles, one line instead of one per level.
#define UW_MODE_ALL 0
#define UW_MODE_TRIGGER 1
#define UW_MODE_LIST 2
#define UW_MODE_LIST1 3
#define UW_MODE_RESUME 4
#define UW_MODE_IS_LIST(m) ((m) == UW_MODE_LIST || (m) == UW_MODE_LIST1 || (m) == UW_MODE_RESUME)

// The column code and the kernels have internal linkage: every unit that includes a column-code
// header (FP64, fast, mixed, tangent) carries its own copies under the same names.
namespace {

// One column per lane: column i_in of A when `active` (in UW_MODE_RESUME, i_in is a hand-off slot).
// All 32 lanes of the warp must call it together (it starts with a warp ballot).  `tbl` is the saturation table in shared memory.  In
// UW_MODE_TRIGGER, convecting columns are appended to wl / *wl_count.
// FAST = 1: the fast-FP64 precision mode (conden_fast in place of conden), not bit-exact.
// ZW = 1: compute_zwshcu (zwshcu.F90), which reads A.omega and the zw_* options; compiled out of the
// compute_uwshcu instantiations.
template <int KP, int NC, int MODE, int FAST, int ZW = 0>
__device__ __forceinline__ void uw_column(const UwArgs& A, const double* __restrict__ tbl, const int i_in,
                                          const bool active, int* __restrict__ wl, int* __restrict__ wl_count)
{
    const int i = (MODE == UW_MODE_RESUME && active) ? A.hand->col[i_in] : i_in;
    // Code size bounds the worklist passes: with the loops unrolled by the compiler and exp, log and pow
    // inlined at each use their kernels were 833 kB (LIST1) and 631 kB (RESUME), far beyond the
    // instruction caches that 16 warps at different places share, and at full occupancy a warp waited 4.4
    // to 6.5 cycles per instruction for its next one.  So the loops here are not unrolled (but for the resumed
    // slopes, by tracer, and the state copies of uw_state.cuh) and the transcendentals are calls.
#define CONDEN(...) conden_call<FAST>(__VA_ARGS__)
// qsat_qs(t, p) right after a CONDEN call at that temperature and pressure: its first lookup
#define UW_QSAT_OF_CONDEN(t, p) rvj
    bool cand = false;
    // lanes of this warp that run a column; UW_SYNC() joins them where every one of them arrives
    const unsigned live = __ballot_sync(0xffffffffu, active);
#define UW_SYNC() __syncwarp(live)
// one level of slope: the limited slope from the difference quotients above and below
#define UW_SLOPE(above, below) ((above) > 0.0 ? MX(0.0, MN(above, below)) : MN(0.0, MX(above, below)))
    if (active) {

    const int mix = A.mix, mkx = A.mkx, ncnst = A.ncnst;
    const double dt = A.dt;
    const double xlv = c.xlv, xls = c.xls, cp = c.cp, zvir = c.zvir, r = c.r, g = c.g, p00 = c.p00,
                 rovcp = c.rovcp, rpen = c.rpen;
    const double rle = c.rle, rkm = c.rkm, rkfre = 1.0, rmaxfrac = 0.10, mumin1 = 0.906, rbuoy = 1.0,
                 rdrag = 1.0, epsvarw = 5.e-4, PGFc = 0.7, criqc = c.criqc, frc_rasn = 1.0, kevp = 2.e-6;
    const int ixnumliq = c.ixnumliq, ixnumice = c.ixnumice;

    // Row of level k in the caller's arrays: bottom-up (compute_uwshcu) or CAM's top-down order
    // (compute_uwshcu_inv, uwshcu.F90:380-469, where interface k and layer k both sit at row mkx-k).
    const int inv = A.inv;
#define RI(k) (inv ? (mkx - (k)) : (k))
#define RL(k) (inv ? (mkx - (k)) : ((k) - 1))
#define GI(a, k) __ldg(&A.a[(size_t)RI(k) * mix + i])
#define GL(a, k) __ldg(&A.a[(size_t)RL(k) * mix + i])
#define GT(m, k) __ldg(&A.tr0[((size_t)((m) - 1) * mkx + RL(k)) * mix + i])
#define OI(a, k) A.a[(size_t)RI(k) * mix + i]
#define OL(a, k) A.a[(size_t)RL(k) * mix + i]
#define OT(m, k) A.trten[((size_t)((m) - 1) * mkx + RL(k)) * mix + i]
#define CNT(x) (inv ? (double)(mkx + 1) - (x) : (x))
#define DLV(j, k) A.diag_level[((size_t)(j) * (mkx + 1) + (k)) * mix + i]
// uemf(k), evaluated on demand with the same expressions as :3416-3422
#define UEMF(kk)                                                                                          \
    ((kk) <= kinv - 2 ? cbmf * (ps0[0] - ps0[(kk)]) / (ps0[0] - ps0[kinv - 1])                             \
                      : ((kk) <= krel - 1 ? cbmf : ((kk) <= kbup - 1 ? umf[(kk)] : ((kk) <= kpen - 1 ? emf[(kk)] : 0.0))))
// the profiles that the per-level diagnostics show outside the updraft's levels as well
#define ZERO_DIAG_PROFILES()                                                                              \
    _Pragma("unroll 1") for (int k = 0; k <= mkx; k++) {                                                  \
        ufrc[k] = 0.0; thlu[k] = 0.0; qtu[k] = 0.0; thvu[k] = 0.0; uu[k] = 0.0; vu[k] = 0.0;              \
        dwten[k] = 0.0; diten[k] = 0.0; fer[k] = 0.0; fdr[k] = 0.0;                                       \
    }
// per-level diagnostics of the current state, levels bottom-up in both level orders
// (uwshcu.F90:1945-1990 and :4383-4433)
#define PUT_DIAG_LEVEL()                                                                                  \
    if (A.diag_level) {                                                                                   \
        _Pragma("unroll 1") for (int k = 0; k <= mkx; k++) {                                              \
            DLV(UW_DL_UFRC, k) = ufrc[k];                                                                 \
            DLV(UW_DL_QTU, k) = qtu[k];                                                                   \
            DLV(UW_DL_THLU, k) = thlu[k];                                                                 \
            DLV(UW_DL_THVU, k) = thvu[k];                                                                 \
            DLV(UW_DL_UU, k) = uu[k];                                                                     \
            DLV(UW_DL_VU, k) = vu[k];                                                                     \
            DLV(UW_DL_UEMF, k) = UEMF(k);                                                                 \
            DLV(UW_DL_FLXRAIN, k) = flxrain[k];                                                           \
            DLV(UW_DL_FLXSNOW, k) = flxsnow[k];                                                           \
        }                                                                                                 \
        _Pragma("unroll 1") for (int j = UW_DL_FER; j < UW_NDL; j++) DLV(j, 0) = 0.0;                     \
        _Pragma("unroll 1") for (int k = 1; k <= mkx; k++) {                                              \
            DLV(UW_DL_FER, k) = fer[k];                                                                   \
            DLV(UW_DL_FDR, k) = fdr[k];                                                                   \
            DLV(UW_DL_DWTEN, k) = dwten[k];                                                               \
            DLV(UW_DL_DITEN, k) = diten[k];                                                               \
        }                                                                                                 \
    }

    // ---- thread-private profiles ---------------------------------------------------------------
    double ps0[KP], p0[KP], dp0[KP], zs0[KP], exn0[KP], exns0[KP];
    double qv0[KP], ql0[KP], qi0[KP], t0[KP], s0[KP], qt0[KP], thl0[KP];
    double ssthl0[KP], ssqt0[KP], ssu0[KP], ssv0[KP], sstr0[NC][KP];
    double thv0bot[KP], thv0top[KP], thvl0bot[KP], thvl0top[KP];
    double thv0bot_o[KP], thv0top_o[KP], thvl0bot_o[KP], thvl0top_o[KP];
    double umf[KP], emf[KP], thlu[KP], qtu[KP], uu[KP], vu[KP], thvu[KP], wu[KP], ufrc[KP], rei[KP];
    double fer[KP], fdr[KP], dwten[KP], diten[KP], tru[NC][KP];
    double thlu_emf[KP], qtu_emf[KP], uu_emf[KP], vu_emf[KP], tru_emf[NC][KP];
    double slflx[KP], qtflx[KP], uflx[KP], vflx[KP], trflx[NC][KP], xflx[KP];
    double qlten_sink[KP], qiten_sink[KP], nlten_sink[KP], niten_sink[KP];
    double uten[KP], vten[KP], uf[KP], vf[KP], qrten[KP], qsten[KP], slten[KP], qtten[KP];
    double qlten[KP], qiten[KP], qvten[KP], sten[KP], qc[KP], qc_l[KP], qc_i[KP], evapc[KP];
    double flxrain[KP], flxsnow[KP], cufrc[KP], qcu[KP], qlu[KP], qiu[KP], trten[NC][KP];
    double qw0[KP], trflx_d[KP], trflx_u[KP];
#if !UW_TAPE_ORDER
    double qltop[KP], qitop[KP], env_thv[KP], env_exc[KP], env_rho[KP], env_rei[KP];
#endif
    double trsrc[NC], tre[NC];

    unsigned int errbits = 0;
    int xflags = 0, lflags = 0;
    bool id_exit = false;
    // stop: the column leaves the scheme (the Fortran's `go to 333`); every later section skips.
    bool stop = false;
    int kinv = 0, klcl = 0, klfc = 0, krel = 0, kbup = 0, kpen = 0;
    int kinv_s = 0, klcl_s = 0, klfc_s = 0, krel_s = 0, kbup_s = 0, kpen_s = 0;
    double cin = 0, cinlcl = 0, plcl = 0, plfc = 0, prel = 0, exlcl = 1.0, exprel = 1.0, tkeavg = 0,
           thvlmin = 0, qtsrc = 0, thlsrc = 0, thvlsrc = 0, usrc = 0, vsrc = 0, thv0lcl = 0, thv0rel = 0;
    double cin_i = 0, cinlcl_i = 0, ke = 0, kinv_o_d = 0;
    int kinv_o = 0, klcl_o = 0, klfc_o = 0;
    double plcl_o = 0, plfc_o = 0, tkeavg_o = 0, thvlmin_o = 0, qtsrc_o = 0, thvlsrc_o = 0, thlsrc_o = 0,
           usrc_o = 0, vsrc_o = 0, thv0lcl_o = 0, trsrc_o[NC];
    double cin_s = -1.0, cinlcl_s = -1.0, plcl_s = 0, plfc_s = 0, pinv_s = 0, pbup_s = 0, ppen_s = 0,
           tkeavg_s = 0;
    double cbmf = 0, wlcl = 0, ufrclcl = 0, ppen = 0, precip = 0, snow = 0, rliq = 0, cush, cnt, cnb;
    double thlu_top = 0, qtu_top = 0, exntop = 1.0, drage = 0, bogbot = 0, bogtop = 0, rho0j = 0,
           wtwb = 0, wtw = 0, xs1 = 0, xs2 = 0, xc1 = 0, xc2 = 0;
    double thj = 0, qvj = 0, qlj = 0, qij = 0, rvj = 0;
    (void)rvj;
    double rainflx = 0, snowflx = 0;
    (void)kinv_o_d;
    const double pblh = __ldg(&A.pblh[i]);
    double tscaleh_r = 0.0;   // UW_MODE_RESUME: tscaleh of the iteration handed over
    bool handed = false;      // UW_MODE_LIST1: the column continues in UW_MODE_RESUME

    if constexpr (MODE != UW_MODE_RESUME) {   // uniform

    // The Fortran zeroes every output here (uwshcu.F90:1087-1124).  Every way out of the column below
    // writes all of them (the final outputs, label 333, or the explicit-CIN branch of iteration 2),
    // so nothing is stored twice.

    // ---- inputs and findsp (uwshcu.F90:1216-1259), and non-finite inputs ----------------------
    // Non-finite inputs have no counterpart in the Fortran, where a NaN or Inf propagates into the
    // column's outputs or stops the model in findsp: a column with a non-finite value in any input
    // the scheme reads takes the exit path (label-333 outputs), is marked UW_X_NONFINITE and sets
    // only that status bit (no findsp at or above the bad level, no conden).  The values are checked
    // as they are loaded; z0 and tke, which the scheme reads later and only at some levels, once here.
    bool nonfinite = !uw_isfinite(pblh) || !uw_isfinite(A.cush[i]);
#pragma unroll 1
    for (int k = 0; k <= mkx; k++) {
        ps0[k] = GI(ps0, k);
        zs0[k] = GI(zs0, k);
        nonfinite |= !uw_isfinite(ps0[k]) || !uw_isfinite(zs0[k]) || !uw_isfinite(GI(tke, k));
        exns0[k] = uw_pow(ps0[k] / p00, rovcp);
    }
#pragma unroll 1
    for (int k = 1; k <= mkx; k++) {
        p0[k] = GL(p0, k);
        dp0[k] = GL(dp0, k);
        qv0[k] = GL(qv0, k);
        ql0[k] = GL(ql0, k);
        qi0[k] = GL(qi0, k);
        t0[k] = GL(t0, k);
        s0[k] = GL(s0, k);
        nonfinite |= !uw_isfinite(p0[k]) || !uw_isfinite(dp0[k]) || !uw_isfinite(qv0[k]) || !uw_isfinite(ql0[k]) ||
                     !uw_isfinite(qi0[k]) || !uw_isfinite(t0[k]) || !uw_isfinite(s0[k]) || !uw_isfinite(GL(z0, k));
        exn0[k] = uw_pow(p0[k] / p00, rovcp);
        qt0[k] = (qv0[k] + ql0[k] + qi0[k]);
        thl0[k] = (t0[k] - xlv * ql0[k] / cp - xls * qi0[k] / cp) / exn0[k];
        qw0[k] = nonfinite ? 0.0 : findsp_point(qv0[k], t0[k], p0[k], errbits, tbl);
    }
    cush = A.cush[i];
    {
        double tmpf[KP];
        slope<KP>(mkx, thl0, p0, ssthl0);
        slope<KP>(mkx, qt0, p0, ssqt0);
#pragma unroll 1
        for (int k = 1; k <= mkx; k++) {
            tmpf[k] = GL(u0, k);
            nonfinite |= !uw_isfinite(tmpf[k]);
        }
        slope<KP>(mkx, tmpf, p0, ssu0);
#pragma unroll 1
        for (int k = 1; k <= mkx; k++) {
            tmpf[k] = GL(v0, k);
            nonfinite |= !uw_isfinite(tmpf[k]);
        }
        slope<KP>(mkx, tmpf, p0, ssv0);
#pragma unroll 1
        for (int m = 1; m <= ncnst; m++) {
#pragma unroll 1
            for (int k = 1; k <= mkx; k++) {
                tmpf[k] = GT(m, k);
                nonfinite |= !uw_isfinite(tmpf[k]);
            }
            slope<KP>(mkx, tmpf, p0, sstr0[m - 1]);
        }
    }
    if (nonfinite) {
        xflags |= UW_X_NONFINITE;
        errbits = UW_ERRBIT_NONFINITE;   // findsp of the levels below the bad one reports nothing
        id_exit = true;
        stop = true;
    }
    // thv0 at layer bottom/top (:1275-1299)
#pragma unroll 1
    for (int k = 1; k <= mkx && !nonfinite; k++) {
        double thl0bot = thl0[k] + ssthl0[k] * (ps0[k - 1] - p0[k]);
        double qt0bot = qt0[k] + ssqt0[k] * (ps0[k - 1] - p0[k]);
        if (CONDEN(ps0[k - 1], exns0[k - 1], thl0bot, qt0bot, thj, qvj, qlj, qij, rvj, tbl)) {
            xflags |= UW_X_CONDEN;
            id_exit = true;
            stop = true;
            break;
        }
        thv0bot[k] = thj * (1.0 + zvir * qvj - qlj - qij);
        thvl0bot[k] = thl0bot * (1.0 + zvir * qt0bot);
        double thl0top = thl0[k] + ssthl0[k] * (ps0[k] - p0[k]);
        double qt0top = qt0[k] + ssqt0[k] * (ps0[k] - p0[k]);
        if (CONDEN(ps0[k], exns0[k], thl0top, qt0top, thj, qvj, qlj, qij, rvj, tbl)) {
            xflags |= UW_X_CONDEN;
            id_exit = true;
            stop = true;
            break;
        }
        thv0top[k] = thj * (1.0 + zvir * qvj - qlj - qij);
        thvl0top[k] = thl0top * (1.0 + zvir * qt0top);
        thv0bot_o[k] = thv0bot[k];
        thv0top_o[k] = thv0top[k];
        thvl0bot_o[k] = thvl0bot[k];
        thvl0top_o[k] = thvl0top[k];
    }
    if (!stop) {
    // The Fortran zeroes some 80 profiles here and again at the implicit-CIN restore (:1333-1408,
    // :1759-1889).  The sections below write every level that they, or the outputs, read (the zeroes
    // outside the cloud included), each level once; only the per-level diagnostics show the others.
    if (A.diag_level) ZERO_DIAG_PROFILES();
    cnt = (double)mkx;
    cnb = 0.0;
    }
    } else {   // uniform
        // the state UW_MODE_LIST1 stored at the implicit-CIN branch of iteration 2 (uw_state.cuh), and
        // the environment profiles that the set-up builds from the inputs, with the same operations
        UW_LOAD_STATE(A.hand->state + i_in, (size_t)A.hand->cap, tscaleh_r);
#pragma unroll 1
        for (int k = 0; k <= mkx; k++) {
            ps0[k] = GI(ps0, k);
            zs0[k] = GI(zs0, k);
        }
#pragma unroll 1
        for (int k = 1; k <= mkx; k++) {
            p0[k] = GL(p0, k);
            dp0[k] = GL(dp0, k);
        }
#pragma unroll 1
        for (int k = 1; k <= mkx; k++) {
            qv0[k] = GL(qv0, k);
            ql0[k] = GL(ql0, k);
            qi0[k] = GL(qi0, k);
            t0[k] = GL(t0, k);
            s0[k] = GL(s0, k);
            qt0[k] = (qv0[k] + ql0[k] + qi0[k]);
            thl0[k] = (t0[k] - xlv * ql0[k] / cp - xls * qi0[k] / cp) / exn0[k];
        }
        {
            // as in the set-up
            double pp = p0[1], pt = thl0[1], pq = qt0[1], pu = GL(u0, 1), pv = GL(v0, 1), bt = 0.0, bq = 0.0, bu = 0.0,
                   bv = 0.0, ptr[NC], btr[NC];
#pragma unroll (NC <= 5 ? NC : 1)
            for (int m = 0; m < NC; m++) {
                btr[m] = 0.0;
                ptr[m] = 0.0;
                if (m < ncnst) {
                    ptr[m] = GT(m + 1, 1);
                }
            }
#pragma unroll 1
            for (int k = 2; k <= mkx; k++) {
                const double xu = GL(u0, k), xv = GL(v0, k), xt = thl0[k], xq = qt0[k], xp = p0[k], dpk = xp - pp;
                const double at = (xt - pt) / dpk, aq = (xq - pq) / dpk, au = (xu - pu) / dpk, av = (xv - pv) / dpk;
                if (k == 2) {
                    bt = at;
                    bq = aq;
                    bu = au;
                    bv = av;
                }
                ssthl0[k - 1] = UW_SLOPE(at, bt);
                ssqt0[k - 1] = UW_SLOPE(aq, bq);
                ssu0[k - 1] = UW_SLOPE(au, bu);
                ssv0[k - 1] = UW_SLOPE(av, bv);
#pragma unroll (NC <= 5 ? NC : 1)
                for (int m = 0; m < NC; m++) {
                    if (m < ncnst) {
                        const double xr = GT(m + 1, k), ar = (xr - ptr[m]) / dpk;
                        if (k == 2) btr[m] = ar;
                        sstr0[m][k - 1] = UW_SLOPE(ar, btr[m]);
                        btr[m] = ar;
                        ptr[m] = xr;
                    }
                }
                pp = xp; pt = xt; pq = xq; pu = xu; pv = xv;
                bt = at; bq = aq; bu = au; bv = av;
            }
            ssthl0[mkx] = ssthl0[mkx - 1];
            ssqt0[mkx] = ssqt0[mkx - 1];
            ssu0[mkx] = ssu0[mkx - 1];
            ssv0[mkx] = ssv0[mkx - 1];
#pragma unroll 1
            for (int m = 0; m < ncnst; m++) sstr0[m][mkx] = sstr0[m][mkx - 1];
        }
        if (A.diag_level) ZERO_DIAG_PROFILES();
    }

    UW_SYNC();

    // ---- implicit-CIN loop (uwshcu.F90:1421-4331) --------------------------------------------
    // Lockstep skeleton.  Every lane of the warp runs the same iterations of this loop and of every
    // level loop inside it: a column's own level range and its exits are per-lane predicates.  Each
    // section is `if (!stop) do { ... } while (0);`, so an exit (`stop = true; break;`) skips the
    // rest of the section and every later one, and the lanes meet again at UW_SYNC() between
    // sections.  (Lanes that leave a loop at different iterations otherwise run apart for the rest
    // of the column: the worklist kernel ran with 1.9 of 32 lanes active.)  Loops marked `uniform`
    // have the same trip count on every live lane; UW_SYNC() appears only directly inside them.
#pragma unroll 1
    for (int iter = (MODE == UW_MODE_RESUME ? 2 : 1); iter <= (MODE == UW_MODE_TRIGGER ? 1 : 2); iter++) {   // uniform
        double tscaleh = tscaleh_r;
        if constexpr (MODE != UW_MODE_RESUME) {   // uniform
        if (!stop) do {
        tscaleh = cush;
        cush = -1.0;

        // kinv (:1455-1468): the first interface from the top whose layer brackets pblh + 5
        kinv = 1;
        {
            bool found = false;
#pragma unroll 1
            for (int k = mkx - 1; k >= 1; k--) {
                if (!found && (pblh + 5.0 - zs0[k]) * (pblh + 5.0 - zs0[k + 1]) < 0.0) {
                    kinv = k + 1;
                    found = true;
                }
            }
        }
        if (kinv <= 1) {
            xflags |= UW_X_KINV1;
            id_exit = true;
            stop = true;
            break;
        }
        // tkeavg, thvlmin (:1484-1499)
        {
            double dpsum = 0.0;
            tkeavg = 0.0;
            thvlmin = 1000.0;
#pragma unroll 1
            for (int k = 0; k <= mkx; k++) {
                if (k > kinv - 1) continue;
                double dpi;
                if (k == 0) dpi = ps0[0] - p0[1];
                else if (k == (kinv - 1)) dpi = p0[kinv - 1] - ps0[kinv - 1];
                else dpi = p0[k] - p0[k + 1];
                dpsum = dpsum + dpi;
                tkeavg = tkeavg + dpi * GI(tke, k);
                if (k != 0) thvlmin = MN(thvlmin, MN(thvl0bot[k], thvl0top[k]));
            }
            tkeavg = tkeavg / dpsum;
        }
        // source air (:1509-1516)
        qtsrc = qt0[1];
        thvlsrc = thvlmin;
        thlsrc = thvlsrc / (1.0 + zvir * qtsrc);
        usrc = GL(u0, kinv - 1) + ssu0[kinv - 1] * (ps0[kinv - 1] - p0[kinv - 1]);
        vsrc = GL(v0, kinv - 1) + ssv0[kinv - 1] * (ps0[kinv - 1] - p0[kinv - 1]);
#pragma unroll 1
        for (int m = 1; m <= ncnst; m++) trsrc[m - 1] = GT(m, 1);
        } while (0);
        UW_SYNC();
        // LCL (:1533-1549)
        if (!stop) do {
        plcl = qsinvert(qtsrc, thlsrc, ps0[0], exns0[0], tbl);
        klcl = mkx;
        {
            bool found = false;
#pragma unroll 1
            for (int k = 0; k <= mkx; k++) {
                if (!found && ps0[k] < plcl) {
                    klcl = k;
                    found = true;
                }
            }
        }
        klcl = MX(1, klcl);
        if (plcl < 30000.0) {
            xflags |= UW_X_KLCLMKX;
            id_exit = true;
            stop = true;
            break;
        }
        exlcl = exnf(plcl);
        {
            double thl0lcl = thl0[klcl] + ssthl0[klcl] * (plcl - p0[klcl]);
            double qt0lcl = qt0[klcl] + ssqt0[klcl] * (plcl - p0[klcl]);
            if (CONDEN(plcl, exlcl, thl0lcl, qt0lcl, thj, qvj, qlj, qij, rvj, tbl)) {
                xflags |= UW_X_CONDEN;
                id_exit = true;
                stop = true;
            break;
            }
            thv0lcl = thj * (1.0 + zvir * qvj - qlj - qij);
        }
        } while (0);
        UW_SYNC();
        // CIN (:1592-1685).  One loop over k = kinv .. mkx-1 serves both cases of the Fortran (LCL at
        // or above kinv, LCL below kinv), with one conden call at ps0(k) per level for every lane.
        // When the LCL is below kinv the Fortran also calls conden at ps0(k-1) with the same source
        // air; above the first level that repeats the previous level's call bit for bit, so only
        // the first level makes it here.
        if (!stop) {
            cin = 0.0;
            cinlcl = 0.0;
            plfc = 0.0;
            klfc = mkx;
        }
        {
            const bool lcl_above = (klcl >= kinv);
            double thvubot = 0.0, thvutop = 0.0;
            bool ldone = stop;
#pragma unroll 1
            for (int k = 2; k <= mkx - 1; k++) {   // uniform (kinv >= 2)
                if (!ldone && k >= kinv) do {
                    if (lcl_above && k < klcl) {
                        thvubot = thvlsrc;
                        thvutop = thvlsrc;
                        cin = cin + single_cin(ps0[k - 1], exns0[k - 1], thv0bot[k], ps0[k], exns0[k], thv0top[k], thvubot, thvutop);
                        break;
                    }
                    if (!lcl_above && k == kinv) {
                        if (CONDEN(ps0[k - 1], exns0[k - 1], thlsrc, qtsrc, thj, qvj, qlj, qij, rvj, tbl)) {
                            xflags |= UW_X_CONDEN;
                            id_exit = true;
                            stop = true;
                            break;
                        }
                        thvutop = thj * (1.0 + zvir * qvj - qlj - qij);
                    }
                    const bool atlcl = lcl_above && k == klcl;
                    if (atlcl) {
                        thvubot = thvlsrc;
                        thvutop = thvlsrc;
                        cin = cin + single_cin(ps0[k - 1], exns0[k - 1], thv0bot[k], plcl, exlcl, thv0lcl, thvubot, thvutop);
                        if (cin < 0.0) lflags |= UW_L_CINLCL;
                        cinlcl = MX(cin, 0.0);
                        cin = cinlcl;
                        thvubot = thvlsrc;
                    } else {
                        thvubot = thvutop;
                    }
                    if (CONDEN(ps0[k], exns0[k], thlsrc, qtsrc, thj, qvj, qlj, qij, rvj, tbl)) {
                        xflags |= UW_X_CONDEN;
                        id_exit = true;
                        stop = true;
                        break;
                    }
                    thvutop = thj * (1.0 + zvir * qvj - qlj - qij);
                    getbuoy(atlcl ? plcl : ps0[k - 1], atlcl ? exlcl : exns0[k - 1], atlcl ? thv0lcl : thv0bot[k],
                            ps0[k], exns0[k], thv0top[k], thvubot, thvutop, plfc, cin);
                    if (plfc > 0.0) {
                        klfc = k;
                        ldone = true;
                    }
                } while (0);
                if (stop) ldone = true;
            }
        }
        UW_SYNC();
        if (!stop) do {
        // (label 35, :1676-1685)
        if (cin < 0.0) lflags |= UW_L_CIN;
        cin = MX(0.0, cin);
        if (klfc >= mkx) {
            klfc = mkx;
            xflags |= UW_X_KLFCMKX;
            id_exit = true;
            stop = true;
            break;
        }
        if (iter == 1) {
            cin_i = cin;
            cinlcl_i = cinlcl;
            ke = rbuoy / (rkfre * tkeavg + epsvarw);
            kinv_o = kinv; klcl_o = klcl; klfc_o = klfc; plcl_o = plcl; plfc_o = plfc;
            tkeavg_o = tkeavg; thvlmin_o = thvlmin; qtsrc_o = qtsrc; thvlsrc_o = thvlsrc;
            thlsrc_o = thlsrc; usrc_o = usrc; vsrc_o = vsrc; thv0lcl_o = thv0lcl;
#pragma unroll 1
            for (int m = 0; m < ncnst; m++) trsrc_o[m] = trsrc[m];
        } else {
            double del_CIN = cin - cin_i;
            if (del_CIN > 0.0) {
                // implicit CIN: restore the iteration-1 state (:1759-1889)
                double alpha = compute_alpha(del_CIN, ke);
                cin = cin_i + alpha * del_CIN;
                cinlcl = cinlcl_i;
                kinv = kinv_o; klcl = klcl_o; klfc = klfc_o; plcl = plcl_o; plfc = plfc_o;
                tkeavg = tkeavg_o; thvlmin = thvlmin_o; qtsrc = qtsrc_o; thvlsrc = thvlsrc_o;
                thlsrc = thlsrc_o; usrc = usrc_o; vsrc = vsrc_o; thv0lcl = thv0lcl_o;
#pragma unroll 1
                for (int m = 0; m < ncnst; m++) trsrc[m] = trsrc_o[m];
                exlcl = exnf(plcl);
#pragma unroll 1
                for (int k = 1; k <= mkx; k++) {
                    qv0[k] = GL(qv0, k);
                    ql0[k] = GL(ql0, k);
                    qi0[k] = GL(qi0, k);
                    t0[k] = GL(t0, k);
                    s0[k] = GL(s0, k);
                    qt0[k] = (qv0[k] + ql0[k] + qi0[k]);
                    thl0[k] = (t0[k] - xlv * ql0[k] / cp - xls * qi0[k] / cp) / exn0[k];
                    thv0bot[k] = thv0bot_o[k];
                    thv0top[k] = thv0top_o[k];
                    thvl0bot[k] = thvl0bot_o[k];
                    thvl0top[k] = thvl0top_o[k];
                }
                slope<KP>(mkx, thl0, p0, ssthl0);
                slope<KP>(mkx, qt0, p0, ssqt0);
                if (A.diag_level) ZERO_DIAG_PROFILES();
                precip = 0.0; snow = 0.0; rliq = 0.0; cbmf = 0.0;
                cnt = (double)mkx; cnb = 0.0; ufrclcl = 0.0; wlcl = 0.0;
            } else {
                // explicit CIN: iteration 1's results are the column's (the Fortran's *_s copies,
                // :1891-2011, :4177-4277).  The profiles still hold them (this iteration has rebuilt
                // the environment only) and cush is in tscaleh; flxprc1/flxsnow1 are zero on this path.
                lflags |= UW_L_DELCIN;
#pragma unroll 1
                for (int k = 0; k <= mkx; k++) {
                    OI(umf, k) = umf[k];
                    OI(wu, k) = wu[k];
                    OI(slflx, k) = slflx[k];
                    OI(qtflx, k) = qtflx[k];
                    OI(flxprc1, k) = 0.0;
                    OI(flxsnow1, k) = 0.0;
                }
#pragma unroll 1
                for (int k = 1; k <= mkx; k++) {
                    OL(qvten, k) = qvten[k]; OL(qlten, k) = qlten[k]; OL(qiten, k) = qiten[k];
                    OL(sten, k) = sten[k]; OL(uten, k) = uten[k]; OL(vten, k) = vten[k];
                    OL(qrten, k) = qrten[k]; OL(qsten, k) = qsten[k]; OL(evapc, k) = evapc[k];
                    OL(cufrc, k) = cufrc[k]; OL(qcu, k) = qcu[k]; OL(qlu, k) = qlu[k];
                    OL(qiu, k) = qiu[k]; OL(qc, k) = qc[k];
#pragma unroll 1
                    for (int m = 1; m <= ncnst; m++) OT(m, k) = trten[m - 1][k];
                }
                A.precip[i] = precip;
                A.snow[i] = snow;
                A.cush[i] = tscaleh;
                A.cbmf[i] = cbmf;
                A.rliq[i] = rliq;
                A.cnt[i] = CNT(cnt);
                A.cnb[i] = CNT(cnb);
                if (A.diag_real) {
                    A.diag_real[UW_DR_CIN * (size_t)mix + i] = cin_s;
                    A.diag_real[UW_DR_CINLCL * (size_t)mix + i] = cinlcl_s;
                    A.diag_real[UW_DR_PLCL * (size_t)mix + i] = plcl_s;
                    A.diag_real[UW_DR_PLFC * (size_t)mix + i] = plfc_s;
                    A.diag_real[UW_DR_PINV * (size_t)mix + i] = pinv_s;
                    A.diag_real[UW_DR_PBUP * (size_t)mix + i] = pbup_s;
                    A.diag_real[UW_DR_PPEN * (size_t)mix + i] = ppen_s;
                    A.diag_real[UW_DR_TKEAVG * (size_t)mix + i] = tkeavg_s;
                }
                kinv = kinv_s; klcl = klcl_s; klfc = klfc_s; krel = krel_s; kbup = kbup_s; kpen = kpen_s;
                PUT_DIAG_LEVEL();
                id_exit = false;
                stop = true;
            break;
            }
        }

        } while (0);
        UW_SYNC();
        }   // MODE != UW_MODE_RESUME
        if constexpr (MODE == UW_MODE_LIST1) {   // uniform
        if (iter == 2) {   // uniform
            // implicit CIN: the rest of the column runs in the UW_MODE_RESUME launch; without a free
            // slot it goes on here
            const unsigned want = __ballot_sync(live, !stop);
            if (want) {
                const UwHand& H = *A.hand;
                const unsigned ln = threadIdx.x & 31u;
                const int leader = __ffs(want) - 1;
                int base = 0;
                if ((int)ln == leader) base = atomicAdd(H.count, __popc(want));
                base = __shfl_sync(live, base, leader);
                const int slot = base + __popc(want & ((1u << ln) - 1u));
                if (!stop && slot < H.cap) {
                    H.col[slot] = i;
                    H.key[slot] = krel_s * 64 + 63 - MN(MX(kpen_s - krel_s, 0), 63);
                    UW_SAVE_STATE(H.state + slot, (size_t)H.cap, tscaleh);
                    handed = true;
                    stop = true;
                }
            }
        }
        }
        // ---- release level and closure (:2035-2184) ------------------------------------------
        if (!stop) do {
        if (klcl < kinv) {
            krel = kinv;
            prel = ps0[krel - 1];
            exprel = exns0[krel - 1];
            thv0rel = thv0bot[krel];
        } else {
            krel = klcl;
            prel = plcl;
            exprel = exlcl;
            thv0rel = thv0lcl;
        }
        {
            double wcrit = sqrt(2.0 * cin * rbuoy);
            // compute_zwshcu computes rho0inv first and lowers wcrit by the large-scale ascent at
            // the PBL top (zwshcu.F90:2277, 2295-2303); the same value of rho0inv for both schemes
            double rho0inv = ps0[kinv - 1] / (r * thv0top[kinv - 1] * exns0[kinv - 1]);
            double sigmaw = sqrt(rkfre * tkeavg + epsvarw);
            if constexpr (ZW) {
                if (c.zw_lf) {
                    const double tmp1 = MN(MX(-GL(omega, kinv - 1), 0.0), 3.0);
                    wcrit = wcrit - tmp1 / rho0inv / 9.8;
                    wcrit = MX(wcrit, 0.0);
                }
                wcrit = wcrit * c.zw_fwcrit;
            }
            double mu = wcrit / sigmaw / 1.4142;
            if (mu >= 3.0) {
                id_exit = true;
                stop = true;
            break;
            }
            cbmf = (rho0inv * sigmaw / 2.5066) * uw_exp(-(mu * mu));
            double cbmflimit = 0.9 * dp0[kinv - 1] / g / dt;
            double mumin0 = 0.0;
            if (cbmf > cbmflimit) mumin0 = sqrt(-uw_log(2.5066 * cbmflimit / rho0inv / sigmaw));
            mu = MX(MX(mu, mumin0), mumin1);
            double mulcl = sqrt(2.0 * cinlcl * rbuoy) / 1.4142 / sigmaw;
            double ta = uw_exp(-(mu * mu)) / 2.5066, te = uw_erfc(mu);
            double mulclstar = sqrt(MX(0.0, 2.0 * (ta * ta) * (1.0 / (te * te) - 0.25 / (rmaxfrac * rmaxfrac))));
            if (mulcl > 1.e-8 && mulcl > mulclstar) {
                double mumin2 = compute_mumin2(mulcl, rmaxfrac, mu);
                if (mu > mumin2) errbits |= UW_ERRBIT_MU;
                mu = MX(mu, mumin2);
                if (mu == mumin2) lflags |= UW_L_UFRC;
            }
            if (mu == mumin0) lflags |= UW_L_CBMF;
            if (mu == mumin1) lflags |= UW_L_UFRC;
            cbmf = (rho0inv * sigmaw / 2.5066) * uw_exp(-(mu * mu));
            double winv = sigmaw * (2.0 / 2.5066) * uw_exp(-(mu * mu)) / uw_erfc(mu);
            wtw = winv * winv - 2.0 * cinlcl * rbuoy;
            if (wtw <= 0.0) {
                xflags |= UW_X_WTW;
                id_exit = true;
                stop = true;
            break;
            }
            wlcl = sqrt(wtw);
            ufrclcl = cbmf / wlcl / rho0inv;
            if (ufrclcl <= 0.0001) {
                xflags |= UW_X_UFRC;
                id_exit = true;
                stop = true;
            break;
            }
            ufrc[krel - 1] = ufrclcl;
#pragma unroll 1
            for (int k = 0; k <= mkx; k++) {
                const bool sub = k >= kinv - 1 && k <= krel - 1;
                umf[k] = sub ? cbmf : 0.0;
                wu[k] = sub ? winv : 0.0;
            }
            fer[krel] = 0.0;   // read at kpen = krel when no level is left for the updraft
        }
        } while (0);
        if (MODE == UW_MODE_TRIGGER) {
            // the column convects past the closure: hand it to the worklist pass
            if (!stop) {
                cand = true;
                stop = true;
            }
        }
        UW_SYNC();
        if (MODE != UW_MODE_TRIGGER) {   // uniform
#if !UW_TAPE_ORDER
        // Condensate of the final updraft at the release level, at the interfaces above it (qltop, qitop)
        // and at the cumulus top; id_top: the adjustment at the top did not close.  The tendencies and
        // the in-cloud diagnostics need it again; the Fortran repeats the conden calls there, with the
        // same arguments.
        double ql_rel = 0.0, qi_rel = 0.0, ql_top = 0.0, qi_top = 0.0;
        bool id_top = false;
#endif
        // updraft at the release level (:2205-2236)
        if (!stop) do {
        emf[krel - 1] = 0.0;
        umf[krel - 1] = cbmf;
        wu[krel - 1] = wlcl;
        thlu[krel - 1] = thlsrc;
        qtu[krel - 1] = qtsrc;
        if (CONDEN(prel, exprel, thlsrc, qtsrc, thj, qvj, qlj, qij, rvj, tbl)) {
            xflags |= UW_X_CONDEN;
            id_exit = true;
            stop = true;
            break;
        }
        thvu[krel - 1] = thj * (1.0 + zvir * qvj - qlj - qij);
#if !UW_TAPE_ORDER
        ql_rel = qlj;
        qi_rel = qij;
#endif
        {
            double uplus = 0.0, vplus = 0.0;
            if (krel == kinv) {
                uplus = PGFc * ssu0[kinv] * (prel - ps0[kinv - 1]);
                vplus = PGFc * ssv0[kinv] * (prel - ps0[kinv - 1]);
            } else {
#pragma unroll 1
                for (int k = 0; k <= mkx; k++) {
                    if (k < kinv || k > MX(krel - 1, kinv)) continue;
                    uplus = uplus + PGFc * ssu0[k] * (ps0[k] - ps0[k - 1]);
                    vplus = vplus + PGFc * ssv0[k] * (ps0[k] - ps0[k - 1]);
                }
                uplus = uplus + PGFc * ssu0[krel] * (prel - ps0[krel - 1]);
                vplus = vplus + PGFc * ssv0[krel] * (prel - ps0[krel - 1]);
            }
            uu[krel - 1] = usrc + uplus;
            vu[krel - 1] = vsrc + vplus;
        }
#pragma unroll 1
        for (int m = 0; m < ncnst; m++) tru[m][krel - 1] = trsrc[m];
        } while (0);
        UW_SYNC();

        {
#if !UW_TAPE_ORDER
            int kenv = krel - 1;   // the environment at the midpoints of layers krel .. kenv is known
#endif
            double scaleh = tscaleh;
            if (tscaleh < 0.0) scaleh = 1000.0;
            // ---- buoyancy-sorting updraft, iter_scaleh loop (:2306-2952) ----------------------
#pragma unroll 1
            for (int iter_scaleh = 1; iter_scaleh <= 3; iter_scaleh++) {   // uniform
                double pe = 0.0, dpe = 0.0, exne = 1.0, thvebot = 0.0, thle = 0.0, qte = 0.0, ue = 0.0, ve = 0.0;
                const bool last = UW_TAPE_ORDER || iter_scaleh == 3;
#if !UW_TAPE_ORDER
                // The first two passes only find the scale height: the winds and tracers of the updraft feed
                // nothing back into it, and of the level profiles only wu (an output at every level) and
                // fer outlive the pass, so the last pass alone computes and stores the rest.  (The
                // per-level diagnostics also show what an earlier, deeper pass left above the cloud top;
                // they hold no tracers.)
                const bool full = last || A.diag_level != nullptr;
                // the updraft at the level below
                double thlu_b = 0.0, qtu_b = 0.0, thvu_b = 0.0, umf_b = 0.0;
#endif
                if (!stop) {
                    kbup = krel;
                    kpen = krel;
                    wtw = wlcl * wlcl;
                    pe = 0.5 * (prel + ps0[krel]);
                    dpe = prel - ps0[krel];
                    exne = exnf(pe);
                    thvebot = thv0rel;
                    thle = thl0[krel] + ssthl0[krel] * (pe - p0[krel]);
                    qte = qt0[krel] + ssqt0[krel] * (pe - p0[krel]);
#if !UW_TAPE_ORDER
                    thlu_b = thlu[krel - 1];
                    qtu_b = qtu[krel - 1];
                    thvu_b = thvu[krel - 1];
                    umf_b = umf[krel - 1];
                    if (full) {   // uniform
#endif
                    ue = GL(u0, krel) + ssu0[krel] * (pe - p0[krel]);
                    ve = GL(v0, krel) + ssv0[krel] * (pe - p0[krel]);
#if !UW_TAPE_ORDER
                    }
#endif
#pragma unroll 1
                    for (int m = 0; last && m < ncnst; m++) tre[m] = GT(m + 1, krel) + sstr0[m][krel] * (pe - p0[krel]);
                }

#if UW_TAPE_ORDER
                // levels k = krel .. mkx-1, taken by every lane as k = krel + j
                bool ldone = stop;
#pragma unroll 1
                for (int j = 0; j <= mkx - 2; j++) {   // uniform
                    const int k = krel + j;
                    if (k > mkx - 1) ldone = true;
                    if (!ldone) do {
                    const int km1 = k - 1;
                    double thlue = thlu[km1];
                    double qtue = qtu[km1];
                    double wue = wu[km1];
                    wtwb = wtw;
                    bool xdone = false;
                    // environment at the layer midpoint: the same in both iter_xc passes, so the
                    // second pass reuses the first one's conden and qsat results (same bits)
                    double thv0j = 0.0, excess0 = 0.0;
#pragma unroll 1
                    for (int iter_xc = 1; iter_xc <= 2; iter_xc++) {
                        if (!xdone && !stop) do {
                        wtw = wu[km1] * wu[km1];
                        if (iter_xc == 1) {
                            if (CONDEN(pe, exne, thle, qte, thj, qvj, qlj, qij, rvj, tbl)) {
                                xflags |= UW_X_CONDEN;
                                id_exit = true;
                                stop = true;
                                break;
                            }
                            thv0j = thj * (1.0 + zvir * qvj - qlj - qij);
                            excess0 = qte - qsat_qs(thle * exne, pe, tbl);
                        }
                        rho0j = pe / (r * thv0j * exne);
                        if (CONDEN(pe, exne, thlue, qtue, thj, qvj, qlj, qij, rvj, tbl)) {
                            xflags |= UW_X_CONDEN;
                            id_exit = true;
                            stop = true;
            break;
                        }
                        // condensate above criqc leaves the updraft; without it the Fortran's
                        // second conden call repeats the first one's arguments and results
                        if ((qlj + qij) > criqc) {
                            double exql = ((qlj + qij) - criqc) * qlj / (qlj + qij);
                            double exqi = ((qlj + qij) - criqc) * qij / (qlj + qij);
                            qtue = qtue - exql - exqi;
                            thlue = thlue + (xlv / cp / exne) * exql + (xls / cp / exne) * exqi;
                            if (CONDEN(pe, exne, thlue, qtue, thj, qvj, qlj, qij, rvj, tbl)) {
                                xflags |= UW_X_CONDEN;
                                id_exit = true;
                                stop = true;
                                break;
                            }
                        }
                        double thvj = thj * (1.0 + zvir * qvj - qlj - qij);
                        double excessu = qtue - qsat_qs(thlue * exne, pe, tbl);
                        double cridis = rle * scaleh;
                        double xc;
                        if ((excessu <= 0.0 && excess0 <= 0.0) || (excessu >= 0.0 && excess0 >= 0.0)) {
                            xc = MN(1.0, MX(0.0, 1.0 - 2.0 * rbuoy * g * cridis / (wue * wue) * (1.0 - thvj / thv0j)));
                        } else {
                            double xsat = excessu / (excessu - excess0);
                            double thlxsat = thlue + xsat * (thle - thlue);
                            double qtxsat = qtue + xsat * (qte - qtue);
                            if (CONDEN(pe, exne, thlxsat, qtxsat, thj, qvj, qlj, qij, rvj, tbl)) {
                                xflags |= UW_X_CONDEN;
                                id_exit = true;
                                stop = true;
            break;
                            }
                            double thvxsat = thj * (1.0 + zvir * qvj - qlj - qij);
                            double x_cu = 0.0, x_en = 0.0;
#pragma unroll 1
                            for (int kk = 1; kk <= 2; kk++) {
                                double thv_x0, thv_x1;
                                if (kk == 1) {
                                    thv_x0 = thvj;
                                    thv_x1 = (1.0 - 1.0 / xsat) * thvj + (1.0 / xsat) * thvxsat;
                                } else {
                                    thv_x1 = thv0j;
                                    thv_x0 = (xsat / (xsat - 1.0)) * thv0j + (1.0 / (1.0 - xsat)) * thvxsat;
                                }
                                double aquad = wue * wue;
                                double bquad = 2.0 * rbuoy * g * cridis * (thv_x1 - thv_x0) / thv0j - 2.0 * (wue * wue);
                                double cquad = 2.0 * rbuoy * g * cridis * (thv_x0 - thv0j) / thv0j + (wue * wue);
                                if (kk == 1) {
                                    if ((bquad * bquad - 4.0 * aquad * cquad) >= 0.0) {
                                        roots(aquad, bquad, cquad, xs1, xs2);
                                        x_cu = MN(1.0, MX(0.0, MN(xsat, MN(xs1, xs2))));
                                    } else {
                                        x_cu = xsat;
                                    }
                                } else {
                                    if ((bquad * bquad - 4.0 * aquad * cquad) >= 0.0) {
                                        roots(aquad, bquad, cquad, xs1, xs2);
                                        x_en = MN(1.0, MX(0.0, MX(xsat, MN(xs1, xs2))));
                                    } else {
                                        x_en = 1.0;
                                    }
                                }
                            }
                            if (x_cu == xsat) xc = MX(x_cu, x_en);
                            else xc = x_cu;
                        }
                        double ee2 = xc * xc;
                        double ud2 = 1.0 - 2.0 * xc + xc * xc;
                        rei[k] = (0.5 * rkm / GL(z0, k) / g / rho0j);
                        if (xc > 0.5) rei[k] = MN(rei[k], 0.9 * uw_log(dp0[k] / g / dt / umf[km1] + 1.0) / dpe / (2.0 * xc - 1.0));
                        fer[k] = rei[k] * ee2;
                        fdr[k] = rei[k] * ud2;
                        // compute_zwshcu's entrainment option (zwshcu.F90:2818-2844)
                        if (ZW && c.zw_ent) {
                            bogbot = rbuoy * (thvu[km1] / thvebot - 1.0) * g;
                            fer[k] = c.zw_ent0 * bogbot / MX(wue * wue, 1.0e-4);
                            double fer_min = 0.0;
                            if (bogbot > 1.e-4) fer_min = 1.e-4;
                            fer[k] = MN(MX(fer[k], fer_min), 3.0e-2);
                        }
                        umf[k] = umf[km1] * uw_exp(dpe * (fer[k] - fdr[k]));
                        emf[k] = 0.0;
                        if (fer[k] * dpe < 1.e-4) {
                            thlu[k] = thlu[km1] + (thle + ssthl0[k] * dpe / 2.0 - thlu[km1]) * fer[k] * dpe;
                            qtu[k] = qtu[km1] + (qte + ssqt0[k] * dpe / 2.0 - qtu[km1]) * fer[k] * dpe;
                            uu[k] = uu[km1] + (ue + ssu0[k] * dpe / 2.0 - uu[km1]) * fer[k] * dpe - PGFc * ssu0[k] * dpe;
                            vu[k] = vu[km1] + (ve + ssv0[k] * dpe / 2.0 - vu[km1]) * fer[k] * dpe - PGFc * ssv0[k] * dpe;
#pragma unroll 1
                            for (int m = 0; m < ncnst; m++)
                                tru[m][k] = tru[m][km1] + (tre[m] + sstr0[m][k] * dpe / 2.0 - tru[m][km1]) * fer[k] * dpe;
                        } else {
                            const double ef = uw_exp(-fer[k] * dpe);
                            thlu[k] = (thle + ssthl0[k] / fer[k] - ssthl0[k] * dpe / 2.0) -
                                      (thle + ssthl0[k] * dpe / 2.0 - thlu[km1] + ssthl0[k] / fer[k]) * ef;
                            qtu[k] = (qte + ssqt0[k] / fer[k] - ssqt0[k] * dpe / 2.0) -
                                     (qte + ssqt0[k] * dpe / 2.0 - qtu[km1] + ssqt0[k] / fer[k]) * ef;
                            uu[k] = (ue + (1.0 - PGFc) * ssu0[k] / fer[k] - ssu0[k] * dpe / 2.0) -
                                    (ue + ssu0[k] * dpe / 2.0 - uu[km1] + (1.0 - PGFc) * ssu0[k] / fer[k]) * ef;
                            vu[k] = (ve + (1.0 - PGFc) * ssv0[k] / fer[k] - ssv0[k] * dpe / 2.0) -
                                    (ve + ssv0[k] * dpe / 2.0 - vu[km1] + (1.0 - PGFc) * ssv0[k] / fer[k]) * ef;
#pragma unroll 1
                            for (int m = 0; m < ncnst; m++)
                                tru[m][k] = (tre[m] + sstr0[m][k] / fer[k] - sstr0[m][k] * dpe / 2.0) -
                                            (tre[m] + sstr0[m][k] * dpe / 2.0 - tru[m][km1] + sstr0[m][k] / fer[k]) * ef;
                        }
                        if (CONDEN(ps0[k], exns0[k], thlu[k], qtu[k], thj, qvj, qlj, qij, rvj, tbl)) {
                            xflags |= UW_X_CONDEN;
                            id_exit = true;
                            stop = true;
            break;
                        }
                        if ((qlj + qij) > criqc) {
                            double exql = ((qlj + qij) - criqc) * qlj / (qlj + qij);
                            double exqi = ((qlj + qij) - criqc) * qij / (qlj + qij);
                            qtu[k] = qtu[k] - exql - exqi;
                            thlu[k] = thlu[k] + (xlv / cp / exns0[k]) * exql + (xls / cp / exns0[k]) * exqi;
                            dwten[k] = exql;
                            diten[k] = exqi;
                            if (CONDEN(ps0[k], exns0[k], thlu[k], qtu[k], thj, qvj, qlj, qij, rvj, tbl)) {
                                xflags |= UW_X_CONDEN;
                                id_exit = true;
                                stop = true;
                                break;
                            }
                        } else {
                            // nothing removed: the Fortran's second conden call repeats the first
                            dwten[k] = 0.0;
                            diten[k] = 0.0;
                        }
                        thvu[k] = thj * (1.0 + zvir * qvj - qlj - qij);
                        bogbot = rbuoy * (thvu[km1] / thvebot - 1.0);
                        bogtop = rbuoy * (thvu[k] / thv0top[k] - 1.0);
                        double delbog = bogtop - bogbot;
                        drage = fer[k] * (1.0 + rdrag);
                        double expfac = uw_exp(-2.0 * drage * dpe);
                        wtwb = wtw;
                        if (drage * dpe > 1.e-3)
                            wtw = wtw * expfac + (delbog + (1.0 - expfac) * (bogbot + delbog / (-2.0 * drage * dpe))) / (rho0j * drage);
                        else
                            wtw = wtw + dpe * (bogbot + bogtop) / rho0j;
                        if (wtw > 0.0) {
                            thlue = 0.5 * (thlu[km1] + thlu[k]);
                            qtue = 0.5 * (qtu[km1] + qtu[k]);
                            wue = 0.5 * sqrt(MX(wtwb + wtw, 0.0));
                        } else {
                            xdone = true;   // go to 111
                        }
                        } while (0);
                    }
                    if (stop) break;
                    // (label 111, :2726-2793)
                    if (umf[k] == 0.0) wtw = -1.0;
                    if (bogtop > 0.0 && wtw > 0.0) kbup = k;
                    if (wtw <= 0.0) {
                        kpen = k;
                        ldone = true;
                        break;   // go to 45
                    }
                    wu[k] = sqrt(wtw);
                    if (wu[k] > 100.0) {
                        xflags |= UW_X_WU;
                        id_exit = true;
                        stop = true;
            break;
                    }
                    {
                        double rhos0j = ps0[k] / (r * 0.5 * (thv0bot[k + 1] + thv0top[k]) * exns0[k]);
                        ufrc[k] = umf[k] / (rhos0j * wu[k]);
                        if (ufrc[k] > rmaxfrac) {
                            lflags |= UW_L_UFRC;
                            ufrc[k] = rmaxfrac;
                            umf[k] = rmaxfrac * rhos0j * wu[k];
                            fdr[k] = fer[k] - uw_log(umf[k] / umf[km1]) / dpe;
                        }
                    }
                    pe = p0[k + 1];
                    dpe = dp0[k + 1];
                    exne = exn0[k + 1];
                    thvebot = thv0bot[k + 1];
                    thle = thl0[k + 1];
                    qte = qt0[k + 1];
                    ue = GL(u0, k + 1);
                    ve = GL(v0, k + 1);
#pragma unroll 1
                    for (int m = 0; m < ncnst; m++) tre[m] = GT(m + 1, k + 1);
                    } while (0);
                    if (stop) ldone = true;
                    UW_SYNC();
                }
#else
                // levels k = krel .. mkx-1, taken by every lane as k = krel + j
                bool ldone = stop;
#pragma unroll 1
                for (int j = 0; j <= mkx - 2; j++) {   // uniform
                    const int k = krel + j;
                    if (k > mkx - 1) ldone = true;
                    if (!ldone) do {
                    const double wu_b = wu[k - 1];   // (carried like the others, the FMA-contracted modes would round
                                                     // wu_b * wu_b with what follows it)
                    double thlue = thlu_b;
                    double qtue = qtu_b;
                    double wue = wu_b;
                    wtwb = wtw;
                    bool xdone = false;
                    // environment at the layer midpoint: the same in both iter_xc passes and in every
                    // updraft of this iteration, so the first one to reach the level computes it
                    double thv0j = 0.0, excess0 = 0.0, reib = 0.0;
                    if (k > kenv) {
                        if (CONDEN(pe, exne, thle, qte, thj, qvj, qlj, qij, rvj, tbl)) {
                            xflags |= UW_X_CONDEN;
                            id_exit = true;
                            stop = true;
                            break;
                        }
                        thv0j = thj * (1.0 + zvir * qvj - qlj - qij);
                        excess0 = qte - UW_QSAT_OF_CONDEN(thle * exne, pe);
                        rho0j = pe / (r * thv0j * exne);
                        reib = (0.5 * rkm / GL(z0, k) / g / rho0j);
                        env_thv[k] = thv0j;
                        env_exc[k] = excess0;
                        env_rho[k] = rho0j;
                        env_rei[k] = reib;
                        kenv = k;
                    } else {
                        thv0j = env_thv[k];
                        excess0 = env_exc[k];
                        rho0j = env_rho[k];
                        reib = env_rei[k];
                    }
                    double lgf = 0.0;        // the factor of the entrainment limit below, once it is needed
                    bool lgf_set = false;
                    double thlu_k = 0.0, qtu_k = 0.0, thvu_k = 0.0, fer_k = 0.0, fdr_k = 0.0, rei_k = 0.0, ef_k = 0.0,
                           dmf_k = 0.0, dw_k = 0.0, di_k = 0.0;
                    const double cridis = rle * scaleh;
#pragma unroll 1
                    for (int iter_xc = 1; iter_xc <= 2; iter_xc++) {
                        if (!xdone && !stop) do {
                        wtw = wu_b * wu_b;
                        if (CONDEN(pe, exne, thlue, qtue, thj, qvj, qlj, qij, rvj, tbl)) {
                            xflags |= UW_X_CONDEN;
                            id_exit = true;
                            stop = true;
                            break;
                        }
                        // condensate above criqc leaves the updraft; without it the Fortran's
                        // second conden call repeats the first one's arguments and results
                        if ((qlj + qij) > criqc) {
                            double exql = ((qlj + qij) - criqc) * qlj / (qlj + qij);
                            double exqi = ((qlj + qij) - criqc) * qij / (qlj + qij);
                            qtue = qtue - exql - exqi;
                            thlue = thlue + (xlv / cp / exne) * exql + (xls / cp / exne) * exqi;
                            if (CONDEN(pe, exne, thlue, qtue, thj, qvj, qlj, qij, rvj, tbl)) {
                                xflags |= UW_X_CONDEN;
                                id_exit = true;
                                stop = true;
                                break;
                            }
                        }
                        double thvj = thj * (1.0 + zvir * qvj - qlj - qij);
                        double excessu = qtue - UW_QSAT_OF_CONDEN(thlue * exne, pe);
                        double xc;
                        if ((excessu <= 0.0 && excess0 <= 0.0) || (excessu >= 0.0 && excess0 >= 0.0)) {
                            xc = MN(1.0, MX(0.0, 1.0 - 2.0 * rbuoy * g * cridis / (wue * wue) * (1.0 - thvj / thv0j)));
                        } else {
                            double xsat = excessu / (excessu - excess0);
                            double thlxsat = thlue + xsat * (thle - thlue);
                            double qtxsat = qtue + xsat * (qte - qtue);
                            if (CONDEN(pe, exne, thlxsat, qtxsat, thj, qvj, qlj, qij, rvj, tbl)) {
                                xflags |= UW_X_CONDEN;
                                id_exit = true;
                                stop = true;
                                break;
                            }
                            double thvxsat = thj * (1.0 + zvir * qvj - qlj - qij);
                            double x_cu = 0.0, x_en = 0.0;
#pragma unroll 1
                            for (int kk = 1; kk <= 2; kk++) {
                                double thv_x0, thv_x1;
                                if (kk == 1) {
                                    thv_x0 = thvj;
                                    thv_x1 = (1.0 - 1.0 / xsat) * thvj + (1.0 / xsat) * thvxsat;
                                } else {
                                    thv_x1 = thv0j;
                                    thv_x0 = (xsat / (xsat - 1.0)) * thv0j + (1.0 / (1.0 - xsat)) * thvxsat;
                                }
                                double aquad = wue * wue;
                                double bquad = 2.0 * rbuoy * g * cridis * (thv_x1 - thv_x0) / thv0j - 2.0 * (wue * wue);
                                double cquad = 2.0 * rbuoy * g * cridis * (thv_x0 - thv0j) / thv0j + (wue * wue);
                                if (kk == 1) {
                                    if ((bquad * bquad - 4.0 * aquad * cquad) >= 0.0) {
                                        roots(aquad, bquad, cquad, xs1, xs2);
                                        x_cu = MN(1.0, MX(0.0, MN(xsat, MN(xs1, xs2))));
                                    } else {
                                        x_cu = xsat;
                                    }
                                } else {
                                    if ((bquad * bquad - 4.0 * aquad * cquad) >= 0.0) {
                                        roots(aquad, bquad, cquad, xs1, xs2);
                                        x_en = MN(1.0, MX(0.0, MX(xsat, MN(xs1, xs2))));
                                    } else {
                                        x_en = 1.0;
                                    }
                                }
                            }
                            if (x_cu == xsat) xc = MX(x_cu, x_en);
                            else xc = x_cu;
                        }
                        double ee2 = xc * xc;
                        double ud2 = 1.0 - 2.0 * xc + xc * xc;
                        rei_k = reib;
                        if (xc > 0.5) {
                            if (!lgf_set) {
                                lgf = 0.9 * uw_log(dp0[k] / g / dt / umf_b + 1.0) / dpe;
                                lgf_set = true;
                            }
                            rei_k = MN(rei_k, lgf / (2.0 * xc - 1.0));
                        }
                        fer_k = rei_k * ee2;
                        fdr_k = rei_k * ud2;
                        // compute_zwshcu's entrainment option (zwshcu.F90:2818-2844)
                        if (ZW && c.zw_ent) {
                            bogbot = rbuoy * (thvu_b / thvebot - 1.0) * g;
                            fer_k = c.zw_ent0 * bogbot / MX(wue * wue, 1.0e-4);
                            double fer_min = 0.0;
                            if (bogbot > 1.e-4) fer_min = 1.e-4;
                            fer_k = MN(MX(fer_k, fer_min), 3.0e-2);
                        }
                        dmf_k = dpe * (fer_k - fdr_k);
                        if (fer_k * dpe < 1.e-4) {
                            thlu_k = thlu_b + (thle + ssthl0[k] * dpe / 2.0 - thlu_b) * fer_k * dpe;
                            qtu_k = qtu_b + (qte + ssqt0[k] * dpe / 2.0 - qtu_b) * fer_k * dpe;
                        } else {
                            ef_k = uw_exp(-fer_k * dpe);
                            thlu_k = (thle + ssthl0[k] / fer_k - ssthl0[k] * dpe / 2.0) -
                                     (thle + ssthl0[k] * dpe / 2.0 - thlu_b + ssthl0[k] / fer_k) * ef_k;
                            qtu_k = (qte + ssqt0[k] / fer_k - ssqt0[k] * dpe / 2.0) -
                                    (qte + ssqt0[k] * dpe / 2.0 - qtu_b + ssqt0[k] / fer_k) * ef_k;
                        }
                        if (CONDEN(ps0[k], exns0[k], thlu_k, qtu_k, thj, qvj, qlj, qij, rvj, tbl)) {
                            xflags |= UW_X_CONDEN;
                            id_exit = true;
                            stop = true;
                            break;
                        }
                        if ((qlj + qij) > criqc) {
                            double exql = ((qlj + qij) - criqc) * qlj / (qlj + qij);
                            double exqi = ((qlj + qij) - criqc) * qij / (qlj + qij);
                            qtu_k = qtu_k - exql - exqi;
                            thlu_k = thlu_k + (xlv / cp / exns0[k]) * exql + (xls / cp / exns0[k]) * exqi;
                            dw_k = exql;
                            di_k = exqi;
                            if (CONDEN(ps0[k], exns0[k], thlu_k, qtu_k, thj, qvj, qlj, qij, rvj, tbl)) {
                                xflags |= UW_X_CONDEN;
                                id_exit = true;
                                stop = true;
                                break;
                            }
                        } else {
                            // nothing removed: the Fortran's second conden call repeats the first
                            dw_k = 0.0;
                            di_k = 0.0;
                        }
                        thvu_k = thj * (1.0 + zvir * qvj - qlj - qij);
                        bogbot = rbuoy * (thvu_b / thvebot - 1.0);
                        bogtop = rbuoy * (thvu_k / thv0top[k] - 1.0);
                        double delbog = bogtop - bogbot;
                        drage = fer_k * (1.0 + rdrag);
                        double expfac = uw_exp(-2.0 * drage * dpe);
                        wtwb = wtw;
                        if (drage * dpe > 1.e-3)
                            wtw = wtw * expfac + (delbog + (1.0 - expfac) * (bogbot + delbog / (-2.0 * drage * dpe))) / (rho0j * drage);
                        else
                            wtw = wtw + dpe * (bogbot + bogtop) / rho0j;
                        if (wtw > 0.0) {
                            thlue = 0.5 * (thlu_b + thlu_k);
                            qtue = 0.5 * (qtu_b + qtu_k);
                            wue = 0.5 * sqrt(MX(wtwb + wtw, 0.0));
                        } else {
                            xdone = true;   // go to 111
                        }
                        } while (0);
                    }
                    if (stop) break;
                    fer[k] = fer_k;
                    // the mass flux and, in the last pass, the level's profiles with the final fer and fdr
                    // (the Fortran evaluates them in each iter_xc pass)
                    double umf_k = umf_b * uw_exp(dmf_k);
                    if (full) {
                        const int km1 = k - 1;
                        rei[k] = rei_k;
                        thlu[k] = thlu_k;
                        qtu[k] = qtu_k;
                        thvu[k] = thvu_k;
                        dwten[k] = dw_k;
                        diten[k] = di_k;
                        qltop[k] = qlj;
                        qitop[k] = qij;
                        if (fer_k * dpe < 1.e-4) {
                            uu[k] = uu[km1] + (ue + ssu0[k] * dpe / 2.0 - uu[km1]) * fer_k * dpe - PGFc * ssu0[k] * dpe;
                            vu[k] = vu[km1] + (ve + ssv0[k] * dpe / 2.0 - vu[km1]) * fer_k * dpe - PGFc * ssv0[k] * dpe;
#pragma unroll 1
                            for (int m = 0; last && m < ncnst; m++)
                                tru[m][k] = tru[m][km1] + (tre[m] + sstr0[m][k] * dpe / 2.0 - tru[m][km1]) * fer_k * dpe;
                        } else {
                            uu[k] = (ue + (1.0 - PGFc) * ssu0[k] / fer_k - ssu0[k] * dpe / 2.0) -
                                    (ue + ssu0[k] * dpe / 2.0 - uu[km1] + (1.0 - PGFc) * ssu0[k] / fer_k) * ef_k;
                            vu[k] = (ve + (1.0 - PGFc) * ssv0[k] / fer_k - ssv0[k] * dpe / 2.0) -
                                    (ve + ssv0[k] * dpe / 2.0 - vu[km1] + (1.0 - PGFc) * ssv0[k] / fer_k) * ef_k;
#pragma unroll 1
                            for (int m = 0; last && m < ncnst; m++)
                                tru[m][k] = (tre[m] + sstr0[m][k] / fer_k - sstr0[m][k] * dpe / 2.0) -
                                            (tre[m] + sstr0[m][k] * dpe / 2.0 - tru[m][km1] + sstr0[m][k] / fer_k) * ef_k;
                        }
                    }
                    // (label 111, :2726-2793)
                    if (umf_k == 0.0) wtw = -1.0;
                    if (bogtop > 0.0 && wtw > 0.0) kbup = k;
                    if (wtw <= 0.0) {
                        kpen = k;
                        ldone = true;
                        if (full) {
                            umf[k] = umf_k;
                            fdr[k] = fdr_k;
                        }
                        break;   // go to 45
                    }
                    wu[k] = sqrt(wtw);
                    if (wu[k] > 100.0) {
                        xflags |= UW_X_WU;
                        id_exit = true;
                        stop = true;
                        break;
                    }
                    {
                        double rhos0j = ps0[k] / (r * 0.5 * (thv0bot[k + 1] + thv0top[k]) * exns0[k]);
                        double ufrc_k = umf_k / (rhos0j * wu[k]);
                        if (ufrc_k > rmaxfrac) {
                            lflags |= UW_L_UFRC;
                            ufrc_k = rmaxfrac;
                            umf_k = rmaxfrac * rhos0j * wu[k];
                            fdr_k = fer_k - uw_log(umf_k / umf_b) / dpe;
                        }
                        if (full) {
                            ufrc[k] = ufrc_k;
                            umf[k] = umf_k;
                            fdr[k] = fdr_k;
                        }
                    }
                    thlu_b = thlu_k;
                    qtu_b = qtu_k;
                    thvu_b = thvu_k;
                    umf_b = umf_k;
                    pe = p0[k + 1];
                    dpe = dp0[k + 1];
                    exne = exn0[k + 1];
                    thvebot = thv0bot[k + 1];
                    thle = thl0[k + 1];
                    qte = qt0[k + 1];
                    if (full) {
                        ue = GL(u0, k + 1);
                        ve = GL(v0, k + 1);
#pragma unroll 1
                        for (int m = 0; last && m < ncnst; m++) tre[m] = GT(m + 1, k + 1);
                    }
                    } while (0);
                    if (stop) ldone = true;
                    UW_SYNC();
                }
#endif
                UW_SYNC();
                // (label 45) penetration depth (:2884-2907)
                if (!stop) do {
#if UW_TAPE_ORDER
                const double thlu_b = thlu[kpen - 1], qtu_b = qtu[kpen - 1];
#else
                // the updraft at kpen - 1 (the release level's when no level stopped it: kpen = krel)
                if (kpen == krel) {
                    thlu_b = thlu[krel - 1];
                    qtu_b = qtu[krel - 1];
                }
#endif
                if (drage == 0.0) {
                    double aquad = (bogtop - bogbot) / (ps0[kpen] - ps0[kpen - 1]);
                    double bquad = 2.0 * bogbot;
                    double cquad = -(wu[kpen - 1] * wu[kpen - 1]) * rho0j;
                    int status = roots(aquad, bquad, cquad, xc1, xc2);
                    if (status == 0) {
                        if (xc1 <= 0.0 && xc2 <= 0.0) {
                            ppen = MX(xc1, xc2);
                            ppen = MN(0.0, MX(-dp0[kpen], ppen));
                        } else if (xc1 > 0.0 && xc2 > 0.0) {
                            ppen = -dp0[kpen];
                        } else {
                            ppen = MN(xc1, xc2);
                            ppen = MN(0.0, MX(-dp0[kpen], ppen));
                        }
                    } else {
                        ppen = -dp0[kpen];
                    }
                } else {
                    ppen = compute_ppen(wtwb, drage, bogbot, bogtop, rho0j, dp0[kpen]);
                }
                if (ppen == -dp0[kpen] || ppen == 0.0) lflags |= UW_L_PPEN;
                // condensate at the cumulus top (:2917-2942)
                if (fer[kpen] * (-ppen) < 1.e-4) {
                    thlu_top = thlu_b + (thl0[kpen] + ssthl0[kpen] * (-ppen) / 2.0 - thlu_b) * fer[kpen] * (-ppen);
                    qtu_top = qtu_b + (qt0[kpen] + ssqt0[kpen] * (-ppen) / 2.0 - qtu_b) * fer[kpen] * (-ppen);
                } else {
                    const double ef = uw_exp(-fer[kpen] * (-ppen));
                    thlu_top = (thl0[kpen] + ssthl0[kpen] / fer[kpen] - ssthl0[kpen] * (-ppen) / 2.0) -
                               (thl0[kpen] + ssthl0[kpen] * (-ppen) / 2.0 - thlu_b + ssthl0[kpen] / fer[kpen]) * ef;
                    qtu_top = (qt0[kpen] + ssqt0[kpen] / fer[kpen] - ssqt0[kpen] * (-ppen) / 2.0) -
                              (qt0[kpen] + ssqt0[kpen] * (-ppen) / 2.0 - qtu_b + ssqt0[kpen] / fer[kpen]) * ef;
                }
                exntop = uw_pow((ps0[kpen - 1] + ppen) / p00, rovcp);
                if (CONDEN(ps0[kpen - 1] + ppen, exntop, thlu_top, qtu_top, thj, qvj, qlj, qij, rvj, tbl)) {
                    xflags |= UW_X_CONDEN;
                    id_exit = true;
                    stop = true;
            break;
                }
#if UW_TAPE_ORDER
                if ((qlj + qij) > criqc) {
                    dwten[kpen] = ((qlj + qij) - criqc) * qlj / (qlj + qij);
                    diten[kpen] = ((qlj + qij) - criqc) * qij / (qlj + qij);
                    qtu_top = qtu_top - dwten[kpen] - diten[kpen];
                    thlu_top = thlu_top + (xlv / cp / exntop) * dwten[kpen] + (xls / cp / exntop) * diten[kpen];
                } else {
                    dwten[kpen] = 0.0;
                    diten[kpen] = 0.0;
                }
#else
                if (full) {
                    if ((qlj + qij) > criqc) {
                        dwten[kpen] = ((qlj + qij) - criqc) * qlj / (qlj + qij);
                        diten[kpen] = ((qlj + qij) - criqc) * qij / (qlj + qij);
                        qtu_top = qtu_top - dwten[kpen] - diten[kpen];
                        thlu_top = thlu_top + (xlv / cp / exntop) * dwten[kpen] + (xls / cp / exntop) * diten[kpen];
                        id_top = CONDEN(ps0[kpen - 1] + ppen, exntop, thlu_top, qtu_top, thj, qvj, qlj, qij, rvj, tbl) != 0;
                    } else {
                        dwten[kpen] = 0.0;
                        diten[kpen] = 0.0;
                        id_top = false;
                    }
                    ql_top = qlj;
                    qi_top = qij;
                }
#endif
                {
                    double rhos0j = ps0[kpen - 1] / (r * 0.5 * (thv0bot[kpen] + thv0top[kpen - 1]) * exns0[kpen - 1]);
                    cush = zs0[kpen - 1] - ppen / rhos0j / g;
                }
                scaleh = cush;
                } while (0);
                UW_SYNC();
            }
        }
        // forcedCu filter (:2964-2992)
        if (!stop) do {
        if (kbup == krel) {
            lflags |= UW_L_SHCU;
            xflags |= UW_X_CUFILTER;
            id_exit = true;
            stop = true;
            break;
        }
        lflags &= ~UW_L_SHCU;
#pragma unroll 1
        for (int k = kpen; k <= mkx; k++) umf[k] = 0.0;
        ufrc[kpen] = 0.0;
        if (A.diag_level) {
#pragma unroll 1
            for (int k = kpen + 1; k <= mkx; k++) {
                ufrc[k] = 0.0;
                dwten[k] = 0.0;
                diten[k] = 0.0;
                fer[k] = 0.0;
                fdr[k] = 0.0;
            }
        }
        // penetrative entrainment (:3055-3183)
        // (the *_emf profiles are read at kbup .. kpen - 1 only)
#pragma unroll 1
        for (int k = mkx; k >= 0; k--) {
            if (k > kpen - 1 || k < kbup) continue;
            double rhos0j = ps0[k] / (r * 0.5 * (thv0bot[k + 1] + thv0top[k]) * exns0[k]);
            if (k == kpen - 1) {
                if ((umf[k] * ppen * rei[kpen] * rpen) < -0.1 * rhos0j) lflags |= UW_L_EMF;
                if ((umf[k] * ppen * rei[kpen] * rpen) < -0.9 * dp0[kpen] / g / dt) lflags |= UW_L_EMF;
                emf[k] = MX(MX(umf[k] * ppen * rei[kpen] * rpen, -0.1 * rhos0j), -0.9 * dp0[kpen] / g / dt);
                thlu_emf[k] = thl0[kpen] + ssthl0[kpen] * (ps0[k] - p0[kpen]);
                qtu_emf[k] = qt0[kpen] + ssqt0[kpen] * (ps0[k] - p0[kpen]);
                uu_emf[k] = GL(u0, kpen) + ssu0[kpen] * (ps0[k] - p0[kpen]);
                vu_emf[k] = GL(v0, kpen) + ssv0[kpen] * (ps0[k] - p0[kpen]);
#pragma unroll 1
                for (int m = 0; m < ncnst; m++) tru_emf[m][k] = GT(m + 1, kpen) + sstr0[m][kpen] * (ps0[k] - p0[kpen]);
            } else {
                if ((emf[k + 1] - umf[k] * dp0[k + 1] * rei[k + 1] * rpen) < -0.1 * rhos0j) lflags |= UW_L_EMF;
                if ((emf[k + 1] - umf[k] * dp0[k + 1] * rei[k + 1] * rpen) < -0.9 * dp0[k + 1] / g / dt) lflags |= UW_L_EMF;
                emf[k] = MX(MX(emf[k + 1] - umf[k] * dp0[k + 1] * rei[k + 1] * rpen, -0.1 * rhos0j), -0.9 * dp0[k + 1] / g / dt);
                if (fabs(emf[k]) > fabs(emf[k + 1])) {
                    thlu_emf[k] = (thlu_emf[k + 1] * emf[k + 1] + thl0[k + 1] * (emf[k] - emf[k + 1])) / emf[k];
                    qtu_emf[k] = (qtu_emf[k + 1] * emf[k + 1] + qt0[k + 1] * (emf[k] - emf[k + 1])) / emf[k];
                    uu_emf[k] = (uu_emf[k + 1] * emf[k + 1] + GL(u0, k + 1) * (emf[k] - emf[k + 1])) / emf[k];
                    vu_emf[k] = (vu_emf[k + 1] * emf[k + 1] + GL(v0, k + 1) * (emf[k] - emf[k + 1])) / emf[k];
#pragma unroll 1
                    for (int m = 0; m < ncnst; m++)
                        tru_emf[m][k] = (tru_emf[m][k + 1] * emf[k + 1] + GT(m + 1, k + 1) * (emf[k] - emf[k + 1])) / emf[k];
                } else {
                    thlu_emf[k] = thl0[k + 1];
                    qtu_emf[k] = qt0[k + 1];
                    uu_emf[k] = GL(u0, k + 1);
                    vu_emf[k] = GL(v0, k + 1);
#pragma unroll 1
                    for (int m = 0; m < ncnst; m++) tru_emf[m][k] = GT(m + 1, k + 1);
                }
            }
        }
        // 1. PBL fluxes (:3255-3290)
        {
            double xsrc = qtsrc, xmean = qt0[kinv];
            double xtop = qt0[kinv + 1] + ssqt0[kinv + 1] * (ps0[kinv] - p0[kinv + 1]);
            double xbot = qt0[kinv - 1] + ssqt0[kinv - 1] * (ps0[kinv - 1] - p0[kinv - 1]);
            fluxbelowinv(cbmf, ps0, kinv, dt, xsrc, xmean, xtop, xbot, xflx);
#pragma unroll 1
            for (int k = 0; k <= mkx; k++) if (k <= kinv - 1) qtflx[k] = xflx[k];
            xsrc = thlsrc;
            xmean = thl0[kinv];
            xtop = thl0[kinv + 1] + ssthl0[kinv + 1] * (ps0[kinv] - p0[kinv + 1]);
            xbot = thl0[kinv - 1] + ssthl0[kinv - 1] * (ps0[kinv - 1] - p0[kinv - 1]);
            fluxbelowinv(cbmf, ps0, kinv, dt, xsrc, xmean, xtop, xbot, xflx);
#pragma unroll 1
            for (int k = 0; k <= mkx; k++) if (k <= kinv - 1) slflx[k] = cp * exns0[k] * xflx[k];
            xsrc = usrc;
            xmean = GL(u0, kinv);
            xtop = GL(u0, kinv + 1) + ssu0[kinv + 1] * (ps0[kinv] - p0[kinv + 1]);
            xbot = GL(u0, kinv - 1) + ssu0[kinv - 1] * (ps0[kinv - 1] - p0[kinv - 1]);
            fluxbelowinv(cbmf, ps0, kinv, dt, xsrc, xmean, xtop, xbot, xflx);
#pragma unroll 1
            for (int k = 0; k <= mkx; k++) if (k <= kinv - 1) uflx[k] = xflx[k];
            xsrc = vsrc;
            xmean = GL(v0, kinv);
            xtop = GL(v0, kinv + 1) + ssv0[kinv + 1] * (ps0[kinv] - p0[kinv + 1]);
            xbot = GL(v0, kinv - 1) + ssv0[kinv - 1] * (ps0[kinv - 1] - p0[kinv - 1]);
            fluxbelowinv(cbmf, ps0, kinv, dt, xsrc, xmean, xtop, xbot, xflx);
#pragma unroll 1
            for (int k = 0; k <= mkx; k++) if (k <= kinv - 1) vflx[k] = xflx[k];
#pragma unroll 1
            for (int m = 0; m < ncnst; m++) {
                xsrc = trsrc[m];
                xmean = GT(m + 1, kinv);
                xtop = GT(m + 1, kinv + 1) + sstr0[m][kinv + 1] * (ps0[kinv] - p0[kinv + 1]);
                xbot = GT(m + 1, kinv - 1) + sstr0[m][kinv - 1] * (ps0[kinv - 1] - p0[kinv - 1]);
                fluxbelowinv(cbmf, ps0, kinv, dt, xsrc, xmean, xtop, xbot, xflx);
#pragma unroll 1
                for (int k = 0; k <= mkx; k++) if (k <= kinv - 1) trflx[m][k] = xflx[k];
            }
        }
        // 2. non-buoyancy-sorting fluxes (:3300-3313)
        {
            double uplus = 0.0, vplus = 0.0;
#pragma unroll 1
            for (int k = 0; k <= mkx; k++) {
                if (k < kinv || k > krel - 1) continue;
                const int kp1 = k + 1;
                qtflx[k] = cbmf * (qtsrc - (qt0[kp1] + ssqt0[kp1] * (ps0[k] - p0[kp1])));
                slflx[k] = cbmf * (thlsrc - (thl0[kp1] + ssthl0[kp1] * (ps0[k] - p0[kp1]))) * cp * exns0[k];
                uplus = uplus + PGFc * ssu0[k] * (ps0[k] - ps0[k - 1]);
                vplus = vplus + PGFc * ssv0[k] * (ps0[k] - ps0[k - 1]);
                uflx[k] = cbmf * (usrc + uplus - (GL(u0, kp1) + ssu0[kp1] * (ps0[k] - p0[kp1])));
                vflx[k] = cbmf * (vsrc + vplus - (GL(v0, kp1) + ssv0[kp1] * (ps0[k] - p0[kp1])));
#pragma unroll 1
                for (int m = 0; m < ncnst; m++)
                    trflx[m][k] = cbmf * (trsrc[m] - (GT(m + 1, kp1) + sstr0[m][kp1] * (ps0[k] - p0[kp1])));
            }
        }
        // 3. buoyancy-sorting fluxes (:3322-3331)
#pragma unroll 1
        for (int k = 0; k <= mkx; k++) {
            if (k < krel || k > kbup - 1) continue;
            const int kp1 = k + 1;
            slflx[k] = cp * exns0[k] * umf[k] * (thlu[k] - (thl0[kp1] + ssthl0[kp1] * (ps0[k] - p0[kp1])));
            qtflx[k] = umf[k] * (qtu[k] - (qt0[kp1] + ssqt0[kp1] * (ps0[k] - p0[kp1])));
            uflx[k] = umf[k] * (uu[k] - (GL(u0, kp1) + ssu0[kp1] * (ps0[k] - p0[kp1])));
            vflx[k] = umf[k] * (vu[k] - (GL(v0, kp1) + ssv0[kp1] * (ps0[k] - p0[kp1])));
#pragma unroll 1
            for (int m = 0; m < ncnst; m++)
                trflx[m][k] = umf[k] * (tru[m][k] - (GT(m + 1, kp1) + sstr0[m][kp1] * (ps0[k] - p0[kp1])));
        }
        // 4. penetrative-entrainment fluxes (:3392-3401)
#pragma unroll 1
        for (int k = 0; k <= mkx; k++) {
            if (k < kbup || k > kpen - 1) continue;
            slflx[k] = cp * exns0[k] * emf[k] * (thlu_emf[k] - (thl0[k] + ssthl0[k] * (ps0[k] - p0[k])));
            qtflx[k] = emf[k] * (qtu_emf[k] - (qt0[k] + ssqt0[k] * (ps0[k] - p0[k])));
            uflx[k] = emf[k] * (uu_emf[k] - (GL(u0, k) + ssu0[k] * (ps0[k] - p0[k])));
            vflx[k] = emf[k] * (vu_emf[k] - (GL(v0, k) + ssv0[k] * (ps0[k] - p0[k])));
#pragma unroll 1
            for (int m = 0; m < ncnst; m++)
                trflx[m][k] = emf[k] * (tru_emf[m][k] - (GT(m + 1, k) + sstr0[m][k] * (ps0[k] - p0[k])));
        }
        // none above
#pragma unroll 1
        for (int k = MX(kpen, kbup); k <= mkx; k++) {
            slflx[k] = 0.0;
            qtflx[k] = 0.0;
            uflx[k] = 0.0;
            vflx[k] = 0.0;
#pragma unroll 1
            for (int m = 0; m < ncnst; m++) trflx[m][k] = 0.0;
        }
        } while (0);
        UW_SYNC();
        // condensate tendency by compensating subsidence (:3416-3476)
        {
            bool ldone = stop;
#pragma unroll 1
            for (int k = 1; k <= mkx; k++) {   // uniform
                if (k > kpen) ldone = true;
                if (!ldone) do {
                double comsub = 0.5 * (UEMF(k) + UEMF(k - 1));
                double thlten_sub, qtten_sub, qlten_sub, qiten_sub, nlten_sub, niten_sub;
                if (comsub >= 0.0) {
                    if (k == mkx) {
                        thlten_sub = 0.0; qtten_sub = 0.0; qlten_sub = 0.0; qiten_sub = 0.0;
                        nlten_sub = 0.0; niten_sub = 0.0;
                    } else {
                        thlten_sub = g * comsub * (thl0[k + 1] - thl0[k]) / (p0[k] - p0[k + 1]);
                        qtten_sub = g * comsub * (qt0[k + 1] - qt0[k]) / (p0[k] - p0[k + 1]);
                        qlten_sub = g * comsub * (ql0[k + 1] - ql0[k]) / (p0[k] - p0[k + 1]);
                        qiten_sub = g * comsub * (qi0[k + 1] - qi0[k]) / (p0[k] - p0[k + 1]);
                        nlten_sub = g * comsub * (GT(ixnumliq, k + 1) - GT(ixnumliq, k)) / (p0[k] - p0[k + 1]);
                        niten_sub = g * comsub * (GT(ixnumice, k + 1) - GT(ixnumice, k)) / (p0[k] - p0[k + 1]);
                    }
                } else {
                    if (k == 1) {
                        thlten_sub = 0.0; qtten_sub = 0.0; qlten_sub = 0.0; qiten_sub = 0.0;
                        nlten_sub = 0.0; niten_sub = 0.0;
                    } else {
                        thlten_sub = g * comsub * (thl0[k] - thl0[k - 1]) / (p0[k - 1] - p0[k]);
                        qtten_sub = g * comsub * (qt0[k] - qt0[k - 1]) / (p0[k - 1] - p0[k]);
                        qlten_sub = g * comsub * (ql0[k] - ql0[k - 1]) / (p0[k - 1] - p0[k]);
                        qiten_sub = g * comsub * (qi0[k] - qi0[k - 1]) / (p0[k - 1] - p0[k]);
                        nlten_sub = g * comsub * (GT(ixnumliq, k) - GT(ixnumliq, k - 1)) / (p0[k - 1] - p0[k]);
                        niten_sub = g * comsub * (GT(ixnumice, k) - GT(ixnumice, k - 1)) / (p0[k - 1] - p0[k]);
                    }
                }
                double thl_prog = thl0[k] + thlten_sub * dt;
                double qt_prog = MX(qt0[k] + qtten_sub * dt, 1.e-12);
                if (CONDEN(p0[k], exn0[k], thl_prog, qt_prog, thj, qvj, qlj, qij, rvj, tbl)) {
                    id_exit = true;
                    stop = true;
            break;
                }
                qlten_sink[k] = MX(qlten_sub, -ql0[k] / dt);
                qiten_sink[k] = MX(qiten_sub, -qi0[k] / dt);
                nlten_sink[k] = MX(nlten_sub, -GT(ixnumliq, k) / dt);
                niten_sink[k] = MX(niten_sub, -GT(ixnumice, k) / dt);
                } while (0);
                if (stop) ldone = true;
            }
        }
        UW_SYNC();
        if (!stop) do {
        // momentum tendency (:3488-3501)
#pragma unroll 1
        for (int k = 1; k <= mkx; k++) {
            if (k > kpen) {
                uten[k] = 0.0;
                vten[k] = 0.0;
                continue;
            }
            uten[k] = (uflx[k - 1] - uflx[k]) * g / dp0[k];
            vten[k] = (vflx[k - 1] - vflx[k]) * g / dp0[k];
            uf[k] = GL(u0, k) + uten[k] * dt;
            vf[k] = GL(v0, k) + vten[k] * dt;
        }
        // thermodynamic tendencies (:3511-3791)
        rliq = 0.0;
        rainflx = 0.0;
        snowflx = 0.0;
        } while (0);
        UW_SYNC();
        {
            double qlubelow = 0.0, qiubelow = 0.0;
            bool ldone = stop;
#pragma unroll 1
            for (int k = 1; k <= mkx; k++) {   // uniform
                if (k > kpen) {
                    ldone = true;
                    qrten[k] = 0.0; qsten[k] = 0.0; qlten[k] = 0.0; qiten[k] = 0.0; qvten[k] = 0.0;
                    sten[k] = 0.0; qc[k] = 0.0;
                    trten[ixnumliq - 1][k] = 0.0;
                    trten[ixnumice - 1][k] = 0.0;
                }
                if (!ldone) do {
                const int km1 = k - 1;
                if (k < krel) {   // below the updraft
                    dwten[k] = 0.0;
                    diten[k] = 0.0;
                    fdr[k] = 0.0;
                }
                dwten[k] = dwten[k] * 0.5 * (umf[k - 1] + umf[k]) * g / dp0[k];
                diten[k] = diten[k] * 0.5 * (umf[k - 1] + umf[k]) * g / dp0[k];
                qrten[k] = frc_rasn * dwten[k];
                qsten[k] = frc_rasn * diten[k];
                rainflx = rainflx + qrten[k] * dp0[k] / g;
                snowflx = snowflx + qsten[k] * dp0[k] / g;
                slten[k] = (slflx[km1] - slflx[k]) * g / dp0[k];
                if (k == 1) {
                    const double u1 = GL(u0, k), u2 = GL(u0, k + 1), v1 = GL(v0, k), v2 = GL(v0, k + 1);
                    slten[k] = slten[k] - g / 4.0 / dp0[k] *
                                              (uflx[k] * (uf[k + 1] - uf[k] + u2 - u1) +
                                               vflx[k] * (vf[k + 1] - vf[k] + v2 - v1));
                } else if (k >= 2 && k <= kpen - 1) {
                    const double um = GL(u0, k - 1), u1 = GL(u0, k), u2 = GL(u0, k + 1);
                    const double vm = GL(v0, k - 1), v1 = GL(v0, k), v2 = GL(v0, k + 1);
                    slten[k] = slten[k] - g / 4.0 / dp0[k] *
                                              (uflx[k] * (uf[k + 1] - uf[k] + u2 - u1) +
                                               uflx[k - 1] * (uf[k] - uf[k - 1] + u1 - um) +
                                               vflx[k] * (vf[k + 1] - vf[k] + v2 - v1) +
                                               vflx[k - 1] * (vf[k] - vf[k - 1] + v1 - vm));
                } else if (k == kpen) {
                    const double um = GL(u0, k - 1), u1 = GL(u0, k), vm = GL(v0, k - 1), v1 = GL(v0, k);
                    slten[k] = slten[k] - g / 4.0 / dp0[k] *
                                              (uflx[k - 1] * (uf[k] - uf[k - 1] + u1 - um) +
                                               vflx[k - 1] * (vf[k] - vf[k - 1] + v1 - vm));
                }
                qtten[k] = (qtflx[km1] - qtflx[k]) * g / dp0[k];

                double qlu_mid, qiu_mid;
                if (k < krel || k > kpen) {
                    qlu_mid = 0.0;
                    qiu_mid = 0.0;
                    qlj = 0.0;
                    qij = 0.0;
                } else {
                    // the release level, the cloud top and the levels between
                    const bool atrel = (k == krel), attop = (k != krel && k == kpen);
#if UW_TAPE_ORDER
                    if (atrel) {
                        if (CONDEN(prel, exprel, thlu[krel - 1], qtu[krel - 1], thj, qvj, qlj, qij, rvj, tbl)) {
                            xflags |= UW_X_CONDEN;
                            id_exit = true;
                            stop = true;
                            break;
                        }
                        qlubelow = qlj;
                        qiubelow = qij;
                    }
                    if (CONDEN(attop ? ps0[k - 1] + ppen : ps0[k], attop ? exntop : exns0[k], attop ? thlu_top : thlu[k],
                               attop ? qtu_top : qtu[k], thj, qvj, qlj, qij, rvj, tbl)) {
                        xflags |= UW_X_CONDEN;
                        id_exit = true;
                        stop = true;
                        break;
                    }
#else
                    if (attop && id_top) {
                        xflags |= UW_X_CONDEN;
                        id_exit = true;
                        stop = true;
                        break;
                    }
                    if (atrel) {
                        qlubelow = ql_rel;
                        qiubelow = qi_rel;
                    }
                    qlj = attop ? ql_top : qltop[k];
                    qij = attop ? qi_top : qitop[k];
#endif
                    if (atrel) {
                        qlu_mid = 0.5 * (qlubelow + qlj) * (prel - ps0[k]) / (ps0[k - 1] - ps0[k]);
                        qiu_mid = 0.5 * (qiubelow + qij) * (prel - ps0[k]) / (ps0[k - 1] - ps0[k]);
                    } else if (attop) {
                        qlu_mid = 0.5 * (qlubelow + qlj) * (-ppen) / (ps0[k - 1] - ps0[k]);
                        qiu_mid = 0.5 * (qiubelow + qij) * (-ppen) / (ps0[k - 1] - ps0[k]);
                    } else {
                        qlu_mid = 0.5 * (qlubelow + qlj);
                        qiu_mid = 0.5 * (qiubelow + qij);
                    }
                }
                qlubelow = qlj;
                qiubelow = qij;

                double qc_lm, qc_im, nc_lm, nc_im;
                qc_l[k] = (1.0 - frc_rasn) * dwten[k];
                qc_i[k] = (1.0 - frc_rasn) * diten[k];
                const double trl = GT(ixnumliq, k), tri = GT(ixnumice, k);
                if (k <= kbup) {
                    qc_l[k] = qc_l[k] + g * 0.5 * (umf[k - 1] + umf[k]) * fdr[k] * qlu_mid;
                    qc_i[k] = qc_i[k] + g * 0.5 * (umf[k - 1] + umf[k]) * fdr[k] * qiu_mid;
                    qc_lm = -g * 0.5 * (umf[k - 1] + umf[k]) * fdr[k] * ql0[k];
                    qc_im = -g * 0.5 * (umf[k - 1] + umf[k]) * fdr[k] * qi0[k];
                    nc_lm = -g * 0.5 * (umf[k - 1] + umf[k]) * fdr[k] * trl;
                    nc_im = -g * 0.5 * (umf[k - 1] + umf[k]) * fdr[k] * tri;
                } else {
                    qc_lm = 0.0;
                    qc_im = 0.0;
                    nc_lm = 0.0;
                    nc_im = 0.0;
                }
                if (k == kbup) {
                    qc_l[k] = qc_l[k] + g * umf[k] * qlj / (ps0[k - 1] - ps0[k]);
                    qc_i[k] = qc_i[k] + g * umf[k] * qij / (ps0[k - 1] - ps0[k]);
                    qc_lm = qc_lm - g * umf[k] * ql0[k] / (ps0[k - 1] - ps0[k]);
                    qc_im = qc_im - g * umf[k] * qi0[k] / (ps0[k - 1] - ps0[k]);
                    nc_lm = nc_lm - g * umf[k] * trl / (ps0[k - 1] - ps0[k]);
                    nc_im = nc_im - g * umf[k] * tri / (ps0[k - 1] - ps0[k]);
                    double ql_emf_kbup, qi_emf_kbup, thjj, qvjj;
                    if (CONDEN(p0[k], exn0[k], thlu_emf[k], qtu_emf[k], thjj, qvjj, ql_emf_kbup, qi_emf_kbup, rvj, tbl)) {
                        id_exit = true;
                        stop = true;
            break;
                    }
                    double nl_emf_kbup = (ql_emf_kbup > 0.0) ? tru_emf[ixnumliq - 1][k] : 0.0;
                    double ni_emf_kbup = (qi_emf_kbup > 0.0) ? tru_emf[ixnumice - 1][k] : 0.0;
                    qc_lm = qc_lm - g * emf[k] * (ql_emf_kbup - ql0[k]) / (ps0[k - 1] - ps0[k]);
                    qc_im = qc_im - g * emf[k] * (qi_emf_kbup - qi0[k]) / (ps0[k - 1] - ps0[k]);
                    nc_lm = nc_lm - g * emf[k] * (nl_emf_kbup - trl) / (ps0[k - 1] - ps0[k]);
                    nc_im = nc_im - g * emf[k] * (ni_emf_kbup - tri) / (ps0[k - 1] - ps0[k]);
                }
                qlten[k] = qc_l[k] + frc_rasn * dwten[k] + (MX(0.0, ql0[k] + (qc_lm + qlten_sink[k]) * dt) - ql0[k]) / dt;
                qiten[k] = qc_i[k] + frc_rasn * diten[k] + (MX(0.0, qi0[k] + (qc_im + qiten_sink[k]) * dt) - qi0[k]) / dt;
                trten[ixnumliq - 1][k] = MX(nc_lm + nlten_sink[k], -trl / dt);
                trten[ixnumice - 1][k] = MX(nc_im + niten_sink[k], -tri / dt);
                qvten[k] = qtten[k] - qlten[k] - qiten[k];
                sten[k] = slten[k] + xlv * qlten[k] + xls * qiten[k];
                qc[k] = qc_l[k] + qc_i[k];
                rliq = rliq + qc[k] * dp0[k] / g / 1000.0;
                } while (0);
                if (stop) ldone = true;
            }
        }
        UW_SYNC();
        // evaporation and melting of precipitation (:3808-3934)
        if (!stop) do {
        {
            double evpint_rain = 0.0, evpint_snow = 0.0;
#pragma unroll 1
            for (int k = 0; k <= mkx; k++) {
                flxrain[k] = 0.0;
                flxsnow[k] = 0.0;
            }
#pragma unroll 1
            for (int k = mkx; k >= 1; k--) {
                double snowmlt;
                if (t0[k] > 273.16) snowmlt = MX(0.0, flxsnow[k] * g / dp0[k]);
                else snowmlt = 0.0;
                double qs1 = qsat_qs(t0[k], p0[k], tbl);
                double subsat = MX((1.0 - qv0[k] / qs1), 0.0);
                double evprain = kevp * subsat * sqrt(flxrain[k] + snowmlt * dp0[k] / g);
                double evpsnow = kevp * subsat * sqrt(MX(flxsnow[k] - snowmlt * dp0[k] / g, 0.0));
                double evplimit = MX(0.0, (qw0[k] - qv0[k]) / dt);
                double evplimit_rain = MN(evplimit, (flxrain[k] + snowmlt * dp0[k] / g) * g / dp0[k]);
                evplimit_rain = MN(evplimit_rain, (rainflx - evpint_rain) * g / dp0[k]);
                evprain = MX(0.0, MN(evplimit_rain, evprain));
                double evplimit_snow = MN(evplimit, MX(flxsnow[k] - snowmlt * dp0[k] / g, 0.0) * g / dp0[k]);
                evplimit_snow = MN(evplimit_snow, (snowflx - evpint_snow) * g / dp0[k]);
                evpsnow = MX(0.0, MN(evplimit_snow, evpsnow));
                if ((evprain + evpsnow) > evplimit) {
                    double tmp1 = evprain * evplimit / (evprain + evpsnow);
                    double tmp2 = evpsnow * evplimit / (evprain + evpsnow);
                    evprain = tmp1;
                    evpsnow = tmp2;
                }
                evapc[k] = evprain + evpsnow;
                cufrc[k] = 0.0; qcu[k] = 0.0; qlu[k] = 0.0; qiu[k] = 0.0;   // in cloud: below
                evpint_rain = evpint_rain + evprain * dp0[k] / g;
                evpint_snow = evpint_snow + evpsnow * dp0[k] / g;
                double ntraprd = qrten[k] - evprain + snowmlt;
                double ntsnprd = qsten[k] - evpsnow - snowmlt;
                flxrain[k - 1] = flxrain[k] + ntraprd * dp0[k] / g;
                flxsnow[k - 1] = flxsnow[k] + ntsnprd * dp0[k] / g;
                flxrain[k - 1] = MX(flxrain[k - 1], 0.0);
                flxsnow[k - 1] = MX(flxsnow[k - 1], 0.0);
                qlten[k] = qlten[k] - qrten[k];
                qiten[k] = qiten[k] - qsten[k];
                qvten[k] = qvten[k] + evprain + evpsnow;
                qtten[k] = qlten[k] + qiten[k] + qvten[k];
                if ((qv0[k] + qvten[k] * dt) < c.qmin[0] || (ql0[k] + qlten[k] * dt) < c.qmin[1] ||
                    (qi0[k] + qiten[k] * dt) < c.qmin[2])
                    lflags |= UW_L_NEGCON;
                sten[k] = sten[k] - xlv * evprain - xls * evpsnow - (xls - xlv) * snowmlt;
                slten[k] = sten[k] - xlv * qlten[k] - xls * qiten[k];
            }
            precip = (flxrain[0] + flxsnow[0]) / 1000.0;
            snow = flxsnow[0] / 1000.0;
        }
        // remove detrained condensate (:3966-3981)
#pragma unroll 1
        for (int k = 1; k <= mkx; k++) {
            if (k > kpen) continue;
            qtten[k] = qtten[k] - qc[k];
            qlten[k] = qlten[k] - qc_l[k];
            qiten[k] = qiten[k] - qc_i[k];
            slten[k] = slten[k] + (xlv * qc_l[k] + xls * qc_i[k]);
            sten[k] = sten[k] - (xls - xlv) * qc_i[k];
        }
        // positive_moisture_single (uwshcu.F90:5096-5162 via :3995-4001); state after the tendencies
        {
            const double qvmin = c.qmin[0], qlmin = c.qmin[1], qimin = c.qmin[2];
            double qvs[KP];
#pragma unroll 1
            for (int k = 1; k <= mkx; k++) qvs[k] = qv0[k] + qvten[k] * dt;
            double dqv = 0.0;
#pragma unroll 1
            for (int k = mkx; k >= 1; k--) {
                double qlk = ql0[k] + qlten[k] * dt;
                double qik = qi0[k] + qiten[k] * dt;
                double dql = MX(0.0, 1.0 * qlmin - qlk);
                double dqi = MX(0.0, 1.0 * qimin - qik);
                qlten[k] = qlten[k] + dql / dt;
                qiten[k] = qiten[k] + dqi / dt;
                qvten[k] = qvten[k] - (dql + dqi) / dt;
                sten[k] = sten[k] + xlv * (dql / dt) + xls * (dqi / dt);
                qvs[k] = qvs[k] - dql - dqi;
                dqv = MX(0.0, 1.0 * qvmin - qvs[k]);
                qvten[k] = qvten[k] + dqv / dt;
                qvs[k] = qvs[k] + dqv;
                if (k != 1) {
                    qvs[k - 1] = qvs[k - 1] - dqv * dp0[k] / dp0[k - 1];
                    qvten[k - 1] = qvten[k - 1] - dqv * dp0[k] / dp0[k - 1] / dt;
                }
                qvs[k] = MX(qvs[k], qvmin);
            }
            if (dqv > 1.e-20) {
                double sum = 0.0;
#pragma unroll 1
                for (int k = 1; k <= mkx; k++)
                    if (qvs[k] > 2.0 * qvmin) sum = sum + qvs[k] * dp0[k];
                double aa = dqv * dp0[1] / MX(1.e-20, sum);
                if (aa < 0.5) {
#pragma unroll 1
                    for (int k = 1; k <= mkx; k++) {
                        if (qvs[k] > 2.0 * qvmin) {
                            double dum = aa * qvs[k];
                            qvs[k] = qvs[k] - dum;
                            qvten[k] = qvten[k] - dum / dt;
                        }
                    }
                }
            }
        }
#pragma unroll 1
        for (int k = 1; k <= mkx; k++) {
            qtten[k] = qvten[k] + qlten[k] + qiten[k];
            slten[k] = sten[k] - xlv * qlten[k] - xls * qiten[k];
        }
        // tracer tendencies (:4007-4076)
#pragma unroll 1
        for (int m = 1; m <= ncnst; m++) {
            if (m < 4) {
                if (m != ixnumliq && m != ixnumice) {   // qv, ql and qi: their tendencies are outputs of their own
#pragma unroll 1
                    for (int k = 1; k <= mkx; k++) trten[m - 1][k] = 0.0;
                }
            } else if (m != ixnumliq && m != ixnumice) {
                const double trmin = c.qmin[m - 1];
                const bool wet = c.wet[m - 1] != 0;
#pragma unroll 1
                for (int k = 0; k <= mkx; k++) {
                    trflx_d[k] = 0.0;
                    trflx_u[k] = 0.0;
                }
#pragma unroll 1
                for (int k = 1; k <= mkx - 1; k++) {
                    double pdelx = wet ? dp0[k] : GL(dpdry0, k);
                    double dum = (GT(m, k) - trmin) * pdelx / g / dt + trflx[m - 1][k - 1] - trflx[m - 1][k] + trflx_d[k - 1];
                    trflx_d[k] = MN(0.0, dum);
                }
#pragma unroll 1
                for (int k = mkx; k >= 2; k--) {
                    double pdelx = wet ? dp0[k] : GL(dpdry0, k);
                    double dum = (GT(m, k) - trmin) * pdelx / g / dt + trflx[m - 1][k - 1] - trflx[m - 1][k] +
                                 trflx_d[k - 1] - trflx_d[k] - trflx_u[k];
                    trflx_u[k - 1] = MX(0.0, -dum);
                }
#pragma unroll 1
                for (int k = 1; k <= mkx; k++) {
                    double pdelx = wet ? dp0[k] : GL(dpdry0, k);
                    trten[m - 1][k] = (trflx[m - 1][k - 1] - trflx[m - 1][k] + trflx_d[k - 1] - trflx_d[k] +
                                       trflx_u[k - 1] - trflx_u[k]) * g / pdelx;
                }
            }
        }
        // in-cloud diagnostics (:4092-4158)
#if UW_TAPE_ORDER
        if (CONDEN(prel, exprel, thlu[krel - 1], qtu[krel - 1], thj, qvj, qlj, qij, rvj, tbl)) {
            xflags |= UW_X_CONDEN;
            id_exit = true;
            stop = true;
            break;
        }
#else
        qlj = ql_rel;
        qij = qi_rel;
#endif
        } while (0);
        UW_SYNC();
        {
            double qcubelow = qlj + qij, qlubelow = qlj, qiubelow = qij;
            bool ldone = stop;
#pragma unroll 1
            for (int j = 0; j <= mkx; j++) {   // uniform
                const int k = krel + j;
                if (k > kpen) ldone = true;
                if (!ldone) do {
                const bool attop = (k == kpen);
#if UW_TAPE_ORDER
                const int idc = CONDEN(attop ? ps0[k - 1] + ppen : ps0[k], attop ? exntop : exns0[k],
                                       attop ? thlu_top : thlu[k], attop ? qtu_top : qtu[k], thj, qvj, qlj, qij, rvj, tbl);
#else
                const bool idc = attop && id_top;
                qlj = attop ? ql_top : qltop[k];
                qij = attop ? qi_top : qitop[k];
#endif
                if (idc) {
                    xflags |= UW_X_CONDEN;
                    id_exit = true;
                    stop = true;
                    break;
                }
                qcu[k] = 0.5 * (qcubelow + qlj + qij);
                qlu[k] = 0.5 * (qlubelow + qlj);
                qiu[k] = 0.5 * (qiubelow + qij);
                // compute_zwshcu's cloud-fraction option (zwshcu.F90:4413-4431, 4449)
                double zw_tmp2 = 0.0, zw_tmp3 = 1.0;
                if (ZW && c.zw_cloud_sh) {
                    zw_tmp3 = 0.5 * c.zw_ufrc0;
                    double tmp1 = (GL(z0, k) - GL(z0, krel)) / (GL(z0, kpen) - GL(z0, krel) + 10.0);
                    tmp1 = 1.0 + c.zw_ufrcz * tmp1;
                    zw_tmp3 = zw_tmp3 * tmp1;
                    zw_tmp2 = fdr[k] * umf[k] * (zs0[k] - zs0[k - 1]) * dt / dp0[k] * 9.8 * c.zw_ufrcd;
                    zw_tmp2 = MN(1.0 - rmaxfrac, zw_tmp2);
                }
                cufrc[k] = (ufrc[k - 1] + ufrc[k]);
                if (k == krel) {
                    cufrc[k] = (ufrclcl + ufrc[k]) * (prel - ps0[k]) / (ps0[k - 1] - ps0[k]);
                } else if (k == kpen) {
                    cufrc[k] = (ufrc[k - 1] + 0.0) * (-ppen) / (ps0[k - 1] - ps0[k]);
                    if ((qlj + qij) > criqc) {
                        qcu[k] = 0.5 * (qcubelow + criqc);
                        qlu[k] = 0.5 * (qlubelow + criqc * qlj / (qlj + qij));
                        qiu[k] = 0.5 * (qiubelow + criqc * qij / (qlj + qij));
                    }
                }
                if constexpr (ZW) cufrc[k] = zw_tmp3 * cufrc[k] + zw_tmp2;
                qcubelow = qlj + qij;
                qlubelow = qlj;
                qiubelow = qij;
                } while (0);
                if (stop) ldone = true;
            }
        }
        UW_SYNC();
        if (!stop) do {
        cnt = (double)kpen;
        cnb = (double)(krel - 1);

        if (iter == 1) {
            cin_s = cin; cinlcl_s = cinlcl; plcl_s = plcl; pinv_s = ps0[kinv - 1]; plfc_s = plfc;
            pbup_s = ps0[kbup]; ppen_s = ps0[kpen - 1] + ppen; tkeavg_s = tkeavg;
            kinv_s = kinv; klcl_s = klcl; klfc_s = klfc; krel_s = krel; kbup_s = kbup; kpen_s = kpen;
            // advance the state for the second CIN estimate (:4177-4184, :4285-4327)
#pragma unroll 1
            for (int k = 1; k <= mkx; k++) {
                double qv0s = qv0[k] + qvten[k] * dt;
                double ql0s = ql0[k] + qlten[k] * dt;
                double qi0s = qi0[k] + qiten[k] * dt;
                double s0s = s0[k] + sten[k] * dt;
                double t0s = t0[k] + sten[k] * dt / cp;
                qv0[k] = qv0s;
                ql0[k] = ql0s;
                qi0[k] = qi0s;
                s0[k] = s0s;
                t0[k] = t0s;
                qt0[k] = (qv0[k] + ql0[k] + qi0[k]);
                thl0[k] = (t0[k] - xlv * ql0[k] / cp - xls * qi0[k] / cp) / exn0[k];
            }
            slope<KP>(mkx, thl0, p0, ssthl0);
            slope<KP>(mkx, qt0, p0, ssqt0);
        }
        } while (0);
        UW_SYNC();
        if (iter == 1) {   // uniform
            bool ldone = stop;
#pragma unroll 1
            for (int k = 1; k <= mkx; k++) {   // uniform
                if (!ldone) do {
                double thl0bot = thl0[k] + ssthl0[k] * (ps0[k - 1] - p0[k]);
                double qt0bot = qt0[k] + ssqt0[k] * (ps0[k - 1] - p0[k]);
                if (CONDEN(ps0[k - 1], exns0[k - 1], thl0bot, qt0bot, thj, qvj, qlj, qij, rvj, tbl)) {
                    xflags |= UW_X_CONDEN;
                    id_exit = true;
                    stop = true;
                    break;
                }
                thv0bot[k] = thj * (1.0 + zvir * qvj - qlj - qij);
                thvl0bot[k] = thl0bot * (1.0 + zvir * qt0bot);
                double thl0top = thl0[k] + ssthl0[k] * (ps0[k] - p0[k]);
                double qt0top = qt0[k] + ssqt0[k] * (ps0[k] - p0[k]);
                if (CONDEN(ps0[k], exns0[k], thl0top, qt0top, thj, qvj, qlj, qij, rvj, tbl)) {
                    xflags |= UW_X_CONDEN;
                    id_exit = true;
                    stop = true;
                    break;
                }
                thv0top[k] = thj * (1.0 + zvir * qvj - qlj - qij);
                thvl0top[k] = thl0top * (1.0 + zvir * qt0top);
                } while (0);
                if (stop) ldone = true;
            }
        }
        UW_SYNC();
        }   // MODE != UW_MODE_TRIGGER
    }

    // ---- final outputs (uwshcu.F90:4337-4370) --------------------------------------------------
    if (!stop) {
#pragma unroll 1
    for (int k = 0; k <= mkx; k++) {
        OI(umf, k) = umf[k];
        OI(wu, k) = wu[k];
        OI(slflx, k) = slflx[k];
        OI(qtflx, k) = qtflx[k];
        OI(flxprc1, k) = flxrain[k] + flxsnow[k];
        OI(flxsnow1, k) = flxsnow[k];
    }
#pragma unroll 1
    for (int k = 1; k <= mkx; k++) {
        OL(qvten, k) = qvten[k]; OL(qlten, k) = qlten[k]; OL(qiten, k) = qiten[k];
        OL(sten, k) = sten[k]; OL(uten, k) = uten[k]; OL(vten, k) = vten[k];
        OL(qrten, k) = qrten[k]; OL(qsten, k) = qsten[k]; OL(evapc, k) = evapc[k];
        OL(cufrc, k) = cufrc[k]; OL(qcu, k) = qcu[k]; OL(qlu, k) = qlu[k];
        OL(qiu, k) = qiu[k]; OL(qc, k) = qc[k];
#pragma unroll 1
        for (int m = 1; m <= ncnst; m++) OT(m, k) = trten[m - 1][k];
    }
    A.precip[i] = precip;
    A.snow[i] = snow;
    A.cush[i] = cush;
    A.cbmf[i] = cbmf;
    A.rliq[i] = rliq;
    A.cnt[i] = CNT(cnt);
    A.cnb[i] = CNT(cnb);
    if (A.diag_real) {
        A.diag_real[UW_DR_CIN * (size_t)mix + i] = cin;
        A.diag_real[UW_DR_CINLCL * (size_t)mix + i] = cinlcl;
        A.diag_real[UW_DR_PLCL * (size_t)mix + i] = plcl;
        A.diag_real[UW_DR_PLFC * (size_t)mix + i] = plfc;
        A.diag_real[UW_DR_PINV * (size_t)mix + i] = ps0[kinv - 1];
        A.diag_real[UW_DR_PBUP * (size_t)mix + i] = ps0[kbup];
        A.diag_real[UW_DR_PPEN * (size_t)mix + i] = ps0[kpen - 1] + ppen;
        A.diag_real[UW_DR_TKEAVG * (size_t)mix + i] = tkeavg;
    }
    PUT_DIAG_LEVEL();
    }

    // (label 333, :4448-4549)
    if (!cand && !handed) {
    if (id_exit) {
        xflags |= UW_X_UWCU;
#pragma unroll 1
        for (int k = 0; k <= mkx; k++) {
            OI(umf, k) = 0.0;
            OI(wu, k) = 0.0;
            OI(slflx, k) = 0.0;
            OI(qtflx, k) = 0.0;
            OI(flxprc1, k) = 0.0;
            OI(flxsnow1, k) = 0.0;
        }
#pragma unroll 1
        for (int k = 1; k <= mkx; k++) {
            OL(qvten, k) = 0.0; OL(qlten, k) = 0.0; OL(qiten, k) = 0.0; OL(sten, k) = 0.0;
            OL(uten, k) = 0.0; OL(vten, k) = 0.0; OL(qrten, k) = 0.0; OL(qsten, k) = 0.0;
            OL(evapc, k) = 0.0; OL(cufrc, k) = 0.0; OL(qcu, k) = 0.0; OL(qlu, k) = 0.0;
            OL(qiu, k) = 0.0; OL(qc, k) = 0.0;
#pragma unroll 1
            for (int m = 1; m <= ncnst; m++) OT(m, k) = 0.0;
        }
        A.precip[i] = 0.0;
        A.snow[i] = 0.0;
        A.cush[i] = -1.0;
        A.cbmf[i] = 0.0;
        A.rliq[i] = 0.0;
        A.cnt[i] = CNT(1.0);
        A.cnb[i] = CNT((double)mkx);
        if (A.diag_real) {
            A.diag_real[UW_DR_CIN * (size_t)mix + i] = -1.0;
            A.diag_real[UW_DR_CINLCL * (size_t)mix + i] = -1.0;
#pragma unroll 1
            for (int j = UW_DR_PLCL; j < UW_NDR; j++) A.diag_real[j * (size_t)mix + i] = 0.0;
        }
        if (A.diag_level)
#pragma unroll 1
            for (int j = 0; j < UW_NDL; j++)
#pragma unroll 1
                for (int k = 0; k <= mkx; k++) DLV(j, k) = 0.0;
        kinv = klcl = klfc = krel = kbup = kpen = 0;
    }
    if (A.diag_int) {
        A.diag_int[UW_DI_EXIT * (size_t)mix + i] = xflags;
        A.diag_int[UW_DI_LIMIT * (size_t)mix + i] = lflags;
        A.diag_int[UW_DI_KINV * (size_t)mix + i] = kinv;
        A.diag_int[UW_DI_KLCL * (size_t)mix + i] = klcl;
        A.diag_int[UW_DI_KLFC * (size_t)mix + i] = klfc;
        A.diag_int[UW_DI_KREL * (size_t)mix + i] = krel;
        A.diag_int[UW_DI_KBUP * (size_t)mix + i] = kbup;
        A.diag_int[UW_DI_KPEN * (size_t)mix + i] = kpen;
    }
    // the column's place in the next call's first worklist launch (uwshcu_set_depth_order): the
    // explicit-CIN columns first, then by updraft depth
    if (A.depth_key) {
        const int depth = kpen - krel;
        A.depth_key[i] = ((lflags & UW_L_DELCIN) ? 0 : 64) + (depth < 0 ? 0 : (depth > 63 ? 63 : depth));
    }
    }
    if (MODE == UW_MODE_TRIGGER && A.trig_key) A.trig_key[i] = (unsigned char)(cand ? krel : 0);
    if (errbits) atomicOr(A.err, errbits);
    }  // active
    if (MODE == UW_MODE_TRIGGER && !A.trig_key) {
        // warp-aggregated append of this warp's candidates
        const unsigned lane = threadIdx.x & 31u;
        const unsigned mask = __ballot_sync(0xffffffffu, cand);
        if (mask) {
            const int leader = __ffs(mask) - 1;
            int base = 0;
            if ((int)lane == leader) base = atomicAdd(wl_count, __popc(mask));
            base = __shfl_sync(0xffffffffu, base, leader);
            if (cand) wl[base + __popc(mask & ((1u << lane) - 1u))] = i;
        }
    }
#undef UW_SYNC
#undef UW_SLOPE
#undef CONDEN
#undef UW_QSAT_OF_CONDEN
#undef RI
#undef RL
#undef CNT
#undef GI
#undef GL
#undef GT
#undef OI
#undef OL
#undef OT
#undef DLV
#undef PUT_DIAG_LEVEL
#undef ZERO_DIAG_PROFILES
#undef UEMF
}

// ---- kernels ---------------------------------------------------------------------------------------

// Register caps (resident blocks of 128 per SM).  The worklist launches take 128 and 80 registers (4 and 6
// blocks) for short worklists, whose warps each run alone on their scheduler and lose to every spill, and
// 72 (7 blocks) for long ones (`dense`; where the line lies, with both sides measured: uw_short_list), whose
// warps hide each other's waits for memory and instructions; 5, 6 and 8 blocks for both are no better at either
// end.  Which it is the device decides by handing each of the two launches its count, the worklist's or 0: a
// test of the length at the kernel's entry changed the compiler's code (1,048,576 columns 104.2 -> 106.0 ms).
// The trigger pass takes 80 (6 blocks: 8.9 ms at 1,048,576 columns, 9.6 ms at 5), the single pass 168.
#define UW_LIST_MINB(m, dense)                                                                            \
    ((m) == UW_MODE_RESUME ? ((dense) ? 7 : 6)                                                            \
                           : (UW_MODE_IS_LIST(m) ? ((dense) ? 7 : 4) : ((m) == UW_MODE_TRIGGER ? 6 : 3)))
template <int KP, int NC, int MODE, int ZW = 0, int DENSE = 0>
__global__ void __launch_bounds__(128, UW_LIST_MINB(MODE, DENSE))
uwshcu_fp64_kernel(const __grid_constant__ UwArgs A, int* __restrict__ wl, int* __restrict__ wl_count)
{
    __shared__ double tbl[UW_TBL];
    for (int t = threadIdx.x; t < UW_TBL; t += blockDim.x) tbl[t] = c_estbl[t];
    __syncthreads();

    const int tid = blockIdx.x * blockDim.x + threadIdx.x;
    int i;
    bool active;
    if (MODE == UW_MODE_LIST || MODE == UW_MODE_LIST1) {
        const int t = uw_spread(*wl_count, A.spread, tid);
        active = t >= 0;
        i = active ? wl[t] : 0;
    } else if (MODE == UW_MODE_RESUME) {
        const int t = uw_spread(MN(*A.hand->count, A.hand->cap), A.spread, tid);
        active = t >= 0;
        i = active ? A.hand->order[t] : 0;   // a hand-off slot
    } else {
        active = tid < A.iend;
        i = tid;
    }
    uw_column<KP, NC, MODE, 0, ZW>(A, tbl, i, active, wl, wl_count);
}

// Batched trigger pass: every column of every member of B (members of one level/tracer class).
// Blocks [block_start[m], block_start[m+1]) cover member m; its convecting columns go to
// wl[m] / count[m].  FAST selects the column code of the fast-FP64 mode.
template <int KP, int NC, int FAST>
__global__ void __launch_bounds__(128, 5) uwshcu_batch_trigger(const __grid_constant__ UwBatch B)
{
    __shared__ double tbl[UW_TBL];
    for (int t = threadIdx.x; t < UW_TBL; t += blockDim.x) tbl[t] = c_estbl[t];
    __syncthreads();

    int m = 0;
    while (m + 1 < B.nm && (int)blockIdx.x >= B.block_start[m + 1]) m++;
    const int tid = ((int)blockIdx.x - B.block_start[m]) * blockDim.x + threadIdx.x;
    const bool active = tid < B.m[m].iend;
    uw_column<KP, NC, UW_MODE_TRIGGER, FAST>(B.m[m], tbl, tid, active, B.wl[m], B.count + m);
}

// Batched worklist pass, persistent: each warp takes the next task (32 * B.chunk consecutive queue
// entries of one member) from the device counter *B.task_head until the queues are drained, so a
// warp never mixes members (their level counts differ).  Task t of member m covers entries
// [t * 32 * chunk, (t + 1) * 32 * chunk) of wl[m].  LMODE: UW_MODE_LIST, or UW_MODE_LIST1 for the
// sorted schedule (each member hands its implicit-CIN columns to its own region, B.m[m].hand).
template <int KP, int NC, int MINB, int FAST, int LMODE = UW_MODE_LIST>
__global__ void __launch_bounds__(128, MINB) uwshcu_batch_list(const __grid_constant__ UwBatch B)
{
    __shared__ double tbl[UW_TBL];
    for (int t = threadIdx.x; t < UW_TBL; t += blockDim.x) tbl[t] = c_estbl[t];
    __syncthreads();

    const int lane = threadIdx.x & 31;
    const int per_task = 32 * B.chunk;
    for (;;) {
        int task = 0;
        if (lane == 0) task = atomicAdd(B.task_head, 1);
        task = __shfl_sync(0xffffffffu, task, 0);
        int m = -1, first = 0;
        for (int j = 0; j < B.nm; j++) {
            const int nt = (B.count[j] + per_task - 1) / per_task;
            if (m < 0) {
                if (task < nt) {
                    m = j;
                    first = task * per_task;
                } else {
                    task -= nt;
                }
            }
        }
        if (m < 0) break;   // same task on every lane: the whole warp leaves
        const int n = B.count[m];
        for (int c = 0; c < B.chunk; c++) {
            const int idx = first + c * 32 + lane;
            const bool active = idx < n;
            const int i = active ? B.wl[m][idx] : 0;
            uw_column<KP, NC, LMODE, FAST>(B.m[m], tbl, i, active, nullptr, nullptr);
        }
    }
}

// Batched resume launch of the sorted schedule, persistent: each warp takes the next task (32
// consecutive entries of one member's hand-off slots in sorted order) from *B.task_head2 until every
// member's slots are done.  Member m has min(*count, cap) slots in its region B.m[m].hand.
template <int KP, int NC, int FAST, int MINB = 5>
__global__ void __launch_bounds__(128, MINB) uwshcu_batch_resume(const __grid_constant__ UwBatch B)
{
    __shared__ double tbl[UW_TBL];
    for (int t = threadIdx.x; t < UW_TBL; t += blockDim.x) tbl[t] = c_estbl[t];
    __syncthreads();

    const int lane = threadIdx.x & 31;
    for (;;) {
        int task = 0;
        if (lane == 0) task = atomicAdd(B.task_head2, 1);
        task = __shfl_sync(0xffffffffu, task, 0);
        int m = -1, first = 0;
        for (int j = 0; j < B.nm; j++) {
            const int nt = (MN(*B.m[j].hand->count, B.m[j].hand->cap) + 31) / 32;
            if (m < 0) {
                if (task < nt) {
                    m = j;
                    first = task * 32;
                } else {
                    task -= nt;
                }
            }
        }
        if (m < 0) break;   // same task on every lane: the whole warp leaves
        const UwHand& H = *B.m[m].hand;
        const int idx = first + lane;
        const bool active = idx < MN(*H.count, H.cap);
        const int slot = active ? H.order[idx] : 0;
        uw_column<KP, NC, UW_MODE_RESUME, FAST>(B.m[m], tbl, slot, active, nullptr, nullptr);
    }
}

// The fast-FP64 precision mode: same launch shapes as uwshcu_fp64_kernel.
template <int KP, int NC, int MODE>
__global__ void __launch_bounds__(128, UW_LIST_MINB(MODE, 0))
uwshcu_fast_kernel(const __grid_constant__ UwArgs A, int* __restrict__ wl, int* __restrict__ wl_count)
{
    __shared__ double tbl[UW_TBL];
    for (int t = threadIdx.x; t < UW_TBL; t += blockDim.x) tbl[t] = c_estbl[t];
    __syncthreads();

    const int tid = blockIdx.x * blockDim.x + threadIdx.x;
    int i;
    bool active;
    if (MODE == UW_MODE_LIST || MODE == UW_MODE_LIST1) {
        const int t = uw_spread(*wl_count, A.spread, tid);
        active = t >= 0;
        i = active ? wl[t] : 0;
    } else if (MODE == UW_MODE_RESUME) {
        const int t = uw_spread(MN(*A.hand->count, A.hand->cap), A.spread, tid);
        active = t >= 0;
        i = active ? A.hand->order[t] : 0;   // a hand-off slot
    } else {
        active = tid < A.iend;
        i = tid;
    }
    uw_column<KP, NC, MODE, 1>(A, tbl, i, active, wl, wl_count);
}

}  // namespace
