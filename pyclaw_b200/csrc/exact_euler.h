// exact_euler.h -- exact Riemann solver of the 1D Euler equations (the normal
// direction of a 2D interface), used by the CUDA kernels (the CPU oracle
// restates it independently in oracle/claw_oracle.cpp).
//
// Method: Toro, Riemann Solvers and Numerical Methods for Fluid Dynamics, 3rd
// ed., Springer 2009, ch. 4: p* is the root of
//     f(p) = f_L(p) + f_R(p) + (u_R - u_L),
// f_K = shock branch (p > p_K) or rarefaction branch (p <= p_K) (eqs. 4.6-4.7,
// derivatives 4.37), found by Newton's method; u* from eq. 4.9; star densities
// from the shock / isentropic relations; the state at x/t = 0 by sampling the
// wave fan (sec. 4.5).  Initial guesses: the adaptive PVRS / two-rarefaction /
// two-shock choice of sec. 9.5.1 ("plain" guess), or a caller-supplied one
// (the learned guess), which is used only if finite and positive.
//
// Stopping rule: each Newton step |f/f'| is compared with tol * p; a step
// below it is the last one (applied, since f and f' are already at hand, which
// leaves p* at machine precision) and is not counted: `iters` counts the
// steps that were needed, so a guess already within tolerance costs none.
//
// Plain C++ with EX_HD on every function, so host code of the library can use
// it too.
#pragma once

#include <math.h>

#ifdef __CUDACC__
#define EX_HD __host__ __device__ __forceinline__
#else
#define EX_HD inline
#endif

#ifdef __CUDACC__
#include "claw2_types.cuh"
#endif

namespace exact_euler {

// Powers and square roots.  On the device x^y = exp(y ln x) (x > 0 wherever
// the solver takes a power) and the branch-free claw2::sqrt_nr: CUDA's pow
// handles every sign and integer case of its arguments in code that, inlined
// at the Newton, fan and sampling sites, outgrew the instruction cache of the
// step kernel (whose top stall was instruction fetch); the relative error of
// exp(y ln x) is about |y ln x| ulps, 1e-14 at most for the pressure and
// density ratios met here.  The host keeps the library functions.
EX_HD double ex_pow(double x, double y) {
#ifdef __CUDA_ARCH__
    return exp(y * log(x));
#else
    return pow(x, y);
#endif
}
// w = x^y and w - 1 for x <= 1, y > 0, the difference exact where it is small: with z = y ln x,
// the series z + z^2 / 2! + ... to z^11 / 11! (the next term is 2e-19 of z at -1/8), which
// is all that interfaces of a smooth flow need (g1 = 1/7: pressure ratios down to 0.42)
// and takes half of an exponential's instructions.
EX_HD double ex_powm1(double x, double y, double& w) {
    const double z = y * log(x);
    if (z < -0.125) {
        w = exp(z);
        return w - 1.0;
    }
    double s = 1.0 / 39916800.0;
    s = fma(s, z, 1.0 / 3628800.0);
    s = fma(s, z, 1.0 / 362880.0);
    s = fma(s, z, 1.0 / 40320.0);
    s = fma(s, z, 1.0 / 5040.0);
    s = fma(s, z, 1.0 / 720.0);
    s = fma(s, z, 1.0 / 120.0);
    s = fma(s, z, 1.0 / 24.0);
    s = fma(s, z, 1.0 / 6.0);
    s = fma(s, z, 1.0 / 2.0);
    const double e = fma(s * z, z, z);
    w = 1.0 + e;
    return e;
}
EX_HD double ex_sqrt(double x) {
#ifdef __CUDA_ARCH__
    return claw2::sqrt_nr(x);
#else
    return sqrt(x);
#endif
}
// 1/x: the branch-free claw2::rcp_nr on the device (quotients in the Newton
// loop and the fan become products with it)
EX_HD double ex_rcp(double x) {
#ifdef __CUDA_ARCH__
    return claw2::rcp_nr(x);
#else
    return 1.0 / x;
#endif
}

struct Gas {
    double g, g1, g2, g3, g4, g5, g6, g7;  // gamma and Toro's constants G1..G7
};

EX_HD Gas make_gas(double gamma) {
    Gas G;
    G.g = gamma;
    G.g1 = (gamma - 1.0) / (2.0 * gamma);
    G.g2 = (gamma + 1.0) / (2.0 * gamma);
    G.g3 = 2.0 * gamma / (gamma - 1.0);
    G.g4 = 2.0 / (gamma - 1.0);
    G.g5 = 2.0 / (gamma + 1.0);
    G.g6 = (gamma - 1.0) / (gamma + 1.0);
    G.g7 = (gamma - 1.0) / 2.0;
    return G;
}

// f_K and f_K' at pressure p (Toro eqs. 4.6, 4.7, 4.37); x = (p / p_K)^g1 - 1 of a
// rarefaction, 2 for a shock.  (The difference as it is: formed from the power, its
// rounding is g4 c_K = 5 c_K times 2^-54 of f, what bounded u* and p*.)
EX_HD void prefun(const Gas& G, double p, double rk, double pk, double ck, double& f, double& fd, double& x) {
    if (p <= pk) {
        const double prat = p * ex_rcp(pk);
        double pw;
        x = ex_powm1(prat, G.g1, pw);
        f = G.g4 * ck * x;
        fd = pw * ex_rcp(prat * rk * ck);  // (1/(rho c)) * prat^(-g2), with prat^(-g2) = prat^g1 / prat
    } else {
        const double ak = G.g5 * ex_rcp(rk);
        const double bk = G.g6 * pk;
        const double ibp = ex_rcp(bk + p);
        const double qrt = ex_sqrt(ak * ibp);
        f = (p - pk) * qrt;
        fd = (1.0 - 0.5 * (p - pk) * ibp) * qrt;
        x = 2.0;
    }
}

// Adaptive noniterative guess (Toro sec. 9.5.1): PVRS when the pressure ratio
// is small and PVRS stays inside [pmin, pmax], else two-rarefaction (TRRS)
// below pmin or two-shock (TSRS) above.
EX_HD double guess_pvrs(const Gas& G, double rl, double ul, double pl, double cl, double rr, double ur, double pr,
                        double cr) {
    const double cup = 0.25 * (rl + rr) * (cl + cr);
    double ppv = 0.5 * (pl + pr) + 0.5 * (ul - ur) * cup;
    ppv = fmax(0.0, ppv);
    const double pmin = fmin(pl, pr), pmax = fmax(pl, pr);
    // (the pressure ratio pmax / pmin <= 2, compared without the quotient)
    if (pmax <= 2.0 * pmin && pmin <= ppv && ppv <= pmax) return ppv;
    if (ppv < pmin) {
        const double icl = ex_rcp(cl), icr = ex_rcp(cr);
        const double pq = ex_pow(pl * ex_rcp(pr), G.g1);
        const double um = (pq * ul * icl + ur * icr + G.g4 * (pq - 1.0)) * ex_rcp(pq * icl + icr);
        const double ptl = 1.0 + G.g7 * (ul - um) * icl;
        const double ptr = 1.0 + G.g7 * (um - ur) * icr;
        return 0.5 * (pl * ex_pow(ptl, G.g3) + pr * ex_pow(ptr, G.g3));
    }
    const double gel = ex_sqrt(G.g5 * ex_rcp(rl * (G.g6 * pl + ppv)));
    const double ger = ex_sqrt(G.g5 * ex_rcp(rr * (G.g6 * pr + ppv)));
    return (gel * pl + ger * pr - (ur - ul)) * ex_rcp(gel + ger);
}

// true if the data generate vacuum (Toro eq. 4.82)
EX_HD bool vacuum(const Gas& G, double ul, double cl, double ur, double cr) { return G.g4 * (cl + cr) <= ur - ul; }

// Newton iteration for p*; returns p*, u*, and per side xl, xr = (p*/p_K)^g1 - 1
// where the last evaluation was on the rarefaction branch, else 2; `iters` =
// updates applied.  p0: starting pressure (<= 0 or non-finite: use the adaptive
// guess).
//
// The last step, at most tol * p, is applied to p and, to first order, to f_L, f_R
// and the powers: what that leaves out is of second order in the step (tol^2
// relative, 1e-24 at the default tolerance, far below a rounding), and it saves the
// evaluation that used to follow, up to two powers of four to six per
// interface.  The step counted is the one that p took after its rounding, so that u* and
// the powers belong to the p* that is returned.
EX_HD void star(const Gas& G, double rl, double ul, double pl, double cl, double rr, double ur, double pr, double cr,
                double p0, double tol, int maxit, double& pstar, double& ustar, int& iters, double& xl, double& xr) {
    iters = 0;
    if (rl == rr && ul == ur && pl == pr) {
        pstar = pl;
        ustar = ul;
        xl = xr = 0.0;
        return;
    }
    double p = p0;
    if (!(p > 0.0) || !(p < 1e300)) p = guess_pvrs(G, rl, ul, pl, cl, rr, ur, pr, cr);
    if (!(p > tol)) p = tol;
    const double du = ur - ul;
    double fl = 0.0, fr = 0.0;
    for (int k = 0; k <= maxit; ++k) {
        double fld, frd;
        prefun(G, p, rl, pl, cl, fl, fld, xl);
        prefun(G, p, rr, pr, cr, fr, frd, xr);
        const double step = (fl + fr + du) * ex_rcp(fld + frd);
        double pn = p - step;
        if (pn < 0.0) pn = tol;
        if (fabs(step) <= tol * p || k == maxit) {
            if (k < maxit) {
                const double taken = p - pn, rel = G.g1 * taken * ex_rcp(p);
                fl = fl - fld * taken;
                fr = fr - frd * taken;
                xl = xl - (1.0 + xl) * rel;
                xr = xr - (1.0 + xr) * rel;
                p = pn;
            }
            break;
        }
        p = pn;
        ++iters;
    }
    pstar = p;
    ustar = 0.5 * (ul + ur + fr - fl);
}
EX_HD void star(const Gas& G, double rl, double ul, double pl, double cl, double rr, double ur, double pr, double cr,
                double p0, double tol, int maxit, double& pstar, double& ustar, int& iters) {
    double xl, xr;
    star(G, rl, ul, pl, cl, rr, ur, pr, cr, p0, tol, maxit, pstar, ustar, iters, xl, xr);
}

// Primitive state at x/t = s of the solution with star values (ps, us)
// (Toro sec. 4.5, SAMPLE).  Also returns the star densities and the two
// acoustic wave speeds used by the wave-propagation correction (shock speed,
// or the mean of head and tail speeds of a rarefaction).
struct Fan {
    double rsl, rsr;  // rho*_L, rho*_R
    double s1, s3;    // left / right acoustic wave speeds (the shock speed of a shock)
    double cml, cmr;  // sound speeds behind a left / right rarefaction (0 for a shock)
};

// Star density and sound speed behind a rarefaction of pressure p_K -> p*, e = star()'s
// (p*/p_K)^g1 - 1: c (1 + e), and rho (p*/p_K)^(1/gamma) = rho p* / (p_K (1 + e)^2)
// (1/gamma = 1 - 2 g1), so no power is taken here.  Down to ratios of 0.7 (e = -0.05) the
// density is formed as the difference from rho, whose terms p* - p_K and p_K e (2 + e) are
// small and exact; beyond, where little is left of rho, as the quotient.  Either quotient is
// corrected by its residual, the roundings of its denominator included.  rms errors of the
// density in units of 1e-17 rho, for ratios within 15% of one, within 60%, over four decades:
// 6.7, 6.9, 9.8; by a power, at the p* of differences of rounded powers, 10.8, 10.6,
// 9.9; by the product of rounded factors there 19.7, 18.8, 15.9.  (What this costs, with
// prefun's difference: six steps at 1024^2 2.14 -> 2.23 ms.)
EX_HD void rarefied(const Gas& G, double ps, double rk, double pk, double ck, double e, double& rs, double& cm) {
    const double x = 1.0 + e;
    const bool weak = e > -0.05;
    const double t = pk * x, den = t * x, r = ex_rcp(den);
    const double n = weak ? fma(-pk, e * (2.0 + e), ps - pk) : ps;
    const double q = n * r;
    const double rem = fma(-q, den, n) - q * (fma(t, x, -den) + fma(pk, x, -t) * x);
    rs = fma(rk, fma(rem, r, q), weak ? rk : 0.0);
    cm = fma(ck, e, ck);
}

EX_HD Fan fan(const Gas& G, double rl, double ul, double pl, double cl, double rr, double ur, double pr, double cr,
              double ps, double us, double xl, double xr) {
    // (A wave is what star's last evaluation took it for.  Where its last step went past p_K,
    // within the tolerance, the shock's relations and the isentrope differ by the cube of
    // that step.)
    Fan F;
    if (xl > 1.0) {
        const double pml = ps * ex_rcp(pl);
        F.rsl = rl * (pml + G.g6) * ex_rcp(pml * G.g6 + 1.0);
        F.s1 = ul - cl * ex_sqrt(G.g2 * pml + G.g1);
        F.cml = 0.0;
    } else {
        rarefied(G, ps, rl, pl, cl, xl, F.rsl, F.cml);
        F.s1 = 0.5 * ((ul - cl) + (us - F.cml));
    }
    if (xr > 1.0) {
        const double pmr = ps * ex_rcp(pr);
        F.rsr = rr * (pmr + G.g6) * ex_rcp(pmr * G.g6 + 1.0);
        F.s3 = ur + cr * ex_sqrt(G.g2 * pmr + G.g1);
        F.cmr = 0.0;
    } else {
        rarefied(G, ps, rr, pr, cr, xr, F.rsr, F.cmr);
        F.s3 = 0.5 * ((ur + cr) + (us + F.cmr));
    }
    return F;
}

// Sample at x/t = 0: returns (rho, u, p) and whether the point is left of the contact.
// The shock speeds and the sound speeds behind the rarefactions are the fan's.
EX_HD void sample0(const Gas& G, double rl, double ul, double pl, double cl, double rr, double ur, double pr, double cr,
                   double ps, double us, const Fan& F, double& r, double& u, double& p, bool& left) {
    const double s = 0.0;
    left = s <= us;
    if (left) {
        if (F.cml > 0.0) {  // (a rarefaction)
            const double shl = ul - cl;
            if (s <= shl) { r = rl; u = ul; p = pl; return; }
            const double stl = us - F.cml;
            if (s > stl) { r = F.rsl; u = us; p = ps; return; }
            u = G.g5 * (cl + G.g7 * ul + s);
            const double c = G.g5 * (cl + G.g7 * (ul - s));
            const double crat = c * ex_rcp(cl);
            const double x = ex_pow(crat, G.g4);
            r = rl * x;
            p = pl * (x * (crat * crat));  // crat^g3, g3 = g4 + 2
        } else {
            const double sl = F.s1;
            if (s <= sl) { r = rl; u = ul; p = pl; }
            else { r = F.rsl; u = us; p = ps; }
        }
    } else {
        if (!(F.cmr > 0.0)) {
            const double sr = F.s3;
            if (s >= sr) { r = rr; u = ur; p = pr; }
            else { r = F.rsr; u = us; p = ps; }
        } else {
            const double shr = ur + cr;
            if (s >= shr) { r = rr; u = ur; p = pr; return; }
            const double str = us + F.cmr;
            if (s <= str) { r = F.rsr; u = us; p = ps; return; }
            u = G.g5 * (-cr + G.g7 * ur + s);
            const double c = G.g5 * (cr - G.g7 * (ur - s));
            const double crat = c * ex_rcp(cr);
            const double x = ex_pow(crat, G.g4);
            r = rr * x;
            p = pr * (x * (crat * crat));
        }
    }
}

// The learned guess's input features and scaling (see pyclaw_b200/learned.py):
// x = (log rho_L/rb, log rho_R/rb, u_L/cb, u_R/cb, log p_L/pb, log p_R/pb) with
// rb = sqrt(rho_L rho_R), pb = sqrt(p_L p_R), cb = sqrt(gamma pb / rb); the
// network predicts y and the guess is p0 * exp(w y), w = J^2/(1+J^2),
// J^2 = (drho/rb)^2 + (dp/pb)^2 + (du/cb)^2, p0 the adaptive guess.
EX_HD void features(const Gas& G, double rl, double ul, double pl, double rr, double ur, double pr, float* x,
                    double& w) {
    const double rb = sqrt(rl * rr), pb = sqrt(pl * pr);
    const double cb = sqrt(G.g * pb / rb);
    const double lr = 0.5 * log(rl / rr), lp = 0.5 * log(pl / pr);
    x[0] = (float)lr;
    x[1] = (float)(-lr);
    x[2] = (float)(ul / cb);
    x[3] = (float)(ur / cb);
    x[4] = (float)lp;
    x[5] = (float)(-lp);
    const double dr = (rr - rl) / rb, dp = (pr - pl) / pb, du = (ur - ul) / cb;
    const double j2 = dr * dr + dp * dp + du * du;
    w = j2 / (1.0 + j2);
}

}  // namespace exact_euler
