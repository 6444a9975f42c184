// tpsc_findzero.h -- the reference's root search, for the host and for device
// code whose evaluator is a grid-wide (or block-wide) sum: every thread runs
// the search on the same values, so the control flow is uniform.
#pragma once
#include <math.h>

#ifdef __CUDACC__
#define TPSC_HD __host__ __device__
#else
#define TPSC_HD
#include <cmath>
#endif

namespace tpsc {

#ifndef __CUDACC__
using std::fabs;
using std::isfinite;
using std::sqrt;
#endif

constexpr double kMachEps = 2.220446049250313e-16;

// a double whose operations are rounded one by one (never contracted into
// FMAs), so that the search takes the same iterates on the device as on the host
struct Rn {
    double v;
    TPSC_HD explicit Rn(double x) : v(x) {}
};
#ifdef __CUDA_ARCH__
TPSC_HD inline Rn operator+(Rn a, Rn b) { return Rn(__dadd_rn(a.v, b.v)); }
TPSC_HD inline Rn operator-(Rn a, Rn b) { return Rn(__dsub_rn(a.v, b.v)); }
TPSC_HD inline Rn operator*(Rn a, Rn b) { return Rn(__dmul_rn(a.v, b.v)); }
TPSC_HD inline Rn operator/(Rn a, Rn b) { return Rn(__ddiv_rn(a.v, b.v)); }
#else
TPSC_HD inline Rn operator+(Rn a, Rn b) { return Rn(a.v + b.v); }
TPSC_HD inline Rn operator-(Rn a, Rn b) { return Rn(a.v - b.v); }
TPSC_HD inline Rn operator*(Rn a, Rn b) { return Rn(a.v * b.v); }
TPSC_HD inline Rn operator/(Rn a, Rn b) { return Rn(a.v / b.v); }
#endif
TPSC_HD inline Rn operator-(Rn a) { return Rn(-a.v); }

// the zero of the line through (xm, ym) and (x3, y3)
TPSC_HD inline double secant(double xm, double ym, double x3, double y3) {
    return (-Rn(ym) * (Rn(x3) - Rn(xm)) / (Rn(y3) - Rn(ym)) + Rn(xm)).v;
}

// ---------------------------------------------------------------------------
// Root search with the control flow of generique::find_zero: bracketing
// inverse-quadratic interpolation with secant and bisection fallbacks, tol
// 1e-16 and 20 iterations (src/generique.cpp:604-913); with lims, the bounded
// variant: tol 1e-15, 12 iterations, eps = 2 machine epsilons
// (src/generique.cpp:917-1234).  The evaluator returns false on a device
// error, which aborts the search.
// ---------------------------------------------------------------------------
#ifdef __CUDACC__
#pragma nv_exec_check_disable
#endif
template <typename F>
TPSC_HD bool find_zero(F &&func, const double init[3], double *root, const double *lims, int *nev, bool *dev_err) {
    double tol, eps;
    int itmax;
    if (!lims) {
        tol = 1.0e-16;
        eps = 10.0 * kMachEps;
        itmax = 20;
    } else {
        tol = 1.0e-15;
        eps = 2.0 * kMachEps;
        itmax = 12;
    }
    *nev = 0;
    *dev_err = false;
    auto f = [&](double x, double &y) -> bool {
        ++*nev;
        if (!func(x, y)) {
            *dev_err = true;
            return false;
        }
        return true;
    };
    int nbiter = 0;
    const double dytol = 0.01;
    double x0 = init[0], xmin = init[1], xmax = init[2];
    double ymin, ymax;
    if (!f(xmin, ymin) || !f(xmax, ymax)) return false;
    double x[3] = {x0, xmin, xmax}, y[3] = {0.0, ymin, ymax};
    if (fabs(ymin) < tol) {
        *root = xmin;
        return true;
    }
    if (fabs(ymax) < tol) {
        *root = xmax;
        return true;
    }
    if (ymin * ymax > 0) {
        if (!f(x[0], y[0])) return false;
        if (fabs(y[0]) < tol) {
            *root = x[0];
            return true;
        }
        if (y[0] * y[2] < 0) {
            const double xt = x[0];
            x[0] = (x[0] + x[2]) / 2;
            x[1] = xt;
            y[1] = y[0];
        } else {
            double ytmp = y[0], xtmp = x[0], xtmp1, ytmp1;
            if (fabs(y[1]) < fabs(ytmp)) ytmp = y[1], xtmp = x[1];
            if (fabs(y[2]) < fabs(ytmp)) ytmp = y[2], xtmp = x[2];
            xtmp1 = xtmp + 10 * eps;
            if (!f(xtmp1, ytmp1)) return false;
            xtmp1 = (Rn(xtmp) - Rn(ytmp) * ((Rn(xtmp1) - Rn(xtmp)) / (Rn(ytmp1) - Rn(ytmp)))).v;
            if (!f(xtmp1, ytmp1)) return false;
            nbiter++;
            while (fabs(ytmp1) > tol && nbiter < itmax && ytmp1 * ytmp > 0 && isfinite(xtmp1)) {
                xtmp = xtmp1;
                ytmp = ytmp1;
                xtmp1 = xtmp + 10 * eps;
                if (!f(xtmp1, ytmp1)) return false;
                xtmp1 = (Rn(xtmp) - Rn(ytmp) * ((Rn(xtmp1) - Rn(xtmp)) / (Rn(ytmp1) - Rn(ytmp)))).v;
                if (!f(xtmp1, ytmp1)) return false;
                nbiter++;
            }
            if (fabs(ytmp1) < tol) {
                *root = xtmp1;
                return true;
            }
            if (ytmp1 * ytmp < 0) {
                x[0] = (xtmp + xtmp1) / 2;
                x[1] = xtmp;
                y[1] = ytmp;
                x[2] = xtmp1;
                y[2] = ytmp1;
            }
            if (nbiter >= itmax) return false;
            if (!isfinite(xtmp1)) return false;
        }
    }
    if (lims) {
        if (x[1] < lims[0] || x[1] > lims[1] || x[2] < lims[0] || x[2] > lims[1]) return false;
    }
    if (fabs(xmax - xmin) < eps) {
        *root = xmin;
        return true;
    }
    if (!f(x[0], y[0])) return false;
    if (fabs(y[0]) < tol) {
        *root = x[0];
        return true;
    }
    int ind1, ind2, ind3, indm = 0, indp = 0, indfar, indmid;
    auto classify = [&]() {
        if (y[0] * y[1] > 0)
            ind1 = 0, ind2 = 1;
        else if (y[0] * y[2] > 0)
            ind1 = 0, ind2 = 2;
        else
            ind1 = 1, ind2 = 2;
        ind3 = 3 - ind1 - ind2;
        if (x[ind3] > x[ind1]) {
            if (x[ind1] > x[ind2])
                indfar = ind2, indmid = ind1;
            else
                indfar = ind1, indmid = ind2;
            indm = indmid, indp = ind3;
        } else {
            if (x[ind1] < x[ind2])
                indfar = ind2, indmid = ind1;
            else
                indfar = ind1, indmid = ind2;
            indm = ind3, indp = indmid;
        }
    };
    classify();
    x[indfar] = secant(x[indmid], y[indmid], x[ind3], y[ind3]);
    if (!f(x[indfar], y[indfar])) return false;
    double dy = y[indfar], dyprec;
    Rn a(0.0), b(0.0), c(0.0);
    while (fabs(dy) > tol && nbiter < itmax) {
        classify();
        const Rn x0r(x[0]), x1r(x[1]), x2r(x[2]), y0r(y[0]), y1r(y[1]), y2r(y[2]);
        const Rn den = -x0r * x0r * x2r + x0r * x0r * x1r - x0r * x1r * x1r + x0r * x2r * x2r - x2r * x2r * x1r +
                       x2r * x1r * x1r;
        const double denom = den.v;
        if (fabs(denom) > 0.0) {
            a = (x0r * y2r - x0r * y1r + x2r * y1r - y2r * x1r - y0r * x2r + y0r * x1r) / den;
            b = -(-y2r * x1r * x1r + x1r * x1r * y0r - x2r * x2r * y0r - y1r * x0r * x0r + y2r * x0r * x0r +
                  y1r * x2r * x2r) /
                den;
            c = (y2r * x0r * x0r * x1r - y1r * x0r * x0r * x2r - x1r * x1r * x0r * y2r + x2r * x2r * x0r * y1r +
                 x1r * x1r * y0r * x2r - x2r * x2r * y0r * x1r) /
                den;
        }
        const double disc = (b * b - Rn(4.0) * a * c).v;
        if (disc > 0.0 && fabs(denom) > 0.0) {
            const Rn sq(sqrt(disc)), two_a = Rn(2.0) * a;
            const double xp = ((-b + sq) / two_a).v, xm = ((-b - sq) / two_a).v;
            if (xp > x[indm] && xp < x[indp])
                x[indfar] = xp;
            else if (xm > x[indm] && xm < x[indp])
                x[indfar] = xm;
            else if (fabs(y[ind3] - y[indmid]) > tol)
                x[indfar] = secant(x[indmid], y[indmid], x[ind3], y[ind3]);
            else {
                *root = x[indmid];
                return true;
            }
        } else {
            if (fabs(y[ind3] - y[indmid]) > tol)
                x[indfar] = secant(x[indmid], y[indmid], x[ind3], y[ind3]);
            else {
                *root = x[indmid];
                return true;
            }
        }
        if (!f(x[indfar], y[indfar])) return false;
        dyprec = fabs(dy);
        dy = y[indfar];
        if (fabs(dyprec - fabs(dy)) < dytol * dyprec || dyprec < fabs(dy)) {
            x[indfar] = (x[ind3] + x[indmid]) / 2.0;
            if (!f(x[indfar], y[indfar])) return false;
            dy = y[indfar];
        }
        nbiter++;
    }
    int best = 0;
    *root = x[0];
    if (fabs(y[1]) < fabs(y[best])) {
        *root = x[1];
        best = 1;
    }
    if (fabs(y[2]) < fabs(y[best])) *root = x[2];
    return true;
}

}  // namespace tpsc
