// The spline knots that a straight orbit passes: collected into a list (the
// Gauss rule's segments) or walked one after the other (the closed form's).
// Host and device, so that the walk's ends can be checked without a GPU.
#pragma once

#include <math.h>

#include "upic_common.cuh"

namespace upic {

// Knot crossings per particle orbit that the device kernels can hold
// (breakpoints of both axes plus the two ends).
constexpr int kMaxBreaks = 40;

// An orbit of more cells than this along an axis passes at least kKnotReach - 2
// of its knots, more than kMaxBreaks: it fails before any knot is looked at.
// Both searches below would otherwise step from knot to knot until the first
// one more than 1e-13 along the orbit, which for a displacement of 1e24 cells
// takes 1e11 steps and for an infinite one never ends.  (A NaN displacement
// passes: both searches find no knot in it.)
constexpr double kKnotReach = 64.0;
static_assert(kKnotReach - 2.0 > kMaxBreaks, "such an orbit has to fail for its knots");
UPIC_HD bool beyond_reach(double du) { return fabs(du) > kKnotReach; }

// Appends the fractions at which the orbit a0 + s du (knots at the integers)
// passes a knot of one axis to b[0..nb); false when there are too many.
UPIC_HD bool axis_breaks(double a0, double du, double* b, int& nb) {
    const double tol = 1.0e-13;
    if (beyond_reach(du)) return false;
    const double a1 = a0 + du;
    const double lo = fmin(a0, a1), hi = fmax(a0, a1);
    const long long first = (long long)floor(lo) + 1;
    const long long last = (long long)ceil(hi) - 1;
    for (long long m = first; m <= last; ++m) {
        const double s = ((double)m - a0) / du;
        if (s > tol && s < 1.0 - tol) {
            if (nb >= kMaxBreaks) return false;
            b[nb++] = s;
        }
    }
    return true;
}

// The next knot (integer) that an orbit u0 + s du passes along one axis after
// fraction s (2: none in (0, 1)); s = 0 for the first
// (path_breakpoints_for_particle :2555).  Only s is kept between calls: the
// knot passed at s is the integer nearest u0 + s du.  Needs an orbit within
// reach.
UPIC_HD double next_knot(double u0, double du, double s) {
    const double step = du > 0.0 ? 1.0 : -1.0;
    double m = s > 0.0 ? rint(fma(s, du, u0)) + step : du > 0.0 ? floor(u0) + 1.0 : ceil(u0) - 1.0;
    for (;;) {
        if (fabs(du) < 1.0e-300 || !((m - (u0 + du)) * step < 0.0)) return 2.0;
        s = (m - u0) / du;
        if (s > 1.0e-13) return s < 1.0 - 1.0e-13 ? s : 2.0;
        m += step;
    }
}

// The segments of an orbit between its knots, one after the other; knots
// closer than 1e-12 count once, and more than kMaxBreaks end points fail.
struct KnotWalk {
    double sx, sy, prev;
    int nb;  // end points so far; 0 when no segment is left, -1 when there were too many
    UPIC_HD void init(double ux, double uy, double dux, double duy) {
        sx = sy = 2.0;
        prev = 0.0;
        nb = -1;
        if (beyond_reach(dux) || beyond_reach(duy)) return;
        sx = next_knot(ux, dux, 0.0);
        sy = next_knot(uy, duy, 0.0);
        nb = 2;
    }
    UPIC_HD bool more() const { return nb > 0; }
    UPIC_HD bool next(double ux, double uy, double dux, double duy, double& sa, double& sb) {
        while (nb > 0) {
            double s = fmin(sx, sy);
            if (s < 1.0) {
                const bool ex = sx == s, ey = sy == s;
                if (ex) sx = next_knot(ux, dux, s);
                if (ey) sy = next_knot(uy, duy, s);
                nb += (ex ? 1 : 0) + (ey ? 1 : 0);
                if (nb > kMaxBreaks) {
                    nb = -1;
                    return false;
                }
            } else {
                s = 1.0;
                nb = 0;
            }
            if (s - prev > 1.0e-12) {
                sa = prev;
                sb = s;
                prev = s;
                return true;
            }
        }
        return false;
    }
};

}  // namespace upic
