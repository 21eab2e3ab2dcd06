// Products of many gate factors on the host, as unevaluated sums of two
// doubles: rounded once, at the end (in plain binary64 the product of a few
// hundred factors would round worse than the gates themselves).
#pragma once

#include <math.h>

#include "ff.cuh"

namespace kbwg {

struct Dd {
    double h = 0.0, l = 0.0;
};
inline Dd dd_mul(Dd a, Dd b) {
    const double p = a.h * b.h, e = fma(a.h, b.h, -p) + (a.h * b.l + a.l * b.h), s = p + e;
    return Dd{s, e - (s - p)};
}
inline Dd dd_add(Dd a, Dd b) {
    const double s = a.h + b.h, bb = s - a.h, e = ((a.h - (s - bb)) + (b.h - bb)) + (a.l + b.l), r = s + e;
    return Dd{r, e - (r - s)};
}
// 1 / sqrt(1 + w^2) for |w| <= 1: the rounded value and one Newton step's correction
inline Dd dd_unit(double w) {
    const double w2 = w * w, w2e = fma(w, w, -w2), sh = 1.0 + w2, sl = (w2 - (sh - 1.0)) + w2e;
    const double r = 1.0 / sqrt(sh), r2 = r * r, r2e = fma(r, r, -r2);
    const double e = fma(-r2, sh, 1.0) - (r2 * sl + r2e * sh);
    return Dd{r, 0.5 * r * e};
}

// A complex factor g collected from gates.
struct DdFactor {
    Dd re{1.0, 0.0}, im;
    bool used = false;
    void times(Dd f) {
        used = true;
        re = dd_mul(re, f);
        im = dd_mul(im, f);
    }
    void times(double c, double s) {  // c + i s
        used = true;
        const Dd r{c, 0.0}, i{s, 0.0}, ni{-s, 0.0};
        const Dd nr = dd_add(dd_mul(re, r), dd_mul(im, ni));
        im = dd_add(dd_mul(re, i), dd_mul(im, r));
        re = nr;
    }
};

// x as a program's constants hold it: float (complex64), two floats
// (float-float) or binary64.
enum { ARITH_C64 = 0, ARITH_F64 = 1, ARITH_FF = 2 };
inline double packed_value(int arith, double x) {
    if (arith == ARITH_C64) return (double)(float)x;
    if (arith == ARITH_FF) {
        const ff::f2 v = ff::split_constant(x);
        return (double)v.h + (double)v.l;
    }
    return x;
}

// RX/RY with cos c and sin s of the half angle, the larger one dropped: the
// coefficient left (rounded as packed), whether it is the cotangent, and the
// factor that makes the gate a rotation again.
struct DeferredRotation {
    double w;
    bool cot;
    Dd factor;
};
inline DeferredRotation defer_rotation(int arith, double c, double s) {
    DeferredRotation r;
    r.cot = !(fabs(c) >= fabs(s));
    r.w = packed_value(arith, r.cot ? c / s : s / c);
    r.factor = dd_unit(r.w);
    if ((r.cot ? s : c) < 0.0) r.factor = Dd{-r.factor.h, -r.factor.l};
    return r;
}

// A diagonal diag(u0, u1), |u0| = 1, as u0 diag(1, c + i s).
inline void defer_diagonal(const double u[4], double &c, double &s) {
    const Dd ur{u[0], 0.0}, ui{u[1], 0.0}, nui{-u[1], 0.0}, vr{u[2], 0.0}, vi{u[3], 0.0};
    c = dd_add(dd_mul(vr, ur), dd_mul(vi, ui)).h;
    s = dd_add(dd_mul(vi, ur), dd_mul(vr, nui)).h;
}

}  // namespace kbwg
