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

struct DdComplex {
    Dd re, im;
};

// A complex factor g collected from gates.
struct DdFactor {
    Dd re{1.0, 0.0}, im;
    bool used = false;
    void times(Dd f) {
        used = true;
        re = dd_mul(re, f);
        im = dd_mul(im, f);
    }
    void times(const DdComplex &f) {
        used = true;
        const Dd nr = dd_add(dd_mul(re, f.re), dd_mul(im, Dd{-f.im.h, -f.im.l}));
        im = dd_add(dd_mul(re, f.im), dd_mul(im, f.re));
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

// A diagonal diag(u0, u1) of two phases, rounded: u0 as the factor f, the rest
// diag(1, c + i s).  Both are brought to unit size first (with e = |u|^2 - 1
// of a few last places, 1 - e / 2), or the |1> side would carry twice the
// rounding of |u0| besides its own (binary64 brickwork of 16 qubits, 8 layers,
// against 80-bit arithmetic: 5.1-9.2e-16, so 4.8-5.4e-16).
struct DeferredDiagonal {
    DdComplex f;
    double c, s;
};
inline DeferredDiagonal defer_diagonal(const double u[4]) {
    auto unit = [](double re, double im) {
        const Dd r{re, 0.0}, i{im, 0.0};
        const Dd e = dd_add(dd_add(dd_mul(r, r), dd_mul(i, i)), Dd{-1.0, 0.0});
        const Dd k = dd_add(Dd{1.0, 0.0}, Dd{-0.5 * e.h, -0.5 * e.l});
        return DdComplex{dd_mul(r, k), dd_mul(i, k)};
    };
    const DdComplex a = unit(u[0], u[1]), b = unit(u[2], u[3]);
    const Dd na{-a.im.h, -a.im.l};
    DeferredDiagonal d;
    d.f = a;
    d.c = dd_add(dd_mul(b.re, a.re), dd_mul(b.im, a.im)).h;
    d.s = dd_add(dd_mul(b.im, a.re), dd_mul(b.re, na)).h;
    return d;
}

}  // namespace kbwg
