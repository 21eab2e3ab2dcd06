// Host check of the deferred gate factors (kbw_gb300/csrc/dd.h) against long
// double on seeded angles.  Prints the worst deviations as "name value" lines;
// tests/test_dd_host.py holds the bounds.
//
//   factor      the factor of RZ against the unit phase it stands for
//   rest        factor * (c + i s) against the |1> phase of RZ, brought to unit size
//   norm        | |factor * (c + i s)| - 1 |
//   unit        dd_unit(w) against 1 / sqrt(1 + w^2), relative
#include <math.h>
#include <stdio.h>
#include <stdlib.h>

#include <algorithm>
#include <complex>
#include <random>

#include "../../kbw_gb300/csrc/dd.h"

using namespace kbwg;
typedef std::complex<long double> C;

static long double val(Dd v) { return (long double)v.h + (long double)v.l; }

int main(int argc, char **argv) {
    const long count = argc > 1 ? atol(argv[1]) : 100000;
    std::mt19937_64 rng(7);
    std::uniform_real_distribution<double> U(-7.0, 7.0);
    long double factor = 0, rest = 0, norm = 0, unit = 0;
    for (long i = 0; i < count; i++) {
        const double h = 0.5 * U(rng), u[4] = {cos(-h), sin(-h), cos(h), sin(h)};
        const DeferredDiagonal d = defer_diagonal(u);
        C a(u[0], u[1]), b(u[2], u[3]);
        a /= std::abs(a);
        b /= std::abs(b);
        const C f(val(d.f.re), val(d.f.im)), one = f * C(d.c, d.s);
        factor = std::max(factor, std::abs(f - a));
        rest = std::max(rest, std::abs(one - b));
        norm = std::max(norm, fabsl(std::abs(one) - 1.0L));
        const double w = U(rng) / 7.0;
        unit = std::max(unit, fabsl(val(dd_unit(w)) * sqrtl(1.0L + (long double)w * w) - 1.0L));
    }
    printf("factor %.6Le\nrest %.6Le\nnorm %.6Le\nunit %.6Le\n", factor, rest, norm, unit);
    return 0;
}
