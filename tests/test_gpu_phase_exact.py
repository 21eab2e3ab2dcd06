"""Phase gates a few last places from a power of i: complex128 handles multiply
by the cosine and sine of the angle as given."""
import math

import numpy as np
import pytest

from kbw_gb300 import DenseGB300, _native as N
from kbw_gb300 import circuits as C

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("jit", [N.JIT_OFF, N.JIT_ALWAYS])
@pytest.mark.parametrize("qubit", [0, 6, 12])
def test_angles_next_to_quarter_turns(qubit, jit):
    n = 13
    sim = DenseGB300(n, "c128", jit=jit)
    one = np.zeros(1 << n, np.complex128)
    one[1 << qubit] = 1.0
    for turn in (math.pi / 2, -math.pi / 2, math.pi):
        angle = turn
        for _ in range(4):
            sim.set_state(one)
            sim.apply([(C.P, qubit, (), angle)])
            got = sim.state()[1 << qubit]
            # (the amplitude is 1: the products are exact; the C library rounds both within 2^-53)
            assert abs(got.real - math.cos(angle)) <= 2.0 ** -53 * abs(math.cos(angle))
            assert abs(got.imag - math.sin(angle)) <= 2.0 ** -53
            angle = np.nextafter(angle, 4.0)


@pytest.mark.parametrize("jit", [N.JIT_OFF, N.JIT_ALWAYS])
@pytest.mark.parametrize("n", [11, 13, 14])
def test_sine_of_one(jit, n):
    """Every amplitude of a phase whose sine is +-1 and whose cosine is a rest,
    with and without controls: two products and a sum, each rounded to 2^-53."""
    rng = np.random.default_rng(n)
    a = rng.standard_normal(1 << n) + 1j * rng.standard_normal(1 << n)
    sim = DenseGB300(n, "c128", jit=jit)
    s = np.arange(1 << n)
    for target, control in ((0, ()), (4, (9,)), (6, (2,)), (n - 1, ()), (n - 2, (n - 1, 7))):
        for angle in (math.pi / 2, -math.pi / 2, math.pi / 2 + 1e-8, 1.5 * math.pi):
            sim.set_state(a)
            sim.apply([(C.P, target, control, angle)])
            m = (1 << target) | sum(1 << q for q in control)
            on = (s & m) == m
            c, sn = np.longdouble(math.cos(angle)), np.longdouble(math.sin(angle))
            re, im = np.longdouble(a.real), np.longdouble(a.imag)
            want_re, want_im = np.where(on, re * c - im * sn, re), np.where(on, re * sn + im * c, im)
            got = sim.state()
            size = np.abs(re) + np.abs(im)
            # (the device's constants may be a last place, 2^-53, from the C library's)
            assert (np.abs(got.real - want_re) <= 3 * 2.0 ** -53 * size).all()
            assert (np.abs(got.imag - want_im) <= 3 * 2.0 ** -53 * size).all()
