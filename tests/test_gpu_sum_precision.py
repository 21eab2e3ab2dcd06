"""How exactly expectation values are summed: states whose sums are known in
wide arithmetic, with bounds from the roundings of a binary64 sum."""
import numpy as np
import pytest

from kbw_gb300 import DenseGB300
from kbw_gb300 import circuits as C

pytestmark = pytest.mark.gpu

X, Y, Z = C.PAULI_X, C.PAULI_Y, C.PAULI_Z
U = 2.0 ** -53


@pytest.mark.parametrize("n", [9, 10])
@pytest.mark.parametrize("string", [[(X, 0)], [(Y, 3), (Z, 1)], [(X, 2), (X, 8)]])
def test_one_pair_of_a_small_complex128_register(n, string):
    """One pair of amplitudes: two products, their sum, each rounded once to
    binary64 (twice the value and its sign are exact)."""
    x = sum(1 << q for p, q in string if p in (X, Y))
    sim = DenseGB300(n, "c128")
    rng = np.random.default_rng(n)
    for _ in range(25):
        s = int(rng.integers(1 << n))
        a = np.zeros(1 << n, np.complex128)
        a[s], a[s ^ x] = rng.standard_normal(2) + 1j * rng.standard_normal(2)
        sim.set_state(a)
        got = sim.exp_value([(1.0, string)])
        lo, hi = min(s, s ^ x), max(s, s ^ x)
        re, im = np.longdouble(a.real), np.longdouble(a.imag)
        parts = (re[lo] * re[hi], im[lo] * im[hi]) if string[0][0] == X else (re[lo] * im[hi], -im[lo] * re[hi])
        want = 2 * sum(parts)
        sign = 1 if abs(got - want) < abs(got + want) else -1  # (signs: the parity tests)
        assert abs(got - sign * want) <= 3 * U * 2 * sum(abs(p) for p in parts)


@pytest.mark.parametrize("prec", ["c64", "c128"])
@pytest.mark.parametrize("n,string", [(9, [(Z, 0)]), (9, [(Z, 4), (Z, 7)]), (12, [(X, 0)]), (12, [(Y, 1), (Z, 2)])])
def test_shares_of_a_warp(prec, n, string):
    """Amplitudes of few bits, scaled by lane: every thread's share is exact in
    a float and the sum takes more than the 48 bits of float-float; only the
    result is rounded, in the three conversions of its parts."""
    pair = any(p != Z for p, q in string)
    lanes = np.arange(1 << n) // 8 if pair else np.arange(1 << n) % 32  # (the 8 amplitudes of a window; every 32nd)
    used = lanes < 32
    x = sum(1 << q for p, q in string if p in (X, Y))
    z = sum(1 << q for p, q in string if p in (Y, Z))
    s = np.arange(1 << n)
    sign = 1 - 2 * (np.bitwise_count((s ^ x) & z).astype(np.int64) & 1)
    sim = DenseGB300(n, prec)
    for seed in range(20):
        rng = np.random.default_rng([n, seed])
        re, im = rng.integers(-1023, 1024, (2, 1 << n))
        scale = 2.0 ** -(lanes % 14) * used * 2.0 ** -12
        sim.set_state((re + 1j * im) * scale)
        ar, ai = np.longdouble(re) * scale, np.longdouble(im) * scale
        br, bi = ar[s ^ x], ai[s ^ x]
        odd = any(p == Y for p, q in string)
        parts = (np.array([ar * bi, -ai * br]) if odd else np.array([ar * br, ai * bi])) * sign
        want = parts.sum()
        got = sim.exp_value([(1.0, string)])
        if odd:  # (i^ny of one Y)
            got = -got if abs(got + want) < abs(got - want) else got
        assert abs(got - want) <= 3 * U * np.abs(parts).sum()


def _pick(sim, n, draw):
    states, counts = sim.sample(list(range(n))[::-1], 1, [draw])
    return int(states[0])


@pytest.mark.parametrize("arith", ["c64", "c128", "ff"])
def test_border_between_two_samples(arith):
    """Two weights in blocks of their own, and draws a few last places around
    their border: weights, total and the drawn weight as binary64 rounds them
    (re^2 of a float is exact there, re^2 + im^2 rounded once)."""
    n, rng = 14, np.random.default_rng(4)
    sim = DenseGB300(n, "c64" if arith == "c64" else "c128", fast_c128=arith == "ff")
    for _ in range(40):
        a = np.zeros(1 << n, np.complex64)
        a[0], a[-1] = (rng.uniform(0.3, 1.0, 2) + 1j * rng.uniform(0.3, 1.0, 2)).astype(np.complex64)
        sim.set_state(a)
        if arith == "ff":
            sim.apply([(C.X, 3, (), 0.0)])  # (exact: the two states swap bit 3)
        w = (np.longdouble(a.real) ** 2 + np.longdouble(a.imag) ** 2).astype(np.float64)
        total = w[0] + w[-1]
        scale = total
        while scale * (1.0 - np.finfo(np.float64).eps) >= total:
            scale = np.nextafter(scale, 0.0)
        first, last = (8, (1 << n) - 9) if arith == "ff" else (0, (1 << n) - 1)
        draw = w[0] / scale
        for _ in range(4):
            draw = np.nextafter(draw, 0.0)
        for _ in range(9):
            assert _pick(sim, n, draw) == (first if draw * scale < w[0] else last)
            draw = np.nextafter(draw, 1.0)


@pytest.mark.parametrize("arith", ["c64", "ff"])
@pytest.mark.parametrize("size", [1e25, 1e-13])
def test_samples_far_from_unit_norm(arith, size):
    """Weights beyond float's range."""
    n = 12
    if arith == "c64" and size < 1:
        size = 1e-4  # (complex64 drops amplitudes below 1e-6)
    a = np.zeros(1 << n, np.complex128)
    a[5], a[4000] = 3 * size, 4j * size
    sim = DenseGB300(n, "c64" if arith == "c64" else "c128", fast_c128=arith == "ff")
    sim.set_state(a)
    sim.apply([(C.X, 0, (), 0.0)])
    assert [_pick(sim, n, d) for d in (0.1, 0.35, 0.37, 0.9)] == [4, 4, 4001, 4001]


def test_energy_of_a_gradient_of_two_amplitudes():
    """lambda = Z psi is exact, and psi two complex amplitudes: their squares
    (exact in binary64), the sum of each pair, and the difference."""
    n, rng = 12, np.random.default_rng(8)
    sim = DenseGB300(n, "c64")
    for _ in range(50):
        gates = [(C.RY, 0, (), float(rng.uniform(0.5, 1.0))), (C.RZ, 0, (), float(rng.uniform(0.5, 1.0)))]
        sim.clear()
        sim.apply(gates)
        a = sim.state()
        w = np.longdouble(a.real) ** 2 + np.longdouble(a.imag) ** 2
        e, _ = sim.adjoint_gradient(gates, [0, 1], 2, [(1.0, [(Z, 0)])])
        assert abs(e - (w[0] - w[1])) <= 3 * U * (w[0] + w[1])
