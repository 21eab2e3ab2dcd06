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
