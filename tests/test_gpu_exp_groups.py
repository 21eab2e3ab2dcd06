"""<P> of strings summed in tiled passes: flip masks on the lowest bit (pairs
inside one packed operand), low, lane and high bits, several strings with one
flip mask (both parts, with and without signs), registers from below one tile
to several passes, and several Hamiltonians in one call, against the oracle."""
import numpy as np
import pytest

import oracle
from kbw_gb300 import DenseGB300, batch_exp_value
from kbw_gb300 import circuits as C

pytestmark = pytest.mark.gpu

X, Y, Z = C.PAULI_X, C.PAULI_Y, C.PAULI_Z
# sums are FP64-grade (~1e-14 per unit string); the circuits' own rounding is
# 2^-24 resp. 2^-47 per gate over at most 8n = 152 gates, strings summed <= 60
TOL = {"c64": 60 * 152 * 2.0 ** -24, "c128": 1e-11, "ff": 1e-11}


def strings(n):
    rng = np.random.default_rng(n)
    out = [[(X, 0)], [(Y, 0)], [(Y, 0), (Z, 1)], [(X, 0), (Z, n - 1)], [(X, n - 1)], [(Y, n - 1), (Z, 0)]]
    out += [[(p, q), (p, q + 1)] for q in range(n - 1) for p in (X, Y)]
    out += [[(X, 1), (Y, 2)], [(Y, 1), (X, 2)], [(X, 1), (X, 2), (Z, 0)], [(Y, 1), (Y, 2), (Z, 3)], [(X, 1), (Y, 2), (Z, 0)]]
    for _ in range(8):
        k = int(rng.integers(1, 5))
        out.append([(int(rng.integers(1, 4)), int(q)) for q in rng.choice(n, size=k, replace=False)])
    return [(float(rng.uniform(-1, 1)), t) for t in out]


@pytest.mark.parametrize("arith", ["c64", "c128", "ff"])
@pytest.mark.parametrize("n", [5, 8, 9, 10, 12, 13, 14, 19])
def test_strings_one_by_one_and_together(arith, n):
    circ = C.random_circuit(n, 8 * n, 300 + n)
    prec = "c64" if arith == "c64" else "c128"
    sim = DenseGB300(n, prec, fast_c128=arith == "ff")
    sim.apply(circ)
    ref = oracle.OracleDense(n, "c128")
    ref.apply(circ)
    ham = strings(n)
    assert abs(sim.exp_value(ham) - ref.pauli_expect(ham)) < TOL[arith]
    for s in ham[:: max(1, len(ham) // 12)]:
        assert abs(sim.exp_value([s]) - ref.pauli_expect([s])) < TOL[arith]
    hams = [ham, [], [(0.5, [])], [(1.0, [(Z, q)]) for q in range(n)], ham[3:7]]
    got = batch_exp_value(n, circ, hams, prec=prec, fast_c128=arith == "ff")
    want = [ref.pauli_expect(h) if h else 0.0 for h in hams]
    assert np.abs(got - np.array(want)).max() < TOL[arith]
