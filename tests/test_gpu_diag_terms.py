"""Strings without flips, summed two terms to a packed instruction: one term,
odd counts, full and overfull groups, masks on lane, run and high bits, on
registers of one 512-amplitude run and of many, against the oracle."""
import numpy as np
import pytest

import oracle
from kbw_gb300 import DenseGB300, batch_exp_value
from kbw_gb300 import circuits as C

pytestmark = pytest.mark.gpu

# sums are FP64-grade; the circuit rounds 2^-24 resp. 2^-47 per gate over 4n <= 76 gates, both parts
TOL = {"c64": 2 * 76 * 2.0 ** -24, "c128": 1e-11, "ff": 1e-11}


@pytest.mark.parametrize("arith", ["c64", "c128", "ff"])
@pytest.mark.parametrize("n", [9, 11, 13, 19])
def test_term_counts(arith, n):
    rng = np.random.default_rng(n)
    circ = C.random_circuit(n, 4 * n, 700 + n)
    prec = "c64" if arith == "c64" else "c128"
    ref = oracle.OracleDense(n, "c128")
    ref.apply(circ)
    masks = []
    while len(masks) < 65:
        m = int(rng.integers(1, 1 << n)) if len(masks) >= n else 1 << len(masks)
        if m not in masks:
            masks.append(m)
    terms = [[(C.PAULI_Z, q) for q in range(n) if m >> q & 1] for m in masks]
    want = np.array([ref.pauli_expect([(1.0, t)]) for t in terms])
    sim = DenseGB300(n, prec, fast_c128=arith == "ff")
    sim.apply(circ)
    for count in (1, 2, 3, 31, 32, 33, 65):
        sign = np.where(np.arange(count) % 3 == 1, -1.0, 1.0)
        got = sim.exp_value([(float(s), t) for s, t in zip(sign, terms)])
        assert abs(got - float(sign @ want[:count])) < count * TOL[arith]
        each = batch_exp_value(n, circ, [[(1.0, t)] for t in terms[:count]], prec=prec, fast_c128=arith == "ff")
        assert np.abs(each - want[:count]).max() < TOL[arith]
