"""Readout at the sizes where its kernels change: measurements that end in the
one-block tail (from the first step, in the middle, not at all), samples of a
float-float resident state, P(1) of every qubit, against the oracle with the
same draws."""
import numpy as np
import pytest

import oracle
from kbw_gb300 import DenseGB300
from kbw_gb300 import circuits as C

pytestmark = pytest.mark.gpu

TOL = {"c64": 1e-5, "c128": 1e-12, "ff": 1e-12}  # the parity tests' bounds


@pytest.mark.parametrize("arith", ["c64", "c128", "ff"])
@pytest.mark.parametrize("n", [1, 4, 11, 12, 13, 14, 17])
def test_readout(arith, n):
    prec = "c64" if arith == "c64" else "c128"
    rng = np.random.default_rng(n)
    circ = [(C.H, q, (), 0.0) for q in range(n)] + (C.random_circuit(n, 10 * n, 500 + n) if n > 1 else [(C.RY, 0, (), 0.4)])
    for qubits in (list(rng.permutation(n)), list(rng.permutation(n)[: (n + 1) // 2]), [n - 1]):
        qubits = [int(q) for q in qubits]
        sim = DenseGB300(n, prec, fast_c128=arith == "ff")
        ref = oracle.OracleDense(n, prec)
        sim.apply(circ)
        ref.apply(circ)
        for q in range(n):
            assert abs(sim.measure_p1(q) - ref.measure_p1(q)) < TOL[arith]
        if arith != "c64":  # (complex64 prefixes differ by more than a basis state's weight)
            draws = C.uniform_draws(300, n)
            for a, b in zip(sim.sample(qubits, 300, draws), ref.sample(qubits, 300, draws)):
                assert np.array_equal(a, b)
        bits = C.uniform_draws(len(qubits), 7 * n)
        assert sim.measure(qubits, bits) == ref.measure(qubits, bits)
        want = ref.state()
        assert np.linalg.norm(sim.state() - want) < TOL[arith] * np.linalg.norm(want)
