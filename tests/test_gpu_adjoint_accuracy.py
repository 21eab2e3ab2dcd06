"""Gradients with deferred factors against binary64: circuits of one and of many
reverse sweeps, with every kind of differentiated gate.  Roundings of the gates
(2^-24 / 2^-47, two states there and back) add in quadrature; eight times that
on a Hamiltonian of coefficient sum c stays far below a term lost or a factor
wrong by a thousandth."""
import math

import numpy as np
import pytest

from kbw_gb300 import DenseGB300
from kbw_gb300 import circuits as C

pytestmark = pytest.mark.gpu

U = {"c64": 2.0 ** -24, "ff": 2.0 ** -47}


@pytest.mark.parametrize("arith", ["c64", "ff"])
@pytest.mark.parametrize("ask", [0, 20])
@pytest.mark.parametrize("n,count", [(13, 60), (13, 700), (16, 300)])
def test_against_binary64(arith, ask, n, count):
    kinds = [C.RX, C.RY, C.RZ, C.P, C.H, C.X, C.Z]
    gates = C.brickwork(n, 1, 4) + C.random_circuit(n, count, n + count, max_controls=1, kinds=kinds)
    index, k = [], 0
    for g in gates:
        index.append(k if g[0] in C.PARAMETRIC else -1)
        k += g[0] in C.PARAMETRIC
    ham = C.tfim_ring(n, 0.8, 0.6) + [(0.5, [(C.PAULI_Y, 1), (C.PAULI_Y, n - 1)])]
    with DenseGB300(n, "c128") as ref:
        e0, g0 = ref.adjoint_gradient(gates, index, k, ham)
    with DenseGB300(n, "c64" if arith == "c64" else "c128", fast_c128=arith == "ff") as sim:
        e1, g1 = sim.adjoint_gradient(gates, index, k, ham, max_checkpoints=ask)
    tol = 8 * math.sqrt(4 * len(gates)) * U[arith] * sum(abs(c) for c, _ in ham)
    assert np.abs(g0).max() > 0.05 and tol < 1e-3
    assert abs(e1 - e0) <= tol and np.abs(g1 - g0).max() <= tol
