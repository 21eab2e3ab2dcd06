"""Gradients of Hamiltonians with large coefficients: a power of two on the
whole Hamiltonian only scales energy and gradient, also where the reverse
sweeps' deferred factors multiply lambda."""
import numpy as np
import pytest

from kbw_gb300 import DenseGB300
from kbw_gb300 import circuits as C

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("arith", ["c64", "c128", "ff"])
@pytest.mark.parametrize("power", [31, 60, 110])
def test_scaled_hamiltonian(arith, power):
    n = 13
    rng = np.random.default_rng(power)
    # quarter turns grow the states most: eighty of them in one sweep
    gates = [(C.RY if i % 2 else C.RX, int(rng.integers(11)), (), float(np.pi / 2 + 0.01 * rng.uniform(-1, 1)))
             for i in range(160)]
    index = list(range(160))
    ham = C.tfim_ring(n, 1.0, 0.5)
    sim = DenseGB300(n, "c64" if arith == "c64" else "c128", fast_c128=arith == "ff")
    e0, g0 = sim.adjoint_gradient(gates, index, 160, ham)
    e1, g1 = sim.adjoint_gradient(gates, index, 160, [(c * 2.0 ** power, t) for c, t in ham])
    # (only subnormal numbers round differently: 2^-149 of 2^13 amplitudes, far below this)
    tol = 1e-16 * sum(abs(c) for c, _ in ham)
    assert np.isfinite(g0).all() and abs(e1 * 2.0 ** -power - e0) <= tol
    assert np.abs(g1 * 2.0 ** -power - g0).max() <= tol
