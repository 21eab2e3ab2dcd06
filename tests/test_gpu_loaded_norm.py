"""Gates on states far from unit norm (loaded amplitudes, a collapse with the
caller's factor): a power of two on the state only scales the result, also
through circuits whose deferred factors grow the state most."""
import math

import numpy as np
import pytest

from kbw_gb300 import DenseGB300
from kbw_gb300 import circuits as C

pytestmark = pytest.mark.gpu

N = 13
RNG = np.random.default_rng(5)
TURNS = [(int(RNG.choice([C.RX, C.RY, C.H])), q % N, (), float(math.pi / 2 * (1 if q % 3 else -1))) for q in range(400)]
# rounding per gate 2^-24 / 2^-47 / 2^-53 over 400 gates, in either of the two runs
TOL = {"c64": 800 * 2.0 ** -24, "ff": 800 * 2.0 ** -47, "c128": 800 * 2.0 ** -53}


def handle(arith):
    return DenseGB300(N, "c64" if arith == "c64" else "c128", fast_c128=arith == "ff")


@pytest.mark.parametrize("arith", ["c64", "c128", "ff"])
@pytest.mark.parametrize("power", [-40, 10, 60])
def test_loaded_amplitudes(arith, power):
    a = RNG.standard_normal(1 << N) + 1j * RNG.standard_normal(1 << N)
    a /= np.linalg.norm(a)
    out = []
    for scale in (1.0, 2.0 ** power):
        sim = handle(arith)
        sim.set_state(a * scale)
        sim.apply(TURNS)
        out.append(sim.state().astype(np.complex128) / scale)
    assert np.linalg.norm(out[1] - out[0]) <= TOL[arith]


@pytest.mark.parametrize("arith", ["c64", "c128", "ff"])
def test_collapse_with_a_large_factor(arith):
    out = []
    for p in (2.0 ** 0.5, 2.0 ** 70.5):
        sim = handle(arith)
        sim.apply([(C.H, 0, (), 0.0)])
        sim.measure_collapse(0, False, p)
        sim.apply(TURNS)
        out.append(sim.state().astype(np.complex128) / p * 2.0 ** 0.5)
        sim.clear()  # (the norm is one again)
        sim.apply(TURNS)
        assert abs(np.linalg.norm(sim.state()) - 1.0) <= TOL[arith]
    assert np.linalg.norm(out[1] - out[0]) <= TOL[arith]
