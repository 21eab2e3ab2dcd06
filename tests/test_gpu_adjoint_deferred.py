"""Adjoint gradient with deferred gate factors: sweeps with more growing gates
than one run of deferred factors takes, several checkpoint segments, controls,
every gate kind, angles where a coefficient vanishes; against the
parameter-shift rule on the binary64 engine."""
import math

import numpy as np
import pytest

from kbw_gb300 import DenseGB300, _native as N
from kbw_gb300 import circuits as C

pytestmark = pytest.mark.gpu

# energies of unit-norm strings with coefficients summing below 40; rounding
# 2^-24 / 2^-47 / 2^-53 per gate, twice 700 gates forward and back, linearly
TOL = {"c64": 40 * 1400 * 2.0 ** -24, "ff": 40 * 1400 * 2.0 ** -47, "c128": 40 * 1400 * 2.0 ** -53}


def circuit(n, gates, seed):
    rng = np.random.default_rng(seed)
    circ, index, k = [], [], 0
    for i in range(gates):
        kind = int(rng.choice([C.H, C.X, C.Y, C.Z, C.RX, C.RY, C.RY, C.RZ, C.P]))
        t = int(rng.integers(n))
        ctrl = (int((t + 1 + rng.integers(n - 1)) % n),) if rng.random() < 0.2 else ()
        a = 0.0
        if kind in C.PARAMETRIC:
            a = float(rng.choice([0.0, math.pi, math.pi / 2, -math.pi])) if rng.random() < 0.2 else float(rng.uniform(-4, 4))
        take = kind in C.PARAMETRIC and not ctrl and rng.random() < 0.3
        circ.append((kind, t, ctrl, a))
        index.append(k if take else -1)
        k += take
    return circ, index, k


@pytest.mark.parametrize("n,gates", [(13, 40), (13, 300), (14, 700)])
def test_against_parameter_shift(n, gates):
    circ, index, k = circuit(n, gates, n + gates)
    ham = C.tfim_ring(n, 1.0, 0.5) + [(0.3, [(C.PAULI_Y, 0), (C.PAULI_Y, n - 1)])]
    ref = DenseGB300(n, "c128", jit=N.JIT_OFF)
    e0, g0 = ref.param_shift_gradient(circ, index, k, ham)
    for arith in ("c128", "ff", "c64"):
        for jit in (N.JIT_OFF, N.JIT_ALWAYS) if gates == 40 else (N.JIT_OFF,):
            sim = DenseGB300(n, "c64" if arith == "c64" else "c128", fast_c128=arith == "ff", jit=jit)
            e, g = sim.adjoint_gradient(circ, index, k, ham)
            assert abs(e - e0) < TOL[arith] and np.abs(g - g0).max() < TOL[arith]
            e2, g2 = sim.adjoint_gradient(circ, index, k, ham, max_checkpoints=0)
            assert e2 == e or abs(e2 - e0) < TOL[arith]
            assert np.abs(g2 - g0).max() < TOL[arith]
