"""Uniform factors of gates left to one multiplication of the state (H's
1/sqrt(2), RZ's phase, the larger of cos and sin of an RX/RY) against the
restated Dense: every rotation form at the angles where it changes, targets on
lane, register and warp bits and outside the tile, lists short enough to keep
the full forms and long enough to be rescaled in between, interpreted and
specialised kernels."""
import math

import numpy as np
import pytest

import oracle
from kbw_gb300 import DenseGB300, _native as N
from kbw_gb300 import circuits as C

pytestmark = pytest.mark.gpu

# at pi/2 + k pi of the full angle the two forms meet, at k pi a coefficient vanishes
ANGLES = [0.0, math.pi / 2, -math.pi / 2, math.pi, -math.pi, 2 * math.pi, 3 * math.pi, math.pi / 2 + 1e-9,
          math.pi - 1e-7, 1e-7, 3.5 * math.pi, -5.9]
# rounding per gate 2^-24 (complex64) / 2^-47 (float-float) / 2^-53, at most 500
# gates in these circuits and errors adding at worst linearly
TOL = {"c64": 500 * 2.0 ** -24, "ff": 500 * 2.0 ** -47, "c128": 500 * 2.0 ** -53}


def rotations(n, count, seed, kinds):
    rng = np.random.default_rng(seed)
    out = []
    for i in range(count):
        kind = int(rng.choice(kinds))
        a = ANGLES[int(rng.integers(len(ANGLES)))] if rng.random() < 0.7 else float(rng.uniform(-7, 7))
        t = int(rng.integers(n))
        ctrl = ()
        if rng.random() < 0.15:
            ctrl = (int((t + 1 + rng.integers(n - 1)) % n),)
        out.append((kind, t, ctrl, a if kind in C.PARAMETRIC else 0.0))
    return out


def check(n, arith, circ, jit):
    prec = "c64" if arith == "c64" else "c128"
    sim = DenseGB300(n, prec, fast_c128=arith == "ff", jit=jit)
    ref = oracle.OracleDense(n, "c128")
    for part in (C.brickwork(n, 1, 5), circ):
        sim.apply(part)
        ref.apply(part)
        sim.flush()
    got, want = sim.state(), ref.state()
    assert np.linalg.norm(got - want) / np.linalg.norm(want) < TOL[arith]


@pytest.mark.parametrize("arith", ["c64", "c128", "ff"])
@pytest.mark.parametrize("n,count", [(11, 40), (13, 1), (13, 2), (13, 3), (14, 430), (16, 60)])
def test_interpreted(arith, n, count):
    check(n, arith, rotations(n, count, 3 * n + count, [C.RX, C.RY, C.RZ, C.H, C.P]), N.JIT_OFF)


@pytest.mark.parametrize("arith", ["c64", "c128", "ff"])
@pytest.mark.parametrize("kinds", [[C.RX], [C.RY], [C.RX, C.RY, C.RZ, C.H, C.X]])
def test_specialised(arith, kinds):
    check(15, arith, rotations(15, 60, 9 + len(kinds), kinds), N.JIT_ALWAYS)


@pytest.mark.parametrize("arith", ["c64", "ff"])
def test_many_cotangents_stay_in_range(arith):
    # every gate at its largest growth: pi/2 turns, far beyond one run of deferred factors
    n = 13
    circ = [(C.RY, q % n, (), math.pi / 2 * (1 if q % 3 else -1)) for q in range(420)]
    check(n, arith, circ, N.JIT_OFF)
