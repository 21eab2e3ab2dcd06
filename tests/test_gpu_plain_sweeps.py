"""Sweeps without deferred rotations and merged signs (a kernel of their own in
complex64 and float-float) against the oracle, alone and between sweeps that
hold some, on every tile; large lists with few gates to defer against binary64;
merged signs and 64-bit state indices on 33 qubits."""
import gc
import math

import numpy as np
import pytest

import oracle
from kbw_gb300 import DenseGB300, _native as N, batch_release
from kbw_gb300 import circuits as C

pytestmark = pytest.mark.gpu

# rounding per gate 2^-24 / 2^-47, errors adding at worst linearly over the gates
U = {"c64": 2.0 ** -24, "ff": 2.0 ** -47}


def handle(n, arith, **kw):
    return DenseGB300(n, "c64" if arith == "c64" else "c128", fast_c128=arith == "ff", **kw)


def controlled(n, count, seed):
    rng, out = np.random.default_rng(seed), []
    for _ in range(count):
        q = [int(x) for x in rng.choice(n, 3, replace=False)]
        kind = int(rng.integers(0, 8))
        out.append((kind, q[0], tuple(q[1:1 + int(rng.integers(1, 3))]),
                    float(rng.uniform(-4, 4)) if kind in C.PARAMETRIC else 0.0))
    return out


@pytest.mark.parametrize("arith", ["c64", "ff"])
@pytest.mark.parametrize("tile", [11, 12, 13])
@pytest.mark.parametrize("mixed", [False, True])
def test_controlled_lists(arith, tile, mixed):
    if arith == "ff" and tile == 13:
        pytest.skip("no such float-float tile")
    n = 15
    sim, ref = handle(n, arith, jit=N.JIT_OFF), oracle.OracleDense(n, "c128")
    sim.set_tuning(tile_qubits=tile)
    parts = [C.brickwork(n, 1, 2), controlled(n, 120, 7)]
    if mixed:  # one flush: sweeps of both kinds
        parts = [C.brickwork(n, 1, 2), controlled(n, 300, 8) + C.hea(n, 3, np.linspace(-2, 2, 90)) + controlled(n, 300, 9)]
    count = sum(len(p) for p in parts)
    for p in parts:
        sim.apply(p)
        ref.apply(p)
        sim.flush()
    got, want = sim.state(), ref.state()
    assert np.linalg.norm(got - want) / np.linalg.norm(want) < count * U[arith]


@pytest.mark.parametrize("arith,n,jit", [("c64", 24, N.JIT_OFF), ("c64", 25, N.JIT_OFF), ("c64", 26, N.JIT_OFF),
                                         ("c64", 26, N.JIT_ALWAYS), ("ff", 25, N.JIT_OFF)])
@pytest.mark.parametrize("family", ["random", "controlled"])
def test_large_lists_with_few_gates_to_defer(arith, n, jit, family):
    gc.collect()
    start = [(C.H, q, (), 0.0) for q in range(0, n, 3)]
    gates = C.random_circuit(n, 100, 5, max_controls=2) if family == "random" else controlled(n, 100, 11)
    out = []
    for sim in (handle(n, arith, jit=jit), DenseGB300(n, "c128", jit=N.JIT_OFF)):
        with sim:
            sim.apply(start)
            sim.flush()
            sim.apply(gates)
            out.append(sim.state())
    assert np.linalg.norm(out[0] - out[1]) < (len(start) + len(gates)) * U[arith]


def test_signs_above_32_qubits():
    """Z and CZ gates of one flush (merged: pairs of tile, warp and outside
    qubits, more than 32 of them outside the tile), then the same ones two to a
    flush (as given), give |0...0> back between Hadamards on every qubit."""
    n = 33
    gc.collect()
    batch_release()
    rng = np.random.default_rng(33)
    signs = [(C.Z, q, (), 0.0) for q in (0, 6, 12, 20, 32)]
    signs += [(C.Z, 32, (q,), 0.0) for q in (0, 5, 9, 12, 13, 31)]
    signs += [(C.Z, int(a), (int(b),), 0.0) for a, b in (rng.choice(np.arange(13, 33), 2, replace=False) for _ in range(45))]
    signs += [(C.Z, int(a), (int(b),), 0.0) for a, b in (rng.choice(13, 2, replace=False) for _ in range(12))]
    mixer = [(C.H, q, (), 0.0) for q in range(n)]
    with DenseGB300(n, "c64", jit=N.JIT_OFF) as sim:
        sim.apply(mixer)
        sim.flush()
        sim.apply(signs)
        sim.flush()
        assert abs(sim.exp_value([(1.0, [(C.PAULI_X, q)]) for q in range(n)])) < n * 0.5  # (the phases are there)
        for i in range(0, len(signs), 2):
            sim.apply(signs[i:i + 2])
            sim.flush()
        sim.apply(mixer)
        ham = [(1.0, [(C.PAULI_Z, q)]) for q in range(n)]
        assert math.isclose(sim.exp_value(ham), n, rel_tol=(2 * n + 2 * len(signs)) * U["c64"])
    gc.collect()
