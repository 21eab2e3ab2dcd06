"""Z and CZ gates merged into one sign per amplitude: rings, dense graphs,
repeated pairs (which cancel), lone Z gates, pairs inside the tile, across its
edge and outside it, with gates in between that keep some of them apart; the
merged sweeps against sweeps that apply every gate as given (bit for bit: signs
are exact and the other gates here have no factor to defer), interpreted and
specialised, and against the oracle."""
import numpy as np
import pytest

import oracle
from kbw_gb300 import DenseGB300, batch_circuits_exp_value, _native as N
from kbw_gb300 import circuits as C

pytestmark = pytest.mark.gpu


def signs(n, count, seed):
    rng = np.random.default_rng(seed)
    out = [(C.Z, (i + 1) % n, (i,), 0.0) for i in range(n)]
    for _ in range(count):
        r = rng.random()
        a, b = (int(q) for q in rng.choice(n, size=2, replace=False))
        if r < 0.7:
            out.append((C.Z, a, (b,), 0.0))
            if r < 0.1:
                out.append((C.Z, b, (a,), 0.0))
        elif r < 0.85:
            out.append((C.Z, a, (), 0.0))
        elif r < 0.9:
            out.append((C.X, a, (), 0.0))
        elif r < 0.95:
            out.append((C.X, a, (b,), 0.0))
        else:
            out.append((C.Z, a, tuple(q for q in range(n) if q not in (a, b))[:2], 0.0))
    return out


@pytest.mark.parametrize("prec,fast", [("c64", False), ("c128", False), ("c128", True)])
@pytest.mark.parametrize("n,count", [(11, 30), (13, 60), (15, 150), (18, 200), (21, 120)])
def test_equal_to_gate_by_gate(prec, fast, n, count):
    rng = np.random.default_rng(n)
    init = rng.standard_normal(1 << n) + 1j * rng.standard_normal(1 << n)
    init = (init / np.linalg.norm(init)).astype(np.complex64 if prec == "c64" else np.complex128)
    circ = signs(n, count, n + count)
    out = []
    for fold, jit in ((False, N.JIT_OFF), (True, N.JIT_OFF)) + (((True, N.JIT_ALWAYS),) if n == 15 else ()):
        sim = DenseGB300(n, prec, fast_c128=fast, fold=fold, jit=jit)
        sim.set_state(init)
        sim.apply(circ)
        out.append(sim.state())
    ref = oracle.OracleDense(n, prec)
    ref.set_state(init)
    ref.apply(circ)
    for s in out[1:]:
        assert np.array_equal(s, out[0])
    if not fast:  # (float-float keeps 48 of the 53 bits of `init`)
        assert np.array_equal(out[0], ref.state().astype(out[0].dtype))


@pytest.mark.parametrize("n", [12, 14, 17])
def test_in_batches_and_gradients(n):
    p = C.hea_params(n, 3, n)
    circ = C.hea(n, 3, p) + signs(n, 40, 5) + C.hea(n, 1, p[: 2 * n])
    ham = C.tfim_ring(n)
    ref = oracle.OracleDense(n, "c128")
    ref.apply(circ)
    want = ref.pauli_expect(ham)
    index = [-1] * len(circ)
    for k in range(2 * n):
        index[k] = k
    for prec, fast, tol in (("c64", False, 5e-5), ("c128", False, 1e-10), ("c128", True, 1e-10)):
        got = batch_circuits_exp_value([(n, circ, ham)], prec=prec, fast_c128=fast)[0]
        assert abs(got - want) < tol
        sim = DenseGB300(n, prec, fast_c128=fast, jit=N.JIT_OFF)
        e, g = sim.adjoint_gradient(circ, index, 2 * n, ham)
        assert abs(e - want) < tol
        for k in (0, n, 2 * n - 1):
            d = []
            for h in (np.pi / 2, -np.pi / 2):
                c = list(circ)
                c[k] = (c[k][0], c[k][1], c[k][2], c[k][3] + h)
                o = oracle.OracleDense(n, "c128")
                o.apply(c)
                d.append(o.pauli_expect(ham))
            assert abs(g[k] - 0.5 * (d[0] - d[1])) < tol
