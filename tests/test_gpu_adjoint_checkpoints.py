"""Checkpoints of the adjoint gradient: a request above 16 is met (seen in the
memory the handle keeps), with results that do not depend on it, in every form
of the forward state, across calls that grow and shrink it, and above 32 qubits
as far as memory allows."""
import gc

import numpy as np
import pytest

from kbw_gb300 import DenseGB300, batch_release
from kbw_gb300 import circuits as C

pytestmark = pytest.mark.gpu

FORMS = [("c64", False, True), ("c64", False, False), ("c128", False, True), ("c128", True, True),
         ("c128", True, False)]
# rounding per gate and state 2^-24 / 2^-53 / 2^-47 over 2 x 140 gates, on
# derivatives of a Hamiltonian whose coefficients sum to 1.5 n = 21
TOL = {"c64": 280 * 21 * 2.0 ** -24, "c128": 280 * 21 * 2.0 ** -53, "ff": 280 * 21 * 2.0 ** -47}


def problem(n, layers, seed):
    params = C.hea_params(n, layers, seed)
    return C.hea(n, layers, params), C.hea_param_index(n, layers), len(params), C.tfim_ring(n, 1.0, 0.5)


@pytest.mark.parametrize("prec,fast,fusion", FORMS)
def test_requests_are_met_and_change_nothing(prec, fast, fusion):
    import torch
    n = 20  # 8 or 16 MiB a state
    p = problem(n, 2, 3)
    gc.collect()
    batch_release()
    with DenseGB300(n, prec, fast_c128=fast, fusion=fusion) as sim:
        e0, g0 = sim.adjoint_gradient(*p, max_checkpoints=0)
        free = torch.cuda.mem_get_info()[0]
        state = (16 if prec == "c128" else 8) << n
        for ask, kept in ((17, 17), (40, 40), (0, 40), (25, 40)):
            e, g = sim.adjoint_gradient(*p, max_checkpoints=ask)
            used = free - torch.cuda.mem_get_info()[0]
            assert kept * state <= used <= kept * state + (96 << 20)  # (and programs, grown with the segments)
            tol = TOL["ff" if fast else prec]
            assert abs(e - e0) <= tol and np.abs(g - g0).max() <= tol


@pytest.mark.parametrize("prec,fast", [("c64", False), ("c128", True)])
def test_kept_checkpoints_equal_a_fresh_handle(prec, fast):
    n = 14
    with DenseGB300(n, prec, fast_c128=fast) as sim:
        for layers, seed, ask in ((3, 1, 20), (1, 2, 30), (5, 3, 17), (3, 1, 64), (2, 4, 0), (3, 1, 20)):
            p = problem(n, layers, seed)
            e, g = sim.adjoint_gradient(*p, max_checkpoints=ask)
            with DenseGB300(n, prec, fast_c128=fast) as fresh:
                e1, g1 = fresh.adjoint_gradient(*p, max_checkpoints=ask)
            assert e == e1 and np.array_equal(g, g1)


def test_more_than_the_circuit_has_gates():
    p = problem(12, 1, 9)
    with DenseGB300(12, "c64") as sim:
        e0, g0 = sim.adjoint_gradient(*p, max_checkpoints=0)
        e1, g1 = sim.adjoint_gradient(*p, max_checkpoints=100000)
        assert abs(e1 - e0) <= TOL["c64"] and np.abs(g1 - g0).max() <= TOL["c64"]


def test_checkpoint_above_32_qubits():
    # state, lambda and those of the twelve checkpoints that fit, 64 GiB each
    n = 33
    gates = [(C.RY, q, (), 0.1 * (q + 1)) for q in (0, 7, 13, 20, 31, 32)] + [(C.X, 32, (5,), 0.0)]
    gates += [(C.RX, q, (), 0.2 * (q % 5 + 1)) for q in (32, 1, 8, 21)] + [(C.RZ, 32, (), 0.4), (C.RY, 32, (), -0.3)]
    index, k = [], 0
    for g in gates:
        index.append(k if g[0] in C.PARAMETRIC else -1)
        k += g[0] in C.PARAMETRIC
    ham = [(0.7, [(C.PAULI_X, 32)]), (-0.4, [(C.PAULI_Z, 7), (C.PAULI_Z, 32)]), (0.3, [(C.PAULI_Y, 1), (C.PAULI_X, 32)])]
    gc.collect()
    batch_release()
    with DenseGB300(n, "c64") as sim:
        e0, g0 = sim.adjoint_gradient(gates, index, k, ham, max_checkpoints=0)
        e1, g1 = sim.adjoint_gradient(gates, index, k, ham, max_checkpoints=17)
        assert abs(e1 - e0) <= TOL["c64"] and np.abs(g1 - g0).max() <= TOL["c64"]
    gc.collect()
