"""The binding's native packers against its Python path: the same arrays, and
the Python path for whatever the packers do not take (numpy numbers, repeated
or large controls, values out of range)."""
import numpy as np
import pytest

from kbw_gb300 import _native as N
from kbw_gb300 import circuits as C
from kbw_gb300 import dense as D


def python_path(monkeypatch):
    monkeypatch.setattr(N, "_pack", None)
    monkeypatch.setattr(N, "_pack_tried", True)


CIRCUITS = [[], C.grover(6, 3, 2), C.hea(5, 2, np.linspace(-1, 1, 20)), C.random_circuit(9, 200, 1, max_controls=4),
            [(C.P, 3, [0, 1], 2), (C.X, 0, (5,), 0.0)], [(np.int64(3), np.int32(1), (np.int64(2),), np.float64(0.5))],
            ((C.H, 1, (), 0.0),), [[C.RY, 2, [], 1.25]], [(C.Z, 4, (63,), 0.0)]]
HAMS = [[], [(1.0, [])], C.tfim_ring(7), [(2, [(3, 1), (1, 0)]), (np.float64(0.5), [(np.int64(2), 3)])],
        [(-0.25, ((1, 2),))]]


@pytest.mark.parametrize("i", range(len(CIRCUITS)))
def test_gate_arrays(i, monkeypatch):
    got = bytes(memoryview(D._gate_array(CIRCUITS[i])).cast("B"))
    python_path(monkeypatch)
    assert got == bytes(memoryview(D._gate_array(CIRCUITS[i])).cast("B"))


@pytest.mark.parametrize("i", range(len(HAMS)))
def test_hamiltonian_arrays(i, monkeypatch):
    got = D._ham_arrays(HAMS[i])
    python_path(monkeypatch)
    want = D._ham_arrays(HAMS[i])
    assert got[4] == want[4]
    for x, y in zip(got[:4], want[:4]):
        assert x.dtype == y.dtype and np.array_equal(x, y)


@pytest.mark.parametrize("bad", [[(0, 1, (70,), 0.0)], [(0, -1, (), 0.0)], [(0, 1, (), "x")], [(0, 1, ())]])
def test_what_was_refused_stays_refused(bad, monkeypatch):
    with pytest.raises(Exception) as native:
        D._gate_array(bad)
    python_path(monkeypatch)
    with pytest.raises(type(native.value)):
        D._gate_array(bad)
