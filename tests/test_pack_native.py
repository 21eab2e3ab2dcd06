"""The native packers are there, under this interpreter's ABI tag, and take
what they are for."""
import os
import shutil
import sysconfig

import numpy as np
import pytest

from kbw_gb300 import _native as N
from kbw_gb300 import build as B
from kbw_gb300 import circuits as C
from kbw_gb300 import dense as D

pytestmark = pytest.mark.skipif(
    not (shutil.which("gcc") or shutil.which("cc"))
    or not os.path.exists(os.path.join(sysconfig.get_paths()["include"], "Python.h")) or B.PACK_NAME is None,
    reason="no C compiler, Python headers or lock-holding interpreter")


@pytest.fixture(autouse=True)
def unloaded(monkeypatch):
    monkeypatch.setattr(N, "_pack", None)
    monkeypatch.setattr(N, "_pack_tried", False)


def test_built_for_this_interpreter(monkeypatch):
    path = B.build_pack()
    assert os.path.basename(path) == "_kbwgpack" + sysconfig.get_config_var("EXT_SUFFIX")
    assert N._packer() is not None and N._packer()._name == path
    # a file of another interpreter is not this one's
    monkeypatch.setattr(B, "PACK_NAME", "_kbwgpack.cpython-399-none.so")
    monkeypatch.setattr(N, "_pack", None)
    monkeypatch.setattr(N, "_pack_tried", False)
    assert N._packer() is None


@pytest.mark.parametrize("circuit,taken", [
    (C.grover(5, 3, 1), True), (C.hea(4, 1, np.linspace(0, 1, 8).tolist()), True), ([[C.X, 2, [0, 63], 1]], True),
    ([(np.int64(0), 1, (), 0.0)], False), ([(C.X, 1, (2, 2), 0.0)], False), ([(C.X, 1, (64,), 0.0)], False),
    ([(C.X, -1, (), 0.0)], False), ([(C.X, 1, (), None)], False)])
def test_gate_lists(circuit, taken):
    B.build_pack()
    buf = np.zeros(max(len(circuit), 1), D._GATE_DT)
    assert N.pack_gates(circuit, buf, len(circuit)) is taken


@pytest.mark.parametrize("ham,taken", [
    (C.tfim_ring(5), True), ([(1, [[3, 0]])], True), ([], True), ([(np.float64(1.0), [(3, 0)])], False),
    ([(1.0, [(3, np.int64(0))])], False), ([(1.0, [(300, 0)])], False), ([(1.0, [(3, -1)])], False)])
def test_hamiltonians(ham, taken):
    B.build_pack()
    assert (N.pack_terms(ham) is not None) is taken
