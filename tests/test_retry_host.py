"""Allocations ask for the buffer kept between batch calls before they fail:
the decision on the host (tests/ff_host/retry_check.cpp, a fake allocator), and
on the GPU a register that fits only without that buffer."""
import os
import shutil
import subprocess

import pytest

from conftest import ROOT

SRC = os.path.join(ROOT, "tests", "ff_host", "retry_check.cpp")


def test_retry_decision(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    exe = str(tmp_path / "retry_check")
    r = subprocess.run([cxx, "-std=c++17", "-Wall", "-Werror", SRC, "-o", exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout


@pytest.mark.gpu
@pytest.mark.parametrize("call", ["register", "gradient"])
def test_register_after_a_batch_call(call):
    import gc

    import torch

    from kbw_gb300 import DenseGB300, batch_circuits_exp_value, batch_release
    from kbw_gb300 import circuits as C

    gc.collect()
    batch_release()
    torch.cuda.empty_cache()
    free = torch.cuda.mem_get_info()[0]
    gib = 1 << 30
    small = DenseGB300(26, "c128") if call == "gradient" else None  # 1 GiB
    # twelve registers of 24 qubits: 3 GiB stay with the process
    ham = [(1.0, [(C.PAULI_Z, 0)])]
    batch_circuits_exp_value([(24, [(C.H, 0, (), 0.0)], ham)] * 12, prec="c128")
    assert free - torch.cuda.mem_get_info()[0] > 3 * gib
    filler = torch.empty(torch.cuda.mem_get_info()[0] - gib // 2, dtype=torch.uint8, device="cuda")
    try:
        if call == "register":
            DenseGB300(27, "c128").close()  # 2 GiB
        else:
            e, g = small.adjoint_gradient([(C.RX, 0, (), 0.3)], [0], 1, ham)
            assert abs(e - 0.955336489125606) < 1e-12 and abs(g[0] + 0.2955202066613396) < 1e-12
    finally:
        del filler
        torch.cuda.empty_cache()
        batch_release()
