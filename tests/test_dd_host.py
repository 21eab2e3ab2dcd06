"""The deferred gate factors (dd.h) on the host: tests/ff_host/dd_check.cpp is
compiled with g++ (contraction off) and compared with long double.  The two
numbers a deferred RZ leaves are rounded to binary64 (2^-54 each, so sqrt(2)
2^-54 together); nothing else of it is."""
import os
import shutil
import subprocess

import pytest

from conftest import ROOT

SRC = os.path.join(ROOT, "tests", "ff_host", "dd_check.cpp")
TINY = 2.0 ** -62  # long double's own roundings, and the second order of 1 - e / 2
BOUNDS = {"factor": TINY, "rest": 2.0 ** -53.5 + TINY, "norm": 2.0 ** -53.5 + TINY, "unit": TINY}


def test_deferred_factors_are_unit_phases(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    exe = str(tmp_path / "dd_check")
    r = subprocess.run([cxx, "-std=c++17", "-O2", "-ffp-contract=off", SRC, "-o", exe, "-lm"],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([exe, "100000"], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr
    got = {k: float(v) for k, v in (line.split() for line in r.stdout.split("\n") if line.strip())}
    assert set(got) == set(BOUNDS)
    for k, bound in BOUNDS.items():
        assert got[k] <= bound, (k, got[k], bound)
