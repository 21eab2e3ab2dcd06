"""Phase gates a few last places from a power of i: complex128 handles multiply
by the cosine and sine of the angle as given."""
import math

import numpy as np
import pytest

from kbw_gb300 import DenseGB300, _native as N
from kbw_gb300 import circuits as C

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("jit", [N.JIT_OFF, N.JIT_ALWAYS])
@pytest.mark.parametrize("qubit", [0, 6, 12])
def test_angles_next_to_quarter_turns(qubit, jit):
    n = 13
    sim = DenseGB300(n, "c128", jit=jit)
    one = np.zeros(1 << n, np.complex128)
    one[1 << qubit] = 1.0
    for turn in (math.pi / 2, -math.pi / 2, math.pi):
        angle = turn
        for _ in range(4):
            sim.set_state(one)
            sim.apply([(C.P, qubit, (), angle)])
            got = sim.state()[1 << qubit]
            # (the amplitude is 1: the products are exact; the C library rounds both within 2^-53)
            assert abs(got.real - math.cos(angle)) <= 2.0 ** -53 * abs(math.cos(angle))
            assert abs(got.imag - math.sin(angle)) <= 2.0 ** -53
            angle = np.nextafter(angle, 4.0)
