"""Scratch a gradient call leaves with its handle: lambda and the checkpoints
while they take at most a sixteenth of the device's memory, whatever the size
of one state."""
import gc

import pytest

from kbw_gb300 import DenseGB300, batch_release
from kbw_gb300 import circuits as C

pytestmark = pytest.mark.gpu


def test_many_checkpoints_of_a_small_state_are_given_back():
    import torch
    n, count = 22, 700  # 64 MiB each: 43.8 GiB, a sixteenth is about 17
    gc.collect()
    batch_release()
    torch.cuda.empty_cache()
    sim = DenseGB300(n, "c128")
    ham = C.tfim_ring(n)
    gates = [(C.RY, i % n, (), 0.01 * i) for i in range(count + 1)]
    index = [0] * len(gates)
    sim.adjoint_gradient(gates[:30], index[:30], 1, ham, 0)
    free, total = torch.cuda.mem_get_info()
    sim.adjoint_gradient(gates, index, 1, ham, count)
    assert free - torch.cuda.mem_get_info()[0] <= total // 16
    sim.close()
