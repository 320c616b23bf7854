"""The qubit sets of generated passes (host only): tiles of a large register move in few tensor copies."""
import numpy as np
import pytest

from mindquantum_b200 import _native as N, workloads
from mindquantum_b200.simulator.lowering import plan_schedule


def _copies(qmask):
    """Tensor copies per tile: the low run of consecutive qubits and four more in one, twice as many per further run."""
    q = int(qmask)
    runs = bin(q & ~(q << 1)).count('1')
    return 2 ** max(0, runs - 5)


@pytest.mark.parametrize('n,p,seed', [(26, 10, 0), (28, 10, 0), (30, 10, 0), (30, 5, 1), (24, 5, 2)])
def test_maxcut_passes_move_whole_tiles(n, p, seed):
    """A searched schedule took fewer passes, but some over sets of nine runs, which moved a tile of 30 qubits in 16 copies
    and took 2.4 times as long."""
    circ = workloads.qaoa_maxcut(n, p, seed)[0]
    _, _, qmask, fused = plan_schedule(circ, n, N.MQB_PREC_C64)
    copies = [_copies(q) for q, f in zip(qmask, fused) if f]
    assert max(copies) <= 4 and np.mean(copies) <= 1.5
