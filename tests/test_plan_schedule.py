"""The host-only plan is the schedule that a program runs."""
import numpy as np
import pytest

from mindquantum_b200 import _native as N
from mindquantum_b200.core import gates as G
from mindquantum_b200.core.circuit import Circuit
from mindquantum_b200.simulator import lowering
from reference_circuits import hea_circuit


def _dense_blocks(n, layers):
    """Dense two-qubit gates inside blocks of six qubits: more matrix entries than one pass may hold."""
    rng, c = np.random.default_rng(n), Circuit()
    m = G.UnivMathGate('m', G.Rxx(0.3).matrix())
    for _ in range(layers):
        for a in range(0, n - 5, 6):
            qs = [int(q) for q in a + rng.permutation(6)]
            for x, y in zip(qs[::2], qs[1::2]):
                c += m.on([x, y])
    return c


@pytest.mark.gpu
@pytest.mark.parametrize('prec', [N.MQB_PREC_C64, N.MQB_PREC_C128])
@pytest.mark.parametrize('n', [6, 12, 14, 16, 18, 20])
@pytest.mark.parametrize('tile', [0, 10, 13])
def test_passes_and_tiles_of_a_program(prec, n, tile):
    for circ in (hea_circuit(n, 8), _dense_blocks(n, 60)):
        prog = lowering.Program(circ, n, prec, circ.params_name, tile_bits=tile)
        _, _, qmask, fused = lowering.plan_schedule(circ, n, prec, tile_bits=tile)
        assert len(qmask) == prog.info.n_passes
        assert {bin(int(q)).count('1') for q, f in zip(qmask, fused) if f} <= {prog.info.tile_bits}
