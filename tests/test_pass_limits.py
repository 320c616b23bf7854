"""Shared memory of the generated pass kernels over circuits that fill their passes (host only)."""
import numpy as np
import pytest

from mindquantum_b200 import _native as N
from mindquantum_b200.core import gates as G
from mindquantum_b200.core.circuit import Circuit
from mindquantum_b200.simulator import lowering

BLOCK_SMEM = 227 * 1024


def _blocks(n, width, layers, rng):
    """Layers of U3 and dense two-qubit gates inside blocks of ``width`` neighbouring qubits: a pass takes whole blocks,
    as many gates as its matrix table and its gradient rows hold."""
    c, k = Circuit(), 0
    for _ in range(layers):
        for q in range(n):
            c += G.U3(f'p{k}', f'p{k + 1}', f'p{k + 2}').on(q)
            k += 3
        for a in range(0, n, width):
            qs = [int(q) for q in a + rng.permutation(min(width, n - a))]
            for x, y in zip(qs[::2], qs[1::2]):
                c += [G.Rxx(f'p{k}'), G.FSim(f'p{k}', f'p{k + 1}'), G.UnivMathGate('m', G.Rxx(0.3).matrix())][k % 3].on([x, y])
                k += 2
    return c


@pytest.mark.parametrize('prec', [N.MQB_PREC_C64, N.MQB_PREC_C128])
@pytest.mark.parametrize('n_hams', [0, 1, 2, 3, 4])
def test_every_kernel_fits_a_block(prec, n_hams):
    full = 0
    for seed, (n, width, layers) in enumerate([(18, 6, 20), (18, 6, 25), (20, 5, 20), (24, 8, 15), (22, 4, 30), (26, 6, 12)]):
        c = _blocks(n, width, layers, np.random.default_rng(seed))
        used = lowering.jit_smem(c, n, prec, n_hams)
        assert used <= BLOCK_SMEM
        full = max(full, used)
    assert full > 0.5 * BLOCK_SMEM or prec == N.MQB_PREC_C64   # the circuits do fill the passes
