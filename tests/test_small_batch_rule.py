"""The block-per-sample kernel and the tile kernels agree where a batch goes from one to the other.

The limit is one sample per SM at 10 qubits and doubles per qubit less (a state alone in complex64: twice that).  In
complex64 a gradient runs in FP64 in the block and in FP32 in the tiles: the bounds are those of complex64.
"""
import numpy as np
import pytest
import torch

from mindquantum_b200 import complex64, complex128
from mindquantum_b200.core.operators import Hamiltonian, QubitOperator
from mindquantum_b200.simulator import Simulator
from reference_circuits import hea_circuit


@pytest.mark.gpu
@pytest.mark.parametrize('dtype,tol', [(complex64, (1e-5, 1e-4)), (complex128, (1e-11, 1e-11))])
@pytest.mark.parametrize('n,n_hams', [(7, 2), (8, 2), (8, 4), (9, 1), (10, 1), (10, 4)])
def test_gradients_at_the_limit(n, n_hams, dtype, tol):
    limit = torch.cuda.get_device_properties(0).multi_processor_count << (10 - n)
    circ = hea_circuit(n, 2)
    hams = [Hamiltonian(QubitOperator(f'Z{q}') + QubitOperator(f'X{q + 1}', 0.5)) for q in range(n_hams)]
    p = torch.as_tensor(np.random.default_rng(n).uniform(0, 2 * np.pi, size=(limit + 1, len(circ.params_name))), device='cuda')
    be = Simulator('mqvector_b200', n, dtype=dtype).backend
    f, g = be.expectation_with_grad_tensor(hams, circ, p, circ.params_name)
    for rows in (slice(0, limit), slice(1, limit + 1)):
        f1, g1 = be.expectation_with_grad_tensor(hams, circ, p[rows], circ.params_name)
        assert torch.allclose(f1, f[rows], atol=tol[0], rtol=0)
        assert torch.allclose(g1, g[rows], atol=tol[1], rtol=0)
