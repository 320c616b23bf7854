"""Grad operators called with numpy arrays inside torch's modes, and the storage of the device call's results."""
import numpy as np
import pytest
import torch

from mindquantum_b200 import complex64, complex128
from mindquantum_b200.core.operators import Hamiltonian, QubitOperator
from mindquantum_b200.simulator import Simulator
from reference_circuits import hea_circuit


@pytest.mark.gpu
@pytest.mark.parametrize('n', [4, 12])
@pytest.mark.parametrize('dtype', [complex64, complex128])
@pytest.mark.parametrize('mode', [torch.inference_mode, torch.no_grad])
def test_numpy_call_inside_a_mode(n, dtype, mode):
    circ = hea_circuit(n, 2)
    hams = [Hamiltonian(QubitOperator('Z0')), Hamiltonian(QubitOperator(f'X{n - 1}'))]
    op = Simulator('mqvector_b200', n, dtype=dtype).get_expectation_with_grad(hams, circ)
    p = np.random.default_rng(n).uniform(0, 2 * np.pi, size=len(circ.params_name))
    f, g = op(p)
    with mode():
        f1, g1 = op(p)
    assert f1.shape == f.shape == (1, 2) and g1.shape == g.shape == (1, 2, len(p))
    assert np.allclose(f1, f, atol=1e-6) and np.allclose(g1, g, atol=1e-6)


@pytest.mark.gpu
def test_device_results_have_storages_of_their_own():
    circ = hea_circuit(4, 1)
    be = Simulator('mqvector_b200', 4, dtype=complex128).backend
    f, g = be.expectation_with_grad_tensor([Hamiltonian(QubitOperator('Z0'))], circ,
                                           torch.zeros(3, len(circ.params_name), device='cuda'), circ.params_name)
    assert f.untyped_storage().data_ptr() != g.untyped_storage().data_ptr()
    assert f.untyped_storage().nbytes() == f.numel() * 8
