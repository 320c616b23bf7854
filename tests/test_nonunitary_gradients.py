"""Gradients through matrices that are not unitary: the state before them is a stored one, not one rebuilt by the
conjugate transpose.  Against central differences of the expectation in complex128 (step 1e-5: truncation and rounding below
1e-8 for values of order one) and complex64 against complex128.
"""
import numpy as np
import pytest

from mindquantum_b200 import complex64, complex128
from mindquantum_b200.core import gates as G
from mindquantum_b200.core.circuit import Circuit
from mindquantum_b200.core.operators import Hamiltonian, QubitOperator
from mindquantum_b200.simulator import Simulator


def _fading(x):
    return np.array([[np.exp(-0.3 * x), 0], [0.2 * np.sin(x), np.cos(x)]], dtype=complex)


def _d_fading(x):
    return np.array([[-0.3 * np.exp(-0.3 * x), 0], [0.2 * np.cos(x), -np.sin(x)]], dtype=complex)


CUSTOM = G.gene_univ_parameterized_gate('fading', _fading, _d_fading)
DAMPED = G.UnivMathGate('damped', np.diag([1, 0.3]).astype(complex))
SHEAR = G.UnivMathGate('shear', np.array([[1, 0.4j], [0, 0.9]]))


def _circuit(n, kind):
    a, b = 0, n // 2
    c = Circuit()
    for q in {a, b, n - 1}:
        c += G.RY(f'y{q}').on(q)
    c += {'diagonal': DAMPED, 'dense': SHEAR}[kind].on(b) if kind != 'custom' else CUSTOM('c').on(b)
    if n > 1:
        c += G.X.on(n - 1, a)
        c += SHEAR.on(a, n - 1) if kind == 'dense' else DAMPED.on(a) if kind == 'diagonal' else CUSTOM('c').on(a, n - 1)
    for q in {a, b, n - 1}:
        c += G.RX(f'x{q}').on(q)
    return c


def _operator(n, kind, dtype, count):
    hams = [Hamiltonian(QubitOperator(f'Z{n // 2}', 0.8) + QubitOperator('X0', -0.5)), Hamiltonian(QubitOperator(f'Y{n - 1}'))]
    c = _circuit(n, kind)
    return c, Simulator('mqvector_b200', n, dtype=dtype).get_expectation_with_grad(hams[:count], c.as_encoder())


# 1 and 5 qubits: a block per sample; 10: the same, at both sides of its batch rule; 12: tile passes
@pytest.mark.gpu
@pytest.mark.parametrize('n,batch,count', [(1, 1, 1), (5, 3, 2), (10, 2, 1), (10, 400, 1), (12, 2, 2)])
@pytest.mark.parametrize('kind', ['diagonal', 'dense', 'custom'])
def test_against_central_differences(n, batch, count, kind):
    if kind == 'custom' and n > 10:
        pytest.skip('larger registers undo custom gates by their conjugate transposes')
    c, op = _operator(n, kind, complex128, count)
    p = np.random.default_rng(n).uniform(0, 2 * np.pi, size=(batch, len(c.params_name)))
    _, g = op(p)
    for k in range(p.shape[1]):
        d = np.zeros(p.shape[1])
        d[k] = 1e-5
        num = (op(p + d)[0] - op(p - d)[0]) / 2e-5
        assert np.allclose(g[:, :, k], num, atol=1e-7, rtol=0)
    f32, g32 = _operator(n, kind, complex64, count)[1](p)
    f64, _ = op(p)
    assert np.allclose(f32, f64, atol=1e-5, rtol=0) and np.allclose(g32, g, atol=1e-4, rtol=0)
