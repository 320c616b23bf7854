"""Diagonal gates of the generated passes in complex64: what their rounding does to expectations and gradients.

A rotation's entries are conjugates, so that their rounding scales the state as a whole.  A pair applied by its rounded
ratio r multiplies the two halves by |r| differently, the same way at every gate: after m equal gates <Z> is off by
m (|r|^2 - 1) / 2, some 2e-5 for m = 1200 and half of all angles.  Products of equal moduli leave a random walk at worst:
2 m products (into a table, then to the amplitude) of a relative rounding error of 2^-24 times 0.6 (rms) each;
the bound is six times that.
"""
import numpy as np
import pytest
import torch

from mindquantum_b200 import complex64, complex128
from mindquantum_b200.core import gates as G
from mindquantum_b200.core.circuit import Circuit
from mindquantum_b200.core.operators import Hamiltonian, QubitOperator
from mindquantum_b200.simulator import Simulator

N_QUBITS = 18   # the smallest register of the generated passes
GATES = 1200
BOUND = 6 * 0.6 * 2.0 ** -24 * np.sqrt(2 * GATES)


@pytest.mark.gpu
@pytest.mark.parametrize('qubits', [(0,), (7,), (12,), (17,), (0, 1), (4, 15), (16, 17)])
def test_diagonal_rotations_do_not_tilt_the_state(qubits):
    c = Circuit([G.H.on(q) for q in range(N_QUBITS)])
    for _ in range(GATES):
        c += G.RZ('t').on(qubits[0]) if len(qubits) == 1 else G.Rzz('t').on(list(qubits))
    ham = Hamiltonian(QubitOperator(' '.join(f'Z{q}' for q in qubits)))
    sim = Simulator('mqvector_b200', N_QUBITS, dtype=complex64)
    angles = np.random.default_rng(7).uniform(0.3, 3.0, size=(12, 1))
    f, g = sim.get_expectation_with_grad(ham, c.as_encoder())(angles)
    assert np.abs(f).max() <= BOUND
    # no diagonal gate changes the expectation; m partials of the same bound each
    assert np.abs(g).max() <= 2 * GATES * BOUND


def _errors(make):
    """Mean over ten parameter sets of |f - f64| and of |g - g64| / |g64|, complex64 against complex128."""
    rng = np.random.default_rng(64)
    circ, ham, params = make(rng)
    p = torch.tensor(params, device='cuda')
    out = []
    for dtype in (complex64, complex128):
        be = Simulator('mqvector_b200', N_QUBITS, dtype=dtype).backend
        f, g = be.expectation_with_grad_tensor([ham], circ, p, circ.params_name)
        out.append((f[:, 0, 0].cpu().numpy(), g[:, 0].cpu().numpy()))
    (f, g), (f64, g64) = out
    return np.abs(f - f64).mean(), (np.linalg.norm(g - g64, axis=1) / np.linalg.norm(g64, axis=1)).mean()


def _ansatz(rng):
    c = Circuit()
    for layer in range(8):
        for q in range(N_QUBITS):
            c += G.RY(f'y{layer}_{q}').on(q)
        for q in range(N_QUBITS):
            c += G.RZ(f'z{layer}_{q}').on(q)
        c += Circuit([G.X.on(q + 1, q) for q in range(N_QUBITS - 1)])
    op = QubitOperator()
    for q in range(N_QUBITS - 1):
        op += QubitOperator(f'Z{q} Z{q + 1}', float(rng.normal()))
    for q in range(N_QUBITS):
        op += QubitOperator(f'X{q}', float(rng.normal()))
    return c, Hamiltonian(op), rng.uniform(0, 2 * np.pi, size=(10, len(c.params_name)))


def _qaoa(rng):
    edges = [(q, (q + 1) % N_QUBITS) for q in range(N_QUBITS)] + [(q, q + N_QUBITS // 2) for q in range(N_QUBITS // 2)]
    c, op = Circuit([G.H.on(q) for q in range(N_QUBITS)]), QubitOperator()
    for layer in range(10):
        for e in edges:
            c += G.Rzz(f'c{layer}').on(list(e))
        for q in range(N_QUBITS):
            c += G.RX(f'm{layer}').on(q)
    for a, b in edges:
        op += QubitOperator(f'Z{a} Z{b}')
    return c, Hamiltonian(op), rng.uniform(0, np.pi, size=(10, len(c.params_name)))


@pytest.mark.gpu
@pytest.mark.parametrize('make,most_f,most_g', [(_ansatz, 8.622e-8, 5.940e-7), (_qaoa, 2.613e-6, 2.623e-6)])
def test_errors_against_64_bits(make, most_f, most_g):
    """No more than with every gate of a run multiplied in on its own pair in complex64 (measured)."""
    f, g = _errors(make)
    print(f'{make.__name__}: f {f:.2e} g {g:.2e}')
    assert f <= most_f and g <= most_g
