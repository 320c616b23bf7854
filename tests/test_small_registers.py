"""The block-per-sample kernel of small registers and the phase factors of the generated passes.

Tolerances as in the tile kernels' tests: complex128 1e-10, complex64 1e-5 on f and 1e-4 on the
gradients (a few hundred gates of 6e-8 each, Hamiltonians of norm below 4).
"""
import numpy as np
import pytest
import torch

from mindquantum_b200 import _native as N, complex64, complex128
from mindquantum_b200.core import gates as G
from mindquantum_b200.core.circuit import Circuit
from mindquantum_b200.core.operators import Hamiltonian, QubitOperator
from mindquantum_b200.simulator import Simulator, lowering
from oracle import oracle as O
from reference_circuits import hea_circuit

TOL = {complex128: (1e-10, 1e-10), complex64: (1e-5, 1e-4)}


def _circuit(n, rng, depth):
    """Every kind of gate the kernel dispatches on: dense and diagonal, one and two targets, X, controls."""
    c, k = Circuit(), 0
    for _ in range(depth):
        q = [int(x) for x in rng.permutation(n)]
        pick = rng.integers(0, 12)
        one = [G.RX(f'p{k}'), G.RY(f'p{k}'), G.RZ(f'p{k}'), G.PhaseShift(f'p{k}'), G.H, G.T, G.X,
               G.U3(f'p{k}', f'p{k + 1}', f'p{k + 2}')]
        if pick < 8 or n < 2:
            g = one[int(pick) % 8]
            c += g.on(q[0], q[1]) if n > 1 and rng.random() < 0.3 else g.on(q[0])
        else:
            g = [G.Rzz(f'p{k}'), G.Rxx(f'p{k}'), G.SWAP, G.FSim(f'p{k}', f'p{k + 1}')][int(pick) - 8]
            c += g.on(q[:2], q[2]) if n > 2 and rng.random() < 0.3 and g is not G.SWAP else g.on(q[:2])
        k += 3
    return c + Circuit([G.RY(f'p{k}').on(0)])


def _hams(n, count):
    ops = [QubitOperator('Z0', 0.7) + QubitOperator(f'X{n - 1}', -0.4) + QubitOperator('', 0.25), QubitOperator('Y0'),
           QubitOperator(f'Z0 Y{n - 1}' if n > 1 else 'X0', 0.6), QubitOperator(f'X{n // 2}', 1.1)]
    return [Hamiltonian(op) for op in ops[:count]]


def _against_oracle(sim, n, hams, circ, params, dtype):
    circ.as_encoder()
    f, g = sim.get_expectation_with_grad(hams, circ)(params)
    ref = O.get_expectation_with_grad(n, hams, circ, params, np.zeros(0), circ.params_name, [], np.complex128, None)
    assert np.allclose(f, ref[:, :, 0], atol=TOL[dtype][0], rtol=0)
    assert np.allclose(g, ref[:, :, 1:], atol=TOL[dtype][1], rtol=0)


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [complex128, complex64])
@pytest.mark.parametrize("n,n_hams,batch", [(1, 1, 3), (2, 4, 1), (5, 2, 7), (6, 1, 2), (9, 3, 2), (10, 1, 1), (10, 4, 2)])
def test_small_register_gradient(dtype, n, n_hams, batch):
    rng = np.random.default_rng(17 * n + n_hams)
    circ = _circuit(n, rng, 40)
    params = rng.uniform(0, 2 * np.pi, size=(batch, len(circ.params_name)))
    _against_oracle(Simulator('mqvector_b200', n, dtype=dtype), n, _hams(n, n_hams), circ, params, dtype)


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [complex128, complex64])
@pytest.mark.parametrize("n", [1, 3, 8, 10])
def test_small_register_apply_from_a_state(dtype, n):
    rng = np.random.default_rng(n)
    circ = _circuit(n, rng, 60)
    prd = dict(zip(circ.params_name, rng.uniform(0, 2 * np.pi, len(circ.params_name))))
    v = rng.normal(size=1 << n) + 1j * rng.normal(size=1 << n)
    v /= np.linalg.norm(v)
    sim = Simulator('mqvector_b200', n, dtype=dtype)
    sim.set_qs(v)
    sim.apply_circuit(circ, prd)
    ref = O.OracleSim(n, np.complex128, v).apply_circuit(circ, prd).qs
    assert np.allclose(sim.get_qs(), ref, atol=1e-11 if dtype == complex128 else 5e-6, rtol=0)


@pytest.mark.gpu
def test_both_sides_of_the_batch_rule_agree():
    """9 qubits: 296 samples run a block each, more run on the tile kernels."""
    n = 9
    rng = np.random.default_rng(5)
    circ = hea_circuit(n, 2)
    ham = _hams(n, 1)
    params = torch.as_tensor(rng.uniform(0, 2 * np.pi, size=(400, len(circ.params_name))), device='cuda')
    be = Simulator('mqvector_b200', n, dtype=complex128).backend
    many = be.expectation_with_grad_tensor(ham, circ, params, circ.params_name)
    few = be.expectation_with_grad_tensor(ham, circ, params[:20], circ.params_name)
    assert torch.allclose(many[0][:20], few[0], atol=1e-11, rtol=0)
    assert torch.allclose(many[1][:20], few[1], atol=1e-11, rtol=0)


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [complex128, complex64])
@pytest.mark.parametrize("n,n_hams", [(10, 1), (12, 1), (13, 2), (14, 4)])
def test_diagonal_gates_in_every_place(dtype, n, n_hams):
    """Diagonal gates of known unitaries (RZ, PS, GP, RZZ, S, T, CZ; controlled or not) between rotations, so
    that their targets and controls fall on registers, lanes, warps and outside the tile."""
    rng = np.random.default_rng(90 + n)
    c, k = Circuit(), 0
    for _ in range(4):
        for q in range(n):
            c += G.RY(f'p{k}').on(q)
            k += 1
        for _ in range(3 * n):
            a, b, d = (int(x) for x in rng.permutation(n)[:3])
            pick = rng.integers(0, 9)
            g = [G.RZ(f'p{k}').on(a), G.RZ(f'p{k}').on(a, b), G.PhaseShift(f'p{k}').on(a), G.PhaseShift(f'p{k}').on(a, [b, d]),
                 G.GlobalPhase(f'p{k}').on(a), G.Rzz(f'p{k}').on([a, b]), G.Rzz(f'p{k}').on([a, b], d), G.Z.on(a, b),
                 (G.S if pick % 2 else G.T).on(a)][int(pick)]
            c += g
            k += 1
    params = rng.uniform(0, 2 * np.pi, size=(2, len(c.params_name)))
    _against_oracle(Simulator('mqvector_b200', n, dtype=dtype, jit=True), n, _hams(n, n_hams), c, params, dtype)


def test_set_search_keeps_the_order_and_saves_passes():
    """A layered circuit in wedges: valid reordering, about half the passes that program order takes (31)."""
    n = 26
    c = hea_circuit(n, 12)
    order, pass_of, qmask, fused = lowering.plan_schedule(c, n, N.MQB_PREC_C64, tile_bits=12)
    gates = list(c)
    pos = {int(g): i for i, g in enumerate(order)}
    last = {}
    for i, g in enumerate(gates):
        for q in list(g.obj_qubits) + list(g.ctrl_qubits):
            if q in last:
                assert pos[last[q]] < pos[i]
            last[q] = i
    for e, gi in enumerate(order):
        for q in gates[gi].obj_qubits:
            assert int(qmask[pass_of[e]]) >> q & 1 or gates[gi].name == 'RZ'
    assert all(fused) and len(qmask) <= 16
