"""Circuits of very different sizes evaluated from two host threads at once."""
import threading

import numpy as np
import pytest
import torch

from mindquantum_b200 import complex128
from mindquantum_b200.core.operators import Hamiltonian, QubitOperator
from mindquantum_b200.simulator import Simulator
from reference_circuits import hea_circuit


def _in_threads(jobs, repeats):
    """What every job returned at each repeat, the jobs in threads of their own with streams of their own."""
    out, errors = [[] for _ in jobs], []
    start = threading.Barrier(len(jobs))

    def work(i):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                start.wait(60)
                for _ in range(repeats):
                    out[i].append(jobs[i]())
        except Exception as e:  # pylint: disable=broad-except
            errors.append(e)

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(jobs))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    if errors:
        raise errors[0]
    return out


# 10 qubits: the block-per-sample kernel, 39 against 170 KB of shared memory; 12: tile passes
@pytest.mark.gpu
@pytest.mark.parametrize('n,layers', [(10, (1, 40)), (12, (1, 12))])
def test_launch_limits_of_two_circuits(n, layers):
    jobs, expected = [], []
    for k in layers:
        circ = hea_circuit(n, k)
        ham = Hamiltonian(QubitOperator('Z0') + QubitOperator(f'X{n - 1}', 0.5))
        op = Simulator('mqvector_b200', n, dtype=complex128).get_expectation_with_grad(ham, circ)
        p = np.random.default_rng(k).uniform(0, 2 * np.pi, size=len(circ.params_name))
        expected.append(op(p))
        jobs.append(lambda op=op, p=p: op(p))
    for got, (f, g) in zip(_in_threads(jobs, 300), expected):
        for f1, g1 in got:
            assert np.allclose(f1, f, atol=1e-12) and np.allclose(g1, g, atol=1e-11)


@pytest.mark.gpu
@pytest.mark.parametrize('backend,n', [('mqvector_b200', 9), ('mqmatrix_b200', 4)])
def test_first_gradients_of_one_circuit(backend, n):
    """Threads that evaluate one circuit share its program, whose gradient schedules are made on first use."""
    for seed in range(10):
        circ = hea_circuit(n, 1 + seed % 3)
        hams = [Hamiltonian(QubitOperator(f'Z{q}')) for q in range(4)]
        p = np.random.default_rng(seed).uniform(0, 2 * np.pi, size=len(circ.params_name))
        if backend == 'mqmatrix_b200':   # one simulator, whose doubled circuit is kept for all calls
            sims = [Simulator(backend, n, dtype=complex128)] * 4
        else:
            sims = [Simulator(backend, n, dtype=complex128) for _ in range(4)]
        jobs = [lambda op=sim.get_expectation_with_grad(hams[:k + 1], circ): op(p) for k, sim in enumerate(sims)]
        got = _in_threads(jobs, 1)
        for k, ((f, g),) in enumerate(got):
            f1, g1 = Simulator(backend, n, dtype=complex128).get_expectation_with_grad(hams[:k + 1], hea_circuit(n, 1 + seed % 3))(p)
            assert np.allclose(f, f1, atol=1e-11) and np.allclose(g, g1, atol=1e-11)
