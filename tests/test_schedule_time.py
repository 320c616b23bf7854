"""The time that building a schedule takes (host only)."""
import ctypes
import time

import numpy as np

from mindquantum_b200 import _native as N
from mindquantum_b200.core import gates as G
from mindquantum_b200.core.circuit import Circuit
from mindquantum_b200.simulator.lowering import lower_circuit


def _seconds(gates, n_qubits):
    """The best of three times of planning ``gates``, and the number of passes."""
    descs, _, _, _, _ = lower_circuit(Circuit(gates), [])
    table, pool, n = (N.GateDesc * len(descs))(*descs), np.zeros(2), len(descs)
    out = [np.zeros(n, t) for t in (np.int32, np.int32, np.uint64, np.int32)]
    passes = ctypes.c_int()
    best = 1e9
    for _ in range(3):
        t0 = time.perf_counter()
        N.call('mqb_plan_schedule', n_qubits, N.MQB_PREC_C64, table, n, pool.ctypes.data_as(ctypes.c_void_p), 1, 0, 1,
               ctypes.byref(passes), *[a.ctypes.data_as(ctypes.c_void_p) for a in out], None)
        best = min(best, time.perf_counter() - t0)
    return best, passes.value


def test_unfused_gates_take_linear_time():
    """A register too small for tile passes runs a pass per gate: four times the gates take about four times as long
    (copying what is left after every gate made it sixteen)."""

    def seconds(count):
        best, passes = _seconds([G.RX(0.1 * (i % 7)).on(i % 4) for i in range(count)], 4)
        assert passes == count
        return best

    assert seconds(60000) < 8 * seconds(15000) + 0.05


def test_idle_qubits_cost_nothing():
    """A register of 26 qubits of which 24 are used is planned about as fast as one of 24 (every scan used to run to
    the end of the circuit: ten times as long)."""
    rng = np.random.default_rng(3)
    gates = []
    for _ in range(15000):
        a, b = (int(q) for q in rng.permutation(24)[:2])
        gates.append(G.RX(0.3).on(a, b) if rng.random() < 0.5 else G.RZ(0.2).on(a))
    assert _seconds(gates, 26)[0] < 4 * _seconds(gates, 24)[0] + 0.02
