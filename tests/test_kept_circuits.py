"""The circuits that a backend keeps rewritten are found by content and share nothing with the caller's."""
import copy

import pytest

from mindquantum_b200.core import gates as G
from mindquantum_b200.core.circuit import Circuit
from mindquantum_b200.simulator.mqmatrix_b200 import doubled_circuit
from mindquantum_b200.simulator.utils import KeptCircuits


def _circ():
    return Circuit([G.RX('a').on(0), G.X.on(1), G.Measure('m').on(0)])


def _unmeasured(gates):
    return Circuit([g for g in gates if not isinstance(g, G.Measure)])


def test_same_content_is_kept_and_other_content_is_not():
    kept = KeptCircuits()
    first = kept.get(_circ(), _unmeasured)
    assert kept.get(_circ(), _unmeasured) is first
    assert kept.get(Circuit([G.RX('b').on(0), G.X.on(1)]), _unmeasured) is not first


@pytest.mark.parametrize('rewrite', [_unmeasured, lambda gates: doubled_circuit(gates[:2], 3)])
def test_a_gate_changed_in_place_leaves_what_was_kept(rewrite):
    kept = KeptCircuits()
    circ = _circ()
    before = [str(g) for g in kept.get(circ, rewrite)]
    list(circ)[1].obj_qubits = [2]
    assert [str(g) for g in kept.get(circ, rewrite)] == [str(g) for g in rewrite(list(circ))]
    assert [str(g) for g in kept.get(circ, rewrite)] != before
    assert [str(g) for g in kept.get(_circ(), rewrite)] == before


class _OwnGate(G.FixedGate):
    def __init__(self):
        super().__init__('own', G.X.matrix())


def _matrix(x):
    return G.RX(float(x)).matrix()


def test_gates_known_by_name_only_are_not_kept():
    kept = KeptCircuits()
    for gate in (_OwnGate().on(0), G.ParamNonHerm('rx', 1, _matrix, _matrix, 'a').on(0)):
        circ = Circuit([gate])
        assert kept.get(circ, _unmeasured) is not kept.get(circ, _unmeasured)


def test_a_copy_starts_empty():
    kept = KeptCircuits()
    first = kept.get(_circ(), _unmeasured)
    assert copy.deepcopy(kept).get(_circ(), _unmeasured) is not first
