"""Performance cases of the state-vector and density-matrix simulators, through the public API.

A case names a family and its sizes; ``listed()`` gives the standing cases and ``draw()`` more of
the same ranges.  The families are what programs of this framework do:

* ``vqe``: one expectation and gradient of a hardware-efficient ansatz in complex128, numpy in and
  out, as an optimiser calls it (4 to 16 qubits; the smallest calls, where latency counts);
* ``hea``: gradients of several parameter sets of a wide ansatz at once in complex64, on device
  tensors (18 to 26 qubits; the largest states);
* ``qnn``: a training step of a torch layer, encoder samples against shared weights, several
  observables (4 to 20 qubits);
* ``qaoa``: MaxCut on a 3-regular graph, few shared parameters, ZZ gates between distant qubits;
* ``uneven``: circuits of different registers evaluated together in one CUDA graph;
* ``apply``: a circuit of mixed gates, controlled and two-qubit ones among them, applied to |0...0>
  (the forward direction alone);
* ``expect``: the expectation of a Hamiltonian of many random Pauli strings (molecules);
* ``sample``: measurement shots of a noiseless circuit;
* ``noise``: shots of a noisy circuit, one trajectory each;
* ``density``: a gradient of a noisy circuit on the density-matrix backend.

A circuit is a list of (gate name, targets, controls, parameter indices), the parameters numbered in
the order of their first use; its structure depends on the case alone, its parameters on the seed.  ``exact`` evaluates the same list in plain torch in 64
bits.
"""
import math
import random

import numpy as np
import torch

from mindquantum_b200 import complex64, complex128
from mindquantum_b200.core import gates as G
from mindquantum_b200.core.circuit import Circuit
from mindquantum_b200.core.operators import Hamiltonian, QubitOperator
from mindquantum_b200.framework import MQAnsatzOnlyOps, MQEncoderOnlyOps, MQLayer
from mindquantum_b200.simulator import Simulator
from mindquantum_b200.simulator.batch import CircuitBatch


def listed():
    return [
        # one optimiser call on a small molecule's register: launches and host time
        {"name": "vqe_8q", "family": "vqe", "n": 8, "layers": 2},
        # the 16-qubit, 8-layer ansatz in complex128, one parameter set
        {"name": "vqe_16q", "family": "vqe", "n": 16, "layers": 8},
        # the wide ansatz at 26 qubits and 12 layers (624 parameters), two parameter sets
        {"name": "hea_26q", "family": "hea", "n": 26, "layers": 12, "batch": 2},
        # a mid-size odd register with an odd batch
        {"name": "hea_21q", "family": "hea", "n": 21, "layers": 5, "batch": 7},
        # a classifier's training step on a mini-batch of small circuits
        {"name": "qnn_6q", "family": "qnn", "n": 6, "layers": 3, "samples": 32, "obs": 2},
        # the 20-qubit classifier with four observables
        {"name": "qnn_20q", "family": "qnn", "n": 20, "layers": 6, "samples": 64, "obs": 4},
        # MaxCut on 26 vertices, p = 10
        {"name": "qaoa_26q", "family": "qaoa", "n": 26, "p": 10},
        # ten random circuits of 10 to 19 qubits as one unit
        {"name": "uneven", "family": "uneven", "members": 10, "n_min": 10, "n_max": 19, "layers": 8, "structure": 3},
        # 300 mixed gates applied to 25 qubits: the forward direction
        {"name": "apply_25q", "family": "apply", "n": 25, "gates": 300, "structure": 7},
        # a molecular Hamiltonian's expectation: hundreds of Pauli strings
        {"name": "expect_20q", "family": "expect", "n": 20, "terms": 400, "structure": 11},
        # shots of a 20-qubit circuit
        {"name": "sample_20q", "family": "sample", "n": 20, "layers": 2, "shots": 4096},
        # a noisy 7-qubit gradient with exact channels
        {"name": "density_7q", "family": "density", "n": 7, "layers": 2},
    ]


def draw(rng):
    def size(lo, hi):   # spread over the logarithm
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    family = rng.choice(["vqe", "vqe", "hea", "qnn", "qnn", "qaoa", "uneven", "apply", "expect", "sample", "noise",
                         "density"])
    if family == "vqe":
        return {"family": family, "n": rng.randint(4, 16), "layers": rng.randint(1, 8)}
    if family == "hea":
        n = rng.randint(18, 25)
        return {"family": family, "n": n, "layers": rng.randint(2, 8), "batch": size(1, max(1, min(16, 1 << (26 - n))))}
    if family == "qnn":
        n = rng.randint(4, 19)
        return {"family": family, "n": n, "layers": rng.randint(1, 5), "samples": size(1, 100), "obs": rng.randint(1, 4)}
    if family == "qaoa":
        return {"family": family, "n": 2 * rng.randint(4, 12), "p": rng.randint(1, 8)}
    if family == "uneven":
        lo = rng.randint(6, 14)
        return {"family": family, "members": rng.randint(3, 12), "n_min": lo, "n_max": lo + rng.randint(1, 4),
                "layers": rng.randint(2, 10), "structure": rng.randint(0, 999)}
    if family == "apply":
        return {"family": family, "n": rng.randint(8, 25), "gates": size(30, 300), "structure": rng.randint(0, 999)}
    if family == "expect":
        return {"family": family, "n": rng.randint(8, 21), "terms": size(10, 500), "structure": rng.randint(0, 999)}
    if family == "sample":
        return {"family": family, "n": rng.randint(6, 21), "layers": rng.randint(1, 3), "shots": size(100, 10000)}
    if family == "noise":
        return {"family": family, "n": rng.randint(4, 13), "layers": rng.randint(1, 3), "shots": size(10, 200)}
    return {"family": family, "n": rng.randint(3, 8), "layers": rng.randint(1, 3)}


# ------------------------------------------------------------------------------ circuits as lists
def _hea(n, layers):
    ops, k = [], 0
    for _ in range(layers):
        for name in ("RY", "RZ"):
            for q in range(n):
                ops.append((name, (q,), (), (k,)))
                k += 1
        ops += [("X", (q + 1,), (q,), ()) for q in range(n - 1)]
    return ops, k


def _hea_terms(n, rng):
    terms = [(((i, "Z"), (i + 1, "Z")), rng.normal()) for i in range(n - 1)]
    return terms + [(((i, "X"),), rng.normal()) for i in range(n)]


def _qnn(n, layers):
    ops = [("RX", (q,), (), (q,)) for q in range(n)]
    k = n
    for _ in range(layers):
        for name in ("RY", "RZ"):
            for q in range(n):
                ops.append((name, (q,), (), (k,)))
                k += 1
        ops += [("Z", ((q + 1) % n,), (q,), ()) for q in range(n)]
    return ops, k


def _cubic_graph(n):
    """Edges of a 3-regular graph on n (even) vertices: a cycle and a fixed random perfect matching."""
    rng = random.Random(n)
    cycle = {tuple(sorted((i, (i + 1) % n))) for i in range(n)}
    while True:
        v = list(range(n))
        rng.shuffle(v)
        chords = {tuple(sorted(v[i:i + 2])) for i in range(0, n, 2)}
        if not chords & cycle:
            return sorted(cycle | chords)


def _qaoa(n, p):
    edges = _cubic_graph(n)
    ops = [("H", (q,), (), ()) for q in range(n)]
    for layer in range(p):
        ops += [("Rzz", e, (), (2 * layer,)) for e in edges]
        ops += [("RX", (q,), (), (2 * layer + 1,)) for q in range(n)]
    return ops, 2 * p, [(((i, "Z"), (j, "Z")), 1.0) for i, j in edges]


def _u3_brick(n, layers):
    ops, k = [], 0
    for layer in range(layers):
        for q in range(n):
            ops.append(("U3", (q,), (), (k, k + 1, k + 2)))
            k += 3
        ops += [("X", (q + 1,), (q,), ()) for q in range(layer % 2, n - 1, 2)]
    return ops, k


def _mixed(n, gates, structure):
    rng = random.Random(1000 * n + structure)
    ops, k = [], 0
    kinds = ["H", "S", "T", "RX", "RY", "RZ", "U3", "PhaseShift", "X", "Z", "SWAP", "Rxx", "Rzz", "FSim"]
    for _ in range(gates):
        name = rng.choice(kinds)
        qs = rng.sample(range(n), 3)
        two = name in ("SWAP", "Rxx", "Rzz", "FSim")
        targets = tuple(qs[:2]) if two else (qs[0],)
        ctrl = (qs[2],) if name in ("X", "Z") or (not two and rng.random() < 0.2) else ()
        count = {"U3": 3, "FSim": 2, "RX": 1, "RY": 1, "RZ": 1, "PhaseShift": 1, "Rxx": 1, "Rzz": 1}.get(name, 0)
        ops.append((name, targets, ctrl, tuple(range(k, k + count))))
        k += count
    return ops, k


def _random_terms(n, count, structure, max_weight):
    rng = np.random.default_rng(1000 * n + structure)
    terms = {}
    for _ in range(count):
        qs = sorted(int(q) for q in rng.permutation(n)[:int(rng.integers(1, max_weight + 1))])
        terms[tuple((q, "XYZ"[int(rng.integers(0, 3))]) for q in qs)] = float(rng.normal())
    return list(terms.items())


def _circuit(ops, names):
    circ = Circuit()
    for name, targets, ctrl, ps in ops:
        gate = getattr(G, name)
        gate = gate(*[names[p] for p in ps]) if ps else gate
        circ += gate.on(list(targets), list(ctrl)) if ctrl else gate.on(list(targets))
    return circ


def _ham(terms):
    op = QubitOperator()
    for paulis, c in terms:
        op += QubitOperator(" ".join(f"{p}{q}" for q, p in paulis), float(c))
    return Hamiltonian(op)


def _uneven_members(case):
    rng = random.Random(case["structure"])
    lo, hi = case["n_min"], case["n_max"]
    ns = [lo, hi] + [rng.randint(lo, hi) for _ in range(case["members"] - 2)]
    return [(n, *_u3_brick(n, case["layers"]), _random_terms(n, 10, i, 4)) for i, n in enumerate(ns)]


def _channels(n):
    return [G.DepolarizingChannel(0.02).on(q) for q in range(n)] + [G.AmplitudeDampingChannel(0.05).on(q) for q in range(n)]


def _noisy(n, layers, names, measure):
    ops, k = _hea(n, layers)
    per = len(ops) // layers
    circ = Circuit()
    for layer in range(layers):
        circ += _circuit(ops[layer * per:(layer + 1) * per], names)
        for c in _channels(n):
            circ += c
    if measure:
        for q in range(n):
            circ += G.Measure(f"m{q}").on(q)
    return circ


def _names(k):
    return [f"p{i}" for i in range(k)]


def _angles(rng, *shape):
    return rng.uniform(0, 2 * np.pi, size=shape)


# ------------------------------------------------------------------------------ inputs of a case
def _inputs(case, seed):
    """What the seed makes: numpy arrays in float64 (float32 values where the case's tensors are float32)."""
    rng = np.random.default_rng(seed)
    f = case["family"]
    f32 = lambda a: a.astype(np.float32).astype(np.float64)  # noqa: E731
    if f in ("vqe", "density"):
        n = case["n"]
        return {"params": _angles(rng, 2 * n * case["layers"]), "terms": _hea_terms(n, rng)}
    if f == "hea":
        n = case["n"]
        return {"params": f32(_angles(rng, case["batch"], 2 * n * case["layers"])), "terms": _hea_terms(n, rng)}
    if f == "qnn":
        n = case["n"]
        return {"enc": f32(rng.uniform(0, np.pi, size=(case["samples"], n))), "w": f32(_angles(rng, 2 * n * case["layers"])),
                "target": f32(rng.uniform(-1, 1, size=(case["samples"], case["obs"])))}
    if f == "qaoa":
        return {"params": f32(rng.uniform(0, np.pi, size=2 * case["p"]))}
    if f == "uneven":
        return {"params": [_angles(rng, 3 * m[0] * case["layers"]) for m in _uneven_members(case)]}
    if f == "apply":
        return {"params": _angles(rng, _mixed(case["n"], case["gates"], case["structure"])[1])}
    if f == "expect":
        return {"params": _angles(rng, 2 * case["n"])}
    return {"params": _angles(rng, 2 * case["n"] * case["layers"]), "seed": int(rng.integers(1, 1 << 20))}


def prepare(case, seed):
    f, x = case["family"], _inputs(case, seed)
    s = {"case": case}
    if f in ("vqe", "density"):
        n = case["n"]
        names = _names(2 * n * case["layers"])
        circ = _circuit(_hea(n, case["layers"])[0], names) if f == "vqe" else _noisy(n, case["layers"], names, False)
        sim = Simulator("mqvector_b200" if f == "vqe" else "mqmatrix_b200", n, dtype=complex128)
        s.update(sim=sim, params=x["params"], grad=sim.get_expectation_with_grad(_ham(x["terms"]), circ))
    elif f == "hea":
        n = case["n"]
        circ = _circuit(_hea(n, case["layers"])[0], _names(2 * n * case["layers"])).as_encoder()
        sim = Simulator("mqvector_b200", n, dtype=complex64)
        s.update(sim=sim, op=MQEncoderOnlyOps(sim.get_expectation_with_grad(_ham(x["terms"]), circ)),
                 params=torch.tensor(x["params"], dtype=torch.float32, device="cuda", requires_grad=True))
    elif f == "qnn":
        n = case["n"]
        ops, k = _qnn(n, case["layers"])
        names = [f"x{q}" for q in range(n)] + [f"w{i}" for i in range(k - n)]
        circ = _circuit(ops[:n], names).as_encoder() + _circuit(ops[n:], names)
        sim = Simulator("mqvector_b200", n, dtype=complex64)
        hams = [_ham([(((q, "Z"),), 1.0)]) for q in range(case["obs"])]
        layer = MQLayer(sim.get_expectation_with_grad(hams, circ), torch.tensor(x["w"], dtype=torch.float32)).cuda()
        s.update(sim=sim, layer=layer, enc=torch.tensor(x["enc"], dtype=torch.float32, device="cuda"),
                 target=torch.tensor(x["target"], dtype=torch.float32, device="cuda"))
    elif f == "qaoa":
        ops, k, terms = _qaoa(case["n"], case["p"])
        sim = Simulator("mqvector_b200", case["n"], dtype=complex64)
        s.update(sim=sim, op=MQAnsatzOnlyOps(sim.get_expectation_with_grad(_ham(terms), _circuit(ops, _names(k)))),
                 params=torch.tensor(x["params"], dtype=torch.float32, device="cuda", requires_grad=True))
    elif f == "uneven":
        members = [(n, _circuit(ops, _names(k)), _ham(terms)) for n, ops, k, terms in _uneven_members(case)]
        s.update(batch=CircuitBatch(members, dtype=complex64), params=[torch.tensor(p).cuda() for p in x["params"]])
    elif f == "apply":
        ops, k = _mixed(case["n"], case["gates"], case["structure"])
        s.update(sim=Simulator("mqvector_b200", case["n"], dtype=complex64), circ=_circuit(ops, _names(k)), params=x["params"])
    elif f == "expect":
        n = case["n"]
        sim = Simulator("mqvector_b200", n, dtype=complex128)
        sim.apply_circuit(_circuit(_hea(n, 1)[0], _names(2 * n)), x["params"])
        s.update(sim=sim, ham=_ham(_random_terms(n, case["terms"], case["structure"], 4)))
    elif f == "sample":
        n = case["n"]
        circ = _circuit(_hea(n, case["layers"])[0], _names(2 * n * case["layers"]))
        for q in range(n):
            circ += G.Measure(f"m{q}").on(q)
        s.update(sim=Simulator("mqvector_b200", n, dtype=complex128), circ=circ, params=x["params"], seed=x["seed"])
    else:
        n = case["n"]
        circ = _noisy(n, case["layers"], _names(2 * n * case["layers"]), True)
        s.update(sim=Simulator("mqvector_b200", n, dtype=complex128), circ=circ, params=x["params"], seed=x["seed"])
    return s


def run(state):
    case = state["case"]
    f = case["family"]
    if f in ("vqe", "density"):
        return state["grad"](state["params"])
    if f in ("hea", "qaoa"):
        out = state["op"](state["params"])
        (g,) = torch.autograd.grad(out.sum(), state["params"])
        return out.detach(), g
    if f == "qnn":
        layer = state["layer"]
        layer.zero_grad(set_to_none=True)
        out = layer(state["enc"])
        loss = torch.nn.functional.mse_loss(out, state["target"])
        loss.backward()
        return out.detach(), loss.detach(), layer.weight.grad
    if f == "uneven":   # a float32 optimiser's view of the batch's values and gradients
        fs, gs = state["batch"](state["params"])
        return [x.real.float() for x in fs], [g.float() for g in gs]
    sim = state["sim"]
    if f == "apply":
        sim.reset()
        sim.apply_circuit(state["circ"], state["params"])
        return sim.backend.state
    if f == "expect":
        return np.complex128(sim.get_expectation(state["ham"]))
    return sim.sampling(state["circ"], state["params"], shots=case["shots"], seed=state["seed"]).samples


# ------------------------------------------------------------------------------ necessary work
def work(case):
    """Bytes: the final state written once (and read once where it is measured), and the results; flops:
    the gates on the state, and in a gradient the gates on the state and every adjoint state once more
    with one inner product per parameter."""
    f = case["family"]
    c64 = f in ("hea", "qnn", "qaoa", "uneven", "apply")
    if f == "uneven":
        parts = [(n, ops, 1, 1) for n, ops, _, _ in _uneven_members(case)]
    elif f == "qnn":
        parts = [(case["n"], _qnn(case["n"], case["layers"])[0], case["samples"], case["obs"])]
    elif f == "qaoa":
        parts = [(case["n"], _qaoa(case["n"], case["p"])[0], 1, 1)]
    elif f == "apply":
        parts = [(case["n"], _mixed(case["n"], case["gates"], case["structure"])[0], 1, 0)]
    elif f == "expect":
        dim = float(1 << case["n"])
        return {"bytes": 16 * dim, "flops": 8 * dim * case["terms"]}
    else:
        n = 2 * case["n"] if f == "density" else case["n"]
        grads = 0 if f in ("sample", "noise") else 1
        times = case["shots"] if f == "noise" else case.get("batch", 1)
        ops = _hea(case["n"], case["layers"])[0]
        parts = [(n, ops * (2 if f == "density" else 1), times, grads)]
    total = {"bytes": 0.0, "flops": 0.0}
    for n, ops, times, grads in parts:
        amps = float(1 << n) * times
        per = sum({"X": 0, "RZ": 6, "Rzz": 6, "Z": 1, "S": 1, "T": 6, "PhaseShift": 3, "SWAP": 0, "RY": 6, "RX": 6, "H": 6}
                  .get(g[0], 14) for g in ops)
        slots = sum(len(g[3]) for g in ops)
        total["bytes"] += amps * (8 if c64 else 16) * (1 if f == "apply" else 2 + grads)
        total["flops"] += amps * (per * (1 if not grads else 2 + grads) + 4 * slots * grads)
    return total


# ------------------------------------------------------------------------------ 64-bit reference
_I2 = [[1, 0], [0, 1]]


def _matrix(name, t):
    """The gate's matrix (bit 0 of the index is the first target) and its derivatives; a diagonal gate
    as the list of its diagonal."""
    c, s = (math.cos(t[0] / 2), math.sin(t[0] / 2)) if t else (1, 0)
    e = lambda a: complex(math.cos(a), math.sin(a))  # noqa: E731
    r = math.sqrt(0.5)
    if name == "RX":
        return [[c, -1j * s], [-1j * s, c]], [[[-s / 2, -0.5j * c], [-0.5j * c, -s / 2]]]
    if name == "RY":
        return [[c, -s], [s, c]], [[[-s / 2, -c / 2], [c / 2, -s / 2]]]
    if name == "RZ":
        return [e(-t[0] / 2), e(t[0] / 2)], [[-0.5j * e(-t[0] / 2), 0.5j * e(t[0] / 2)]]
    if name == "Rzz":
        a, b = e(-t[0] / 2), e(t[0] / 2)
        return [a, b, b, a], [[-0.5j * a, 0.5j * b, 0.5j * b, -0.5j * a]]
    if name == "PhaseShift":
        return [1, e(t[0])], [[0, 1j * e(t[0])]]
    if name == "U3":
        p, la = e(t[1]), e(t[2])
        return ([[c, -la * s], [p * s, p * la * c]],
                [[[-s / 2, -la * c / 2], [p * c / 2, -p * la * s / 2]], [[0, 0], [1j * p * s, 1j * p * la * c]],
                 [[0, -1j * la * s], [0, 1j * p * la * c]]])
    if name == "Rxx":
        m = np.eye(4, dtype=complex) * c
        for i in range(4):
            m[i, 3 - i] = -1j * s
        return m.tolist(), None
    if name == "FSim":
        c2, s2 = math.cos(t[0]), math.sin(t[0])
        return [[1, 0, 0, 0], [0, c2, -1j * s2, 0], [0, -1j * s2, c2, 0], [0, 0, 0, e(-t[1])]], None
    return {"H": [[r, r], [r, -r]], "X": [[0, 1], [1, 0]], "Z": [1, -1], "S": [1, 1j], "T": [1, e(math.pi / 4)],
            "SWAP": [[1, 0, 0, 0], [0, 0, 1, 0], [0, 1, 0, 0], [0, 0, 0, 1]]}[name], []


def _slices(psi, n, targets, ctrl):
    """Views of psi by the targets' bits (controls set)."""
    out = []
    for r in range(1 << len(targets)):
        fixed = {q: 1 for q in ctrl}
        fixed.update({q: r >> i & 1 for i, q in enumerate(targets)})
        shape, index, top = [], [], n
        for q in sorted(fixed, reverse=True):
            shape += [1 << (top - q - 1), 2]
            index += [slice(None), fixed[q]]
            top = q
        out.append(psi.view(*shape, 1 << top)[tuple(index)])
    return out


def _apply(psi, n, targets, ctrl, m, adjoint=False):
    v = _slices(psi, n, targets, ctrl)
    if not isinstance(m[0], (list, tuple)):
        for x, d in zip(v, m):
            d = complex(d).conjugate() if adjoint else d
            if d != 1:
                x.mul_(d)
        return
    if adjoint:
        m = [[complex(m[j][i]).conjugate() for j in range(len(m))] for i in range(len(m))]
    new = []
    for row in m:
        acc = None
        for a, x in zip(row, v):
            if a != 0:
                acc = x * a if acc is None else acc.add_(x, alpha=a)
        new.append(acc)
    for x, y in zip(v, new):
        x.copy_(y)


def _inner(lam, psi, n, targets, ctrl, d):
    """Re <lam| D |psi>."""
    a, b = _slices(lam, n, targets, ctrl), _slices(psi, n, targets, ctrl)
    total = 0.0
    for i, x in enumerate(a):
        for j, y in enumerate(b):
            w = (d[i] if i == j else 0) if not isinstance(d[0], (list, tuple)) else d[i][j]
            if w != 0:
                total = total + w * torch.sum(x.conj() * y)
    return total.real


def _apply_terms(psi, n, terms):
    out = torch.zeros_like(psi)
    idx = torch.arange(1 << n, device=psi.device)
    for paulis, c in terms:
        flip = sum(1 << q for q, p in paulis if p in "XY")
        sign, ny = None, 0
        for q, p in paulis:
            if p in "YZ":   # P|i> picks (-1)^bit of the ket's index
                b = (idx >> q) & 1
                sign = b if sign is None else sign ^ b
                ny += p == "Y"
        y = psi if sign is None else psi * (1 - 2 * sign)
        y = y[idx ^ flip] if flip else y
        out.add_(y, alpha=c * 1j ** ny)
    return out


def _zero(n):
    psi = torch.zeros(1 << n, dtype=torch.complex128, device="cuda" if torch.cuda.is_available() else "cpu")
    psi[0] = 1
    return psi


def _gradient(n, ops, p, hams):
    """f[h] and df[h]/dp of one parameter vector by the adjoint method."""
    psi = _zero(n)
    mats = [_matrix(name, [p[i] for i in ps]) for name, _, _, ps in ops]
    for (_, t, c, _), (m, _) in zip(ops, mats):
        _apply(psi, n, t, c, m)
    lams = [_apply_terms(psi, n, h) for h in hams]
    f = torch.stack([torch.sum(psi.conj() * la).real for la in lams])
    g = [[0.0] * len(p) for _ in hams]
    for (_, t, c, ps), (m, ds) in zip(reversed(ops), reversed(mats)):
        _apply(psi, n, t, c, m, adjoint=True)
        for h, la in enumerate(lams):
            for i, d in zip(ps, ds):
                g[h][i] = g[h][i] + 2 * _inner(la, psi, n, t, c, d)
            _apply(la, n, t, c, m, adjoint=True)
    return f, torch.stack([torch.stack(row) for row in g])


def _exact_density(case, x):
    """Tr(H rho) of the noisy circuit with dense matrices; the gradient by torch's autograd."""
    n, layers = case["n"], case["layers"]
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    p = torch.tensor(x["params"], device=dev, requires_grad=True)
    ops = _hea(n, layers)[0]
    per = len(ops) // layers
    const = lambda m: torch.tensor(m, dtype=torch.complex128, device=dev)  # noqa: E731
    pauli = [const(m) for m in (_I2, [[0, 1], [1, 0]], [[0, -1j], [1j, 0]], [[1, 0], [0, -1]])]
    rho = (_zero(n)[:, None] * _zero(n)[None, :].conj()).view([2] * (2 * n))

    def both(rho, ks, qs):   # sum_k K rho K^dag on qubits qs (axis n - 1 - q is qubit q)
        out, d = 0, len(qs)
        rows, cols = [n - 1 - q for q in qs], [2 * n - 1 - q for q in qs]
        for k in ks:
            k = k.view([2] * (2 * d))
            y = torch.movedim(torch.tensordot(k, rho, dims=(list(range(d, 2 * d)), rows)), list(range(d)), rows)
            y = torch.movedim(torch.tensordot(k.conj(), y, dims=(list(range(d, 2 * d)), cols)), list(range(d)), cols)
            out = out + y
        return out

    dep = [pauli[0] * math.sqrt(1 - 0.75 * 0.02)] + [m * math.sqrt(0.02 / 4) for m in pauli[1:]]
    damp = [const([[1, 0], [0, math.sqrt(0.95)]]), const([[0, math.sqrt(0.05)], [0, 0]])]
    cnot = const([[1, 0, 0, 0], [0, 1, 0, 0], [0, 0, 0, 1], [0, 0, 1, 0]])
    for layer in range(layers):
        for name, t, c, ps in ops[layer * per:(layer + 1) * per]:
            if name == "X":
                rho = both(rho, [cnot], [c[0], t[0]])
                continue
            a = p[ps[0]] / 2
            gen = pauli[2] if name == "RY" else pauli[3]
            rho = both(rho, [torch.cos(a) * pauli[0] - 1j * torch.sin(a) * gen], [t[0]])
        for ks in (dep, damp):
            for q in range(n):
                rho = both(rho, ks, [q])
    rho = rho.reshape(1 << n, 1 << n)
    h = torch.stack([_apply_terms(col, n, x["terms"]) for col in torch.eye(1 << n, dtype=torch.complex128, device=dev)]).T
    f = torch.sum(h * rho.T).real
    (g,) = torch.autograd.grad(f, p)
    return f.detach(), g


def exact(case, seed):
    f, x = case["family"], _inputs(case, seed)
    if f in ("sample", "noise"):
        return None
    if f in ("vqe", "density"):
        v, g = (_gradient(case["n"], _hea(case["n"], case["layers"])[0], x["params"].tolist(), [x["terms"]]) if f == "vqe"
                else _exact_density(case, x))
        return v.reshape(1, 1).to(torch.complex128), g.reshape(1, 1, -1).to(torch.complex128)
    if f == "hea":
        ops = _hea(case["n"], case["layers"])[0]
        rows = [_gradient(case["n"], ops, p.tolist(), [x["terms"]]) for p in x["params"]]
        return torch.stack([r[0] for r in rows]), torch.stack([r[1][0] for r in rows])
    if f == "qaoa":
        ops, _, terms = _qaoa(case["n"], case["p"])
        v, g = _gradient(case["n"], ops, x["params"].tolist(), [terms])
        return v.reshape(1, 1), g[0]
    if f == "qnn":
        if case["samples"] * case["obs"] * case["layers"] * case["n"] > 10000:
            return None
        n, (ops, _) = case["n"], _qnn(case["n"], case["layers"])
        hams = [[(((q, "Z"),), 1.0)] for q in range(case["obs"])]
        rows = [_gradient(n, ops, e.tolist() + x["w"].tolist(), hams) for e in x["enc"]]
        out, g = torch.stack([r[0] for r in rows]), torch.stack([r[1][:, n:] for r in rows])
        diff = out - torch.tensor(x["target"], device=out.device)
        return out, (diff ** 2).mean(), torch.einsum("smp,sm->p", g, 2 * diff / diff.numel())
    if f == "uneven":
        rows = [_gradient(n, ops, p.tolist(), [terms]) for (n, ops, _, terms), p in zip(_uneven_members(case), x["params"])]
        return [r[0] for r in rows], [r[1] for r in rows]
    n, psi = case["n"], _zero(case["n"])
    ops = _mixed(n, case["gates"], case["structure"])[0] if f == "apply" else _hea(n, 1)[0]
    for name, t, c, ps in ops:
        _apply(psi, n, t, c, _matrix(name, [x["params"][i] for i in ps])[0])
    if f == "apply":
        return psi
    return torch.sum(psi.conj() * _apply_terms(psi, n, _random_terms(n, case["terms"], case["structure"], 4)))
