"""The work that a program has this framework do, as cases that can be timed.

Each case is one pass through the public entry points of ``wqc_cuda``: whole
circuits on one state, circuits read layer by layer, a layer on a loaded state,
many circuits in one batch, readout of a loaded state, a gradient, and the two
kinds of contraction tree.  ``run`` resets the state where the pass starts from
|0...0>, so a state can be run any number of times.

The outputs are what does not depend on the gauge of the singular vectors: the
state vector, amplitudes, expectation values, gradients, shots, and the bonds
as whole numbers.
"""
from __future__ import annotations

import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "wqc-core_b200"))

import wqc_cuda as W  # noqa: E402
from wqc_cuda import circuits as C  # noqa: E402
from wqc_cuda import exact as X  # noqa: E402
from wqc_cuda import exact_plan as XP  # noqa: E402
from wqc_cuda import network as N  # noqa: E402
from wqc_cuda import network_plan as NP  # noqa: E402

PRECISION = {"fp64": W.PRECISION_FP64, "fp32": W.PRECISION_FP32}
RULE = {"reference": W.SPLIT_RULE_REFERENCE, "exact": W.SPLIT_RULE_EXACT}


def listed():
    return [
        # The smallest call: a short circuit on a few qubits, read as a state
        # vector (a notebook, a unit test, one point of a parameter scan).
        {"name": "circuit_8q_chi16", "kind": "circuit", "gates": "brickwork", "n": 8, "depth": 6, "chi": 16,
         "rule": "reference", "precision": "fp64"},
        # The brickwork of the tests and the benchmark, at its own size: bonds
        # reach chi_max and every later split truncates.
        {"name": "circuit_16q_chi32", "kind": "circuit", "gates": "brickwork", "n": 16, "depth": 20, "chi": 32,
         "rule": "reference", "precision": "fp64"},
        # The same kind of circuit in the precision form, an odd register and a
        # bond that is no power of two.
        {"name": "circuit_19q_chi48_fp32", "kind": "circuit", "gates": "brickwork", "n": 19, "depth": 16, "chi": 48,
         "rule": "reference", "precision": "fp32"},
        # The headline's circuit family (random one-qubit gates, CZ/CNOT
        # brickwork, routed long-range CNOTs) at its chi_max, on a register
        # whose amplitudes are still read in earnest; exact splits.
        {"name": "circuit_28q_chi128", "kind": "circuit", "gates": "random", "n": 28, "depth": 10, "chi": 128,
         "rule": "exact", "precision": "fp64"},
        # The largest bond the backend takes: two-site matrices of 512 x 512.
        {"name": "circuit_20q_chi256", "kind": "circuit", "gates": "blocks", "n": 20, "depth": 9, "chi": 256,
         "rule": "exact", "precision": "fp64"},
        # The trace loop: the amplitudes of every qubit are read before each
        # layer, so the host waits for the device at every step.
        {"name": "trace_20q_chi64", "kind": "trace", "n": 20, "depth": 12, "chi": 64},
        # One brickwork step on a state that comes from elsewhere at a fixed
        # bond (a compressed state of low rank), under the reference's split
        # rule: uploads, range-finder splits of 250 x 250, state vector back.
        # (The reference's test matrix keeps the rank of such a state at odd
        # bonds; at 128 its rows repeat and the result is rounding alone.)
        {"name": "loaded_step_16q_chi125", "kind": "loaded", "n": 16, "chi": 125, "rank": 12},
        # Many independent circuits of mixed width, depth and bond in one batch.
        {"name": "batch_48", "kind": "batch", "slices": 48, "lo": 16, "hi": 28, "depth": 14, "chi": 64},
        # Readout of a wide state that is in hand: energy, one-site
        # amplitudes, shots.
        {"name": "readout_50q_chi128", "kind": "readout", "n": 50, "chi": 128, "shots": 1000},
        # A variational step on the 32-qubit ansatz: energy and its gradient by
        # the adjoint, with checkpoints.
        {"name": "gradient_32q_chi64", "kind": "gradient", "n": 32, "layers": 6, "chi": 64},
        # An exact contraction tree at the widest state it admits, for 64 basis
        # vectors at once.
        {"name": "exact_tree_25q", "kind": "exact_tree", "n": 25, "depth": 20},
        # A network contraction tree of a two-dimensional circuit.
        {"name": "network_tree_25q", "kind": "network_tree", "side": 5, "depth": 12},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["circuit", "circuit", "circuit", "trace", "loaded", "batch", "readout", "gradient",
                       "exact_tree", "network_tree"])
    if kind == "circuit":
        gates = rng.choice(["brickwork", "brickwork", "random", "blocks"])
        n = {"brickwork": rng.randint(4, 20), "random": rng.randint(12, 28), "blocks": rng.randint(8, 20)}[gates]
        depth = {"brickwork": rng.randint(2, 20), "random": rng.randint(3, 8), "blocks": rng.randint(2, 9)}[gates]
        # Cuts of the random family at small bonds fall between equal singular
        # values (its gates are partly Clifford): what is kept is then arbitrary.
        chi = rng.randint(80, 160) if gates == "random" else _log(rng, 8, 160)
        return {"kind": kind, "gates": gates, "n": n, "depth": depth, "chi": chi,
                "rule": "exact", "precision": rng.choice(["fp64", "fp64", "fp64", "fp32"])}
    if kind == "trace":
        return {"kind": kind, "n": rng.randint(8, 24), "depth": rng.randint(2, 12), "chi": 64}
    if kind == "loaded":
        return {"kind": kind, "n": rng.randint(4, 16), "chi": 2 * rng.randint(50, 62) + 1,
                "rank": rng.randint(3, 12)}
    if kind == "batch":
        lo = rng.randint(8, 20)
        return {"kind": kind, "slices": _log(rng, 2, 48), "lo": lo, "hi": rng.randint(lo, 28),
                "depth": rng.randint(4, 14), "chi": rng.choice([16, 32, 64])}
    if kind == "readout":
        return {"kind": kind, "n": rng.randint(8, 50), "chi": _log(rng, 8, 128), "shots": _log(rng, 16, 1000)}
    if kind == "gradient":
        return {"kind": kind, "n": rng.randint(6, 32), "layers": rng.randint(2, 6), "chi": 64}
    if kind == "exact_tree":
        return {"kind": kind, "n": rng.randint(6, 25), "depth": rng.randint(3, 20)}
    return {"kind": kind, "side": rng.randint(2, 4), "depth": rng.randint(3, 12)}


# --- inputs ------------------------------------------------------------------

def _turned(gates, seed):
    """The same circuit with rotation angles of this seed."""
    turn = np.isin(gates["kind"], (C.RX, C.RY, C.RZ))
    gates["angle"][turn] = np.random.default_rng(seed).uniform(0.0, 2.0 * math.pi, int(turn.sum()))
    return gates


def _gates(case, seed):
    n, depth = case["n"], case["depth"]
    make = {"brickwork": C.ry_rz_brickwork, "random": C.random_layers, "blocks": C.large_chi}[case["gates"]]
    return _turned(C.gates_array(make(n, depth, 20261204)), seed)


def _slices(case, seed):
    """(width, chi_max, gates) of every slice; chi_max is one of chi, chi/2, chi/4."""
    shape = np.random.default_rng(case["slices"])
    out = []
    for i in range(case["slices"]):
        n = int(shape.integers(case["lo"], case["hi"] + 1))
        depth = int(shape.integers(max(2, case["depth"] // 3), case["depth"] + 1))
        out.append((n, case["chi"] >> (i % 3), C.gates_array(C.ry_rz_brickwork(n, depth, 1000 * seed + i))))
    return out


def _bonds(n, chi):
    return [min(2 ** min(i, n - i, 30), chi) for i in range(n + 1)]


def _random_mps(n, chi, seed):
    """Right-canonical random sites of norm 1, as numpy arrays [l][2][r]."""
    rng = np.random.default_rng(seed)
    b = _bonds(n, chi)
    sites = []
    for q in range(n):
        l, r = b[q], b[q + 1]
        a = rng.standard_normal((2 * r, l)) + 1j * rng.standard_normal((2 * r, l))
        sites.append(np.ascontiguousarray(np.linalg.qr(a)[0].conj().T.reshape(l, 2, r)))
    return sites


def _padded_mps(n, chi, rank, seed):
    """A random state of bond rank `rank` carried at bond `chi` on every inner
    bond, its norm brought down as truncation does (no split renormalises)."""
    rng = np.random.default_rng(seed)
    core = [0.03 * t for t in _random_mps(n, rank, seed)]
    frames = [np.ones((1, 1))]
    for q in range(n - 1):
        r = core[q].shape[2]
        a = rng.standard_normal((chi, r)) + 1j * rng.standard_normal((chi, r))
        frames.append(np.linalg.qr(a)[0])
    frames.append(np.ones((1, 1)))
    return [np.ascontiguousarray(np.einsum("xa,asb,yb->xsy", frames[q], core[q], frames[q + 1].conj(), optimize=True))
            if q else np.ascontiguousarray(np.einsum("asb,yb->asy", core[q], frames[q + 1].conj()))
            for q in range(n)]


def _step(n):
    """A brickwork step: a rotation on every qubit, then CZ / CNOT on the even and on the odd pairs."""
    gates = [C.g1(C.RY, q, 0.3 + 0.1 * q) for q in range(n)]
    for first in (0, 1):
        gates += [C.g2(C.CNOT if q % 4 < 2 else C.CZ, q, q + 1) for q in range(first, n - 1, 2)]
    return C.gates_array(gates)


def _tree_circuit(case, seed):
    if case["kind"] == "exact_tree":
        return _turned(C.ry_cnot_brickwork(case["n"], case["depth"]), seed)
    return _turned(C.grid(case["side"], case["depth"]), seed)


def _basis_vectors(n, seed):
    return np.random.default_rng(seed + 1).integers(0, 2**n, size=64, dtype=np.uint64)


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case}
    if kind == "circuit":
        s["gates"] = _gates(case, seed)
        s["mps"] = W.CudaMps(case["n"], case["chi"], precision=PRECISION[case["precision"]])
        s["mps"].set_split_rule(RULE[case["rule"]])
        s["observable"] = C.zz_x_observable(case["n"])
    elif kind == "trace":
        n = case["n"]
        all_gates = C.gates_array(C.ry_rz_brickwork(n, case["depth"], seed))
        s["layers"], at = [], 0
        for layer in range(case["depth"]):
            two = len(range(layer % 2, n - 1, 2))
            s["layers"].append((all_gates[at:at + 2 * n], all_gates[at + 2 * n:at + 2 * n + two]))
            at += 2 * n + two
        s["mps"] = W.CudaMps(n, case["chi"])
    elif kind == "loaded":
        s["sites"] = _padded_mps(case["n"], case["chi"], case["rank"], seed)
        s["gates"] = _step(case["n"])
        s["mps"] = W.CudaMps(case["n"], case["chi"])
    elif kind == "batch":
        slices = _slices(case, seed)
        s["gates"] = [g for _, _, g in slices]
        s["batch"] = W.CudaBatch([n for n, _, _ in slices], [c for _, c, _ in slices])
    elif kind == "readout":
        s["mps"] = W.CudaMps(case["n"], case["chi"])
        for q, t in enumerate(_random_mps(case["n"], case["chi"], seed)):
            s["mps"].set_site(q, t)
        s["observable"] = C.zz_x_observable(case["n"])
        s["seed"] = seed
    elif kind == "gradient":
        s["gates"], s["pidx"], _ = C.hea_ansatz(case["n"], case["layers"], seed)
        s["checkpoints"] = C.hea_checkpoints(case["n"], case["layers"])
        s["observable"] = C.zz_x_observable(case["n"])
    elif kind == "exact_tree":
        s["gates"] = _tree_circuit(case, seed)
        s["tree"] = XP.plan_greedy(case["n"], s["gates"])
        s["bits"] = _basis_vectors(case["n"], seed)
        s["contractor"] = X.ExactContractor()
    else:
        s["gates"] = _tree_circuit(case, seed)
        s["tree"] = NP.greedy_tree(case["side"] ** 2, s["gates"])
        s["contractor"] = N.NetworkContractor()
    return s


# --- one pass ----------------------------------------------------------------

def _read(m, n, observable):
    if n <= 20:
        return {"state": m.contract_to_statevector(), "bonds": m.bond_dims()}
    return {"amplitudes": m.site_amplitudes_many(range(n)), "zero": np.array(m.amplitude_at_compact_zero()),
            "energy": np.array(m.expectation(*observable)), "bonds": m.bond_dims()}


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "circuit":
        m = state["mps"]
        m.reset()
        m.apply_gates(state["gates"])
        return {**_read(m, case["n"], state["observable"]), "kept": m.split_records()["chi"].copy()}
    if kind == "trace":
        m = state["mps"]
        m.reset()
        reads = []
        for one, two in state["layers"]:
            m.apply_gates(one)
            reads.append(m.site_amplitudes_many(range(case["n"])))
            m.apply_adjacent_disjoint_gates(two)
        reads.append(m.site_amplitudes_many(range(case["n"])))
        return {"reads": np.stack(reads), "bonds": m.bond_dims()}
    if kind == "loaded":
        m = state["mps"]
        m.reset()
        for q, t in enumerate(state["sites"]):
            m.set_site(q, t)
        m.apply_gates(state["gates"])
        return {"state": m.contract_to_statevector(), "bonds": m.bond_dims(),
                "kept": m.split_records()["chi"].copy()}
    if kind == "batch":
        b = state["batch"]
        b.reset()
        b.apply_slices(state["gates"])
        return {"amplitudes": b.amplitudes(), "bonds": b.bond_dims()}
    if kind == "readout":
        m = state["mps"]
        return {"energy": np.array(m.expectation(*state["observable"])),
                "amplitudes": m.site_amplitudes_many(range(case["n"])),
                "shots": m.sample(range(min(case["n"], 62)), case["shots"], state["seed"]).astype(np.int64)}
    if kind == "gradient":
        f, grad = W.adjoint_gradient(case["n"], case["chi"], state["gates"], state["pidx"], *state["observable"],
                                     checkpoints=state["checkpoints"])
        return {"energy": f, "gradient": grad}
    if kind == "exact_tree":
        return state["contractor"].contract(case["n"], state["gates"], state["tree"], state["bits"])
    return {"amplitude": np.array(state["contractor"].contract(case["side"] ** 2, state["gates"], state["tree"]))}


# --- what a pass cannot do without ---------------------------------------------

def _split_work(n, chi, gates):
    """Complex multiply-add flops of the merges and SVDs of a gate list whose
    bonds grow as fast as chi_max lets them."""
    bond = [1] * (n + 1)
    flops = 0.0

    def split(p):
        nonlocal flops
        m, k, r = 2 * bond[p], bond[p + 1], 2 * bond[p + 2]
        lo, hi = min(m, r), max(m, r)
        flops += 8.0 * m * k * r + W.svd_flops(hi, lo)
        bond[p + 1] = min(lo, chi)

    for g in gates:
        kind = int(g["kind"])
        pairs = []
        if kind in (C.CNOT, C.CZ):
            pairs = [(int(g["q0"]), int(g["q1"]))]
        elif kind == C.CCNOT:
            a, b, t = int(g["q0"]), int(g["q1"]), int(g["q2"])
            pairs = [(b, t), (a, t), (b, t), (a, t), (a, b), (a, b)]
        for x, y in pairs:
            lo, hi = min(x, y), max(x, y)
            route = list(range(hi - 1, lo, -1))
            for p in route + [lo] + route[::-1]:
                split(p)
    return flops


def work(case):
    kind = case["kind"]
    if kind == "circuit":
        g = _gates(case, 1)
        out = 16 * 2 ** case["n"] if case["n"] <= 20 else 32 * case["n"]
        return {"bytes": 24 * len(g) + out, "flops": _split_work(case["n"], case["chi"], g)}
    if kind == "trace":
        g = C.gates_array(C.ry_rz_brickwork(case["n"], case["depth"], 1))
        return {"bytes": 24 * len(g) + 32 * case["n"] * (case["depth"] + 1),
                "flops": _split_work(case["n"], case["chi"], g)}
    if kind == "loaded":
        n, chi, r = case["n"], case["chi"], case["rank"]
        side = 2.0 * chi
        # Interior even pairs: the merge and one pass of a rank-2r factorisation.
        per = 8.0 * side * side * chi + 8.0 * side * side * 2 * r
        return {"bytes": 32.0 * chi * chi * n + 16 * 2 ** n, "flops": per * max(1, n // 2 - 2)}
    if kind == "batch":
        slices = _slices(case, 1)
        return {"bytes": sum(24 * len(g) + 16 for _, _, g in slices),
                "flops": sum(_split_work(n, chi, g) for n, chi, g in slices)}
    if kind == "readout":
        b = _bonds(case["n"], case["chi"])
        size = sum(2.0 * b[q] * b[q + 1] for q in range(case["n"]))
        # One transfer of the three-state operator per site, the environments
        # of the shots, and two vector-matrix products per shot and site.
        flops = sum(8.0 * 2 * b[q] * b[q + 1] * (b[q] + b[q + 1]) * 4 for q in range(case["n"]))
        return {"bytes": 16 * size + 8 * case["shots"], "flops": flops + 8.0 * 2 * size * case["shots"]}
    if kind == "gradient":
        g, _, _ = C.hea_ansatz(case["n"], case["layers"], 1)
        fwd = _split_work(case["n"], case["chi"], g)
        return {"bytes": 24 * len(g) + 8 * 2 * case["n"] * case["layers"], "flops": 2 * fwd}
    g = _tree_circuit(case, 1)
    if kind == "exact_tree":
        size = 2.0 ** case["n"]
        return {"bytes": 2 * 16 * size, "flops": 8.0 * size * case["n"] * (case["depth"] - 1)}
    tree = NP.greedy_tree(case["side"] ** 2, g)
    return {"bytes": float(24 * len(g) + tree.get("peak_bytes", 0)), "flops": _tree_flops(case["side"] ** 2, g, tree)}


def _tree_flops(n, gates, tree):
    legs_of = {tuple(ref.items())[0]: list(legs) for ref, legs in NP.leaves(n, gates)}
    flops, nodes = 0.0, []

    def legs(ref):
        (name, index), = ref.items()
        return nodes[index] if name == "node" else legs_of[(name, index)]

    for node in tree["nodes"]:
        a, b = legs(node["left"]), legs(node["right"])
        flops += 8.0 * 2.0 ** len(set(a) | set(b))
        nodes.append(sorted(set(a) ^ set(b)))
    return flops


# --- the same in plain numpy and torch, 64 bits ----------------------------------

def _mat1(kind, angle):
    c, s, r = math.cos(angle / 2), math.sin(angle / 2), math.sqrt(0.5)
    return {
        C.H: np.array([[r, r], [r, -r]]), C.X: np.array([[0, 1], [1, 0]]), C.Y: np.array([[0, -1j], [1j, 0]]),
        C.Z: np.diag([1, -1]), C.S: np.diag([1, 1j]), C.T: np.diag([1, complex(r, r)]),
        C.RX: np.array([[c, -1j * s], [-1j * s, c]]), C.RY: np.array([[c, -s], [s, c]]),
        C.RZ: np.diag([complex(c, -s), complex(c, s)]),
    }[kind].astype(np.complex128)


_CNOT = np.array([[1, 0, 0, 0], [0, 1, 0, 0], [0, 0, 0, 1], [0, 0, 1, 0]], dtype=np.complex128).reshape(2, 2, 2, 2)
_CZ = np.diag([1, 1, 1, -1]).astype(np.complex128).reshape(2, 2, 2, 2)
_SWAP = np.array([[1, 0, 0, 0], [0, 0, 1, 0], [0, 1, 0, 0], [0, 0, 0, 1]], dtype=np.complex128).reshape(2, 2, 2, 2)


class _Mps:
    """Sites [l][2][r]; a two-site gate is an SVD cut at chi, sqrt(S) on both sides."""

    def __init__(self, n, chi, sites=None):
        self.n, self.chi = n, chi
        self.sites = [np.array([[[1.0], [0.0]]], dtype=np.complex128) for _ in range(n)] if sites is None else \
            [t.copy() for t in sites]

    def pair(self, p, u):
        """u[s'][t'][s][t] on sites p, p + 1."""
        a, b = self.sites[p], self.sites[p + 1]
        l, r = a.shape[0], b.shape[2]
        theta = (a.reshape(2 * l, -1) @ b.reshape(b.shape[0], -1)).reshape(l, 2, 2, r)
        theta = np.einsum("xyst,lstr->lxyr", u, theta).reshape(2 * l, 2 * r)
        us, sv, vh = np.linalg.svd(theta, full_matrices=False)
        k = min(max(int((sv > 1e-12).sum()), 1), self.chi)
        root = np.sqrt(sv[:k])
        self.sites[p] = (us[:, :k] * root).reshape(l, 2, k)
        self.sites[p + 1] = (root[:, None] * vh[:k]).reshape(k, 2, r)

    def routed(self, c, t, u):
        lo, hi = min(c, t), max(c, t)
        for p in range(hi - 1, lo, -1):
            self.pair(p, _SWAP)
        self.pair(lo, u if c < t else u.transpose(1, 0, 3, 2))
        for p in range(lo + 1, hi):
            self.pair(p, _SWAP)

    def apply(self, gates):
        for g in gates:
            kind = int(g["kind"])
            if kind in (C.CNOT, C.CZ):
                self.routed(int(g["q0"]), int(g["q1"]), _CNOT if kind == C.CNOT else _CZ)
            else:
                q = int(g["q0"])
                self.sites[q] = np.einsum("xs,lsr->lxr", _mat1(kind, float(g["angle"])), self.sites[q])
        return self

    def dense(self):
        v = np.ones((1, 1), dtype=np.complex128)
        for t in self.sites:  # the later qubit is the higher bit
            v = np.einsum("pl,lsr->spr", v, t).reshape(-1, t.shape[2])
        return v[:, 0]

    def zero(self):
        v = np.ones(1)
        for t in self.sites:
            v = v @ t[:, 0]
        return v[0]

    def site_amplitudes(self):
        """(n, 2): the amplitudes with qubit t at 0 and at 1, each summed over the other qubits."""
        left, right = [np.ones(1)], [np.ones(1)]
        for t in self.sites[:-1]:
            left.append(left[-1] @ t.sum(1))
        for t in self.sites[:0:-1]:
            right.append(t.sum(1) @ right[-1])
        right = right[::-1]
        return np.array([[left[q] @ t[:, s] @ right[q] for s in (0, 1)] for q, t in enumerate(self.sites)])

    def energy(self):
        """<psi| sum Z Z + 0.5 sum X |psi> by left environments: identity, an open Z, the terms done."""
        z, x = np.diag([1.0, -1.0]), np.array([[0.0, 1.0], [1.0, 0.0]])
        one = np.ones((1, 1), dtype=np.complex128)
        env, opened, done = one, None, 0 * one

        def step(e, t, op):
            return np.einsum("xsr,xsq->rq", t.conj(), np.einsum("st,xtq->xsq", op, np.einsum("xy,ytq->xtq", e, t,
                                                                                        optimize=True)),
                             optimize=True)

        for t in self.sites:
            new_done = step(done, t, np.eye(2)) + 0.5 * step(env, t, x)
            if opened is not None:
                new_done = new_done + step(opened, t, z)
            env, opened, done = step(env, t, np.eye(2)), step(env, t, z), new_done
        return complex(done[0, 0])


def _dense_gate(psi, n, g):
    kind, q = int(g["kind"]), int(g["q0"])
    if kind in (C.CNOT, C.CZ):
        t = int(g["q1"])
        lo, hi = min(q, t), max(q, t)
        v = psi.view(2 ** (n - 1 - hi), 2, 2 ** (hi - lo - 1), 2, 2 ** lo)
        if kind == C.CZ:
            v[:, 1, :, 1] *= -1
        elif q == hi:
            v[:, 1] = v[:, 1].flip(2)
        else:
            v[:, :, :, 1] = v[:, :, :, 1].flip(1)
        return
    u = _mat1(kind, float(g["angle"]))
    v = psi.view(2 ** (n - 1 - q), 2, 2 ** q)
    a, b = v[:, 0].clone(), v[:, 1].clone()
    v[:, 0] = complex(u[0, 0]) * a + complex(u[0, 1]) * b
    v[:, 1] = complex(u[1, 0]) * a + complex(u[1, 1]) * b


def _dense(n, gates, psi=None):
    if psi is None:
        psi = torch.zeros(2 ** n, dtype=torch.complex128, device="cuda" if torch.cuda.is_available() else "cpu")
        psi[0] = 1
    for g in gates:
        _dense_gate(psi, n, g)
    return psi


def _ansatz_energy(n, layers, angles):
    """The ansatz as untruncated sites (a CZ ladder doubles every bond) and its
    energy, differentiable in `angles` (layers, n, 2)."""
    cd = torch.complex128
    sign = torch.tensor([[1.0, 1.0], [1.0, -1.0]], dtype=torch.float64).to(cd)  # (-1)^(j s)
    zero = torch.zeros((), dtype=torch.float64)
    sites = []
    for q in range(n):
        t = torch.zeros(1, 2, 1, dtype=cd)
        t[0, 0, 0] = 1
        for layer in range(layers):
            ry, rz = angles[layer, q, 0], angles[layer, q, 1]
            c, s = torch.cos(ry / 2), torch.sin(ry / 2)
            u = torch.stack([torch.stack([c, -s]), torch.stack([s, c])]).to(cd)
            ph = torch.stack([torch.complex(zero, -rz / 2), torch.complex(zero, rz / 2)]).exp()
            t = torch.einsum("s,st,ltr->lsr", ph, u, t)
            if q > 0:  # Z^j from the pair on the left
                l, _, r = t.shape
                t = torch.einsum("js,lsr->ljsr", sign, t).reshape(2 * l, 2, r)
            if q < n - 1:  # the projector of the pair on the right
                l, _, r = t.shape
                t = torch.einsum("ks,lsr->lsrk", torch.eye(2, dtype=cd), t).reshape(l, 2, 2 * r)
        sites.append(t)
    z = torch.tensor([1.0, -1.0], dtype=torch.float64).to(cd)
    one = torch.ones(1, 1, dtype=cd)
    env, opened, done = one, 0 * one, 0 * one
    for t in sites:
        tc = t.conj()

        def step(e, right):
            return torch.einsum("xsr,xsq->rq", tc, torch.einsum("xy,ysq->xsq", e, right))

        tz, tx = z[None, :, None] * t, t.flip(1)
        env, opened, done = step(env, t), step(env, tz), step(done, t) + step(opened, tz) + 0.5 * step(env, tx)
    return done[0, 0].real


def exact(case, seed):
    kind = case["kind"]
    if kind == "circuit":
        n, gates = case["n"], _gates(case, seed)
        if np.any(gates["kind"] == C.CCNOT):
            return None
        m = _Mps(n, case["chi"]).apply(gates)
        if n <= 20:
            return {"state": m.dense(), "bonds": None, "kept": None}
        return {"amplitudes": m.site_amplitudes(), "zero": np.array(m.zero()), "energy": np.array(m.energy()), "bonds": None,
                "kept": None}
    if kind == "trace":
        n = case["n"]
        gates = C.gates_array(C.ry_rz_brickwork(n, case["depth"], seed))
        at, reads, psi = 0, [], None

        def sums():
            return np.array([psi.view(2 ** (n - 1 - q), 2, 2 ** q).sum((0, 2)).cpu().numpy() for q in range(n)])

        for layer in range(case["depth"]):
            two = len(range(layer % 2, n - 1, 2))
            psi = _dense(n, gates[at:at + 2 * n], psi)
            reads.append(sums())
            psi = _dense(n, gates[at + 2 * n:at + 2 * n + two], psi)
            at += 2 * n + two
        reads.append(sums())
        return {"reads": np.stack(reads), "bonds": None}
    if kind == "loaded":
        n = case["n"]
        m = _Mps(n, case["chi"], _padded_mps(n, case["chi"], case["rank"], seed)).apply(_step(n))
        return {"state": m.dense(), "bonds": None, "kept": None}
    if kind == "batch":
        return {"amplitudes": np.array([_Mps(n, chi).apply(g).zero()
                                        for n, chi, g in _slices(case, seed)]), "bonds": None}
    if kind == "readout":
        m = _Mps(case["n"], case["chi"], _random_mps(case["n"], case["chi"], seed))
        return {"energy": np.array(m.energy()), "amplitudes": m.site_amplitudes(), "shots": None}
    if kind == "gradient":
        _, _, params = C.hea_ansatz(case["n"], case["layers"], seed)
        angles = torch.tensor(params.reshape(case["layers"], case["n"], 2), dtype=torch.float64, requires_grad=True)
        f = _ansatz_energy(case["n"], case["layers"], angles)
        f.backward()
        return {"energy": float(f.detach()), "gradient": angles.grad.reshape(-1).numpy()}
    gates = _tree_circuit(case, seed)
    if kind == "exact_tree":
        psi = _dense(case["n"], gates)
        return psi[torch.from_numpy(_basis_vectors(case["n"], seed).astype(np.int64)).to(psi.device)].cpu().numpy()
    return {"amplitude": np.array(complex(_dense(case["side"] ** 2, gates)[0]))}
