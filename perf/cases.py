"""The work users of this engine have it do, as cases that can be timed.

A case is a dict of plain values.  ``prepare`` makes what a program holds before
the call (a register handle, gate lists, Hamiltonians, draws), ``run`` is one
pass through the package's public entry points, ``work`` the bytes and
operations such a pass cannot do without, and ``exact`` the same outputs in
binary64 by plain torch.

Kinds of pass
  circuit     a register set to |0...0>, a gate list, the whole state read on the device
  grover      the reference's example program: gate list, dump of every qubit, samples
  energy      one evaluation of a variational loop: whole circuit, <H> and every <Z_q> in one call
  expect      <H> of a state that stays on the device
  experiment  a circuit, P(1) of every qubit, samples, then a measurement of the register
  gradient    energy and every derivative by the adjoint method
  batch       many circuits with their own gates and Hamiltonians in one call

``arith``: "c64", "c128" (binary64 arithmetic) or "ff" (complex128 with
FLAG_FAST_C128).  ``repeat`` circuits keep their structure from call to call and
only the angles change, as in a parameter scan: the program has run the
structure before (and waited for its specialised kernels).  The others are run
once by their program, so specialised kernels never come into play (jit off).
"""
import math

import numpy as np
import torch

import kbw_gb300 as kbw
from kbw_gb300 import _native
from kbw_gb300 import circuits as C
from kbw_gb300.dense import batch_circuits_prepare, batch_circuits_run

GRID = {"c64": 8, "c128": 16, "ff": 16}  # bytes per amplitude


def listed():
    return [
        # the reference's own example program, through the C ABI's small calls (latency)
        {"name": "grover_12q", "kind": "grover", "n": 12, "iterations": 50, "shots": 1024, "arith": "ff"},
        # a small VQE's energy evaluation with the entry's default arithmetic
        {"name": "energy_14q_c128", "kind": "energy", "n": 14, "layers": 4, "ham": "tfim", "arith": "c128"},
        # a mid-size VQE's energy evaluation in single precision
        {"name": "energy_19q_c64", "kind": "energy", "n": 19, "layers": 6, "ham": "heisenberg", "arith": "c64"},
        # a small gradient step, odd register size
        {"name": "gradient_17q_ff", "kind": "gradient", "n": 17, "layers": 5, "ham": "tfim", "arith": "ff"},
        # the gradient benchmark: 480 parameters on 24 qubits
        {"name": "gradient_24q_c64", "kind": "gradient", "n": 24, "layers": 10, "ham": "tfim", "arith": "c64"},
        # a circuit run once: every gate kind with up to two controls
        {"name": "once_23q_ff", "kind": "circuit", "n": 23, "family": "random", "size": 300, "repeat": False,
         "arith": "ff"},
        # binary64 gate arithmetic, the default of a complex128 handle
        {"name": "brickwork_25q_c128", "kind": "circuit", "n": 25, "family": "brickwork", "size": 8, "repeat": True,
         "arith": "c128"},
        # single precision, the reference's default, on a large register
        {"name": "brickwork_28q_c64", "kind": "circuit", "n": 28, "family": "brickwork", "size": 20, "repeat": True,
         "arith": "c64"},
        # the headline benchmark: 30 qubits, 20 layers, complex128
        {"name": "brickwork_30q_ff", "kind": "circuit", "n": 30, "family": "brickwork", "size": 20, "repeat": True,
         "arith": "ff"},
        # the observable of the variational benchmarks on a resident state
        {"name": "expect_27q_ff", "kind": "expect", "n": 27, "ham": "tfim", "arith": "ff"},
        # one shot of a whole experiment with every kind of readout
        {"name": "experiment_24q_ff", "kind": "experiment", "n": 24, "layers": 2, "shots": 1024, "arith": "ff"},
        # the batched workload: circuits of 8..20 qubits, 2..8 layers, each with its own Hamiltonian
        {"name": "batch_1024_c64", "kind": "batch", "circuits": 1024, "min_n": 8, "max_n": 20, "arith": "c64"},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["circuit", "circuit", "circuit", "grover", "energy", "expect", "experiment", "gradient",
                       "gradient", "batch"])
    arith = rng.choice(["c64", "c128", "ff"])
    if kind == "circuit":
        family = rng.choice(["brickwork", "random", "hea"])
        n = rng.randint(10, 25 if arith == "c128" else 29)
        size = _log_int(rng, 20, 400) if family == "random" else rng.randint(1, 20 if n < 29 else 12)
        return {"kind": kind, "n": n, "family": family, "size": size, "repeat": rng.random() < 0.6, "arith": arith}
    if kind == "grover":
        return {"kind": kind, "n": rng.randint(6, 14), "iterations": _log_int(rng, 3, 60),
                "shots": _log_int(rng, 16, 4096), "arith": rng.choice(["c128", "ff"])}
    if kind == "energy":
        return {"kind": kind, "n": rng.randint(6, 19), "layers": rng.randint(1, 8),
                "ham": rng.choice(["tfim", "heisenberg", "molecule", "fields"]), "arith": arith}
    if kind == "expect":
        return {"kind": kind, "n": rng.randint(13, 27), "ham": rng.choice(["tfim", "heisenberg", "molecule", "fields"]),
                "arith": arith}
    if kind == "experiment":
        return {"kind": kind, "n": rng.randint(12, 24), "layers": rng.randint(1, 4), "shots": _log_int(rng, 16, 1024),
                "arith": rng.choice(["c128", "ff"])}
    if kind == "gradient":
        n = rng.randint(13, 20 if arith == "c128" else 23)
        return {"kind": kind, "n": n, "layers": rng.randint(1, 10), "ham": rng.choice(["tfim", "heisenberg"]),
                "arith": arith}
    lo = rng.randint(4, 12)
    return {"kind": "batch", "circuits": _log_int(rng, 16, 1024), "min_n": lo, "max_n": rng.randint(lo, 20),
            "arith": arith}


# ---- inputs ---------------------------------------------------------------------
def _hamiltonian(name, n, rng):
    """tfim: ring transverse-field Ising; heisenberg: open XXX chain in a field;
    molecule: Jordan-Wigner strings (two or four X/Y with Z in between, and
    ZZ densities); fields: Z on every qubit, ZZ on random pairs."""
    co = lambda: float(rng.uniform(-1.0, 1.0))  # noqa: E731
    if name == "tfim":
        return C.tfim_ring(n, co() + 1.5, co())
    if name == "heisenberg":
        j, h = co() + 1.5, co()
        out = [(j, [(p, i), (p, i + 1)]) for i in range(n - 1) for p in (C.PAULI_X, C.PAULI_Y, C.PAULI_Z)]
        return out + [(h, [(C.PAULI_Z, i)]) for i in range(n)]
    if name == "fields":
        out = [(co(), [(C.PAULI_Z, i)]) for i in range(n)]
        for _ in range(n):
            a, b = rng.choice(n, size=2, replace=False)
            out.append((co(), [(C.PAULI_Z, int(a)), (C.PAULI_Z, int(b))]))
        return out
    out = []
    for _ in range(4 * n):
        ends = sorted(int(q) for q in rng.choice(n, size=4 if n >= 4 and rng.random() < 0.5 else 2, replace=False))
        terms = {}
        for lo, hi in zip(ends[::2], ends[1::2]):
            for q in range(lo + 1, hi):
                terms[q] = C.PAULI_Z
            terms[lo] = terms[hi] = C.PAULI_X if rng.random() < 0.5 else C.PAULI_Y
        out.append((0.1 * co(), [(p, q) for q, p in sorted(terms.items())]))
    return out + [(co(), [(C.PAULI_Z, i)]) for i in range(n)]


def _circuit(case, rng):
    """The case's gate list.  A repeated structure is the case's own (its seed
    follows from the sizes), with angles of `rng`; else all of it is rng's."""
    n, family, size = case["n"], case["family"], case["size"]
    structure = 1000 * n + size if case["repeat"] else int(rng.integers(1 << 31))
    if family == "hea":
        return C.hea(n, size, rng.uniform(-math.pi, math.pi, 2 * n * size))
    g = C.brickwork(n, size, structure) if family == "brickwork" else C.random_circuit(n, size, structure)
    turn = (C.RX, C.RY, C.RZ) if family == "brickwork" else C.PARAMETRIC  # (S and T keep their angles)
    return [(k, t, c, float(rng.uniform(0.0, 2.0 * math.pi)) if k in turn else a) for k, t, c, a in g]


def _inputs(case, seed):
    """Everything of a case that comes from the seed, on the host."""
    rng = np.random.default_rng([seed, 77])
    kind, n = case["kind"], case.get("n")
    if kind == "circuit":
        return {"gates": _circuit(case, rng)}
    if kind == "grover":
        return {"gates": C.grover(n, int(rng.integers(1 << n)), case["iterations"]),
                "draws": C.uniform_draws(case["shots"], seed)}
    if kind in ("energy", "gradient"):
        layers = case["layers"]
        ham = _hamiltonian(case["ham"], n, rng)
        return {"gates": C.hea(n, layers, rng.uniform(-math.pi, math.pi, 2 * n * layers)),
                "index": C.hea_param_index(n, layers), "params": 2 * n * layers, "ham": ham,
                "hams": [ham] + [[(1.0, [(C.PAULI_Z, q)])] for q in range(n)]}
    if kind == "expect":
        return {"gates": C.hea(n, 2, rng.uniform(-math.pi, math.pi, 4 * n)), "ham": _hamiltonian(case["ham"], n, rng)}
    if kind == "experiment":
        layers = case["layers"]
        return {"gates": C.hea(n, layers, rng.uniform(-math.pi, math.pi, 2 * n * layers)),
                "draws": C.uniform_draws(case["shots"], seed), "bits": C.uniform_draws(n, seed + 1)}
    out = []
    for m, layers, params in C.hea_batch(case["circuits"], seed, case["min_n"], case["max_n"]):
        out.append((m, C.hea(m, layers, params), C.tfim_ring(m, 1.0, 0.5)))
    return {"circuits": out}


def _prec(case):
    return {"prec": "c64" if case["arith"] == "c64" else "c128", "fast_c128": case["arith"] == "ff"}


class _OnDevice:
    """The register's amplitudes in device memory, for torch to view in place."""

    def __init__(self, sim, ptr, n, prec):
        self.sim = sim
        self.__cuda_array_interface__ = {"shape": (1 << n,), "typestr": "<c8" if prec == _native.C64 else "<c16",
                                         "data": (ptr, False), "version": 3, "strides": None}


def _state(sim):
    n, prec, ptr, _ = sim.device_info()
    return torch.as_tensor(_OnDevice(sim, ptr, n, prec), device="cuda")


def _values(case, x):
    """Energies and derivatives in the precision of the register they come
    from: a complex64 program keeps them in single precision, beside its
    parameters."""
    return np.asarray(x, dtype=np.float32 if case["arith"] == "c64" else np.float64)


def _shots(hist, shots):
    """A histogram (states, counts) in arrays of `shots` entries, -1 after its last."""
    out = np.full((2, shots), -1, np.int64)
    out[0, : hist[0].size], out[1, : hist[1].size] = hist
    return out


def prepare(case, seed):
    st = {"case": case, "kind": case["kind"], **_inputs(case, seed)}
    if case["kind"] == "batch":
        st["packed"] = batch_circuits_prepare(st.pop("circuits"))
        return st
    if case["kind"] == "energy":
        # the loop's earlier evaluations of the same ansatz
        run(st)
        run(st)
        return st
    once = case["kind"] == "circuit" and not case["repeat"]
    st["sim"] = sim = kbw.DenseGB300(case["n"], jit=_native.JIT_OFF if once else None, **_prec(case))
    if case["kind"] == "expect":
        sim.apply(st["gates"])
        sim.flush()
    elif not once:
        for _ in range(2):
            run(st)
        sim.jit_wait()
        run(st)
    return st


def run(st):
    kind, case = st["kind"], st["case"]
    if kind == "circuit":
        sim = st["sim"]
        sim.clear()
        sim.apply(st["gates"])
        return _state(sim)
    if kind == "energy":
        return _values(case, kbw.batch_exp_value(case["n"], st["gates"], st["hams"], **_prec(case)))
    if kind == "expect":
        return _values(case, st["sim"].exp_value(st["ham"]))
    if kind == "gradient":
        e, g = st["sim"].adjoint_gradient(st["gates"], st["index"], st["params"], st["ham"])
        return {"energy": _values(case, e), "gradient": _values(case, g)}
    if kind == "batch":
        p = _prec(case)
        return _values(case, batch_circuits_run(st["packed"], p["prec"], p["fast_c128"]))
    sim, qubits = st["sim"], list(range(case["n"]))[::-1]
    sim.clear()
    sim.apply(st["gates"])
    if kind == "grover":
        states, re, im = sim.dump(qubits)
        hist = sim.sample(qubits, case["shots"], st["draws"])
        return {"states": states.astype(np.int64), "re": re, "im": im, "sampled": _shots(hist, case["shots"])}
    ones = np.array([sim.measure_p1(q) for q in range(len(qubits))])
    hist = sim.sample(qubits, case["shots"], st["draws"])
    outcome = sim.measure(qubits, st["bits"])
    return {"p1": ones, "sampled": _shots(hist, case["shots"]), "outcome": outcome, "state": _state(sim)}


# ---- what a pass cannot do without -------------------------------------------------
# operations per amplitude of an uncontrolled gate: X, Y, Z move or negate; H
# adds and scales; RX and RY are two products and a sum per part; P and RZ a
# complex product on one half (RZ up to a global phase)
_OPS = {C.X: 0, C.Y: 0, C.Z: 0, C.H: 4, C.P: 3, C.RX: 6, C.RY: 6, C.RZ: 3}


def _flops(gates, n):
    return float(sum(_OPS[k] * 2.0 ** (n - len(c)) for k, _, c, _ in gates))


def work(case):
    inp = _inputs(case, 1)
    kind = case["kind"]
    if kind == "batch":
        fl = sum(_flops(g, m) + 8.0 * len(h) * 2.0 ** m for m, g, h in inp["circuits"])
        return {"bytes": 32.0 * sum(len(g) for _, g, _ in inp["circuits"]) + 8.0 * case["circuits"], "flops": fl}
    n = case["n"]
    size = float(GRID[case["arith"]]) * 2.0 ** n
    fl = _flops(inp["gates"], n)
    if kind == "expect":
        return {"bytes": size, "flops": 8.0 * len(inp["ham"]) * 2.0 ** n}
    if kind == "energy":
        return {"bytes": size, "flops": fl + (8.0 * len(inp["ham"]) + 4.0 * n) * 2.0 ** n}
    if kind == "gradient":  # forward, and back on two states with one inner product per parameter
        return {"bytes": 2.0 * size, "flops": 3.0 * fl + 8.0 * (len(inp["ham"]) + inp["params"]) * 2.0 ** n}
    if kind == "experiment":  # the state written, read for the readouts, written collapsed
        return {"bytes": 3.0 * size, "flops": fl + 4.0 * n * 2.0 ** n}
    return {"bytes": size, "flops": fl}


# ---- the same outputs in binary64 by plain torch -----------------------------------
def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _zero(n, batch=None):
    psi = torch.zeros((batch or 1, 1 << n), dtype=torch.complex128, device=_device())
    psi[:, 0] = 1.0
    return psi


def _halves(psi, n, target, controls):
    """Views of the amplitudes with the controls set and the target 0 / 1."""
    v = psi.view([psi.shape[0]] + [2] * n)
    ix = [slice(None)] * (n + 1)
    for c in controls:
        ix[n - c] = 1
    ix[n - target] = 0
    a = v[tuple(ix)]
    ix[n - target] = 1
    return a, v[tuple(ix)]


def _apply(psi, n, kind, target, controls, angle, inverse=False):
    """One gate in place.  `angle`: a number, or one per row of psi."""
    a, b = _halves(psi, n, target, controls)
    if torch.is_tensor(angle):
        angle = angle.to(psi.device).view([-1] + [1] * (a.dim() - 1))
        cos, sin = torch.cos, torch.sin
    else:
        cos, sin = math.cos, math.sin
    if inverse:
        angle = -angle
    if kind == C.X:
        t = a.clone()
        a.copy_(b)
        b.copy_(t)
    elif kind == C.Y:
        t = a * 1j
        a.copy_(b).mul_(-1j)
        b.copy_(t)
    elif kind == C.Z:
        b.neg_()
    elif kind == C.H:
        t = a - b
        a.add_(b).mul_(math.sqrt(0.5))
        b.copy_(t).mul_(math.sqrt(0.5))
    elif kind == C.P:
        b.mul_(cos(angle) + 1j * sin(angle))
    elif kind == C.RZ:
        a.mul_(cos(angle / 2) - 1j * sin(angle / 2))
        b.mul_(cos(angle / 2) + 1j * sin(angle / 2))
    else:
        c, s = cos(angle / 2), sin(angle / 2)
        t = a.clone()
        if kind == C.RX:
            a.mul_(c).add_(b * (-1j * s))
            b.mul_(c).add_(t.mul_(-1j * s))
        else:
            a.mul_(c).sub_(b * s)
            b.mul_(c).add_(t.mul_(s))


def _evolve(psi, n, gates, inverse=False):
    for k, t, c, angle in (reversed(gates) if inverse else gates):
        _apply(psi, n, k, t, c, angle, inverse)
    return psi


def _times_pauli(psi, n, terms):
    """The Pauli string's image of psi (a copy)."""
    out = psi.clone()
    for p, q in terms:
        _apply(out, n, {C.PAULI_X: C.X, C.PAULI_Y: C.Y, C.PAULI_Z: C.Z}[p], q, (), 0.0)
    return out


def _times_hamiltonian(psi, n, ham):
    """H psi."""
    out = torch.zeros_like(psi)
    index = torch.arange(1 << n, device=psi.device)
    diagonal = None
    for coef, terms in ham:
        if all(p == C.PAULI_Z for p, _ in terms):
            par = torch.zeros_like(index)
            for _, q in terms:
                par ^= index >> q
            sign = (1 - 2 * (par & 1)).to(torch.float64).mul_(coef)
            diagonal = sign if diagonal is None else diagonal.add_(sign)
        else:
            out.add_(_times_pauli(psi, n, terms), alpha=coef)
    if diagonal is not None:
        out.addcmul_(psi, diagonal.to(torch.complex128)[None])
    return out


def _dot(a, b):
    return (a.conj() * b).sum(-1)


def _expect(psi, n, ham):
    return _dot(psi, _times_hamiltonian(psi, n, ham)).real


def exact(case, seed):
    inp = _inputs(case, seed)
    kind, n = case["kind"], case.get("n")
    if kind == "batch":
        return _exact_batch(inp["circuits"])
    psi = _evolve(_zero(n), n, inp["gates"])
    if kind == "circuit":
        out = psi.view(-1)
        return out.to(torch.complex128)
    if kind in ("energy", "expect"):
        e = float(_expect(psi, n, inp["ham"])[0])
        if kind == "expect":
            return np.array(e)
        w = (psi.real.square() + psi.imag.square()).view([2] * n)
        z = [float(w.select(n - 1 - q, 0).sum() - w.select(n - 1 - q, 1).sum()) for q in range(n)]
        return np.array([e] + z)
    if kind == "gradient":
        return _exact_gradient(psi, n, inp)
    if kind == "grover":
        out = psi.view(-1).cpu().numpy()
        # (samples are whole numbers; every basis state is in the dump)
        return {"states": None, "re": out.real.copy(), "im": out.imag.copy(), "sampled": None}
    w = (psi.real.square() + psi.imag.square()).view([2] * n)
    ones = np.array([float(w.select(n - 1 - q, 1).sum()) for q in range(n)])
    # (the collapsed state is scaled by the engine's own outcome probabilities)
    return {"p1": ones, "sampled": None, "outcome": None, "state": None}


def _exact_gradient(psi, n, inp):
    lam = _times_hamiltonian(psi, n, inp["ham"])
    energy = float(_dot(psi, lam).real[0])
    grad = torch.zeros(inp["params"], dtype=torch.float64, device=psi.device)
    pauli = {C.RX: C.X, C.RY: C.Y, C.RZ: C.Z}
    for (k, t, c, angle), p in zip(reversed(inp["gates"]), reversed(inp["index"])):
        if p >= 0:  # dU/dtheta = -i/2 P U: dE/dtheta = Im <lambda|P|psi>
            image = psi.clone()
            _apply(image, n, pauli[k], t, c, 0.0)
            grad[p] += _dot(lam, image).imag[0]
        _apply(psi, n, k, t, c, angle, True)
        _apply(lam, n, k, t, c, angle, True)
    return {"energy": np.array(energy), "gradient": grad.cpu().numpy()}


def _exact_batch(circuits):
    """Circuits of one size and depth share their structure: evolved together."""
    out = np.zeros(len(circuits))
    groups = {}
    for i, (m, g, _) in enumerate(circuits):
        groups.setdefault((m, len(g)), []).append(i)
    for (m, _), members in groups.items():
        step = max(1, (1 << 26) >> m)
        for at in range(0, len(members), step):
            part = members[at: at + step]
            psi = _zero(m, len(part))
            lists = [circuits[i][1] for i in part]
            for row in zip(*lists):
                k, t, c, _ = row[0]
                angles = torch.tensor([x[3] for x in row], dtype=torch.float64)
                _apply(psi, m, k, t, c, angles if k in C.PARAMETRIC else 0.0)
            out[part] = _expect(psi, m, circuits[part[0]][2]).cpu().numpy()
    return out
