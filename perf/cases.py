"""The calls that programs make of the engine, over the sizes they make them at.

Circuits are the seeded generators of ``dqsim.workloads`` (the layered circuits
of the reference's statevector benchmark, U3 + CX brickwork, QFT, and the
hardware-efficient ansatz) and go through the public Python API:

* ``shots``: ``StatevectorSimulator.simulate_shots`` of a terminally measured
  circuit, the call most programs make;
* ``dynamic``: the same call on a circuit with mid-circuit measurements, a
  conditional gate and resets, which runs one trajectory per shot;
* ``state``: ``simulate`` and the whole statevector;
* ``observe``: ``simulate`` and what a program asks of a state too large to
  copy out: marginal probabilities, chosen amplitudes, Pauli expectations;
* ``queries``: the queries alone, on a result that the program keeps;
* ``batch``: ``BatchedCircuits``, many uneven circuits in one run.

Seeded counts are whole numbers that depend on every bit of the running sums,
so the single-precision form is asked for floating results, in single
precision, and counts come from the double-precision form.
"""

import cmath
import math
import sys
from pathlib import Path

import numpy as np
import torch

_PACKAGE = str(Path(__file__).resolve().parents[1] / "classical-quantum-sim-optimizer_b200")
if _PACKAGE not in sys.path:
    sys.path.insert(0, _PACKAGE)

import dqsim  # noqa: E402
from dqsim import _core, workloads  # noqa: E402

MEMORY_MB = 65536  # of 180 GB: room for every size here, as a program of that size sets it


def listed():
    return [
        # The reference benchmark's terminal case: a small circuit asked for a few counts,
        # as a parameter sweep or a classroom notebook does over and over.
        {"name": "shots_12q_layers", "kind": "shots", "circuit": "layers", "qubits": 12, "depth": 8,
         "shots": 256, "precision": "complex128"},
        # The reference benchmark's dynamic case: mid-circuit measurement feeding a gate.
        {"name": "dynamic_10q", "kind": "dynamic", "qubits": 10, "depth": 3, "rounds": 1, "shots": 128,
         "precision": "complex128"},
        # Repeated syndrome-like rounds (measure, conditional gate, reset) on a register of
        # odd size, more shots.
        {"name": "dynamic_15q_rounds", "kind": "dynamic", "qubits": 15, "depth": 2, "rounds": 3, "shots": 300,
         "precision": "complex128"},
        # The reference benchmark's unitary case: a state computed and copied to the host.
        {"name": "state_16q_layers", "kind": "state", "circuit": "layers", "qubits": 16, "depth": 8,
         "precision": "complex128"},
        # The plain workload of the benchmark configuration: 20 qubits, depth 20, 1000 shots.
        {"name": "shots_20q_brickwork", "kind": "shots", "circuit": "brickwork", "qubits": 20, "depth": 20,
         "shots": 1000, "precision": "complex128"},
        # The same at depth 40 on a state far larger than L2 (2 GiB), odd qubit count.
        {"name": "shots_27q_brickwork", "kind": "shots", "circuit": "brickwork", "qubits": 27, "depth": 40,
         "shots": 1000, "precision": "complex128"},
        # QFT in double precision: controlled phases over all pairs, then swaps.
        {"name": "observe_25q_qft", "kind": "observe", "circuit": "qft", "qubits": 25, "depth": 1,
         "precision": "complex128", "execution": "auto"},
        # One launch per operation, the form that profiles and per-operation checks run.
        {"name": "observe_23q_per_gate", "kind": "observe", "circuit": "hea", "qubits": 23, "depth": 6,
         "precision": "complex128", "execution": "per_gate"},
        # A variational step in single precision (tensor-core passes) and its observables.
        {"name": "observe_22q_hea_c64", "kind": "observe", "circuit": "hea", "qubits": 22, "depth": 6,
         "precision": "complex64", "execution": "auto"},
        # The headline size: 30 qubits, depth 40, single precision (8 GiB).
        {"name": "observe_30q_brickwork_c64", "kind": "observe", "circuit": "brickwork", "qubits": 30, "depth": 40,
         "precision": "complex64", "execution": "auto"},
        # A kept result questioned several times.
        {"name": "queries_24q", "kind": "queries", "circuit": "hea", "qubits": 24, "depth": 4, "shots": 2048,
         "precision": "complex128"},
        # Uneven ansatz circuits in one run, 1024 shots and <Z0Z1> each (a population of
        # candidates or a data set of circuits).
        {"name": "batch_64_hea_c64", "kind": "batch", "count": 64, "qmin": 12, "qmax": 20, "dmin": 4, "dmax": 16,
         "shots": 1024, "precision": "complex64"},
    ]


def _log_int(rng, lo, hi):
    return min(hi, int(math.exp(rng.uniform(math.log(lo), math.log(hi + 1)))))


def draw(rng):
    kind = rng.choice(["shots", "shots", "dynamic", "state", "observe", "observe", "queries", "batch"])
    both = rng.choice(["complex128", "complex64"])
    if kind == "shots":
        return {"kind": kind, "circuit": rng.choice(["layers", "brickwork", "qft", "hea"]),
                "qubits": rng.randint(5, 26), "depth": _log_int(rng, 2, 40), "shots": _log_int(rng, 64, 4096),
                "precision": "complex128"}
    if kind == "dynamic":
        return {"kind": kind, "qubits": rng.randint(4, 16), "depth": rng.randint(1, 4), "rounds": rng.randint(1, 3),
                "shots": _log_int(rng, 32, 400), "precision": "complex128"}
    if kind == "state":
        return {"kind": kind, "circuit": rng.choice(["layers", "brickwork", "qft", "hea"]),
                "qubits": rng.randint(5, 20), "depth": _log_int(rng, 2, 24), "precision": both}
    if kind == "observe":
        per_gate = both == "complex128" and rng.random() < 0.3
        return {"kind": kind, "circuit": rng.choice(["brickwork", "qft", "hea"]),
                "qubits": rng.randint(14, 24 if per_gate else 26 if both == "complex128" else 28),
                "depth": _log_int(rng, 2, 24), "precision": both, "execution": "per_gate" if per_gate else "auto"}
    if kind == "queries":
        return {"kind": kind, "circuit": "hea", "qubits": rng.randint(12, 26), "depth": _log_int(rng, 2, 8),
                "shots": _log_int(rng, 64, 4096), "precision": "complex128"}
    return {"kind": kind, "count": _log_int(rng, 8, 64), "qmin": rng.randint(8, 12), "qmax": rng.randint(13, 20),
            "dmin": rng.randint(2, 4), "dmax": rng.randint(5, 16), "shots": _log_int(rng, 128, 1024),
            "precision": both}


def _layers(n, depth, rng):
    """The layers of workloads.benchmark_layers with seeded angles around its own."""
    ins = workloads.benchmark_layers(n, depth)
    shift = rng.uniform(-0.2, 0.2, size=len(ins))
    for op, s in zip(ins, shift):
        for key in ("theta", "phi"):
            if key in op:
                op[key] += float(s)
    return ins


def _measure_all(n):
    return [{"kind": "measure", "qubit": q, "cbit": q} for q in range(n)]


def _circuit(case, seed, measure):
    n, depth = case["qubits"], case["depth"]
    if case["circuit"] == "layers":
        ins = _layers(n, depth, np.random.default_rng(seed))
        return workloads.TransportCircuit(n, ins + (_measure_all(n) if measure else []), n if measure else 0)
    if case["circuit"] == "brickwork":
        return workloads.brickwork(n, depth, seed, measure)
    if case["circuit"] == "hea":
        return workloads.hea(n, depth, seed, measure)
    return workloads.qft(n, seed, measure)


def _dynamic(case, seed):
    """Layers, then rounds of: measure a qubit, a gate on its outcome, reset another
    qubit, layers again; everything measured at the end."""
    n, rng = case["qubits"], np.random.default_rng(seed)
    ins = _layers(n, case["depth"], rng)
    for r in range(case["rounds"]):
        ins.append({"kind": "measure", "qubit": r, "cbit": r})
        ins.append({"kind": "conditional", "condition": {"creg_base": r, "creg_size": 1, "creg_value": 1},
                    "op": {"kind": "x", "qubit": n - 1 - r}})
        if r:
            ins.append({"kind": "reset", "qubit": r})
        ins += _layers(n, case["depth"], rng)
    return workloads.TransportCircuit(n, ins + _measure_all(n), n)


def _simulator(case):
    return dqsim.StatevectorSimulator(seed=7, max_memory_mb=MEMORY_MB, precision=case["precision"],
                                      execution=case.get("execution", "auto"))


def _pauli_strings(n):
    """Neighbouring ZZ terms and one transverse string, as a spin Hamiltonian has."""
    strings = []
    for a in (0, 1, n // 2):
        s = ["I"] * n
        s[n - 1 - a] = s[n - 2 - a] = "Z"
        strings.append("".join(s))
    s = ["I"] * n
    s[n - 1] = "X"
    strings.append("".join(s))
    return strings


def _questions(case, seed):
    """Register parts and basis indices that a program asks about."""
    n, rng = case["qubits"], np.random.default_rng(seed + 1)
    return {
        "part": [int(q) for q in rng.choice(n, size=min(8, n), replace=False)],
        "high": list(range(n - 1, max(-1, n - 11), -1)),
        "indices": rng.integers(0, 1 << n, size=4096).astype(np.uint64),
        "paulis": _pauli_strings(n) if case["circuit"] == "hea" else [],
    }


def _batch_circuits(case, seed):
    return workloads.hea_batch(case["count"], seed, case["qmin"], case["qmax"], case["dmin"], case["dmax"])


def prepare(case, seed):
    kind = case["kind"]
    state = {"case": case, "sim": _simulator(case)}
    if kind == "batch":
        state["batch"] = _core.BatchedCircuits(state["sim"], _batch_circuits(case, seed), shots=case["shots"],
                                               tensor_cores=case["precision"] == "complex64")
        return state
    if kind == "dynamic":
        state["circuit"] = _dynamic(case, seed)
    else:
        state["circuit"] = _circuit(case, seed, kind == "shots")
    state["circuit"].model_dump_json()
    if kind in ("observe", "queries"):
        state["ask"] = _questions(case, seed)
    if kind == "queries":
        state["result"] = state["sim"].simulate(state["circuit"])
    return state


def _real(case, values):
    return np.asarray(values, dtype=np.float32 if case["precision"] == "complex64" else np.float64)


def _amplitudes(case, values):
    return values.astype(np.complex64) if case["precision"] == "complex64" else values


def _table(case, probabilities, qubits):
    """A query's {index: p} as a table."""
    out = np.zeros(1 << len(qubits))
    out[list(probabilities.keys())] = list(probabilities.values())
    return _real(case, out)


def _outcomes(counts):
    """A histogram as the sorted list of its shots' outcomes."""
    keys = sorted(counts)
    bits = np.frombuffer("".join(keys).encode(), dtype=np.uint8).reshape(len(keys), -1) - ord("0")
    values = bits @ (np.int64(1) << np.arange(bits.shape[1] - 1, -1, -1, dtype=np.int64))
    return np.repeat(values, [counts[k] for k in keys])


def _observed(case, ask, result):
    out = {"part": _table(case, result.probabilities(ask["part"]), ask["part"]),
           "high": _table(case, result.probabilities(ask["high"]), ask["high"]),
           "amplitudes": _amplitudes(case, result.amplitudes(ask["indices"]))}
    if ask["paulis"]:
        out["paulis"] = _real(case, [result.expectation_value(p) for p in ask["paulis"]])
    return out


def run(state):
    case, sim = state["case"], state["sim"]
    kind = case["kind"]
    if kind in ("shots", "dynamic"):
        return {"outcomes": _outcomes(sim.simulate_shots(state["circuit"], case["shots"]))}
    if kind == "state":
        return {"statevector": _amplitudes(case, sim.simulate(state["circuit"]).statevector)}
    if kind == "observe":
        return _observed(case, state["ask"], sim.simulate(state["circuit"]))
    if kind == "queries":
        out = _observed(case, state["ask"], state["result"])
        out["sampled"] = _outcomes(state["result"].counts(case["shots"], seed=11))
        return out
    state["batch"].run()
    return {"zz": _real(case, state["batch"].expect_zz())}


# Real operations per amplitude of one gate (a complex product 6, a sum 2): a 2x2
# matrix 14, a phase on half or a quarter of the state 3 or 1.5; moves none.
_GATE_FLOPS = {"u3": 14.0, "ry": 14.0, "h": 14.0, "rz": 6.0, "cp": 1.5, "cz": 0.5}


def _gates_flops(instructions, n):
    return sum(_GATE_FLOPS.get(op["kind"], 0.0) for op in instructions) * (1 << n)


def work(case):
    """A state written once and read once by what is asked of it, and the gates' arithmetic."""
    amp = 8 if case["precision"] == "complex64" else 16
    if case["kind"] == "batch":
        sizes = [c for c in _batch_circuits(case, 0)]
        return {"bytes": float(sum(2 * amp << c.num_qubits for c in sizes)),
                "flops": float(sum(_gates_flops(c.data["instructions"], c.num_qubits) for c in sizes))}
    n = case["qubits"]
    if case["kind"] == "dynamic":
        c = _dynamic(case, 0)
        # Every shot ends in a state of its own; the part before the first measurement is shared.
        first = next(i for i, op in enumerate(c.data["instructions"]) if op["kind"] == "measure")
        ins = c.data["instructions"]
        return {"bytes": float(case["shots"] * 2 * amp << n),
                "flops": float(_gates_flops(ins[:first], n) + case["shots"] * _gates_flops(ins[first:], n))}
    if case["kind"] == "queries":  # a read of the state for each question that covers it
        return {"bytes": float((3 + len(_pauli_strings(n))) * amp << n),
                "flops": float((3 * 3 + 8 * len(_pauli_strings(n))) << n)}
    c = _circuit(case, 0, False)
    return {"bytes": float(2 * amp << n), "flops": float(_gates_flops(c.data["instructions"], n))}


# --------------------------------------------------------------------------
# The same results from plain torch in 64 bits
# --------------------------------------------------------------------------
EXACT_MAX_QUBITS = 26


def _matrix(op):
    if op["kind"] == "h":
        r = math.sqrt(0.5)
        return [[r, r], [r, -r]]
    if op["kind"] == "x":
        return [[0, 1], [1, 0]]
    if op["kind"] == "ry":
        c, s = math.cos(op["theta"] / 2), math.sin(op["theta"] / 2)
        return [[c, -s], [s, c]]
    if op["kind"] == "rz":
        return [[cmath.exp(-0.5j * op["phi"]), 0], [0, cmath.exp(0.5j * op["phi"])]]
    if op["kind"] == "u3":
        c, s = math.cos(op["theta"] / 2), math.sin(op["theta"] / 2)
        return [[c, -cmath.exp(1j * op["lam"]) * s],
                [cmath.exp(1j * op["phi"]) * s, cmath.exp(1j * (op["phi"] + op["lam"])) * c]]
    return None


def _pair(psi, n, a, b):
    """psi as (.., bit of the higher qubit, .., bit of the lower one, ..)."""
    lo, hi = min(a, b), max(a, b)
    return psi.view(1 << (n - 1 - hi), 2, 1 << (hi - lo - 1), 2, 1 << lo)


def _bits(view, a, b, va, vb):
    """The part where qubit a reads va and qubit b reads vb."""
    hi, lo = (va, vb) if a > b else (vb, va)
    return view[:, hi, :, lo, :]


def _exact_state(circuit):
    n = circuit.num_qubits
    device = "cuda" if torch.cuda.is_available() else "cpu"
    psi = torch.zeros(1 << n, dtype=torch.complex128, device=device)
    psi[0] = 1
    for op in circuit.data["instructions"]:
        kind = op["kind"]
        m = _matrix(op)
        if m is not None:
            v = psi.view(1 << (n - 1 - op["qubit"]), 2, 1 << op["qubit"])
            x, y = v[:, 0].clone(), v[:, 1].clone()
            v[:, 0] = m[0][0] * x + m[0][1] * y
            v[:, 1] = m[1][0] * x + m[1][1] * y
        elif kind in ("cx", "cz", "cp"):
            c, t = op["control"], op["target"]
            v = _pair(psi, n, c, t)
            if kind == "cx":
                one, zero = _bits(v, c, t, 1, 1), _bits(v, c, t, 1, 0)
                keep = one.clone()
                one.copy_(zero)
                zero.copy_(keep)
            else:
                _bits(v, c, t, 1, 1).mul_(-1.0 if kind == "cz" else cmath.exp(1j * op["lam"]))
        elif kind == "swap":
            v = _pair(psi, n, op["a"], op["b"])
            one, two = _bits(v, op["a"], op["b"], 0, 1), _bits(v, op["a"], op["b"], 1, 0)
            keep = one.clone()
            one.copy_(two)
            two.copy_(keep)
        elif kind != "measure":
            raise ValueError(f"no plain form of {kind!r}")
    return psi


def _exact_part(psi, n, qubits):
    """Marginal probabilities with qubits[0] as the most significant bit."""
    p = psi.abs().square().view((2,) * n)  # axis n-1-q is qubit q
    rest = [n - 1 - q for q in range(n) if q not in qubits]
    if rest:
        p = p.sum(dim=rest)
    kept = sorted(qubits, reverse=True)  # the axes left, in order
    return p.permute([kept.index(q) for q in qubits]).reshape(-1).cpu().numpy()


def _exact_pauli(psi, n, pauli):
    index = torch.arange(psi.numel(), device=psi.device)
    sign = torch.zeros_like(index)
    flip = 0
    for pos, ch in enumerate(pauli):
        q = n - 1 - pos
        if ch == "Z":
            sign ^= (index >> q) & 1
        elif ch == "X":
            flip |= 1 << q
    return float((psi.conj() * (1 - 2 * sign) * psi[index ^ flip]).sum().real)


def exact(case, seed):
    kind = case["kind"]
    if kind in ("shots", "dynamic"):
        return None
    if kind == "batch":
        zz = []
        for c in _batch_circuits(case, seed):
            zz.append(_exact_pauli(_exact_state(c), c.num_qubits, "I" * (c.num_qubits - 2) + "ZZ"))
        return {"zz": np.array(zz)}
    n = case["qubits"]
    if n > EXACT_MAX_QUBITS:
        return None
    psi = _exact_state(_circuit(case, seed, False))
    if kind == "state":
        return {"statevector": psi.cpu().numpy()}
    ask = _questions(case, seed)
    out = {"part": _exact_part(psi, n, ask["part"]), "high": _exact_part(psi, n, ask["high"]),
           "amplitudes": psi[torch.from_numpy(ask["indices"].astype(np.int64)).to(psi.device)].cpu().numpy()}
    if ask["paulis"]:
        out["paulis"] = np.array([_exact_pauli(psi, n, p) for p in ask["paulis"]])
    return out
