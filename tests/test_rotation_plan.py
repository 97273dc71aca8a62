"""complex128 rotation passes (csrc/rotations.cpp, csrc/rotation_pass.cu).

On the CPU a numpy replay of each pass's program, step by step as the kernel
runs it, against the oracle, over every gate kind the form takes, tile sizes
and circuit families; on the GPU the default complex128 path where it can go
wrong (smallest and largest tiles, tiles sharing a CTA, programs too large for
a launch argument, several trajectories).
"""

import struct

import numpy as np
import pytest

from helpers import GATES, Circuit, brickwork, hea, inst, qft, random_circuit
from oracle import oracle as o

import dqsim
from dqsim import _core, workloads

PLAIN, SIGNED, KEPT, IMAG = range(4)
TABLE, SLOTS, MODULI = 1 << 16, 1 << 17, 1 << 18
SLOT_BITS = 9


def parity(x):
    x = np.asarray(x, dtype=np.uint64).copy()
    for s in (32, 16, 8, 4, 2, 1):
        x ^= x >> np.uint64(s)
    return (x & np.uint64(1)).astype(np.int64)


def sign(x):
    return 1 - 2 * parity(x)


def linear(x, vectors):
    """XOR of vectors[b] over the set bits b of x."""
    x = np.asarray(x, dtype=np.int64)
    out = np.zeros_like(x)
    for b, v in enumerate(vectors):
        out ^= ((x >> b) & 1) * int(v)
    return out


def deposit(x, positions):
    return linear(x, [1 << p for p in positions])


def swizzle(p):
    return p ^ (((p >> 3) ^ (p >> 6) ^ (p >> 9) ^ (p >> 12)) & 7)


def pair(word):
    return struct.unpack("<dd", struct.pack("<IIII", *word))


def rotate(a, d, kind, t, u, signs):
    low = d & -d
    for v in range(16):
        if v & low:
            continue
        s = -1 if (signs >> v) & 1 else 1
        assert kind != PLAIN or s == 1
        x, y = a[:, :, v], a[:, :, v ^ d]
        if kind == KEPT:
            x -= s * t * y
            y *= u
            y += s * t * x
        elif kind == IMAG:
            x -= 1j * s * t * y
            y -= 1j * s * u * x
        else:
            x -= s * t * y
            y += s * u * x


def run_phase(a, words, data, head, index):
    at = head[2][1]
    for step in words[head[0][0]:head[0][0] + head[0][1]]:
        todo = [(1 << j, ((step[0] >> (2 * j)) & 3) - 1) for j in range(4) if (step[0] >> (2 * j)) & 3]
        if (step[0] >> 8) & 15:
            todo.append(((step[0] >> 8) & 15, (step[0] >> 12) & 3))
        for d, kind in todo:
            t, u = pair(words[at])
            at, signs, f = at + 1, 0, 1
            if kind != PLAIN:
                signs, mask = words[at][:2]
                at, f = at + 1, sign(mask & index)
            rotate(a, d, kind, t * f, u if kind == KEPT else u * f, signs)
        if step[0] & TABLE:
            a *= np.array([complex(*pair(w)) for w in words[data + step[1]:data + step[1] + 16]])
        if step[0] & (SLOTS | MODULI):
            n, signs = step[3] & 0xFFFF, step[3] >> 16
            first = data + step[2]
            plus = np.ones(index.shape, dtype=np.complex128)
            minus = plus.copy()
            for i in range(n):
                s = sign(words[first + i // 4][i % 4] & index)
                x, y = pair(words[first + (n + 3) // 4 + i])
                if step[0] & SLOTS:
                    plus *= x + 1j * y * s
                    minus *= x - 1j * y * s
                else:
                    plus *= np.where(s < 0, y, x)
                    minus *= np.where(s < 0, x, y)
            for v in range(16):
                a[:, :, v] *= minus if (signs >> v) & 1 else plus


def replay(plan):
    n = plan["n"]
    state = np.zeros(1 << n, dtype=np.complex128)
    state[0] = 1.0
    for p in plan["passes"]:
        tile = p["qubits"]
        m = len(tile)
        words = [tuple(int(x) for x in w) for w in np.array(p["words"], dtype=np.uint32).reshape(-1, 4)]
        outer = np.arange(1 << (n - m))
        index = deposit(outer, [q for q in range(n) if q not in tile])[:, None] | deposit(np.arange(1 << m), tile)
        places = np.empty((outer.size, 1 << m), dtype=np.complex128)
        places[:, swizzle(np.arange(1 << m))] = state[index]
        slot = np.arange(1 << (m - 4))
        for ph in range(p["phases"]):
            head = words[3 * ph:3 * ph + 3]
            halves = [h for w in (head[0][2:], head[1], head[2][:1]) for x in w for h in (x & 0xFFFF, x >> 16)]
            full = linear(slot, halves[4:4 + m - 4])[:, None] ^ linear(np.arange(16), halves[:4])[None, :]
            assert np.array_equal(np.sort(full.ravel()), np.arange(1 << m))  # every place once
            a = places[:, full]
            run_phase(a, words, p["data"], head, slot[None, :] | outer[:, None] << SLOT_BITS)
            places[:, full] = a
        e = np.arange(1 << m)
        at = linear(e, p["out_dir"])[None, :] ^ p["out_const"] ^ linear(outer, p["out_outer"][:n - m])[:, None]
        flips = parity(p["sign_local"] & e)[None, :] ^ parity(p["sign_outer"] & outer)[:, None] ^ p["sign_const"]
        state[index] = np.take_along_axis(places, at, axis=1) * (1 - 2 * flips)
    return state


def oracle_state(circuit):
    return o.OracleSimulator(seed=1).simulate(circuit).statevector


def layers(n, depth):
    return workloads.TransportCircuit(n, workloads.benchmark_layers(n, depth))


@pytest.mark.parametrize("tile", [5, 8, 10])
@pytest.mark.parametrize("maker", [lambda: brickwork(9, 8, seed=1, measure=False), lambda: qft(10, seed=3),
                                   lambda: hea(10, 6, seed=4), lambda: layers(9, 8)])
def test_rotation_passes_reproduce_the_oracle(maker, tile):
    c = maker()
    plan = _core.rotation_plan_dump(c.model_dump_json(), tile)
    assert all(p["ok"] for p in plan["passes"])
    np.testing.assert_allclose(replay(plan), oracle_state(c), atol=1e-13, rtol=0)


def kinds():
    """One instruction of every kind that random circuits draw."""
    found = {}
    for seed in range(40):
        for g in random_circuit(seed, 6, 60):
            found.setdefault((g["kind"], g.get("name")), g)
    return sorted(found.items(), key=str)


@pytest.mark.parametrize("name,gate", kinds(), ids=lambda x: str(x) if isinstance(x, tuple) else "")
def test_every_gate_kind_between_entangling_layers(name, gate):
    before = [inst("u3", qubit=q, theta=0.3 + q, phi=0.2 * q, lam=1.1 * q) for q in range(6)]
    before += [inst("cx", control=q, target=q + 1) for q in range(5)]
    after = [inst("u3", qubit=q, theta=1.3 * q, phi=0.4, lam=-0.7 * q) for q in range(6)]
    c = Circuit(6, before + [gate] + after)
    try:
        plan = _core.rotation_plan_dump(c.model_dump_json(), 6)
    except ValueError:
        assert name[0] == "rc3x"  # wider than any tile operation
        return
    if not all(p["ok"] for p in plan["passes"]):
        assert name[0] in ("rccx", "gate")  # dense matrices that are no Pauli rotation run in register phases
        return
    np.testing.assert_allclose(replay(plan), oracle_state(c), atol=1e-14, rtol=0)


@pytest.mark.gpu
@pytest.mark.parametrize("n,tile", [(5, 5), (6, 5), (9, 5), (9, 9), (13, 13), (14, 13), (15, 12), (16, 0)])
def test_rotation_kernel_against_the_oracle(n, tile):
    for c in (brickwork(n, 7, seed=n, measure=False), qft(n, seed=n), hea(n, 5, seed=n), layers(n, 4)):
        sim = dqsim.StatevectorSimulator(seed=1, tile_qubits=tile)
        assert np.max(np.abs(sim.simulate(c).statevector - oracle_state(c))) <= 1e-12


@pytest.mark.gpu
def test_rotation_programs_larger_than_a_launch_argument():
    c = brickwork(11, 120, seed=2, measure=False)  # one pass holds every operation
    words = [len(p["words"]) // 4 for p in _core.rotation_plan_dump(c.model_dump_json(), 12)["passes"]]
    assert min(words) > 1980
    assert np.max(np.abs(dqsim.StatevectorSimulator(seed=1).simulate(c).statevector - oracle_state(c))) <= 1e-12


@pytest.mark.gpu
@pytest.mark.parametrize("n", [5, 7, 10, 13])
def test_rotation_passes_in_trajectories(n):
    """Batches of states (tiles of several states to a CTA, ragged counts) with seeded counts equal to the oracle's."""
    ins = workloads.benchmark_layers(n, 2) + [inst("measure", qubit=0, cbit=0)] + workloads.benchmark_layers(n, 2)
    c = Circuit(n, ins + [inst("measure", qubit=q, cbit=q) for q in range(n)], n)
    got = dqsim.StatevectorSimulator(seed=3).simulate_shots(c, shots=67)
    assert got == o.OracleSimulator(seed=3).simulate_shots(c, shots=67)


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["one_phase", "brickwork", "qft"])
def test_rotation_passes_with_many_tiles_to_an_sm(kind):
    """1,024 tiles of 12 qubits (six or seven to an SM of 148): two teams of a CTA in turn, ends with one and with both."""
    n = 22
    c = {"one_phase": lambda: Circuit(n, [inst("ry", qubit=q, theta=0.1 + q) for q in range(4)]),
         "brickwork": lambda: brickwork(n, 4, seed=5, measure=False), "qft": lambda: qft(n, seed=3)}[kind]()
    assert np.max(np.abs(dqsim.StatevectorSimulator(seed=1).simulate(c).statevector - oracle_state(c))) <= 1e-12


@pytest.mark.gpu
def test_trajectories_with_many_tiles_to_an_sm():
    ins = workloads.benchmark_layers(13, 2) + [inst("measure", qubit=0, cbit=0)] + workloads.benchmark_layers(13, 2)
    c = Circuit(13, ins + [inst("measure", qubit=q, cbit=q) for q in range(13)], 13)
    got = dqsim.StatevectorSimulator(seed=3).simulate_shots(c, shots=451)  # 902 tiles
    assert got == o.OracleSimulator(seed=3).simulate_shots(c, shots=451)


def moved(n, tile, how):
    """Distinct amplitudes, then relabellings only."""
    ins = [inst("u3", qubit=q, theta=0.3 + q, phi=0.1 * q, lam=0.7) for q in range(n)]
    if how == "cx":
        return Circuit(n, ins + [inst("cx", control=q, target=(q + d) % n) for d in (5, 3, 2) for q in range(n)])
    ins += [inst("swap", a=q, b=n - 1 - q) for q in range(n // 2)]
    if how == "swaps_x_z":
        ins += [inst("x", qubit=q) for q in (1, n - 2, n // 2)] + [inst("z", qubit=q) for q in (2, n - 3)]
    ins += [inst("swap", a=q, b=q + n // 2) for q in range(n // 2)]
    ins += [inst("swap", a=q, b=n - 2 - q) for q in range(1, n // 2 - 1)]
    return Circuit(n, ins)


@pytest.mark.gpu
@pytest.mark.parametrize("how", ["swaps", "swaps_x_z", "cx"])
@pytest.mark.parametrize("n,tile", [(9, 5), (13, 5), (14, 8)])
def test_passes_that_only_move_amplitudes(n, tile, how):
    """Swap networks trade places where they are, other permutations go through tiles; tiles with and without qubit 0."""
    c = moved(n, tile, how)
    passes = _core.rotation_plan_dump(c.model_dump_json(), tile)["passes"]
    assert any(p["phases"] == 0 for p in passes)
    got = dqsim.StatevectorSimulator(seed=1, tile_qubits=tile).simulate(c).statevector
    assert np.max(np.abs(got - oracle_state(c))) <= 1e-13


@pytest.mark.parametrize("n,tile,low", [(19, 12, 0), (20, 12, 2), (20, 11, 0), (21, 13, 2)])
def test_tiles_of_wide_registers_hold_the_low_qubits(n, tile, low):
    ins = [inst("ry", qubit=q, theta=0.1 + q) for q in range(n)] + [inst("cx", control=q, target=(q + 7) % n) for q in range(n)]
    passes = _core.rotation_plan_dump(Circuit(n, ins).model_dump_json(), tile)["passes"]
    assert all(p["ok"] and len(p["qubits"]) == tile for p in passes)
    assert all(set(range(low)) <= set(p["qubits"]) for p in passes)


# What random circuits below draw from: every gate with a rotation form (no dense matrices but RXX).
FORMS = [g for g in GATES if g[0] not in ("rccx", "rc3x")]
SPECIAL = [0.0, np.pi, -np.pi, np.pi / 2, -np.pi / 2, np.pi / 4, 2 * np.pi, 1.0, -0.3]


def form_circuit(seed, n, gates, names=None):
    """Gates with a rotation form on random qubits; a third of the angles are multiples of pi/4 or the like."""
    rng = np.random.default_rng(seed)
    forms = [g for g in FORMS if len(g[1]) <= n and (names is None or g[0] in names)]
    ins = []
    for _ in range(gates):
        kind, qubits, params = forms[int(rng.integers(len(forms)))]
        fields = dict(zip(qubits, rng.choice(n, size=len(qubits), replace=False).tolist()))
        for p in params:
            fields[p] = float(rng.choice(SPECIAL) if rng.random() < 1 / 3 else rng.uniform(-np.pi, np.pi))
        ins.append(inst(kind, **fields))
    return Circuit(n, ins)


def mixed_layers(n, depth, seed, kinds, two):
    """Layers of one-qubit gates (kinds[layer % len] everywhere, or drawn from a tuple of them) and bricks of `two`."""
    rng = np.random.default_rng(seed)
    ins = []
    for layer in range(depth):
        for q in range(n):
            kind = kinds[layer % len(kinds)]
            kind = kind if isinstance(kind, str) else str(rng.choice(kind))
            params = next(g[2] for g in GATES if g[0] == kind)
            ins.append(inst(kind, qubit=q, **{p: float(rng.uniform(-np.pi, np.pi)) for p in params}))
        for a in range(layer % 2, n - 1, 2):
            ins.append(inst("rxx", a=a, b=a + 1, theta=float(rng.uniform(-np.pi, np.pi))) if two == "rxx" else
                       inst(two, control=a, target=a + 1))
    return Circuit(n, ins)


def replay_error(c, tile):
    plan = _core.rotation_plan_dump(c.model_dump_json(), tile)
    assert all(p["ok"] for p in plan["passes"])
    return np.max(np.abs(replay(plan) - oracle_state(c))), plan


def kinds_by_phase(plan):
    """Per phase of every pass, the kinds of its rotations."""
    for p in plan["passes"]:
        words = np.array(p["words"], dtype=np.uint32).reshape(-1, 4).tolist()
        for ph in range(p["phases"]):
            first, steps = words[3 * ph][:2]
            found = set()
            for w in words[first:first + steps]:
                found |= {((w[0] >> (2 * j)) & 3) - 1 for j in range(4) if (w[0] >> (2 * j)) & 3}
                if (w[0] >> 8) & 15:
                    found.add((w[0] >> 12) & 3)
            yield found


# Layers in which rotations without the factor i (RX, SX, RXX) meet those with it.
MIXED = [(("rx", "ry"), "cx"), (("rx", "ry"), "cz"), ((("sx", "t", "h"),), "cx"), ((("sx", "t", "h"),), "cz"),
         ((("rx", "h"),), "cx"), ((("rx", "h"),), "cz"), ((("sx", "u3"),), "cx"), ((("sx", "u3"),), "cz"),
         (("ry",), "rxx"), ((("rx", "ry"),), "rxx")]


@pytest.mark.parametrize("kinds,two", MIXED, ids=str)
def test_layers_of_rotations_with_and_without_the_factor_i(kinds, two):
    for n, depth in ((5, 2), (6, 3), (7, 8), (8, 5), (9, 6), (10, 12)):
        c = mixed_layers(n, depth, n, kinds, two)
        for tile in {5, n}:
            assert replay_error(c, tile)[0] <= 1e-13, (n, depth, tile)


@pytest.mark.parametrize("kinds,two", [(("rx", "ry"), "cx"), ((("sx", "t", "h"),), "cx"), (("ry",), "rxx")], ids=str)
def test_those_layers_hold_phases_of_both_kinds(kinds, two):
    """Kept rotations and rotations without the factor i in one phase, so that the replay above covers it."""
    plan = replay_error(mixed_layers(10, 12, 10, kinds, two), 10)[1]
    assert any({KEPT, IMAG} <= found for found in kinds_by_phase(plan))


@pytest.mark.parametrize("instructions", [
    [inst("sx", qubit=4), inst("cx", control=3, target=4), inst("h", qubit=4), inst("cx", control=3, target=4),
     inst("sx", qubit=4)],
    [inst("rx", qubit=4, theta=1.1), inst("cx", control=3, target=4), inst("ry", qubit=4, theta=1.2),
     inst("cx", control=3, target=4), inst("rx", qubit=4, theta=0.7)],
    [inst("rx", qubit=2, theta=1.0), inst("rxx", a=3, b=0, theta=0.8), inst("rxx", a=4, b=2, theta=0.8),
     inst("h", qubit=2), inst("h", qubit=4)]])
def test_few_gates_that_owe_different_factors(instructions):
    assert replay_error(Circuit(5, instructions), 5)[0] <= 1e-15


@pytest.mark.parametrize("n", [5, 6, 7, 8, 9])
def test_random_circuits_of_every_gate_with_a_rotation_form(n):
    for seed in range(30):
        for gates, names in ((60, None), (25, ("h", "x", "sx", "t", "rx", "ry", "rz", "u3", "cx", "cz", "rxx", "rzz"))):
            c = form_circuit(1000 * n + seed, n, gates, names)
            for tile in {5, min(n, 6 + seed % 3)}:
                assert replay_error(c, tile)[0] <= 1e-13, (seed, gates, tile)


@pytest.mark.gpu
@pytest.mark.parametrize("kinds,two", [(("rx", "ry"), "cx"), ((("sx", "t", "h"),), "cz"), (("ry",), "rxx")], ids=str)
def test_mixed_rotations_on_the_device(kinds, two):
    """The default complex128 form as a state, as shots and in a batch."""
    sizes = [(5, 4), (8, 6), (13, 5), (15, 3)]
    plain = [mixed_layers(n, depth, n, kinds, two) for n, depth in sizes]
    measured = [Circuit(n, c.data["instructions"] + [inst("measure", qubit=q, cbit=q) for q in range(n)], n)
                for (n, _), c in zip(sizes, plain)]
    batch = _core.BatchedCircuits(dqsim.StatevectorSimulator(seed=3), measured, shots=200)
    batch.run()
    for i, (n, _) in enumerate(sizes):
        want = oracle_state(plain[i])
        assert np.max(np.abs(dqsim.StatevectorSimulator(seed=1).simulate(plain[i]).statevector - want)) <= 1e-12
        assert np.max(np.abs(batch.statevector(i, n) - want)) <= 1e-12
        seed = (3 + i * _core.BATCH_SEED_STRIDE) % (1 << 64)
        counts = o.OracleSimulator(seed=seed).simulate_shots(measured[i], shots=200)
        assert dqsim.StatevectorSimulator(seed=seed).simulate_shots(measured[i], shots=200) == counts
        assert batch.counts(i) == counts


def product_of_entries(c):
    """The gates' double entries applied in long double."""
    n = c.data["qregs"]["q"]["size"]
    r = 0.7071067811865476
    psi = np.zeros(1 << n, dtype=np.clongdouble)
    psi[0] = 1
    for op in c.data["instructions"]:
        if op["kind"] in ("cx", "cz"):
            i = np.arange(1 << n)
            held = ((i >> op["control"]) & 1) == 1
            psi = (psi[np.where(held, i ^ (1 << op["target"]), i)] if op["kind"] == "cx" else
                   np.where(held & (((i >> op["target"]) & 1) == 1), -psi, psi))
            continue
        half = op.get("theta", op.get("phi", 0.0)) / 2
        co, si = np.cos(half), np.sin(half)
        m = {"h": [[r, r], [r, -r]], "ry": [[co, -si], [si, co]],
             "rz": [[complex(co, -si), 0], [0, complex(co, si)]]}[op["kind"]]
        v = psi.reshape(1 << (n - 1 - op["qubit"]), 2, 1 << op["qubit"])
        x, y = v[:, 0].copy(), v[:, 1].copy()
        v[:, 0] = np.clongdouble(m[0][0]) * x + np.clongdouble(m[0][1]) * y
        v[:, 1] = np.clongdouble(m[1][0]) * x + np.clongdouble(m[1][1]) * y
    return psi


@pytest.mark.parametrize("gate", [{"kind": "h"}, {"kind": "ry", "theta": 0.3}], ids=lambda g: g["kind"])
def test_the_scale_of_rounded_entries_is_kept(gate):
    """2,400 times one gate, whose entries' norm is 7e-17 (H) and 5e-17 (RY) off one: 1.6e-13 and 1.2e-13 in all.
    The rounding of 2,400 gates (three roundings of 1.1e-16, signs at random) is some 1.6e-14."""
    n = 12
    ins = []
    for layer in range(200):
        ins += [inst(gate["kind"], qubit=q, **{k: v for k, v in gate.items() if k != "kind"}) for q in range(n)]
        ins += [inst("cx", control=q, target=q + 1) for q in range(layer % 2, n - 1, 2)]
    c = Circuit(n, ins)
    got = replay(_core.rotation_plan_dump(c.model_dump_json(), n))
    assert np.linalg.norm((got - product_of_entries(c)).astype(np.complex128)) <= 4e-14


def test_angles_below_the_rounding_of_one_add_up():
    """1,000 turns of 2e-16 with gates between that keep them apart: 1e-13 in an amplitude."""
    ins = [inst("h", qubit=q) for q in range(5)]
    for k in range(1000):
        ins += [inst("rz", qubit=0, phi=2e-16), inst("cz", control=0, target=1 + k % 4)]
    c = Circuit(5, ins)
    got = replay(_core.rotation_plan_dump(c.model_dump_json(), 5))
    assert np.max(np.abs(got - product_of_entries(c))) <= 2e-15


# A U3 whose angles' sum is rounded to 1e-11: its entries are 1e-12 from a unitary matrix.
FAR = [inst("ry", qubit=0, theta=0.77), inst("cx", control=0, target=1),
       inst("u3", qubit=0, theta=-1.348, phi=1e-12, lam=98103.878)]


def test_matrices_further_from_unitary_than_rounding_have_no_rotation_form():
    assert not any(p["ok"] for p in _core.rotation_plan_dump(Circuit(5, FAR).model_dump_json(), 5)["passes"])


@pytest.mark.gpu
def test_matrices_further_from_unitary_than_rounding_are_applied_as_they_are():
    c = Circuit(5, FAR)
    assert np.max(np.abs(dqsim.StatevectorSimulator(seed=1).simulate(c).statevector - oracle_state(c))) <= 1e-15


@pytest.mark.parametrize("tile,tables", [(6, 4), (5, 5)])
def test_controlled_rotations_take_no_phases_between(tile, tables):
    """A ring of CRY as rotations about Y and Z Y, controls in the tile and outside: the tables settle what rotations owe."""
    c = Circuit(6, [inst("ry", qubit=q, theta=0.3 + q) for q in range(6)] +
                [inst("cry", control=q, target=(q + 1) % 6, theta=0.9 + q) for q in range(6)])
    error, plan = replay_error(c, tile)
    assert error <= 1e-15
    assert sum(p["slot_phases"] for p in plan["passes"]) == 0
    assert sum(p["rotations"] for p in plan["passes"]) == 18
    assert sum(p["tables"] for p in plan["passes"]) <= tables


@pytest.mark.parametrize("maker", [lambda: brickwork(5, 90, seed=1, measure=False), lambda: brickwork(9, 60, seed=2, measure=False),
                                   lambda: mixed_layers(8, 90, 3, ("rx", "ry"), "cx"), lambda: form_circuit(4, 9, 900)])
def test_programs_larger_than_a_launch_argument_in_parts(maker):
    """Cut between phases: each part fits, and run one after another they are the whole."""
    c = maker()
    n = c.data["qregs"]["q"]["size"]
    for tile in {5, n}:
        plan = _core.rotation_plan_dump(c.model_dump_json(), tile)
        assert tile < n or any("parts" in p for p in plan["passes"])
        parts = [dict(part, qubits=p["qubits"]) for p in plan["passes"] for part in p.get("parts", [p])]
        assert all(len(p["words"]) // 4 <= 1980 for p in parts)
        for p in plan["passes"]:
            assert sum(part["phases"] for part in p.get("parts", [p])) == p["phases"]
        np.testing.assert_allclose(replay({"n": n, "passes": parts}), oracle_state(c), atol=1e-13, rtol=0)


def test_a_phase_fits_a_launch_argument():
    """The longest phases: many rotations that commute, each with a table before it (X X on all pairs), on 20 qubits."""
    n = 20
    rng = np.random.default_rng(1)
    ins = [inst("rxx", a=a, b=b, theta=float(rng.uniform(-3, 3))) for _ in range(3) for a in range(8) for b in range(a)]
    ins += [inst("ry", qubit=q, theta=0.1 + q) for q in range(n)]
    for p in _core.rotation_plan_dump(Circuit(n, ins + ins).model_dump_json(), 12)["passes"]:
        assert p["ok"]
        assert all(len(part["words"]) // 4 <= 1980 for part in p.get("parts", [p]))


def ring(n, layers, kind):
    """Layers of RY on every qubit and one gate of `kind` on every third (of three qubits: neighbours)."""
    ins = []
    for layer in range(layers):
        ins += [inst("ry", qubit=q, theta=0.3 + q + layer) for q in range(n)]
        for q in range(layer % 3, n - 2, 3):
            ins.append({"cz": inst("cz", control=q, target=q + 1), "cu3": inst("cu3", control=q, target=q + 2, theta=0.4, phi=1.1, lam=q),
                        "ccx": inst("ccx", control1=q, control2=q + 1, target=q + 2),
                        "rxx": inst("rxx", a=q, b=q + 2, theta=0.7)}[kind])
    return Circuit(n, ins)


@pytest.mark.parametrize("n,kind,quicker", [(5, "cu3", True), (9, "cu3", True), (11, "cu3", True), (12, "cu3", False),
                                            (20, "cu3", False), (8, "ccx", True), (8, "rxx", True), (9, "cz", False)])
def test_the_form_of_small_registers(n, kind, quicker):
    assert _core.rotation_plan_dump(ring(n, 6, kind).model_dump_json(), 12)["register_phases_quicker"] == quicker


@pytest.mark.gpu
@pytest.mark.parametrize("n", [5, 8, 9, 10, 11, 12])
@pytest.mark.parametrize("kind", ["cu3", "ccx", "rxx", "cz"])
def test_both_forms_of_small_registers(n, kind):
    """The default against register phases (an explicit fusion width), rotations (an explicit tile) and the oracle."""
    c = ring(n, 6, kind)
    want = oracle_state(c)
    for options in ({}, {"fusion_width": 2}, {"tile_qubits": 12}):
        got = dqsim.StatevectorSimulator(seed=1, **options).simulate(c).statevector
        assert np.max(np.abs(got - want)) <= 1e-13, options


@pytest.mark.gpu
def test_parts_of_a_program_with_many_tiles_to_an_sm():
    """40 layers on 12 of 22 qubits: parts with and without teams, intermediate ones in place."""
    c = Circuit(22, brickwork(12, 40, seed=3, measure=False).data["instructions"])
    passes = _core.rotation_plan_dump(c.model_dump_json(), 12)["passes"]
    assert any(len(p.get("parts", [])) > 1 for p in passes)
    assert np.max(np.abs(dqsim.StatevectorSimulator(seed=1).simulate(c).statevector - oracle_state(c))) <= 1e-12
