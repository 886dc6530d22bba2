"""Rotation-phase plans of circuits with CX between any qubits: address maps that CX has
changed a lot, on the CPU (plans interpreted against the oracle) and on the GPU.

Tolerance: the fused path's 1e-12; a few thousand gates on unit-norm states round to below
1e-13.
"""
import math
import struct

import numpy as np
import pytest

import _oracle
from _circuits import JsonCircuit, g
from _sweep_emu import canonical, emulate, plan
from dqsim_bosonic_b200 import _native as nat
from dqsim_bosonic_b200.circuit import decode_circuit_json, encode
from dqsim_bosonic_b200.statevector import run_program

ATOL = 1e-12


def u3(rng, q):
    return g("u3", q, *[float(x) for x in rng.uniform(0, 6, 3)])


def all_to_all(n, layers, rng):
    insts = []
    for _ in range(layers):
        insts += [u3(rng, q) for q in range(n)]
        insts += [g("cx", a, b) for a in range(n) for b in range(a + 1, n)]
    return insts


def pauli_evolution(n, strings, rng):
    insts = []
    for _ in range(strings):
        qs = rng.permutation(n)[: rng.integers(2, min(n, 8) + 1)].tolist()
        ps = [rng.integers(3) for _ in qs]
        ladder = [g("cx", a, b) for a, b in zip(qs, qs[1:])]
        insts += [x for q, p in zip(qs, ps) for x in [[g("h", q)], [g("rx", q, math.pi / 2)], []][p]]
        insts += ladder + [g("rz", qs[-1], float(rng.uniform(0, 6)))] + ladder[::-1]
        insts += [x for q, p in zip(qs, ps) for x in [[g("h", q)], [g("rx", q, -math.pi / 2)], []][p]]
    return insts


def random_cx(n, gates, rng, share, diagonal=False):
    """`share` of u3, the rest CX on any two qubits (half of it cz, cp and rzz)."""
    insts = []
    for _ in range(gates):
        a, b = rng.permutation(n)[:2].tolist()
        if rng.random() < share:
            insts.append(u3(rng, a))
        elif diagonal and rng.random() < 0.5:
            insts.append([g("cz", a, b), g("cp", a, b, 0.4), g("rzz", a, b, 0.9)][rng.integers(3)])
        else:
            insts.append(g("cx", a, b))
    return insts


def smallest(n, _, rng):
    # three CX onto qubit 10's address and two that pass it on: thread bits reach half the banks
    return [g("rx", 0, 0.7)] + [g("cx", a, b) for a, b in [(1, 2), (3, 2), (6, 2), (3, 10), (2, 10)]]


def outside(n, cxs, rng, controls=1, targets=8):
    """CX controlled from outside the tile: each phase takes four."""
    return [u3(rng, 0)] + [g("cx", n - 1 - i % controls, i // controls % targets) for i in range(cxs)]


def outside_pairs(n, cxs, rng):
    """The same, then a phase for every pair of qubits: a last flush of every size."""
    pairs = [g("cp", a, b, float(rng.uniform(0, 6))) for a in range(n) for b in range(a + 1, n)]
    return outside(n, cxs, rng) + pairs


FAMILIES = {
    "outside": outside,
    "outside_one": lambda n, k, rng: outside(n, k, rng, 1, 1),
    "outside_many": lambda n, k, rng: outside(n, k, rng, 5),
    "outside_pairs": outside_pairs,
    "smallest": smallest,
    "all_to_all": all_to_all,
    "pauli": pauli_evolution,
    "cx_half": lambda n, k, rng: random_cx(n, k, rng, 0.5),
    "cx_most": lambda n, k, rng: random_cx(n, k, rng, 0.1),
    "cx_nearly_all": lambda n, k, rng: random_cx(n, k, rng, 0.02),
    "cx_diagonal": lambda n, k, rng: random_cx(n, k, rng, 0.1, True),
}


def program(kind, n, size, seed):
    insts = FAMILIES[kind](n, size, np.random.default_rng(seed))
    return encode(decode_circuit_json(JsonCircuit(n, [g("u3", 0, 0.3, 0.2, 0.1)] + insts).model_dump_json()))


def oracle_case(kind, n, size, seed):
    prog = program(kind, n, size, seed)
    rng = np.random.default_rng(seed)
    v = rng.normal(size=1 << n) + 1j * rng.normal(size=1 << n)
    v /= np.linalg.norm(v)
    want, _, rc, _ = _oracle.run(prog, 0, v)
    assert rc == 0
    return prog, v, want


SMALL = [("smallest", 11, 0), ("all_to_all", 11, 3), ("all_to_all", 13, 2), ("pauli", 11, 20), ("pauli", 14, 12),
         ("cx_half", 11, 400), ("cx_half", 12, 1000), ("cx_most", 11, 200), ("cx_most", 12, 1000), ("cx_most", 14, 400),
         ("cx_nearly_all", 12, 400), ("cx_diagonal", 11, 300), ("cx_diagonal", 13, 500),
         # programs of more than one sweep's room
         ("outside", 14, 200), ("outside", 13, 800), ("outside_one", 14, 800), ("outside_many", 16, 480),
         ("outside_pairs", 13, 60), ("outside_pairs", 13, 80), ("outside_pairs", 13, 120), ("outside_pairs", 14, 160), ("outside_pairs", 13, 280), ("outside_pairs", 13, 320)]


@pytest.mark.parametrize("kind,n,size", SMALL)
@pytest.mark.parametrize("seed", range(4))
def test_plans_match_oracle(engine_lib, kind, n, size, seed):
    prog, v, want = oracle_case(kind, n, size, seed)
    got, perm, _ = emulate(prog, v)
    assert np.max(np.abs(canonical(got, perm) - want)) < ATOL


# sizes the oracle is slow for: every program has a plan, of rotation phases
@pytest.mark.parametrize("kind,size", [("all_to_all", 1), ("all_to_all", 5), ("pauli", 30), ("cx_half", 1000),
                                       ("cx_most", 3000), ("cx_nearly_all", 1000), ("cx_diagonal", 3000),
                                       ("outside", 3000), ("outside_one", 800), ("outside_many", 2000),
                                       ("outside_pairs", 120)])
@pytest.mark.parametrize("n", [17, 20, 24, 30])
def test_every_program_has_a_plan(engine_lib, kind, size, n):
    for seed in range(8):
        blobs = plan(program(kind, n, size, seed))[0]
        assert blobs and all(struct.unpack_from("<I", b, 112)[0] for b in blobs)


@pytest.mark.parametrize("n,kind,cxs", [(14, "outside", 200), (20, "outside", 480), (20, "outside_many", 480)])
def test_cx_from_one_control_share_phases(engine_lib, n, kind, cxs):
    # four CX a phase, whatever their controls outside the tile
    blobs = plan(program(kind, n, cxs, 0))[0]
    assert sum(struct.unpack_from("<4I", b, 0)[2] for b in blobs) <= cxs // 4 + 4 * len(blobs)


@pytest.mark.gpu
@pytest.mark.parametrize("kind,n,size,seed", [(k, n, s, 1) for k, n, s in SMALL]
                         + [("all_to_all", 20, 2, 0), ("cx_most", 20, 600, 0), ("cx_diagonal", 18, 600, 0)])
def test_kernel(gpu, kind, n, size, seed):
    prog, v, want = oracle_case(kind, n, size, seed)
    st = nat.State(n, 0)
    st.upload(v)
    run_program(st, prog, 0, nat.SEM_SIMULATE, nat.EXEC_FUSED)
    assert np.max(np.abs(st.download() - want)) < ATOL


@pytest.mark.gpu
def test_batch_items(gpu):
    # tiles of 2^12 amplitudes and 8 thread bits, as a batch's larger items run
    from dqsim_bosonic_b200.batch import run_batch

    cases = [("all_to_all", 17, 1), ("cx_most", 17, 500), ("cx_diagonal", 17, 400), ("pauli", 18, 15),
             ("outside", 17, 900), ("outside_pairs", 17, 200)]
    progs = [program(k, n, s, 3) for k, n, s in cases]
    _, states, st = run_batch(progs, range(len(progs)), want_states=True)
    for (k, n, s), prog, got in zip(cases, progs, states):
        assert np.max(np.abs(got - _oracle.run(prog, 0)[0])) < ATOL, (k, n, s)
    assert st.engine_items == 0
