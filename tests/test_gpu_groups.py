"""Gates applied several in one pass against the same gates launched one by one.

The arithmetic is the same, so the states are equal bit for bit.  A profiled run
times every gate and therefore launches them singly.
"""
import numpy as np
import pytest

from _circuits import JsonCircuit, cond, g, random_gate
from dqsim_bosonic_b200 import _native as nat
from dqsim_bosonic_b200.circuit import decode_circuit_json, encode
from dqsim_bosonic_b200.statevector import run_program

pytestmark = pytest.mark.gpu


def both(insts, n, ncbits=0):
    prog = encode(decode_circuit_json(JsonCircuit(n, insts, ncbits).model_dump_json()))
    rng = np.random.default_rng(n)
    v = rng.normal(size=1 << n) + 1j * rng.normal(size=1 << n)
    v /= np.linalg.norm(v)
    out = []
    for profile in (False, True):
        st = nat.State(n, 0)
        st.upload(v)
        bits, prof = run_program(st, prog, 5, nat.SEM_SIMULATE, nat.EXEC_PER_GATE, 0, profile)
        out.append((st.download().view(np.uint64), bits, prof))
    (a, ba, pa), (b, bb, pb) = out
    assert np.array_equal(a, b) and np.array_equal(ba, bb)
    assert (pa.apply_one_qubit_calls, pa.apply_n_qubit_calls) == (pb.apply_one_qubit_calls, pb.apply_n_qubit_calls)
    return pa.kernel_launches, pb.kernel_launches


@pytest.mark.parametrize("n,seed", [(8, 0), (13, 1), (14, 2), (16, 3)])
def test_random_gates(gpu, n, seed):
    rng = np.random.default_rng(seed)
    insts = []
    while len(insts) < 200:
        # runs on a few qubits (grouped), low ones, high ones or any
        k = int(rng.integers(1, 6))
        qs = rng.permutation(n)[:max(k, 1)]
        for _ in range(int(rng.integers(1, 8))):
            d = random_gate(rng, n if rng.random() < 0.3 else max(k, 1))
            if all(q < len(qs) for q in d["qubits"]) and rng.random() < 0.8:
                d = {f: (int(qs[x]) if isinstance(x, int) else x) for f, x in d.items() if f not in ("qubits", "params")}
                d["qubits"], d["params"] = [], []
            insts.append(d)
    fewer, singly = both(insts, n)
    assert fewer < singly


@pytest.mark.parametrize("n", [13, 15])
def test_groups_end_at_measurements_and_conditions(gpu, n):
    rng = np.random.default_rng(n)
    insts = []
    for r in range(6):
        insts += [random_gate(rng, n) for _ in range(6)]
        insts += [g("measure", r, r), g("reset", r + 1)]
        insts += [cond(r, 1, 1, g("rx", q, 0.3 + q)) for q in range(3)]
        insts += [g("cx", 0, 1), g("swap", n - 1, 0), g("t", 0), g("cz", 2, 3), g("rzz", 0, n - 2, 0.4)]
    both(insts, n, 6)
