"""Sweeps of rotation phases (one-qubit gates split into phases and rotations, X and CX as
address changes): the planner on the CPU, the kernel on the GPU, both against the oracle.

Tolerance: the fused path's 1e-12; the rounding of a few hundred gates on unit-norm states
is below 1e-14.
"""
import math

import numpy as np
import pytest

import _oracle
from _circuits import JsonCircuit, g
from _sweep_emu import canonical, emulate
from dqsim_bosonic_b200 import _native as nat
from dqsim_bosonic_b200.circuit import decode_circuit_json, encode
from dqsim_bosonic_b200.statevector import run_program

ATOL = 1e-12


def circuit(n, depth, seed, special):
    """u3-type gates among X, CX, phases, cp, rzz, swaps; `special` angles make cos or sin
    of a rotation zero, tiny or equal."""
    rng = np.random.default_rng(seed)
    insts = []
    for _ in range(depth):
        k = rng.integers(9)
        a, b = rng.permutation(n)[:2].tolist()
        if k < 4:
            th = float(rng.uniform(0, 2 * math.pi))
            if special:
                th = float(rng.choice([0.0, math.pi, math.pi / 2, -math.pi / 2, 2 * math.pi, 1e-9, math.pi - 1e-9,
                                       math.pi + 1e-17, 3.0]))
            insts.append(g("u3", a, th, float(rng.uniform(0, 6)), float(rng.uniform(0, 6))))
        elif k == 4:
            insts.append(g("x", a))
        elif k == 5:
            insts.append(g("cx", a, b))
        elif k == 6:
            insts.append(g("cx", a, b))
        elif k == 7:
            insts.append([g("cp", a, b, 0.7), g("rzz", a, b, 1.1), g("cz", a, b), g("swap", a, b)][rng.integers(4)])
        else:
            insts.append([g("h", a), g("ry", a, 0.4), g("sx", a), g("t", a), g("y", a)][rng.integers(5)])
    return JsonCircuit(n, insts + [g("u3", 0, 0.3, 0.2, 0.1)])


CASES = [(11, 120, 1, False, 0), (12, 200, 2, False, 0), (13, 200, 3, True, 0), (14, 160, 4, True, 5),
         (16, 260, 5, False, 40)]


def case(n, depth, seed, special):
    prog = encode(decode_circuit_json(circuit(n, depth, seed, special).model_dump_json()))
    rng = np.random.default_rng(seed)
    v = rng.normal(size=1 << n) + 1j * rng.normal(size=1 << n)
    v /= np.linalg.norm(v)
    want, _, rc, _ = _oracle.run(prog, 0, v)
    assert rc == 0
    return prog, v, want


@pytest.mark.parametrize("n,depth,seed,special,cost", CASES)
def test_planned(engine_lib, n, depth, seed, special, cost):
    prog, v, want = case(n, depth, seed, special)
    got, perm, _ = emulate(prog, v, nat.RunOpts(0, nat.EXEC_FUSED, 0, 0, 0, cost))
    assert np.max(np.abs(canonical(got, perm) - want)) < ATOL


@pytest.mark.gpu
@pytest.mark.parametrize("n,depth,seed,special,cost", CASES + [(20, 300, 6, False, 0), (21, 300, 7, True, 0)])
def test_kernel(gpu, n, depth, seed, special, cost):
    prog, v, want = case(n, depth, seed, special)
    st = nat.State(n, 0)
    st.upload(v)
    run_program(st, prog, 0, nat.SEM_SIMULATE, nat.EXEC_FUSED, 0, False, False, cost)
    assert np.max(np.abs(st.download() - want)) < ATOL
    # from a basis state (generated and skipped tiles)
    st.reset()
    run_program(st, prog, 0, nat.SEM_SIMULATE, nat.EXEC_FUSED, 0, False, False, cost)
    assert np.max(np.abs(st.download() - _oracle.run(prog, 0)[0])) < ATOL


@pytest.mark.gpu
@pytest.mark.parametrize("n", [11, 14])
def test_norm_does_not_drift(gpu, n):
    # 16 n gates that each round the 2-norm by about eps: independent, they add to
    # 4 sqrt(n) eps (root mean square over circuits); factors a little off modulus one
    # that pile up would be several times that
    drift = []
    for seed in range(10):
        rng = np.random.default_rng(seed)
        insts = []
        for layer in range(8):
            insts += [g("rx" if layer % 2 else "ry", q, float(rng.uniform(-math.pi, math.pi))) for q in range(n)]
            insts += [g("rzz", q, (q + 1) % n, float(rng.uniform(-math.pi, math.pi))) for q in range(n)]
        prog = encode(decode_circuit_json(JsonCircuit(n, insts).model_dump_json()))
        st = nat.State(n, 0)
        run_program(st, prog, 0, nat.SEM_SIMULATE, nat.EXEC_FUSED, 0, False, False, 0)
        v = np.asarray(st.download()).astype(np.clongdouble)
        drift.append(float(np.vdot(v, v).real - 1))
    assert np.sqrt(np.mean(np.square(drift))) < 4 * math.sqrt(n) * np.finfo(float).eps
