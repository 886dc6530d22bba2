"""Small states: whole programs and sampling in one launch each, against the oracle."""
import numpy as np
import pytest

import _oracle
from _circuits import JsonCircuit, cond, g, gate, random_gate
from dqsim_bosonic_b200 import _native as nat
from dqsim_bosonic_b200.circuit import decode_circuit_json, encode
from dqsim_bosonic_b200.statevector import SimulationResult, run_program

pytestmark = pytest.mark.gpu


def prog_of(c):
    return encode(decode_circuit_json(c.model_dump_json()))


def mixed(n, depth, seed):
    rng = np.random.default_rng(seed)
    insts = []
    for k in range(depth):
        r = rng.random()
        q = int(rng.integers(n))
        if r < 0.12:
            insts.append(g("measure", q, int(rng.integers(6))))
        elif r < 0.18:
            insts.append(g("reset", q))
        elif r < 0.3:
            insts.append(cond(int(rng.integers(5)), 2, int(rng.integers(4)), random_gate(rng, n)))
        elif r < 0.34 and n > 1:
            insts.append(g("swap", q, (q + 1) % n))
        else:
            insts.append(random_gate(rng, n))
    return JsonCircuit(n, insts, ncbits=6)


# one amplitude per thread and many, the last size that takes the path and the first that
# does not, programs of one instruction
@pytest.mark.parametrize("mode", [nat.EXEC_PER_GATE, nat.EXEC_FUSED])
@pytest.mark.parametrize("n,depth", [(1, 1), (1, 40), (2, 60), (4, 90), (7, 120), (9, 7), (9, 150), (10, 150), (12, 120),
                                     (13, 60)])
def test_program_matches_oracle(gpu, n, depth, mode):
    prog = prog_of(mixed(n, depth, 50 + n))
    rng = np.random.default_rng(n)
    v = rng.normal(size=1 << n) + 1j * rng.normal(size=1 << n)
    v /= np.linalg.norm(v)
    for init in (None, v):
        want, wcb, rc, _ = _oracle.run(prog, 5, init)
        assert rc == 0
        st = nat.State(n, 0)
        if init is not None:
            st.upload(init)
        cb, prof = run_program(st, prog, 5, nat.SEM_SIMULATE, mode)
        assert prof.boundary_draws == 0 and cb.tolist() == wcb.tolist()
        assert np.max(np.abs(st.download() - want)) < 1e-12
        executed = prof.apply_one_qubit_calls + prof.apply_n_qubit_calls + prof.measure_qubit_calls
        assert executed > 0 or depth == 1 or mode == nat.EXEC_FUSED


def test_unsupported_gate_stops_the_program(gpu):
    insts = [g("x", 0), g("h", 1), g("measure", 0, 0), gate("nope", [0]), g("x", 1)]
    prog = prog_of(JsonCircuit(3, insts, ncbits=1))
    st = nat.State(3, 0)
    with pytest.raises(NotImplementedError, match="nope"):
        run_program(st, prog, 1, nat.SEM_SIMULATE, nat.EXEC_PER_GATE)
    want = np.zeros(8, dtype=complex)
    want[1] = want[3] = 1 / np.sqrt(2)  # what came before it was applied
    assert np.max(np.abs(st.download() - want)) < 1e-15


# one block's scan of 2048 entries, its neighbours, sums of several terms, no shots
@pytest.mark.parametrize("n,k,shots", [(1, 1, 10), (1, 0, 5), (5, 5, 1000), (11, 11, 5000), (12, 12, 300), (11, 5, 257),
                                       (8, 3, 0), (6, 6, 16385)])
def test_samples_match_oracle(gpu, n, k, shots):
    rng = np.random.default_rng(n * 7 + k)
    v = rng.normal(size=1 << n) + 1j * rng.normal(size=1 << n)
    v[rng.random(1 << n) < 0.3] = 0
    v[0] += 1
    v /= np.linalg.norm(v)
    st = nat.State(n, 0)
    st.upload(v)
    qs = rng.permutation(n)[:k].tolist()
    res = SimulationResult(st, n, {}, None)
    got = res.sample_indices(shots, qs, seed=3)
    assert res.last_boundary_draws == 0
    assert got.tolist() == _oracle.sample(v, qs, 3, shots).tolist()


# the collapse divides by multiplying and correcting: every result equals the division, for
# zeros, numbers near the ends of the range, and norms that are not representable sums
@pytest.mark.parametrize("n", [1, 5, 14])
@pytest.mark.parametrize("p1", [0.5, 1 / 3, 1e-14, 0.9999999, 1.0])
@pytest.mark.parametrize("outcome", [0, 1])
def test_collapse_is_a_division(gpu, n, p1, outcome):
    rng = np.random.default_rng(n)
    v = (rng.normal(size=1 << n) + 1j * rng.normal(size=1 << n)) * 2.0 ** rng.integers(-60, 3, size=1 << n)
    v.real[rng.random(1 << n) < 0.1] = -0.0
    v[rng.random(1 << n) < 0.05] = 1e-308 + 5e-324j
    v[rng.random(1 << n) < 0.05] = 1e-251 - 1e280j
    st = nat.State(n, 0)
    st.upload(v)
    q = n // 2
    nat.check(nat.lib().dq_collapse(st.handle, q, outcome, p1))
    norm = max(np.sqrt(p1 if outcome else max(1.0 - p1, 0.0)), 1e-15)
    keep = ((np.arange(1 << n) >> q) & 1) == outcome
    want = np.where(keep, v.real / norm, 0.0) + 1j * np.where(keep, v.imag / norm, 0.0)
    got = st.download()
    assert got.tobytes() == want.tobytes() or (
        np.array_equal(got.real, want.real) and np.array_equal(got.imag, want.imag))


# norms of unnormalised states: infinite and undefined ones, and ones so large that quotients
# are denormal
@pytest.mark.parametrize("n", [1, 5, 14])
@pytest.mark.parametrize("p1", [np.inf, np.nan, 1e302, 1e140, 1e100])
def test_collapse_by_extreme_norms(gpu, n, p1):
    rng = np.random.default_rng(n)
    v = (rng.normal(size=1 << n) + 1j * rng.normal(size=1 << n)) * 2.0 ** rng.integers(-820, 500, size=1 << n)
    v.real[rng.random(1 << n) < 0.1] = -0.0
    st = nat.State(n, 0)
    st.upload(v)
    q = n // 2
    nat.check(nat.lib().dq_collapse(st.handle, q, 1, p1))
    norm = max(np.sqrt(p1), 1e-15) if p1 == p1 else p1
    keep = ((np.arange(1 << n) >> q) & 1) == 1
    got = st.download()
    assert np.array_equal(got.real, np.where(keep, v.real / norm, 0.0), equal_nan=True)
    assert np.array_equal(got.imag, np.where(keep, v.imag / norm, 0.0), equal_nan=True)


@pytest.mark.parametrize("n", [3, 12, 14])
@pytest.mark.parametrize("mode", [nat.EXEC_PER_GATE, nat.EXEC_FUSED])
def test_measurement_of_an_infinite_norm(gpu, n, mode):
    # p1 overflows: outcome 1, and every finite amplitude over infinity is zero
    prog = prog_of(JsonCircuit(n, [g("measure", 0, 0)], ncbits=1))
    v = np.full(1 << n, 1e160 + 1e-3j)
    want, wcb, rc, _ = _oracle.run(prog, 3, v)
    assert rc == 0
    st = nat.State(n, 0)
    st.upload(v)
    cb, _ = run_program(st, prog, 3, nat.SEM_SIMULATE, mode)
    assert cb.tolist() == wcb.tolist() == [1]
    assert np.array_equal(st.download(), want)


@pytest.mark.parametrize("mode", [nat.EXEC_PER_GATE, nat.EXEC_FUSED])
@pytest.mark.parametrize("n", [3, 10])
def test_program_without_memory_for_its_tables(gpu, alloc_limit, n, mode):
    # 3000 instructions take more than 64 KiB of tables; the measurements come back one by one
    prog = prog_of(mixed(n, 3000, 3))
    want, wcb, rc, _ = _oracle.run(prog, 5)
    assert rc == 0
    st = nat.State(n, 0)
    with alloc_limit(1 << 16):
        cb, prof = run_program(st, prog, 5, nat.SEM_SIMULATE, mode)
        got = st.download()
    assert prof.boundary_draws == 0 and cb.tolist() == wcb.tolist()
    assert np.max(np.abs(got - want)) < 1e-12


# one launch where measurements are many for the gates, sweeps or grouped launches where they
# are few, with the same results either way
@pytest.mark.parametrize("mode,gates,meas,one_launch", [
    (nat.EXEC_FUSED, 400, 1, False), (nat.EXEC_FUSED, 30, 6, True), (nat.EXEC_PER_GATE, 400, 1, True)])
@pytest.mark.parametrize("n", [10, 12])
def test_deep_programs_run_in_sweeps(gpu, mode, gates, meas, one_launch, n):
    rng = np.random.default_rng(n)
    insts = []
    for k in range(gates):
        if k % (gates // meas) == gates // meas - 1:
            insts.append(g("measure", int(rng.integers(n)), 0))
        a, b = rng.permutation(n)[:2].tolist()
        insts.append([g("ry", a, 0.3), g("rz", a, 0.7), g("cp", a, b, 0.4), g("u3", a, 0.1, 0.2, 0.3)][k % 4])
    prog = prog_of(JsonCircuit(n, insts, ncbits=1))
    want, wcb, rc, _ = _oracle.run(prog, 9)
    assert rc == 0
    st = nat.State(n, 0)
    cb, prof = run_program(st, prog, 9, nat.SEM_SIMULATE, mode)
    assert prof.boundary_draws == 0 and cb.tolist() == wcb.tolist()
    assert np.max(np.abs(st.download() - want)) < 1e-12
    assert (prof.kernel_launches == 1 and prof.sweeps == 0) == one_launch


# both sides of the line between one block and separate launches: the same indices
@pytest.mark.parametrize("n,k,shots", [(11, 11, 4608), (11, 11, 4609), (13, 9, 3072), (13, 9, 3073), (14, 10, 1024),
                                       (14, 11, 1024), (17, 11, 100)])
def test_samples_beside_the_line(gpu, n, k, shots):
    rng = np.random.default_rng(n * k)
    v = rng.normal(size=1 << n) + 1j * rng.normal(size=1 << n)
    v /= np.linalg.norm(v)
    st = nat.State(n, 0)
    st.upload(v)
    qs = rng.permutation(n)[:k].tolist()
    res = SimulationResult(st, n, {}, None)
    got = res.sample_indices(shots, qs, seed=3)
    assert res.last_boundary_draws == 0
    assert got.tolist() == _oracle.sample(v, qs, 3, shots).tolist()
