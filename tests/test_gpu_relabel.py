"""Materialising a qubit relabeling (swap gates run as relabelings) against numpy.

The program holds swaps only, so the state is the input with its index bits
permuted: the comparison is exact.
"""
import numpy as np
import pytest

from _circuits import JsonCircuit, g
from dqsim_bosonic_b200 import _native as nat
from dqsim_bosonic_b200.circuit import decode_circuit_json, encode
from dqsim_bosonic_b200.statevector import run_program

pytestmark = pytest.mark.gpu


# below, at and above the 8 local positions of a tile pair, one tile pair per warp
# and several, with positions that pair up inside, across and outside the tile
@pytest.mark.parametrize("n", [2, 5, 7, 8, 9, 10, 11, 13, 16, 21])
@pytest.mark.parametrize("case", ["reverse", "one", "random", "cycle"])
def test_relabelled_state(gpu, n, case):
    rng = np.random.default_rng(n)
    if case == "reverse":
        pairs = [(q, n - 1 - q) for q in range(n // 2)]
    elif case == "one":
        pairs = [(0, n - 1)]
    elif case == "cycle":
        pairs = [(q, q + 1) for q in range(n - 1)]
    else:
        pairs = [tuple(rng.choice(n, 2, replace=False).tolist()) for _ in range(2 * n)]
    v = rng.normal(size=1 << n) + 1j * rng.normal(size=1 << n)
    want = v.reshape((2,) * n)  # axis n - 1 - q is qubit q
    for a, b in pairs:
        want = np.swapaxes(want, n - 1 - a, n - 1 - b)
    prog = encode(decode_circuit_json(JsonCircuit(n, [g("swap", a, b) for a, b in pairs]).model_dump_json()))
    st = nat.State(n, 0)
    st.upload(v)
    run_program(st, prog, 0, nat.SEM_SIMULATE, nat.EXEC_FUSED)
    assert np.array_equal(st.download(), want.reshape(-1))
