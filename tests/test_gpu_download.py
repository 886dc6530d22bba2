"""Copies of device results into host arrays (staged through pinned memory)."""
import numpy as np
import pytest

from _circuits import brickwork_u3_cx
from dqsim_bosonic_b200 import _native as nat
from dqsim_bosonic_b200.batch import run_batch
from dqsim_bosonic_b200.circuit import decode_circuit_json, encode

pytestmark = pytest.mark.gpu


# below one staging chunk (2^16 amplitudes), one, several, and more than the staging ring holds
@pytest.mark.parametrize("n", [0, 1, 9, 16, 17, 20, 22])
def test_download_returns_what_was_uploaded(gpu, n):
    rng = np.random.default_rng(n)
    v = rng.normal(size=1 << n) + 1j * rng.normal(size=1 << n)
    st = nat.State(n, 0)
    st.upload(v)
    assert np.array_equal(st.download(), v)


@pytest.mark.parametrize("want", [True, {0}, {1, 4}, {2, 3, 5}, set()])
def test_batch_states_land_in_their_arrays(gpu, want):
    # shared-memory and HBM items, with pieces that share and that cross staging chunks
    progs = [encode(decode_circuit_json(brickwork_u3_cx(n, 3, k).model_dump_json()))
             for k, n in enumerate((10, 18, 16, 12, 17, 19))]
    _, all_states, _ = run_batch(progs, range(6), want_states=True)
    _, states, _ = run_batch(progs, range(6), want_states=want)
    for k, s in enumerate(states):
        if want is True or k in want:
            assert np.array_equal(s, all_states[k])
            assert abs(np.vdot(s, s).real - 1.0) < 1e-12
        else:
            assert s is None


# nothing, and less than the staging ring, for pinned memory
@pytest.mark.parametrize("limit", [1, 4 << 20])
def test_downloads_without_pinned_memory(gpu, alloc_limit, limit):
    rng = np.random.default_rng(1)
    v = rng.normal(size=1 << 21) + 1j * rng.normal(size=1 << 21)
    st = nat.State(21, 0)
    st.upload(v)
    with alloc_limit(limit):
        assert np.array_equal(st.download(), v)


def test_batch_states_without_pinned_memory(gpu, alloc_limit):
    # 17 states of 256 KiB: their device buffer is within the limit, five chunks are not
    progs = [encode(decode_circuit_json(brickwork_u3_cx(14, 2, k).model_dump_json())) for k in range(17)]
    _, want, _ = run_batch(progs, range(17), want_states=True)
    with alloc_limit(17 << 18):
        _, got, _ = run_batch(progs, range(17), want_states=True)
    for a, b in zip(got, want):
        assert np.array_equal(a, b)


def test_download_into_pinned_memory(gpu):
    import torch

    n = 21
    rng = np.random.default_rng(2)
    v = rng.normal(size=1 << n) + 1j * rng.normal(size=1 << n)
    st = nat.State(n, 0)
    st.upload(v)
    out = torch.empty(1 << n, dtype=torch.complex128, pin_memory=True)
    nat.check(nat.lib().dq_state_download(st.handle, out.data_ptr(), 1 << n))
    assert np.array_equal(out.numpy(), v)
