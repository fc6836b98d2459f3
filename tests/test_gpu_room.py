"""A device without room for all that a call would like: it takes less and
gives the same results.  mb2_debug_room stands in for such a device."""
import contextlib

import numpy as np
import pytest

from menos_b200._lib import MB2Error, lib
from menos_b200.engine import trajectories
from test_dm import noisy_circuit

pytestmark = pytest.mark.gpu


@contextlib.contextmanager
def room(ctx, size):
    assert lib().mb2_debug_room(ctx.h, size) == 0
    try:
        yield
    finally:
        lib().mb2_debug_room(ctx.h, 0)


def least_room(ctx, d, paulis):
    """About the least room in which two trajectories run."""
    size = 16 << 10
    while True:
        with room(ctx, size):
            try:
                trajectories(ctx, d, 2, 9, paulis)
                return size
            except MB2Error as e:
                assert e.code == 2  # the resource error
        size += size // 8


# A batch of 64 in a room for two: refused for its states (1 MiB at 10
# qubits), or beside states that fit (16 KiB at 4) for its draws, values and
# scratch.
@pytest.mark.parametrize("n", [10, 4])
def test_a_batch_that_is_refused_runs_one_by_one(ctx, n):
    _, d = noisy_circuit(n, 60, np.random.default_rng(n), widest=2)
    paulis = [(3, 0), (0, 5), (1, 2)]
    targets = [(q, q) for q in range(n)]
    whole = trajectories(ctx, d, 70, 9, paulis, None, 70, targets)
    with room(ctx, least_room(ctx, d, paulis)):
        got = trajectories(ctx, d, 70, 9, paulis, None, 70, targets)
    assert np.array_equal(got["terms"], whole["terms"])
    assert got["standard_error"] == whole["standard_error"]
    assert got["counts"] == whole["counts"]
