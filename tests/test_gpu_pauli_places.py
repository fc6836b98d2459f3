"""Where a grouped Pauli term's sum is kept: in a register (regular pairs,
then Z strings, eight in all), in shared memory, one for each thread or -- where
that would leave an SM room for one CTA only -- for each pair of threads; with
three tile buffers or two.  Values against the oracle's sequential sum (the
parity tests' 1e-12), a state by itself and in a batch."""
import numpy as np
import pytest

from menos_b200 import DeviceState, workloads
from menos_b200._lib import C64, C128
from menos_b200.engine import sweep_batch
from test_oracle_pin import rand_state

pytestmark = pytest.mark.gpu


def groups(n, rng):
    z = lambda: int(rng.integers(0, 1 << n))
    top = 1 << (n - 1)
    yield "Z strings", [(0, z()) for _ in range(16)]
    yield "one Z string", [(0, z())] + [(top, z())]
    yield "pairs, then Z strings", [(top, z()) for _ in range(5)] + [(0, z()) for _ in range(9)]
    yield "more pairs than registers", [(0, z())] + [(top, z()) for _ in range(11)] + [(0, z())]
    yield "no pair in registers", [(int(x), z()) for x in rng.integers(1, 1 << 8, 16)]
    yield "twelve of them", [(int(x), z()) for x in rng.integers(1, 1 << 8, 12)] + [(0, z()) for _ in range(4)]
    yield "every kind", [(x, z()) for x in (0, 1, top, top | 1, 0, 3, top | 5, 2, 0, top, 7, top, 0, 1, top | 3, 0)]
    yield "chain", [p for i in range(n - 1) for p in ((3 << i, 0), (3 << i, 3 << i), (0, 3 << i))]


@pytest.mark.parametrize("n", [10, 11, 12, 15])
def test_every_place(ctx, oracle, n):
    rng = np.random.default_rng(40 + n)
    s = rand_state(n, rng)
    for precision, given in ((C128, s), (C64, s.astype(np.complex64))):
        st = DeviceState(ctx, n, precision)
        st.copy_in(given)
        exact = given.astype(np.complex128)
        for name, terms in groups(n, rng):
            want = np.array([oracle.expectation(exact, x, z) for x, z in terms])
            assert np.max(np.abs(st.expectation(terms) - want)) < 1e-12, name


@pytest.mark.parametrize("n", [11, 13])
def test_every_place_in_a_batch(ctx, n):
    rng = np.random.default_rng(60 + n)
    circ = workloads.hea(n, 2, 5)
    rows = rng.uniform(-3, 3, size=(7, sum(len(op[2]) for op in circ.ops)))
    for name, terms in groups(n, rng):
        coefs = rng.normal(size=len(terms))
        values, states, _ = sweep_batch(ctx, circ, rows, terms, coefs, want_states=True)
        st = DeviceState(ctx, n)
        for value, state in zip(values, states):
            st.copy_in(state)
            # The same sums, added in another order: at most 48 terms of coefficients around one.
            assert abs(value - np.sum(coefs * st.expectation(terms).real)) < 1e-12, name
