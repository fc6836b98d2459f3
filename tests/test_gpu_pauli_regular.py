"""Grouped Pauli terms where the group's shape changes its path: terms whose
pairs differ in the highest tile bit (their sums in registers, eight at most),
dependent and repeated X masks, Z strings, X masks in the low bits only, both
kinds of pair sum, tiles of two and four own amplitudes per thread.  Values
against the oracle's sequential sum (the parity tests' 1e-12)."""
import numpy as np
import pytest

from menos_b200 import DeviceState
from menos_b200._lib import C64
from test_oracle_pin import rand_state

pytestmark = pytest.mark.gpu


def term_lists(n, rng):
    def draw(k, x=None):
        return [(int(rng.integers(0, 1 << n)) if x is None else x(), int(rng.integers(0, 1 << n))) for _ in range(k)]
    basis = [int(rng.integers(1, 1 << n)) for _ in range(3)]
    span = lambda: basis[0] * int(rng.integers(2)) ^ basis[1] * int(rng.integers(2)) ^ basis[2] * int(rng.integers(2))
    top = 1 << (n - 1)
    yield draw(1)
    yield draw(8)
    yield draw(64)
    yield draw(16, span)                                        # 16 terms in a span of three
    yield draw(12, lambda: top) + draw(4, lambda: 0)            # one X mask, more terms than registers hold
    yield draw(10, lambda: int(rng.integers(0, 8)))             # X in the low bits
    yield [(0, 0), (top, top), (top, 0), ((1 << n) - 1, (1 << n) - 1)] + draw(9)


@pytest.mark.parametrize("n", [9, 10, 11, 12, 14, 17])
def test_terms_against_the_sequential_sum(ctx, oracle, n):
    rng = np.random.default_rng(n)
    s = rand_state(n, rng)
    st, lo = DeviceState(ctx, n), DeviceState(ctx, n, C64)
    st.copy_in(s)
    lo.copy_in(s.astype(np.complex64))
    s64 = s.astype(np.complex64).astype(np.complex128)
    for terms in term_lists(n, rng):
        want = np.array([oracle.expectation(s, x, z) for x, z in terms])
        assert np.max(np.abs(st.expectation(terms) - want)) < 1e-12
        want = np.array([oracle.expectation(s64, x, z) for x, z in terms])
        assert np.max(np.abs(lo.expectation(terms) - want)) < 1e-12
