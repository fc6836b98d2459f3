"""Branches of the sampling path that ordinary states and calls do not take:
no room on the device for the draws' sort and the counts, an infinite
amplitude, a sort bucket beyond what shared memory holds; and the sizes where
its rules turn (3000 shots, up to which the host draws and counts; buckets of
at most 512 words on average, up to 1024 each sorted in shared memory)."""
import ctypes as C

import numpy as np
import pytest

from menos_b200 import Circuit, DensityMatrix
from menos_b200._lib import lib
from test_gpu_parity import dev_state
from test_gpu_room import room
from test_oracle_pin import rand_state

pytestmark = pytest.mark.gpu


def identity(n):
    return [(q, q) for q in range(n)]


@pytest.mark.parametrize("n", [3, 13])
@pytest.mark.parametrize("shots", [1, 2999, 3000, 3001, 4096, 4097])
def test_counts_where_the_device_takes_over(ctx, oracle, n, shots):
    s = rand_state(n, np.random.default_rng(shots))
    st = dev_state(ctx, s)
    for seed in (1, 2 ** 63):
        assert st.sample(shots, seed, identity(n)) == oracle.sample(s, shots, seed, identity(n))


@pytest.mark.parametrize("n", [12, 16])
@pytest.mark.parametrize("reverse", [False, True])
def test_counts_without_room_for_the_sort(ctx, oracle, n, reverse):
    # 16 bytes a shot fit the 4 MiB, the sort's 36 and more do not.
    shots, targets = 150000, [(q, n - 1 - q if reverse else q) for q in range(n)]
    s = rand_state(n, np.random.default_rng(n))
    st = dev_state(ctx, s)
    with room(ctx, 4 << 20):
        assert st.sample(shots, 8, targets) == oracle.sample(s, shots, 8, targets)


def test_density_counts_without_room_for_the_sort(ctx):
    n, shots = 6, 150000
    c = Circuit(n)
    for q in range(n):
        c.gate("ry", [q], [0.3 + 0.4 * q])
        c.channel([q], [np.sqrt(0.9) * np.eye(2), np.sqrt(0.1) * np.array([[0, 1], [1, 0]])])

    def rho():
        r = DensityMatrix(ctx, n)
        r.init()
        r.apply(c)
        return r

    whole = rho().sample(shots, 8, identity(n))
    with room(ctx, 4 << 20):
        assert rho().sample(shots, 8, identity(n)) == whole


@pytest.mark.parametrize("n,at", [(10, 77), (13, 0), (13, 5000), (14, 16383)])
def test_an_infinite_amplitude(ctx, oracle, n, at):
    # The sums before it are exact; every later uniform is below its sum.
    s = rand_state(n, np.random.default_rng(at))
    s[at] = np.inf
    st = dev_state(ctx, s)
    assert st.sample(3000, 2, identity(n)) == oracle.sample(s, 3000, 2, identity(n))


def mt_key(x):
    """A state word of mt19937_64 as a uniform's numerator (the published tempering, then 53 bits)."""
    x = x ^ ((x >> np.uint64(29)) & np.uint64(0x5555555555555555))
    x = x ^ ((x << np.uint64(17)) & np.uint64(0x71D67FFFEDA60000))
    x = x ^ ((x << np.uint64(37)) & np.uint64(0xFFF7EEE000000000))
    return (x ^ (x >> np.uint64(43))) >> np.uint64(11)


@pytest.mark.parametrize("count", [1, 2, 511, 512, 513, 1024, 1025, 70000])
def test_sort_sizes(ctx, count):
    words = np.random.default_rng(count).integers(0, 2 ** 64, count, np.uint64)
    out = np.zeros(count)
    assert lib().mb2_debug_sort_words(ctx.h, words.ctypes.data, count, out.ctypes.data) == 0
    assert np.array_equal(out, np.sort(mt_key(words).astype(np.float64) * 2.0 ** -53))


@pytest.mark.parametrize("crowd", [0, 1023, 1024, 1025, 3000, 4096])
def test_a_crowded_bucket(ctx, crowd):
    # 4096 words go to 8 buckets; `crowd` of them to the sixth.
    pool = np.random.default_rng(crowd).integers(0, 2 ** 64, 60000, np.uint64)
    sixth = (mt_key(pool) >> np.uint64(50)) == 5
    words = np.concatenate([pool[sixth][:crowd], pool[~sixth][:4096 - crowd]])
    words = np.random.default_rng(1).permutation(words)
    out = np.zeros(words.size)
    assert lib().mb2_debug_sort_words(ctx.h, words.ctypes.data, words.size, out.ctypes.data) == 0
    assert np.array_equal(out, np.sort(mt_key(words).astype(np.float64) * 2.0 ** -53))
