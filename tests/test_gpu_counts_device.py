"""Sampling from the seed to the counts on the device: the generator and the
sort at the sizes where their kernels change shape (a twist is 312 words, runs
are counted in tiles of 1024; where one CTA's sort ends:
test_gpu_counts_branches.py), sums that cross binades inside one chunk, and the short walk over a
density matrix's diagonal.  Counts are whole numbers: identical, always."""
import numpy as np
import pytest

from menos_b200 import Circuit, DensityMatrix, DeviceState
from menos_b200._lib import MB2Error
from test_gpu_parity import dev_state
from test_oracle_pin import rand_state

pytestmark = pytest.mark.gpu


def identity(n):
    return [(q, q) for q in range(n)]


@pytest.mark.parametrize("n,shots", [(1, 1), (4, 2), (5, 311), (11, 312), (12, 313), (12, 1023), (13, 1025),
                                     (12, 4095), (9, 4096), (14, 4097), (16, 8193), (13, 65537), (18, 1 << 20)])
def test_counts_at_the_edges_of_the_kernels(ctx, oracle, n, shots):
    s = rand_state(n, np.random.default_rng(shots + n))
    st = dev_state(ctx, s)
    for seed in (0, 2 ** 64 - 1, 123456789):
        assert st.sample(shots, seed, identity(n)) == oracle.sample(s, shots, seed, identity(n))


@pytest.mark.parametrize("kind", ["growing", "leading zeros", "one run", "tiny", "spikes"])
def test_binade_crossings_inside_a_chunk(ctx, oracle, kind):
    n = 14
    rng = np.random.default_rng(5)
    i = np.arange(1 << n)
    mag = {"growing": np.exp(i * (60.0 / (1 << n)) - 60.0), "leading zeros": np.where(i < 9001, 0.0, rng.uniform(0, 1, i.size)),
           "one run": np.where((i >> 4) == 300, rng.uniform(0, 1, i.size), 0.0),
           "tiny": np.where(i < 6000, 1e-150 * rng.uniform(0, 1, i.size), rng.uniform(0, 1, i.size)),
           "spikes": np.where(i % 777 == 5, 1.0, 1e-9)}[kind]
    s = (mag / np.linalg.norm(mag)).astype(np.complex128)
    st = dev_state(ctx, s)
    p = s.real * s.real + s.imag * s.imag
    assert st.norm_exact() == np.add.accumulate(p)[-1]
    assert st.sample(20000, 3, identity(n)) == oracle.sample(s, 20000, 3, identity(n))


def test_a_state_that_is_no_state(ctx, oracle):
    # A NaN amplitude: the sums before it are exact, and no later one exceeds a uniform.
    n = 13
    s = rand_state(n, np.random.default_rng(8))
    s[5000] = np.nan
    st = dev_state(ctx, s)
    assert st.sample(3000, 2, identity(n)) == oracle.sample(s, 3000, 2, identity(n))


@pytest.mark.parametrize("targets", [[(3, 0), (1, 1)], [(q, 11 - q) for q in range(12)], [(0, 40), (11, 2)], []])
def test_targets_that_are_not_the_basis_states(ctx, oracle, targets):
    s = rand_state(12, np.random.default_rng(6))
    st = dev_state(ctx, s)
    assert st.sample(30000, 4, targets) == oracle.sample(s, 30000, 4, targets)


def test_capacity_is_refused_before_anything_is_written(ctx):
    import ctypes as C
    from menos_b200._lib import lib
    st = dev_state(ctx, rand_state(12, np.random.default_rng(9)))
    t = np.asarray(identity(12), np.uint32).ravel()
    out, cnt, cap = np.full(8, 7, np.uint64), np.full(8, 7, np.uint64), C.c_uint64(8)
    rc = lib().mb2_sample(st.h, 1000, 1, t.ctypes.data, 12, out.ctypes.data, cnt.ctypes.data, C.byref(cap))
    assert rc == 1 and np.all(out == 7) and np.all(cnt == 7)
    with pytest.raises(MB2Error):
        st.sample(10, 1, [(12, 0)])


@pytest.mark.parametrize("n", [1, 5, 10, 11, 12])
def test_density_walk(ctx, oracle, n):
    rng = np.random.default_rng(n)
    c = Circuit(n)
    for q in range(n):
        c.gate("ry", [q], [float(rng.uniform(0, 3))])
        c.channel([q], [np.sqrt(0.9) * np.eye(2), np.sqrt(0.1) * np.array([[0, 1], [1, 0]])])
    rho = DensityMatrix(ctx, n)
    rho.init()
    rho.apply(c)
    diag = np.real(np.diagonal(rho.matrix())).copy()
    # Entries below zero make the running sum fall: the walk takes the first index that exceeds the uniform.
    if n >= 5:
        diag[3::7] = -1e-3 * diag[3::7]
        full = rho.state.copy_out()
        full[np.arange(1 << n) * ((1 << n) + 1)] = diag
        rho.state.copy_in(full)
    sums = np.add.accumulate(diag)
    for shots, seed in [(1, 3), (700, 4), (5000, 5)]:
        u = np.sort(oracle.uniforms(seed, shots))
        first = np.searchsorted(np.maximum.accumulate(sums), u, side="right")
        first = np.minimum(first, (1 << n) - 1)
        want = dict(zip(*(v.tolist() for v in np.unique(first, return_counts=True))))
        assert rho.sample(shots, seed, identity(n)).to_dict() == want
