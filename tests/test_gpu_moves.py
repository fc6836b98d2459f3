"""Permutations taken by the tile's map instead of moving amplitudes: X, CX
(either way round, its control in the tile or outside it), SWAP, and blocks
that are one of them and a one-qubit gate, with wide blocks (which need the
amplitudes at their own index), diagonals and permutations of three qubits
between them.  Complex128 states are the oracle's to the bit at every tile
width; complex64 and batched states within their rounding."""
import numpy as np
import pytest

import pyoracle
from menos_b200 import Circuit, DeviceState
from menos_b200._lib import C64
from menos_b200.engine import sweep_batch
from test_oracle_pin import bits_equal

pytestmark = pytest.mark.gpu


def moving_circuit(n, gates, rng, wide=True):
    names = ["x", "cx", "cx", "cx", "swap", "y", "u", "rz", "ry", "h", "cz", "cp", "t"] + (["ccx", "unitary"] if n > 2 and wide else [])
    a, b = Circuit(n), pyoracle.Circuit(n)
    for _ in range(gates):
        name = names[rng.integers(len(names))]
        if name == "unitary":
            k = int(rng.integers(1, min(4, n) + 1))
            m = np.linalg.qr(rng.normal(size=(1 << k, 1 << k)) + 1j * rng.normal(size=(1 << k, 1 << k)))[0]
            q = [int(v) for v in rng.choice(n, size=k, replace=False)]
            for c in (a, b):
                c.unitary(q, m)
            continue
        k = {"cx": 2, "swap": 2, "cz": 2, "cp": 2, "ccx": 3}.get(name, 1)
        q = [int(v) for v in rng.choice(n, size=k, replace=False)]
        p = [float(v) for v in rng.uniform(-3, 3, size={"u": 3, "rz": 1, "ry": 1, "cp": 1}.get(name, 0))]
        for c in (a, b):
            c.gate(name, q, p)
    return a, b


@pytest.mark.parametrize("n,tile", [(4, 4), (5, 4), (7, 5), (9, 6), (11, 11), (12, 11), (12, 12), (13, 4), (13, 9), (14, 11),
                                    (14, 12), (16, 11)])
@pytest.mark.parametrize("fuse", [True, False])
def test_states_are_the_oracles_to_the_bit(ctx, oracle, n, tile, fuse):
    rng = np.random.default_rng(100 * n + tile)
    st = DeviceState(ctx, n)
    for gates in (12, 90):
        for wide in (True, False):
            a, b = moving_circuit(n, gates, rng, wide)
            st.init(0.0)
            st.apply_program(a, fuse_gates=fuse, tile_qubits=tile)
            assert bits_equal(st.copy_out(), oracle.run(b, fuse_gates=fuse)), (gates, wide)


@pytest.mark.parametrize("n", [12, 13, 16, 20])
@pytest.mark.parametrize("fuse", [True, False])
def test_ladders(ctx, oracle, n, fuse):
    # CX chains up, down and from a far control, between rotations, at the default tile.
    rng = np.random.default_rng(n)
    a, b = Circuit(n), pyoracle.Circuit(n)
    for layer in range(4):
        for q in range(n):
            t = float(rng.uniform(-3, 3))
            for c in (a, b):
                c.gate("ry", [q], [t])
                c.gate("rz", [q], [t / 3])
        pairs = [(q, q + 1) for q in range(n - 1)] if layer % 2 == 0 else [(q + 1, q) for q in range(n - 1)]
        for q, r in pairs + [(n - 1, 0), (0, n - 1), (n // 2, 1)]:
            for c in (a, b):
                c.gate("cx", [q, r])
        for c in (a, b):
            c.gate("x", [layer])
    st = DeviceState(ctx, n)
    st.init(0.0)
    st.apply_program(a, fuse_gates=fuse)
    assert bits_equal(st.copy_out(), oracle.run(b, fuse_gates=fuse))


@pytest.mark.parametrize("n", [5, 12, 13, 15])
def test_complex64(ctx, oracle, n):
    rng = np.random.default_rng(n)
    st = DeviceState(ctx, n, C64)
    for fuse in (True, False):
        for tile in sorted({min(n, t) for t in (5, 12, 13)}):
            a, b = moving_circuit(n, 60, rng)
            st.init(0.0)
            st.apply_program(a, fuse_gates=fuse, tile_qubits=tile, c64_kernel="simt")
            # 60 gates, each amplitude a sum of at most 16 products rounded to 2^-24.
            assert np.max(np.abs(st.copy_out() - oracle.run(b, fuse_gates=fuse))) < 60 * 16 * 2.0 ** -24


@pytest.mark.parametrize("n", [6, 12, 14])
def test_batched_bindings(ctx, oracle, n):
    rng = np.random.default_rng(n)
    a, b = moving_circuit(n, 60, rng, wide=False)
    slots = [len(op[2]) for op in a.ops]
    rows = rng.uniform(-3, 3, size=(5, sum(slots)))
    _, states, _ = sweep_batch(ctx, a, rows, [(0, 0)], [1.0], want_states=True)
    for row, got in zip(rows, states):
        k = 0
        for i, s in enumerate(slots):
            oc, qs, ps, m, *rest = b.ops[i]
            b.ops[i] = (oc, qs, tuple(float(v) for v in row[k:k + s]) if s else ps, m, *rest)
            k += s
        assert bits_equal(got, oracle.run(b, fuse_gates=False))


@pytest.mark.parametrize("n,tile", [(4, 4), (9, 6), (12, 12), (13, 11)])
def test_real_blocks_on_the_two_diagonals(ctx, oracle, n, tile):
    # Channel superoperators' shape on every ordered operand pair, zeros and signs among the entries.
    rng = np.random.default_rng(n)
    a, b = Circuit(n), pyoracle.Circuit(n)
    for q in range(n):
        for c in (a, b):
            c.gate("u", [q], [0.3 + q, 1.1, 0.2])
    for q in range(n):
        for r in range(n):
            if q == r:
                continue
            m = np.zeros((4, 4))
            v = rng.normal(size=(4, 2)) * 0.7
            for i in range(4):
                m[i, i], m[i, 3 - i] = v[i]
            if (q + r) % 3 == 0:
                m[1, 2] = m[2, 1] = 0.0
            for c in (a, b):
                c.unitary([q, r], m)
    st = DeviceState(ctx, n)
    st.init(0.0)
    st.apply_program(a, fuse_gates=False, tile_qubits=tile)
    assert bits_equal(st.copy_out(), oracle.run(b, fuse_gates=False))
