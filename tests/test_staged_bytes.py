"""What a pass stages in shared memory stays within the limit that the kernels'
tile buffers leave, at every tile width and in both precisions, whatever the
blocks make of their phases: a plan above it is refused at its launch.

Long runs of exact permutations (X, CX), diagonals (T) and blocks of three
qubits (CCX, applied from shared memory) open the most phase records per
block: one to bring moved amplitudes back before a wide block, one for the
diagonal behind it."""
import ctypes as C
import random

import numpy as np
import pytest

from menos_b200 import DeviceState, _lib
from menos_b200.circuit import Circuit, to_mb2_ops
from menos_b200.engine import C64, C128
from test_host import as_oracle_circuit
from test_oracle_pin import bits_equal


def staged(circ, tile, precision):
    arr, keep = to_mb2_ops(circ)
    opts = _lib.SweepOptions(0, 0, tile, 0, 1)  # unfused; the FP32 SIMT passes
    most, limit = C.c_uint64(), C.c_uint64()
    rc = _lib.lib().mb2_debug_staged_bytes(arr, len(circ.ops), C.byref(opts), circ.num_qubits, precision,
                                           C.byref(most), C.byref(limit))
    assert rc == 0
    del keep
    return most.value, limit.value


def x_t_ccx_t(n):
    c = Circuit(n)
    for _ in range(300):
        c.gate("x", [0]).gate("t", [0]).gate("ccx", [0, 1, 2]).gate("t", [0])
    return c


def cx_t_ccx_u(n):
    # Controls outside an 11-qubit tile, and dense one-qubit blocks between.
    c = Circuit(n)
    for i in range(200):
        c.gate("cx", [n - 1 - i % 5, 3]).gate("t", [3]).gate("ccx", [0, 1, 2]).gate("t", [0])
        c.gate("u", [i % 7], [0.1 * i, 0.2, 0.3])
    return c


def diagonals(n):
    # Sign runs, phases and two-qubit diagonals with moves and wide blocks between.
    c = Circuit(n)
    for i in range(400):
        c.gate(("z", "t", "s")[i % 3], [i % 9]).gate("cp", [i % 9, (i + 4) % 9], [0.1 * i])
        if i % 3 == 0:
            c.gate("swap", [i % 9, (i + 1) % 9])
        if i % 7 == 0:
            c.gate("ccx", [0, 4, 8])
    return c


def any_order(n):
    rng = random.Random(7)
    c = Circuit(n)
    for _ in range(2500):
        a, b, d = rng.sample(range(n), 3)
        kind = rng.randrange(8)
        if kind == 0:
            c.gate("ccx", [a, b, d])
        elif kind == 1:
            c.gate("swap", [a, b]).gate("ccx", [a, b, d])
        elif kind == 2:
            c.gate("u", [a], [rng.random(), 0.2, 0.3])
        elif kind == 3:
            c.gate("t", [a])
        elif kind == 4:
            c.gate("x", [a])
        elif kind == 5:
            c.gate("cp", [a, b], [rng.random()])
        elif kind == 6:
            c.gate("y", [a])
        else:
            c.gate("cx", [a, b])
    return c


@pytest.mark.parametrize("family", [x_t_ccx_t, cx_t_ccx_u, diagonals, any_order], ids=lambda f: f.__name__)
@pytest.mark.parametrize("precision,widths", [(C128, range(4, 13)), (C64, range(4, 14))], ids=["c128", "c64"])
def test_staged_within_the_limit(family, precision, widths):
    circ = family(16)
    for tile in widths:
        most, limit = staged(circ, tile, precision)
        assert 0 < most <= limit, tile


@pytest.mark.gpu
@pytest.mark.parametrize("precision,tile", [(C128, 11), (C128, 12), (C64, 12), (C64, 13)])
def test_the_longest_passes_run(ctx, oracle, precision, tile):
    n = 13
    circ = Circuit(n)
    for q in range(n):
        circ.gate("u", [q], [0.4 + q, 0.3, 0.2 * q])
    circ.ops += x_t_ccx_t(n).ops
    st = DeviceState(ctx, n, precision)
    st.init(0.0)
    st.apply_program(circ, fuse_gates=False, tile_qubits=tile, c64_kernel="simt")
    expect = oracle.run(as_oracle_circuit(circ), fuse_gates=False)
    got = st.copy_out()
    if precision == C128:
        assert bits_equal(got, expect)
    else:  # 613 blocks that round (u and t), each a sum of at most two complex products rounded to 2^-24
        assert np.max(np.abs(got - expect)) < 613 * 4 * 2.0 ** -24
