"""Sweeps whose passes are of both kinds, with the tile's map and without, on
either side of the state size from which they run a kernel each: the oracle's
bits on both."""
import numpy as np
import pytest

import pyoracle
from menos_b200 import Circuit, DeviceState
from test_oracle_pin import bits_equal

pytestmark = pytest.mark.gpu


def both_kinds(n, wide, rng):
    a, b = Circuit(n), pyoracle.Circuit(n)

    def layer():
        for q in range(n):
            p = [float(v) for v in rng.uniform(-3, 3, 3)]
            for c in (a, b):
                c.gate("u", [q], p)
        if wide:  # dense two-qubit blocks: the full kernels
            m = np.linalg.qr(rng.normal(size=(4, 4)) + 1j * rng.normal(size=(4, 4)))[0]
            for c in (a, b):
                c.unitary([0, n - 1], m)
                c.unitary([n // 2, 1], m)

    layer()
    for c in (a, b):
        for q in range(n - 1):
            c.gate("cx", [q, q + 1])
        c.gate("swap", [0, n - 2])
    layer()
    return a, b


@pytest.mark.parametrize("n,tile", [(9, 8), (14, 11), (14, 12), (22, 11), (23, 11), (23, 12)])
@pytest.mark.parametrize("wide", [False, True], ids=["lean", "full"])
def test_bits(ctx, oracle, n, tile, wide):
    a, b = both_kinds(n, wide, np.random.default_rng(n))
    st = DeviceState(ctx, n)
    st.init(0.0)
    st.apply_program(a, fuse_gates=False, tile_qubits=tile)
    assert bits_equal(st.copy_out(), oracle.run(b, fuse_gates=False))
