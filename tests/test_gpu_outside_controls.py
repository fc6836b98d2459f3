"""CX controls outside a pass's tile: seven of them, all that a phase record
holds, and the eighth, which the pass takes into the tile or leaves to the
next."""
import numpy as np
import pytest

import pyoracle
from menos_b200 import Circuit, DeviceState
from test_oracle_pin import bits_equal

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("controls", [6, 7, 8, 9])
@pytest.mark.parametrize("room", [0, 2], ids=["full tile", "two qubits free"])
def test_outside_controls(ctx, oracle, controls, room):
    tile, n = 8, 18
    inside = tile - room
    a, b = Circuit(n), pyoracle.Circuit(n)
    for c in (a, b):
        for q in range(n - 1, -1, -1):  # the tile's qubits last, with their CX behind them
            c.gate("ry", [q], [0.3 + 0.17 * q])
        for i in range(controls):
            c.gate("cx", [n - 1 - i, i % inside])
        for q in range(inside):
            c.gate("u", [q], [0.2 * q, 0.5, 0.7])
        for i in range(controls):  # and undone in part, so that the map's columns meet again
            c.gate("cx", [n - 1 - i, (i + i % 2) % inside])
        c.gate("x", [1])
    st = DeviceState(ctx, n)
    st.init(0.0)
    st.apply_program(a, fuse_gates=False, tile_qubits=tile)
    assert bits_equal(st.copy_out(), oracle.run(b, fuse_gates=False))
