"""What describes a sweep's plan -- the schedule and the time estimate -- plans
as the sweep does: the complex64 tile width and form by state size, and what
its kernels do for each block."""
import ctypes as C

import numpy as np
import pytest

from menos_b200 import Circuit, _lib, workloads
from menos_b200.circuit import to_mb2_ops
from menos_b200.engine import C64, C128


@pytest.mark.parametrize("n", [20, 24, 25, 27, 28, 30])
@pytest.mark.parametrize("family", ["brick", "hea"])
@pytest.mark.parametrize("fuse", [0, 1])
@pytest.mark.parametrize("kernel", [0, 1])
def test_the_schedules_passes_are_the_plans(n, family, fuse, kernel):
    # (Few enough layers for the tensor cores that no pass is split for its phase matrices.)
    circ = getattr(workloads, family)(n, 6 if kernel == 1 else 3 if family == "brick" else 1, 5)
    arr, keep = to_mb2_ops(circ)
    lib, opts = _lib.lib(), _lib.SweepOptions(fuse, 0, 0, 0, kernel)
    stats = np.zeros(6, np.uint64)
    assert lib.mb2_debug_run_plan(arr, len(circ.ops), C.byref(opts), n, C64, None, stats.ctypes.data) == 0
    nb, ml = C.c_uint64(len(circ.ops)), C.c_uint64(64 * 2 * len(circ.ops))
    at, k = np.zeros(nb.value, np.uint32), np.zeros(nb.value, np.uint32)
    q, m = np.zeros(6 * nb.value, np.uint32), np.zeros(ml.value)
    assert lib.mb2_debug_schedule(arr, len(circ.ops), C.byref(opts), n, at.ctypes.data, k.ctypes.data, q.ctypes.data,
                                  m.ctypes.data, C.byref(nb), C.byref(ml), C64) == 0
    del keep
    assert at[:nb.value].max() + 1 == stats[0]


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [C128, C64])
def test_permutations_are_priced_as_the_map_they_are(ctx, precision):
    def seconds(circ, fuse):
        arr, keep = to_mb2_ops(circ)
        opts, out = _lib.SweepOptions(fuse, 0, 0, 0, 0), C.c_double()
        assert _lib.lib().mb2_estimate_sweep_time(ctx.h, arr, len(circ.ops), C.byref(opts), circ.num_qubits, precision,
                                                  C.byref(out)) == 0
        del keep
        return out.value

    plain, ladder, moves = Circuit(22), Circuit(22), Circuit(22)
    for c in (plain, ladder, moves):
        for j in range(11):
            c.gate("ry", [j], [0.1 + j])
    for c in (ladder, moves):
        for j in range(10):
            c.gate("cx", [j, j + 1])
    moves.gate("swap", [2, 7]).gate("x", [4])
    # One pass each: the moves add nothing to it.
    assert seconds(moves, 0) == seconds(plain, 0)
    # A rotation that fusion joined to a CX is priced as the rotation.
    assert seconds(ladder, 1) <= 1.0001 * seconds(plain, 1)
