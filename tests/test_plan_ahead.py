"""Planning looks for exact moves behind the block that closed a pass.  A
qubit without blocks, or with one only at the program's end, does not make it
look through the whole rest of the program for each pass."""
import ctypes as C
import time

import numpy as np
import pytest

from menos_b200 import _lib, workloads
from menos_b200.circuit import Circuit, to_mb2_ops
from menos_b200.engine import C128


def plan(circ):
    """(passes, seconds of this process)"""
    arr, keep = to_mb2_ops(circ)
    stats = np.zeros(6, np.uint64)
    opts = _lib.SweepOptions(0, 0, 0, 0, 0)
    best = float("inf")
    for _ in range(3):
        t = time.process_time()
        assert _lib.lib().mb2_debug_run_plan(arr, len(circ.ops), C.byref(opts), circ.num_qubits, C128, None,
                                             stats.ctypes.data) == 0
        best = min(best, time.process_time() - t)
    del keep
    return int(stats[0]), best


@pytest.mark.parametrize("family", ["brick", "hea"])
@pytest.mark.parametrize("last", [False, True], ids=["idle", "at the end"])
def test_a_qubit_that_waits(family, last):
    n, depth = 15, 900 if family == "brick" else 400
    layers = getattr(workloads, family)(n, depth, 3)
    whole, t0 = plan(layers)
    waiting = Circuit(n + 1)
    waiting.ops = list(layers.ops)
    if last:
        waiting.gate("x", [n])
    passes, t1 = plan(waiting)
    assert passes <= whole + whole // 50 + 1
    # The same blocks: about the same time (0.8 to 1.3 times it), five to six
    # times it when every pass looked through the rest.
    assert t1 < 3 * t0 + 0.005
