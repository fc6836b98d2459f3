"""X, CX and SWAP in programs for the tensor cores: they are part of a phase's
matrix like any other block, and do not wait behind the other blocks of their
pass as they do in the SIMT programs, whose kernels take them by the tile's
map."""
import ctypes as C

import numpy as np
import pytest

from menos_b200 import _lib, workloads
from menos_b200.circuit import to_mb2_ops
from menos_b200.engine import C64
from test_host import as_oracle_circuit
from test_tc_plan import mixed_circuit, run_plan


# Passes and register layouts of the unfused RY/RZ + CX ansatz of 10 layers as
# they are without the maps; with the permutations waiting 81, 86 and 90
# layouts, and a pass more at 26 and 30 qubits.
@pytest.mark.parametrize("n,passes,layouts", [(26, 19, 75), (28, 21, 79), (30, 14, 85)])
def test_unfused_ladders(n, passes, layouts):
    circ = workloads.hea(n, 10, 3)
    arr, keep = to_mb2_ops(circ)
    stats = np.zeros(6, np.uint64)
    opts = _lib.SweepOptions(0, 0, 0, 0, 0)
    assert _lib.lib().mb2_debug_run_plan(arr, len(circ.ops), C.byref(opts), n, C64, None, stats.ctypes.data) == 0
    del keep
    assert stats[0] == stats[1] <= passes and stats[5] <= layouts


@pytest.mark.parametrize("name", ["hea", "mixed"])
@pytest.mark.parametrize("n,tile", [(12, 11), (14, 12), (15, 13)])
def test_unfused_plans_match_the_oracle(oracle, name, n, tile):
    # (The mixed circuit's three-qubit blocks keep passes in SIMT form.)
    circ = workloads.hea(n, 4, n) if name == "hea" else mixed_circuit(n, 5, n)
    got, stats = run_plan(circ, tile=tile, fuse=False)
    assert name == "mixed" or stats["tc_passes"] > 0
    assert np.max(np.abs(got - oracle.run(as_oracle_circuit(circ), fuse_gates=False))) <= 1e-12
