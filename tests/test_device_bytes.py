"""What a trajectory run and a sampling call are said to hold on the device,
for callers that account for its memory: never less than they take."""
import ctypes as C

import numpy as np
import pytest

from menos_b200 import _lib
from menos_b200.circuit import to_mb2_ops
from menos_b200.engine import trajectories
from test_dm import noisy_circuit


def said(circ, count, terms, monitored=False):
    arr, keep = to_mb2_ops(circ)
    batch, size = C.c_uint64(), C.c_uint64()
    assert _lib.lib().mb2_trajectories_bytes(circ.num_qubits, arr, len(circ.ops), count, terms, int(monitored),
                                             C.byref(batch), C.byref(size)) == 0
    del keep
    return batch.value, size.value


@pytest.mark.parametrize("n,count,batch", [(3, 5, 5), (16, 80, 64), (20, 80, 16), (24, 2, 1), (30, 8, 1)])
def test_a_batch_counts_all_its_states(n, count, batch):
    _, d = noisy_circuit(n, 8, np.random.default_rng(n), widest=2)
    b, size = said(d, count, 4)
    assert b == batch and size >= batch * (16 << n)
    one, least = said(d, count, 4, monitored=True)
    assert one == 1 and 16 << n <= least <= size


def test_draws():
    lib = _lib.lib()
    assert lib.mb2_draw_bytes(0) == 0
    for shots in (1, 512, 513, 10 ** 6):
        assert 36 * shots <= lib.mb2_draw_bytes(shots) <= 64 * shots + (64 << 10)


@pytest.mark.gpu
@pytest.mark.parametrize("n,count,terms", [(4, 70, 3), (10, 64, 20), (16, 80, 6), (17, 3, 1), (20, 20, 2)])
def test_a_run_holds_no_more(ctx, n, count, terms):
    from cuda.bindings import driver as dv
    from cuda.bindings import runtime as rt

    def pool(attribute, value=None):
        err, p = rt.cudaDeviceGetDefaultMemPool(0)
        assert err == 0
        if value is not None:
            assert rt.cudaMemPoolSetAttribute(p, attribute, value)[0] == 0
            return None
        err, v = rt.cudaMemPoolGetAttribute(p, attribute)
        assert err == 0
        return int(v)

    high = rt.cudaMemPoolAttr.cudaMemPoolAttrUsedMemHigh
    _, d = noisy_circuit(n, 24, np.random.default_rng(n), widest=2)
    paulis = [(i % (1 << n), (3 * i) % (1 << n)) for i in range(1, terms + 1)]
    before = pool(rt.cudaMemPoolAttr.cudaMemPoolAttrUsedMemCurrent)
    pool(high, dv.cuuint64_t(0))
    trajectories(ctx, d, count, 3, paulis)
    taken = pool(high) - before
    batch, size = said(d, count, terms)
    # The pool hands out at its own granularity (at most 2 MiB more for each of the three pieces).
    assert batch * (16 << n) <= taken <= size + (6 << 20)
