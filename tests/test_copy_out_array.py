"""DeviceState.copy_out into an array of the caller's: the library fills it
through its address, so an array of another type, size or layout is refused
before it is called."""
import numpy as np
import pytest

from menos_b200 import DeviceState
from menos_b200.engine import C64, C128


def host_only(n, precision):
    """A state without its device side: what copy_out looks at before the call."""
    st = DeviceState.__new__(DeviceState)
    st.n, st.precision, st.h, st.ctx = n, precision, None, None
    return st


def read_only(a):
    a.flags.writeable = False
    return a


@pytest.mark.parametrize("out", [
    np.zeros(8, np.complex64), np.zeros(8, np.float64), np.zeros(7, np.complex128), np.zeros(16, np.complex128),
    np.zeros(16, np.complex128)[::2], np.zeros((2, 4), np.complex128).T, read_only(np.zeros(8, np.complex128)),
    np.zeros(8, ">c16"), np.zeros(129, np.uint8)[1:].view(np.complex128), [0j] * 8,
], ids=["complex64", "float64", "short", "long", "strided", "transposed", "read-only", "byte order", "misaligned", "list"])
def test_refused(out):
    with pytest.raises(ValueError):
        host_only(3, C128).copy_out(out)


def test_precision_is_the_states():
    with pytest.raises(ValueError):
        host_only(3, C64).copy_out(np.zeros(8, np.complex128))


@pytest.mark.gpu
@pytest.mark.parametrize("precision,dtype", [(C128, np.complex128), (C64, np.complex64)])
def test_taken(ctx, precision, dtype):
    st = DeviceState(ctx, 5, precision)
    st.init(0.5)
    own = st.copy_out()
    for out in (np.ones(32, dtype), np.ones((4, 8), dtype), st.host_array()):
        assert st.copy_out(out) is out
        assert np.array_equal(out.ravel(), own)
