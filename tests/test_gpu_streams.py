"""States' streams come from a pool of their context: many states at once,
one after another, from several threads, and states that outlive the handle
of the context they came from."""
import threading

import numpy as np
import pytest

import pyoracle
from menos_b200 import Context, DeviceState, workloads
from test_oracle_pin import bits_equal

pytestmark = pytest.mark.gpu


def test_states_reuse_streams(ctx, oracle):
    c = workloads.brick(10, 3, 4)
    o = pyoracle.Circuit(10)
    o.ops = list(c.ops)
    want = oracle.run(o)
    for count in (1, 40, 3):  # more than the pool keeps
        states = [DeviceState(ctx, 10) for _ in range(count)]
        assert len({s.stream_handle() for s in states}) == count  # no stream is anyone else's while in use
        for s in states:
            s.init(0.0)
            s.apply_program(c)
        assert all(bits_equal(s.copy_out(), want) for s in states)
        for s in states:
            s.free()


def test_threads(ctx, oracle):
    c = workloads.brick(9, 4, 5)
    o = pyoracle.Circuit(9)
    o.ops = list(c.ops)
    want, bad = oracle.run(o), []

    def work():
        for _ in range(20):
            s = DeviceState(ctx, 9)
            s.init(0.0)
            s.apply_program(c)
            if not bits_equal(s.copy_out(), want):
                bad.append(1)
            s.free()
    threads = [threading.Thread(target=work) for _ in range(6)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad


def test_a_state_outlives_its_contexts_handle():
    mine = Context(0)
    s = DeviceState(mine, 8)
    s.init(0.0)
    assert np.abs(s.copy_out()[0]) == 1.0
    mine.close()
    s.free()
