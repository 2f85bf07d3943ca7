"""What a kernel reports through the engine's error flag: a wait that ran out is named, and a
host read of results raises.  The wait is one that nothing ends; it gives up by itself after 2 s."""
import time

import pytest

pytestmark = pytest.mark.gpu


def test_a_wait_that_ran_out_is_named(gpu):
    from cupoly_b200 import _lib
    from cupoly_b200.engine import FORWARD, Engine, QBase, UNIFORM, _stream
    e = Engine(2, 0, 4096, 256)
    e.check()
    t = time.perf_counter()
    _lib.call("cp_wait_test", e.handle, _stream())
    with pytest.raises(_lib.CupolyError) as ei:
        e.check()
    assert time.perf_counter() - t < 10
    assert ei.value.code == 5
    assert "tensor-core" in str(ei.value) and "sampler" not in str(ei.value)
    # the flag is cleared and the context still works
    x = e.empty(QBase, 1)
    e.sample(x, QBase, UNIFORM, 1, 0)
    e.dgt(x, QBase, FORWARD)
    e.check()
