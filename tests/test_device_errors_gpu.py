"""What a kernel reports through the engine's error flag: a wait that ran out is named, and a
host read of results raises.  The wait is one that nothing ends; it gives up by itself after 2 s."""
import subprocess
import time

import numpy as np
import pytest

from tests.common import random_poly_residues

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


def test_host_reads_raise_what_a_kernel_reported(gpu):
    from cupoly_b200 import _lib, cupoly as cu
    from cupoly_b200.batch import MixedPolymul
    from cupoly_b200.engine import _stream

    def run_out(e):
        _lib.call("cp_wait_test", e.handle, _stream())

    mp = MixedPolymul([(2048, 1)], kmax=1)
    e = mp.groups[2048]["engine"]
    a = random_poly_residues(3, e.Q, 2048)
    one = np.zeros_like(a)
    one[:, 0] = 1
    mp.set_inputs(0, a, one)
    mp.run()
    assert np.array_equal(mp.result(0), a)
    run_out(e)
    with pytest.raises(_lib.CupolyError, match="wait"):
        mp.result(0)
    assert np.array_equal(mp.result(0), a)

    x = e.zeros(0, 1)
    run_out(e)
    with pytest.raises(_lib.CupolyError, match="wait"):
        e.export_residues(x, 0, 0)
    assert len(e.export_residues(x, 0, 0)) == e.wire_bytes(0, 1)

    cu.CUDAEngine.init(2, 3, 4096, 256)
    ctx = cu.Context()
    p = cu.poly_t()
    cu.poly_init(ctx, p)
    cu.poly_set_coeff(ctx, p, 3, 7)
    cu.poly_add(ctx, p, p, p)
    run_out(cu.CUDAEngine.engine)
    with pytest.raises(_lib.CupolyError, match="wait"):
        cu.poly_get_coeff(ctx, p, 3)
    assert cu.poly_get_coeff(ctx, p, 3) == 14
    run_out(cu.CUDAEngine.engine)
    with pytest.raises(_lib.CupolyError, match="wait"):
        cu.poly_export_residues(ctx, p)
    cu.CUDAEngine.destroy()


def test_cxx_host_reads_raise_what_a_kernel_reported(gpu, tmp_path):
    from tests.test_cxx_host import CXX_DIR, _compile
    exe = _compile(CXX_DIR + "/wait_error.cpp", str(tmp_path / "wait_error"))
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout.count("wait") == 2 and r.stdout.rstrip().endswith("14"), r.stdout + r.stderr
