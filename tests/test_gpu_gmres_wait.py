"""The grid barriers of the one-launch GMRES give up after a bounded wait: with a limit of one poll (the launch's blocks
start microseconds apart) a solve and an adjoint solve report an error status, and with the default limit the same
handle then gives the same solutions as before."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_barrier_waits_that_run_out_are_reported():
    from tramonto_gb300 import native, setup
    p = setup.slit_pore(dict(ndim=1, nx=(1201, 1, 1), dx=0.01, rho_b=0.5, kT=1.5))
    s = native.Solver(p)
    s.fill(setup.initial_state(s, p, max_enhancement=1.0))
    b = np.random.default_rng(3).standard_normal(s.shape)
    for precision in (native.FP64, native.FP32):
        s.set_precision(precision)
        for solve in (s.solve, s.adjoint_solve):
            x, it, rr = solve(b, tol=1e-6)
            assert s.lib.tgpu_set_gmres_wait_limit(s.h, C.c_long(1)) == 0
            with pytest.raises(native.TgpuError) as e:
                solve(b, tol=1e-6)
            assert e.value.status == -2 and "bounded wait ran out" in str(e.value)
            assert s.lib.tgpu_set_gmres_wait_limit(s.h, C.c_long(0)) == 0
            again, it2, rr2 = solve(b, tol=1e-6)
            assert it2 == it > 0 and rr2 == rr < 1e-6 and np.array_equal(again, x)
    s.close()


def test_limit_is_refused_elsewhere():
    from tramonto_gb300 import native, setup
    p = setup.slit_pore(dict(ndim=2, nx=(40, 40, 1), dx=0.1, rho_b=0.5, kT=1.5))
    s = native.Solver(p)
    assert s.lib.tgpu_set_gmres_wait_limit(s.h, C.c_long(1)) == -4
    s.close()
