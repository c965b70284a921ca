"""FP32 products of several components in the one-launch GMRES: each density's stencil sums are FP32 sums, their sum over
the densities is formed in FP64.  Components 1 and 3 are alike and enter the mean field with strengths +E and -E, so
their sums cancel exactly, and component 2's, E / 2^27 of them, is what is left: FP32 additions would lose it.

Three steps of a solve with FP32 products against three with FP64 products: FP32 sums carry 1e-6 of what is left, and
three steps of a well-conditioned system pass that on with a factor of order ten: 1e-4."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_components_add_in_fp64():
    from tramonto_gb300 import native, setup
    from tramonto_gb300.problem import BC_PERIODIC, UATT
    n, nc = 301, 3
    one = [[1.0] * nc] * nc
    rng = np.random.default_rng(4)
    v = 0.3 * rng.standard_normal((2, n))
    p = setup.build_problem(1, (n, 1, 1), (0.05,), ((BC_PERIODIC, BC_PERIODIC),), hs_diam=[1.0] * nc,
                            rho_b=[0.1, 0.2, 0.1], attraction=True, sigma=one, eps=[[0.5] * nc] * nc,
                            rcut=[[2.0] * nc] * nc, vext=np.stack([v[0], v[1], v[0]]))
    s = native.Solver(p)
    x = setup.initial_state(s, p, max_enhancement=2.0)
    s.close()
    for i in range(nc):
        for j, scale in enumerate((2.0 ** 27, 1.0, -2.0 ** 27)):
            off, w, hw = p.stencils[(UATT, i + nc * j)]
            p.stencils[(UATT, i + nc * j)] = (off, scale * w, hw)
    s = native.Solver(p)
    s.fill(x)
    b = np.zeros(s.shape)
    b[:nc] = rng.standard_normal((nc, n))
    b[2] = b[0]
    want = [s.solve(b, tol=1e-14, max_iter=k) for k in (1, 2, 3)]
    s.set_precision(native.FP32)
    for k, (dx, it, rel) in enumerate(want, 1):
        got, it32, rel32 = s.solve(b, tol=1e-14, max_iter=k)
        err = np.abs(got[:nc] - dx[:nc]).max() / np.abs(dx[:nc]).max()
        print(k, rel, rel32, err)
        assert it == it32 == k and abs(rel32 - rel) <= 1e-4 * rel and err <= 1e-4
    s.close()
