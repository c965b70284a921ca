"""FP32 products of several components in 2-D, with their sums as FP32 transforms: one density's FP32 sums are added to the
others' in FP64.  Components 1 and 3 are alike and enter the mean field with strengths +E and -E, so their sums cancel
exactly, and component 2's, E / 2^27 of them, is what is left: FP32 additions would lose it.  The mesh is large enough
for the transforms to be the faster sums (attraction 5300 points a pair, balls and shells 385, 250 x 240 nodes).

Products against FP64 ones to 1e-5 of the largest entry, as for every FP32 product."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_components_add_in_fp64():
    from goldens import rel_err
    from tramonto_gb300 import native, setup
    from tramonto_gb300.problem import BC_IN_WALL, BC_PERIODIC, DELTA, THETA, UATT
    nx, ny, nc = 250, 240, 3
    one = [[1.0] * nc] * nc
    rng = np.random.default_rng(4)
    v = 0.3 * rng.standard_normal((2, nx * ny))
    p = setup.build_problem(2, (nx, ny, 1), (0.05,) * 2, ((BC_IN_WALL, BC_IN_WALL), (BC_PERIODIC, BC_PERIODIC)),
                            hs_diam=[1.0] * nc, rho_b=[0.1, 0.2, 0.1], attraction=True, sigma=one,
                            eps=[[0.5] * nc] * nc, rcut=[[2.0] * nc] * nc, vext=np.stack([v[0], v[1], v[0]]))
    s = native.Solver(p)
    x = setup.initial_state(s, p, max_enhancement=2.0)
    s.close()
    for i in range(nc):
        for j, scale in enumerate((2.0 ** 27, 1.0, -2.0 ** 27)):
            off, w, hw = p.stencils[(UATT, i + nc * j)]
            p.stencils[(UATT, i + nc * j)] = (off, scale * w, hw)
    s = native.Solver(p)
    s.fill(x)
    v2 = rng.standard_normal((nc, nx * ny))
    v2[2] = v2[0]
    J = np.zeros(s.shape)
    J[:nc] = v2
    S64, J64 = s.schur(v2), s.jv(J)
    s.set_precision(native.FP32)
    for _ in range(5):         # (a choice timed while the host was held up is made again)
        s.set_fft32_policy(-1)
        s.schur(v2)
        if s.fft32_choice(DELTA)["forward"] == s.fft32_choice(DELTA)["transposed"] == 1:
            break
    for _ in range(3):
        e = rel_err(s.schur(v2), S64), rel_err(s.jv(J), J64)
        print(e)
        assert max(e) <= 1e-5
    assert s.fft32_choice(THETA)["forward"] == s.fft32_choice(DELTA)["forward"] == 1
    assert s.fft32_choice(THETA)["transposed"] == s.fft32_choice(DELTA)["transposed"] == 1
    s.close()
