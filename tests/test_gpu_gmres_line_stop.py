"""Cycles of the one-launch GMRES that converge after one, two and three steps, many times each: the block that solves
for the result leaves the loop ahead of the others there.  A cycle that stops on its tolerance after k steps and one cut
off at k steps build the same Krylov space and sum in the same order, so their solutions are equal."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

WALL, BULK, PER = -1, 0, 1


@pytest.mark.parametrize("n,nc,att,bc", [(9, 1, True, (PER, PER)), (1200, 1, False, (WALL, BULK)),
                                         (2001, 2, True, (WALL, BULK)), (9664, 1, True, (WALL, WALL))])
def test_early_convergence(n, nc, att, bc):
    from tramonto_gb300 import native, setup
    rng = np.random.default_rng(n)
    one = [[1.0] * nc] * nc
    p = setup.build_problem(1, (n, 1, 1), (0.5 if n < 100 else 0.05,), (bc,), hs_diam=[1.0, 0.8][:nc],
                            rho_b=[0.3, 0.2][:nc], functional=2 if nc > 1 else 0, attraction=att, sigma=one,
                            eps=[[0.5] * nc] * nc, rcut=[[2.0] * nc] * nc, vext=0.3 * rng.standard_normal((nc, n)))
    s = native.Solver(p)
    s.fill(setup.initial_state(s, p, max_enhancement=2.0))
    b = rng.standard_normal(s.shape)
    for solve in (s.solve, s.adjoint_solve):
        cut = [solve(b, tol=1e-14, max_iter=k) for k in (1, 2, 3)]
        assert 1.0 > cut[0][2] > cut[1][2] > cut[2][2]
        for k, (dx, it, rr) in enumerate(cut, 1):
            for _ in range(100):
                got, its, rel = solve(b, tol=rr * (1.0 + 1e-9), max_iter=50)
                assert it == its == k and rel == rr and np.array_equal(got, dx)
    s.close()
