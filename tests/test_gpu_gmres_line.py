"""GMRES of 1-D problems in one launch, at the edges of its split: meshes smaller than a tile, one node past a tile,
the smallest and largest numbers of nodes per block (8 and 64) and the first mesh that takes the separate kernels,
one to three components (with and without attraction), bulk, wall, periodic and reflecting boundaries, zero-density
nodes, and cycles that end at the iteration limit.

The solution is checked by the matrix-free products: J dx = b and J^T lambda = g to 1e-8 of the right-hand side (the
linear tolerance 1e-11 on the preconditioned residual times the range of the densities, under 1e3); FP32 products to
1e-4 with tolerance 1e-6; and a solve cut off after k steps reports k steps and the residual of the Krylov space,
no larger than one step earlier."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

WALL, BULK, PER, REFL = -1, 0, 1, 2
CASES = [(5, 1, False, (WALL, BULK)), (8, 1, True, (PER, PER)), (9, 2, True, (WALL, WALL)), (301, 1, True, (WALL, WALL)),
         (1200, 1, False, (WALL, BULK)), (1209, 1, True, (REFL, BULK)), (2001, 2, False, (BULK, BULK)),
         (1417, 3, True, (WALL, BULK)), (9664, 1, True, (WALL, BULK)), (9665, 1, False, (PER, PER))]


def problem(n, nc, att, bc):
    from tramonto_gb300 import setup
    rng = np.random.default_rng(n)
    dx = 0.5 if n < 100 else 0.05
    vext = 0.5 * rng.standard_normal((nc, n))
    if n > 100:
        vext[:, rng.choice(n, n // 30, replace=False)] = 10.0
    one = [[1.0] * nc] * nc
    return setup.build_problem(1, (n, 1, 1), (dx,), (bc,), hs_diam=[1.0, 0.8, 0.6][:nc], rho_b=[0.3, 0.2, 0.1][:nc],
                               functional=2 if nc > 1 else 0, attraction=att, sigma=one, eps=[[0.5] * nc] * nc,
                               rcut=[[2.0] * nc] * nc, vext=vext), rng


@pytest.mark.parametrize("n,nc,att,bc", CASES)
def test_one_launch_gmres(n, nc, att, bc):
    from tramonto_gb300 import native, setup
    from tramonto_gb300.native import Solver
    p, rng = problem(n, nc, att, bc)
    if n < 100 and PER in bc:
        p.bc = ((PER, PER),)
    s = Solver(p)
    s.fill(setup.initial_state(s, p, max_enhancement=2.0))
    b = rng.standard_normal(s.shape)
    dx, it, rr = s.solve(b, tol=1e-11)
    err = np.linalg.norm(s.jv(dx) - b) / np.linalg.norm(b)
    lam, ita, rra = s.adjoint_solve(b, tol=1e-11)
    erra = np.linalg.norm(s.jtv(lam) - b) / np.linalg.norm(b)
    print(n, nc, "solve", it, rr, err, "adjoint", ita, rra, erra)
    assert rr < 1e-11 and err <= 1e-8 and rra < 1e-11 and erra <= 1e-8
    rels = [s.solve(b, tol=1e-14, max_iter=k)[1:] for k in (1, 2, 5)]
    assert [r[0] for r in rels] == [1, 2, 5] or it < 5
    assert rels[0][1] >= rels[1][1] >= rels[2][1]
    assert np.abs(s.solve(np.zeros(s.shape))[0]).max() == 0.0
    s.set_precision(native.FP32)
    dx32, it32, rr32 = s.solve(b, tol=1e-6)
    err32 = np.linalg.norm(s.jv(dx32) - b) / np.linalg.norm(b)
    print("FP32", it32, rr32, err32)
    assert rr32 < 1e-6 and err32 <= 1e-4
    with pytest.raises(native.TgpuError) as e:
        s.solve(np.full(s.shape, np.nan))
    assert e.value.status == -6
    s.close()
