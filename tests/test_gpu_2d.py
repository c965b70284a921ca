"""2-D problems: the point sums with split taps (nodes past a warp's 32 and a chunk's 256 taps), the FP32 products by
FFT or direct sums as their timing chooses, and GMRES with one, several and many chunks of eight basis vectors.

FP64 residuals and J v against the oracle to 1e-12; FP32 products against FP64 to 1e-5 of their max norms, both before
and after the choices; solutions by J dx = b to 1e-8 (linear tolerance 1e-11, densities spread over less than 1e3), the
residual estimate falling with every added step, the adjoint alike."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

WALL, BULK, PER, REFL = -1, 0, 1, 2
CASES = [((9, 7), 0.25, ((WALL, BULK), (REFL, REFL)), 1, False), ((33, 31), 0.2, ((WALL, WALL), (PER, PER)), 1, True),
         ((65, 40), 0.1, ((WALL, BULK), (PER, PER)), 2, True), ((50, 64), 0.1, ((BULK, BULK), (WALL, BULK)), 1, True)]


@pytest.mark.parametrize("n,dx,bc,nc,att", CASES)
def test_2d(n, dx, bc, nc, att):
    import orc
    from goldens import rel_err
    from tramonto_gb300 import native, setup
    rng = np.random.default_rng(n[0])
    N = n[0] * n[1]
    vext = 0.5 * rng.standard_normal((nc, N))
    vext[:, rng.choice(N, N // 20, replace=False)] = 10.0
    one = [[1.0] * nc] * nc
    p = setup.build_problem(2, n + (1,), (dx,) * 2, bc, hs_diam=[1.0, 0.6][:nc], rho_b=[0.3, 0.2][:nc],
                            functional=2 if nc > 1 else 0, attraction=att, sigma=one, eps=[[0.5] * nc] * nc,
                            rcut=[[2.0] * nc] * nc, vext=vext)
    s = native.Solver(p)
    x = setup.initial_state(s, p, max_enhancement=2.0)
    R = s.fill(x)
    o = orc.Oracle(p)
    err = np.abs(R - o.resid(x)).max()
    print(n, "fill against the oracle", err)
    assert err <= 1e-12
    b, v2 = rng.standard_normal(s.shape), rng.standard_normal((nc, N))
    J64, S64 = s.jv(b), s.schur(v2)
    dx_, it, rr = s.solve(b, tol=1e-11)
    lam, ita, rra = s.adjoint_solve(b, tol=1e-11)
    e1 = np.linalg.norm(s.jv(dx_) - b) / np.linalg.norm(b)
    e2 = np.linalg.norm(s.jtv(lam) - b) / np.linalg.norm(b)
    print("solve", it, rr, e1, "adjoint", ita, rra, e2)
    assert rr < 1e-11 and rra < 1e-11 and e1 <= 1e-8 and e2 <= 1e-8
    rel = [s.solve(b, tol=1e-14, max_iter=k)[2] for k in (1, 7, 8, 9, 10, 17)]
    assert all(u >= v for u, v in zip(rel, rel[1:]))
    s.set_precision(native.FP32)
    for _ in range(3):
        assert rel_err(s.jv(b), J64) <= 1e-5 and rel_err(s.schur(v2), S64) <= 1e-5
    s.close()
