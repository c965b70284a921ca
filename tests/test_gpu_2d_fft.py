"""FP32 sums of 2-D problems by transforms and by direct sums, on meshes where the transforms are the faster ones (the test
asserts that they were taken): unequal ends along x, whose shared boundary value the low end's profile makes up for, walls,
bulk and periodic ends along y, a two-phase interface, one and two components, zero-density nodes.

FP32 fills to 1e-4 and FP32 products to 1e-5 of the FP64 ones' largest entry, as in 3-D; solutions by J dx = b to 1e-4 with
tolerance 1e-6 (the densities spread over less than 1e2)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

WALL, BULK, PER = -1, 0, 1
CASES = [((260, 250), ((WALL, BULK), (PER, PER)), 1, False), ((251, 260), ((BULK, WALL), (WALL, WALL)), 2, False),
         ((262, 245), ((WALL, WALL), (BULK, BULK)), 1, False), ((250, 257), ((BULK, BULK), (PER, PER)), 1, True)]


@pytest.mark.parametrize("n,bc,nc,interface", CASES)
def test_2d_fft(n, bc, nc, interface):
    from goldens import rel_err
    from tramonto_gb300 import native, setup
    from tramonto_gb300.problem import DELTA, THETA
    rng = np.random.default_rng(sum(n))
    N = n[0] * n[1]
    one = [[1.0] * nc] * nc
    vext = 0.3 * rng.standard_normal((nc, N))
    vext[:, rng.choice(N, N // 25, replace=False)] = 10.0
    p = setup.build_problem(2, n + (1,), (0.05,) * 2, bc, hs_diam=[1.0, 0.8][:nc], rho_b=[0.3, 0.2][:nc],
                            functional=2 if nc == 2 else 0, attraction=True, sigma=one, eps=[[0.5] * nc] * nc,
                            rcut=[[2.0] * nc] * nc, vext=vext)
    if interface:
        p.interface = 2
        sides = [setup.bulk_constants(0, [1.0], [r], True, {0: p.stencils[(2, 0)]}, 1) for r in (0.2, 0.4)]
        p.rho_b_lbb, p.rho_b_rtf = np.array([0.2]), np.array([0.4])
        p.dphi_lbb, p.dphi_rtf = sides[0]["dphi_bulk"], sides[1]["dphi_bulk"]
        p.betamu_if = np.array([1.0])
    s = native.Solver(p)
    x = setup.initial_state(s, p, max_enhancement=1.5)
    x[:nc] *= np.exp(0.1 * rng.standard_normal((nc, N)))
    x[nc:] *= 1.0 + 0.05 * rng.standard_normal(x[nc:].shape)
    v, v2, b = rng.standard_normal(x.shape), rng.standard_normal((nc, N)), rng.standard_normal(x.shape)
    R, J, S = s.fill(x), s.jv(v), s.schur(v2)
    for policy, took in ((0, -1), (-1, 1)):
        s.set_precision(native.FP32)
        s.set_fill_arithmetic(native.FILL_FP32)
        for _ in range(5):     # (a choice timed while the host was held up is made again)
            s.set_fft32_policy(policy)
            s.schur(v2)
            if s.fft32_choice(DELTA)["forward"] == s.fft32_choice(DELTA)["transposed"] == took:
                break
        fill = [rel_err(s.fill(x), R) for _ in range(2)]
        prod = [rel_err(s.jv(v), J), rel_err(s.schur(v2), S), rel_err(s.schur(v2), S)]
        dx, it, rr = s.solve(b, tol=1e-6)
        s.set_precision(native.FP64)
        err = np.linalg.norm(s.jv(dx) - b) / np.linalg.norm(b)
        print(n, "policy", policy, "fills", fill, "products", prod, "solve", it, rr, err)
        for t in (THETA, DELTA):
            c = s.fft32_choice(t)
            assert c["forward"] == c["transposed"] == took
        assert max(fill) <= 1e-4 and max(prod) <= 1e-5 and rr < 1e-6 and err <= 1e-4
    s.close()
