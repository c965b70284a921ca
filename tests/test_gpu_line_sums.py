"""1-D point sums, a pass in one launch: meshes below, at and past the 32 nodes of a block, the largest that takes the
launch and the first that does not, stencils of fewer and of more taps than a chunk of 32, one to three components of
equal and unequal sizes, every kind of boundary and zero-density nodes.

FP64 residuals and Jacobian products against the oracle to 1e-12 of the largest entry (a few hundred roundings of
1e-16); FP32 products to 1e-5 of it.  The reference's FMT3 Jacobian drops the sign of mirrored vector densities, so
there the products are held to the central difference of the oracle's residual, to 1e-7 (step 1e-6: truncation 1e-12
times third derivatives of up to 1e4, roundings 1e-16 / 1e-6)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

WALL, BULK, PER, REFL = -1, 0, 1, 2
CASES = [(5, 0.5, 1, False, (PER, PER)), (31, 0.1, 1, True, (WALL, WALL)), (32, 0.1, 2, True, (WALL, BULK)),
         (33, 0.1, 1, False, (REFL, BULK)), (301, 0.02, 1, True, (BULK, BULK)), (70, 0.05, 3, True, (REFL, REFL)),
         (32768, 0.05, 1, True, (WALL, BULK)), (32769, 0.05, 1, True, (WALL, BULK))]


@pytest.mark.parametrize("n,dx,nc,att,bc", CASES)
@pytest.mark.parametrize("same", [False, True])
def test_line_sums(n, dx, nc, att, bc, same):
    import orc
    from goldens import rel_err
    from tramonto_gb300 import native, setup
    if same and nc == 1 and n > 100:
        pytest.skip("one component has one size")
    rng = np.random.default_rng(n)
    vext = 0.5 * rng.standard_normal((nc, n))
    if n > 30:
        vext[:, rng.choice(n, n // 30, replace=False)] = 10.0
    one = [[1.0] * nc] * nc
    p = setup.build_problem(1, (n, 1, 1), (dx,), (bc,), hs_diam=[1.0] * nc if same else [1.0, 0.8, 0.6][:nc],
                            rho_b=[0.3, 0.2, 0.1][:nc], functional=0 if nc == 1 or same else 2, attraction=att, sigma=one,
                            eps=[[0.5] * nc] * nc, rcut=[[2.0] * nc] * nc, vext=vext)
    s = native.Solver(p)
    x = setup.initial_state(s, p, max_enhancement=2.0)
    o = orc.Oracle(p)
    R, R0 = s.fill(x), o.resid(x)
    v = rng.standard_normal(s.shape)
    mixed = nc > 1 and not same and REFL in bc
    J, J0 = s.jv(v), (o.resid(x + 1e-6 * v) - o.resid(x - 1e-6 * v)) / 2e-6 if mixed else o.jv(x, v)
    print(n, nc, "fill", rel_err(R, R0), "jv", rel_err(J, J0))
    assert np.abs(R - R0).max() <= 1e-12 * max(1.0, np.abs(R0).max()) and rel_err(J, J0) <= (1e-7 if mixed else 1e-12)
    s.set_precision(native.FP32)
    assert rel_err(s.jv(v), J0) <= 1e-5
    s.close()
