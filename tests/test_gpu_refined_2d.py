"""TGPU_FILL_REFINED in 2-D where a refined fill makes the handle's first FP32 sums (the choice between direct and FFT sums
falls inside it): a fill of x1 after one of x0, and a second step from there, against the FP64 fill.

The FP32 sums cover the change of the state alone, so their rounding is about 3e-7 of the change's sums; those are at
most 30 times the largest change of the residual here (rows in which terms cancel), which gives 1e-5 of it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

WALL, BULK, PER = -1, 0, 1
CASES = [((33, 31), 0.2, ((WALL, BULK), (PER, PER)), 1, False), ((65, 40), 0.1, ((WALL, WALL), (PER, PER)), 1, True),
         ((50, 64), 0.1, ((BULK, BULK), (WALL, BULK)), 2, True)]


@pytest.mark.parametrize("reopened", [False, True])
@pytest.mark.parametrize("n,dx,bc,nc,att", CASES)
def test_refined_fill_2d(n, dx, bc, nc, att, reopened):
    from tramonto_gb300 import native, setup
    rng = np.random.default_rng(n[0])
    N = n[0] * n[1]
    one = [[1.0] * nc] * nc
    p = setup.build_problem(2, n + (1,), (dx,) * 2, bc, hs_diam=[1.0, 0.6][:nc], rho_b=[0.3, 0.2][:nc],
                            functional=2 if nc > 1 else 0, attraction=att, sigma=one, eps=[[0.5] * nc] * nc,
                            rcut=[[2.0] * nc] * nc, vext=0.3 * rng.standard_normal((nc, N)))
    s = native.Solver(p)
    x = [setup.initial_state(s, p, max_enhancement=2.0)]
    for _ in range(2):
        x.append(x[-1] * (1.0 + 1e-4 * rng.uniform(-1, 1, x[0].shape)))
    R = [s.fill(v) for v in x]
    if reopened:   # a choice made and taken back
        s.set_precision(native.FP32)
        s.schur(rng.standard_normal((nc, N)))
        s.set_precision(native.FP64)
        s.set_fft32_policy(-1)
    s.set_fill_arithmetic(native.FILL_REFINED, tau=1e-3)
    assert np.abs(s.fill(x[0]) - R[0]).max() == 0.0   # FP64 sums, the reference
    s.reset_stats()
    for k in (1, 2):
        err, change = np.abs(s.fill(x[k]) - R[k]).max(), np.abs(R[k] - R[0]).max()
        print(n, k, "error", err, "change", change)
        assert err <= 1e-5 * change
    assert s.stats()["fp64_refreshes"] == 0
    s.close()
