"""FFT sums over boxes that share one boundary value between both ends of a dimension (F >= n + reach instead of
n + 2 reach), against the direct FP64 sums: every pair of wall and bulk ends along x (unequal ends need the low end's
profile), equal and unequal ends along y and z, reflecting and periodic ones beside them, meshes shorter than the
stencils' reach, a two-phase interface, two components, and a moved bulk state.

FP64 fills to 1e-12 (transform rounding as in test_gpu_fft_lengths), FP32 fills to 1e-4 and FP32 products to 1e-5 of
their max norms, FP64-accurate products to 1e-12."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

WALL, BULK, PER, REFL = -1, 0, 1, 2
CASES = [((23, 12, 14), ((WALL, BULK), (PER, PER), (PER, PER)), 1, False), ((26, 13, 15), ((BULK, WALL), (WALL, WALL), (BULK, BULK)), 1, False),
         ((21, 15, 13), ((WALL, WALL), (BULK, WALL), (REFL, REFL)), 2, False), ((24, 14, 13), ((BULK, BULK), (WALL, BULK), (PER, PER)), 2, False),
         ((9, 14, 12), ((WALL, BULK), (WALL, WALL), (PER, PER)), 1, False), ((17, 12, 13), ((REFL, BULK), (BULK, BULK), (PER, PER)), 1, False),
         ((22, 12, 13), ((BULK, BULK), (PER, PER), (PER, PER)), 1, True)]


@pytest.mark.parametrize("box,bc,nc,interface", CASES)
def test_fft_boundaries(box, bc, nc, interface):
    from goldens import rel_err
    from tramonto_gb300 import native, setup
    rng = np.random.default_rng(sum(box))
    N = int(np.prod(box))
    one = [[1.0] * nc] * nc
    vext = 0.3 * rng.standard_normal((nc, N))
    vext[:, rng.choice(N, N // 25, replace=False)] = 10.0
    p = setup.build_problem(3, box, (0.2,) * 3, bc, hs_diam=[1.0, 0.8][:nc], rho_b=[0.3, 0.2][:nc],
                            functional=2 if nc == 2 else 0, attraction=True, sigma=one, eps=[[0.5] * nc] * nc,
                            rcut=[[2.0] * nc] * nc, vext=vext)
    if interface:
        p.interface = 2
        sides = [setup.bulk_constants(0, [1.0], [r], True, {0: p.stencils[(2, 0)]}, 1) for r in (0.2, 0.4)]
        p.rho_b_lbb, p.rho_b_rtf = np.array([0.2]), np.array([0.4])
        p.dphi_lbb, p.dphi_rtf = sides[0]["dphi_bulk"], sides[1]["dphi_bulk"]
        p.betamu_if = np.array([1.0])
    s = native.Solver(p)
    x = setup.initial_state(s, p, max_enhancement=2.0)
    x[:nc] *= np.exp(0.1 * rng.standard_normal((nc, N)))
    x[nc:] *= 1.0 + 0.05 * rng.standard_normal(x[nc:].shape)
    v, v2 = rng.standard_normal(x.shape), rng.standard_normal((nc, N))
    for moved in (False, True):
        if moved:
            if interface:
                break
            s.set_bulk(0.9 * np.asarray(p.rho_b))
        s.set_fill_arithmetic(native.FILL_FP64)
        s.set_precision(native.FP64)
        R, J, S = s.fill(x), s.jv(v), s.schur(v2)
        s.set_fill_arithmetic(native.FILL_FFT)
        s.set_precision(native.FP64_FFT)
        s.set_fft_threshold(0)
        e = [np.abs(s.fill(x) - R).max(), rel_err(s.jv(v), J), rel_err(s.schur(v2), S)]
        s.set_precision(native.FP32)
        s.set_fft32_policy(1)
        s.set_fill_arithmetic(native.FILL_FP32)
        e32 = [rel_err(s.fill(x), R), rel_err(s.jv(v), J), rel_err(s.schur(v2), S), rel_err(s.schur(v2), S)]
        print(box, "FP64 FFT", e, "FP32", e32)
        assert max(e) <= 1e-12
        assert e32[0] <= 1e-4 and max(e32[1:]) <= 1e-5
    s.close()
