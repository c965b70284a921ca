"""The FFT passes at every length class: each register radix (1 to 27) as first and second factor, the three ranges
of first radices, the longest transform (432), lengths of one radix only, odd numbers of lines (the last complex line
of the x passes holds one real line) and tiles with idle lines.

Periodic boxes of hard spheres whose stencils reach one node, so that the transforms run on the box's own lengths (343 has
no two radices and is padded).
With every sum by FFT the FP64 fill equals the direct FP64 one to 1e-12 (transform rounding ~eps log2 of the box,
4e-15, times the sums' scale of a few, with two orders to spare) and the FP32 products the FP64 ones to 1e-5 of their
max norms."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

BOXES = [(432, 25, 9), (27, 432, 4), (24, 5, 384), (405, 18, 5), (20, 400, 3), (375, 6, 15), (9, 27, 25), (250, 10, 12),
         (8, 324, 8), (16, 16, 160), (360, 12, 3), (5, 135, 225),
         (70, 7, 21), (14, 98, 9), (196, 5, 105), (5, 420, 28), (343, 3, 7)]


def problem(box):
    from tramonto_gb300 import setup
    from tramonto_gb300.problem import BC_PERIODIC
    bc = ((BC_PERIODIC, BC_PERIODIC),) * 3
    return setup.build_problem(3, box, (0.5,) * 3, bc, hs_diam=[1.0], rho_b=[0.5])


@pytest.mark.parametrize("box", BOXES)
def test_fft_lengths(box):
    from goldens import rel_err
    from tramonto_gb300 import native, setup
    p = problem(box)
    s = native.Solver(p)
    rng = np.random.default_rng(box[0])
    x = setup.initial_state(s, p)
    x[0] *= np.exp(0.2 * rng.standard_normal(p.nnodes))
    x[1:] *= 1.0 + 0.05 * rng.standard_normal(x[1:].shape)
    R64 = s.fill(x)
    v, v2 = rng.standard_normal(x.shape), rng.standard_normal((1, p.nnodes))
    S64, J64 = s.schur(v2), s.jv(v)
    s.set_fill_arithmetic(native.FILL_FFT)
    s.set_fft_threshold(0)
    err = np.abs(s.fill(x) - R64).max()
    s.set_precision(native.FP32)
    s.set_fft32_policy(1)
    S32, S32b, J32 = s.schur(v2), s.schur(v2), s.jv(v)
    print(box, "FP64 fill", err, "FP32 products", rel_err(S32, S64), rel_err(S32b, S64), rel_err(J32, J64))
    assert err <= 1e-12
    assert max(rel_err(S32, S64), rel_err(S32b, S64), rel_err(J32, J64)) <= 1e-5
    s.close()
