"""The arithmetic of the transposed sums in 3-D, chosen by the caller: tgpu_set_fft_threshold 0 takes the FP64 transforms,
a length that no stencil has the direct FP64 sums.  J^T w by each against the oracle's, entry by entry, to 1e-12 of the
largest entry of its row (a sum of up to a few thousand terms; the transforms of these boxes carry 16 roundings of their
largest value), with the number of sums to tell which ran: the transforms take one per component and direction.  With
direct sums a non-finite entry stays within the stencils' reach."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

WALL, BULK, PER, REFL = -1, 0, 1, 2
CASES = [((23, 20, 21), ((WALL, BULK), (PER, PER), (PER, PER)), 1, True),
         ((21, 19, 22), ((BULK, WALL), (WALL, WALL), (BULK, BULK)), 2, False),
         ((22, 21, 20), ((PER, PER), (WALL, BULK), (PER, PER)), 2, True)]


def problem(box, bc, nc, att):
    from tramonto_gb300 import setup
    rng = np.random.default_rng(sum(box))
    N = int(np.prod(box))
    vext = 0.3 * rng.standard_normal((nc, N))
    vext[:, rng.choice(N, N // 20, replace=False)] = 10.0
    pair = [[1.0] * nc] * nc
    return setup.build_problem(3, box, (0.2,) * 3, bc, hs_diam=[1.0, 0.8][:nc], rho_b=[0.3, 0.2][:nc],
                               functional=2 if nc == 2 else 0, attraction=att, sigma=pair, eps=pair,
                               rcut=[[1.6] * nc] * nc, vext=vext), rng, N


@pytest.mark.parametrize("box,bc,nc,att", CASES)
def test_both_ways_against_the_oracle(box, bc, nc, att):
    import orc
    from tramonto_gb300 import native, setup
    p, rng, N = problem(box, bc, nc, att)
    s = native.Solver(p)
    x = setup.initial_state(s, p)
    s.fill(x)
    w = rng.standard_normal((p.nunk, N))
    want = orc.Oracle(p).jtv(x, w)
    scale = np.abs(want).max(axis=1)
    for threshold in (0, 2 ** 31 - 1, 0):
        s.set_fft_threshold(threshold)
        s.jtv(w)
        s.reset_stats()
        got = s.jtv(w)
        sums = s.stats()["conv_launches"]
        err = (np.abs(got - want).max(axis=1) / scale).max()
        print(box, threshold, "error", err, "sums", sums)
        assert err <= 1e-12
        assert sums == 2 * nc if threshold == 0 else sums >= 4 * nc
    s.set_fft_threshold(2 ** 31 - 1)
    w[nc, N // 2] = np.inf     # the row of n3: read over the ball's reach (three nodes each way)
    bad = ~np.isfinite(s.jtv(w))
    assert 0 < bad.sum() <= nc * 7 ** 3 + 1
    s.close()


def test_reflecting_boundaries_stay_direct():
    from tramonto_gb300 import native, setup
    p, rng, N = problem((20, 21, 19), ((WALL, BULK), (REFL, REFL), (PER, PER)), 1, False)
    s = native.Solver(p)
    s.fill(setup.initial_state(s, p))
    w = rng.standard_normal((p.nunk, N))
    sums = []
    for threshold in (2 ** 31 - 1, 0, -1):
        s.set_fft_threshold(threshold)
        s.reset_stats()
        s.jtv(w)
        sums.append(s.stats()["conv_launches"])
    assert sums[0] == sums[1] == sums[2] >= 4
    s.close()


def test_adjoint_products_do_not_build_the_fills_spectra():
    import torch
    from tramonto_gb300 import native, setup
    p = setup.config2(n=64)[0]
    s = native.Solver(p)
    x = setup.initial_state(s, p)
    s.fill(x)
    s.jtv(np.ones(s.shape))
    free = torch.cuda.mem_get_info()[0]
    s.set_fill_arithmetic(native.FILL_FFT)
    s.fill(x)
    # theta, delta and attraction: twelve spectra and three boxes of (F / 2 + 1) x 64 x 64 points, F at least 64
    assert free - torch.cuda.mem_get_info()[0] >= 15 * 33 * 64 * 64 * 16
    s.close()
