"""The adjoint's transposed sums as FP64 FFT convolutions (3-D, no reflecting boundary): <u, J v> = <J^T u, v> to 1e-12 of
|u| |J v| against the direct FP64 J v, for every other boundary condition, ragged boxes, one and two components
(seven spectral terms with a binary attraction), and zero-density nodes.  The meshes are large enough for the rule to
choose the transforms; the reflecting box keeps the direct sums."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

WALL, BULK, PER, REFL = -1, 0, 1, 2
CASES = [
    ((31, 27, 29), ((WALL, BULK), (PER, PER), (PER, PER)), 1, True),
    ((30, 33, 28), ((WALL, WALL), (BULK, BULK), (PER, PER)), 1, False),
    ((29, 30, 31), ((BULK, WALL), (WALL, WALL), (BULK, BULK)), 2, False),
    ((32, 26, 30), ((PER, PER), (WALL, BULK), (PER, PER)), 2, True),
    ((28, 30, 27), ((WALL, BULK), (REFL, REFL), (PER, PER)), 1, True),
]


@pytest.mark.parametrize("box,bc,ncomp,att", CASES)
def test_adjoint_fft_dot_identity(box, bc, ncomp, att):
    from tramonto_gb300 import native, setup
    rng = np.random.default_rng(sum(box))
    N = int(np.prod(box))
    vext = 0.3 * rng.standard_normal((ncomp, N))
    vext[:, rng.choice(N, N // 20, replace=False)] = 10.0
    pair = [[1.0] * ncomp] * ncomp
    p = setup.build_problem(3, box, (0.2,) * 3, bc, hs_diam=[1.0, 0.8][:ncomp], rho_b=[0.3, 0.2][:ncomp],
                            functional=2 if ncomp == 2 else 0, attraction=att, sigma=pair, eps=pair,
                            rcut=[[2.0] * ncomp] * ncomp, vext=vext)
    s = native.Solver(p)
    s.fill(setup.initial_state(s, p))
    u, v = rng.standard_normal((p.nunk, N)), rng.standard_normal((p.nunk, N))
    jv, jtu = s.jv(v), s.jtv(u)
    a, b = float(np.vdot(u, jv)), float(np.vdot(jtu, v))
    scale = float(np.linalg.norm(u) * np.linalg.norm(jv))
    print(box, "<u, Jv>", a, "<Jtu, v>", b, "rel", abs(a - b) / scale)
    assert abs(a - b) <= 1e-12 * scale
    s.close()
