"""The work that a program using this package has it do, through its public entry points.

A case is a dict of plain values; ``kind`` names the entry point:

newton   ``Solver.newton_solve_device``: a whole Newton solve from its initial state to a residual target
sens     ``Solver.grad_vext``: the sensitivity of the adsorption to the external field (an adjoint solve), host arrays
fill     ``Solver.fill_device``: the FP64-accurate residual of a state, which also keeps the Jacobian's state
schur    ``Solver.schur_device``: one product with the Schur complement, the operator of the GMRES iterations
jv       ``Solver.jv_device``: one Jacobian product
jtv      ``Solver.jtv_device``: one product with the transposed Jacobian

``fluid`` and ``ndim`` choose the problem:

wall 1-D     hard spheres (FMT1) against a planar hard wall, dx = 0.01
slit 1-D     FMT1 + WCA fluid in a slit pore, dx = 0.01 (300 to 4000 nodes in an isotherm sweep)
slit 2-D     the chemically patterned slit of the same sweep, dx = 0.05 (100 x 100 to 400 x 400 nodes)
rough 3-D    FMT1 + WCA fluid next to a rough 12-3 wall, dx = 0.1 or 0.08, periodic in y and z
pore 3-D     binary White-Bear mixture of hard spheres in a cylindrical pore, dx = 0.1

Problems are built by ``tramonto_gb300.setup`` as in a user's program; the states and vectors that go in are made here
with torch, from the seed alone.
"""
import math

import numpy as np
import torch

from tramonto_gb300 import isotherm, native, setup
from tramonto_gb300.problem import BC_IN_BULK, BC_IN_WALL, BC_PERIODIC, DELTA, FMT3, THETA, UATT

ARITH = {"fp64": native.FP64, "fp32": native.FP32, "fp16tc": native.FP16TC, "fp64fft": native.FP64_FFT}


def listed():
    return [
        # the smallest solves: a planar wall in 1-D, FP64 throughout; latency and launches count
        dict(name="newton_1d_wall", kind="newton", fluid="wall", ndim=1, nx=2001, ny=1, nz=1, dx=0.01, arith="fp64"),
        # state points of an isotherm sweep, in its mixed-precision mode: 1-D and 2-D slit pores
        dict(name="newton_1d_slit", kind="newton", fluid="slit", ndim=1, nx=1487, ny=1, nz=1, dx=0.01, arith="fp32"),
        dict(name="newton_2d_slit", kind="newton", fluid="slit", ndim=2, nx=201, ny=201, nz=1, dx=0.05, arith="fp32"),
        # the derivative that goes with a state point of the sweep
        dict(name="sens_1d_slit", kind="sens", fluid="slit", ndim=1, nx=801, ny=1, nz=1, dx=0.01, arith="fp64"),
        # a Jacobian product of the sweep's FP64 mode, an odd mesh
        dict(name="jv_2d_slit", kind="jv", fluid="slit", ndim=2, nx=157, ny=143, nz=1, dx=0.05, arith="fp64"),
        # the benchmark's solve: 128^3, mixed precision
        dict(name="newton_3d_128", kind="newton", fluid="rough", ndim=3, nx=128, ny=128, nz=128, dx=0.1,
             arith="fp16tc"),
        # the operations inside that solve, each by itself: the accurate residual and the FP32 Schur product
        dict(name="fill_3d_128", kind="fill", fluid="rough", ndim=3, nx=128, ny=128, nz=128, dx=0.1, arith="fp64fft"),
        dict(name="schur_3d_128", kind="schur", fluid="rough", ndim=3, nx=128, ny=128, nz=128, dx=0.1, arith="fp32"),
        # a ragged box whose lengths were tuned for nothing
        dict(name="fill_3d_ragged", kind="fill", fluid="rough", ndim=3, nx=83, ny=101, nz=70, dx=0.1,
             arith="fp64fft"),
        # the mixture in the pore: the product of its Newton solve and the adjoint product of its sensitivities
        dict(name="jv_3d_pore", kind="jv", fluid="pore", ndim=3, nx=96, ny=96, nz=64, dx=0.1, arith="fp64fft"),
        dict(name="jtv_3d_pore", kind="jtv", fluid="pore", ndim=3, nx=96, ny=96, nz=64, dx=0.1, arith="fp64"),
        # the largest workload: 256^3 at dx = 0.08
        dict(name="fill_3d_256", kind="fill", fluid="rough", ndim=3, nx=256, ny=256, nz=256, dx=0.08,
             arith="fp64fft"),
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    what = rng.choice(["wall", "slit1", "slit1", "slit2", "slit2", "solve3", "rough3", "rough3", "rough3", "pore3"])
    if what == "wall":
        return dict(kind="newton", fluid="wall", ndim=1, nx=size(400, 4000), ny=1, nz=1, dx=0.01, arith="fp64")
    if what == "slit1":
        kind = rng.choice(["newton", "sens", "jtv", "schur"])
        return dict(kind=kind, fluid="slit", ndim=1, nx=size(301, 4000), ny=1, nz=1, dx=0.01,
                    arith="fp32" if kind == "newton" else "fp64")
    if what == "slit2":
        kind = rng.choice(["newton", "jv", "schur", "fill"])
        n = size(100, 300)
        return dict(kind=kind, fluid="slit", ndim=2, nx=n, ny=n if kind == "newton" else size(100, 300), nz=1, dx=0.05,
                    arith="fp32" if kind == "newton" else "fp64")
    if what == "solve3":
        n = rng.randint(56, 120)
        return dict(kind="newton", fluid="rough", ndim=3, nx=n, ny=n, nz=n, dx=0.1, arith="fp16tc")
    kind = rng.choice(["fill", "schur", "schur", "jv"] if what == "rough3" else ["fill", "schur", "jv", "jtv"])
    arith = {"fill": "fp64fft", "jtv": "fp64", "jv": "fp64fft"}.get(kind) or rng.choice(["fp32", "fp64fft"])
    lo, hi = (48, 160) if what == "rough3" else (48, 110)
    return dict(kind=kind, fluid="rough" if what == "rough3" else "pore", ndim=3, nx=size(lo, hi), ny=size(lo, hi),
                nz=size(lo, hi), dx=0.1, arith=arith)


# ---- the problem ---------------------------------------------------------------------------------------------

def problem(case, seed):
    rng = np.random.default_rng(seed)
    nx = (case["nx"], case["ny"], case["nz"])
    es = (case["dx"],) * case["ndim"]
    if case["fluid"] == "wall":
        return setup.build_problem(1, nx, es, ((BC_IN_WALL, BC_IN_BULK),), hs_diam=[1.0],
                                   rho_b=[rng.uniform(0.6, 0.7)])
    if case["fluid"] == "slit":   # a dense fluid off the vapour-liquid loop, so that every state point has one solution
        return setup.slit_pore(dict(ndim=case["ndim"], nx=nx, dx=case["dx"], rho_b=rng.uniform(0.52, 0.58), kT=1.5,
                                    eps_w=rng.uniform(0.8, 1.0)))
    if case["fluid"] == "rough":
        if nx[0] == nx[1] == nx[2]:
            return setup.config2(n=nx[0], esize=case["dx"], seed=seed)[0]
        kT = 1.2
        vext, _ = setup.rough_wall_vext(nx, es, kT=kT, seed=seed)
        bc = ((BC_IN_WALL, BC_IN_BULK), (BC_PERIODIC, BC_PERIODIC), (BC_PERIODIC, BC_PERIODIC))
        return setup.build_problem(3, nx, es, bc, hs_diam=[1.0], rho_b=[0.6], attraction=True, sigma=[[1.0]],
                                   eps=[[1.0 / kT]], rcut=[[2.5]], vext=vext)
    return setup.config3(nx=nx, esize=case["dx"], seed=seed, pore_radius=0.45 * case["dx"] * min(nx[0], nx[1]))[0]


class Physics:
    """The residual of a problem as plain torch operations in 64 bits on its arrays: stencil sums as FFTs over boxes
    padded by the boundary rules, the rest written out.  Products with the Jacobian are its derivatives."""

    def __init__(self, p):
        self.p = p
        nd = self.nd = p.ndim
        self.shape = tuple(int(p.nx[d]) for d in range(nd))[::-1]          # [z][y][x]
        self.h = [max(int(np.abs(o[:, d]).max()) for o, _, _ in p.stencils.values()) for d in range(nd)]
        self.box = tuple(int(p.nx[d]) + 2 * self.h[d] for d in range(nd))[::-1]
        t = dict(dtype=torch.float64, device="cuda")
        self.vext = torch.tensor(np.asarray(p.vext), **t).reshape((p.ncomp,) + self.shape)
        self.live = torch.tensor(np.asarray(p.zero_density) == 0, device="cuda").reshape((p.ncomp,) + self.shape)
        self.full = self.live & (self.vext != p.vext_max)                  # rows of the Euler-Lagrange equation

    def kernel(self, off, coef):
        g = torch.zeros(self.box, dtype=torch.float64, device="cuda")
        at = tuple(torch.tensor((-off[:, d].astype(np.int64)) % self.box[self.nd - 1 - d], device="cuda")
                   for d in range(self.nd - 1, -1, -1))
        g.index_put_(at, torch.tensor(np.ascontiguousarray(coef), dtype=torch.float64, device="cuda"), accumulate=True)
        return torch.fft.rfftn(g)

    def spectrum(self, f, bulk):
        for d in range(self.nd - 1, -1, -1):      # x last: the first dimension out of range decides
            ax, h, n = self.nd - 1 - d, self.h[d], f.shape[self.nd - 1 - d]
            ends = []
            for side in (0, 1):
                if self.p.bc[d][side] == BC_PERIODIC:
                    ends.append(f.narrow(ax, n - h if side == 0 else 0, h))
                else:
                    s = list(f.shape)
                    s[ax] = h
                    v = bulk if self.p.bc[d][side] == BC_IN_BULK else 0.0
                    ends.append(torch.full(s, v, dtype=f.dtype, device=f.device))
            f = torch.cat([ends[0], f, ends[1]], ax)
        return torch.fft.rfftn(f)

    def back(self, F):
        f = torch.fft.irfftn(F, s=self.box)
        for d in range(self.nd):
            f = f.narrow(self.nd - 1 - d, self.h[d], int(self.p.nx[d]))
        return f

    def sums(self, rho, bulk):
        """The weighted densities (rows n3 n2 n1 n0 V2 V1; copies left out for one particle size) and mean fields."""
        p, nd = self.p, self.nd
        rb, mf = [0.0] * p.nrb, [0.0] * p.ncomp
        for j in range(p.ncomp):
            F = self.spectrum(torch.where(self.live[j], rho[j], torch.zeros_like(rho[j])), float(p.rho_b[j]) * bulk)
            f = float(p.fac_overlap[j])
            off, w, _ = p.stencils[(THETA, j)]
            rb[0] = rb[0] + self.back(F * self.kernel(off, f * w))
            off, w, _ = p.stencils[(DELTA, j)]
            n2 = self.back(F * self.kernel(off, f * w))
            v2 = [self.back(F * self.kernel(off, f * w * off[:, d] * p.esize[d] * p.inv_rad[j])) for d in range(nd)]
            rb[1] = rb[1] + n2
            rb[2] = rb[2] + n2 * float(p.inv_4pir[j])
            rb[3] = rb[3] + n2 * float(p.inv_4pirsq[j])
            for d in range(nd):
                rb[4 + d] = rb[4 + d] + v2[d]
                rb[4 + nd + d] = rb[4 + nd + d] + v2[d] * float(p.inv_4pir[j])
            if p.attraction:
                for i in range(p.ncomp):
                    off, w, _ = p.stencils[(UATT, i + p.ncomp * j)]
                    mf[i] = mf[i] + self.back(F * self.kernel(off, w))
        return rb, mf

    def dphi(self, n3, n2, n1, n0, V2, V1):
        a = 1.0 / (1.0 - n3)
        q = sum(v * v for v in V2)
        d12 = sum(u * v for u, v in zip(V1, V2))
        g, g2, gv = n2 ** 3 - 3.0 * n2 * q, 3.0 * n2 * n2 - 3.0 * q, -6.0 * n2
        if self.p.functional == FMT3:
            cut = n3 <= 1e-10                       # third term and all second derivatives end there
            t = torch.where(cut, torch.full_like(n3, 0.3), n3)
            o = 1.0 - t
            lg = torch.log(o)
            f = (t + o * o * lg) / (36.0 * math.pi * t * t * o * o)
            f1 = (t - 2.0 * o * lg) / (36.0 * math.pi * t * t * o * o) \
                + (t + o * o * lg) / (36.0 * math.pi) * (-2.0 / (t ** 3 * o * o) + 2.0 / (t * t * o ** 3))
        else:
            cut = torch.zeros_like(n3, dtype=torch.bool)
            f, f1 = a * a / (24.0 * math.pi), a ** 3 / (12.0 * math.pi)
        zero = torch.zeros_like(n3)

        def stop(v):
            return torch.where(cut, v.detach(), v)

        return (stop(-torch.log(1.0 - n3)), stop(n2 * a), torch.where(cut, zero, n1 * a + g2 * f),
                torch.where(cut, zero, n0 * a + (n1 * n2 - d12) * a * a + g * f1),
                [stop(-v * a) for v in V2], [torch.where(cut, zero, -u * a + gv * f * v) for u, v in zip(V1, V2)])

    def residual(self, x):
        p, nd, nc = self.p, self.nd, self.p.ncomp
        x = x.reshape((p.nunk,) + self.shape)
        rho, rb = x[:nc], x[nc:nc + p.nrb]
        sums, mf = self.sums(rho, 1.0)
        n3, n2, n1, n0 = rb[0], rb[1], rb[2], rb[3]
        d0, d1, d2, d3, dv1, dv2 = self.dphi(n3, n2, n1, n0, [rb[4 + d] for d in range(nd)],
                                             [rb[4 + nd + d] for d in range(nd)])
        out = []
        db = [float(v) for v in p.dphi_bulk]
        for i in range(nc):
            f, r1, r2 = float(p.fac_overlap[i]), float(p.inv_4pir[i]), float(p.inv_4pirsq[i])
            off, w, _ = p.stencils[(DELTA, i)]
            T = self.spectrum(f * (d0 * r2 + d1 * r1 + d2), f * (db[0] * r2 + db[1] * r1 + db[2])) * self.kernel(off, w)
            for d in range(nd):
                T = T - self.spectrum(f * (dv1[d] * r1 + dv2[d]), 0.0) \
                    * self.kernel(off, w * off[:, d] * p.esize[d] * p.inv_rad[i])
            off, w, _ = p.stencils[(THETA, i)]
            T = T + self.spectrum(f * d3, f * db[3]) * self.kernel(off, w)
            mu = -math.log(p.rho_b[i]) - float(p.betamu_hs_ex[i]) - (float(p.betamu_att[i]) if p.attraction else 0.0)
            row = torch.log(torch.where(self.full[i], rho[i], torch.ones_like(rho[i]))) + mu + self.vext[i] + self.back(T)
            if p.attraction:
                row = row + x[nc + p.nrb + i]
            out.append(torch.where(self.full[i], row, rho[i]))
        for k in range(p.nrb):
            s = sums[k]
            if p.single_size and k in (2, 3):
                s = rb[1] * float(p.inv_4pir[0] if k == 2 else p.inv_4pirsq[0])
            elif p.single_size and k >= 4 + nd:
                s = rb[k - nd] * float(p.inv_4pir[0])
            out.append(s - rb[k])
        if p.attraction:
            out += [mf[i] - x[nc + p.nrb + i] for i in range(nc)]
        return torch.stack(out).reshape(p.nunk, -1)

    def jv(self, x, v):
        return torch.func.jvp(self.residual, (x,), (v,))[1]

    def jtv(self, x, w):
        x = x.detach().requires_grad_(True)
        return torch.autograd.grad(self.residual(x), x, w)[0]

    def schur(self, x, v2):
        p, nc = self.p, self.p.ncomp
        u = self.jv(x, torch.cat([v2, torch.zeros_like(x[nc:])]))
        y = -u
        if p.single_size:                          # the copies n1, n0, V1 follow n2 and V2
            y[nc + 2] -= float(p.inv_4pir[0]) * u[nc + 1]
            y[nc + 3] -= float(p.inv_4pirsq[0]) * u[nc + 1]
            for d in range(self.nd):
                y[nc + 4 + self.nd + d] -= float(p.inv_4pir[0]) * u[nc + 4 + d]
        y[:nc] = 0.0
        return u[:nc] - self.jv(x, y)[:nc]


def initial(ph):
    """The state a solve starts from: densities rho_b exp(-V) (at most rho_b in the pores' wells), with their own
    weighted densities and mean fields."""
    p = ph.p
    x = torch.zeros((p.nunk,) + ph.shape, dtype=torch.float64, device="cuda")
    for i in range(p.ncomp):
        r = float(p.rho_b[i]) * torch.exp(-ph.vext[i].clamp(max=50.0))
        if p.bc[0][1] != BC_IN_BULK:
            r = r.clamp(max=float(p.rho_b[i]))
        x[i] = torch.where(ph.full[i], r, torch.zeros_like(r))
    rb, mf = ph.sums(x[:p.ncomp], 1.0)
    for k in range(p.nrb):
        x[p.ncomp + k] = rb[k]
    x[p.ncomp][x[p.ncomp].abs() < 1e-9] = 0.0      # deep inside walls the sums are empty
    if p.attraction:
        for i in range(p.ncomp):
            x[p.ncomp + p.nrb + i] = mf[i]
    return x.reshape(p.nunk, -1)


def vectors(case, ph, seed):
    """A state in the middle of a solve (weighted densities a little off their sums) and the vector of a product: a
    residual weighted with the densities, as the Krylov vectors of the diagonally preconditioned GMRES (and the
    adjoint solutions) are."""
    p = ph.p
    gen = torch.Generator(device="cuda").manual_seed(int(seed) % (1 << 31) + 17)

    def noise(rows):
        return torch.randn((rows, p.nnodes), dtype=torch.float64, device="cuda", generator=gen)

    def smooth(rows):    # a random field that varies over a particle's size, as residuals do, with a little noise
        f = noise(rows).reshape((rows,) + ph.shape)
        dims = tuple(range(1, 1 + ph.nd))
        k2 = sum((2 * math.pi * torch.fft.fftfreq(n, case["dx"], device="cuda", dtype=torch.float64)
                  .reshape([-1 if a == d else 1 for a in range(ph.nd)])) ** 2 for d, n in enumerate(ph.shape))
        f = torch.fft.ifftn(torch.fft.fftn(f, dim=dims) * torch.exp(-0.05 * k2), dim=dims).real
        return (f / f.std()).reshape(rows, -1) + 0.1 * noise(rows)

    x = initial(ph)
    x[:p.ncomp] *= torch.exp(0.05 * noise(p.ncomp))
    x[p.ncomp:] *= 1.0 + 1e-3 * noise(p.nunk - p.ncomp)
    v = smooth(p.nunk)
    v[:p.ncomp] *= torch.where(ph.full.reshape(p.ncomp, -1), x[:p.ncomp], torch.ones_like(x[:p.ncomp]))
    if case["kind"] == "schur":
        v = v[:p.ncomp].contiguous()
    return x, v


# ---- the interface -------------------------------------------------------------------------------------------

def prepare(case, seed):
    p = problem(case, seed)
    ph = Physics(p)
    s = native.Solver(p)
    s.set_stream(torch.cuda.current_stream().cuda_stream)
    st = dict(kind=case["kind"], s=s, fp32=case["arith"] == "fp32")
    if case["kind"] in ("newton", "sens"):
        st["x0"] = initial(ph)
        st["x"] = st["x0"].clone()
    if case["kind"] == "newton":
        if case["ndim"] < 3 and case["arith"] == "fp32":
            isotherm.set_mode(s, True)
            st["how"] = dict(resid_tol=1e-10, lin_tol=1e-6, lin_max_iter=300)
        elif case["ndim"] < 3:
            st["how"] = dict(resid_tol=1e-10, lin_tol=1e-12, lin_max_iter=500)
        else:
            s.set_precision(ARITH[case["arith"]])
            s.set_fill_arithmetic(native.FILL_MIXED_FFT, switch_norm=0.1)
            st["how"] = dict(resid_tol=1e-8, lin_tol=1e-6, lin_max_iter=300)
        s.newton_solve_device(st["x"], **st["how"])         # the handle's choices and workspaces
    elif case["kind"] == "sens":                            # at a converged state
        s.newton_solve_device(st["x"], resid_tol=1e-10, lin_tol=1e-12, lin_max_iter=500)
        st["xh"] = st["x"].cpu().numpy()
    else:
        st["x"], st["v"] = vectors(case, ph, seed)
        st["R"] = torch.empty_like(st["x"])
        st["y"] = torch.empty_like(st["v"])
        s.set_precision(native.FP64 if case["kind"] == "fill" else ARITH[case["arith"]])
        s.set_fill_arithmetic(native.FILL_FFT if case["ndim"] == 3 else native.FILL_FP64)
        s.fill_device(st["x"], st["R"], 0)
        if case["kind"] != "fill":
            run(st)                                         # the handle's choices and workspaces
    return st


def run(st):
    s, kind = st["s"], st["kind"]
    if kind == "newton":
        st["x"].copy_(st["x0"])
        s.newton_solve_device(st["x"], **st["how"])
        return st["x"]
    if kind == "sens":
        return s.grad_vext(st["xh"], kind=1, icomp=0, tol=1e-11, max_iter=500)
    if kind == "fill":
        s.fill_device(st["x"], st["R"], 0)
        return st["R"]
    if kind == "schur":
        s.schur_device(st["v"], st["y"])
    elif kind == "jv":
        s.jv_device(st["v"], st["y"])
    else:
        s.jtv_device(st["v"], st["y"])
    return st["y"].float() if st["fp32"] else st["y"]       # an FP32 product's result has FP32's digits


def work(case):
    """Vectors read and written once; arithmetic as transforms of the unpadded mesh (2.5 N log2 N each way) for the
    stencil sums a pass cannot do without, and a few dozen operations per node for the local physics."""
    nd, nc = case["ndim"], 2 if case["fluid"] == "pore" else 1
    N = case["nx"] * case["ny"] * case["nz"]
    att = case["fluid"] in ("slit", "rough")
    nunk = nc + 4 + 2 * nd + (nc if att else 0)
    fwd = nc + 4 + 2 * nd + nc * nc * att if nc > 1 else 2 + nd + att + 1
    tr = nc * (nd + 2) + nc
    flops = (fwd + tr) * 2.5 * N * math.log2(N) + 60.0 * N
    byts = 8.0 * N * {"fill": 2 * nunk + nc, "schur": 2 * nc + nunk, "jv": 3 * nunk, "jtv": 3 * nunk,
                      "newton": 2 * nunk + nc, "sens": nunk + 2 * nc}[case["kind"]]
    # a solve takes at least a handful of fills and some tens of products, an adjoint solve some tens of products
    return dict(bytes=byts, flops=flops * {"newton": 40, "sens": 20}.get(case["kind"], 1))


def exact(case, seed):
    if case["kind"] in ("newton", "sens"):
        return None      # the result of an iteration
    ph = Physics(problem(case, seed))
    x, v = vectors(case, ph, seed)
    with torch.set_grad_enabled(case["kind"] == "jtv"):
        r = ph.residual(x) if case["kind"] == "fill" else getattr(ph, case["kind"])(x, v)
    return r.detach()
