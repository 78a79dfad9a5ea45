"""Performance cases of the library: what a program that uses it has it do.

``listed()`` names fixed cases, ``draw(rng)`` gives others of the same ranges.
``prepare(case, seed)`` makes what a program holds before the call (the
configuration, the device-resident state, device or host arrays),
``run(state)`` is one pass through the public entry points, ``work(case)`` the
bytes and operations that pass cannot do without, and ``exact(case, seed)`` the
pass's results in 64 bits from plain torch, without the library.

Kinds of case:

  step      one time step of a run in its steady state (Solver.step)
  startup   a state uploaded from pinned host memory and the first four steps,
            which rebuild the solver tables three times (Solver.set_state, step)
  ensemble  several runs advanced together (ensemble_run, graph replay)
  helm      isolated batched vertical solves on device arrays
  column    one penalty system on host arrays (Solver.penalty_main)
  legacy    the reference's routines on host fields (horfft, dpdz, filter,
            interface average)
  diag      the run's statistics (Solver.diag)
"""
import math

import numpy as np
import torch

import iwrepo_b200 as iw
from iwrepo_b200 import config as cf


def listed():
    return [
        # the smallest 3-D run (64 x 64 x (4 x 17)) in the parity precision: launches and latency
        dict(name="step_64_fp64", kind="step", nx=64, ny=64, nzloc=17, nsubd=4, prec="fp64", tune=False),
        # the FP64 production size of the parity runs (256 x 256 x (8 x 25))
        dict(name="step_256_fp64", kind="step", nx=256, ny=256, nzloc=25, nsubd=8, prec="fp64", tune=True),
        # the benchmark run: 512 x 512 x (12 x 33), mixed precision, launch choices autotuned as bench.py does
        dict(name="step_512_mixed", kind="step", nx=512, ny=512, nzloc=33, nsubd=12, prec="mixed", tune=True),
        # mixed-radix lengths in x and y and an odd number of points: a run sized by its physics
        dict(name="step_ragged_mixed", kind="step", nx=192, ny=120, nzloc=22, nsubd=5, prec="mixed", tune=False),
        # the reference's shipped 2-D forced run: paddle, adaptive time step, uneven subdomains
        dict(name="step_2d_forced", kind="step", nx=256, ny=1, nzloc=25, nsubd=12, prec="fp64", tune=False),
        # the start of a run or a restart of its multistep scheme: upload, solver tables, start-up steps
        dict(name="startup_96_mixed", kind="startup", nx=96, ny=96, nzloc=21, nsubd=6, prec="mixed"),
        # a parameter study: 12 runs of uneven sizes, four steps of each per call
        dict(name="ensemble_12_mixed", kind="ensemble", members=12, pick=2024, steps=4, prec="mixed"),
        # isolated Helmholtz solves (33024 columns of 8 x 25 points), FP64
        dict(name="helm_256_fp64", kind="helm", nx=256, ny=256, nzloc=25, nsubd=8, mode=0),
        # the same with FP32 factors and one FP64 residual sweep
        dict(name="helm_256_refined", kind="helm", nx=256, ny=256, nzloc=25, nsubd=8, mode=1),
        # a Fortran program's own penalty solve: one system of 12 x 25 points on host arrays
        dict(name="column_300", kind="column", nzloc=25, nsubd=12, bot=1, top=1),
        # a Fortran program's diagnostics on host fields
        dict(name="legacy_128", kind="legacy", nx=128, ny=128, nzloc=17, nsubd=4),
        # the statistics of a running simulation
        dict(name="diag_256_mixed", kind="diag", nx=256, ny=256, nzloc=25, nsubd=8, prec="mixed"),
    ]


def _smooth(lo, hi):
    out = []
    for n in range(lo, hi + 1, 2):
        m = n
        for r in (2, 3, 5):
            while m % r == 0:
                m //= r
        if m == 1:
            out.append(n)
    return out


def _log_pick(rng, values):
    x = math.exp(rng.uniform(math.log(values[0]), math.log(values[-1])))
    return min(values, key=lambda v: abs(math.log(v / x)))


def draw(rng):
    kind = rng.choices(["step", "startup", "ensemble", "helm", "column", "legacy", "diag"],
                       [10, 2, 2, 3, 1, 1, 1])[0]
    prec = rng.choice(["fp64", "mixed"])
    while kind == "ensemble":
        c = dict(kind=kind, members=rng.randint(2, 10), pick=rng.randrange(1, 10000), steps=rng.randint(2, 6),
                 prec=prec)
        if c["steps"] * sum(m.grid_points for m in _members(c)) <= (6e7 if prec == "mixed" else 3e7):
            return c
    nzloc, nsubd = rng.randint(9, 33), rng.randint(2, 12)
    if kind == "column":
        bc = rng.choice([(0, 0), (0, 1), (1, 1)])
        return dict(kind=kind, nzloc=nzloc, nsubd=nsubd, bot=bc[0], top=bc[1])
    if kind == "step" and rng.random() < 0.15:
        return dict(kind=kind, nx=_log_pick(rng, _smooth(32, 512)), ny=1, nzloc=rng.randint(11, 31), nsubd=12,
                    prec="fp64", tune=False)
    top = {"step": 512, "startup": 160, "helm": 320, "legacy": 192, "diag": 384}[kind]
    most = {"step": 3.0e7 if prec == "mixed" else 1.5e7, "startup": 1.5e6, "helm": 1.5e7, "legacy": 1.2e6,
            "diag": 1.5e7}[kind]
    while True:
        nx, ny = _log_pick(rng, _smooth(32, top)), _log_pick(rng, _smooth(16, top))
        if nx * ny * nzloc * nsubd <= most:
            break
        nzloc, nsubd = rng.randint(9, 33), rng.randint(2, 12)
    c = dict(kind=kind, nx=nx, ny=ny, nzloc=nzloc, nsubd=nsubd)
    if kind == "helm":
        c["mode"] = rng.choice([0, 0, 1])
    elif kind != "legacy":
        c["prec"] = prec
    if kind == "step":
        c["tune"] = rng.random() < 0.3
    return c


# ----------------------------------------------------------------------
# configurations and states
# ----------------------------------------------------------------------
def _config(c):
    prec = cf.IW_PREC_MIXED if c.get("prec") == "mixed" else cf.IW_PREC_FP64
    if c["kind"] == "step" and c["ny"] == 1:
        return cf.shipped_2d(nx=c["nx"], nzloc=c["nzloc"], nsubd=c["nsubd"], precision=prec)
    nz = c["nzloc"] * c["nsubd"]
    dt = 1e-3 if nz <= 100 else 5e-4 if nz <= 250 else 2.5e-4
    re_ = 1000.0 if nz <= 100 else 2000.0 if nz <= 250 else 5000.0
    nx, ny = c.get("nx", 16), c.get("ny", 16)
    return cf.Config(nx=nx, ny=ny, nzloc=c["nzloc"], nsubd=c["nsubd"], dt=dt, xnu=1 / re_, xkappa=1 / re_,
                     precision=prec).validate()


def _nodes(n):
    """Gauss-Legendre-Lobatto points of degree n - 1, ascending."""
    leg = np.polynomial.legendre.Legendre.basis(n - 1)
    x = leg.deriv().roots().real
    for _ in range(3):  # Newton steps on P'
        x = x - leg.deriv()(x) / leg.deriv(2)(x)
    x = np.concatenate([[-1.0], np.sort(x), [1.0]])
    return 0.5 * (x - x[::-1])


def _levels(cfg):
    x = _nodes(cfg.nzloc)
    return np.concatenate([z + 0.5 * h * (x + 1.0) for z, h in zip(cfg.z0, cfg.zh)])


def _physical(cfg, seed):
    """u, v, w, rho: a mode-1 internal wave along x, in 3-D a weaker oblique one, and seeded noise in the bottom
    fifth of the depth."""
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    f8 = dict(device="cuda", dtype=torch.float64)
    ampl = (0.05 if cfg.forcing == 0 else 0.002) * (0.9 + 0.2 * torch.rand(1, generator=gen, **f8))
    phase = 2 * math.pi * torch.rand(2, generator=gen, **f8)
    kx, ky, m = 2 * math.pi / cfg.xlen, 2 * math.pi / cfg.ylen, math.pi / cfg.zlen
    rc = cfg.rho0 * cfg.brunt ** 2 / cfg.grav
    z = torch.tensor(_levels(cfg), **f8)[:, None, None]
    x = kx * cfg.xlen / cfg.nx * torch.arange(cfg.nx, **f8)[None, None, :]
    y = ky * cfg.ylen / cfg.ny * torch.arange(cfg.ny, **f8)[None, :, None]
    waves = [(ampl, kx, 0.0, x + phase[0])]
    if cfg.ny > 1:
        waves.append((0.4 * ampl, kx, ky, x + y + phase[1]))
    low = (z < 0.2 * cfg.zlen).to(torch.float64)
    for q in range(4):
        f = torch.zeros((cfg.nz, cfg.ny, cfg.nx), **f8)
        for a, k, l, th in waves:
            k2 = k * k + l * l
            om = cfg.brunt * math.sqrt(k2 / (k2 + m * m))
            if q < 2:
                f -= a * (l if q else k) / k2 * m * torch.cos(m * z) * torch.sin(th)
            elif q == 2:
                f += a * torch.sin(m * z) * torch.cos(th)
            else:
                f -= a / om * rc * torch.sin(m * z) * torch.sin(th)
        if q < 3 and (q != 1 or cfg.ny > 1):
            f += (0.002 * ampl) * low * (2 * torch.rand(f.shape, generator=gen, **f8) - 1)
        yield f


def _spectral(cfg, seed):
    """The four fields as the library stores them, (nz, ny, nxpp) in its storage type."""
    store = torch.float32 if cfg.precision == cf.IW_PREC_MIXED else torch.float64
    for f in _physical(cfg, seed):
        yield torch.view_as_real(_forward(f)).reshape(cfg.nz, cfg.ny, cfg.nxpp).to(store)


class _Buffer:
    """A device field of a Solver as torch sees it; keeps the Solver alive."""

    def __init__(self, solver, f):
        c = solver.cfg
        self.solver = solver
        self.__cuda_array_interface__ = dict(
            shape=(c.nz, c.ny, c.nxpp), typestr="<f4" if c.precision == cf.IW_PREC_MIXED else "<f8",
            data=(solver.field_ptr(f), False), version=2)


def _solver(cfg, seed):
    s = iw.Solver(cfg)
    fields = [torch.as_tensor(_Buffer(s, f), device="cuda") for f in range(4)]
    for dst, src in zip(fields, _spectral(cfg, seed)):
        dst.copy_(src)
    torch.cuda.synchronize()  # the library works on streams of its own
    return s, fields


def _start_steps(cfg):
    return 22 if cfg.imaxcalc else 3  # the adaptive rule acts after 20 steps


def _members(c):
    prec = cf.IW_PREC_MIXED if c["prec"] == "mixed" else cf.IW_PREC_FP64
    return [m.replace(precision=prec) for m in cf.ensemble_members(c["members"], c["pick"])]


def _helm_lambda(c):
    kx = np.arange(c["nx"] // 2 + 1)
    ky = np.fft.fftfreq(c["ny"], 1.0 / c["ny"])
    return (kx[None, :] ** 2 + ky[:, None] ** 2).ravel() + 11.0 / (6 * 1e-3)


def _helm_rhs(c, seed):
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    return torch.randn((c["ny"] * (c["nx"] // 2 + 1), c["nzloc"] * c["nsubd"], 2), generator=gen, device="cuda",
                       dtype=torch.float64)


def _column(c, seed):
    rng = np.random.default_rng(int(seed))
    n = c["nzloc"] * c["nsubd"]
    eps = float(10.0 ** rng.uniform(-3, -1))
    bcs = tuple(rng.uniform(-0.5, 0.5, 4)) if c["bot"] else (0.0, 0.0, 0.0, 0.0)
    return eps, bcs, rng.standard_normal(n), rng.standard_normal(n)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "column":
        s = iw.Solver(_config(case))
        return dict(kind=kind, s=s, bc=(case["bot"], case["top"]), col=_column(case, seed))
    if kind == "helm":
        s = iw.Solver(_config(case))
        lam = torch.tensor(_helm_lambda(case), device="cuda")
        rhs = _helm_rhs(case, seed)
        return dict(kind=kind, s=s, lam=lam, rhs=rhs, out=torch.zeros_like(rhs), mode=case["mode"])
    if kind == "ensemble":
        runs = [_solver(cfg, seed * 101 + i) for i, cfg in enumerate(_members(case))]
        iw.ensemble_run([s for s, _ in runs], 3)
        return dict(kind=kind, runs=[s for s, _ in runs], out=[f for _, f in runs], steps=case["steps"])
    cfg = _config(case)
    if kind == "legacy":
        f = next(_spectral(cfg, seed)).cpu().numpy()
        return dict(kind=kind, s=iw.Solver(cfg), f=f)
    if kind == "startup":
        host = torch.empty((4, cfg.nz, cfg.ny, cfg.nxpp), dtype=torch.float64, pin_memory=True)
        for q, f in enumerate(_spectral(cfg, seed)):
            host[q].copy_(f)
        s = iw.Solver(cfg)
        fields = [torch.as_tensor(_Buffer(s, f), device="cuda") for f in range(4)]
        return dict(kind=kind, s=s, host=host, state=host.numpy(), out=fields)
    s, fields = _solver(cfg, seed)
    if kind == "diag":
        return dict(kind=kind, s=s, out=fields)
    s.step(_start_steps(cfg))
    if case["tune"]:
        s.autotune()
    return dict(kind=kind, s=s, out=fields)


def run(state):
    kind = state["kind"]
    if kind == "step":
        state["s"].step(1)
        return state["out"]
    if kind == "startup":
        state["s"].set_state(state["state"], t=0.0, istep=0)
        state["s"].step(4)
        return state["out"]
    if kind == "ensemble":
        iw.ensemble_run(state["runs"], state["steps"])
        return state["out"]
    if kind == "helm":
        rhs = state["rhs"]
        iw.helm_solve_batched(state["s"], state["lam"].data_ptr(), rhs.shape[0], 0, 1, rhs.data_ptr(),
                              state["out"].data_ptr(), state["mode"])
        return state["out"]
    if kind == "column":
        eps, bcs, rr, ri = state["col"]
        state["s"].penalty_setup(eps)
        return state["s"].penalty_main(eps, *state["bc"], bcs, rr, ri)
    if kind == "legacy":
        s, f = state["s"], state["f"]
        phys = s.horfft(f, 1)
        back = s.horfft(phys, -1)
        avg, count = s.interface_avg3d(f)
        return [phys, back, s.dpdz(f), s.filter_3dlegenfourier(f), avg, count]
    d = state["s"].diag()
    return dict(ke=d["ke"], eps=d["eps"], wrms=d["wrms_bottom"], cfl=list(d["cfl"]), minmax=list(d["minmax"]))


# ----------------------------------------------------------------------
# work: each input read once, each output written once
# ----------------------------------------------------------------------
def _fft_flops(cfg, transforms):
    """`transforms` real fields through x (half-length complex) and y."""
    m = cfg.nx // 2
    x = cfg.ny * cfg.nz * (5 * m * math.log2(m) + 8 * m)
    y = 0 if cfg.ny == 1 else cfg.nz * (m + 1) * 5 * cfg.ny * math.log2(cfg.ny)
    return transforms * (x + y)


def _step_work(cfg):
    # state: u, v, w, rho at n, n-1, n-2 and the nonlinear terms at n-1, n-2 read; three levels written.
    # operations: 12 inverse and 12 forward transforms, the products, D on 4 + 4 fields, the filter on 4, and the
    # block products of the solves (pressure: inverse and two D; u, v, w, rho: inverse) on real and imaginary parts
    item = 4 if cfg.precision == cf.IW_PREC_MIXED else 8
    n, N = cfg.ntot, cfg.nzloc
    flops = _fft_flops(cfg, 24) + 60.0 * n + 2.0 * N * n * (4 + 4 + 4 + 3 + 4)
    return 32.0 * n * item, flops


def work(case):
    kind = case["kind"]
    if kind == "column":
        n, N = case["nzloc"] * case["nsubd"], case["nzloc"]
        return dict(bytes=6.0 * 8 * n, flops=2.0 * n * N * 2 * N + 2 * 2.0 * n * 3 * N)
    if kind == "ensemble":
        each = [_step_work(m) for m in _members(case)]
        return dict(bytes=case["steps"] * sum(b for b, _ in each), flops=case["steps"] * sum(f for _, f in each))
    cfg = _config(case)
    n, N = cfg.ntot, cfg.nzloc
    if kind == "helm":
        ncol, sys = cfg.ncol, len(set(_helm_lambda(case).tolist()))
        # one band system of N sub- and super-diagonals per distinct lambda, right-hand sides in, solutions out
        return dict(bytes=32.0 * ncol * cfg.nz + 8.0 * sys * cfg.nz * 2 * N, flops=2.0 * 2 * N * cfg.nz * 2 * ncol)
    if kind == "legacy":
        return dict(bytes=8.0 * 8 * n, flops=_fft_flops(cfg, 2) + 2.0 * N * n * 2 + 10.0 * n)
    b, f = _step_work(cfg)
    if kind == "step":
        return dict(bytes=b, flops=f)
    if kind == "startup":
        return dict(bytes=4 * b + 4 * 8.0 * n, flops=4 * f)
    item = 4 if cfg.precision == cf.IW_PREC_MIXED else 8  # diag: 13 physical fields of 4 spectral ones
    return dict(bytes=4.0 * n * item, flops=_fft_flops(cfg, 13) + 2.0 * N * n * 3 + 40.0 * n)


# ----------------------------------------------------------------------
# exact results: the method in plain torch, 64 bits
# ----------------------------------------------------------------------
def _forward(f):
    """Physical (.., ny, nx) -> spectral (.., ny, nx/2+1); the x-Nyquist column is scaled, not transformed, in y."""
    s = torch.fft.rfft(f, dim=-1, norm="forward")
    nyq = s[..., -1:] / f.shape[-2]
    return torch.cat([torch.fft.fft(s[..., :-1], dim=-2, norm="forward"), nyq], dim=-1)


def _inverse(s, nx):
    """Spectral -> physical; the x-Nyquist column is taken as it is, real parts only at kx = 0 and Nyquist."""
    g = torch.cat([torch.fft.ifft(s[..., :-1], dim=-2, norm="forward"), s[..., -1:]], dim=-1)
    g[..., 0] = g[..., 0].real.to(g.dtype)
    g[..., -1] = g[..., -1].real.to(g.dtype)
    return torch.fft.irfft(g, n=nx, dim=-1, norm="forward")


def _project(s):
    """What an inverse and a forward transform leave of a spectral field."""
    out = s.clone()
    out[..., 0] = 0.5 * (s[..., 0] + torch.conj(torch.roll(torch.flip(s[..., 0], [-1]), 1, -1)))
    out[..., -1] = (s[..., -1].real / s.shape[-2]).to(s.dtype)
    return out


class _Exact:
    """The time step in 64 bits."""

    def __init__(self, cfg):
        dev, f8 = "cuda", torch.float64
        self.cfg, N = cfg, cfg.nzloc
        t = lambda a: torch.tensor(np.asarray(a), device=dev, dtype=f8)  # noqa: E731
        x, n = _nodes(N), N - 1
        leg = np.stack([np.polynomial.legendre.Legendre.basis(k)(x) for k in range(N)])  # [k, point]
        wg = 2.0 / (n * (n + 1) * leg[n] ** 2)
        dx = x[:, None] - x[None, :] + np.eye(N)
        c = np.prod(dx, axis=1)
        D = c[:, None] / (c[None, :] * dx) * (1 - np.eye(N))
        D -= np.diag(D.sum(1))
        D2 = 2 * (np.diag(D)[:, None] * D - D / dx) * (1 - np.eye(N))
        D2 -= np.diag(D2.sum(1))
        ck = np.arange(N) + 0.5
        ck[n] = 0.5 * n
        kc = int(cfg.fackc * n)
        th = np.clip((np.arange(N) - kc) / (n - kc), 0, None)
        sig = np.where(np.arange(N) >= kc, np.exp(-cfg.amp * th ** (2 * cfg.p)), 1.0)
        self.L = t((leg.T * (sig * ck)) @ (leg * wg))
        self.D, self.D2, self.h = t(D), t(D2), t(cfg.zh)
        self.kx = t(2 * math.pi / cfg.xlen * np.arange(cfg.nx // 2 + 1))[None, None, :]
        nyh = cfg.ny // 2
        j = np.arange(cfg.ny)
        self.ky = t(2 * math.pi / cfg.ylen * np.where(j < nyh, j, j - cfg.ny) * (cfg.ny > 1))[None, :, None]
        ak = torch.sqrt(self.kx ** 2 + self.ky ** 2)
        akmax = math.sqrt(float(self.kx.max()) ** 2 + float(self.ky.abs().max()) ** 2)
        self.cf = torch.exp(-cfg.amp * (ak / akmax) ** (2 * cfg.pf))
        self.k2, self.inv = torch.unique((self.kx ** 2 + self.ky ** 2).reshape(-1), return_inverse=True)
        z = _levels(cfg)
        self.z = t(z)[:, None, None]
        self.meang = 1.0 - torch.exp(-cfg.xbcrit * ((self.z - cfg.zcen) / cfg.xlen) ** 2)
        zf = np.concatenate([[z[0]], z.reshape(cfg.nsubd, N)[:, 1:].ravel()])
        dz = np.concatenate([[z[0] - z[-1]], np.diff(zf)])  # merged levels; the lowest is taken from the top
        g = (np.arange(cfg.nsubd)[:, None] * n + np.arange(N)[None, :]).ravel()
        self.dzinv = t(np.where(np.arange(cfg.nz) < cfg.nz - 1, 1.0 / dz[g], 0.0))[:, None, None]
        self.t, self.dt, self.istep = 0.0, cfg.dt, 0
        self.co = dict(f=(1.0, 0.0, 0.0), b=(1.0, 0.0, 0.0), v=1.0)
        self.cdt, self.changing, self.since = 1.0, False, 0
        kx1, m1 = 2 * math.pi / cfg.xlen, math.pi / cfg.zlen
        self.om = cfg.brunt * kx1 / math.sqrt(kx1 ** 2 + m1 ** 2)
        self.ready = {}

    def blocks(self, a):
        return a.reshape((self.cfg.nsubd, self.cfg.nzloc) + tuple(a.shape[1:]))

    def apply(self, op, a):
        b = self.blocks(a)
        return torch.einsum("ij,sj...->si...", op.to(a.dtype), b).reshape(a.shape)

    def dz(self, a):
        b = self.blocks(self.apply(self.D, a))
        return (b * (2.0 / self.h).reshape((-1,) + (1,) * (b.dim() - 1))).reshape(a.shape)

    def penalty(self, eps, bc, h):
        """(alpha, beta, tau) of one end of a subdomain of height h; bc 0 Dirichlet, 1 Neumann, 2 interface."""
        c, N = self.cfg, self.cfg.nzloc
        om = 2.0 / ((N + 1) * (N + 2))
        if bc == 0:
            return 1.0, 0.0, c.facdir * (2 / h) ** 2 * eps / om ** 2
        if bc == 1:
            return 0.0, 1.0, torch.full_like(eps, c.facneumn * 2 / h / om)
        fac = torch.where(1 / eps >= 1e5, c.facrobin, 1.0)
        return 1.0, 1.0, fac / (om * eps) * (eps + 2 * om - 2 * torch.sqrt(om ** 2 + eps * om)) * 2 / h

    def matrix(self, eps, bot, top):
        c, N, ns = self.cfg, self.cfg.nzloc, self.cfg.nsubd
        A = torch.zeros((eps.numel(), c.nz, c.nz), device="cuda", dtype=torch.float64)
        A += torch.eye(c.nz, device="cuda", dtype=torch.float64)
        e, t1b, t2t = eps[:, None], None, None
        for k in range(ns):
            m, h = k * N, c.zh[k]
            r = slice(m, m + N)
            A[:, r, r] -= eps[:, None, None] * (2 / h) ** 2 * self.D2
            a, b, tau = self.penalty(eps, bot if k == 0 else 2, h)
            A[:, m, m] += tau * a
            A[:, m, r] -= tau[:, None] * b * e * (2 / h) * self.D[0]
            if k == 0:
                t1b = tau
            else:
                A[:, m, m] -= 0.5 * tau * a
                A[:, m, r] += 0.5 * tau[:, None] * b * e * (2 / h) * self.D[0]
                A[:, m, m - 1] -= 0.5 * tau * a
                A[:, m, m - N:m] += 0.5 * tau[:, None] * b * e * (2 / c.zh[k - 1]) * self.D[N - 1]
            q = m + N - 1
            a, b, tau = self.penalty(eps, top if k == ns - 1 else 2, h)
            A[:, q, q] += tau * a
            A[:, q, r] += tau[:, None] * b * e * (2 / h) * self.D[N - 1]
            if k == ns - 1:
                t2t = tau
            else:
                A[:, q, q] -= 0.5 * tau * a
                A[:, q, r] -= 0.5 * tau[:, None] * b * e * (2 / h) * self.D[N - 1]
                A[:, q, q + 1] -= 0.5 * tau * a
                A[:, q, q + 1:q + 1 + N] -= 0.5 * tau[:, None] * b * e * (2 / c.zh[k + 1]) * self.D[0]
        return A, t1b, t2t

    def columns(self, eps, bot, top, rhs, wall=None):
        """Solves the system of every (kx, ky) for the fields rhs (each (nz, ny, nxh+1) complex); eps per distinct
        k^2.  Systems without a finite eps (k = 0 of the pressure) give 0.  wall: Neumann data, bottom and top."""
        c, out = self.cfg, [torch.zeros_like(r) for r in rhs]
        cols = [r.reshape(c.nz, -1) for r in rhs]
        order = torch.argsort(self.inv, stable=True)
        count = torch.bincount(self.inv, minlength=self.k2.numel())
        first = torch.cumsum(count, 0) - count
        most = int(count.max())
        step = max(1, int(2e9) // (8 * c.nz * c.nz))
        for s in range(0, self.k2.numel(), step):
            s1 = min(self.k2.numel(), s + step)
            ok = torch.isfinite(eps[s:s1])
            e = torch.where(ok, eps[s:s1], torch.ones_like(eps[s:s1]))
            A, t1, t2 = self.matrix(e, bot, top)
            slot = torch.arange(most, device="cuda")[None, :]
            col = order[torch.clamp(first[s:s1, None] + slot, max=order.numel() - 1)]  # (systems, slots)
            B = torch.cat([q[:, col.reshape(-1)].reshape(c.nz, s1 - s, most) for q in cols], -1).permute(1, 0, 2)
            B = B * e[:, None, None]
            if wall is not None:
                lo, hi = (w.reshape(-1)[col.reshape(-1)].reshape(s1 - s, most) for w in wall)
                B[:, 0] -= (t1 * e)[:, None] * lo
                B[:, -1] += (t2 * e)[:, None] * hi
            X = torch.linalg.solve(A, torch.cat([B.real, B.imag], -1))
            X = torch.complex(X[..., :B.shape[-1]], X[..., B.shape[-1]:]) * ok[:, None, None]
            live = slot < count[s:s1, None]
            for i, o in enumerate(out):
                o.reshape(c.nz, -1)[:, col[live]] = X[:, :, i * most:(i + 1) * most].permute(1, 0, 2)[:, live]
        return out

    def variable(self, d1, d2, d3):
        d12, d23, d123 = d1 + d2, d2 + d3, d1 + d2 + d3
        f = (1 + d1 * (2 * d1 + 6 * d2 + 3 * d3) / (6 * d2 * d23), -d1 * (2 * d1 + 3 * d2 + 3 * d3) / (6 * d2 * d3),
             d1 * (2 * d1 + 3 * d2) / (6 * d3 * d23))
        b = (1 + d1 / d2 + d1 / d123 + d1 ** 2 / (d123 * d2) + d1 ** 2 * d12 / (d123 * d23 * d2),
             -(d1 ** 2 / (d12 * d2) + d1 ** 2 / (d2 * d123) + d1 ** 2 * d12 / (d2 * d23 * d123)
               + d1 ** 2 * d12 / (d3 * d23 * d123)), d1 ** 2 * d12 / (d3 * d23 * d123))
        return f, b, 1 + d1 / d12 + d1 / d123

    def start(self, fields):
        c = self.cfg
        self.F = [torch.view_as_complex(f.double().reshape(c.nz, c.ny, -1, 2).contiguous()) for f in fields]
        zero = torch.zeros_like(self.F[0])
        self.Fn, self.Fnm, self.Sn, self.Snm = ([zero] * 4 for _ in range(4))

    def adapt(self):
        c = self.cfg
        if not int(self.t / self.dt) > 20:
            return
        u, w = (_inverse(self.F[q], c.nx) for q in (0, 2))
        cx = float(u.abs().max()) * self.dt * c.nx / c.xlen
        cz = float((w.abs() * self.dzinv).max()) * self.dt
        if not (cz > 0.7 or cz < 0.1 or cx > 0.16):
            return
        r = 1.25 if cz > 0.7 or cx > 0.16 else max(0.8, self.dt / (2 * math.pi / (50 * self.om)))
        self.dt, self.cdt = self.dt / r, r
        f, b, v = self.variable(self.dt, r * self.dt, r * self.dt)
        self.co, self.changing, self.since = dict(f=f, b=b, v=v), True, 0

    def step(self):
        c, D = self.cfg, self.dz
        self.istep += 1
        if c.imaxcalc:
            self.adapt()
        if self.changing:
            self.since += 1
        F1 = [_project(f) for f in self.F]
        F1[2][:, 0, 0] = 0
        inv = lambda a: _inverse(a, c.nx)  # noqa: E731
        u, v, w, r = (inv(f) for f in F1)
        rg = -c.rho0 * c.brunt ** 2 / c.grav
        Q, tau = [], 0.5 * (c.nzloc + 1) * (c.nzloc + 2) / 2
        N, ns = c.nzloc, c.nsubd
        for q, a in enumerate((u, v, w)):
            Q.append(-0.5 * (u * inv(1j * self.kx * F1[q]) + v * inv(1j * self.ky * F1[q]) + w * inv(D(F1[q]))))
        Q[2] += c.brunt ** 2 / rg * r
        Q.append(-w * rg)
        lo, hi = [k * N for k in range(1, ns)], [k * N - 1 for k in range(1, ns)]
        tl = (tau * 2.0 / self.h)[:, None, None]
        if ns > 1:
            for q, a in enumerate((u, v, w, r)):  # upwind interface penalty
                Q[q][lo] -= tl[1:] * torch.clamp(w[lo], min=0) * (a[lo] - a[hi])
                Q[q][hi] -= tl[:-1] * torch.clamp(-w[hi], min=0) * (a[hi] - a[lo])
        if c.forcing:
            xk, xm = 2 * math.pi / c.xlen, math.pi / c.zlen
            om = c.brunt * xk / math.sqrt(xk * xk + xm * xm)
            on = 1.0 if self.t <= c.fwave * 2 * math.pi / om else 0.0
            a = c.xacrit * c.umax * c.umax / c.xlen * on
            th = xk * c.xlen / c.nx * torch.arange(c.nx, device="cuda", dtype=torch.float64) - om * self.t
            cz, sz = torch.cos(xm * self.z), torch.sin(xm * self.z)
            lev = torch.ones_like(self.z)
            if c.forcing == cf.IW_PADDLE_ABOVE_BOTTOM:
                lev[0] = 0
            Q[0] += lev * (-a * xm / xk) * cz * torch.sin(th)
            Q[2] += lev * a * sz * torch.cos(th)
            Q[3] += lev * (-a / om * c.brunt ** 2 * c.rho0 / c.grav) * sz * torch.sin(th)
        S = []
        for q, a in enumerate((u, v, w, r)):
            h = -0.5 if q < 3 else -1.0
            S.append(_forward(Q[q]) + 1j * self.kx * _forward(h * u * a) + 1j * self.ky * _forward(h * v * a)
                     + D(_forward(h * w * a)))
        f, b, dt = self.co["f"], self.co["b"], self.dt
        rot = [((self.kx ** 2 + self.ky ** 2) * lw[2] + 1j * self.kx * D(lw[0]) + 1j * self.ky * D(lw[1]))[[0, -1]]
               for lw in ([_project(x) for x in F1[:3]], self.Fn[:3], self.Fnm[:3])]
        wall = [f[0] * S[2][k] + f[1] * self.Sn[2][k] + f[2] * self.Snm[2][k]
                - c.xnu * (f[0] * rot[0][i] + f[1] * rot[1][i] + f[2] * rot[2][i]) for i, k in enumerate((0, -1))]
        F2 = [_project(x) for x in F1]
        new = []
        for q in range(4):
            g = dt * (f[0] * S[q] + f[1] * self.Sn[q] + f[2] * self.Snm[q]) + b[0] * F2[q] + b[1] * self.Fn[q] \
                + b[2] * self.Fnm[q]
            new.append(self.cf * self.apply(self.L, g) if c.ispecfilternl == 1 else g)
        self.Snm, self.Sn, self.Fnm, self.Fn = self.Sn, S, self.Fn, F2
        if self.istep < 2:
            self.co["f"], self.co["b"] = (2.0, -1.0, 0.0), (2.0, -0.5, 0.0)
        elif self.changing and self.since < 2:
            self.co["f"], self.co["b"], _ = self.variable(dt, dt, self.cdt * dt)
        else:
            self.co["f"], self.co["b"] = (3.0, -3.0, 1.0), (3.0, -1.5, 1 / 3)
        # pressure and projection
        U, V, W, R = new
        div = (1j * self.kx * U + 1j * self.ky * V + D(W)) / dt
        phi = self.apply(self.L, self.columns(1 / self.k2, 1, 1, [-div], wall)[0])
        U, V = U - dt * 1j * self.kx * phi, V - dt * 1j * self.ky * phi
        W = W - dt * D(phi)
        W[:, 0, 0] = 0
        noslip = c.bc_variant == cf.IW_BC_NOSLIP
        if noslip:
            U[0], V[0], W[0] = 0, 0, 0
        # Helmholtz solves
        nu, ka, bv = c.xnu * dt, c.xkappa * dt, self.co["v"]
        eu, et = 1 / (self.k2 + bv / nu), 1 / (self.k2 + bv / ka)
        U, V = self.columns(eu, 0 if noslip else 1, 1, [U / nu, V / nu])
        W = self.columns(torch.where(self.k2 == 0, float("inf"), eu), 0, 0, [W / nu])[0]
        R = self.columns(et, 1, 1, [R / ka])[0]
        self.F = [self.apply(self.L, x) for x in (U, V, W, R)]
        if c.meanu_damping:
            self.F[0][:, 0, 0] *= self.meang[:, 0, 0]
        if self.istep < 2:
            self.co["v"] = 1.5
        elif self.changing and self.since < 2:
            self.co["v"] = self.variable(dt, dt, self.cdt * dt)[2]
            self.cdt, self.changing = 1.0, False
        else:
            self.co["v"] = 11 / 6
        self.t += dt
        self.F = [self.average(x)[0] for x in self.F]

    def average(self, s):
        """Adaptive interface averaging; the averaged field and the number of averaged points."""
        c, out = self.cfg, _project(s)
        if c.nsubd < 2:
            return out, 0
        i = torch.arange(1, c.nsubd, device="cuda") * c.nzloc
        ph = _inverse(s[torch.stack([i - 2, i - 1, i, i + 1])], c.nx)
        hit = (ph[2] - ph[1]).abs() / (ph[2] + ph[1]).abs() > 0.005
        mid = 0.5 * (ph[0] + ph[3])
        out[i - 1] += _forward(torch.where(hit, mid - ph[1], 0.0))
        out[i] += _forward(torch.where(hit, mid - ph[2], 0.0))
        return out, int(hit.sum())

    def fields(self):
        c = self.cfg
        return [torch.view_as_real(f.contiguous()).reshape(c.nz, c.ny, c.nxpp) for f in self.F]


def _too_long(cfg, steps):
    """Whether the dense solves, the bulk of exact(), would take over about 20 seconds."""
    kx = (np.arange(cfg.nx // 2 + 1) / cfg.xlen) ** 2
    ky = (np.arange(cfg.ny // 2 + 1) / cfg.ylen) ** 2 if cfg.ny > 1 else np.zeros(1)
    systems = np.unique((kx[None, :] + ky[:, None]).round(12)).size
    return 4 * steps * systems * cfg.nz ** 3 > 1e12


def exact(case, seed):
    kind = case["kind"]
    if kind == "ensemble":
        cfgs, steps = _members(case), 3 + case["steps"]
        if len(cfgs) > 4 or any(_too_long(m, len(cfgs) * steps) for m in cfgs):
            return None
        out = []
        for i, cfg in enumerate(cfgs):
            m = _Exact(cfg)
            m.start(list(_spectral(cfg, seed * 101 + i)))
            for _ in range(steps):
                m.step()
            out.append(m.fields())
        return out
    cfg = _config(case)
    if kind == "column":
        m, (eps, bcs, rr, ri) = _Exact(cfg), _column(case, seed)
        e = torch.tensor([eps], device="cuda", dtype=torch.float64)
        A, t1, t2 = m.matrix(e, case["bot"], case["top"])
        B = -eps * torch.tensor(np.stack([rr, ri], -1), device="cuda")
        scaled = B.T.cpu().numpy().copy()
        b = B.clone()
        lo, hi = (torch.tensor(bcs[k:k + 2], device="cuda", dtype=torch.float64) for k in (0, 2))
        b[0] += t1 * lo if case["bot"] == 0 else -t1 * eps * lo
        b[-1] += t2 * hi if case["top"] == 0 else t2 * eps * hi
        x = torch.linalg.solve(A[0], b).T.cpu().numpy()
        return x[0], x[1], scaled[0], scaled[1]
    if kind == "helm":
        m, rhs = _Exact(cfg), _helm_rhs(case, seed)
        lam, inv = np.unique(_helm_lambda(case), return_inverse=True)
        if lam.size * cfg.nz ** 3 > 1e12:
            return None
        out, order = torch.empty_like(rhs), np.argsort(inv, kind="stable")
        first = np.searchsorted(inv[order], np.arange(lam.size + 1))
        most, step = int(np.diff(first).max()), max(1, int(2e9) // (8 * cfg.nz ** 2))
        for s in range(0, lam.size, step):
            s1 = min(lam.size, s + step)
            e = torch.tensor(1.0 / lam[s:s1], device="cuda")
            col = order[np.minimum(first[s:s1, None] + np.arange(most), order.size - 1)]
            live = torch.tensor(np.arange(most) < np.diff(first)[s:s1, None], device="cuda")
            col = torch.tensor(col, device="cuda")
            B = rhs[col].permute(0, 2, 1, 3).reshape(s1 - s, cfg.nz, most * 2)
            X = torch.linalg.solve(m.matrix(e, 0, 1)[0], B).reshape(s1 - s, cfg.nz, most, 2).permute(0, 2, 1, 3)
            out[col[live]] = X[live]
        return out
    if kind == "legacy":
        m = _Exact(cfg)
        m.start([next(_spectral(cfg, seed))])
        f, real = m.F[0], lambda a: torch.view_as_real(a.contiguous()).reshape(cfg.nz, cfg.ny, cfg.nxpp).cpu().numpy()
        phys = _inverse(f, cfg.nx)
        padded = torch.nn.functional.pad(phys, (0, 2)).cpu().numpy()
        avg, _ = m.average(f)
        return [padded, real(_forward(phys)), real(m.dz(f)), real(m.cf * m.apply(m.L, f)), real(avg), None]
    if kind == "diag":
        return _exact_diag(cfg, seed)
    steps = 4 if kind == "startup" else _start_steps(cfg) + 1
    if _too_long(cfg, steps):
        return None
    m = _Exact(cfg)
    m.start(list(_spectral(cfg, seed)))
    for _ in range(steps):
        m.step()
    return m.fields()


def _exact_diag(cfg, seed):
    m = _Exact(cfg)
    m.start(list(_spectral(cfg, seed)))
    ke = eps = 0.0
    cfl, ext = [], []
    rg = -cfg.rho0 * cfg.brunt ** 2 / cfg.grav
    scale = [cfg.dt * cfg.nx / cfg.xlen, cfg.dt * cfg.ny / cfg.ylen, cfg.dt * m.dzinv]
    for q, f in enumerate(m.F):
        p = _inverse(f, cfg.nx)
        if q < 3:
            ke += 0.5 * float((p[1:] ** 2).sum())
            for d in (1j * m.kx * f, 1j * m.ky * f, m.dz(f)):
                eps += cfg.xnu * float((_inverse(d, cfg.nx)[1:] ** 2).sum())
            cfl.append(max(0.0, float((p.abs() * scale[q]).max())))
        if q == 2:
            low = p[(m.z < 0.2 * cfg.zlen).reshape(-1)]
            wrms = float((low ** 2).mean().sqrt())
        if q == 3:
            p = p + 1.0 + rg * m.z
        ext += [min(float(p.min()), 1.0 if q == 3 else 0.0), max(float(p.max()), 0.0)]
    return dict(ke=ke, eps=eps, wrms=wrms, cfl=cfl, minmax=ext)
