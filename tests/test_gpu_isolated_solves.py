"""The isolated penalty solves at the edges of their kernels.

* iw_helm_solve_batched, mode 0: block inverses on the tensor cores with one
  FP64 residual sweep for systems of moderate condition, band LU for the others
  (small lambda) and for arrays that are only 8-byte aligned.  The penalty rows
  are far larger than the others, so the measure is the normwise backward error
  |b - A x| / (|A| |x| + |b|) (maximum norms): sums of at most 3 N + 1 terms, each
  term of relative error eps = 1.1e-16, give (3 N + 1) eps; twice that for the two
  triangular sweeps, and a factor 4 for pivot growth: 8 (3 N + 1) eps.
* mode 1: FP32 sweeps with a right-hand side per lane must give the same bits as
  the warp-per-column kernel, which runs when solutions replace right-hand sides.
* penalty_main_: the band LU in shared memory equals the oracle's SGBTF2 bit
  for bit for subdomain sizes around the warp and the CTA.
* the tables follow a change of dt: a run whose dt changes there and back
  equals one that keeps it, bit for bit, from a re-uploaded state.
"""
import numpy as np
import pytest

from iwrepo_b200 import config as cf

pytestmark = pytest.mark.gpu


def _backward_error(o, lam, sol, rhs, cols, bot, top):
    worst = 0.0
    for c in cols:
        A = o.penalty_matrix(1.0 / lam[c], bot, top)
        for p in (0, 1):
            x, b = sol[c, :, p], rhs[c, :, p]
            den = np.abs(A).sum(1).max() * np.abs(x).max() + np.abs(b).max()
            worst = max(worst, np.abs(b - A @ x).max() / den)
    return worst


@pytest.mark.parametrize("nzloc,nsubd", [(3, 4), (8, 1), (9, 3), (16, 2), (17, 16), (25, 8), (33, 3), (40, 2), (44, 2)])
def test_batched_solves(nzloc, nsubd):
    import torch
    import iwrepo_b200 as iw
    from oracle import Oracle
    cfg = cf.Config(nx=16, ny=12, nzloc=nzloc, nsubd=nsubd, dt=1e-3).validate()
    s, o = iw.Solver(cfg), Oracle(cfg)
    rng = np.random.default_rng(nzloc)
    # 1 to 9 columns per lambda, one system far above the condition bound of the block inverses
    lam = np.repeat(1.0e4 * (1 + np.arange(9.0)), np.arange(1, 10))
    lam[-1] = 1.0e-2
    rng.shuffle(lam)
    ncol, n = lam.size, cfg.nz
    rhs = rng.standard_normal((ncol, n, 2))
    dl = torch.tensor(lam, device="cuda")
    cols = list(range(0, ncol, 7)) + [int(np.argmin(lam))]
    for mode in (0, 1):
        dr = torch.tensor(rhs, device="cuda")
        ds = torch.zeros_like(dr)
        iw.helm_solve_batched(s, dl.data_ptr(), ncol, 0, 1, dr.data_ptr(), ds.data_ptr(), mode)
        torch.cuda.synchronize()
        sol = ds.cpu().numpy()
        if mode == 0:
            assert _backward_error(o, lam, sol, rhs, cols, 0, 1) <= 8 * (3 * nzloc + 1) * 1.1e-16
            # 8-byte aligned arrays
            br, bs = (torch.zeros(ncol * n * 2 + 1, dtype=torch.float64, device="cuda") for _ in range(2))
            br[1:] = dr.reshape(-1)
            iw.helm_solve_batched(s, dl.data_ptr(), ncol, 0, 1, br.data_ptr() + 8, bs.data_ptr() + 8, 0)
            torch.cuda.synchronize()
            other = bs[1:].cpu().numpy().reshape(sol.shape)
            assert _backward_error(o, lam, other, rhs, cols, 0, 1) <= 8 * (3 * nzloc + 1) * 1.1e-16
        else:
            iw.helm_solve_batched(s, dl.data_ptr(), ncol, 0, 1, dr.data_ptr(), dr.data_ptr(), 1)
            torch.cuda.synchronize()
            assert np.array_equal(dr.cpu().numpy(), sol)
    s.close()


@pytest.mark.parametrize("nzloc,nsubd", [(3, 1), (3, 5), (4, 12), (16, 3), (17, 2), (32, 1), (33, 9), (48, 3)])
def test_band_lu_bit_identical(nzloc, nsubd):
    import iwrepo_b200 as iw
    from oracle import Oracle
    cfg = cf.Config(nx=16, ny=8, nzloc=nzloc, nsubd=nsubd, dt=1e-3).validate()
    s, o = iw.Solver(cfg), Oracle(cfg)
    rng = np.random.default_rng(nsubd)
    r1, r2 = rng.standard_normal(cfg.nz), rng.standard_normal(cfg.nz)
    for eps, bot, top in ((1e-2, 0, 1), (2e-5, 1, 1)):
        s.penalty_setup(eps)
        o.penalty_setup(eps)
        a = s.penalty_main(eps, bot, top, (0.1, 0.2, -0.3, 0.4), r1, r2)
        b = o.penalty_main(eps, bot, top, (0.1, 0.2, -0.3, 0.4), r1, r2)
        for x, y in zip(a, b):
            assert np.array_equal(x, y)
    s.close()


@pytest.mark.parametrize("solver", [cf.IW_SOLVE_AUTO, cf.IW_SOLVE_LU])
def test_tables_follow_a_change_of_dt(solver):
    import iwrepo_b200 as iw
    cfg = cf.Config(nx=16, ny=12, nzloc=9, nsubd=3, dt=1e-3, solver=solver).validate()
    third = dict(fac=(3.0, -3.0, 1.0), bdf=(3.0, -1.5, 1 / 3), bdfv=11 / 6)
    a, b = iw.Solver(cfg), iw.Solver(cfg)
    a.init_mode1(0.05, 1e-3, 3)
    a.step(4)
    levels = [a.state(lev) for lev in range(5)]
    b.set_state(*levels, t=0.0, istep=4)
    b.step_coefs(dt=2.0, **third)   # few refined tasks become many, and back
    b.step_coefs(dt=5e-4, **third)
    b.set_state(*levels, t=0.0, istep=4)
    for s in (a, b):
        s.step_coefs(dt=1e-3, **third)
    assert all(np.array_equal(a.state(lev), b.state(lev)) for lev in range(5))
    a.close()
    b.close()
