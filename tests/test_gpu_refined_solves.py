"""iw_helm_solve_batched, mode 1: few columns take the kernel with a warp per column, many the one with a
lane per right-hand side; a column's solution has the same bits on either side of the line, and at the
first call with some columns as at later ones."""
import numpy as np
import pytest

from iwrepo_b200 import config as cf

pytestmark = pytest.mark.gpu


def _solve(s, lam, rhs, mode):
    import torch
    import iwrepo_b200 as iw
    sol = torch.zeros_like(rhs)
    torch.cuda.synchronize()
    iw.helm_solve_batched(s, lam.data_ptr(), lam.numel(), 0, 1, rhs.data_ptr(), sol.data_ptr(), mode)
    torch.cuda.synchronize()
    return sol


# per-SM waves of 8 columns (4 where the vectors fill shared memory); nzloc around the prefetching variants
@pytest.mark.parametrize("nzloc,nsubd", [(5, 2), (9, 3), (17, 2), (25, 3), (33, 2), (34, 2), (40, 2), (47, 1), (33, 20)])
def test_same_bits_for_few_and_many_columns(nzloc, nsubd):
    import torch
    import iwrepo_b200 as iw
    s = iw.Solver(cf.Config(nx=16, ny=8, nzloc=nzloc, nsubd=nsubd, dt=1e-3).validate())
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    wave = (4 if nzloc * nsubd > 597 else 8) * sms
    line = wave * (1 if nzloc <= 33 else 3)
    gen = torch.Generator(device="cuda").manual_seed(nzloc)
    ncol = line + 5
    lam = torch.tensor(np.resize(np.geomspace(0.5, 4.0e4, 37), ncol), device="cuda")
    rhs = torch.randn((ncol, nzloc * nsubd, 2), generator=gen, device="cuda", dtype=torch.float64)
    many = _solve(s, lam, rhs, 1)
    assert torch.isfinite(many).all()
    assert torch.equal(_solve(s, lam, rhs, 1), many)
    for k in (1, 16, 17, line):
        assert torch.equal(_solve(s, lam[:k], rhs[:k].contiguous(), 1), many[:k]), k
    s.close()


@pytest.mark.parametrize("nzloc,nsubd", [(9, 3), (25, 4), (44, 2)])
@pytest.mark.parametrize("low", [0, 3, 12])
def test_tables_made_by_need(nzloc, nsubd, low):
    """The tables are made by the first call that needs them.  Whatever the order of the modes and of aligned and
    only 8-byte aligned arrays, and with none, some or all of the 12 lambdas below the condition bound (the band LU then
    factors only those in mode 0), every call has the bits that it has on a handle of its own."""
    import torch
    import iwrepo_b200 as iw
    cfg = cf.Config(nx=16, ny=8, nzloc=nzloc, nsubd=nsubd, dt=1e-3).validate()
    gen = torch.Generator(device="cuda").manual_seed(7 * nzloc + low)
    base = np.concatenate([np.geomspace(1e-3, 0.1, low), np.geomspace(1.0e5, 4.0e5, 12 - low)])
    lam = torch.tensor(np.resize(base, 40), device="cuda")
    rhs = torch.randn((40, cfg.nz, 2), generator=gen, device="cuda", dtype=torch.float64)
    odd = torch.zeros(rhs.numel() + 1, device="cuda", dtype=torch.float64)
    odd[1:] = rhs.reshape(-1)

    def call(s, what):
        if what != "odd":
            return _solve(s, lam, rhs, what)
        sol = torch.zeros_like(odd)
        torch.cuda.synchronize()
        iw.helm_solve_batched(s, lam.data_ptr(), 40, 0, 1, odd.data_ptr() + 8, sol.data_ptr() + 8, 0)
        torch.cuda.synchronize()
        return sol[1:].reshape(rhs.shape)

    want = {}
    for what in (0, 1, "odd"):
        s = iw.Solver(cfg)
        want[what] = call(s, what)
        s.close()
    for order in ((0, 1, "odd", 0), (1, 0, "odd", 1), ("odd", 0, 1, 0), (0, "odd", 1, 1)):
        s = iw.Solver(cfg)
        for what in order:
            assert torch.equal(call(s, what), want[what]), (order, what)
        s.close()


def test_failed_allocation_of_the_tables():
    """A refused allocation is reported, writes no solution, and the next call is a complete one."""
    import torch
    import iwrepo_b200 as iw
    from iwrepo_b200 import IwError, _lib
    cfg = cf.Config(nx=16, ny=8, nzloc=9, nsubd=3, dt=1e-3).validate()
    lam = torch.tensor(np.resize(np.concatenate([[1e-3], np.geomspace(1.0e5, 4.0e5, 11)]), 40), device="cuda")
    rhs = torch.ones((40, cfg.nz, 2), device="cuda", dtype=torch.float64)
    for mode in (0, 1):
        s = iw.Solver(cfg)
        want = _solve(s, lam, rhs, mode)
        s.close()
        failed = 0
        for nth in range(1, 20):
            s = iw.Solver(cfg)
            _lib.check(_lib.lib().iw_fail_allocation(s.h, nth))
            try:
                assert torch.equal(_solve(s, lam, rhs, mode), want)
                done = True
            except IwError as e:
                assert e.code == 6
                done, failed = False, failed + 1
            _lib.check(_lib.lib().iw_fail_allocation(s.h, 0))
            assert torch.equal(_solve(s, lam, rhs, mode), want)
            s.close()
            if done:
                break
        assert done and failed >= 2
