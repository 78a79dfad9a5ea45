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
