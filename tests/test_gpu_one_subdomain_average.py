"""interface_avg3d_ with one subdomain has no interface: the field comes back as one round trip through physical
space leaves it.  Lengths of one and of several blocks of rows."""
import numpy as np
import pytest

from iwrepo_b200 import config as cf
from oracle import Oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [cf.IW_PREC_FP64, cf.IW_PREC_MIXED])
@pytest.mark.parametrize("nx,ny,nzloc", [(12, 8, 5), (16, 1, 9), (8, 300, 5)])
def test_one_subdomain_average(nx, ny, nzloc, precision):
    import iwrepo_b200 as iw
    cfg = cf.Config(nx=nx, ny=ny, nzloc=nzloc, nsubd=1, dt=1e-3, precision=precision).validate()
    f = np.random.default_rng(3).standard_normal((cfg.nz, cfg.ny, cfg.nxpp))
    want, _ = Oracle(cfg).interface_avg3d(f)
    with iw.Solver(cfg) as s:
        got, count = s.interface_avg3d(f)
    assert count == 0
    # two FFT passes of at most 12 doublings in the oracle: 24 roundings of 1.1e-16, four operations each
    assert np.linalg.norm(got - want) <= 1e-14 * np.linalg.norm(want)
