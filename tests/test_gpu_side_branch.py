"""A step runs its wall term and its refined pressure columns beside the other kernels; while the phases
are timed everything runs on one stream.  The kernels and their inputs are the same, so the bits are."""
import numpy as np
import pytest

from iwrepo_b200 import config as cf

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [cf.IW_PREC_FP64, cf.IW_PREC_MIXED])
@pytest.mark.parametrize("nx,ny,nzloc,nsubd", [(16, 8, 9, 3), (64, 64, 17, 4), (96, 30, 21, 6), (64, 1, 12, 3)])
def test_side_branch_gives_the_same_bits(nx, ny, nzloc, nsubd, precision):
    import iwrepo_b200 as iw
    cfg = cf.Config(nx=nx, ny=ny, nzloc=nzloc, nsubd=nsubd, dt=1e-3, precision=precision).validate()
    runs = []
    for timed in (False, True):
        s = iw.Solver(cfg)
        s.init_mode1(0.05, 1e-3, 23)
        s.profile(timed)
        for _ in range(6):
            s.step(1)
        s.profile(False)
        runs.append([s.state(lev) for lev in range(5)])
        s.close()
    for a, b in zip(*runs):
        assert all(np.array_equal(a[q], b[q]) for q in range(4))
