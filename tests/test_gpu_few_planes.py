"""y transforms of FP32 columns of 16 and 32 rows: narrow tiles where there are fewer wide ones than SMs, wide ones above.
Steps and the budget (transforms of one field) have the same bits with the tile chosen by size as with 4 columns."""
import numpy as np
import pytest

from iwrepo_b200 import config as cf

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ny", [16, 32])
@pytest.mark.parametrize("nx,nzloc,nsubd", [(12, 5, 1), (32, 9, 2), (60, 9, 8), (60, 15, 10), (64, 17, 3)])
def test_few_planes(nx, ny, nzloc, nsubd):
    import iwrepo_b200 as iw
    cfg = cf.Config(nx=nx, ny=ny, nzloc=nzloc, nsubd=nsubd, dt=1e-3, precision=cf.IW_PREC_MIXED).validate()
    runs = []
    for tile in (0, 4):
        with iw.Solver(cfg) as s:
            s.set_launch("y_tile", tile)
            s.init_mode1(0.02, 1e-3, 9)
            s.step(3)
            runs.append([s.state(level) for level in range(5)] + list(s.postp()))
    assert all(np.array_equal(a, b) for a, b in zip(*runs))
