"""y tiles of 2 and 4 columns (a warp per column; power-of-two lengths have kernels of their own) against the
tile taken by size, through whole steps: every transform direction, with and without the i ky fold, at lengths
around the values per lane of the kernels (ny <= 128, 256, 512, 1024)."""
import numpy as np
import pytest

from iwrepo_b200 import config as cf

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [cf.IW_PREC_FP64, cf.IW_PREC_MIXED])
@pytest.mark.parametrize("ny", [2, 6, 16, 64, 90, 128, 144, 256, 300, 512, 540, 1000, 1024])
def test_narrow_tiles(ny, precision):
    import iwrepo_b200 as iw
    cfg = cf.Config(nx=12, ny=ny, nzloc=5, nsubd=2, dt=1e-3, precision=precision).validate()
    runs = []
    for tile in (0, 4, 2):
        s = iw.Solver(cfg)
        s.set_launch("y_tile", tile)
        s.init_mode1(0.02, 1e-3, 5)
        s.step(3)
        runs.append(s.state())
        s.close()
    # rounding of the passes, 1e-16 or 6e-8 each, in three steps and relative to the largest velocity (v is noise)
    tol = 1e-13 if precision == cf.IW_PREC_FP64 else 1e-5
    big = max(np.linalg.norm(runs[0][q]) for q in range(3))
    for r in runs[1:]:
        for q in range(4):
            assert np.linalg.norm(r[q] - runs[0][q]) <= tol * (big if q < 3 else np.linalg.norm(runs[0][3])), q
