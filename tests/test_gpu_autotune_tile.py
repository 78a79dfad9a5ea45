"""iw_autotune times the y tile that an untuned run takes among its candidates and keeps it where the
narrower ones are slower: by a third and more at these sizes (16 columns for ny <= 128, which the choice 8
stands for; at ny = 512 in FP64 two transforms fit in shared memory with 4 columns, one with 8)."""
import numpy as np
import pytest

from iwrepo_b200 import config as cf

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,precision", [(64, 64, cf.IW_PREC_FP64), (64, 64, cf.IW_PREC_MIXED), (192, 120, cf.IW_PREC_FP64),
                                             (192, 120, cf.IW_PREC_MIXED), (256, 128, cf.IW_PREC_FP64),
                                             (256, 128, cf.IW_PREC_MIXED), (128, 512, cf.IW_PREC_FP64)])
def test_tuned_run_keeps_the_wide_tile(nx, ny, precision):
    import iwrepo_b200 as iw
    cfg = cf.Config(nx=nx, ny=ny, nzloc=17, nsubd=4, dt=5e-4, precision=precision).validate()
    s = iw.Solver(cfg)
    s.init_mode1(0.05, 1e-4, 3)
    s.step(3)
    assert s.autotune()["y_tile"] == 8
    assert s.get_launch("y_tile") == 8
    s.close()


@pytest.mark.parametrize("ny", [1, 2, 48, 1000])
def test_tuned_run_keeps_its_results(ny):
    """One row, fewer rows than a tile has columns, a mixed length and one whose tiles are all narrow."""
    import iwrepo_b200 as iw
    cfg = cf.Config(nx=16, ny=ny, nzloc=9, nsubd=2, dt=1e-3).validate()
    runs = []
    for tune in (False, True):
        s = iw.Solver(cfg)
        s.init_mode1(0.02, 1e-4, 3)
        s.step(2)
        if tune:
            s.autotune()
        s.step(2)
        runs.append(s.state())
        s.close()
    for q in range(4):  # tiles of another width transform with other radices: rounding of FP64, 1e-16 per pass and step
        n = max(np.linalg.norm(runs[0][0]), np.linalg.norm(runs[0][q]))
        assert np.linalg.norm(runs[0][q] - runs[1][q]) <= 1e-13 * n
