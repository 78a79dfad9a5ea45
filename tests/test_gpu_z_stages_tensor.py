"""The tensor-core z stages (k_stageA_t, k_stageE_t) and the whole-column hand-over
from stage E to the solves, at the edges of their tiles, against the tiled
kernels and the strided solves.

FP64: stage A and stage E form the same FMA chains with D as the tiled stage A,
so only stage E's contraction of the products differs (1e-11 of the field after
3 steps, as between the older stage-E variants).  Mixed: the products are
rounded once instead of after every term, a difference of FP32 rounding (1e-5).
Row counts around the tiles of 8; planes that are no multiple of 8 points, and
FP32 planes whose rows do not start on 16 bytes (ny = 1).
"""
import numpy as np
import pytest

from iwrepo_b200 import config as cf

pytestmark = pytest.mark.gpu

SHAPES = [(16, 12, 3, 2), (18, 6, 8, 3), (20, 10, 9, 1), (16, 16, 16, 2), (30, 12, 17, 4), (16, 8, 25, 3), (24, 18, 33, 2),
          (16, 8, 39, 2), (16, 8, 40, 2), (30, 1, 21, 3), (32, 1, 12, 2)]


@pytest.mark.parametrize("precision", [cf.IW_PREC_FP64, cf.IW_PREC_MIXED])
@pytest.mark.parametrize("nx,ny,nzloc,nsubd", SHAPES)
def test_tensor_core_z_stages(nx, ny, nzloc, nsubd, precision):
    import iwrepo_b200 as iw
    cfg = cf.Config(nx=nx, ny=ny, nzloc=nzloc, nsubd=nsubd, dt=1e-3, precision=precision).validate()
    runs = []
    for old in (False, True):
        s = iw.Solver(cfg)
        if old:
            s.set_launch("stage_a", 0)
            s.set_launch("stage_e", 0)
            s.set_launch("solve", 1)
        s.init_mode1(0.05, 1e-3, 19)
        s.step(3)
        runs.append([s.state(lev) for lev in range(5)])
        s.close()
    tol = 1e-11 if precision == cf.IW_PREC_FP64 else 1e-5
    for a, b in zip(*runs):
        scale = max(np.linalg.norm(b[q]) for q in (0, 2)) if ny == 1 else 0.0
        for q in range(4):
            n = max(np.linalg.norm(b[q]), 1e-3 * scale)
            assert np.linalg.norm(a[q] - b[q]) <= tol * (n if n > 0 else 1.0), q
