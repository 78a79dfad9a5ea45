"""The tensor-core solves (k_solve_tc, k_press_tc) at the edges of their tiles.

They form every sum as the FMA chain of the FP64-pipe kernels (the matrix
instruction adds its products one after the other), so a run on variant 2 must
equal the run on variant 1 bit for bit: row counts around the tiles of 8 and
the k steps of 4, one and sixteen subdomains, blocks of unequal height, tasks
of one tile (nx != ny: two columns per system) and of two, in both precisions,
no-slip and free-slip.
"""
import numpy as np
import pytest

from iwrepo_b200 import config as cf

pytestmark = pytest.mark.gpu

UNEQUAL = dict(z0=[0.0, 0.2, 0.35], zh=[0.2, 0.15, 0.65])
SHAPES = [(3, 2), (4, 3), (7, 4), (8, 3), (9, 16), (12, 1), (15, 3), (16, 5), (17, 4), (23, 2), (24, 3), (25, 8), (31, 2),
          (32, 3), (33, 3), (39, 2), (40, 2)]


@pytest.mark.parametrize("precision", [cf.IW_PREC_FP64, cf.IW_PREC_MIXED])
@pytest.mark.parametrize("nzloc,nsubd", SHAPES)
def test_tensor_core_solve_gives_the_same_bits(nzloc, nsubd, precision):
    import iwrepo_b200 as iw
    kw = dict(UNEQUAL) if nsubd == 3 else {}
    square = nzloc % 2 == 0
    cfg = cf.Config(nx=24 if square else 32, ny=24 if square else 18, nzloc=nzloc, nsubd=nsubd, dt=1e-3,
                    bc_variant=cf.IW_BC_NOSLIP if square else cf.IW_BC_FREESLIP, precision=precision, **kw).validate()
    runs = []
    for variant in (1, 2):
        s = iw.Solver(cfg)
        s.set_launch("solve", variant)
        s.init_mode1(0.05, 1e-3, 11)
        s.step(4)
        runs.append([s.state(lev) for lev in range(5)])
        s.close()
    for a, b in zip(*runs):
        assert np.array_equal(a, b)


def test_default_solve_variant_is_the_tensor_core_kernel():
    import iwrepo_b200 as iw
    s = iw.Solver(cf.Config(nx=16, ny=16, nzloc=9, nsubd=2, dt=1e-3).validate())
    assert s.get_launch("solve") == 2
    s.close()
