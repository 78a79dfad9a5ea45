"""x rows and y transforms of every kind of length, against the oracle in FP64.

nx / 2 = R0 * NB with R0 in 2, 4, 6, 8, 10 and NB in 8, 16, 32 takes the kernel whose first and last
passes run in registers; other lengths (10, 15, 25, 36, 54, 100, 8, 9 and the longest) the general one.
ny covers last CTAs with fewer rows than their places, short columns that share a warp, and
mixed radices.  One step from a seeded state: both sides round transforms of at most 2^10 points and
solve the same systems, so they agree as in the parity test (1e-12; v, which holds noise alone, 1e-11).
"""
import numpy as np
import pytest

from iwrepo_b200 import config as cf

pytestmark = pytest.mark.gpu

SHAPES = [(32, 6), (48, 10), (64, 5 * 2), (96, 6), (128, 18), (160, 6), (192, 2), (256, 6), (320, 10), (384, 4),
          (512, 6), (640, 6), (20, 12), (30, 24), (50, 30), (72, 36), (108, 48), (200, 60), (768, 4),
          (1024, 4), (16, 120), (16, 128), (18, 256), (20, 150)]


@pytest.mark.parametrize("nx,ny", SHAPES)
def test_transform_lengths_match_oracle(nx, ny):
    import iwrepo_b200 as iw
    from oracle import Oracle
    cfg = cf.Config(nx=nx, ny=ny, nzloc=8, nsubd=2, dt=1e-3, precision=cf.IW_PREC_FP64).validate()
    o, s = Oracle(cfg, fourier_scale=True), iw.Solver(cfg)
    for x in (o, s):
        x.init_mode1(0.05, 1e-4, 7)
        x.step(2)
    a, b = s.state(0), o.state(0)
    for q in range(4):
        assert np.linalg.norm(a[q] - b[q]) <= (1e-11 if q == 1 else 1e-12) * np.linalg.norm(b[q]), q
    s.close()


@pytest.mark.parametrize("forcing", [1, 2])
@pytest.mark.parametrize("nx", [64, 96, 100])
def test_forced_rows_match_oracle(nx, forcing):
    """The paddle terms are added in the same kernels (registers of two values per thread)."""
    import iwrepo_b200 as iw
    from oracle import Oracle
    cfg = cf.Config(nx=nx, ny=6, nzloc=8, nsubd=2, dt=1e-3, forcing=forcing, xacrit=0.5, precision=cf.IW_PREC_FP64).validate()
    o, s = Oracle(cfg, fourier_scale=True), iw.Solver(cfg)
    for x in (o, s):
        x.init_mode1(0.05, 1e-4, 7)
        x.step(2)
    a, b = s.state(0), o.state(0)
    for q in range(4):
        assert np.linalg.norm(a[q] - b[q]) <= (1e-11 if q == 1 else 1e-12) * np.linalg.norm(b[q]), q
    s.close()
