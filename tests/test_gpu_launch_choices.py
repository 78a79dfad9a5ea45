"""Launch choices that iw_autotune reports or iw_get_launch reads can be set on another handle of the same sizes,
which then gives the same bits: also nzloc above the register-column kernels' 33 and FP32 planes that are no
whole number of 16 bytes, where the tuner keeps the tensor-core stage E."""
import ctypes as C

import numpy as np
import pytest

from iwrepo_b200 import config as cf

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,nzloc,precision", [
    (16, 16, 33, cf.IW_PREC_MIXED), (16, 16, 34, cf.IW_PREC_FP64), (16, 16, 40, cf.IW_PREC_MIXED),
    (16, 16, 41, cf.IW_PREC_MIXED), (16, 1, 17, cf.IW_PREC_MIXED)])
def test_choices_can_be_set_again(nx, ny, nzloc, precision):
    import iwrepo_b200 as iw
    from iwrepo_b200 import _lib
    cfg = cf.Config(nx=nx, ny=ny, nzloc=nzloc, nsubd=2, dt=1e-3, precision=precision).validate()
    runs = [iw.Solver(cfg) for _ in range(3)]
    for s in runs:
        s.init_mode1(0.05, 1e-3, 11)
    tuned, reported, read = runs
    ch = (C.c_int * 4)()
    _lib.check(_lib.lib().iw_autotune(tuned.h, ch))
    for which, value in zip(("y_tile", "stage_a", "stage_e", "solve_pressure"), ch):
        assert tuned.get_launch(which) == value
        reported.set_launch(which, value)
    for which in tuned.LAUNCH:
        read.set_launch(which, tuned.get_launch(which))
    for s in runs:
        s.step(4)
    for level in range(5):
        want = tuned.state(level)
        assert np.array_equal(reported.state(level), want)
        assert np.array_equal(read.state(level), want)
    for s in runs:
        s.close()


def test_reported_z_kernels():
    import iwrepo_b200 as iw
    for nzloc, kernel in ((40, "tensor-core"), (41, "tiled")):
        with iw.Solver(cf.Config(nx=16, ny=16, nzloc=nzloc, nsubd=2, dt=1e-3).validate()) as s:
            s.init_mode1(0.05, 1e-3, 11)
            assert s.autotune()["z_kernels"] == {"stage_a": kernel, "stage_e": kernel}


@pytest.mark.parametrize("nx,own", [(32, True), (96, True), (640, True), (48, False), (512, True), (100, False), (1024, False)])
def test_x_row_threads_where_the_length_has_the_choice(nx, own):
    """Lengths with a kernel of their own leave the choice alone."""
    import iwrepo_b200 as iw
    cfg = cf.Config(nx=nx, ny=4, nzloc=5, nsubd=1, dt=1e-3, precision=cf.IW_PREC_MIXED).validate()
    with iw.Solver(cfg) as s:
        s.init_mode1(0.05, 1e-3, 11)
        s.set_launch("x_row_threads", 256)
        ch = s.autotune()["x_row_threads"]
        assert ch == 256 if own else ch in (128, 256)
