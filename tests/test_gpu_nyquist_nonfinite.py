"""The imaginary part of the x-Nyquist column is not part of a real field: the round-trip projection drops
it, so a step accepts any value there, NaN included, and computes the same as without it.  A
non-finite value that the projection keeps is reported."""
import numpy as np
import pytest

from iwrepo_b200 import config as cf

pytestmark = pytest.mark.gpu


def _run(cfg, spoil, stage_a, value):
    import iwrepo_b200 as iw
    s = iw.Solver(cfg)
    s.init_mode1(0.05, 1e-3, 5)
    st = s.state()
    if spoil == "imag":
        st[:, 2, 1, cfg.nx + 1] = value
    elif spoil == "real":
        st[0, 2, 1, cfg.nx] = value
    elif spoil == "mean":
        st[1, 2, 0, 0] = value
    s.set_launch("stage_a", stage_a)
    s.set_state(st)
    try:
        s.step(2)
        s.sync()
        return s.state()
    finally:
        s.close()


@pytest.mark.parametrize("stage_a", [-1, 0])
@pytest.mark.parametrize("precision", [cf.IW_PREC_FP64, cf.IW_PREC_MIXED])
@pytest.mark.parametrize("nx,ny,nzloc,nsubd", [(16, 8, 9, 2), (18, 6, 17, 2)])
def test_nyquist_imaginary_part(nx, ny, nzloc, nsubd, precision, stage_a):
    from iwrepo_b200 import IwError
    cfg = cf.Config(nx=nx, ny=ny, nzloc=nzloc, nsubd=nsubd, dt=1e-3, precision=precision).validate()
    want = _run(cfg, None, stage_a, 0.0)
    for value in (np.nan, np.inf, 0.25):
        assert np.array_equal(_run(cfg, "imag", stage_a, value), want)
    for spoil in ("real", "mean"):
        with pytest.raises(IwError):
            _run(cfg, spoil, stage_a, np.nan)
