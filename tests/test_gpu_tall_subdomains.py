"""Steps with more points per subdomain than the tensor-core stages take (nzloc 41 to 48), against the
oracle: stage E's tiled kernel then needs more shared memory than a kernel gets unasked (FP64, nzloc >= 42)."""
import numpy as np
import pytest

from iwrepo_b200 import config as cf

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [cf.IW_PREC_FP64, cf.IW_PREC_MIXED])
@pytest.mark.parametrize("nzloc,nsubd", [(41, 2), (42, 2), (44, 3), (48, 1), (48, 2)])
def test_steps_match_the_oracle(nzloc, nsubd, precision):
    import iwrepo_b200 as iw
    from oracle import Oracle
    cfg = cf.Config(nx=16, ny=8, nzloc=nzloc, nsubd=nsubd, dt=1e-3, precision=precision).validate()
    o, s = Oracle(cfg, fourier_scale=True), iw.Solver(cfg)
    o.init_mode1(0.05, 1e-4, 9)
    s.init_mode1(0.05, 1e-4, 9)
    o.step(5)
    s.step(4)
    s.run(1)  # from a captured graph
    a, b = s.state(), o.state()
    # FP64: rounding of the solves, as in the smaller configurations; mixed: FP32 storage, 6e-8 a step and value, of
    # the largest velocity (v is noise, 500 times smaller than u)
    big = max(np.linalg.norm(b[q]) for q in range(3))
    for q in range(4):
        n = np.linalg.norm(b[q])
        tol = (1e-10 if q == 1 else 1e-11) * n if precision == cf.IW_PREC_FP64 else 1e-5 * (big if q < 3 else n)
        assert np.linalg.norm(a[q] - b[q]) <= tol, (q, np.linalg.norm(a[q] - b[q]) / n)
    s.close()
