"""Columns of more points than four warps' right-hand sides leave room for in shared memory (nz > 1816), solved
with the band LU: steps against the oracle on either side of the line and at the largest nz."""
import numpy as np
import pytest

from iwrepo_b200 import config as cf

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nzloc,nsubd", [(47, 38), (48, 38), (48, 64)])
def test_steps_match_the_oracle(nzloc, nsubd):
    import iwrepo_b200 as iw
    from oracle import Oracle
    cfg = cf.Config(nx=8, ny=4, nzloc=nzloc, nsubd=nsubd, dt=1e-4).validate()
    o, s = Oracle(cfg, fourier_scale=True), iw.Solver(cfg)
    o.init_mode1(0.05, 1e-4, 9)
    s.init_mode1(0.05, 1e-4, 9)
    o.step(2)
    s.step(2)
    a, b = s.state(), o.state()
    # The same factors and the same order of operations in the sweeps, transforms and the derivative round differently: 1.1e-16
    # of the velocity times the largest entries of (2 / h) D, 1.5e5 at 48 x 64, is 2e-11 of it; v, noise a thousand
    # times smaller than u, takes its share of that from the pressure.
    big = max(np.linalg.norm(b[q]) for q in range(3))
    for q in range(4):
        assert np.linalg.norm(a[q] - b[q]) <= 1e-10 * (big if q < 3 else np.linalg.norm(b[3])), q
    s.close()
