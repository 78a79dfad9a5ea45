"""Runs of different sizes stepped by threads of their own have the bits of the same runs one after the other: the
shared-memory limit of a kernel is shared by all handles, and their launches ask for different amounts."""
import threading

import numpy as np
import pytest

from iwrepo_b200 import config as cf

pytestmark = pytest.mark.gpu

SIZES = [dict(nx=24, ny=16, nzloc=5, nsubd=2), dict(nx=100, ny=60, nzloc=17, nsubd=4), dict(nx=50, ny=200, nzloc=33, nsubd=3),
         dict(nx=36, ny=12, nzloc=44, nsubd=2)]


@pytest.mark.parametrize("solver", [cf.IW_SOLVE_AUTO, cf.IW_SOLVE_LU])
def test_steps_in_threads(solver):
    import iwrepo_b200 as iw
    runs = {}

    def work(key, size, steps=24):
        s = iw.Solver(cf.Config(dt=1e-3, solver=solver, **size).validate())
        s.init_mode1(0.02, 1e-4, 3)
        for _ in range(steps):
            s.step(1)
        runs[key] = s.state()
        s.close()

    for k, size in enumerate(SIZES):
        work(k, size)
    threads = [threading.Thread(target=work, args=(10 + k, size)) for k, size in enumerate(SIZES)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for k in range(len(SIZES)):
        assert np.array_equal(runs[10 + k], runs[k]), SIZES[k]
