"""Isolated solves of several threads, each with handles of its own that come and go: the tables of one handle are made,
used and freed while the others'."""
import threading

import numpy as np
import pytest

from iwrepo_b200 import config as cf

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", [0, 1])
def test_tables_of_handles_that_come_and_go(mode):
    import torch
    import iwrepo_b200 as iw
    cfg = cf.Config(nx=16, ny=8, nzloc=9, nsubd=3, dt=1e-3).validate()
    sets, repeats, workers = 12, 4, 3
    lam = [torch.tensor(np.resize(np.geomspace(1e-2, 1e5 + k, 11), 40), device="cuda") for k in range(sets)]
    rhs = torch.ones((40, cfg.nz, 2), device="cuda", dtype=torch.float64)
    out = [[torch.zeros_like(rhs) for _ in range(sets)] for _ in range(workers + 1)]
    torch.cuda.synchronize()
    errors = []

    def work(w, many):
        try:
            for _ in range(many):
                with iw.Solver(cfg) as s:
                    for k in range(sets):
                        iw.helm_solve_batched(s, lam[k].data_ptr(), 40, 0, 1, rhs.data_ptr(), out[w][k].data_ptr(), mode)
                    s.sync()
        except Exception as e:  # noqa: BLE001 (reported by the test's thread)
            errors.append(e)

    work(workers, 1)
    threads = [threading.Thread(target=work, args=(w, repeats)) for w in range(workers)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors
    for w in range(workers):
        assert all(torch.equal(a, b) for a, b in zip(out[w], out[workers]))
