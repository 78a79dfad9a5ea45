"""A device allocation that fails while a step builds its solver tables: the step reports
IW_ERR_NOMEM, the handle stays as it was before the step, and a later step gives the same bits as a
run that never failed."""
import numpy as np
import pytest

from iwrepo_b200 import config as cf

pytestmark = pytest.mark.gpu
NOMEM = 6  # IW_ERR_NOMEM


def _solver(precision):
    import iwrepo_b200 as iw
    # the lowest wavenumbers are above the condition bound: raw inverses and a refined prefix
    s = iw.Solver(cf.Config(nx=16, ny=8, nzloc=9, nsubd=3, dt=1e-3, precision=precision).validate())
    s.init_mode1(0.05, 1e-4, 7)
    return s


@pytest.mark.parametrize("precision", [cf.IW_PREC_FP64, cf.IW_PREC_MIXED])
@pytest.mark.parametrize("before", [0, 1, 2])
def test_failed_table_build_leaves_the_handle_usable(precision, before):
    from iwrepo_b200 import IwError, _lib
    lib = _lib.lib()
    ref = _solver(precision)
    ref.step(5)
    want = ref.state()
    ref.close()
    failures = 0
    for nth in range(1, 100):
        s = _solver(precision)
        s.step(before)
        _lib.check(lib.iw_fail_allocation(s.h, nth))
        try:
            s.step(1)
            done = 1
        except IwError as e:
            assert e.code == NOMEM, (nth, str(e))
            done, failures = 0, failures + 1
        _lib.check(lib.iw_fail_allocation(s.h, 0))
        s.step(5 - before - done)
        assert np.array_equal(s.state(), want), nth
        s.close()
        if done:
            break
    else:
        pytest.fail("a step makes more than 99 allocations")
    if before == 0:
        assert failures >= 4 * 7  # tables, column maps and task lists of four kinds of system
