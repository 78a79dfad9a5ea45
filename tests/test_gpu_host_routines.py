"""The routines on host fields (horfft_, dpdz_, filter_3dlegenfourier_, interface_avg3d_) keep their device
scratch and twiddles with the handle: a repeated call allocates nothing, a refused allocation leaves the
caller's array as it was, threads do not meet in the scratch, and fields beyond its bound pass through one
of their own."""
import threading

import numpy as np
import pytest

from iwrepo_b200 import config as cf

pytestmark = pytest.mark.gpu


def _calls(s, f):
    avg, count = s.interface_avg3d(f)
    return [s.horfft(f, 1), s.horfft(f, -1), s.dpdz(f), s.filter_3dlegenfourier(f), avg, np.array([count])]


def _field(cfg, seed):
    return np.random.default_rng(seed).standard_normal((cfg.nz, cfg.ny, cfg.nxpp))


@pytest.mark.parametrize("precision", [cf.IW_PREC_FP64, cf.IW_PREC_MIXED])
@pytest.mark.parametrize("nx,ny,nzloc,nsubd", [(16, 8, 9, 3), (18, 1, 5, 1), (30, 20, 17, 2)])
def test_repeated_calls_allocate_nothing(nx, ny, nzloc, nsubd, precision):
    import iwrepo_b200 as iw
    from iwrepo_b200 import _lib
    lib = _lib.lib()
    cfg = cf.Config(nx=nx, ny=ny, nzloc=nzloc, nsubd=nsubd, dt=1e-3, precision=precision).validate()
    f, g = _field(cfg, 1), _field(cfg, 2)
    s, fresh = iw.Solver(cfg), iw.Solver(cfg)
    first = _calls(s, f)
    _calls(s, g)  # the scratch holds another field's values
    held = s.device_bytes()
    _lib.check(lib.iw_fail_allocation(s.h, 1))
    again = _calls(s, f)
    _lib.check(lib.iw_fail_allocation(s.h, 0))
    assert s.device_bytes() == held
    for a, b, c in zip(first, again, _calls(fresh, f)):
        assert np.array_equal(a, b) and np.array_equal(a, c)
    s.close()
    fresh.close()


def test_refused_allocation_leaves_the_array():
    import iwrepo_b200 as iw
    from iwrepo_b200 import _lib
    lib = _lib.lib()
    cfg = cf.Config(nx=16, ny=8, nzloc=9, nsubd=3, dt=1e-3, precision=cf.IW_PREC_MIXED).validate()
    f = _field(cfg, 3)
    for call in ("horfft", "filter_3dlegenfourier", "interface_avg3d"):
        args = (f, 1) if call == "horfft" else (f,)
        for nth in (1, 2):  # the scratch, the twiddles
            s = iw.Solver(cfg)
            _lib.check(lib.iw_fail_allocation(s.h, nth))
            out = getattr(s, call)(*args)
            if call != "filter_3dlegenfourier" or nth == 1:
                assert lib.iw_last_status() == 6
                assert np.array_equal(out[0] if call == "interface_avg3d" else out, f)
            _lib.check(lib.iw_fail_allocation(s.h, 0))
            a = getattr(s, call)(*args)
            t = iw.Solver(cfg)
            b = getattr(t, call)(*args)
            assert np.array_equal(*((a[0], b[0]) if call == "interface_avg3d" else (a, b)))
            s.close()
            t.close()


def test_threads_on_one_handle():
    import iwrepo_b200 as iw
    cfg = cf.Config(nx=64, ny=60, nzloc=9, nsubd=4, dt=1e-3, precision=cf.IW_PREC_MIXED).validate()
    s = iw.Solver(cfg)
    fields = [_field(cfg, 10 + k) for k in range(4)]
    want = []
    for f in fields:
        t = iw.Solver(cfg)
        want.append((t.horfft(f, 1), t.dpdz(f), t.filter_3dlegenfourier(f)))
        t.close()
    got = [[] for _ in fields]

    def work(k):
        for _ in range(8):
            got[k].append((s.horfft(fields[k], 1), s.dpdz(fields[k]), s.filter_3dlegenfourier(fields[k])))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for k in range(4):
        for r in got[k]:
            assert all(np.array_equal(a, b) for a, b in zip(r, want[k]))
    s.close()


def test_fields_beyond_the_scratch():
    import iwrepo_b200 as iw
    cfg = cf.Config(nx=64, ny=64, nzloc=9, nsubd=2, dt=1e-3).validate()
    s = iw.Solver(cfg)
    nk = (32 << 20) // (66 * 64) + 3  # planes: just over 256 MB
    f = np.random.default_rng(4).standard_normal((nk, 64, 66))
    held = s.device_bytes()
    big = s.horfft(f, 1, nk)
    assert s.device_bytes() == held
    for k in (0, nk // 2, nk - 18):
        assert np.array_equal(big[k:k + 18], s.horfft(f[k:k + 18], 1, 18))
    s.close()
