"""iw_diag from (kx, y) rows (k_xrow_stats) at the edges of its transforms: odd
half lengths, one y row, row lengths of one and of several values per lane,
subdomains beyond the tensor-core derivative (N > 40), in both precisions,
against the same sums and extrema of physical fields from horfft and dpdz.

FP64: sums of n terms of relative error 1e-16 each, transforms of log n passes: 1e-12
covers both with a margin of 100.  Mixed: FP32 transforms, relative error
about 6e-8 log2(n) of the largest value; sums average it: 1e-5 of each quantity.
"""
import numpy as np
import pytest

from iwrepo_b200 import config as cf

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,tol", [(cf.IW_PREC_FP64, 1e-12), (cf.IW_PREC_MIXED, 1e-5)])
@pytest.mark.parametrize("nx,ny,nzloc,nsubd", [(30, 10, 9, 2), (64, 1, 17, 3), (18, 16, 44, 1), (270, 4, 12, 2), (512, 6, 9, 1),
                                               (1080, 2, 5, 1)])
def test_diag_equals_physical_sums(nx, ny, nzloc, nsubd, precision, tol):
    import iwrepo_b200 as iw
    cfg = cf.Config(nx=nx, ny=ny, nzloc=nzloc, nsubd=nsubd, dt=1e-3, precision=precision).validate()
    s = iw.Solver(cfg)
    s.init_mode1(0.05, 1e-2, 5)
    d = s.diag()
    f = s.state(0)
    kx = np.repeat(np.arange(nx // 2 + 1), 2)[None, None, :]
    ky = np.where(np.arange(ny) < ny // 2, np.arange(ny), np.arange(ny) - ny)[None, :, None] * (ny > 1)

    def times_i(a, k):
        b = np.empty_like(a)
        b[..., 0::2], b[..., 1::2] = -(k * a)[..., 1::2], (k * a)[..., 0::2]
        return b

    phys = lambda a: s.horfft(np.ascontiguousarray(a), 1)[..., :nx]  # noqa: E731
    p = [phys(q) for q in f]
    ke = 0.5 * sum((p[q][1:] ** 2).sum() for q in range(3))
    eps = cfg.xnu * sum((phys(g)[1:] ** 2).sum() for q in range(3)
                        for g in (times_i(f[q], kx), times_i(f[q], ky), s.dpdz(f[q])))
    assert abs(d["ke"] - ke) <= tol * ke and abs(d["eps"] - eps) <= tol * eps
    assert abs(d["cfl"][0] - np.abs(p[0]).max() * cfg.dt * nx / cfg.xlen) <= tol * d["cfl"][0]
    for q in range(3):
        lo, hi = min(p[q].min(), 0.0), max(p[q].max(), 0.0)
        m = max(-lo, hi)
        assert abs(d["minmax"][2 * q] - lo) <= tol * m and abs(d["minmax"][2 * q + 1] - hi) <= tol * m
    s.close()
