"""Launches that fail are reported.  A successful cudaFuncSetAttribute resets the CUDA runtime's record of a
launch that failed before it, so shared-memory limits and checks both go through the
helpers that keep the first error (set_smem, launch_error in csrc/iw_lib.cu)."""
import glob
import os
import re

import numpy as np
import pytest

from iwrepo_b200 import config as cf

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "iwrepo_b200", "csrc")


def test_limits_and_checks_go_through_the_helpers():
    for path in glob.glob(os.path.join(CSRC, "*.inl")) + glob.glob(os.path.join(CSRC, "*.cu*")):
        src = re.sub(r"//[^\n]*|/\*.*?\*/", "", open(path).read(), flags=re.S)
        if os.path.basename(path) == "iw_lib.cu":
            i, j = src.index("cudaError_t g_launch_error"), src.index("static inline cudaError_t launch_error()")
            assert "cudaFuncSetAttribute" in src[i:j]
            src = src[:i] + src[j:]
        assert "cudaFuncSetAttribute" not in src, path
        assert not re.search(r"CK\(\s*cuda(GetLast|PeekAtLast)Error", src), path


@pytest.mark.gpu
def test_refused_launch_is_reported_once():
    """Isolated band-LU solves of 1250 points ask for more shared memory than an SM has: the call says so, and the steps
    after it run without a trace of it."""
    import torch
    import iwrepo_b200 as iw
    from iwrepo_b200 import IwError
    cfg = cf.Config(nx=8, ny=4, nzloc=25, nsubd=50, dt=1e-4).validate()
    runs = []
    for ask in (False, True):
        s = iw.Solver(cfg)
        s.init_mode1(0.05, 1e-4, 9)
        if ask:
            lam = torch.full((4,), 1.0e4, dtype=torch.float64, device="cuda")
            rhs = torch.zeros((4, cfg.nz, 2), dtype=torch.float64, device="cuda")
            torch.cuda.synchronize()
            with pytest.raises(IwError):
                iw.helm_solve_batched(s, lam.data_ptr(), 4, 0, 1, rhs.data_ptr(), torch.zeros_like(rhs).data_ptr(), 0)
        s.step(2)
        runs.append(s.state())
        s.close()
    assert np.array_equal(*runs)
