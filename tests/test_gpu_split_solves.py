"""iw_helm_solve_batched, mode 0, with lambdas on both sides of the condition bound: the columns of the band LU are
solved beside those of the block inverses.  A chain of solves, each from the solution before it and the last ones in place,
has the bits of the same chain with a wait after every call, and each column those of a solve of its side alone."""
import numpy as np
import pytest

from iwrepo_b200 import config as cf

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nzloc,nsubd,ncol", [(9, 3, 40), (25, 8, 3000), (36, 4, 700)])
def test_split_columns(nzloc, nsubd, ncol):
    import torch
    import iwrepo_b200 as iw
    s = iw.Solver(cf.Config(nx=16, ny=8, nzloc=nzloc, nsubd=nsubd, dt=1e-3).validate())
    gen = torch.Generator(device="cuda").manual_seed(nzloc)
    low, high = np.geomspace(1e-3, 0.1, 5), np.geomspace(1.0e5, 4.0e5, 7)
    lam = torch.tensor(np.resize(np.concatenate([low, high]), ncol), device="cuda")
    rhs = torch.randn((ncol, nzloc * nsubd, 2), generator=gen, device="cuda", dtype=torch.float64)

    def solve(lam, src, dst):
        iw.helm_solve_batched(s, lam.data_ptr(), lam.numel(), 0, 1, src.data_ptr(), dst.data_ptr(), 0)

    def chain(wait):
        b = [rhs.clone(), torch.zeros_like(rhs), torch.zeros_like(rhs)]
        torch.cuda.synchronize()
        for src, dst in ((0, 1), (1, 2), (2, 0), (0, 0), (0, 1), (1, 1)):
            solve(lam, b[src], b[dst])
            if wait:
                s.sync()
        s.sync()
        return b

    want = chain(True)
    for _ in range(3):
        assert all(torch.equal(x, y) for x, y in zip(chain(False), want))
    one = torch.zeros_like(rhs)
    solve(lam, rhs, one)
    s.sync()
    for side in (lam < 1, lam > 1):
        sub, out = rhs[side].contiguous(), torch.zeros_like(rhs[side])
        part = lam[side].contiguous()
        torch.cuda.synchronize()
        solve(part, sub, out)
        s.sync()
        assert torch.equal(out, one[side])
    s.close()
