"""Periodic levels of odd size above those one launch holds, where the first and
last rows (columns) of a colour are neighbours across the seam: every run of a
V-cycle gives the same iterate, in double and in a single-precision correction,
with tiles on and off, and on a coarsest level of that kind too."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sys_,m,n,xp,yp", [
    (1, 1100, 904, False, True),   # 113 rows
    (0, 600, 512, True, False),    # 75 columns
    (0, 1024, 1022, False, True),  # 511 rows
    (1, 1200, 1200, True, True),   # 75 x 75
    (0, 1000, 1000, True, True),   # 125 x 125: the coarsest level
    (1, 202, 202, True, True),     # 101 x 101 the same, odd at once
])
def test_reproducible(gpu, sys_, m, n, xp, yp):
    import torch
    from incrmt_b200 import capi
    s = capi.MGSolver(sys_, m, n, bx=1.0, by=-1 + 2 * n / m, x_prd=xp, y_prd=yp)
    rng = np.random.default_rng(m * 7 + n)
    rho = 1 + 2 * rng.random((n + 4, m + 4))
    N = s.m_sys * s.n_sys
    b = rng.standard_normal(N)
    bd = torch.tensor(b - b.mean(), device="cuda")
    z0 = rng.standard_normal(N)
    runs = []
    for tiles in (True, False):
        s.set_tiles(tiles)
        s.set_density(rho)
        for _ in range(4):
            z, zm = torch.tensor(z0, device="cuda"), torch.zeros(N, dtype=torch.float64, device="cuda")
            torch.cuda.synchronize()
            s.vcycle_device(bd.data_ptr(), z.data_ptr())
            with pytest.raises(capi.IncrmtError):  # one FP32 correction; the cap is its expected end
                s.solve_device(bd.data_ptr(), zm.data_ptr(), max_vcycles=1, precision=capi.PREC_MIXED)
            torch.cuda.synchronize()
            runs.append((z.cpu().numpy(), zm.cpu().numpy()))
    assert np.isfinite(runs[0][0]).all() and np.isfinite(runs[0][1]).all()
    for z, zm in runs[1:]:
        assert np.array_equal(z, runs[0][0])
        assert np.array_equal(zm, runs[0][1])
    s.close()
