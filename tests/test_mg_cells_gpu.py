"""The smoother by cells (k_smooth_cells), with the transfers and Galerkin
products by tiles, against one launch per colour and per point, bit for bit:
sizes around a tile's edges and around the rules that choose its height, odd
sizes, grids of many or few tiles, arrays that cannot be read by pairs, and
seams in either direction with densities that do not match across them (periodic
sizes that stay even down to the levels one launch holds: a larger odd periodic
level is swept by colours that meet at its seam, in no fixed order)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CASES = [
    # sys, m, n, x_prd, y_prd, zpr, mixed precision
    (0, 512, 512, False, False, False, True),
    (0, 513, 511, False, False, False, False),     # odd, just below and above in a direction
    (0, 721, 601, False, False, True, True),       # 361 cells: a last strip of one cell
    (0, 240, 1201, False, False, False, True),     # two full strips
    (0, 16384, 17, False, False, False, False),    # more strips than blocks in a wave
    (0, 17, 16384, False, False, False, False),    # one strip, many chunks
    (0, 640, 512, True, True, False, False),
    (0, 1536, 320, False, True, True, True),
    (0, 112, 96, False, False, False, True),       # two MAC tiles by four
    (0, 114, 98, False, False, True, True),        # one cell more
    (0, 111, 95, False, False, False, True),
    (0, 128, 160, True, True, False, True),
    (1, 107, 95, False, False, False, True),       # 108 x 96 nodes: two tiles of 27 cells, six of 8
    (1, 108, 96, False, False, True, True),
    (1, 160, 160, True, True, False, True),
    (1, 511, 289, False, False, True, True),       # either height, double
    (1, 760, 900, False, False, False, True),      # either height, single
    (1, 1100, 1024, False, True, False, True),
    (1, 1601, 1499, False, False, False, True),
    (1, 1536, 1536, False, True, True, True),
]


@pytest.mark.parametrize("sys_,m,n,xp,yp,zpr,mixed", CASES)
@pytest.mark.parametrize("shift", [0, 1])
def test_cells_identical_to_colour_launches(gpu, sys_, m, n, xp, yp, zpr, mixed, shift):
    import torch
    from incrmt_b200 import capi
    s = capi.MGSolver(sys_, m, n, bx=-1 + 2 * m / max(m, n), by=-1 + 2 * n / max(m, n), x_prd=xp, y_prd=yp, zpr=zpr)
    rng = np.random.default_rng(m * 7 + n)
    rho = 1 + 2 * rng.random((n + 4, m + 4))
    N = s.m_sys * s.n_sys
    b = rng.standard_normal(N)
    b -= b.mean()
    z0 = rng.standard_normal(N)
    bd = torch.zeros(N + 1, dtype=torch.float64, device="cuda")[shift:shift + N]  # shift 1: rows start off a pair
    bd.copy_(torch.tensor(b))
    out = {}
    for tiles in (True, False):
        s.set_tiles(tiles)
        s.set_density(rho)
        z = torch.tensor(z0, device="cuda")
        zm = torch.zeros(N, dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        s.vcycle_device(bd.data_ptr(), z.data_ptr())
        if mixed:  # one FP32 correction; the cap is its expected end
            with pytest.raises(capi.IncrmtError) as e:
                s.solve_device(bd.data_ptr(), zm.data_ptr(), max_vcycles=1, precision=capi.PREC_MIXED)
            assert e.value.code == capi.ERR_NOCONV
        torch.cuda.synchronize()
        out[tiles] = (z.cpu().numpy(), zm.cpu().numpy())
    assert np.isfinite(out[True][0]).all() and np.isfinite(out[True][1]).all()
    assert np.array_equal(out[True][0], out[False][0])
    assert np.array_equal(out[True][1], out[False][1])
    s.close()
