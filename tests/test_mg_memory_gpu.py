"""Device memory of a solver: the coefficients, iterates, right-hand sides and
stencils of its levels in both precisions, and at most 32 bytes an unknown for
the transfer weights (four in double, or fewer in both precisions), so that a
grid which fits the device keeps fitting."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sys_,m,n,aspect", [(0, 2048, 2048, 1.0), (1, 2048, 2048, 3.0)])
def test_bytes_per_unknown(gpu, sys_, m, n, aspect):
    import torch
    from incrmt_b200 import capi
    from test_tile_indices import hierarchy
    capi.MGSolver(sys_, 64, 64).close()  # loads the kernels
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    s = capi.MGSolver(sys_, m, n, bx=-1 + 2 * aspect)
    used = before - torch.cuda.mem_get_info()[0]
    # level 0: coefficients in both precisions (12 bytes, MAC 24), density 8, b
    # and z 16, the smoothers' buffers 20; below: z, b 16, stencils 108, buffers 20
    levels = [(mm * nn) for (mm, nn, *_) in hierarchy(s.m_sys, s.n_sys, 0, 0, (n * aspect / m) ** 2)]
    fine, coarse = levels[0], sum(levels[1:])
    assert used <= (44 + (24 if sys_ == 0 else 12) + 32) * fine + (144 + 32) * coarse + (32 << 20)
    s.close()
