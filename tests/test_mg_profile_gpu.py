"""The bytes that the smoothing launches of the fine level are credited with:
their operands and result once for both sweeps, no iterate from a zero start."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sys_,words", [(0, 5), (1, 4)])
def test_bytes_of_a_launch(gpu, sys_, words):
    import torch
    from incrmt_b200 import capi
    s = capi.MGSolver(sys_, 320, 256)
    s.set_density(np.ones((260, 324)))
    N = s.m_sys * s.n_sys
    b = np.random.default_rng(1).standard_normal(N)
    b = torch.tensor(b - b.mean(), device="cuda")
    z = torch.zeros(N, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    s.set_profiling(True)
    s.vcycle_device(b.data_ptr(), z.data_ptr())
    torch.cuda.synchronize()
    vc = s.solve_device(b.data_ptr(), z.data_ptr()).vcycles
    ms, nbytes, launches = s.profile()
    assert launches == 2 * (vc + 1) and ms > 0
    assert nbytes == launches * N * 8.0 * words
    s.set_profiling(True)
    z.zero_()
    torch.cuda.synchronize()
    vc = s.solve_device(b.data_ptr(), z.data_ptr(), precision=capi.PREC_MIXED).vcycles
    ms, nbytes, launches = s.profile()
    assert launches == 2 * vc
    assert nbytes == vc * N * 4.0 * (2 * words - 1)  # the first smoothing starts from zero
    s.close()
