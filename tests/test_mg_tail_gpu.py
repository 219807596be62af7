"""The coarse levels' cluster launch (k_tail): convergence to the tolerance, by
an independent residual, at V-cycle counts of a working hierarchy, for
hierarchies that exercise its layouts: one block and strips over the cluster,
levels of 2^k and 2^k + 1 unknowns, odd and thin ones, semi-coarsening in
either direction, even and odd periodic sizes. A wrong transfer or update on
any coarse level costs many V-cycles or the convergence."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# sys, m, n, box width / height
CASES = [
    (0, 6, 6, 1.0), (0, 9, 17, 1.0), (0, 33, 33, 1.0), (0, 65, 64, 1.0), (0, 129, 127, 1.0), (0, 300, 257, 1.0),
    (0, 200, 30, 6.7), (0, 30, 200, 0.15), (0, 160, 160, 3.0), (0, 160, 160, 0.3),
    (1, 6, 6, 1.0), (1, 32, 32, 1.0), (1, 64, 64, 1.0), (1, 128, 100, 1.0), (1, 255, 300, 1.0), (1, 150, 150, 3.0),
]


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("sys_,m,n,aspect", CASES)
def test_walls(gpu, sys_, m, n, aspect, precision):
    from incrmt_b200 import capi
    from oracle import operators
    bx, by = -1 + 2 * max(aspect, 1.0), -1 + 2 * max(1 / aspect, 1.0)
    s = capi.MGSolver(sys_, m, n, bx=bx, by=by)
    rng = np.random.default_rng(m * 11 + n + sys_)
    rho = np.ones((n + 4, m + 4))
    rho[n // 3:n // 2 + 2, m // 4:m // 2 + 2] = 3.0
    s.set_density(rho)
    b = rng.standard_normal((s.n_sys, s.m_sys))
    b -= b.mean()
    z = np.zeros(b.size)
    st = s.solve(b, z, precision=precision)
    dx, dy = (bx + 1) / m, (by + 1) / n
    apply = operators.mac_apply if sys_ == 0 else operators.fem_apply
    r = b - apply(rho, z.reshape(b.shape), dx, dy)
    assert np.linalg.norm(r) <= 1.2e-9 * np.linalg.norm(b)
    assert st.vcycles <= 14
    s.close()


@pytest.mark.parametrize("sys_", [0, 1])
@pytest.mark.parametrize("m,n", [(64, 64), (193, 144), (288, 144), (90, 80), (100, 112), (256, 160), (48, 18)])
def test_channel(gpu, sys_, m, n):
    """y-periodic with the zero-pressure edge: halo rows that wrap around the
    cluster, and 5, 7 and 9 coarse rows, where colours meet across the seam."""
    from incrmt_b200 import capi
    s = capi.MGSolver(sys_, m, n, ax=-1.0, bx=5.0, ay=-1.0, by=1.0, y_prd=True, zpr=True)
    rng = np.random.default_rng(m + n)
    rho = np.ones((n + 4, m + 4))
    rho[n // 2:n // 2 + 3, m // 4:m // 2] = 10.0
    s.set_density(rho)
    b = rng.standard_normal((s.n_sys, s.m_sys))
    if sys_ == 1:
        b[:, -1] = 0
    z = np.zeros(b.size)
    st = s.solve(b, z)
    assert st.vcycles <= 20
    r = b.ravel() - s.apply(z)
    assert np.linalg.norm(r) <= 1.2e-9 * np.linalg.norm(b)
    s.close()
