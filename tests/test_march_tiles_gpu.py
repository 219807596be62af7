"""The march's and the extrapolation's two tile sizes (k_ls_fim_coop,
k_ls_extrap_tiles): windows off on these grids takes
the large tiles over the whole grid, windows on the small ones over the
object's window, whose tiles start elsewhere. After two steps the status has to
be the same, the level set to the rounding of values below one (the two runs
sum the same terms), and the sweeps as many."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPES = {
    "circle": lambda s: s.add_circle(0.13, -0.21, 0.3, 1.0, 2.0),
    "ellipse": lambda s: s.add_ellipse(-0.1, 0.2, 0.35, 0.12, 0.7, 1.0, 2.0),
    "rod": lambda s: s.add_rounded_rod(0.0, 0.05, 0.06, 0.25, 1.0, 2.0),
    "small": lambda s: s.add_circle(0.013, 0.007, 0.02, 1.0, 2.0),  # two to three cells: the whole band in a few tiles
    "corner": lambda s: s.add_circle(0.83, 0.85, 0.1, 1.0, 2.0),  # its band is cut by the walls' ghost rows
}


@pytest.mark.parametrize("shape", list(SHAPES))
@pytest.mark.parametrize("m,n", [(256, 256), (301, 233)])
def test_tile_sizes_agree(gpu, shape, m, n):
    from incrmt_b200 import capi
    out = []
    for windows in (True, False):
        s = capi.Simulation(m, n, ntrace=0)
        SHAPES[shape](s)
        s.set_windows(windows)
        dt = s.initialize()
        s.step(dt, 2)
        st = s.stats()
        out.append((s.get("phi"), s.get("status"), st.march_sweeps, s.get("X"), s.get("Y"), st.extrap_sweeps))
        s.close()
    assert np.array_equal(out[0][1], out[1][1])
    assert np.abs(out[0][0] - out[1][0]).max() <= 1e-14
    assert out[0][2] == out[1][2] and out[0][5] == out[1][5]
    band = (out[0][1] >= 2) & (out[0][1] <= 5)
    for k in (3, 4):
        assert np.abs(out[0][k][band] - out[1][k][band]).max() <= 1e-14


def test_singular_fit_is_reported(gpu):
    """A body below the grid's resolution: the radius-3 window is singular,
    the wider ones of the fallback too."""
    from incrmt_b200 import capi
    s = capi.Simulation(64, 64, ntrace=0)
    s.add_circle(0.013, 0.007, 0.025, 1.0, 2.0)
    dt = s.initialize()
    with pytest.raises(capi.IncrmtError) as e:
        s.step(dt, 2)
    assert e.value.code == capi.ERR_EXTRAP_SINGULAR
    s.close()
