"""The windowed banded LU (SW2GPU_PREC_BAND) at the widths where its tiling changes: a system
narrower than one panel, one, two and three panel rows per lane, right-hand side lengths that are
not multiples of a panel or of a back-substitution block, and a band too wide for the window (the
pivot-by-pivot walk)."""
import numpy as np
import pytest

from adhv8_kraken_b200 import capi, meshgen
from adhv8_kraken_b200.sw2 import SW2GPU

pytestmark = pytest.mark.gpu


# channel nx x ny: 3 (nx + 1)(ny + 1) unknowns, band half-width about 3 (ny + 3) unknowns
@pytest.mark.parametrize("nx,ny", [(1, 1), (5, 1), (9, 2), (31, 5), (20, 11), (33, 16), (29, 20), (21, 32), (45, 41), (50, 48)])
def test_windowed_band_solve_equals_dense_solve(nx, ny):
    m = meshgen.channel(nx=nx, ny=ny, length=10.0 * nx, width=10.0 * ny, dt=10.0, nsteps=2)
    g = SW2GPU(m, precond=capi.SW2GPU_PREC_BAND)
    assert g.step()["status"] == 0
    rp, col, val, _ = g.load()
    V = m.nnodes
    rng = np.random.default_rng(3)
    x_ref = rng.standard_normal(3 * V)
    A = np.zeros((V, 3, V, 3))
    A[np.repeat(np.arange(V), np.diff(rp)), :, col, :] = val
    A = A.reshape(3 * V, 3 * V)
    b = A @ x_ref
    x, its, rc = g.linear_solve(val, b)
    g.close()
    assert rc == 0 and its == 1
    # an LU without pivoting of these diagonally strong systems: condition numbers up to 1e5 times
    # the rounding of a 6,000-unknown system
    assert np.abs(x - x_ref).max() <= 1e-10 * np.abs(x_ref).max()
