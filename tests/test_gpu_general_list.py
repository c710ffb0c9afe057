"""The wet/dry Jacobian kernel takes the listed elements sixteen to a CTA, the + and - passes of a
column in the two halves of a warp.  Lists of one element and around one and two groups against the
oracle's residual and Jacobian, within 1e-12 and 1e-7, the tolerances of the other wet/dry states
(rounding; the truncation and round-off of the central differences)."""
import numpy as np
import pytest

from adhv8_kraken_b200.sw2 import SW2GPU
from conftest import relerr
from helpers import channel_model
from oracle.oracle import Oracle


def old_dry_nodes(model, listed, count):
    """Nodes whose triangles, apart from one another and from the listed ones, the inflow and the
    tailwater, number `count`."""
    tri = model.tri
    degree = np.bincount(tri.ravel(), minlength=model.nnodes)
    busy = np.zeros(model.nnodes, bool)
    busy[model.edges.ravel()] = True
    busy[tri[listed]] = True
    picked, left = [], count
    for d in (6, 3):
        for n in np.flatnonzero(degree == d):
            mine = tri[(tri == n).any(1)]
            if left >= d and not busy[mine].any():
                picked.append(n)
                busy[mine] = True
                left -= d
    assert left == 0, left
    return np.array(picked, int)


@pytest.mark.gpu
@pytest.mark.parametrize("count", [12, 15, 18, 33])
def test_short_lists_of_wet_dry_elements(count):
    model = channel_model()
    # one dry wall node: with the flags of the wet/dry test, twelve listed triangles; the others have
    # a node that was dry two levels ago
    wall = np.flatnonzero((np.bincount(model.tri.ravel()) == 3) & ~np.isin(np.arange(model.nnodes), model.edges))
    dry = wall[len(wall) // 2]
    rng = np.random.default_rng(count)
    h, hoo = model.h0 + rng.normal(0, 0.02, model.nnodes), model.h0.copy()
    h[dry] = -0.05
    u, v = 0.5 + rng.normal(0, 0.1, model.nnodes), rng.normal(0, 0.1, model.nnodes)
    o = Oracle(model)
    for level, depth in ((0, h), (1, model.h0), (2, hoo)):
        o.set_state(level, depth, 0.5**level * u, 0.5**level * v)
    o.set_dt(5.0, model.series_values(0.0, 5.0))
    wd = o.wdflag()
    assert (wd > 0).sum() == 12
    hoo[old_dry_nodes(model, wd > 0, count - 12)] = -0.05
    o.set_state(2, hoo, 0.25 * u, 0.25 * v)
    assert ((wd > 0) | (hoo[model.tri] <= 0).any(1)).sum() == count
    g = SW2GPU(model)
    for level, depth in ((0, h), (1, model.h0), (2, hoo)):
        g.set_state(level, depth, 0.5**level * u, 0.5**level * v)
    g.set_dt(5.0, model.series_values(0.0, 5.0))
    g.set_wd(wd)
    rg, ro = g.resid(), o.resid()
    assert relerr(rg, ro) <= 1e-12
    _, _, vg, rg = g.load()
    vo, ro = o.load()
    assert relerr(rg, ro) <= 1e-12
    assert relerr(vg.reshape(-1), vo.reshape(-1)) <= 1e-7
