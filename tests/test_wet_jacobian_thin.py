"""The closed-form Jacobian (adhv8_kraken_b200/csrc/sw2_wet_jac.cuh) down to the shallowest depth that
takes it: an element whose depths are not all above kWetMargin (1e-6 m) goes the general way."""
import os
import re

import numpy as np
import pytest
from test_wet_jacobian_on_host import CSRC, _call, _column, lib  # noqa: F401


def test_the_margin_is_what_the_depths_below_go_down_to():
    with open(os.path.join(CSRC, "sw2_kernels.cuh")) as fh:
        src = fh.read()
    assert re.search(r"constexpr double kWetMargin = 1e-6;", src)
    assert "h[i] > kWetMargin" in src


@pytest.mark.parametrize("depth", [1e-2, 1e-3, 1e-4, 1e-5, 3e-6, 1.03e-6])
@pytest.mark.parametrize("drag", [0.0, 0.02, 3e-6])
def test_thin_films(lib, drag, depth):  # noqa: F811
    """Drag roughness far above the depth (clipped law) and near it; depths within 1 % of each other,
    so that steps of 2 % keep each above the floors (1.2e-7 and below)."""
    rng = np.random.default_rng(29)
    ph = np.array([9.81, 0.1, 0.4, 0.0, 0.5, 5.0])
    m = np.array([drag, 0.5, 1e-4, 0.0])
    df = np.zeros(3, np.int32)
    for trial in range(10):
        g = np.zeros(29)
        ang = np.array([0.3, 2.2, 4.4]) + rng.uniform(-0.2, 0.2, 3)
        g[0:3], g[3:6] = 20 * np.cos(ang), 20 * np.sin(ang)
        g[6:9] = rng.uniform(-0.1, 0.1, 3)
        g[9:12] = depth * rng.uniform(1.0, 1.01, 3)
        g[12:18] = rng.uniform(0.05, 0.5, 6) * rng.choice([-1, 1], 6)
        g[18:21] = g[9:12]
        g[21:27] = g[12:18]
        J = _call(lib.jac, g, ph, m, df, 81).reshape(3, 3, 3, 3)
        scale = np.abs(J).max()
        for b in range(3):
            for var, off in enumerate((12, 15, 9)):
                k = off + b
                col = _column(lib, g, ph, m, df, k, 0.02 * abs(g[k])).reshape(3, 3)
                # the extrapolated remainder of steps between 2 % and 0.25 % of the value, and the
                # residual's rounding over the smallest
                assert np.abs(J[:, b, :, var] - col).max() <= 1e-6 * scale, (trial, b, var)
