"""The plain form on gridded bathymetry with stretched axes and with axes of the
two fields that are equal, nearly equal or of another spacing rule, against the
oracle."""

import numpy as np
import pytest

from tests import helpers as H

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("axis", ["uniform", "stretched"])
@pytest.mark.parametrize("current", ["equal", "one value off", "last value off", "shorter"])
def test_equal_and_nearly_equal_axes(oracle, axis, current):
    import mantaray_gb300 as mr

    rng = np.random.default_rng(len(axis) + len(current))
    n = 41
    x = np.arange(n, dtype=np.float32) * np.float32(10.0)
    if axis == "stretched":
        x[2:] += np.float32(0.25) * rng.integers(0, 8, n - 2).astype(np.float32)
    cx = x.astype(np.float64)
    if current == "one value off":
        cx[20] += 0.5
    elif current == "last value off":
        cx[-1] += 3.0
    elif current == "shorter":
        cx = cx[:-1]
    depth = rng.uniform(3.0, 60.0, (n, n))
    u, v = rng.normal(0, 0.3, (2, n, cx.size))
    y = x.astype(np.float64)
    m = 200
    k, th = rng.uniform(0.02, 0.4, m), rng.uniform(0, 2 * np.pi, m)
    rays = (rng.uniform(5.0, 395.0, m), rng.uniform(5.0, 395.0, m), k * np.cos(th), k * np.sin(th))
    got = mr.trace(mr.Bathymetry.grid(x, x, depth), mr.Current.grid(cx, y, u, v), *rays, 12.0, 0.4)
    o = oracle.trace(oracle.Bathymetry.grid(x, x, depth), oracle.Current.grid(cx, y, u, v), *rays,
                     0.0, 12.0, 0.4)
    H.assert_parity(got.traj, got.n_rows, o[0], o[1])
    np.testing.assert_array_equal(got.status, o[2])
