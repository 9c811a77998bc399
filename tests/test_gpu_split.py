"""The plain form on gridded bathymetry (csrc/rk4_f64_grid.cu) against the
general kernel and the oracle, at the sizes and places where its dispatch and
its cell records can go wrong: cell edges and the ulps beside them, corners,
the grid's rim, rays leaving the grid, dry and NaN nodes, k = 0, gradients
outside the pairs' domain, the current's three forms, both stop rules, one
ray to a ragged block."""

import numpy as np
import pytest

from tests import helpers as H

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def mr():
    import mantaray_gb300 as m

    m._native.load()
    return m


def _points(axis, rng, n):
    """Grid lines and their neighbouring doubles, the rim, and random points."""
    out = []
    for a in axis[:: max(1, axis.size // 6)].tolist() + [float(axis[-1])]:
        out += [a, np.nextafter(a, -np.inf), np.nextafter(a, np.inf),
                a + 1e-6 * abs(a), a - 1e-6 * abs(a)]
    out += [float(axis[0]) - 0.01, float(axis[-1]) + 0.01]
    return np.concatenate([out, rng.uniform(axis[0], axis[-1], max(0, n - len(out)))])


def _case(form, nx, ny, sp, n, seed):
    rng = np.random.default_rng(seed)
    x = (np.float32(2.3) + np.float32(sp) * np.arange(nx, dtype=np.float32)).astype(np.float32)
    y = (np.float32(-7.7) + np.float32(0.9 * sp) * np.arange(ny, dtype=np.float32)).astype(np.float32)
    depth = rng.uniform(3.0, 60.0, (ny, nx))
    if form == "weird":  # dry, NaN, very deep and very steep nodes
        flat = depth.ravel()
        flat[rng.integers(0, flat.size, 3)] = -1.0
        flat[rng.integers(0, flat.size, 2)] = np.nan
        flat[rng.integers(0, flat.size, 2)] = 3e5
        flat[rng.integers(0, flat.size, 1)] = 1e9
    if form == "constant":
        cur = ("constant", 0.3, -0.2)
    else:
        cx, cy = x.astype(np.float64), y.astype(np.float64)
        if form == "other":
            cx = np.linspace(float(x[0]) - 1.0, float(x[-1]) + 1.0, nx + 3)
            cy = np.linspace(float(y[0]) - 1.0, float(y[-1]) + 1.0, ny + 1)
        cur = ("grid", cx, cy, rng.normal(0, 0.3, (cy.size, cx.size)),
               rng.normal(0, 0.3, (cy.size, cx.size)))
    px, py = _points(x, rng, n), _points(y, rng, n)
    x0 = np.concatenate([px, rng.uniform(x[0], x[-1], py.size), np.repeat(x, 3)[:9].astype(float)])
    y0 = np.concatenate([rng.uniform(y[0], y[-1], px.size), py, np.repeat(y, 3)[:9].astype(float)])
    m = min(x0.size, y0.size)
    keep = rng.permutation(m)[:n] if n < m else np.arange(m)
    x0, y0 = x0[keep], y0[keep]
    th = rng.choice([0.0, np.pi / 2, np.pi, -np.pi / 2, 0.7, 2.1, 4.0], x0.size)
    k = rng.uniform(0.02, 0.4, x0.size)
    if form == "weird" and n > 4:
        k[:2] = (0.0, 1e-9)
    return (x, y, depth), cur, (x0, y0, k * np.cos(th), k * np.sin(th))


def _current(m, spec):
    return m.Current.grid(*spec[1:]) if spec[0] == "grid" else m.Current.constant(*spec[1:])


@pytest.mark.parametrize("stop_rule", [0, 1])
@pytest.mark.parametrize("form", ["same", "other", "constant", "weird"])
@pytest.mark.parametrize("nx,ny,n", [(2, 2, 1), (3, 2, 31), (41, 37, 33), (64, 50, 517)])
def test_grid_kernel_against_general_and_oracle(mr, oracle, form, stop_rule, nx, ny, n):
    grid, cur, rays = _case(form, nx, ny, 10.0, n, 100 * nx + n)
    args = (25 * 0.4, 0.4)
    got = mr.trace(mr.Bathymetry.grid(*grid), _current(mr, cur), *rays, *args, stop_rule=stop_rule)
    o = oracle.trace(oracle.Bathymetry.grid(*grid), _current(oracle, cur), *rays, 0.0, args[0],
                     args[1], stop_rule=stop_rule)
    H.assert_parity(got.traj, got.n_rows, o[0], o[1])
    np.testing.assert_array_equal(got.status, o[2])
    if form == "weird":
        return
    # a depth array one value short takes the general kernel; rays that never
    # read the last cell have the same rows there
    short = mr.trace(mr.Bathymetry.grid(grid[0], grid[1], grid[2].ravel()[:-1]),
                     _current(mr, cur), *rays, *args, stop_rule=stop_rule)
    far = np.nanmax(np.where(np.isfinite(got.traj[1]), got.traj[1], -np.inf), axis=0) < grid[0][-2] - 3
    far &= np.all(np.isfinite(got.traj[1:, -1]), axis=0)
    if far.any():
        H.assert_parity(got.traj[:, :, far], got.n_rows[far], short.traj[:, :, far],
                        short.n_rows[far])


def test_grid_kernel_backward_in_time(mr, oracle):
    # t_end < t0 with a negative step is a positive number of steps
    grid, cur, rays = _case("same", 41, 37, 10.0, 65, 5)
    got = mr.trace(mr.Bathymetry.grid(*grid), _current(mr, cur), *rays, -6.0, -0.3, t0=2.0)
    o = oracle.trace(oracle.Bathymetry.grid(*grid), _current(oracle, cur), *rays, 2.0, -4.0, -0.3)
    H.assert_parity(got.traj, got.n_rows, o[0], o[1])
    np.testing.assert_array_equal(got.status, o[2])
