"""The batched kernel's modes against one another, bit for bit: the same rays
through the build whose scenarios share one geometry, the one that reads each
scenario's, and the single-scenario one, in every launch form; and through
the build for axes of more than 2^22 points, whose cell location converts
where the others add, at grid lines, outside the grid and at NaN."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def mr():
    import mantaray_gb300 as m

    m._native.load()
    return m


def _dev(*arrays):
    import torch

    return [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in arrays]


def _same(a, b, label):
    for name in ("end_state", "n_steps", "n_saved", "status", "saved"):
        x, y = (np.nan_to_num(getattr(r, name).cpu().numpy(), nan=-7.0) for r in (a, b))
        np.testing.assert_array_equal(x, y, err_msg=f"{label} {name}")


def _configs():
    from mantaray_gb300.batch import make_config

    return {"uncapped": make_config(128, 2), "capped": make_config(128, 16),
            "two rays": make_config(64, 4, 2), "ahead": make_config(128, 4, 1, 32, 1, 2),
            "sweeps": make_config(128, 4, 1, 32, 1, 0, 7),
            "capped sweeps": make_config(128, 16, 1, 32, 1, 0, 16)}


@pytest.mark.parametrize("n", [1, 33, 4099])
def test_table_modes_agree(mr, n):
    from mantaray_gb300.batch import BatchTracer

    rng = np.random.default_rng(n)
    ax = np.arange(61) * 20.0

    def scenario(points):
        y = np.arange(points) * 20.0
        b = mr.Bathymetry.grid(ax.astype(np.float32), y.astype(np.float32),
                               rng.uniform(20.0, 60.0, (points, 61)))
        return b, mr.Current.grid(ax, y, rng.normal(0, 0.2, (points, 61)),
                                  rng.normal(0, 0.2, (points, 61)))

    s0, s1, other = scenario(61), scenario(61), scenario(47)
    th = rng.uniform(0, 2 * np.pi, n)
    k = rng.uniform(0.03, 0.3, n)
    rays = _dev(rng.uniform(100, 1100, n), rng.uniform(100, 1100, n), k * np.cos(th),
                k * np.sin(th))
    sid = rng.integers(0, 2, n).astype(np.uint8)
    (dsid,) = _dev(sid)
    one_geometry = BatchTracer([s0, s1])
    two_geometries = BatchTracer([s0, s1, other])
    for label, cfg in _configs().items():
        a = one_geometry.trace(*rays, 0.5, 90, decimation=20, scenario=dsid, config=cfg)
        _same(a, two_geometries.trace(*rays, 0.5, 90, decimation=20, scenario=dsid, config=cfg),
              label)
        for s, tracer in enumerate((BatchTracer([s0]), BatchTracer([s1]))):
            one = tracer.trace(*rays, 0.5, 90, decimation=20, config=cfg)
            idx = np.flatnonzero(sid == s)
            np.testing.assert_array_equal(a.end_state.cpu().numpy()[:, idx],
                                          one.end_state.cpu().numpy()[:, idx], err_msg=label)


def test_wide_axes_agree_with_narrow_ones(mr):
    from mantaray_gb300.batch import BatchTracer, make_config

    rng = np.random.default_rng(3)
    wide, ny = (1 << 22) + 1, 3
    x = np.arange(wide, dtype=np.float32)
    y = np.arange(ny, dtype=np.float32) * np.float32(50.0)
    depth = np.full((ny, wide), 40.0)
    for i in (0, 3000, wide - 4000):
        depth[:, i:i + 1000] = rng.uniform(5.0, 60.0, (ny, 1000))
    depth[1, 3300] = np.nan
    depth[:, 3500] = -1.0
    current = mr.Current.constant(0.2, -0.1)
    tracers = [BatchTracer([(mr.Bathymetry.grid(x[:n], y, depth[:, :n]), current)])
               for n in (wide - 1, wide)]
    n = 300
    x0 = np.concatenate([rng.uniform(0, 900, 100), np.arange(3000, 3090, dtype=float),
                         rng.uniform(wide - 3900, wide - 3100, 100),
                         [0.0, -1.0, -1e-30, 1e30, -1e30, np.nan, 5e6, 900.0, 900.0, 900.0]])
    y0 = rng.uniform(0.0, 100.0, n)
    y0[::7] = 50.0
    y0[-3:] = (np.nan, 1e12, -0.0)
    th = rng.choice([0.0, np.pi, 0.4, 2.5, 4.0], n)
    k = rng.uniform(0.05, 0.5, n)
    k[:3] = (0.0, 1e25, 1e-12)
    rays = _dev(x0, y0, k * np.cos(th), k * np.sin(th))
    for cfg in (make_config(128, 2), make_config(128, 16), make_config(64, 4, 2),
                make_config(128, 4, 1, 32, 1, 0, 9)):
        a, b = (t.trace(*rays, 0.25, 60, decimation=7, config=cfg) for t in tracers)
        _same(a, b, "wide")
    assert len(np.unique(a.status.cpu().numpy())) >= 3
