"""The batched kernel's builds for axes of more than 2^22 points, with the
current on the bathymetry's grid and over two scenarios, against the narrow
builds on the same cells one point shorter: bit for bit, in every launch form."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def fields():
    import mantaray_gb300 as mr

    rng = np.random.default_rng(3)
    wide, ny = (1 << 22) + 1, 3
    x, y = np.arange(wide, dtype=np.float32), np.arange(ny, dtype=np.float32) * np.float32(50.0)
    out = {}
    depth, u = np.full((ny, wide), 40.0), np.zeros((ny, wide))
    for i in (0, wide - 4000):
        depth[:, i:i + 1000] = rng.uniform(5.0, 60.0, (ny, 1000))
        u[:, i:i + 1000] = rng.normal(0.0, 0.3, (ny, 1000))
    for n in (wide - 1, wide):
        xn = x[:n].astype(np.float64)
        out[n] = (mr.Bathymetry.grid(x[:n], y, depth[:, :n]),
                  mr.Current.grid(xn, y.astype(np.float64), u[:, :n], -u[:, :n]))
    return wide, out


@pytest.mark.parametrize("scenarios", ["grid", "grid+grid", "grid+constant"])
def test_wide_builds_agree_with_narrow_ones(fields, scenarios):
    import torch

    import mantaray_gb300 as mr
    from mantaray_gb300.batch import BatchTracer, make_config

    wide, by_length = fields
    rng = np.random.default_rng(len(scenarios))
    n = 300
    x0 = np.concatenate([rng.uniform(0, 900, 150), rng.uniform(wide - 3990, wide - 3100, 146),
                         [-1.0, np.nan, 5e6, 1e30]])
    th, k = rng.uniform(0, 2 * np.pi, n), rng.uniform(0.05, 0.5, n)
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    rays = [dev(a) for a in (x0, rng.uniform(0.0, 100.0, n), k * np.cos(th), k * np.sin(th))]
    kw = {}
    if "+" in scenarios:
        kw["scenario"] = dev((np.arange(n) % 2).astype(np.uint8))
    tracers = []
    for length in (wide - 1, wide):
        b, c = by_length[length]
        second = {"grid+grid": [(b, c)], "grid+constant": [(b, mr.Current.constant(0.2, -0.1))]}
        tracers.append(BatchTracer([(b, c)] + second.get(scenarios, [])))
    for cfg in (make_config(128, 2), make_config(128, 16), make_config(64, 4, 2),
                make_config(128, 4, 1, 32, 1, 0, 9), make_config(128, 16, 1, 32, 1, 0, 9)):
        a, b = (t.trace(*rays, 0.25, 60, decimation=7, config=cfg, **kw) for t in tracers)
        for name in ("end_state", "n_steps", "n_saved", "status", "saved"):
            p, q = (np.nan_to_num(getattr(r, name).cpu().numpy(), nan=-7.0) for r in (a, b))
            np.testing.assert_array_equal(p, q, err_msg=name)
    assert len(np.unique(a.status.cpu().numpy())) >= 2


def test_wide_builds_follow_the_launch_shape(fields):
    # many rays at 16 blocks per SM run a capped build, few the uncapped one:
    # the same rays, bit for bit
    import torch

    from mantaray_gb300.batch import BatchTracer, make_config

    wide, by_length = fields
    tracer = BatchTracer([by_length[wide]])
    few = 1000
    many = 2048 * torch.cuda.get_device_properties(0).multi_processor_count
    rng = np.random.default_rng(9)
    th, k = rng.uniform(0, 2 * np.pi, few), rng.uniform(0.05, 0.5, few)
    rays = [rng.uniform(0, 900, few), rng.uniform(0.0, 100.0, few), k * np.cos(th), k * np.sin(th)]
    cfg = make_config(128, 16)
    ends = []
    for n in (few, many):
        r = tracer.trace(*[torch.from_numpy(np.resize(a, n)).cuda() for a in rays], 0.25, 40,
                         config=cfg)
        ends.append(r.end_state.cpu().numpy()[:, :few])
    np.testing.assert_array_equal(*ends)
