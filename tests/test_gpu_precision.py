"""The kernels on float pairs against the FP64 kernels they stand in for: on
smooth fields, each output's error in norm at most 4 times the FP64 form's own
plus 2^-49 of its norm (8 units of FP64's rounding).  The differentiation form
against diff_reference.cpp (the FP64 kernels serve a call while it is captured),
the plain form against the oracle (the general kernel serves a depth array one
value short).  Pairs that lost their low halves would be off by 2^-24 a term."""

import numpy as np
import pytest

from tests.test_gpu_diff_split import _call, _reference, _tangent, reference  # noqa: F401

pytestmark = pytest.mark.gpu

NODES, SPACING, DT = 200, 200.0, 2.0


def _shelf(seed, n):
    rng = np.random.default_rng(seed)
    x = np.arange(NODES) * SPACING
    length = x[-1]
    X, Y = x[None, :], x[:, None]
    r2 = (X - 0.5 * length) ** 2 + (Y - 0.5 * length) ** 2
    depth = np.maximum(1500.0 - 1490.0 * X / length
                       - 700.0 * np.exp(-r2 / (2.0 * (0.08 * length) ** 2)), 5.0)
    u = np.broadcast_to(np.exp(-((Y - 0.5 * length) ** 2) / (2.0 * (0.05 * length) ** 2)),
                        depth.shape).copy()
    v = 0.2 * np.cos(X / 3000.0) * np.sin(Y / 2500.0)
    th, k = rng.uniform(-0.5, 0.5, n), 10.0 ** rng.uniform(-1.7, -1.0, n)
    rays = np.stack([np.full(n, 0.47 * length) + rng.uniform(0, 100.0, n),
                     length * rng.uniform(0.3, 0.7, n), k * np.cos(th), k * np.sin(th)])
    return rng, x, depth, u, v, rays


def _bounded(pairs, fp64, ref):
    norm = np.linalg.norm(ref)
    assert np.linalg.norm(pairs - ref) <= 4.0 * np.linalg.norm(fp64 - ref) + 2.0 ** -49 * norm


@pytest.mark.parametrize("seed,steps", [(1, 60), (2, 150)])
def test_adjoint_error(reference, seed, steps):  # noqa: F811
    import torch

    from mantaray_gb300 import _native
    from mantaray_gb300.diff import grid

    n = 400
    rng, x, depth, u, v, rays = _shelf(seed, n)
    g = grid(NODES, NODES, 0.0, 0.0, SPACING, SPACING)
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    grad_end = rng.standard_normal((4, n)) * [[1.0], [1.0], [1e3], [1e3]]
    args = (_native.load(), g, g, dev(depth), dev(u), dev(v), dev(rays), DT, steps, 13,
            dev(grad_end))
    pairs, fp64 = _call(*args, captured=False), _call(*args, captured=True)
    ref = _reference(reference, g, g, depth, u, v, rays, DT, steps, grad_end)
    for r in (pairs, fp64, ref):
        assert (r[1] == 0).all()
    assert not np.array_equal(pairs[2], fp64[2])  # the two forms
    for q in (0, 2):
        for part in (slice(0, 2), slice(2, 4)):
            _bounded(pairs[q][part], fp64[q][part], ref[q][part])
    for q in (3, 4, 5):
        _bounded(pairs[q], fp64[q], ref[q])


@pytest.mark.parametrize("seed,steps", [(3, 60), (4, 150)])
@pytest.mark.parametrize("along", ["state", "fields"])
def test_tangent_error(reference, seed, steps, along):  # noqa: F811
    import torch

    from mantaray_gb300.diff import grid, tangent

    n = 400
    rng, x, depth, u, v, rays = _shelf(seed, n)
    g = grid(NODES, NODES, 0.0, 0.0, SPACING, SPACING)
    ds = rng.standard_normal((4, n)) * [[1.0], [1.0], [1e-4], [1e-4]]
    fields = [None, None, None]
    if along == "fields":
        ds = np.zeros_like(ds)
        fields = [50.0 * np.exp(-(depth / 800.0) ** 2), 0.1 * u, 0.3 * v]
    dev = lambda a: None if a is None else torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    args = [dev(a) for a in rays] + [dev(depth), dev(u), dev(v)]
    rest = [dev(ds), *[dev(f) for f in fields]]

    def call():
        return tangent(*args, g, g, DT, steps, *rest)

    pairs = call()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        fp64 = call()
    graph.replay()
    torch.cuda.synchronize()
    pairs, fp64 = ([t.cpu().numpy() for t in r] for r in (pairs, fp64))
    end, status, d_end = _tangent(reference, g, g, depth, u, v, rays, DT, steps, ds, fields)
    assert (pairs[2] == 0).all() and (fp64[2] == 0).all() and (status == 0).all()
    assert not np.array_equal(pairs[1], fp64[1])
    for part in (slice(0, 2), slice(2, 4)):
        _bounded(pairs[0][part], fp64[0][part], end[part])
        _bounded(pairs[1][part], fp64[1][part], d_end[part])


@pytest.mark.parametrize("current", ["grid", "constant"])
def test_plain_error(oracle, current):
    import mantaray_gb300 as mr

    n = 300
    _, x, depth, u, v, rays = _shelf(5, n)
    x32 = x.astype(np.float32)
    make = {"grid": lambda m: m.Current.grid(x, x, u, v),
            "constant": lambda m: m.Current.constant(0.3, -0.2)}[current]
    time = (150 * DT, DT)
    pairs = mr.trace(mr.Bathymetry.grid(x32, x32, depth), make(mr), *rays, *time)
    general = mr.trace(mr.Bathymetry.grid(x32, x32, depth.ravel()[:-1]), make(mr), *rays, *time)
    ref = oracle.trace(oracle.Bathymetry.grid(x32, x32, depth), make(oracle), *rays, 0.0, *time)[0]
    assert np.isfinite(ref).all() and np.isfinite(pairs.traj).all()
    assert not np.array_equal(pairs.traj, general.traj)
    for part in (slice(1, 3), slice(3, 5)):
        _bounded(pairs.traj[part], general.traj[part], ref[part])
