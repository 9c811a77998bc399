"""The FP64 tangent-linear form where the tangents of one call span many
scales: a node of a tangent field far from every ray, one ray's initial
tangent among others', components and fields decades apart.  Against
diff_reference.cpp, each ray's tangent over the ray's own scale, with the
bound of test_gpu_diff_split.py (100 s 2^-45 in norm for s steps)."""

import numpy as np
import pytest

from tests.test_gpu_diff_split import _case, _tangent, reference  # noqa: F401

pytestmark = pytest.mark.gpu

STEPS = 40


def _d_end(g, c, depth, u, v, rays, ds, fields):
    import torch

    from mantaray_gb300.diff import tangent

    dev = lambda a: None if a is None else torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    end, d_end, status = tangent(*dev(rays), dev(depth), dev(u), dev(v), g, c, 5.0, STEPS,
                                 dev(ds), *[dev(f) for f in fields])
    return d_end.cpu().numpy(), status.cpu().numpy()


def _compare(reference, case, ds, fields, scale=1.0):
    """scale: of each ray's tangent (the equations are linear in it)."""
    _, g, c, depth, u, v, rays = case
    got, status = _d_end(g, c, depth, u, v, rays, ds, fields)
    ref = _tangent(reference, g, c, depth, u, v, rays, 5.0, STEPS, ds, fields)
    np.testing.assert_array_equal(status, ref[1])
    ok = status == 0
    assert ok.sum() > status.size // 4
    scale = np.broadcast_to(scale, ok.shape)[ok]
    assert np.isfinite(got[:, ok]).all()
    for q in (slice(0, 2), slice(2, 4)):
        r = ref[2][q][:, ok] / scale
        assert np.linalg.norm(got[q][:, ok] / scale - r) <= 100 * STEPS * 2.0 ** -45 * np.linalg.norm(r)
    return ok


def _inner(n, same):
    """Rays that cannot reach the grids' first cell: below 71 m of water and
    currents of 2 m/s they travel 5.7 km at most."""
    rng, g, c, depth, u, v, rays = _case(n, STEPS, "mixed", same)
    keep = np.hypot(rays[0] + 1000.0, rays[1] - 300.0) > 6500.0
    return rng, g, c, depth, u, v, rays[:, keep]


@pytest.mark.parametrize("same", [True, False])
@pytest.mark.parametrize("node", [9.97e36, 1e20, 1e200, -1e-300])
@pytest.mark.parametrize("field", [0, 1, 2])
def test_one_node_far_away(reference, same, node, field):  # noqa: F811
    case = _inner(600, same)
    rng, _, _, depth, u, v, rays = case
    fields = [10.0 * rng.standard_normal(depth.shape), *(0.1 * rng.standard_normal((2, *u.shape)))]
    fields[field][0, 0] = node
    _compare(reference, case, np.zeros_like(rays), fields)


@pytest.mark.parametrize("same", [True, False])
@pytest.mark.parametrize("size", [1e46, 1e300, 1e-46])
def test_one_ray_of_another_scale(reference, same, size):  # noqa: F811
    case = _inner(600, same)
    rng, rays = case[0], case[6]
    scale = np.ones(rays.shape[1])
    scale[::97] = size
    ds = np.array([[1.0], [1.0], [1e-4], [1e-4]]) * rng.standard_normal(rays.shape) * scale
    _compare(reference, case, ds, [None] * 3, scale)


@pytest.mark.parametrize("same", [True, False])
def test_one_ray_with_a_state_among_others_without(reference, same):  # noqa: F811
    case = _inner(600, same)
    rng, _, _, depth, u, v, rays = case
    ds, scale = np.zeros_like(rays), np.ones(rays.shape[1])
    ds[:, 5], scale[5] = 1e46, 1e46
    fields = [10.0 * rng.standard_normal(depth.shape), *(0.1 * rng.standard_normal((2, *u.shape)))]
    _compare(reference, case, ds, fields, scale)


def test_every_ray_of_its_own_scale(reference):  # noqa: F811
    case = _inner(600, True)
    rng, rays = case[0], case[6]
    scale = 10.0 ** rng.uniform(-60.0, 60.0, rays.shape[1])
    ds = np.array([[1.0], [1.0], [1e-4], [1e-4]]) * rng.standard_normal(rays.shape) * scale
    _compare(reference, case, ds, [None] * 3, scale)


@pytest.mark.parametrize("dk", [1e-12, 1e-20, 1e-30, 0.0])
def test_components_of_different_scales(reference, dk):  # noqa: F811
    case = _inner(600, True)
    rng, rays = case[0], case[6]
    ds = np.array([[1.0], [1.0], [dk], [dk]]) * rng.standard_normal(rays.shape)
    _compare(reference, case, ds, [None] * 3)


@pytest.mark.parametrize("size", [1e-10, 1e-16, 1e-25, 1e25])
def test_small_and_large_fields(reference, size):  # noqa: F811
    # alone, and beside a state tangent of order 1
    case = _inner(600, False)
    rng, _, _, depth, u, v, rays = case
    fields = [10.0 * size * rng.standard_normal(depth.shape),
              *(0.1 * size * rng.standard_normal((2, *u.shape)))]
    _compare(reference, case, np.zeros_like(rays), fields)
    ds = np.array([[1.0], [1.0], [1e-4], [1e-4]]) * rng.standard_normal(rays.shape)
    _compare(reference, case, ds, fields)
