"""The FP64 differentiation kernels on float pairs against the same model in
long double (diff_reference.cpp), and their stopped rays against the FP64
kernels', which serve the call while its stream is being captured.

Tolerances, for s steps: the state is rounded to FP64 once a step (2^-53 of
components up to 3e4 m), and the paths amplify that by up to G, measured on the
reference with starts moved by 2^-40, so end states differ by less than 10 s G
2^-52 of the largest component (G = 1 where they contract); the pairs' terms of the gradients carry 2^-45 each step and follow the states' difference,
so the gradients differ by less than 100 s 2^-45 in norm (s = 40: 1.2e-10)."""

import ctypes
import os
import shutil
import subprocess
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _fields(rng, nx, ny, kind):
    y, x = np.mgrid[0:ny, 0:nx]
    d = 40.0 + 30.0 * np.sin(0.5 * x + 1.0) * np.cos(0.4 * y) + rng.uniform(-1, 1, (ny, nx))
    if kind == "shallow":   # down to the pairs' least depth, and dry
        d = np.abs(d - 40.0) * 0.02 - 0.02
    elif kind == "deep":    # kh from 1 to beyond exp(-2 kh)'s range
        d = d * np.where(x > nx // 2, 200.0, 1.0)
    elif kind == "nan":
        d[ny // 2, nx // 2] = np.nan
    return d


@pytest.fixture(scope="module")
def reference(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("needs g++")
    so = str(tmp_path_factory.mktemp("ref") / "diff_reference.so")
    src = os.path.join(os.path.dirname(os.path.abspath(__file__)), "diff_reference.cpp")
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-o", so, src], check=True)
    return ctypes.CDLL(so)


def _reference(lib, g, c, depth, u, v, rays, dt, steps, grad_end):
    n = rays.shape[1]
    p = lambda a: a.ctypes.data_as(ctypes.c_void_p)  # noqa: E731
    nodes = np.array([g.nx, g.ny, c.nx, c.ny], dtype=np.int64)
    geom = np.array([g.x0, g.y0, g.dx, g.dy, c.x0, c.y0, c.dx, c.dy])
    end, status, g0 = np.empty((4, n)), np.empty(n, dtype=np.uint8), np.empty((4, n))
    cuts = np.linspace(0, n, 9).astype(int)
    parts = [[np.zeros_like(a) for a in (depth, u, v)] for _ in cuts[1:]]
    rays, grad_end = np.ascontiguousarray(rays), np.ascontiguousarray(grad_end)

    def run(i):
        lib.adjoint(p(nodes), p(geom), p(depth), p(u), p(v), ctypes.c_double(dt),
                    *[ctypes.c_int64(int(q)) for q in (steps, n, cuts[i], cuts[i + 1])], p(rays),
                    p(grad_end), p(end), p(status), p(g0), *[p(a) for a in parts[i]])

    with ThreadPoolExecutor(8) as pool:
        list(pool.map(run, range(8)))
    return [end, status, g0, *[sum(a[q] for a in parts) for q in range(3)]]


def _check(got, ref, moved, steps, size):
    np.testing.assert_array_equal(got[1], ref[1])
    ok = ref[1] == 0
    assert np.isnan(got[0][:, ~ok]).all() and (got[2][:, ~ok] == 0.0).all()
    _check_states(got, ref, moved, steps)
    assert np.isfinite(got[2]).all()
    for e, r in zip(got[2:], ref[2:]):
        norm = np.linalg.norm(r / size)
        assert np.linalg.norm((e - r) / size) <= 100 * steps * 2.0 ** -45 * norm


def _check_states(got, ref, moved, steps):
    ok = ref[1] == 0
    for q in (slice(0, 2), slice(2, 4)):  # positions, wavenumbers
        err = np.abs(got[0][q][:, ok] - ref[0][q][:, ok])
        big = np.abs(ref[0][q][:, ok])
        if err.size:
            growth = np.nanmax(np.abs(moved[0][q][:, ok] - ref[0][q][:, ok])) * 2.0 ** 40 / big.max()
            assert err.max() <= 10 * steps * max(growth, 1.0) * 2.0 ** -52 * big.max()


def _tangent(lib, g, c, depth, u, v, rays, dt, steps, ds, fields):
    n = rays.shape[1]
    p = lambda a: None if a is None else a.ctypes.data_as(ctypes.c_void_p)  # noqa: E731
    nodes = np.array([g.nx, g.ny, c.nx, c.ny], dtype=np.int64)
    geom = np.array([g.x0, g.y0, g.dx, g.dy, c.x0, c.y0, c.dx, c.dy])
    end, status, d_end = np.empty((4, n)), np.empty(n, dtype=np.uint8), np.empty((4, n))
    cuts = np.linspace(0, n, 9).astype(int)
    rays, ds = np.ascontiguousarray(rays), np.ascontiguousarray(ds)

    def run(i):
        lib.tangent(p(nodes), p(geom), p(depth), p(u), p(v), ctypes.c_double(dt),
                    *[ctypes.c_int64(int(q)) for q in (steps, n, cuts[i], cuts[i + 1])], p(rays),
                    p(ds), *[p(f) for f in fields], p(end), p(status), p(d_end))

    with ThreadPoolExecutor(8) as pool:
        list(pool.map(run, range(8)))
    return [end, status, d_end]


def _call(lib, g, c, depth, u, v, rays, dt, steps, every, grad_end, captured):
    import torch

    n = rays.shape[1]
    dev = "cuda"
    n_ck = (steps + every - 1) // every
    new = lambda *s: torch.full(s, 7.0, dtype=torch.float64, device=dev)  # noqa: E731
    ck, end, status = new(n_ck, 4, n), new(4, n), torch.zeros(n, dtype=torch.uint8, device=dev)
    seg, g0 = new(every, 16, n), new(4, n)
    grads = [new(*depth.shape), new(*u.shape), new(*u.shape)]
    p = lambda t: t.data_ptr()  # noqa: E731

    def run(stream):
        head = (64, ctypes.byref(g), p(depth), ctypes.byref(c), p(u), p(v), n,
                *[p(r) for r in rays], dt, steps, every)
        assert lib.mr_diff_forward(*head, p(ck), p(end), p(status), stream) == 0
        assert lib.mr_diff_backward(*head, p(ck), p(status), p(grad_end), p(seg), p(g0),
                                    *[p(t) for t in grads], stream) == 0

    torch.cuda.synchronize()
    if captured:
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            run(torch.cuda.current_stream().cuda_stream)
        graph.replay()
    else:
        run(torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    return [t.cpu().numpy() for t in (end, status, g0, *grads)]


def _case(n, steps, kind, same):
    from mantaray_gb300.diff import grid

    rng = np.random.default_rng(n + steps)
    nx, ny = (5, 4) if n == 1 else (33, 21)
    dx = 500.0
    g = grid(nx, ny, -1000.0, 300.0, dx, dx)
    cx, cy = (nx, ny) if same else (nx - 1, ny + 1)
    c = g if same else grid(cx, cy, -1000.0, 300.0 - 0.25 * dx, dx * 1.03125, dx)
    depth = _fields(rng, nx, ny, kind)
    u, v = 0.6 * rng.standard_normal((2, cy, cx))
    x = rng.uniform(-1000.0, -1000.0 + (nx - 1) * dx, n)
    y = rng.uniform(300.0, 300.0 + (ny - 1) * dx, n)
    k = 10.0 ** rng.uniform(-2.0, -0.3, n)
    a = rng.uniform(0.0, 2.0 * np.pi, n)
    if n >= 33:
        x[:4] = [-1000.0, -1000.0 + (nx - 1) * dx, -1000.0 + 3 * dx, np.nan]  # edges, a grid line
        y[:3] = [300.0 + 2 * dx, 300.0 + (ny - 1) * dx, 300.0 + 5 * dx]
        k[4:6] = [0.0, 1e4]
    return rng, g, c, depth, u, v, np.stack([x, y, k * np.cos(a), k * np.sin(a)])


@pytest.mark.parametrize("n,steps,every", [(1, 1, 1), (33, 7, 3), (64, 40, 40), (1000, 40, 7)])
@pytest.mark.parametrize("kind", ["mixed", "shallow", "deep", "nan"])
@pytest.mark.parametrize("same", [True, False])
@pytest.mark.parametrize("size", [1.0, 1e-40, 1e60])
def test_adjoint_on_pairs(reference, n, steps, every, kind, same, size):
    import torch

    from mantaray_gb300 import _native

    rng, g, c, depth, u, v, rays = _case(n, steps, kind, same)
    t = lambda q: torch.from_numpy(np.ascontiguousarray(q)).cuda()  # noqa: E731
    rays = t(rays)
    grad_end = t(np.stack([rng.standard_normal((2, n)), 1e3 * rng.standard_normal((2, n))])
                 .reshape(4, n) * size)
    if n >= 33:
        grad_end[:, 7] = 0.0
    args = (_native.load(), g, c, t(depth), t(u), t(v), rays, 5.0, steps, every, grad_end)
    got = _call(*args, captured=False)
    ref = _reference(reference, g, c, depth, u, v, rays.cpu().numpy(), 5.0, steps,
                     grad_end.cpu().numpy() / size)
    ref = ref[:2] + [r * size for r in ref[2:]]
    moved = _reference(reference, g, c, depth, u, v, rays.cpu().numpy() * (1 + 2.0 ** -40), 5.0,
                       steps, grad_end.cpu().numpy() / size)
    _check(got, ref, moved, steps, size)
    if kind != "shallow" and n >= 33:
        assert (ref[1] == 0).sum() > n // 4
    # the FP64 form serves the call while it is captured
    np.testing.assert_array_equal(_call(*args, captured=True)[1], got[1])


@pytest.mark.parametrize("n,steps", [(1, 1), (33, 7), (1000, 40)])
@pytest.mark.parametrize("kind", ["mixed", "shallow", "deep", "nan"])
@pytest.mark.parametrize("same", [True, False])
@pytest.mark.parametrize("along", ["state", "depth", "all", "inf"])
@pytest.mark.parametrize("size", [1.0, 1e-40])
def test_tangent_on_pairs(reference, n, steps, kind, same, along, size):
    import torch

    from mantaray_gb300 import _native

    rng, g, c, depth, u, v, rays = _case(n, steps, kind, same)
    ds = np.array([[1.0], [1.0], [1e-4], [1e-4]]) * rng.standard_normal((4, n)) * size
    fields = [10.0 * size * rng.standard_normal(depth.shape),
              *(0.1 * size * rng.standard_normal((2, *u.shape)))]
    if along == "state":
        fields = [None, None, None]
    elif along == "depth":
        ds, fields = 0.0 * ds, [fields[0], None, None]
    elif along == "inf":    # one current field, a node of it infinite
        fields = [None, None, fields[2]]
        fields[2][1, 1] = np.inf
    lib = _native.load()
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    d_args = [dev(a) for a in (depth, u, v, rays, ds)]
    d_fields = [None if f is None else dev(f) for f in fields]
    p = lambda a: None if a is None else a.data_ptr()  # noqa: E731

    def call(captured):
        out = [torch.full((4, n), 7.0, dtype=torch.float64, device="cuda") for _ in range(2)]
        status = torch.zeros(n, dtype=torch.uint8, device="cuda")

        def run(stream):
            assert lib.mr_diff_tangent(
                64, ctypes.byref(g), p(d_args[0]), ctypes.byref(c), p(d_args[1]), p(d_args[2]), n,
                *[p(r) for r in d_args[3]], p(d_args[4]), *[p(f) for f in d_fields], 5.0, steps,
                p(out[0]), p(out[1]), p(status), stream) == 0

        torch.cuda.synchronize()
        if captured:
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph):
                run(torch.cuda.current_stream().cuda_stream)
            graph.replay()
        else:
            run(torch.cuda.current_stream().cuda_stream)
        torch.cuda.synchronize()
        return out[0].cpu().numpy(), status.cpu().numpy(), out[1].cpu().numpy()

    got, fp64 = call(False), call(True)
    np.testing.assert_array_equal(got[1], fp64[1])
    ok = got[1] == 0
    assert np.isnan(got[0][:, ~ok]).all() and np.isnan(got[2][:, ~ok]).all()
    np.testing.assert_array_equal(np.isnan(got[2]), np.isnan(fp64[2]))
    if along == "inf":
        return
    ref = _tangent(reference, g, c, depth, u, v, rays, 5.0, steps, ds, fields)
    np.testing.assert_array_equal(got[1], ref[1])
    if ok.any():
        err = np.linalg.norm(got[2][:, ok] / size - ref[2][:, ok] / size)
        assert err <= 100 * steps * 2.0 ** -45 * np.linalg.norm(ref[2][:, ok] / size)
        _check_states(got, ref, _tangent(reference, g, c, depth, u, v, rays * (1 + 2.0 ** -40), 5.0,
                                         steps, ds, fields), steps)
