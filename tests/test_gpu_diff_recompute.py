"""The backward pass where its recomputed states are not the forward's: a ray
that the forward completed may, by rounding, be outside a grid in the
recomputation.  Checkpoints outside the grid, dry and NaN stand for it: the walk
backward ends there, with the gradient it had come to, and no node gets any.
In both FP64 routes (while captured the FP64 kernels serve) and
in FP32."""

import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _backward(dtype, ck, status, grad_end, steps, every, captured):
    import torch

    from mantaray_gb300 import _native
    from mantaray_gb300.diff import grid

    lib = _native.load()
    n = ck.shape[2]
    g = grid(40, 30, 0.0, 0.0, 100.0, 100.0)
    rng = np.random.default_rng(0)
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    depth = rng.uniform(20.0, 40.0, (30, 40))
    depth[20:, 20:] = -1.0
    fields = [dev(a.astype(dtype)) for a in (depth, *rng.normal(0.0, 0.3, (2, 30, 40)))]
    ck, grad_end, status = dev(ck.astype(dtype)), dev(grad_end.astype(dtype)), dev(status)
    seg = torch.zeros((every, 16, n), dtype=ck.dtype, device="cuda")
    g0 = torch.full((4, n), 7.0, dtype=ck.dtype, device="cuda")
    nodes = [torch.full((30, 40), 7.0, dtype=torch.float64, device="cuda") for _ in range(3)]
    p = lambda t: t.data_ptr()  # noqa: E731

    def run():
        assert lib.mr_diff_backward(
            64 if dtype == np.float64 else 32, ctypes.byref(g), p(fields[0]), ctypes.byref(g),
            p(fields[1]), p(fields[2]), n, *[p(ck[0, q]) for q in range(4)], 2.0, steps, every,
            p(ck), p(status), p(grad_end), p(seg), p(g0), *[p(t) for t in nodes],
            torch.cuda.current_stream().cuda_stream) == 0

    torch.cuda.synchronize()
    if captured:
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            run()
        graph.replay()
    else:
        run()
    torch.cuda.synchronize()
    return g0.cpu().numpy(), [t.cpu().numpy() for t in nodes]


@pytest.mark.parametrize("dtype,captured", [(np.float64, False), (np.float64, True),
                                            (np.float32, False)])
@pytest.mark.parametrize("every", [1, 4, 9])
def test_states_without_a_derivative(dtype, captured, every):
    n, steps = 70, 9
    n_ck = (steps + every - 1) // every
    rng = np.random.default_rng(every)
    ck = np.empty((n_ck, 4, n))
    ck[:, 0], ck[:, 1], ck[:, 2], ck[:, 3] = 500.0, 500.0, 0.1, 0.05
    bad = np.arange(n) % 7
    ck[:, 0, bad == 0] = -1e-9
    ck[:, 0, bad == 1] = 3900.0 + 1e-3
    ck[:, 1, bad == 2] = 1e300 if dtype == np.float64 else 1e30
    ck[:, :2, bad == 3] = 2500.0  # dry
    ck[:, 0, bad == 4] = np.nan
    ck[:, 2:, bad == 5] = 0.0
    status = np.zeros(n, dtype=np.uint8)
    status[bad == 6] = 1
    grad_end = rng.standard_normal((4, n))
    g0, nodes = _backward(dtype, ck, status, grad_end, steps, every, captured)
    np.testing.assert_array_equal(g0[:, bad < 6], grad_end.astype(dtype)[:, bad < 6])
    assert (g0[:, bad == 6] == 0.0).all()
    for a in nodes:
        np.testing.assert_array_equal(a, 0.0)


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
def test_states_at_the_edge(dtype):
    # within a step of the rim, where some stages have a derivative and some not
    n, steps = 257, 1
    rng = np.random.default_rng(1)
    a = np.linspace(0.0, 2.0 * np.pi, n)
    ck = np.stack([3900.0 - 30.0 * rng.random(n), 500.0 + 300.0 * rng.random(n), 0.1 * np.cos(a),
                   0.1 * np.sin(a)])[None]
    grad_end = rng.standard_normal((4, n))
    out = [_backward(dtype, ck, np.zeros(n, dtype=np.uint8), grad_end, steps, 1, captured)
           for captured in (False, True)]
    for g0, nodes in out:
        assert np.isfinite(g0).all() and all(np.isfinite(t).all() for t in nodes)
        assert (nodes[0][:, 35:] != 0.0).any() and (nodes[0][:, :30] == 0.0).all()
    tol = 1e-9 if dtype == np.float64 else 0.0
    np.testing.assert_allclose(out[0][0], out[1][0], rtol=tol, atol=tol)
