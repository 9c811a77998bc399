"""Calls of few steps on large grids, where filling the records costs more than
pairs save, and of grids too large for records, take the FP64 kernels: the same
bits as while the stream is captured, when the FP64 kernels always serve.  One
step past the line the pairs serve, with other low bits."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nodes,steps,fp64", [(600, 1, True), (1024, 10, True), (1024, 40, False),
                                              (4098, 300, True), (200, 1, True),
                                              (200, 4, False)])
def test_route(nodes, steps, fp64):
    import torch

    from mantaray_gb300.diff import grid, tangent

    dev = "cuda"
    gen = torch.Generator(device=dev).manual_seed(nodes)
    uni = lambda *s: torch.rand(*s, generator=gen, dtype=torch.float64, device=dev)  # noqa: E731
    g = grid(nodes, nodes, 0.0, 0.0, 100.0, 100.0)
    depth, u, v = 20.0 + 30.0 * uni(nodes, nodes), uni(nodes, nodes), uni(nodes, nodes)
    n, mid = 100, 50.0 * nodes
    rays = [mid + 100.0 * uni(n), mid + 100.0 * uni(n), 0.05 + 0.1 * uni(n), 0.1 * uni(n)]
    ds = torch.ones((4, n), dtype=torch.float64, device=dev)

    def call():
        return tangent(*rays, depth, u, v, g, g, 2.0, steps, dstate0=ds)

    a = call()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        b = call()
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(a[2], b[2])
    same = all(torch.equal(p, q) for p, q in zip(a[:2], b[:2]))
    assert same == fp64
    np.testing.assert_allclose(a[1].cpu().numpy(), b[1].cpu().numpy(), rtol=1e-6, atol=1e-9)
