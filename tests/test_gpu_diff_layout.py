"""diff.tangent with tensors that are not contiguous: the same bits as with
contiguous ones."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", ["float64", "float32"])
@pytest.mark.parametrize("which", ["tangents", "rays and fields"])
def test_strided_tensors(dtype, which):
    import torch

    from mantaray_gb300.diff import grid, tangent

    n, nodes = 300, 64
    gen = torch.Generator(device="cuda").manual_seed(4)
    kw = {"generator": gen, "dtype": getattr(torch, dtype), "device": "cuda"}
    uni = lambda *s: torch.rand(*s, **kw)  # noqa: E731
    g = grid(nodes, nodes, 0.0, 0.0, 100.0, 100.0)
    depth, u, v = 20.0 + 30.0 * uni(nodes, nodes), uni(nodes, nodes), uni(nodes, nodes)
    rays = [2000.0 + 2000.0 * uni(n), 2000.0 + 2000.0 * uni(n), 0.05 + 0.1 * uni(n), 0.1 * uni(n)]
    tangents = [uni(n, 4).T, *[uni(nodes, 2 * nodes)[:, ::2] for _ in range(3)]]
    args = [*rays, depth, u, v]
    if which == "tangents":
        calls = [(args, tangents), (args, [t.contiguous() for t in tangents])]
    else:
        strided = [torch.stack([t, t], -1)[..., 0] for t in args]
        assert not any(t.is_contiguous() for t in strided)
        tangents = [t.contiguous() for t in tangents]
        calls = [(strided, tangents), (args, tangents)]
    a, b = (tangent(*s, g, g, 2.0, 20, *t) for s, t in calls)
    for p, q in zip(a, b):
        np.testing.assert_array_equal(p.cpu().numpy(), q.cpu().numpy())
