"""What an FP64 differentiation call leaves behind on the device."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_records_are_given_back():
    # also after mr_trace, which has the device's default pool keep what is
    # freed: the records of 2,048^2 cells (0.8 GB) are not kept with it
    import torch

    import mantaray_gb300 as mr
    from mantaray_gb300.diff import grid, tangent

    ax = np.arange(64) * 100.0
    mr.trace(mr.Bathymetry.grid(ax.astype(np.float32), ax.astype(np.float32), np.full((64, 64), 50.0)),
             mr.Current.constant(0.1, 0.0), *[np.full(4, q) for q in (100.0, 100.0, 0.1, 0.0)],
             10.0, 1.0)
    nodes = 2049
    g = grid(nodes, nodes, 0.0, 0.0, 100.0, 100.0)
    depth = torch.full((nodes, nodes), 50.0, dtype=torch.float64, device="cuda")
    u = torch.zeros_like(depth)
    rays = [torch.full((64,), q, dtype=torch.float64, device="cuda") for q in (1e5, 1e5, 0.1, 0.0)]

    def call():
        tangent(*rays, depth, u, u, g, g, 2.0, 300)
        torch.cuda.synchronize()
        return torch.cuda.mem_get_info()[0]

    tangent(*rays, depth[:64, :64].contiguous(), u[:64, :64].contiguous(), u[:64, :64].contiguous(),
            grid(64, 64, 1e5 - 3000.0, 1e5 - 3000.0, 100.0, 100.0),
            grid(64, 64, 1e5 - 3000.0, 1e5 - 3000.0, 100.0, 100.0), 2.0, 300)
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    assert free - call() < 100 << 20
