"""The batched kernel's capped and middle builds, taken when a call has more
rays than the uncapped one keeps resident, against the uncapped build on a call
that fits: the same rays, bit for bit, in both launch forms and table modes."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sweep", [0, 16])
@pytest.mark.parametrize("scenarios", [1, 2])
@pytest.mark.parametrize("lanes", [7 * 128, 7 * 128 + 1, 2048])
def test_capped_builds_agree(sweep, scenarios, lanes):
    import torch

    import mantaray_gb300 as mr
    from mantaray_gb300.batch import BatchTracer, make_config

    rng = np.random.default_rng(5)
    ax = np.arange(61) * 20.0
    fields = [(mr.Bathymetry.grid(ax.astype(np.float32), ax.astype(np.float32),
                                  rng.uniform(20.0, 60.0, (61, 61))),
               mr.Current.grid(ax, ax, rng.normal(0, 0.2, (61, 61)),
                               rng.normal(0, 0.2, (61, 61)))) for _ in range(scenarios)]
    few = 4099
    # per SM: what 72 registers hold (7 blocks of 128), one more, and beyond any
    # residency
    many = lanes * torch.cuda.get_device_properties(0).multi_processor_count
    th, k = rng.uniform(0, 2 * np.pi, few), rng.uniform(0.03, 0.3, few)
    rays = [rng.uniform(100, 1100, few), rng.uniform(100, 1100, few), k * np.cos(th),
            k * np.sin(th)]
    sid = rng.integers(0, scenarios, few).astype(np.uint8)
    tracer = BatchTracer(fields)
    cfg = make_config(128, 16, 1, 32, 1, 0, sweep)

    def ends(n):
        dev = [torch.from_numpy(np.resize(a, n)).cuda() for a in rays]
        kw = {"scenario": torch.from_numpy(np.resize(sid, n)).cuda()} if scenarios > 1 else {}
        r = tracer.trace(*dev, 0.5, 40, config=cfg, **kw)
        return r.end_state.cpu().numpy()[:, :few], r.n_steps.cpu().numpy()[:few]

    for a, b in zip(ends(few), ends(many)):
        np.testing.assert_array_equal(a, b)
