"""What a program has this package do, as measurable cases.

Four kinds of work, each through the package's own entry points:

* ``plain``    the FP64 drop-in: ``single_ray`` / ``ray_tracing`` (host arrays
  in, dataset out) and ``trace_device`` (resident buffers, full trajectories);
* ``batched``  the FP32 form: ``BatchTracer.trace`` and a captured
  ``BatchGraph`` over one or several scenarios;
* ``diff``     ray endpoints with their gradients (``ray_endpoints`` and a
  backward pass), or the tangent-linear form, in FP64 or FP32;
* ``seed``     initial states of point sources, made on the device.

Fields, spacings, steps and ray distributions are those of the package's
workloads and tests: a planar beach, a Gaussian seamount in a uniform current,
a shelf with a shoal and a jet, shoals with vortices, and a shelf slope with
rough topography.  Everything is made from the seed alone.
"""

import math

import numpy as np
import torch
import torch.utils.checkpoint

import mantaray_gb300 as mr
from mantaray_gb300 import batch as mr_batch
from mantaray_gb300 import diff as mr_diff
from mantaray_gb300 import initial as mr_initial

G = 9.8
DEV = "cuda"
F64 = torch.float64

# Ray-step arithmetic of the reference's expressions: 4 right-hand sides of
# ~55 operations and their field lookups (~110 each), plus the RK4 update.
FLOPS_STEP = 710
# A step of forward, recompute and reverse sweep: 12 right-hand sides, 4 of
# them with partials and a transpose (about twice the work).
FLOPS_ADJOINT_STEP = 4 * FLOPS_STEP
FLOPS_TANGENT_STEP = 2 * FLOPS_STEP


# ------------------------------------------------------------------- cases --

def listed():
    return [
        # one ray on resident fields, host in and out: a call's latency
        {"name": "single_ray", "kind": "plain", "api": "single_ray", "field": "beach", "nodes": 1000,
         "rays": 1, "steps": 200, "dt": 0.5, "math": "identity"},
        # the reference's published example: 500 rays of 10 s swell, about 10^2
        # steps over 4,000 m of water and a current with eddies, host in and out
        {"name": "ray_tracing_500", "kind": "plain", "api": "ray_tracing", "field": "eddies",
         "nodes": 512, "rays": 500, "steps": 150, "dt": 8.0, "math": "identity"},
        # the planar-beach workload: few rays, many steps, shoaling water
        {"name": "plain_beach_1024", "kind": "plain", "api": "trace_device", "field": "beach",
         "nodes": 1000, "rays": 1024, "steps": 2000, "dt": 0.5, "math": "identity"},
        # the seamount workload, full trajectories on the device
        {"name": "plain_seamount_64k", "kind": "plain", "api": "trace_device", "field": "seamount",
         "nodes": 2001, "rays": 65536, "steps": 2000, "dt": 2.0, "math": "identity"},
        # the reference's own transcendental calls, a ragged number of rays
        {"name": "plain_libm_5003", "kind": "plain", "api": "trace_device", "field": "shelf",
         "nodes": 512, "rays": 5003, "steps": 301, "dt": 4.0, "math": "libm"},
        # the batched form with its default launch and decimated rows
        {"name": "batched_seamount_64k", "kind": "batched", "api": "trace", "field": "seamount",
         "nodes": 2001, "scenarios": 1, "rays": 65536, "steps": 4000, "dt": 1.0,
         "decimation": 100, "order": 0, "sweep": 0, "blocks_per_sm": 4},
        # point sources over several scenarios, uneven lifetimes, ordered queue
        {"name": "batched_sources_1m", "kind": "batched", "api": "trace", "field": "vortices",
         "nodes": 1024, "scenarios": 4, "rays": 1048573, "steps": 1000, "dt": 2.0,
         "decimation": 200, "order": 1, "sweep": 0, "blocks_per_sm": 12},
        # the large single-scenario form: a replayed graph in sweeps, records
        # (1.3 GB) far larger than L2
        {"name": "batched_slope_4m", "kind": "batched", "api": "graph", "field": "slope",
         "nodes": 4096, "scenarios": 1, "rays": 4194304, "steps": 1024, "dt": 2.0,
         "decimation": 0, "order": 1, "sweep": 128, "blocks_per_sm": 12},
        # endpoint loss and its gradients, both precisions
        {"name": "adjoint_fp64", "kind": "diff", "api": "adjoint", "field": "shelf", "nodes": 512,
         "rays": 32768, "steps": 300, "dt": 4.0, "precision": 64},
        {"name": "adjoint_fp32", "kind": "diff", "api": "adjoint", "field": "shelf", "nodes": 512,
         "rays": 131071, "steps": 300, "dt": 4.0, "precision": 32},
        # forward-mode derivative along a state and a depth direction
        {"name": "tangent_fp64", "kind": "diff", "api": "tangent", "field": "shelf", "nodes": 512,
         "rays": 8192, "steps": 500, "dt": 2.0, "precision": 64},
        # initial states of 1,024 point sources x 1,024 rays
        {"name": "seed_sources_1m", "kind": "seed", "field": "vortices", "nodes": 1024,
         "sources": 1024, "per_source": 1024},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["plain", "plain", "plain", "batched", "batched", "diff", "diff", "seed"])
    if kind == "plain":
        api = rng.choice(["ray_tracing", "trace_device", "trace_device"])
        field = rng.choice(["beach", "seamount", "shelf", "eddies", "vortices"])
        rays = _log_int(rng, 1, 2000 if api == "ray_tracing" else 65536)
        steps = min(_log_int(rng, 50, 2000), max(50, 60_000_000 // rays))
        return {"kind": kind, "api": api, "field": field, "nodes": rng.randint(200, 1200),
                "rays": rays, "steps": steps, "dt": rng.choice([0.5, 1.0, 2.0, 4.0]),
                "math": rng.choice(["identity", "identity", "identity", "libm"])
                if rays * steps < 4_000_000 else "identity"}
    if kind == "batched":
        sweep = rng.choice([0, 0, 96, 128])
        order = 1 if sweep else rng.choice([0, 1])
        field = rng.choice(["seamount", "vortices", "slope", "shelf"])
        rays = _log_int(rng, 1000, 2_000_000)
        steps = min(_log_int(rng, 100, 3000), max(100, 800_000_000 // rays))
        return {"kind": kind, "api": rng.choice(["trace", "graph"]), "field": field,
                "nodes": rng.randint(300, 2000), "scenarios": rng.choice([1, 1, 1, 2, 3]),
                "rays": rays, "steps": steps, "dt": rng.choice([1.0, 2.0]),
                "decimation": rng.choice([0, 100]), "order": order, "sweep": sweep,
                "blocks_per_sm": rng.choice([4, 6, 12])}
    if kind == "diff":
        precision = rng.choice([64, 64, 32])
        api = rng.choice(["adjoint", "adjoint", "tangent"])
        rays = _log_int(rng, 100, 30000 if precision == 64 else 130000)
        steps = min(_log_int(rng, 50, 400), max(50, 8_000_000 // rays))
        return {"kind": kind, "api": api, "field": "shelf", "nodes": rng.randint(200, 600),
                "rays": rays, "steps": steps, "dt": rng.choice([1.0, 2.0, 4.0]),
                "precision": precision}
    return {"kind": kind, "field": rng.choice(["vortices", "seamount", "beach"]),
            "nodes": rng.randint(200, 1200), "sources": _log_int(rng, 1, 1000),
            "per_source": _log_int(rng, 10, 1000)}


# ------------------------------------------------------------------ inputs --

def _generator(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _uniform(gen, n, lo, hi):
    return lo + (hi - lo) * torch.rand(n, generator=gen, dtype=F64, device=DEV)


def _field(name, nodes, gen):
    """One scenario: axis (the same for x and y, f64 values that are exact in
    f32), depth, u, v as [y][x] f64 tensors."""
    spacing = {"beach": 10.0, "seamount": 50.0, "shelf": 200.0, "vortices": 100.0,
               "eddies": 100.0, "slope": 50.0}[name]
    x = torch.arange(nodes, dtype=F64, device=DEV) * spacing
    length = float(x[-1])
    X, Y = x[None, :], x[:, None]
    if name == "beach":  # 100 m at x = 0, shoaling; no current
        depth = (100.0 - 90.0 * X / length).clamp_min(2.0).expand(nodes, nodes).contiguous()
        u = torch.zeros_like(depth)
        v = torch.zeros_like(depth)
    elif name == "seamount":  # 4,000 m to 200 m, uniform current
        r2 = (X - 0.5 * length) ** 2 + (Y - 0.5 * length) ** 2
        depth = (4000.0 - 3800.0 * torch.exp(-r2 / (2.0 * (0.15 * length) ** 2))).clamp_min(5.0)
        u = torch.full_like(depth, 0.5)
        v = torch.zeros_like(depth)
    elif name == "shelf":  # a shelf with a shoal, a jet along x
        r2 = (X - 0.5 * length) ** 2 + (Y - 0.5 * length) ** 2
        depth = (3000.0 - 2980.0 * X / length
                 - 1500.0 * torch.exp(-r2 / (2.0 * (0.08 * length) ** 2))).clamp_min(5.0)
        u = torch.exp(-((Y - 0.5 * length) ** 2) / (2.0 * (0.05 * length) ** 2)).expand(
            nodes, nodes).contiguous()
        v = torch.zeros_like(depth)
    else:
        if name == "eddies":  # deep water of one depth
            depth = torch.full((nodes, nodes), 4000.0, dtype=F64, device=DEV)
            u = torch.zeros_like(depth)
        elif name == "vortices":  # seeded shoals
            depth = torch.full((nodes, nodes), 4000.0, dtype=F64, device=DEV)
            for cx, cy, a, s in _uniform(gen, 4 * 12, 0.0, 1.0).reshape(12, 4).tolist():
                depth -= (500.0 + 3000.0 * a) * torch.exp(
                    -((X - cx * length) ** 2 + (Y - cy * length) ** 2)
                    / (2.0 * ((0.05 + 0.12 * s) * length) ** 2))
            depth = depth.clamp(20.0, 4000.0)
            u = torch.zeros_like(depth)
        else:  # slope: a shelf break in x, k^-3 roughness of 50 m rms, a jet
            fx = torch.fft.rfftfreq(nodes, d=spacing, dtype=F64, device=DEV)
            fy = torch.fft.fftfreq(nodes, d=spacing, dtype=F64, device=DEV)
            k = torch.hypot(fy[:, None], fx[None, :])
            amp = torch.where(k > 0, k.clamp_min(1e-12) ** -1.5, torch.zeros_like(k))
            phase = 2.0 * math.pi * torch.rand(k.shape, generator=gen, dtype=F64, device=DEV)
            rough = torch.fft.irfft2(torch.polar(amp, phase), s=(nodes, nodes))
            rough *= 50.0 / rough.square().mean().sqrt()
            depth = (60.0 + 3940.0 * 0.5 * (1.0 - torch.tanh((X - 0.2 * length)
                                                             / (0.03 * length))) + rough)
            depth = depth.clamp_min(5.0)
            yc = 0.5 * length + 0.08 * length * torch.sin(2.0 * math.pi * X / (0.4 * length))
            u = torch.exp(-((Y - yc) ** 2) / (2.0 * (0.05 * length) ** 2))
        v = torch.zeros_like(depth)
        # eddies: u = d(psi)/dy, v = -d(psi)/dx of Gaussian vortices
        for cx, cy, a, s in _uniform(gen, 4 * 8, 0.0, 1.0).reshape(8, 4).tolist():
            sig = (0.02 + 0.06 * s) * length
            peak = (0.2 + 0.8 * abs(2.0 * a - 1.0)) * (1.0 if a > 0.5 else -1.0)
            dx, dy = X - cx * length, Y - cy * length
            g = peak * math.exp(0.5) / sig * torch.exp(-(dx * dx + dy * dy) / (2.0 * sig * sig))
            u -= dy * g
            v += dx * g
    return x, depth, u, v


def _bilinear(x, a, px, py):
    sp = float(x[1] - x[0])
    n = x.numel()
    ix, iy = px / sp, py / sp
    i, j = ix.floor().clamp(0, n - 2), iy.floor().clamp(0, n - 2)
    fx, fy = ix - i, iy - j
    base = (j * n + i).long()
    a = a.reshape(-1)
    return ((1 - fx) * (1 - fy) * a[base] + fx * (1 - fy) * a[base + 1]
            + (1 - fx) * fy * a[base + n] + fx * fy * a[base + n + 1])


def _wavenumber(period, depth):
    """|k| from the dispersion relation, by Newton iteration."""
    w2 = (2.0 * math.pi / period) ** 2
    k = torch.maximum(w2 / G, torch.sqrt(w2 / (G * depth)))
    for _ in range(12):
        th = torch.tanh(k * depth)
        k = k - (G * k * th - w2) / (G * th + G * k * depth * (1 - th * th))
    return k


def _rays(name, n, x, depth, gen):
    """Launch points, directions and periods of the field's workload."""
    length = float(x[-1])
    if name == "vortices":  # point sources away from the edges, all directions
        sources = max(1, min(256, n // 64))
        at = torch.arange(n, device=DEV) % sources
        px = _uniform(gen, sources, 0.1 * length, 0.9 * length)[at]
        py = _uniform(gen, sources, 0.1 * length, 0.9 * length)[at]
        theta, period = _uniform(gen, n, 0.0, 2.0 * math.pi), _uniform(gen, n, 6.0, 18.0)
    else:
        x_start, spread, t_lo, t_hi = {"beach": (0.0, 30.0, 8.0, 12.0),
                                       "seamount": (0.0, 20.0, 8.0, 16.0),
                                       # on the shoal's flank: its shallow water refracts the rays
                                       "shelf": (0.47, 30.0, 8.0, 14.0),
                                       "eddies": (0.0, 0.0, 10.0, 10.0),
                                       "slope": (0.0, 15.0, 10.0, 16.0)}[name]
        px = torch.full((n,), x_start * length, dtype=F64, device=DEV)
        py = _uniform(gen, n, 0.25 * length, 0.75 * length)
        theta = _uniform(gen, n, -math.radians(spread), math.radians(spread))
        period = _uniform(gen, n, t_lo, t_hi)
    k = _wavenumber(period, _bilinear(x, depth, px, py))
    return px, py, k * torch.cos(theta), k * torch.sin(theta)


def _inputs(case, seed):
    """Scenarios, rays and the rays' scenario numbers, from the seed alone."""
    gen = _generator(seed)
    count = case.get("scenarios", 1)
    fields = [_field(case["field"], case["nodes"], gen) for _ in range(count)]
    if case["kind"] == "seed":
        x = fields[0][0]
        length = float(x[-1])
        rays = tuple(_uniform(gen, case["sources"], 0.05 * length, 0.95 * length) for _ in range(2))
        return fields, rays, None
    n = case["rays"]
    per = [n // count + (1 if s < n % count else 0) for s in range(count)]
    parts = [_rays(case["field"], m, f[0], f[1], gen) for m, f in zip(per, fields)]
    rays = tuple(torch.cat(p) for p in zip(*parts))
    scenario = None
    if count > 1:
        scenario = torch.cat([torch.full((m,), s, dtype=torch.uint8, device=DEV)
                              for s, m in enumerate(per)])
    return fields, rays, scenario


def _handles(f):
    x, depth, u, v = (t.cpu().numpy() for t in f)
    x32 = x.astype(np.float32)
    return mr.Bathymetry.grid(x32, x32, depth), mr.Current.grid(x, x, u, v)


def _loss_targets(case, gen, rays):
    """Targets near the endpoints' spread: y and direction of each ray."""
    n = case["rays"]
    return (rays[1] + _uniform(gen, n, -2000.0, 2000.0), _uniform(gen, n, -0.5, 0.5))


def prepare(case, seed):
    fields, rays, scenario = _inputs(case, seed)
    kind = case["kind"]
    state = {"case": case}
    if kind == "diff":
        dtype = F64 if case["precision"] == 64 else torch.float32
        x = fields[0][0]
        sp, n = float(x[1] - x[0]), case["nodes"]
        state["grid"] = mr_diff.grid(n, n, 0.0, 0.0, sp, sp)
        gen = _generator(seed + 1_000_003)
        state["targets"] = tuple(t.to(dtype) for t in _loss_targets(case, gen, rays))
        leaves = [t.to(dtype).contiguous() for t in rays] + [t.to(dtype) for t in fields[0][1:]]
        if case["api"] == "adjoint":
            leaves = [t.requires_grad_() for t in leaves]
        else:
            scale = torch.tensor([[1.0], [1.0], [1e-4], [1e-4]], dtype=F64, device=DEV)
            ds = scale * torch.randn((4, case["rays"]), generator=gen, dtype=F64, device=DEV)
            r2 = (x[None, :] - 0.5 * x[-1]) ** 2 + (x[:, None] - 0.5 * x[-1]) ** 2
            dd = 50.0 * torch.exp(-r2 / (2.0 * (0.06 * x[-1]) ** 2))
            state["dstate"], state["d_depth"] = ds.to(dtype), dd.to(dtype)
        state["leaves"] = leaves
        return state
    if kind == "seed":
        bathymetry, _ = _handles(fields[0])
        state.update(bathymetry=bathymetry, sources=rays, seed=int(seed))
        return state
    handles = [_handles(f) for f in fields]
    n, steps, dt = case["rays"], case["steps"], case["dt"]
    if kind == "plain":
        state["fields"] = handles[0]
        if case["api"] == "trace_device":
            state["rays"] = rays
            state["out"] = (torch.empty((5, steps + 1, n), dtype=F64, device=DEV),
                            torch.empty(n, dtype=torch.int32, device=DEV),
                            torch.empty(n, dtype=torch.uint8, device=DEV))
        else:
            state["rays"] = tuple(t.cpu().numpy() for t in rays)
        return state
    # batched: the tracer, its launch shape, and the output buffers or graph
    tracer = mr_batch.BatchTracer(handles)
    cfg = mr_batch.make_config(128, case["blocks_per_sm"], 1, 32, case["order"], 0, case["sweep"])
    state.update(tracer=tracer, cfg=cfg, rays=rays, scenario=scenario)
    if case["api"] == "graph":
        state["graph"] = tracer.graph(*rays, dt, steps, 0.0, case["decimation"], scenario, cfg)
    else:
        state["out"] = tracer.alloc(n, steps, case["decimation"])
    return state


# --------------------------------------------------------------- one pass --

_ROWS = ("time", "x", "y", "kx", "ky")


def run(state):
    case = state["case"]
    kind, api = case["kind"], case.get("api")
    if kind == "seed":
        return list(mr_initial.seed_point_sources(
            state["bathymetry"], *state["sources"], case["per_source"], (0.0, 2.0 * math.pi),
            (6.0, 18.0), state["seed"]))
    if kind == "plain":
        b, c = state["fields"]
        duration = case["steps"] * case["dt"]
        if api == "trace_device":
            traj, n_rows, status = state["out"]
            mr.trace_device(b, c, *state["rays"], 0.0, duration, case["dt"], traj, n_rows, status,
                            math=case["math"])
            return {"traj": traj, "n_rows": n_rows, "status": status}
        if api == "single_ray":
            ds = mr.single_ray(*(float(a[0]) for a in state["rays"]), duration, case["dt"], b, c,
                               math=case["math"])
        else:
            ds = mr.ray_tracing(*state["rays"], duration, case["dt"], b, c, math=case["math"])
        return {v: np.asarray(ds[v]) for v in _ROWS}
    if kind == "batched":
        if api == "graph":
            state["graph"].launch()
            out = state["graph"].out
        else:
            out = state["tracer"].trace(*state["rays"], case["dt"], case["steps"], 0.0,
                                        case["decimation"], state["scenario"], state["cfg"],
                                        state["out"])
        res = {"end_state": out.end_state, "n_steps": out.n_steps, "n_saved": out.n_saved,
               "status": out.status}
        if case["decimation"]:
            res["saved"] = out.saved
        return res
    grid, leaves = state["grid"], state["leaves"]
    if api == "tangent":
        end, d_end, status = mr_diff.tangent(*leaves, grid, grid, case["dt"], case["steps"],
                                             dstate0=state["dstate"], d_depth=state["d_depth"])
        return {"end": end, "d_end": d_end, "status": status}
    end, status = mr_diff.ray_endpoints(*leaves, grid, grid, case["dt"], case["steps"])
    loss = mr_diff.endpoint_loss(end, status, *state["targets"])
    grads = torch.autograd.grad(loss, leaves)
    return {"end": end.detach(), "status": status, "loss": loss.detach(),
            "grad_state": torch.stack(grads[:4]), "grad_depth": grads[4], "grad_u": grads[5],
            "grad_v": grads[6]}


# ------------------------------------------------------------------- work --

def work(case):
    kind = case["kind"]
    nodes = case["nodes"] ** 2
    if kind == "seed":
        n = case["sources"] * case["per_source"]
        # a Newton solve of about 6 iterations, a sine and a cosine
        return {"bytes": 32 * n + 16 * case["sources"] + 4 * min(nodes, 4 * case["sources"]),
                "flops": 250 * n}
    n, steps = case["rays"], case["steps"]
    # nodes of the fields a call can reach at most: each ray meets at most a
    # few new nodes a step
    reach = min(nodes * case.get("scenarios", 1), 4 * n * steps)
    if kind == "plain":
        return {"bytes": 40 * n * (steps + 1) + 32 * n + 5 * n + 24 * reach,
                "flops": FLOPS_STEP * n * steps}
    if kind == "batched":
        rows = steps // case["decimation"] + 1 if case["decimation"] else 0
        return {"bytes": (32 + 40 + 9 + 20 * rows) * n + 12 * reach,
                "flops": FLOPS_STEP * n * steps}
    size = case["precision"] // 8
    if case["api"] == "tangent":
        return {"bytes": (16 * n + 4 * reach) * size + n, "flops": FLOPS_TANGENT_STEP * n * steps}
    return {"bytes": (12 * n + 3 * reach + 3 * nodes) * size + n,
            "flops": FLOPS_ADJOINT_STEP * n * steps}


# ------------------------------------------------- the model in 64 bits --

def _cells(fields):
    """[scenario * cell][12]: the bilinear coefficients of depth, u and v."""
    out = []
    for _, *abc in fields:
        cols = []
        for a in abc:
            v00, v10, v01, v11 = a[:-1, :-1], a[:-1, 1:], a[1:, :-1], a[1:, 1:]
            cols += [v00, v10 - v00, v01 - v00, (v11 - v10) - (v01 - v00)]
        out.append(torch.stack(cols, dim=-1).reshape(-1, 12))
    return torch.cat(out)


def _derivative(vals, grads, kx, ky):
    """(dx, dy, dkx, dky) from the interpolated (h, u, v) and the cells'
    constant gradients (h_x, h_y, u_x, u_y, v_x, v_y)."""
    h, u, v = vals
    hx, hy, ux, uy, vx, vy = grads
    k = torch.sqrt(kx * kx + ky * ky)
    a = k * h
    th = torch.tanh(a)
    b = torch.clamp(a, max=300.0)  # sinh and cosh stay finite; the terms are 0 there
    sh, ch = torch.sinh(b), torch.cosh(b)
    sq = torch.sqrt(G * k * th)
    cg = 0.5 * G * (th + b / (ch * ch)) / sq
    f = -0.5 * k * sq / (sh * ch)
    return (cg * kx / k + u, cg * ky / k + v, f * hx - kx * ux - ky * vx,
            f * hy - kx * uy - ky * vy)


class _Model:
    """The ray equations on regular grids, everything in FP64."""

    def __init__(self, fields, scenario=None, closed=True):
        x = fields[0][0]
        self.n, self.sp = x.numel(), float(x[1] - x[0])
        self.table = _cells(fields)
        self.offset = 0 if scenario is None else scenario.long() * (self.n - 1) ** 2
        self.closed = closed  # whether a point on the last grid line is inside

    def __call__(self, s):
        """(derivatives, whether each ray has one)."""
        x, y, kx, ky = s
        ix, iy = x / self.sp, y / self.sp
        top = float(self.n - 1)
        hi = (ix <= top) & (iy <= top) if self.closed else (ix < top) & (iy < top)
        ok = (ix >= 0) & (iy >= 0) & hi
        i = torch.nan_to_num(ix).floor().clamp(0, self.n - 2)
        j = torch.nan_to_num(iy).floor().clamp(0, self.n - 2)
        fx, fy = ix - i, iy - j
        c = self.table.index_select(0, (j * (self.n - 1) + i).long() + self.offset).reshape(-1, 3, 4)
        basis = torch.stack([torch.ones_like(fx), fx, fy, fx * fy], dim=-1)
        h, u, v = (c * basis[:, None, :]).sum(-1).unbind(-1)
        g = (c[:, :, 1:3] / self.sp).reshape(-1, 6).unbind(-1)
        ok &= (h > 0) & ((kx != 0) | (ky != 0))
        return torch.stack(_derivative((h, u, v), g, kx, ky)), ok


def _rk4(model, s, dt):
    """One step and whether all four stages had a derivative."""
    k1, o1 = model(s)
    k2, o2 = model(s + k1 * (dt / 2))
    k3, o3 = model(s + k2 * (dt / 2))
    k4, o4 = model(s + k3 * dt)
    return s + (k1 + k2 * 2 + k3 * 2 + k4) * (dt / 6), o1 & o2 & o3 & o4


def _exact_plain(case, fields, rays):
    model = _Model(fields)
    n, steps, dt = case["rays"], case["steps"], case["dt"]
    nan = float("nan")
    traj = torch.full((5, steps + 1, n), nan, dtype=F64, device=DEV)
    s = torch.stack(rays)
    t = 0.0
    alive = torch.ones(n, dtype=torch.bool, device=DEV)
    traj[0, 0], traj[1:, 0] = t, s
    for step in range(1, steps + 1):
        new, ok = _rk4(model, s, dt)
        # a stage without a derivative gives a NaN row, the ray's last
        s = torch.where(alive & ok, new, torch.full_like(new, nan))
        t += dt
        traj[0, step] = torch.where(alive, t, nan)
        traj[1:, step] = s
        alive &= ok
    return traj


def _exact_batched(case, fields, rays, scenario):
    model = _Model(fields, scenario, closed=False)
    n, steps, dt, dec = case["rays"], case["steps"], case["dt"], case["decimation"]
    s = torch.stack(rays)
    alive = torch.ones(n, dtype=torch.bool, device=DEV)
    taken = torch.zeros(n, dtype=F64, device=DEV)
    saved = None
    if dec:
        saved = torch.full((5, steps // dec + 1, n), float("nan"), dtype=F64, device=DEV)
        saved[0, 0], saved[1:, 0] = 0.0, s
    for step in range(1, steps + 1):
        new, ok = _rk4(model, s, dt)
        alive &= ok
        s = torch.where(alive, new, s)
        taken += alive
        if dec and step % dec == 0:
            row = torch.cat([torch.full_like(s[:1], step * dt), s])
            saved[:, step // dec] = torch.where(alive, row, saved[:, step // dec])
    res = {"end_state": torch.cat([(taken * dt)[None], s]), "n_steps": None, "n_saved": None,
           "status": None}
    if dec:
        res["saved"] = saved
    return res


class _DiffModel:
    """The same equations with the nodes as differentiable tensors."""

    def __init__(self, x, depth, u, v):
        self.n, self.sp = x.numel(), float(x[1] - x[0])
        self.nodes = [a.reshape(-1) for a in (depth, u, v)]

    def __call__(self, s):
        x, y, kx, ky = s
        ix, iy = x / self.sp, y / self.sp
        i = ix.detach().floor().clamp(0, self.n - 2)
        j = iy.detach().floor().clamp(0, self.n - 2)
        fx, fy = ix - i, iy - j
        base = (j * self.n + i).long()
        vals, grads = [], []
        for a in self.nodes:
            v00, v10 = a.index_select(0, base), a.index_select(0, base + 1)
            v01 = a.index_select(0, base + self.n)
            v11 = a.index_select(0, base + self.n + 1)
            ex, ey = v10 - v00, v01 - v00
            vals.append(v00 + ex * fx + ey * fy + (v11 - v10 - v01 + v00) * fx * fy)
            grads += [ex / self.sp, ey / self.sp]
        return torch.stack(_derivative(vals, grads, kx, ky)), True


def _exact_diff(case, fields, rays, seed):
    gen = _generator(seed + 1_000_003)
    y_target, theta_target = _loss_targets(case, gen, rays)
    dtype = F64 if case["precision"] == 64 else torch.float32
    cast = lambda t: t.to(dtype).to(F64)  # noqa: E731  (the inputs as the call gets them)
    leaves = [cast(t).requires_grad_() for t in (*rays, *fields[0][1:])]
    n, steps, dt = case["rays"], case["steps"], case["dt"]
    x = fields[0][0]

    def inside(s):
        return bool(((s[:2] >= 0) & (s[:2] <= float(x[-1]))).all())

    def steps_of(s, depth, u, v, count):
        model = _DiffModel(x, depth, u, v)
        for _ in range(count):
            s, _ok = _rk4(model, s, dt)
        return s

    if case["api"] == "tangent":
        scale = torch.tensor([[1.0], [1.0], [1e-4], [1e-4]], dtype=F64, device=DEV)
        ds = cast(scale * torch.randn((4, n), generator=gen, dtype=F64, device=DEV))
        r2 = (x[None, :] - 0.5 * x[-1]) ** 2 + (x[:, None] - 0.5 * x[-1]) ** 2
        dd = cast(50.0 * torch.exp(-r2 / (2.0 * (0.06 * x[-1]) ** 2)))
        plain = [t.detach() for t in leaves]
        zero = torch.zeros_like(plain[5])
        with torch.autograd.forward_ad.dual_level():
            dual = torch.autograd.forward_ad.make_dual
            s = dual(torch.stack(plain[:4]), ds)
            end = steps_of(s, dual(plain[4], dd), dual(plain[5], zero), dual(plain[6], zero), steps)
            end, d_end = torch.autograd.forward_ad.unpack_dual(end)
        return {"end": end, "d_end": d_end, "status": None} if inside(end) else None
    s = torch.stack(leaves[:4])
    chunk, done = 20, 0
    while done < steps:
        m = min(chunk, steps - done)
        s = torch.utils.checkpoint.checkpoint(steps_of, s, *leaves[4:], m, use_reentrant=False)
        done += m
    if not inside(s.detach()):
        return None
    dy = s[1] - cast(y_target)
    dth = torch.atan2(s[3], s[2]) - cast(theta_target)
    loss = (dy * dy + dth * dth).sum()
    grads = torch.autograd.grad(loss, leaves)
    return {"end": s.detach(), "status": None, "loss": loss.detach(),
            "grad_state": torch.stack(grads[:4]), "grad_depth": grads[4], "grad_u": grads[5],
            "grad_v": grads[6]}


def _mix(seed, index):
    """SplitMix64 of seed + (index + 1) * golden as uniforms in [0, 1)."""
    with np.errstate(over="ignore"):
        z = np.uint64(seed) + (index.astype(np.uint64) + np.uint64(1)) * np.uint64(0x9E3779B97F4A7C15)
        z = (z ^ (z >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
        z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
        z = z ^ (z >> np.uint64(31))
    return (z >> np.uint64(11)).astype(np.float64) * 2.0 ** -53


def _exact_seed(case, fields, sources, seed):
    x, depth = fields[0][:2]
    px, py = (t.repeat_interleave(case["per_source"]) for t in sources)
    r = np.arange(px.numel())
    theta = torch.from_numpy(2.0 * math.pi * _mix(seed, 2 * r)).to(DEV)
    period = torch.from_numpy(6.0 + 12.0 * _mix(seed, 2 * r + 1)).to(DEV)
    k = _wavenumber(period, _bilinear(x, depth, px, py))
    return [px, py, k * torch.cos(theta), k * torch.sin(theta)]


def exact(case, seed):
    fields, rays, scenario = _inputs(case, seed)
    kind = case["kind"]
    if kind == "diff":
        return _exact_diff(case, fields, rays, seed)
    if kind == "seed":
        return _exact_seed(case, fields, rays, seed)
    # about 120 operations a stage, each at the launch rate or a pass over n
    if case["steps"] * 4 * 120 * max(7e-6, case["rays"] * 9e-12) > 25.0:
        return None
    if kind == "batched":
        return _exact_batched(case, fields, rays, scenario)
    traj = _exact_plain(case, fields, rays)
    if case["api"] == "trace_device":
        return {"traj": traj, "n_rows": None, "status": None}
    # the dataset ends with the longest ray's last row
    rows = int((~torch.isnan(traj[0])).any(dim=1).sum())
    out = traj[:, :rows, 0] if case["api"] == "single_ray" else traj[:, :rows]
    return {v: out[q].cpu().numpy() for q, v in enumerate(_ROWS)}
