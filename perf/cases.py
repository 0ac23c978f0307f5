"""The work that a user of pyftle_b200 has it do, as cases that can be timed and compared.

Every case calls the package's public entry points on inputs that are already on the
GPU.  The kinds, and what each stands for in use:

steps      the reference-style loop: ``update`` + ``integrate`` once per snapshot, then the
           FTLE of the final positions (small seed sets, custom loops, interactive use)
solver     ``FTLESolver.run`` on one window: the drop-in call, packing included; plain FP64
           HOLD as in the reference, or 16-bit storage with the FP64 judge
window     ``run_window`` over a packed series: one window of a sliding series, plain FP64 or
           16-bit, chunked and cell-sorted as the benchmark runs it
batch      ``WindowBatch.run``: many uneven windows over one series in one launch
pack       ``SnapshotSeries``: a snapshot stack made into a series, paid once per data set
analytic   ``AnalyticalSolver.run`` on a closed-form field
ftle       the FTLE building blocks on advected particle groups
train      one optimisation step of the flow-map surrogate
surrogate  the surrogate's FTLE field (2D fused kernel, 3D layered kernels)

Sizes follow the repository's benchmark and full-size tests (double gyre on 512 x 256,
ABC on 128^3, turbulence on 1024^2, 4 x 256 and 4 x 384 networks, batches of 65,536).
"""

import math

import numpy as np
import torch

from pyftle_b200 import (
    BlendedSnapshotSource,
    EngineOptions,
    FTLESolver,
    GridSpec,
    MemoryBatchSource,
    NeighboringParticles,
    SnapshotSeries,
    create_integrator,
    create_interpolator,
    run_window,
)
from pyftle_b200.api import ABCFlow, AnalyticalSolver, DoubleGyre
from pyftle_b200.batch import WindowBatch, WindowSpecRun
from pyftle_b200.ftle import (
    compute_cauchy_green_2x2,
    compute_cauchy_green_3x3,
    compute_flow_map_jacobian_2x2,
    compute_flow_map_jacobian_3x3,
    compute_ftle_2x2,
    compute_ftle_3x3,
    compute_ftle_from_positions,
    max_eigenvalue_2x2,
    max_eigenvalue_3x3,
)
from pyftle_b200.surrogate import FlowMapMLP

TWO_PI = 2.0 * math.pi
F64 = torch.float64
RECORD_BYTES = {"fp64": 8, "fx16": 2, "fx15": 2, "fp16": 2, "bf16": 2}

# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------


def listed():
    return [
        # interactive use and unit-sized data: launches and host calls are everything
        dict(name="gyre_steps_small", kind="steps", flow="gyre", nx=65, ny=33, nz=0, cx=40, cy=20,
             cz=0, steps=20, h=0.05, integrator="rk4"),
        # the reference's own benchmark window through the drop-in solver
        dict(name="gyre_solver_hold", kind="solver", flow="gyre", nx=512, ny=256, nz=0, cx=400,
             cy=200, cz=0, snaps=101, steps=101, h=0.05, integrator="rk4", precision="fp64",
             judged=False),
        # one whole judged 16-bit window: pack, window, FP64 sample
        dict(name="turb_solver_judged", kind="solver", flow="turb", nx=512, ny=512, nz=0, cx=512,
             cy=256, cz=0, snaps=41, steps=80, h=0.025, integrator="rk4", precision="fx16",
             judged=True),
        # reference-exact window of the 3D flow (also the judge and the surrogate's data)
        dict(name="abc_window_f64", kind="window", flow="abc", nx=128, ny=128, nz=128, cx=65,
             cy=64, cz=63, snaps=16, steps=100, h=0.02, integrator="rk4", precision="fp64",
             mode="blend", chunk=0, update=True),
        # the headline window: 16-bit storage, 50-step chunks, cell sort
        dict(name="abc_window_fx16", kind="window", flow="abc", nx=128, ny=128, nz=128, cx=128,
             cy=128, cz=128, snaps=32, steps=200, h=0.02, integrator="rk4", precision="fx16",
             mode="blend", chunk=50, update=False),
        # many uneven windows in one persistent launch
        dict(name="turb_batch_fx16", kind="batch", flow="turb", nx=1024, ny=1024, nz=0, windows=24,
             cmin=64, cmax=1024, snaps=100, lmin=40, lmax=160, h=0.025, integrator="rk4",
             precision="fx16"),
        # making a data set ready
        dict(name="abc_pack_fx16", kind="pack", flow="abc", nx=128, ny=128, nz=128, snaps=32,
             precision="fx16"),
        # closed-form field, four fields of a sliding start time
        dict(name="gyre_analytic", kind="analytic", flow="gyre", cx=301, cy=150, cz=0, fields=4,
             period=5.0, h=0.1, integrator="rk4"),
        # deformation diagnostics of advected groups
        dict(name="ftle_blocks_3d", kind="ftle", dim=3, groups=600001, chain=True),
        # one Adam step of the 2D surrogate
        dict(name="train_step_2d", kind="train", dim=2, hidden=256, depth=4, freqs=32,
             batch=65536),
        # a surrogate field of a million seeds
        dict(name="surrogate_field_2d", kind="surrogate", dim=2, hidden=256, depth=4, freqs=32,
             seeds=1 << 20),
        # the 3D network on its layered kernels
        dict(name="surrogate_field_3d", kind="surrogate", dim=3, hidden=384, depth=4, freqs=32,
             seeds=1 << 18),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _grid_and_seeds(rng, dim, most):
    """Grid and seed extents; `most` bounds the number of groups."""
    if dim == 2:
        nx, ny = _log(rng, 40, 700), _log(rng, 40, 700)
        cx = _log(rng, 16, min(700, most // 16))
        cy = max(1, min(_log(rng, 16, 700), most // cx))
        return dict(nx=nx, ny=ny, nz=0, cx=cx, cy=cy, cz=0)
    nx = _log(rng, 20, 128)  # the reference's 3D layout: nx == ny
    c = [_log(rng, 8, max(9, int(most ** (1 / 3)))) for _ in range(3)]
    return dict(nx=nx, ny=nx, nz=_log(rng, 20, 128), cx=c[0], cy=c[1], cz=c[2])


def draw(rng):
    kind = rng.choice(["steps", "solver", "solver", "window", "window", "window", "batch", "pack",
                       "analytic", "ftle", "train", "surrogate"])
    dim = rng.choice([2, 3])
    integrator = rng.choice(["rk4", "rk4", "rk4", "ab2", "euler"])
    flow = "abc" if dim == 3 else rng.choice(["gyre", "turb"])
    if kind == "steps":
        flow = "abc" if dim == 3 else "gyre"
        return dict(kind=kind, flow=flow, **_grid_and_seeds(rng, dim, 200000),
                    steps=rng.randint(5, 40), h=0.05, integrator=integrator)
    if kind == "solver":
        hold = rng.random() < 0.5
        steps = rng.randint(20, 150)
        return dict(kind=kind, flow="gyre" if hold and dim == 2 else flow,
                    **_grid_and_seeds(rng, dim, 150000), snaps=steps if hold else 41, steps=steps,
                    h=0.05 if hold else 0.02, integrator=integrator,
                    precision="fp64" if hold else "fx16", judged=not hold)
    if kind == "window":
        precision = rng.choice(["fp64", "fp64", "fx16", "fx16", "fx15", "fp16", "bf16"])
        g = _grid_and_seeds(rng, dim, 300000 if precision == "fp64" else 2000000)
        mode = rng.choice(["hold", "blend", "blend"])
        return dict(kind=kind, flow=flow, **g, snaps=rng.randint(12, 40),
                    steps=rng.randint(30, 160) if mode == "blend" else 12, h=0.02,
                    integrator=integrator, precision=precision, mode=mode,
                    chunk=0 if precision == "fp64" else rng.choice([0, 25, 50]),
                    update=rng.random() < 0.5)
    if kind == "batch":
        g = _grid_and_seeds(rng, dim, 1000)
        return dict(kind=kind, flow="abc" if dim == 3 else "turb", nx=g["nx"], ny=g["ny"],
                    nz=g["nz"], windows=rng.randint(2, 24), cmin=16, cmax=400 if dim == 2 else 60,
                    snaps=rng.randint(20, 60), lmin=20, lmax=rng.randint(40, 160), h=0.02,
                    integrator=integrator, precision=rng.choice(["fx16", "fx15", "fp16"]))
    if kind == "pack":
        g = _grid_and_seeds(rng, dim, 1000)
        return dict(kind=kind, flow=flow, nx=g["nx"], ny=g["ny"], nz=g["nz"],
                    snaps=rng.randint(2, 60),
                    precision=rng.choice(["fp64", "fx16", "fx15", "fp16", "bf16"]))
    if kind == "analytic":
        g = _grid_and_seeds(rng, dim, 100000)
        return dict(kind=kind, flow="gyre" if dim == 2 else "abc", cx=g["cx"], cy=g["cy"],
                    cz=g["cz"], fields=rng.randint(1, 6), period=rng.uniform(1.0, 6.0), h=0.1,
                    integrator=integrator)
    if kind == "ftle":
        return dict(kind=kind, dim=dim, groups=_log(rng, 1000, 2000000), chain=rng.random() < 0.5)
    hidden, freqs = rng.choice([(256, 32), (256, 32), (384, 32), (512, 64), (128, 32)])
    depth = rng.choice([4, 4, 3, 5])
    if kind == "train":
        return dict(kind=kind, dim=dim, hidden=hidden, depth=depth, freqs=freqs,
                    batch=128 * _log(rng, 32, 512))
    return dict(kind=kind, dim=dim, hidden=hidden, depth=depth, freqs=freqs,
                seeds=8 * _log(rng, 500, 32768))


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _u(seed, *key):
    """One number in [0, 1) from the seed and a key."""
    return float(np.random.default_rng([seed, *key]).random())


def _shape(c):
    return (c["nx"], c["ny"]) if not c["nz"] else (c["nx"], c["ny"], c["nz"])


def _grid(c):
    """(shape, origin, spacing, periodic): the gyre's box with both ends, else [0, 2 pi)^d."""
    shape = _shape(c)
    if c["flow"] == "gyre":
        return shape, (0.0, 0.0), (2.0 / (shape[0] - 1), 1.0 / (shape[1] - 1)), False
    return shape, (0.0,) * len(shape), tuple(TWO_PI / n for n in shape), True


def _spec(c):
    shape, origin, spacing, periodic = _grid(c)
    return GridSpec(shape, origin, spacing, periodic)


def _points(c):
    """(dim, nodes) node coordinates on the host, meshgrid order."""
    shape, origin, spacing, _ = _grid(c)
    axes = [o + s * np.arange(n) for n, o, s in zip(shape, origin, spacing)]
    return np.stack([m.ravel() for m in np.meshgrid(*axes)])


def _snap_dt(c):
    """Time between snapshots: the step of HOLD windows, else a spacing that covers them."""
    if c["kind"] == "steps" or c.get("mode") == "hold" or (
            c["kind"] == "solver" and not c["judged"]):
        return c["h"]
    if c["kind"] == "pack":
        return 0.05
    if c["flow"] == "abc":
        return TWO_PI / c["snaps"]  # one period of the flow
    span = c["lmax"] if c["kind"] == "batch" else c["steps"]
    return span * c["h"] / (c["snaps"] - 1)


def _periodic_time(c):
    return c["flow"] == "abc" and _snap_dt(c) != c.get("h")


def _gyre_params(seed):
    return 0.09 + 0.02 * _u(seed, 1), 0.2 + 0.1 * _u(seed, 2), TWO_PI / (9.0 + 2.0 * _u(seed, 3))


def _abc_params(seed):
    return (math.sqrt(3.0) * (0.95 + 0.1 * _u(seed, 1)),
            math.sqrt(2.0) * (0.95 + 0.1 * _u(seed, 2)), 0.95 + 0.1 * _u(seed, 3))


def _snapshots(c, seed, count):
    """(count, dim, nodes) velocities in FP64 on the GPU."""
    shape, origin, spacing, _ = _grid(c)
    ax = [o + s * torch.arange(n, dtype=F64, device="cuda")
          for n, o, s in zip(shape, origin, spacing)]
    times = [i * _snap_dt(c) for i in range(count)]
    dim, nodes = len(shape), math.prod(shape)
    if c["flow"] == "abc":
        out = torch.empty((count, 3, shape[1], shape[0], shape[2]), dtype=F64, device="cuda")
        A, B, C = _abc_params(seed)
        sx, sy, sz = (torch.sin(a) for a in ax)
        cx, cy, cz = (torch.cos(a) for a in ax)
        for s, t in enumerate(times):
            At = A + 0.1 * math.sin(t)
            out[s, 0] = (At * sz)[None, None, :] + (C * cy)[:, None, None]
            out[s, 1] = (B * sx)[None, :, None] + (At * cz)[None, None, :]
            out[s, 2] = (C * sy)[:, None, None] + (B * cx)[None, :, None]
        return out.view(count, 3, nodes)
    out = torch.empty((count, dim, shape[1], shape[0]), dtype=F64, device="cuda")
    if c["flow"] == "gyre":
        A, eps, om = _gyre_params(seed)
        x, y = ax[0][None, :], ax[1][:, None]
        for s, t in enumerate(times):
            e = eps * math.sin(om * t)
            f, df = e * x * x + (1.0 - 2.0 * e) * x, 2.0 * e * x + (1.0 - 2.0 * e)
            out[s, 0] = -math.pi * A * torch.sin(math.pi * f) * torch.cos(math.pi * y)
            out[s, 1] = math.pi * A * torch.cos(math.pi * f) * torch.sin(math.pi * y) * df
        return out.view(count, 2, nodes)
    # 2D turbulence: E(k) ~ k^(-5/3) on 4 <= |k| <= min(128, n/3), each mode with its frequency
    g = _gen(seed)
    kx = torch.fft.fftfreq(shape[0], 1.0 / shape[0], dtype=F64, device="cuda")[None, :]
    ky = torch.fft.fftfreq(shape[1], 1.0 / shape[1], dtype=F64, device="cuda")[:, None]
    k = torch.sqrt(kx * kx + ky * ky)
    keep = (k >= 4.0) & (k <= min(128.0, min(shape) / 3.0))
    amp = torch.where(keep, k.clamp_min(1.0) ** (-7.0 / 3.0), torch.zeros_like(k))
    phase = TWO_PI * torch.rand(k.shape, generator=g, dtype=F64, device="cuda")
    omega = torch.randn(k.shape, generator=g, dtype=F64, device="cuda")
    amp = amp * (0.02 * nodes / math.sqrt(0.25 * float((amp * k).square().sum())))
    for s, t in enumerate(times):
        psi = torch.polar(amp, phase + omega * t)
        out[s, 0] = torch.fft.ifft2(1j * ky * psi).real
        out[s, 1] = torch.fft.ifft2(-1j * kx * psi).real
    return out.view(count, 2, nodes)


def _centroids(c, seed, cx, cy, cz):
    """Regular centroids inside the flow's box, shifted by a fraction of their spacing."""
    if c["flow"] == "gyre":
        lo, hi = (0.02, 0.02), (1.98, 0.98)
    else:
        lo, hi = (0.0,) * 3, (TWO_PI,) * 3
    axes = []
    for a, n in enumerate((cx, cy, cz) if cz else (cx, cy)):
        d = (hi[a] - lo[a]) / n
        axes.append(lo[a] + d * (torch.arange(n, dtype=F64, device="cuda") + _u(seed, 10 + a)))
    mesh = torch.meshgrid(*axes, indexing="xy")
    return torch.stack([m.reshape(-1) for m in mesh], dim=1)


def _groups(cent, delta=5e-4):
    """Role-blocked neighbours [L; R; T; B (; F; Bk)]."""
    dim = cent.shape[1]
    rows = []
    for a in range(dim):
        e = torch.zeros(dim, dtype=F64, device=cent.device)
        e[a] = delta
        rows += [cent - e, cent + e] if a == 0 else [cent + e, cent - e]
    return torch.cat(rows).contiguous()


def _seeds(c, seed):
    return _groups(_centroids(c, seed, c["cx"], c["cy"], c["cz"]))


def _batch_windows(c, seed):
    """(cx, cy, cz, steps, t0) of each window of a batch: the sizes are the case's own, the
    start times the seed's."""
    sizes = np.random.default_rng([c[k] for k in ("windows", "cmin", "cmax", "lmin", "lmax")])
    rng = np.random.default_rng([seed, 77])
    span = c["lmax"] * c["h"] if c["flow"] == "turb" else TWO_PI
    out = []
    for _ in range(c["windows"]):
        n = int(round(math.exp(sizes.uniform(math.log(c["cmin"]), math.log(c["cmax"])))))
        steps = int(sizes.integers(c["lmin"], c["lmax"] + 1))
        t0 = float(rng.uniform(0.0, max(0.0, span - steps * c["h"])))
        out.append((n, max(1, n // 2), max(1, n // 2) if c["nz"] else 0, steps, t0))
    return out


def _deformed(c, seed):
    """(positions at t0, positions after a random stretching of every group)."""
    g, dim, n = _gen(seed), c["dim"], c["groups"]
    cent = TWO_PI * torch.rand((n, dim), generator=g, dtype=F64, device="cuda")
    grad = torch.eye(dim, dtype=F64, device="cuda") + 2.0 * torch.randn(
        (n, dim, dim), generator=g, dtype=F64, device="cuda")
    p0 = _groups(cent)
    off = (p0.view(2 * dim, n, dim) - cent[None]).transpose(0, 1)  # (n, K, dim)
    p1 = cent[:, None, :] + torch.einsum("nij,nkj->nki", grad, off)
    return p0, p1.transpose(0, 1).reshape(-1, dim).contiguous()


def _freq(c, seed):
    """Frequency rows: (kx, ky, kt, phase), 3D (kx, ky, kz, kt, phase, 0, 0, 0)."""
    rng, d, n = np.random.default_rng([seed, 5]), c["dim"], c["freqs"]
    rows = np.zeros((n, 4 * (d - 1)), dtype=np.float32)
    rows[:, :d] = np.round(rng.normal(0.0, 4.0, (n, d)))
    rows[:, 0] += np.all(rows[:, :d] == 0.0, axis=1)
    rows[:, d] = rng.normal(0.0, 0.3, n)
    return rows


def _net(c, seed):
    return FlowMapMLP(_freq(c, seed), hidden=c["hidden"], depth=c["depth"], out_scale=0.05, seed=seed)


def _net_points(c, seed, n, t0=None):
    g = _gen(seed)
    p = TWO_PI * torch.rand((n, c["dim"] + 1), generator=g, dtype=F64, device="cuda")
    p[:, -1] = 0.5 * p[:, -1] if t0 is None else t0
    return p, g


def _train_inputs(c, seed):
    p, g = _net_points(c, seed, c["batch"])
    x = p[:, :c["dim"]]
    target = (torch.sin(x + 0.3 * p[:, -1:]) + 0.3 * torch.sin(3.0 * x.flip(1))).float()
    return p, target.contiguous(), g


def prepare(case, seed):
    c, k = case, case["kind"]
    if k == "steps":
        interp = create_interpolator("grid", _shape(c), periodic=_grid(c)[3])
        snaps = _snapshots(c, seed, c["steps"])
        interp.update(snaps[0], _points(c))
        return dict(case=c, interp=interp, integ=create_integrator(c["integrator"], interp),
                    snaps=snaps, seeds=_seeds(c, seed))
    if k == "solver":
        snaps, points, seeds = _snapshots(c, seed, c["snaps"]), _points(c), _seeds(c, seed)
        periodic = _grid(c)[3]
        if c["judged"]:
            source = BlendedSnapshotSource(snaps, points, seeds, _shape(c), h=c["h"],
                                           num_steps=c["steps"], snapshot_dt=_snap_dt(c),
                                           periodic_space=periodic,
                                           periodic_time=_periodic_time(c))
            options = EngineOptions(precision=c["precision"], time_mode="blend", judge_tol=1e-3)
        else:
            source = MemoryBatchSource(snaps, points, seeds, c["h"], _shape(c),
                                       periodic_space=periodic)
            options = EngineOptions(precision=c["precision"])
        interp = create_interpolator("grid", _shape(c), periodic=periodic)
        return dict(case=c, source=source, options=options,
                    integ=create_integrator(c["integrator"], interp))
    if k == "window":
        series = SnapshotSeries(_spec(c), _snapshots(c, seed, c["snaps"]),
                                precision=c["precision"], periodic_time=_periodic_time(c))
        return dict(case=c, series=series, seeds=_seeds(c, seed))
    if k == "batch":
        series = SnapshotSeries(_spec(c), _snapshots(c, seed, c["snaps"]),
                                precision=c["precision"], periodic_time=_periodic_time(c))
        runs = [WindowSpecRun(_groups(_centroids(c, seed, cx, cy, cz)), t0, c["h"], steps,
                              keep_positions=True)
                for cx, cy, cz, steps, t0 in _batch_windows(c, seed)]
        return dict(case=c, batch=WindowBatch(series, runs, integrator=c["integrator"],
                                              snapshot_dt=_snap_dt(c)))
    if k == "pack":
        return dict(case=c, grid=_spec(c), snaps=_snapshots(c, seed, c["snaps"]))
    if k == "analytic":
        if c["flow"] == "gyre":
            flow = DoubleGyre(*_gyre_params(seed))
        else:
            flow = ABCFlow(*_abc_params(seed))
        part = NeighboringParticles(positions=_seeds(c, seed))
        return dict(case=c, solver=AnalyticalSolver(flow, part, c["h"], c["period"], c["fields"],
                                                    c["integrator"]))
    if k == "ftle":
        p0, p1 = _deformed(c, seed)
        part = NeighboringParticles(positions=p0)
        part.positions.copy_(p1)
        return dict(case=c, part=part)
    net = _net(c, seed)
    if k == "train":
        points, target, g = _train_inputs(c, seed)
        # in mid-training the moments hold the gradients' scale
        net.m.normal_(0.0, 1e-3, generator=g)
        net.v.uniform_(1e-6, 2e-6, generator=g)
        net.step = 1000
        return dict(case=c, net=net, points=points, target=target)
    points, _ = _net_points(c, seed, c["seeds"], t0=1.0)
    if net.supports_fused:
        points = points[:, :2].contiguous()
    return dict(case=c, net=net, points=points)


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------


def run(state):
    c = state["case"]
    k = c["kind"]
    if k == "steps":
        interp, integ, snaps = state["interp"], state["integ"], state["snaps"]
        part = NeighboringParticles(positions=state["seeds"])
        integ.reset()
        for i in range(c["steps"]):
            interp.update(snaps[i])
            integ.integrate(c["h"], part)
        return part.positions, compute_ftle_from_positions(part, (c["steps"] - 1) * c["h"])
    if k == "solver":
        return FTLESolver(state["source"], state["integ"], options=state["options"]).run()
    if k == "window":
        pos = state["seeds"].clone() if c["update"] else state["seeds"]
        ftle = run_window(state["series"], pos, integrator=c["integrator"], time_mode=c["mode"],
                          h=c["h"], num_steps=c["steps"], snapshot_dt=_snap_dt(c),
                          chunk_steps=c["chunk"] or None, keep_positions=not c["update"])
        return (ftle, pos) if c["update"] else ftle
    if k == "batch":
        return state["batch"].run()
    if k == "pack":
        return SnapshotSeries(state["grid"], state["snaps"], precision=c["precision"],
                              periodic_time=_periodic_time(c)).packed
    if k == "analytic":
        return state["solver"].run()
    if k == "ftle":
        part = state["part"]
        if not c["chain"]:
            return compute_ftle_from_positions(part, 2.0)
        if c["dim"] == 2:
            jac = compute_flow_map_jacobian_2x2(part)
            cg = compute_cauchy_green_2x2(jac)
            return jac, cg, max_eigenvalue_2x2(cg), compute_ftle_2x2(jac, 2.0)
        jac = compute_flow_map_jacobian_3x3(part)
        cg = compute_cauchy_green_3x3(jac)
        return jac, cg, max_eigenvalue_3x3(cg), compute_ftle_3x3(jac, 2.0)
    net = state["net"]
    if k == "train":
        loss = net.loss_and_grads(state["points"], state["target"])
        net.adam_step(1e-3)
        return dict(loss=loss, w=net.w, m=net.m, v=net.v)
    if net.supports_fused:
        return net.ftle_fused(state["points"], 1.0, 5.0)
    return net.ftle(state["points"], 5.0)


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------


def _particle_steps(c):
    """(groups, sum over groups of steps) of an advecting case, on average over seeds."""
    if c["kind"] == "batch":
        ln = math.log(c["cmax"] / c["cmin"])
        p = 3 if c["nz"] else 2
        per = (c["cmax"] ** p - c["cmin"] ** p) / (p * ln) / (4 if c["nz"] else 2)
        return c["windows"] * per, c["windows"] * per * 0.5 * (c["lmin"] + c["lmax"])
    n = c["cx"] * c["cy"] * (c["cz"] or 1)
    if c["kind"] == "analytic":
        steps = int(c["period"] / c["h"]) + 1
        return n * c["fields"], n * c["fields"] * steps
    return n, n * c["steps"]


def work(case):
    c, k = case, case["kind"]
    if k == "pack":
        nodes, dim = math.prod(_shape(c)), len(_shape(c))
        record = 2 * (4 if dim == 3 and c["precision"] != "fp64" else dim)
        return {"bytes": nodes * c["snaps"] * (8 * dim + record * RECORD_BYTES[c["precision"]]),
                "flops": 2 * dim * nodes * c["snaps"]}
    if k == "ftle":
        d, n = c["dim"], c["groups"]
        out = 2 * d * d + 2 if c["chain"] else 1
        return {"bytes": 8 * n * (2 * d * d + d + out), "flops": n * (60 if d == 2 else 400)}
    if k in ("train", "surrogate"):
        h, f, d = c["hidden"], 2 * c["freqs"], c["dim"]
        macs = f * h + (c["depth"] - 1) * h * h + h * d
        n = c["batch"] if k == "train" else c["seeds"]
        rows = 3 if k == "train" else 1 + d
        params = macs + c["depth"] * h + d
        return {"bytes": n * 8 * (d + 2) + params * (28 if k == "train" else 2),
                "flops": 2 * macs * n * rows}
    dim = 3 if c.get("cz") or c.get("nz") else 2
    groups, steps = _particle_steps(c)
    stages = 4 if c["integrator"] == "rk4" else 1
    if k == "analytic":
        flops = (60 if dim == 2 else 90) * 2 * dim * steps * stages
        return {"bytes": 8 * groups * (4 * dim * dim + 1), "flops": flops}
    precision = c.get("precision", "fp64")
    nodes = math.prod(_shape(c))
    given = 8 if k in ("steps", "solver") else RECORD_BYTES[precision]
    hold = _snap_dt(c) == c["h"]
    snaps = c["steps"] if hold else c["snaps"]
    # the snapshots are read once where the particles visit every cell, else what they gather
    gathers = 2 * dim * steps * stages * 2 ** dim * (1 if hold else 2)
    bytes_ = min(snaps * nodes, gathers) * dim * given + 8 * groups * (2 * dim * dim + 1)
    per_stage = (40 if dim == 2 else 80) + (0 if hold else 3 * dim * 2 ** dim)
    return {"bytes": bytes_, "flops": per_stage * 2 * dim * steps * stages}


# ---------------------------------------------------------------------------
# the same in 64 bits, in plain torch
# ---------------------------------------------------------------------------


def _field(c, grid, snaps, periodic_time, hold, step, t, x):
    """Multilinear velocity at x (M, dim): snapshot `step` (hold) or blended at time t."""
    shape, origin, spacing, periodic = grid
    S = snaps.shape[0]
    if hold:
        pair = [(snaps[step], 1.0)]
    else:
        tau = t / _snap_dt(c)
        if periodic_time:
            tau %= S
        tau = min(max(tau, 0.0), S if periodic_time else S - 1.0)
        s = min(int(tau), S - 1 if periodic_time else S - 2)
        pair = [(snaps[s], 1.0 - (tau - s)), (snaps[(s + 1) % S], tau - s)]
    idx, frac, inside = [], [], None
    for a, n in enumerate(shape):
        p = (x[:, a] - origin[a]) / spacing[a]
        q = torch.floor(p)
        frac.append(p - q)
        i = q.long()
        if periodic:
            i0 = i % n
            idx.append((i0, (i0 + 1) % n))
        else:
            ok = (p >= 0) & (p < n - 1)
            inside = ok if inside is None else inside & ok
            i0 = i.clamp(0, n - 2)
            idx.append((i0, i0 + 1))
    u = torch.zeros_like(x)
    for corner in range(1 << len(shape)):
        w, j = None, [idx[a][(corner >> a) & 1] for a in range(len(shape))]
        for a in range(len(shape)):
            f = frac[a] if (corner >> a) & 1 else 1.0 - frac[a]
            w = f if w is None else w * f
        node = j[1] * shape[0] + j[0]
        if len(shape) == 3:
            node = node * shape[2] + j[2]
        for snap, weight in pair:
            u += (w * weight)[:, None] * snap[:, node].T
    return u if inside is None else torch.where(inside[:, None], u, torch.zeros_like(u))


def _advect(velocity, x, integrator, h, steps, t0):
    prev = None
    for i in range(steps):
        t = t0 + i * h
        if integrator == "rk4":
            k1 = velocity(i, t, x)
            k2 = velocity(i, t + 0.5 * h, x + 0.5 * h * k1)
            k3 = velocity(i, t + 0.5 * h, x + 0.5 * h * k2)
            k4 = velocity(i, t + h, x + h * k3)
            x = x + (h / 6.0) * (k1 + 2.0 * k2 + 2.0 * k3 + k4)
        else:
            v = velocity(i, t, x)
            x = x + h * (v if prev is None else 1.5 * v - 0.5 * prev)
            prev = v if integrator == "ab2" else None
    return x


def _jacobian(p0, p1):
    dim = p0.shape[1]
    a, b = (p.view(2 * dim, -1, dim) for p in (p0, p1))
    cols = []
    for j in range(dim):
        hi, lo = (1, 0) if j == 0 else (2 * j, 2 * j + 1)
        cols.append((b[hi] - b[lo]) / (a[hi] - a[lo])[:, j:j + 1])
    return torch.stack(cols, dim=2)


def _lambda_max(cg):
    if cg.shape[1] == 2:
        a, b, d = cg[:, 0, 0], cg[:, 0, 1], cg[:, 1, 1]
        return 0.5 * (a + d) + torch.hypot(0.5 * (a - d), b)
    return torch.cat([torch.linalg.eigvalsh(x)[:, -1] for x in cg.split(1 << 13)])


def _ftle(jac, period):
    return torch.log(torch.sqrt(_lambda_max(jac.transpose(1, 2) @ jac))) / period


def _flow_map(c, seed, snaps, seeds, steps, t0):
    """Final positions of a gridded case, in pieces that fit beside the snapshots."""
    grid, hold, pt = _grid(c), _snap_dt(c) == c["h"], _periodic_time(c)

    def velocity(i, t, x):
        return _field(c, grid, snaps, pt, hold, i, t, x)

    return torch.cat([_advect(velocity, x, c["integrator"], c["h"], steps, t0)
                      for x in seeds.split(1 << 22)])


def _closed_form(c, seed, t, x):
    if c["flow"] == "gyre":
        A, eps, om = _gyre_params(seed)
        e = eps * math.sin(om * t)
        f = e * x[:, 0] ** 2 + (1.0 - 2.0 * e) * x[:, 0]
        df = 2.0 * e * x[:, 0] + (1.0 - 2.0 * e)
        return torch.stack((-math.pi * A * torch.sin(math.pi * f) * torch.cos(math.pi * x[:, 1]),
                            math.pi * A * torch.cos(math.pi * f) * torch.sin(math.pi * x[:, 1])
                            * df), dim=1)
    A, B, C = _abc_params(seed)
    At = A + 0.1 * math.sin(t)
    s, o = torch.sin(x), torch.cos(x)
    return torch.stack((At * s[:, 2] + C * o[:, 1], B * s[:, 0] + At * o[:, 2],
                        C * s[:, 1] + B * o[:, 0]), dim=1)


def _net_exact(c, seed):
    """(FP32 weights, frequency rows) of _net's network, drawn as its constructor draws."""
    rng = np.random.default_rng(seed)
    dims = [2 * c["freqs"]] + [c["hidden"]] * c["depth"]
    ws = []
    for l, fan in enumerate(dims):
        last = l == c["depth"]
        std = 0.1 / math.sqrt(fan) if last else math.sqrt(2.0 / fan)
        w = rng.normal(0.0, std, (c["dim"] if last else c["hidden"], fan)).astype(np.float32)
        ws.append(torch.from_numpy(w).cuda())
    return ws, torch.from_numpy(_freq(c, seed)).cuda().double()


def _features(c, freq, p):
    d = c["dim"]
    ph = p @ freq[:, :d + 1].T + freq[:, d + 1]
    return torch.sin(ph), torch.cos(ph)


def _net_ftle(c, seed, pts, period):
    ws, freq = _net_exact(c, seed)
    ws = [w.bfloat16().double() for w in ws]  # the weights that the network evaluates
    d, out = c["dim"], []
    for p in pts.split(1 << 15):
        s, o = _features(c, freq, p)
        h = torch.cat((s, o), dim=1)
        tan = [torch.cat((freq[:, a] * o, -freq[:, a] * s), dim=1) for a in range(d)]
        for w in ws[:-1]:
            z = h @ w.T
            sg = torch.sigmoid(z)
            tan = [(t @ w.T) * (sg * (1.0 + z * (1.0 - sg))) for t in tan]
            h = z * sg
        jac = torch.stack([t @ ws[-1].T for t in tan], dim=2)
        out.append(_ftle(torch.eye(d, dtype=F64, device="cuda") + 0.05 * jac, period))
    return torch.cat(out)


def exact(case, seed):
    c, k = case, case["kind"]
    if k == "pack":
        return None
    if k in ("steps", "solver", "window"):
        stages = 4 if c["integrator"] == "rk4" else 1
        if 2 * _particle_steps(c)[1] * stages * (3 if c["nz"] else 2) > 3e9:
            return None
        seeds = _seeds(c, seed)
        snaps = _snapshots(c, seed, c["steps"] if k == "steps" else c["snaps"])
        x = _flow_map(c, seed, snaps, seeds, c["steps"], 0.0)
        hold = _snap_dt(c) == c["h"]
        f = _ftle(_jacobian(seeds, x), (c["steps"] - hold) * c["h"])
        if k == "steps":
            return x, f
        if k == "solver":
            return f.cpu().numpy()
        return (f, x) if c["update"] else f
    if k == "batch":
        stages = 4 if c["integrator"] == "rk4" else 1
        if 2 * _particle_steps(c)[1] * stages * (3 if c["nz"] else 2) > 1.5e9:
            return None
        snaps, out = _snapshots(c, seed, c["snaps"]), []
        for cx, cy, cz, steps, t0 in _batch_windows(c, seed):
            seeds = _groups(_centroids(c, seed, cx, cy, cz))
            x = _flow_map(c, seed, snaps, seeds, steps, t0)
            out.append(_ftle(_jacobian(seeds, x), steps * c["h"]))
        return out
    if k == "analytic":
        seeds, out = _seeds(c, seed), []
        steps = int(c["period"] / c["h"]) + 1
        for i in range(c["fields"]):
            x = _advect(lambda _, t, y: _closed_form(c, seed, t, y), seeds, c["integrator"],
                        c["h"], steps, i * c["h"])
            out.append(_ftle(_jacobian(seeds, x), (steps - 1) * c["h"]))
        out = torch.stack(out).cpu().numpy()
        return out[0] if c["fields"] == 1 else out
    if k == "ftle":
        jac = _jacobian(*_deformed(c, seed))
        f = _ftle(jac, 2.0)
        if not c["chain"]:
            return f
        cg = jac.transpose(1, 2) @ jac if c["dim"] == 2 else jac @ jac.transpose(1, 2)
        return jac, cg, _lambda_max(cg), f
    if k == "surrogate":
        pts, _ = _net_points(c, seed, c["seeds"], t0=1.0)
        return _net_ftle(c, seed, pts, 5.0)
    pts, target, g = _train_inputs(c, seed)
    w0, freq = _net_exact(c, seed)
    ws = [w.bfloat16().double().requires_grad_(True) for w in w0]
    bs = [torch.zeros(w.shape[0], dtype=F64, device="cuda", requires_grad=True) for w in ws]
    loss = torch.zeros(1, dtype=F64, device="cuda")
    h = torch.cat(_features(c, freq, pts), dim=1)
    for hh, tt in zip(h.split(1 << 13), target.double().split(1 << 13)):
        for w, b in zip(ws[:-1], bs[:-1]):
            hh = torch.nn.functional.silu(hh @ w.T + b)
        part = (hh @ ws[-1].T + bs[-1] - tt).square().sum() / c["batch"]
        part.backward()
        loss += part.detach()
    # flat parameters: each layer's weights, then its biases; 64 rows in the output layer
    grads, params = [], []
    for l, (w, b) in enumerate(zip(ws, bs)):
        pad = 64 - w.shape[0] if l == c["depth"] else 0
        for flat, v, u in ((grads, w.grad, b.grad), (params, w0[l].double(), b.detach())):
            flat += [torch.nn.functional.pad(v, (0, 0, 0, pad)).reshape(-1),
                     torch.nn.functional.pad(u, (0, pad))]
    grad, w = torch.cat(grads), torch.cat(params)
    m = torch.empty(w.numel(), device="cuda").normal_(0.0, 1e-3, generator=g).double()
    v = torch.empty(w.numel(), device="cuda").uniform_(1e-6, 2e-6, generator=g).double()
    m, v = 0.9 * m + 0.1 * grad, 0.999 * v + 0.001 * grad * grad
    c1, c2 = 1.0 - 0.9 ** 1001, 1.0 - 0.999 ** 1001
    w = w - 1e-3 * (m / c1) / (torch.sqrt(v / c2) + 1e-8)
    return dict(loss=loss, w=w, m=m, v=v)
