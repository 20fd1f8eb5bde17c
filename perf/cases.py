"""Timed cases of flursys_b200: what programs that use the framework have it do.

A solver pass is a restart: the state held in page-locked host memory goes
into the solver, the solver advances, and every field of the new state comes
back (``handle.upload`` / ``advance`` / ``handle.download``), so that each pass
does the same work. The batched solver, which has no upload, steps on from
rest. Pressure systems are solved to 1e-12 rather than the benchmark's 1e-8,
which determines the fields, the pressure of the largest grids included, to
the digits that two correct solvers may be held to; an iteration costs the
same.

``exact`` restates each step in 64-bit torch with a direct solve of the
pressure system (cosine transforms on boxes, conjugate gradients run to
rounding where there are solid or outlet cells).
"""
import math

import numpy as np
import torch

from flursys_b200 import (BackendOptions, BatchedIncompressibleSolver, Case, CavityCase, CylinderCase,
                          IncompressibleSolver, LidDrivenCavity3DConfig, LidDrivenCavity3DSolver, SimulationConfig,
                          TimeStepSettings, _abi)
from flursys_b200.learned import CIN, COUT, DEFAULT_WEIGHTS, FcgNet, init_params
from flursys_b200.solver import ChannelSimpleConfig, solve_simple_channel

DEV = "cuda"
RTOL = 1e-12
BATCH_RTOL = 3e-11  # a warm start begins where 1e-12 of its residual is below what mixed precision reaches
ITERS = 60000
F64 = torch.float64


def listed():
    return [
        # the smallest step a program takes: a coarse grid, all latency
        {"name": "cavity2d_48x40_f64", "kind": "cavity2d", "nx": 48, "ny": 40, "precision": "f64",
         "convection": "upwind"},
        # the 2D benchmark grid: 128 x 128, upwind, the default precision
        {"name": "cavity2d_128_f64", "kind": "cavity2d", "nx": 128, "ny": 128, "precision": "f64",
         "convection": "upwind"},
        # a large 2D grid with odd sides in mixed precision, central convection
        {"name": "cavity2d_509x331_mixed", "kind": "cavity2d", "nx": 509, "ny": 331, "precision": "mixed",
         "convection": "central"},
        # flow past a body: solid cells, symmetry sides and a pressure outlet
        {"name": "cylinder_250x100_f64", "kind": "cylinder", "nx": 250, "ny": 100, "precision": "f64",
         "convection": "upwind"},
        # many 2D cavities of uneven size advanced together (the batched workload)
        {"name": "batch2d_64", "kind": "batch", "count": 64, "lo": 64, "hi": 512, "precision": "mixed"},
        # the 3D configuration's own defaults: 32^3, SOR, 64 bits
        {"name": "cavity3d_32_sor", "kind": "cavity3d", "nx": 32, "ny": 32, "nz": 32, "precision": "f64",
         "solver": "sor"},
        # a 3D box with odd sides at the default precision
        {"name": "cavity3d_75x62x51_f64", "kind": "cavity3d", "nx": 75, "ny": 62, "nz": 51, "precision": "f64",
         "solver": "pcg"},
        # the 3D benchmark grid in mixed precision
        {"name": "cavity3d_128_mixed", "kind": "cavity3d", "nx": 128, "ny": 128, "nz": 128, "precision": "mixed",
         "solver": "pcg"},
        # the largest 3D grid of the benchmark, plain conjugate gradients
        {"name": "cavity3d_256_mixed", "kind": "cavity3d", "nx": 256, "ny": 256, "nz": 256, "precision": "mixed",
         "solver": "pcg"},
        # the same grid with the learned preconditioner (network inference)
        {"name": "cavity3d_256_fcg", "kind": "cavity3d", "nx": 256, "ny": 256, "nz": 256, "precision": "mixed",
         "solver": "fcg"},
        # steady SIMPLE on the channel: CSR assembly, BiCGSTAB and CG in 64 bits
        {"name": "channel_1024x256", "kind": "channel", "nx": 1024, "ny": 256, "outer": 2},
        # one gradient of the preconditioner's training: forward and backward
        {"name": "train_64", "kind": "train", "n": 64, "batch": 4},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["cavity2d", "cavity2d", "cylinder", "batch", "sor", "pcg", "pcg", "pcg", "fcg", "channel",
                       "train"])
    if kind == "cavity2d":
        return {"kind": kind, "nx": _log(rng, 24, 700), "ny": _log(rng, 24, 700),
                "precision": rng.choice(["f64", "mixed"]), "convection": rng.choice(["upwind", "central"])}
    if kind == "cylinder":
        nx = _log(rng, 75, 450)
        return {"kind": kind, "nx": nx, "ny": int(nx * rng.uniform(0.35, 0.45)),
                "precision": rng.choice(["f64", "mixed"]), "convection": rng.choice(["upwind", "central"])}
    if kind == "batch":
        return {"kind": kind, "count": _log(rng, 2, 48), "lo": 64, "hi": rng.randint(96, 448), "precision": "mixed"}
    if kind == "channel":
        return {"kind": kind, "nx": _log(rng, 96, 1024), "ny": _log(rng, 32, 256), "outer": 2}
    if kind == "train":
        return {"kind": kind, "n": 8 * rng.randint(4, 12), "batch": rng.randint(1, 4)}
    if kind == "sor":
        side = [_log(rng, 12, 44) for _ in range(3)]
        return {"kind": "cavity3d", "nx": side[0], "ny": side[1], "nz": side[2], "precision": "f64", "solver": "sor"}
    if kind == "fcg":
        side = [8 * rng.randint(5, 20) for _ in range(3)]
        return {"kind": "cavity3d", "nx": side[0], "ny": side[1], "nz": side[2], "precision": "mixed",
                "solver": "fcg"}
    precision = rng.choice(["f64", "mixed", "mixed"])
    hi = 112 if precision == "f64" else 208
    side = [_log(rng, 20, hi) for _ in range(3)]
    return {"kind": "cavity3d", "nx": side[0], "ny": side[1], "nz": side[2], "precision": precision, "solver": "pcg"}


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _sines(n, points, kmax):
    """sin(k pi x) at x = points / n, exactly 0 on the walls."""
    k = torch.arange(1, kmax + 1, dtype=F64, device=DEV)
    t = torch.sin(math.pi / n * torch.outer(points, k))
    t[(points == 0) | (points == n)] = 0.0
    return t


def _line(n, mid):
    p = torch.arange(n if mid else n + 1, dtype=F64, device=DEV)
    return p + 0.5 if mid else p


def _flow2d(nx, ny, lx, ly, seed, peak):
    """Discretely divergence-free face velocities (the differences of a random
    stream function that is 0 on the walls), |u| at most `peak`."""
    km = 6
    rng = np.random.default_rng(seed)
    k = np.arange(1, km + 1)
    c = rng.standard_normal((km, km)) / (k[:, None] ** 2 + k[None, :] ** 2)
    c = torch.from_numpy(c).to(DEV)
    psi = _sines(ny, _line(ny, False), km) @ c @ _sines(nx, _line(nx, False), km).T
    u = (psi[1:, :] - psi[:-1, :]) * (ny / ly)
    v = -(psi[:, 1:] - psi[:, :-1]) * (nx / lx)
    s = peak / max(float(u.abs().max()), float(v.abs().max()))
    return u * s, v * s


def _flow3d(nx, ny, nz, seed, peak=0.5):
    """The same in 3D: the discrete curl of a random vector potential with
    sine modes of amplitude |k|^-2."""
    km = 6
    rng = np.random.default_rng(seed)
    k = np.arange(1, km + 1)
    kk = k[:, None, None] ** 2 + k[None, :, None] ** 2 + k[None, None, :] ** 2
    coef = [torch.from_numpy(rng.standard_normal((km, km, km)) / kk).to(DEV) for _ in range(3)]

    def potential(c, mx, my, mz):  # [z][y][x]
        sx, sy, sz = (_sines(n, _line(n, m), km) for n, m in ((nx, mx), (ny, my), (nz, mz)))
        return torch.einsum("kc,abc,jb,ia->kji", sz, c, sy, sx)

    ax = potential(coef[0], True, False, False)
    ay = potential(coef[1], False, True, False)
    az = potential(coef[2], False, False, True)
    u = torch.diff(az, dim=1) * ny - torch.diff(ay, dim=0) * nz
    v = torch.diff(ax, dim=0) * nz - torch.diff(az, dim=2) * nx
    w = torch.diff(ay, dim=2) * nx - torch.diff(ax, dim=1) * ny
    s = peak / max(float(t.abs().max()) for t in (u, v, w))
    return u * s, v * s, w * s


def _solid(case):
    """Cells inside the cylinder of CylinderCase's defaults (25 x 10, centre
    (5, 5), diameter 1), as [ny][nx]."""
    x = _line(case["nx"], True) * (25.0 / case["nx"]) - 5.0
    y = _line(case["ny"], True) * (10.0 / case["ny"]) - 5.0
    return x[None, :] ** 2 + y[:, None] ** 2 <= 0.25


def _open(solid):
    ny, nx = solid.shape
    uo = torch.ones(ny, nx + 1, dtype=torch.bool, device=DEV)
    uo[:, :-1] &= ~solid
    uo[:, 1:] &= ~solid
    vo = torch.ones(ny + 1, nx, dtype=torch.bool, device=DEV)
    vo[:-1] &= ~solid
    vo[1:] &= ~solid
    return uo, vo


def _inputs2d(case, seed):
    nx, ny = case["nx"], case["ny"]
    if case["kind"] == "cavity2d":
        return _flow2d(nx, ny, 1.0, 1.0, seed, 0.6)
    u, v = _flow2d(nx, ny, 25.0, 10.0, seed, 0.3)
    uo, vo = _open(_solid(case))
    return torch.where(uo, u + 1.0, 0.0), torch.where(vo, v, 0.0)


def _dt2d(case):
    if case["kind"] == "cavity2d":
        h, nu = 1.0 / max(case["nx"], case["ny"]), 0.01
    else:
        h, nu = min(25.0 / case["nx"], 10.0 / case["ny"]), 0.01
    return min(0.25 * h, 0.1 * h * h / nu)


def _dt3d(case):
    h = 1.0 / max(case["nx"], case["ny"], case["nz"])
    return 5.0e-4 if case["solver"] == "sor" else min(0.5 * h, 0.25 * h * h * 400.0 / 3.0)


def _config2d(case, dt):
    c = Case.lid_driven_cavity(CavityCase()) if case["kind"] == "cavity2d" else Case.cylinder(CylinderCase())
    return SimulationConfig(case=c, nx=case["nx"], ny=case["ny"], dt=dt, t_end=1e9, max_steps=1 << 40,
                            minimum_steps=1 << 40, convection=case["convection"], pressure_max_iters=ITERS,
                            backend=BackendOptions(precision=case["precision"], stop_rule="rel-l2",
                                                   pressure_rtol=RTOL))


def _config3d(case):
    if case["solver"] == "sor":  # LidDrivenCavity3DConfig's defaults
        return LidDrivenCavity3DConfig(nx=case["nx"], ny=case["ny"], nz=case["nz"])
    weights = DEFAULT_WEIGHTS if case["solver"] == "fcg" else None
    return LidDrivenCavity3DConfig(nx=case["nx"], ny=case["ny"], nz=case["nz"], reynolds=400.0, dt=_dt3d(case),
                                   pressure_solver=case["solver"], pressure_max_iters=ITERS,
                                   backend=BackendOptions(precision=case["precision"], stop_rule="rel-l2",
                                                          pressure_rtol=RTOL,
                                                          fcg_weights_path=weights))


def _batch_configs(case, seed):
    rng = np.random.default_rng(seed)
    # the largest instance is always there, so that seeds cost alike
    sides = [case["hi"]] + [int(s) for s in np.random.default_rng(7).integers(case["lo"], case["hi"] + 1,
                                                                            size=case["count"] - 1)]
    return [(s, float(re)) for s, re in zip(sides, rng.uniform(100.0, 2000.0, size=case["count"]))]


def _channel_config(case, seed):
    rng = np.random.default_rng(seed)
    return ChannelSimpleConfig(nx=case["nx"], ny=case["ny"], reynolds=float(rng.uniform(50.0, 400.0)),
                               inlet_peak_velocity=float(rng.uniform(0.5, 1.5)),
                               max_outer_iterations=case["outer"], continuity_tolerance=0.0,
                               momentum_solver=(1e-13, 1e-11, 20000), pressure_solver=(1e-13, 1e-10, 60000))


def _pairs(case, seed):
    """Training pairs (b, p) with L p = b on the unit-spacing Neumann operator
    and b of unit RMS: a smooth part and a rough one, as solver residuals have."""
    n, out = case["n"], []
    gen = torch.Generator().manual_seed(seed)
    for _ in range(case["batch"]):
        c = torch.randn(8, 8, 8, generator=gen, dtype=F64).to(DEV)
        k = torch.arange(8, dtype=F64, device=DEV)
        t = torch.cos(math.pi / n * torch.outer(_line(n, True), k))
        p = torch.einsum("kc,abc,jb,ia->kji", t, c / (1.0 + k[:, None, None] + k[:, None] + k) ** 2, t, t)
        p = p + 1e-3 * torch.randn(n, n, n, generator=gen, dtype=F64).to(DEV)
        p = p - p.mean()
        b = _neumann(p)
        s = float(b.square().mean().sqrt())
        b, p = (b / s).float().contiguous(), (p / s).float().contiguous()
        out.append((b, p, float(b.double().square().sum())))
    return out


def _pinned(t):
    return t.detach().to("cpu", F64).contiguous().flatten().pin_memory().numpy()


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        cfgs = [SimulationConfig(case=Case.lid_driven_cavity(CavityCase(reynolds=re)), nx=s, ny=s, dt=1e-3,
                                 time_step=TimeStepSettings(adaptive=True), t_end=1e9, max_steps=1 << 40,
                                 minimum_steps=1 << 40, pressure_max_iters=ITERS,
                                 backend=BackendOptions(precision=case["precision"], stop_rule="rel-l2",
                                                        pressure_rtol=BATCH_RTOL))
                for s, re in _batch_configs(case, seed)]
        return {"kind": kind, "solver": BatchedIncompressibleSolver(cfgs)}
    if kind == "channel":
        return {"kind": kind, "config": _channel_config(case, seed)}
    if kind == "train":
        params = init_params(seed)
        w = torch.from_numpy(params).to(DEV)
        return {"kind": kind, "net": FcgNet(params), "weights": w, "grad": torch.zeros_like(w),
                "loss": torch.zeros(1, dtype=F64, device=DEV), "pairs": _pairs(case, seed), "n": case["n"]}
    if kind == "cavity3d":
        solver = LidDrivenCavity3DSolver(_config3d(case))
        fields = list(zip((_abi.FIELD_U, _abi.FIELD_V, _abi.FIELD_W),
                          _flow3d(case["nx"], case["ny"], case["nz"], seed)))
        cells = case["nx"] * case["ny"] * case["nz"]
    else:
        solver = IncompressibleSolver(_config2d(case, _dt2d(case)))
        fields = list(zip((_abi.FIELD_U, _abi.FIELD_V), _inputs2d(case, seed)))
        cells = case["nx"] * case["ny"]
    fields.append((_abi.FIELD_PRESSURE, torch.zeros(cells, dtype=F64)))
    start = [(f, _pinned(t)) for f, t in fields]
    return {"kind": kind, "solver": solver, "start": start,
            "out": {f: _pinned(torch.zeros(a.size)) for f, a in start}}


def run(s):
    kind = s["kind"]
    if kind == "batch":
        b = s["solver"]
        b.advance(1)
        return [np.concatenate([b.field(i, name) for i in range(len(b))]) for name in ("u", "v", "pressure")]
    if kind == "channel":
        r = solve_simple_channel(s["config"])
        return [r["u"], r["v"], r["p"], r["flux"]]
    if kind == "train":
        s["grad"].zero_()
        s["loss"].zero_()
        s["net"].set_params_device(s["weights"])
        for b, p, norm in s["pairs"]:
            s["net"].train_sample(b, p, norm, s["grad"], s["loss"], (s["n"],) * 3)
        return [s["grad"], s["loss"]]
    h = s["solver"].handle
    for f, a in s["start"]:
        h.upload(f, a)
    if kind == "cavity3d":
        s["solver"].advance(1)
    else:
        s["solver"].advance()
    return [h.download(f, out) for f, out in s["out"].items()]


# ---------------------------------------------------------------------------
# work
# ---------------------------------------------------------------------------
def _iterations(case):
    """Iterations that (preconditioned) conjugate gradients need, within a
    factor of about 1.5: they grow with the longest side."""
    if case["kind"] == "cylinder":
        return 4.5 * max(case["nx"], case["ny"])
    if case["kind"] == "cavity2d":
        return 6.0 * max(case["nx"], case["ny"])
    side = max(case["nx"], case["ny"], case["nz"])
    if case["solver"] == "fcg":
        return 0.38 * side
    return 11.0 * side


def work(case):
    """Bytes: the state read once and the new state written once. Flops: the
    iterations' operator, inner products and vector updates, about 20 per cell
    and iteration; the network's convolutions where it is applied."""
    kind = case["kind"]
    if kind == "train":
        n3, conv = case["n"] ** 3, 0.0
        for (a, b), down in zip(zip(CIN, COUT), (1, 8, 64, 512, 64, 8, 1)):
            conv += 2.0 * 27 * a * b * n3 / down
        return {"bytes": 8.0 * n3 * case["batch"], "flops": 3.0 * conv * case["batch"]}
    if kind == "batch":
        sides = [s for s, _ in _batch_configs(case, 0)]
        return {"bytes": sum(48.0 * s * s for s in sides), "flops": sum(20.0 * 6.0 * s ** 3 for s in sides)}
    if kind == "channel":
        n = case["nx"] * case["ny"]
        return {"bytes": 40.0 * n, "flops": 20.0 * n * 2.9 * case["nx"] * case["outer"]}
    if kind == "cavity3d":
        n = case["nx"] * case["ny"] * case["nz"]
        flops = 20.0 * n * _iterations(case)
        if case["solver"] == "fcg":
            flops += _iterations(case) * n * 2.0 * 27 * (16 + 512 / 8 + 2048 / 64 + 4096 / 512 + 2048 / 64 + 512 / 8 + 16)
        return {"bytes": 64.0 * n, "flops": flops}
    n = case["nx"] * case["ny"]
    return {"bytes": 48.0 * n, "flops": 20.0 * n * _iterations(case)}


# ---------------------------------------------------------------------------
# the same results in 64-bit torch
# ---------------------------------------------------------------------------
def _cosines(n):
    """Orthonormal eigenvectors (columns) and eigenvalues of the 1D Neumann
    second difference."""
    k = torch.arange(n, dtype=F64, device=DEV)
    t = torch.cos(math.pi / n * torch.outer(k + 0.5, k)) * math.sqrt(2.0 / n)
    t[:, 0] = math.sqrt(1.0 / n)
    return t, 2.0 - 2.0 * torch.cos(math.pi / n * k)


def _solve_box(b, inv_h2):
    """Zero-mean x with A x = b - mean(b), A the positive Neumann operator;
    axes are ordered (z,) y, x and inv_h2 with them."""
    lam = torch.zeros((1,) * b.dim(), dtype=F64, device=DEV)
    vecs = []
    for ax, w in enumerate(inv_h2):
        t, l = _cosines(b.shape[ax])
        vecs.append(t)
        lam = lam + (w * l).reshape([-1 if a == ax else 1 for a in range(b.dim())])
    for ax, t in enumerate(vecs):
        b = torch.movedim(torch.tensordot(b, t, dims=([ax], [0])), -1, ax)
    lam.view(-1)[0] = 1.0
    b = b / lam
    b.view(-1)[0] = 0.0
    for ax, t in enumerate(vecs):
        b = torch.movedim(torch.tensordot(b, t, dims=([ax], [1])), -1, ax)
    return b.contiguous()


def _solve_masked(b, fluid, wet, ix2, iy2):
    """Conjugate gradients to rounding: fluid rows couple to wet neighbours;
    other cells are 0."""
    m = wet.to(F64)
    ex, ey = m[:, 1:] * m[:, :-1] * ix2, m[1:] * m[:-1] * iy2
    diag = torch.zeros_like(b)
    diag[:, :-1] += ex
    diag[:, 1:] += ex
    diag[:-1] += ey
    diag[1:] += ey
    f = fluid.to(F64)
    inv = torch.where(diag > 0, 1.0 / diag, 0.0) * f

    def apply(x):
        q = diag * x
        q[:, :-1] -= ex * x[:, 1:]
        q[:, 1:] -= ex * x[:, :-1]
        q[:-1] -= ey * x[1:]
        q[1:] -= ey * x[:-1]
        return q * f

    x, b = torch.zeros_like(b), b * f
    for _ in range(2):  # the second solve, for the residual of the first, removes its rounding
        r = b - apply(x)
        z = inv * r
        d, rz = z.clone(), (r * z).sum()
        stop = float(r.norm()) * 1e-13
        for it in range(20000):
            q = apply(d)
            a = rz / (d * q).sum()
            x += a * d
            r -= a * q
            z = inv * r
            new = (r * z).sum()
            if it % 50 == 49 and float(r.norm()) <= stop:
                break
            d = z + (new / rz) * d
            rz = new
    return x


def _transport(scheme, f, left, right):
    return torch.where(f >= 0, left, right) if scheme == "upwind" else 0.5 * (left + right)


def _step2d(u, v, solid, cavity, scheme, dt, nu, lx, ly, lid=1.0):
    """One projection step (unit density): u [ny][nx+1], v [ny+1][nx]. The
    cavity has four walls and a lid; otherwise an inflow of 1 on the left, an
    outlet of pressure 0 on the right and symmetry above and below."""
    ny, nx = v.shape[0] - 1, v.shape[1]
    dx, dy = lx / nx, ly / ny
    uo, vo = _open(solid)

    def boundaries(u, v):
        u[:, 0] = 0.0 if cavity else 1.0
        u[:, -1] = 0.0 if cavity else u[:, -2]
        v[0] = 0.0
        v[-1] = 0.0

    c = u[:, 1:-1]
    e = torch.where(uo[:, 2:], u[:, 2:], -c)
    w = torch.where(uo[:, :-2], u[:, :-2], -c)
    up, down = torch.empty_like(c), torch.empty_like(c)
    up[:-1] = torch.where(uo[1:, 1:-1], c[1:], -c[:-1])
    up[-1] = 2.0 * lid - c[-1] if cavity else c[-1]
    down[1:] = torch.where(uo[:-1, 1:-1], c[:-1], -c[1:])
    down[0] = -c[0] if cavity else c[0]
    fe, fw = 0.5 * (c + e), 0.5 * (w + c)
    fn, fs = 0.5 * (v[1:, :-1] + v[1:, 1:]), 0.5 * (v[:-1, :-1] + v[:-1, 1:])
    conv = (fe * _transport(scheme, fe, c, e) - fw * _transport(scheme, fw, w, c)) / dx + \
           (fn * _transport(scheme, fn, c, up) - fs * _transport(scheme, fs, down, c)) / dy
    diff = (e - 2.0 * c + w) / dx ** 2 + (up - 2.0 * c + down) / dy ** 2
    us = torch.zeros_like(u)
    us[:, 1:-1] = torch.where(uo[:, 1:-1], c + dt * (nu * diff - conv), 0.0)

    c = v[1:-1]
    up = torch.where(vo[2:], v[2:], -c)
    down = torch.where(vo[:-2], v[:-2], -c)
    e, w = torch.empty_like(c), torch.empty_like(c)
    e[:, :-1] = torch.where(vo[1:-1, 1:], c[:, 1:], -c[:, :-1])
    e[:, -1] = -c[:, -1] if cavity else c[:, -1]
    w[:, 1:] = torch.where(vo[1:-1, :-1], c[:, :-1], -c[:, 1:])
    w[:, 0] = -c[:, 0]
    fe, fw = 0.5 * (u[:-1, 1:] + u[1:, 1:]), 0.5 * (u[:-1, :-1] + u[1:, :-1])
    fn, fs = 0.5 * (c + up), 0.5 * (down + c)
    conv = (fe * _transport(scheme, fe, c, e) - fw * _transport(scheme, fw, w, c)) / dx + \
           (fn * _transport(scheme, fn, c, up) - fs * _transport(scheme, fs, down, c)) / dy
    diff = (e - 2.0 * c + w) / dx ** 2 + (up - 2.0 * c + down) / dy ** 2
    vs = torch.zeros_like(v)
    vs[1:-1] = torch.where(vo[1:-1], c + dt * (nu * diff - conv), 0.0)
    boundaries(us, vs)

    rhs = (torch.diff(us, dim=1) / dx + torch.diff(vs, dim=0) / dy) / dt
    if cavity:
        p = _solve_box(-rhs, (1.0 / dy ** 2, 1.0 / dx ** 2))
    else:
        fluid = ~solid
        fluid[:, -1] = False
        p = _solve_masked(-rhs, fluid, ~solid, 1.0 / dx ** 2, 1.0 / dy ** 2)
    un, vn = us.clone(), vs.clone()
    un[:, 1:-1] = torch.where(uo[:, 1:-1], us[:, 1:-1] - dt * torch.diff(p, dim=1) / dx, 0.0)
    vn[1:-1] = torch.where(vo[1:-1], vs[1:-1] - dt * torch.diff(p, dim=0) / dy, 0.0)
    boundaries(un, vn)
    return un, vn, p


def _sor_box(rhs, inv_h2, cfg):
    """Red-black SOR sweeps from 0 with p(0, 0, 0) held at 0, until the largest
    residual elsewhere is below the tolerance or the sweeps run out; a missing
    neighbour takes the centre value."""
    grid = torch.meshgrid(*[torch.arange(n, device=DEV) for n in rhs.shape], indexing="ij")
    colour = (grid[0] + grid[1] + grid[2]) % 2
    free = torch.ones_like(colour, dtype=torch.bool)
    free[0, 0, 0] = False
    masks = [(colour == c) & free for c in (0, 1)]
    diag = 2.0 * sum(inv_h2)
    p = torch.zeros_like(rhs)

    def neighbours(p):
        s = 0.0
        for ax, w in enumerate(inv_h2):
            n = p.shape[ax]
            s = s + w * (torch.cat((p.narrow(ax, 1, n - 1), p.narrow(ax, n - 1, 1)), ax) +
                         torch.cat((p.narrow(ax, 0, 1), p.narrow(ax, 0, n - 1)), ax))
        return s

    for _ in range(cfg.pressure_max_iters):
        for m in masks:
            p = torch.where(m, p + cfg.pressure_omega * ((neighbours(p) - rhs) / diag - p), p)
        if float(((neighbours(p) - diag * p - rhs) * free).abs().max()) < cfg.pressure_tolerance:
            break
    return p


def _step3d(u, v, w, dt, nu, lid=1.0, sor=None):
    """One step of the 3D cavity on the unit cube (advective central form);
    `sor`: the configuration whose SOR sweeps stand for the pressure solve."""
    nz, ny, nx = u.shape[0], u.shape[1], v.shape[2]

    def around(c, ax, low, high):
        """The neighbours of c along ax, with wall ghosts low and high."""
        a, b = torch.empty_like(c), torch.empty_like(c)
        n = c.shape[ax]
        a.narrow(ax, 1, n - 1).copy_(c.narrow(ax, 0, n - 1))
        a.narrow(ax, 0, 1).copy_(low)
        b.narrow(ax, 0, n - 1).copy_(c.narrow(ax, 1, n - 1))
        b.narrow(ax, n - 1, 1).copy_(high)
        return a, b

    def predict(q, axis, vel):
        """q's interior faces along its own axis; vel: the advecting velocities there by axis (z, y, x)."""
        n = q.shape[axis]
        c = q.narrow(axis, 1, n - 2)
        adv, lap = 0.0, 0.0
        for ax, cells in ((0, nz), (1, ny), (2, nx)):
            if ax == axis:
                lo, hi = q.narrow(axis, 0, n - 2), q.narrow(axis, 2, n - 2)
            else:
                first, last = c.narrow(ax, 0, 1), c.narrow(ax, c.shape[ax] - 1, 1)
                top = 2.0 * lid - last if (axis == 2 and ax == 1) else -last
                lo, hi = around(c, ax, -first, top)
            adv = adv + vel[ax] * (hi - lo) * (0.5 * cells)
            lap = lap + (hi - 2.0 * c + lo) * float(cells) ** 2
        out = torch.zeros_like(q)
        out.narrow(axis, 1, n - 2).copy_(c + dt * (nu * lap - adv))
        return out

    mid = lambda q, ax: 0.5 * (q.narrow(ax, 0, q.shape[ax] - 1) + q.narrow(ax, 1, q.shape[ax] - 1))  # noqa: E731
    us = predict(u, 2, (mid(mid(w, 0), 2), mid(mid(v, 1), 2), u[:, :, 1:-1]))
    vs = predict(v, 1, (mid(mid(w, 0), 1), v[:, 1:-1], mid(mid(u, 2), 1)))
    ws = predict(w, 0, (w[1:-1], mid(mid(v, 1), 0), mid(mid(u, 2), 0)))
    rhs = (torch.diff(us, dim=2) * nx + torch.diff(vs, dim=1) * ny + torch.diff(ws, dim=0) * nz) / dt
    inv_h2 = (float(nz) ** 2, float(ny) ** 2, float(nx) ** 2)
    if sor is None:
        p = _solve_box(-rhs, inv_h2)
        p = p - p[0, 0, 0]
    else:
        rhs[0, 0, 0] = 0.0
        p = _sor_box(rhs, inv_h2, sor)
    un, vn, wn = u.clone(), v.clone(), w.clone()
    un[:, :, 1:-1] = us[:, :, 1:-1] - dt * torch.diff(p, dim=2) * nx
    vn[:, 1:-1] = vs[:, 1:-1] - dt * torch.diff(p, dim=1) * ny
    wn[1:-1] = ws[1:-1] - dt * torch.diff(p, dim=0) * nz
    return un, vn, wn, p


def _neumann(p):
    q = torch.zeros_like(p)
    for ax in range(3):
        d = torch.diff(p, dim=ax)
        q.narrow(ax, 0, p.shape[ax] - 1).sub_(d)
        q.narrow(ax, 1, p.shape[ax] - 1).add_(d)
    return q


def _network(params, b):
    """The preconditioner's encoder-decoder in 64 bits."""
    w, off = [], 0
    for ci, co in zip(CIN, COUT):
        w.append(params[off:off + 27 * ci * co].reshape(co, 3, 3, 3, ci).permute(0, 4, 1, 2, 3))
        off += 27 * ci * co
    conv = lambda x, k: torch.nn.functional.conv3d(x, w[k], padding=1)  # noqa: E731
    pool = lambda x: torch.nn.functional.avg_pool3d(x, 2)  # noqa: E731
    up = lambda x: torch.nn.functional.interpolate(x, scale_factor=2, mode="nearest")  # noqa: E731
    a1 = conv(b[None, None], 0)
    a2 = conv(pool(a1), 1)
    a3 = conv(pool(a2), 2)
    a4 = conv(pool(a3), 3)
    b3 = conv(up(a4) + a3, 4)
    b2 = conv(up(b3) + a2, 5)
    return conv(up(b2) + a1, 6)[0, 0]


def _exact_train(case, seed):
    torch.backends.cudnn.enabled = False  # plain 64-bit convolutions
    params = torch.from_numpy(init_params(seed)).to(DEV, F64).requires_grad_(True)
    total = 0.0
    for b, p, norm in _pairs(case, seed):
        e = _network(params, b.double()) - p.double()
        q = 0.0
        for ax in range(3):
            d = torch.diff(e, dim=ax)
            pad = [0, 0] * (2 - ax)
            q = q + torch.nn.functional.pad(d, pad + [1, 0]) - torch.nn.functional.pad(d, pad + [0, 1])
        loss = q.square().sum() / norm
        loss.backward()
        total += float(loss.detach())
    return [params.grad, torch.tensor([total], dtype=F64)]


def exact(case, seed):
    kind = case["kind"]
    flat = lambda ts: [t.contiguous().flatten() for t in ts]  # noqa: E731
    if kind == "channel":  # a second SIMPLE solver would be needed
        return None
    if kind == "train":
        return _exact_train(case, seed)
    if kind == "cavity3d":
        sor = _config3d(case) if case["solver"] == "sor" else None
        return flat(_step3d(*_flow3d(case["nx"], case["ny"], case["nz"], seed), _dt3d(case),
                            1.0 / (100.0 if sor else 400.0), sor=sor))
    if kind == "batch":
        parts = [[], [], []]
        ts = TimeStepSettings()
        for s, re in _batch_configs(case, seed):
            u = torch.zeros(s, s + 1, dtype=F64, device=DEV)
            v = torch.zeros(s + 1, s, dtype=F64, device=DEV)
            nu, h = 1.0 / re, 1.0 / s
            # from rest only the diffusion number bounds the step
            dt = min(ts.max_dt, ts.target_diffusion_number * h * h / (2.0 * nu), 1e-3 * ts.max_growth_factor)
            solid = torch.zeros(s, s, dtype=torch.bool, device=DEV)
            for part, t in zip(parts, _step2d(u, v, solid, True, "upwind", dt, nu, 1.0, 1.0)):
                part.append(t.contiguous().flatten())
        return [torch.cat(part) for part in parts]
    cavity = kind == "cavity2d"
    solid = torch.zeros(case["ny"], case["nx"], dtype=torch.bool, device=DEV) if cavity else _solid(case)
    lx, ly = (1.0, 1.0) if cavity else (25.0, 10.0)
    return flat(_step2d(*_inputs2d(case, seed), solid, cavity, case["convection"], _dt2d(case), 0.01, lx, ly))
