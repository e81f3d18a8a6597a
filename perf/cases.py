"""Timed cases of the framework, each through an entry point that a program calls.

Four kinds of work, over the sizes that users of a focused-ultrasound solver run:

* ``request``: one whole CW solve by the Python front, host inputs and host results;
* ``cw``: a kept solver handle running one CW solve (reset, settle, record, phasors) with
  the results left in device buffers, as an embedding program does through the C ABI;
* ``heat``: a kept Pennes / CEM43 handle: temperatures in, sub-steps, temperatures and dose out;
* ``fft``: the batched 3-D real transform, forward and inverse, on device buffers.

Media, sources and fields are drawn from the seed: layered tissue with rough interfaces or
ellipsoid inclusions in water, focused bowls with steered phases, focal heating spots.
``exact`` restates each path in 64 bits with plain torch.
"""

from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

import caustica_gb300 as cg
from caustica_gb300 import _lib
from caustica_gb300.device import DeviceLabelMedium
from caustica_gb300.engine import DeviceSolver, make_plan

F0 = 1.0e6  # drive frequency [Hz] of every acoustic case
PML = 10  # sponge cells of every acoustic case
RAMP = 3.0  # drive ramp, periods
EDGE = 2.0  # sponge edge factor
WATER = (0.0253, 1000.0, 1500.0, 3.5)  # alpha [Np/m], rho, c, beta
T_REF = 37.0


def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _gen(seed):
    return np.random.default_rng([int(seed), 7919])


def _ptr(t):
    return C.c_void_p(t.data_ptr())


# ------------------------------------------------------------------ cases --
def listed():
    return [
        # a planner's quick request: the smallest grid that is served, whole call with host data
        {"name": "request_64", "kind": "request", "ndim": 3, "nx": 64, "ny": 64, "nz": 64, "medium": "inclusions",
         "storage": "labels", "nonlinear": False, "harmonics": 1, "batch": 1, "settle": 6, "record": 2, "roi": False},
        # a 2-D slice for set-up checks: little work per launch, ragged size (padded to 135 x 192)
        {"name": "slice_131x187", "kind": "cw", "ndim": 2, "nx": 1, "ny": 131, "nz": 187, "medium": "layers",
         "storage": "labels", "nonlinear": True, "harmonics": 2, "batch": 1, "settle": 8, "record": 2, "roi": False},
        # the plain linear water-tank solve of the benchmark's first configuration
        {"name": "tank_96x96x128", "kind": "cw", "ndim": 3, "nx": 96, "ny": 96, "nz": 128, "medium": "water",
         "storage": "device", "nonlinear": False, "harmonics": 1, "batch": 1, "settle": 6, "record": 2, "roi": False},
        # nonlinear propagation into layered tissue, the benchmark's headline grid, three harmonics
        {"name": "tissue_192x192x256", "kind": "cw", "ndim": 3, "nx": 192, "ny": 192, "nz": 256, "medium": "layers",
         "storage": "device", "nonlinear": True, "harmonics": 3, "batch": 1, "settle": 8, "record": 2, "roi": False},
        # a patient grid of any size (padded to 144 x 180 x 192), only the target region recorded
        {"name": "ragged_139x173x187", "kind": "cw", "ndim": 3, "nx": 139, "ny": 173, "nz": 187, "medium": "inclusions",
         "storage": "labels", "nonlinear": False, "harmonics": 1, "batch": 1, "settle": 6, "record": 1, "roi": True},
        # per-voxel maps (a CT-derived medium), odd row count and odd row length, nonlinear
        {"name": "dense_100x125x135", "kind": "cw", "ndim": 3, "nx": 100, "ny": 125, "nz": 135, "medium": "dense",
         "storage": "dense", "nonlinear": True, "harmonics": 2, "batch": 1, "settle": 6, "record": 1, "roi": False},
        # eight steering positions of one array over one medium in one batch
        {"name": "steer8_160x160x192", "kind": "cw", "ndim": 3, "nx": 160, "ny": 160, "nz": 192, "medium": "inclusions",
         "storage": "device", "nonlinear": False, "harmonics": 1, "batch": 8, "settle": 4, "record": 1, "roi": True},
        # the largest cubic grid of the common GPU comparisons that a whole head at 1 MHz needs
        {"name": "head_400", "kind": "cw", "ndim": 3, "nx": 400, "ny": 400, "nz": 400, "medium": "layers",
         "storage": "device", "nonlinear": False, "harmonics": 1, "batch": 1, "settle": 4, "record": 1, "roi": True},
        # heating with dose on the first configuration's grid: short launches, many of them
        {"name": "heat_96x96x128", "kind": "heat", "nx": 96, "ny": 96, "nz": 128, "storage": "labels", "materials": 4,
         "dose": True, "dirichlet": False, "steps": 200},
        # heating with dose on the largest served grid
        {"name": "heat_256x256x320", "kind": "heat", "nx": 256, "ny": 256, "nz": 320, "storage": "labels",
         "materials": 6, "dose": True, "dirichlet": False, "steps": 60},
        # per-voxel coefficients, held walls, odd sizes
        {"name": "heat_dense_101x117x143", "kind": "heat", "nx": 101, "ny": 117, "nz": 143, "storage": "dense",
         "materials": 0, "dose": True, "dirichlet": True, "steps": 100},
        # the stand-alone transform, forward and inverse
        {"name": "fft_160x160x192_b2", "kind": "fft", "nx": 160, "ny": 160, "nz": 192, "batch": 2},
    ]


def _smooth(n):
    while True:
        m = n
        for p in (2, 3, 5):
            while m % p == 0:
                m //= p
        if m == 1:
            return n
        n += 1


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["cw", "cw", "cw", "cw", "heat", "heat", "fft", "request"])
    if kind == "request":
        return {"kind": kind, "ndim": 3, "nx": size(40, 72), "ny": size(40, 72), "nz": size(48, 80),
                "medium": "inclusions", "storage": "labels", "nonlinear": rng.random() < 0.3, "harmonics": 1,
                "batch": 1, "settle": rng.randint(4, 7), "record": 2, "roi": False}
    if kind == "cw":
        storage = rng.choice(["device", "device", "labels", "dense"])
        nonlinear = rng.random() < 0.5
        if rng.random() < 0.2:
            n = (1, size(64, 320), size(96, 400))
        elif storage == "device":
            n = tuple(_smooth(size(64, 320)) for _ in range(3))
        else:
            n = tuple(size(56, 160) for _ in range(3))
        ndim = 2 if n[0] == 1 else 3
        if ndim == 2 and storage == "device":
            storage = "labels"
        cells = n[0] * n[1] * n[2]
        batch = rng.choice([2, 3, 5, 8]) if cells < 5_000_000 and storage != "dense" and rng.random() < 0.3 else 1
        return {"kind": kind, "ndim": ndim, "nx": n[0], "ny": n[1], "nz": n[2],
                "medium": "dense" if storage == "dense" else rng.choice(["water", "layers", "inclusions"]),
                "storage": storage, "nonlinear": nonlinear, "harmonics": rng.randint(1, 3) if nonlinear else 1,
                "batch": batch, "settle": rng.randint(4, 8) if cells * batch < 10_000_000 else 4, "record": 1,
                "roi": rng.random() < 0.5}
    if kind == "heat":
        storage = rng.choice(["labels", "labels", "dense"])
        hi = 280 if storage == "labels" else 160
        n = [size(48, hi) for _ in range(3)]
        if storage == "labels" and rng.random() < 0.7:
            n[2] += n[2] % 2
        return {"kind": kind, "nx": n[0], "ny": n[1], "nz": n[2], "storage": storage,
                "materials": rng.randint(1, 8) if storage == "labels" else 0, "dose": rng.random() < 0.8,
                "dirichlet": rng.random() < 0.3, "steps": rng.randint(20, 100)}
    return {"kind": "fft", "nx": _smooth(size(32, 320)), "ny": _smooth(size(32, 320)), "nz": _smooth(size(32, 320)),
            "batch": rng.randint(1, 3)}


# --------------------------------------------------------------- acoustics --
def _shape(case):
    return tuple(case[a] for a in ("nx", "ny", "nz"))[3 - case["ndim"]:]


def _padded(case):
    return tuple(_smooth(n) for n in _shape(case))


def _axes(shape, dev):
    out = []
    for d, n in enumerate(shape):
        v = [1] * len(shape)
        v[d] = n
        out.append(torch.arange(n, device=dev, dtype=torch.float32).reshape(v))
    return out


def _label_map(case, shape, rng, dev):
    """uint8 labels (0 = water) of a layered or an inclusion medium."""
    lab = torch.zeros(shape, dtype=torch.uint8, device=dev)
    ax = _axes(shape, dev)
    if case["medium"] == "layers":
        depth = [0.15, 0.22, 0.34]
        for i, d in enumerate(depth):
            relief = torch.zeros((1,) * len(shape), device=dev)
            for _ in range(6):
                amp, ph = rng.uniform(0.3, 1.5), rng.uniform(0, 2 * math.pi)
                arg = ph
                for a in ax[:-1]:
                    arg = arg + float(rng.uniform(-0.4, 0.4)) * a
                relief = relief + amp * torch.sin(torch.as_tensor(arg, device=dev))
            lab[(ax[-1] >= PML + 4 + d * shape[-1] + relief).expand(shape)] = i + 1
    elif case["medium"] == "inclusions":
        for i in range(5):
            r2 = torch.zeros((1,) * len(shape), device=dev)
            for a, n in zip(ax, shape):
                r2 = r2 + ((a - rng.uniform(0.3, 0.75) * n) / rng.uniform(0.06 * n + 1, 0.18 * n + 2)) ** 2
            lab[(r2 <= 1.0).expand(shape)] = i + 1
    return lab


def _table(case, rng):
    rows = {0: WATER}
    for i in range(1, 6):
        rows[i] = (float(rng.uniform(3.0, 14.0)), float(rng.uniform(920.0, 1100.0)), float(rng.uniform(1440.0, 1640.0)),
                   float(rng.uniform(4.0, 6.5)))
    if not case["nonlinear"]:
        rows = {k: v[:3] + (0.0,) for k, v in rows.items()}
    return {k: tuple(float(np.float32(x)) for x in v) for k, v in rows.items()}


def _dense_maps(case, shape, rng, dev):
    """Smoothly varying alpha, rho, c, beta of every voxel (float32)."""
    ax = _axes(shape, dev)
    f = torch.zeros(shape, device=dev)
    for _ in range(8):
        arg = float(rng.uniform(0, 2 * math.pi))
        for a in ax:
            arg = arg + float(rng.uniform(-0.25, 0.25)) * a
        f = f + torch.sin(arg)
    g = torch.Generator(device=dev).manual_seed(int(rng.integers(1 << 30)))
    f = f / 8.0 + 0.02 * torch.randn(shape, device=dev, generator=g)
    f = f.clamp(-1.0, 1.0)
    return (5.0 + 3.0 * f, 1010.0 + 60.0 * f, 1540.0 + 70.0 * f, (5.0 + 1.0 * f) if case["nonlinear"] else 0.0 * f)


def _acoustic(case, seed):
    """Everything a solve is given: plain arrays and numbers."""
    dev = _dev()
    rng = _gen(seed)
    shape = _shape(case)
    dx = 0.25e-3
    s = {"shape": shape, "dx": dx, "dev": dev}
    if case["storage"] == "dense":
        s["maps"] = _dense_maps(case, shape, rng, dev)
        c_max = float(s["maps"][2].max())
    else:
        s["labels"] = _label_map(case, shape, rng, dev)
        s["rows"] = _table(case, rng)
        present = torch.unique(s["labels"]).tolist()
        s["rows"] = {k: v for k, v in s["rows"].items() if k in present}
        c_max = max(v[2] for v in s["rows"].values())
    # a bowl shell on the z = low side, one voxel per lateral position, steered focus
    lat = shape[:-1]
    apex = [n // 2 for n in lat] + [PML + 2]
    roc = 0.55 * shape[-1]
    a = min(0.3 * (min(lat) - 2 * PML), 0.6 * roc)
    r = int(a)
    offs = np.stack(np.meshgrid(*[np.arange(-r, r + 1)] * len(lat), indexing="ij"), -1).reshape(-1, len(lat))
    rr = (offs**2).sum(1)
    offs, rr = offs[rr <= a * a], rr[rr <= a * a]
    z = np.round(roc - np.sqrt(roc * roc - rr)).astype(np.int64) + apex[-1]
    s["idx"] = np.concatenate([offs + np.array(apex[:-1]), z[:, None]], 1).astype(np.int64)
    k0 = 2 * math.pi * F0 / 1500.0
    ph = []
    for _ in range(case["batch"]):
        tgt = np.array([*(apex[:-1] + rng.uniform(-4, 4, len(lat))), apex[-1] + roc + rng.uniform(-6, 6)])
        d = np.linalg.norm((s["idx"] - tgt) * dx, axis=1)
        ph.append(((-k0 * d) % (2 * math.pi)).astype(np.float32))
    s["phases"] = np.stack(ph)
    s["amplitude"] = float(rng.uniform(0.8e5, 1.2e5) * (5.0 if case["nonlinear"] else 1.0))
    period = 1.0 / F0
    spp = max(2, int(math.floor(period / (0.48 * dx / c_max))))
    while period / spp * c_max / dx > 0.50 + 1e-12:  # the hard Courant limit
        spp += 1
    s["spp"], s["dt"] = spp, period / spp
    s["c_max"] = c_max
    s["region"] = tuple(slice(int(0.3 * n), int(0.3 * n) + max(1, int(0.4 * n))) for n in shape) if case["roi"] else None
    return s


def _objects(case, s):
    """The framework's own objects for the solve `s`."""
    grid = cg.Grid(s["shape"], s["dx"], cg.PMLSpec(PML * s["dx"], EDGE))
    if case["storage"] == "dense":
        medium = cg.Medium(*(m.cpu().numpy() for m in s["maps"]))
    elif case["storage"] == "device":
        medium = DeviceLabelMedium(s["labels"], s["rows"])
    else:
        medium = cg.Medium.from_labels(s["labels"].cpu().numpy(), s["rows"])
    source = cg.CWSource(indices=s["idx"], phases=s["phases"][0], amplitude=s["amplitude"], f0=F0, ramp_periods=RAMP)
    # settling runs a fixed number of periods: the flight time is taken to the apex, so that
    # the schedule is max(flight + minimum, ...) = the case's own count
    focus = tuple(int(v) for v in s["idx"][len(s["idx"]) // 2])
    return grid, medium, source, focus


def _prepare_request(case, seed):
    s = _acoustic(case, seed)
    grid, medium, source, focus = _objects(case, s)
    tof = _tof(s, focus)
    spec = cg.CWRunSpec(convergence_tol=0.0, min_settle_periods=1, max_settle_periods=max(1, case["settle"] - tof),
                        n_record_periods=case["record"])
    solver = cg.WesterveltKSpaceGB300() if case["nonlinear"] else cg.LinearKSpaceGB300()
    return {"kind": "request", "solver": solver, "args": (grid, medium, source, spec), "focus": focus,
            "region": s["region"], "harmonics": tuple(range(1, case["harmonics"] + 1))}


def _tof(s, focus):
    """Periods of flight from the farthest source voxel to `focus` at the slowest sound speed."""
    if "maps" in s:
        c_min = float(s["maps"][2].min())
    else:
        c_min = min(v[2] for v in s["rows"].values())
    d = np.linalg.norm((s["idx"] - np.array(focus)) * s["dx"], axis=1).max()
    return max(1, int(math.ceil(d / c_min * F0)))


def _settle_periods(s, case):
    """Settling periods that the schedule of the whole call comes to (tolerance 0: the upper bound)."""
    focus = tuple(int(v) for v in s["idx"][len(s["idx"]) // 2])
    tof = _tof(s, focus)
    lo = tof + max(1, int(math.ceil(RAMP)) + 1)
    return max(tof + max(1, case["settle"] - tof), lo)


def _prepare_cw(case, seed):
    s = _acoustic(case, seed)
    grid, medium, source, focus = _objects(case, s)
    spec = cg.CWRunSpec(convergence_tol=0.0, min_settle_periods=1, max_settle_periods=max(1, case["settle"]),
                        n_record_periods=case["record"])
    harmonics = tuple(range(1, case["harmonics"] + 1))
    plan = make_plan("perf", grid, medium, source, spec, record_region=s["region"], reference_point=focus,
                     nonlinear=case["nonlinear"], harmonics=harmonics)
    solver = DeviceSolver(plan, batch=case["batch"], phases=s["phases"])
    nrec, B, dev = solver.nrec, case["batch"], s["dev"]
    return {"kind": "cw", "solver": solver, "settle": case["settle"], "record": case["record"], "spp": plan.spp,
            "keep": medium, "phasors": torch.empty((B, len(harmonics), nrec, 2), dtype=torch.float32, device=dev),
            "p_max": torch.empty((B, nrec), dtype=torch.float32, device=dev)}


def _run_cw(st):
    solver = st["solver"]
    solver.reset()
    solver.run_periods(st["settle"])
    solver.begin_record()
    solver.run_periods(st["record"], record=True)
    _lib.call("cg_solver_finalize", solver.h, st["record"] * st["spp"], _ptr(st["phasors"]), _ptr(st["p_max"]))
    return {"phasors": st["phasors"], "p_max": st["p_max"]}


def _solve_exact(case, seed, settle):
    """The CW scheme in 64 bits: k-space pseudospectral steps, sponge, source, harmonic sums."""
    s = _acoustic(case, seed)
    dev, shape, nd, B = s["dev"], s["shape"], case["ndim"], case["batch"]
    pad = _padded(case)
    f8 = torch.float64
    if "maps" in s:
        props = [m.to(f8) for m in s["maps"]]
        c_src_map = s["maps"][2]
    else:
        lut = torch.zeros((256, 4), dtype=f8, device=dev)
        for k, v in s["rows"].items():
            lut[k] = torch.tensor(v, dtype=f8)
        props = [lut[:, i][s["labels"].long()] for i in range(4)]
        c_src_map = props[2]
    idx = [torch.as_tensor(s["idx"][:, d], device=dev) for d in range(nd)]
    c_src = c_src_map[tuple(idx)].to(f8)
    for d in range(nd):  # high-end edge replication up to the transform size
        g = torch.arange(pad[d], device=dev).clamp(max=shape[d] - 1)
        props = [p.index_select(d, g) for p in props]
    alpha, rho, c, beta = props
    dt, dx, spp = s["dt"], s["dx"], s["spp"]
    dtr, rc2, ab, b2 = dt / rho, rho * c * c * dt, torch.exp(-alpha * c * dt), 2.0 * beta * dt
    del props, alpha, rho, c, beta
    sp = torch.ones((1,) * nd, dtype=f8, device=dev)
    k2, ik = torch.zeros((1,) * nd, dtype=f8, device=dev), []
    for d, n in enumerate(pad):
        r = torch.arange(n, device=dev)
        e = torch.minimum(r, n - 1 - r)
        w = torch.where(e < PML, torch.exp(-EDGE * ((PML - e).to(f8) / PML) ** 2), torch.ones((), dtype=f8, device=dev))
        v = [1] * nd
        v[d] = n
        sp = sp * w.reshape(v)
        k = 2 * math.pi * (torch.fft.rfftfreq(n, dx, dtype=f8, device=dev) if d == nd - 1
                           else torch.fft.fftfreq(n, dx, dtype=f8, device=dev))
        v[d] = k.numel()
        k2 = k2 + (k * k).reshape(v)
        kd = k.clone()
        if n % 2 == 0:
            kd[n // 2] = 0.0
        ik.append(1j * kd.reshape(v))
    a = 0.5 * s["c_max"] * dt * torch.sqrt(k2)
    kappa = torch.where(a > 0, torch.sin(a) / torch.where(a > 0, a, torch.ones_like(a)), torch.ones_like(a))
    damp = ab * sp
    del a, k2, ab
    dims = tuple(range(1, nd + 1))
    p = torch.zeros((B, *pad), dtype=f8, device=dev)
    u = [torch.zeros_like(p) for _ in range(nd)]
    scale = 2.0 * c_src * dt / dx
    ph = torch.as_tensor(s["phases"], device=dev).to(f8)
    reg = s["region"] or tuple(slice(0, n) for n in shape)
    H = case["harmonics"]
    rshape = tuple(r.stop - r.start for r in reg)
    acc = torch.zeros((B, H, *rshape), dtype=torch.complex128, device=dev)
    pm = torch.zeros((B, *rshape), dtype=f8, device=dev)
    rec_steps = case["record"] * spp
    where = (slice(None), *idx)
    for n in range(settle * spp + rec_steps):
        P = torch.fft.rfftn(p, dim=dims) * kappa
        D = None
        for i in range(nd):
            g = torch.fft.irfftn(P * ik[i], s=pad, dim=dims)
            u[i] = (u[i] - dtr * g) * damp
            del g
            t = torch.fft.rfftn(u[i], dim=dims) * ik[i]
            D = t if D is None else D + t
        div = torch.fft.irfftn(D * kappa, s=pad, dim=dims)
        del P, D, t
        p = (p - ((rc2 + b2 * p) if case["nonlinear"] else rc2) * div) * damp
        tt = n * dt
        env = 0.5 * (1.0 - math.cos(math.pi * min(tt * F0 / RAMP, 1.0)))
        p[where] += s["amplitude"] * env * scale * torch.sin(2 * math.pi * F0 * tt - ph)
        if n >= settle * spp:
            q = p[(slice(None), *reg)]
            pm = torch.maximum(pm, q.abs())
            for h in range(H):
                w = 2 * math.pi * (h + 1) * (n % spp) / spp
                acc[:, h] += q * complex(math.cos(w), math.sin(w))
    acc *= 2.0 / rec_steps
    return acc, pm


# -------------------------------------------------------------------- heat --
def _thermal(case, seed):
    """Plain inputs of a Pennes solve: label table or per-cell maps, Q, T0."""
    dev = _dev()
    rng = _gen(seed)
    shape = _heat_shape(case)
    ax = _axes(shape, dev)
    dx = 0.5e-3
    s = {"shape": shape, "dx": dx, "dev": dev, "dt": 0.05}
    g = torch.Generator(device=dev).manual_seed(int(rng.integers(1 << 30)))
    q = torch.zeros(shape, device=dev)
    for _ in range(3):
        r2 = torch.zeros((1, 1, 1), device=dev)
        for a, n in zip(ax, shape):
            r2 = r2 + ((a - rng.uniform(0.3, 0.7) * n) / rng.uniform(3.0, 0.15 * n + 4.0)) ** 2
        q = q + float(rng.uniform(1e6, 8e6)) * torch.exp(-r2)
    s["q"] = q.contiguous()
    s["T0"] = (T_REF + 0.5 * torch.rand(shape, device=dev, generator=g)).contiguous()
    if case["storage"] == "labels":
        lab = torch.zeros(shape, dtype=torch.uint8, device=dev)
        for i in range(1, case["materials"]):
            r2 = torch.zeros((1, 1, 1), device=dev)
            for a, n in zip(ax, shape):
                r2 = r2 + ((a - rng.uniform(0.2, 0.8) * n) / rng.uniform(0.08 * n + 1, 0.25 * n + 2)) ** 2
            lab[(r2 <= 1.0).expand(shape)] = i
        s["labels"] = lab.contiguous()
        n = case["materials"]
        k = rng.uniform(0.25, 0.6, n)
        rho_c = rng.uniform(2.2e6, 4.0e6, n)
        perf = rng.uniform(0.0, 4.0e3, n)
        s["table"] = np.stack([k, s["dt"] / rho_c, perf, np.zeros(n)], 1).astype(np.float32)
    else:
        f = torch.zeros(shape, device=dev)
        for _ in range(6):
            arg = float(rng.uniform(0, 2 * math.pi))
            for a in ax:
                arg = arg + float(rng.uniform(-0.3, 0.3)) * a
            f = f + torch.sin(arg) / 6.0
        k = 0.45 + 0.15 * f
        inv = 1.0 / (dx * dx)
        s["k"] = k
        s["faces"] = []
        s["walls"] = []
        for d in range(3):
            lo, hi = k.narrow(d, 0, shape[d] - 1), k.narrow(d, 1, shape[d] - 1)
            s["faces"].append((2.0 * lo * hi / (lo + hi) * inv).contiguous())
            s["walls"] += [(2.0 * k.select(d, 0) * inv).reshape(-1), (2.0 * k.select(d, shape[d] - 1) * inv).reshape(-1)]
        s["walls"] = torch.cat(s["walls"]).contiguous()
        s["coeff"] = (s["dt"] / (3.2e6 + 0.6e6 * f)).contiguous()
        s["perf"] = (1.8e3 + 1.5e3 * f).contiguous()
    return s


def _heat_shape(case):
    return tuple(case[a] for a in ("nx", "ny", "nz"))


def _prepare_heat(case, seed):
    s = _thermal(case, seed)
    cfg = _lib.PennesConfig()
    cfg.nx, cfg.ny, cfg.nz = s["shape"]
    cfg.dirichlet, cfg.dose = int(case["dirichlet"]), int(case["dose"])
    cfg.theta_wall, cfg.t_ref = 0.0, T_REF
    cfg.half_dt_min = 0.5 * s["dt"] / 60.0
    handle = _Handle("cg_pennes_create", "cg_pennes_destroy", C.byref(cfg))
    torch.cuda.synchronize()
    if case["storage"] == "labels":
        _lib.call("cg_pennes_set_labels", handle.h, _ptr(s["labels"]), len(s["table"]), _lib.ptr(s["table"]),
                  1.0 / (s["dx"] * s["dx"]), 0, 7, _ptr(s["q"]))
    else:
        _lib.call("cg_pennes_set_coefficients", handle.h, *(_ptr(f) for f in s["faces"]), _ptr(s["walls"]),
                  _ptr(s["perf"]), _ptr(s["coeff"]), _ptr(s["q"]), None)
    out = {k: torch.empty(s["shape"], dtype=torch.float32, device=s["dev"]) for k in ("T", "T_max", "dose")}
    return {"kind": "heat", "handle": handle, "T0": s["T0"], "out": out, "steps": case["steps"], "dose": case["dose"]}


def _run_heat(st):
    h, out = st["handle"].h, st["out"]
    ok = C.c_int(0)
    _lib.call("cg_pennes_set_temperature", h, _ptr(st["T0"]), None, C.byref(ok))
    _lib.call("cg_pennes_run", h, st["steps"])
    _lib.call("cg_pennes_check_finite", h, C.byref(ok))
    _lib.call("cg_pennes_get_temperature", h, _ptr(out["T"]), _ptr(out["T_max"]),
              _ptr(out["dose"]) if st["dose"] else None)
    return {k: v for k, v in out.items() if k != "dose" or st["dose"]}


def _heat_exact(case, seed):
    s = _thermal(case, seed)
    f8, dev, shape = torch.float64, s["dev"], s["shape"]
    inv = 1.0 / (s["dx"] * s["dx"])
    if case["storage"] == "labels":
        tab = torch.as_tensor(s["table"], device=dev).to(f8)
        lab = s["labels"].long()
        k, coeff, perf = (tab[:, i][lab] for i in range(3))
        faces, wall = [], []
        for d in range(3):
            lo, hi = k.narrow(d, 0, shape[d] - 1), k.narrow(d, 1, shape[d] - 1)
            faces.append(2.0 * lo * hi / (lo + hi) * inv)
            wall.append((2.0 * k.select(d, 0) * inv, 2.0 * k.select(d, shape[d] - 1) * inv))
    else:
        coeff, perf = s["coeff"].to(f8), s["perf"].to(f8)
        faces = [f.to(f8) for f in s["faces"]]
        wall, at = [], 0
        for d in range(3):
            pl = tuple(n for i, n in enumerate(shape) if i != d)
            m = pl[0] * pl[1]
            w = s["walls"][at:at + 2 * m].to(f8)
            wall.append((w[:m].reshape(pl), w[m:].reshape(pl)))
            at += 2 * m
    q = s["q"].to(f8)
    th = s["T0"].to(f8) - T_REF
    tm, dose = th.clone(), torch.zeros_like(th)

    def rate(t):
        e = 43.0 - (t + T_REF)
        return torch.where(e < 0, torch.exp2(-e), torch.exp2(-2.0 * e))

    for _ in range(case["steps"]):
        w = q - perf * th
        for d in range(3):
            n = shape[d]
            flux = (th.narrow(d, 1, n - 1) - th.narrow(d, 0, n - 1)) * faces[d]
            w.narrow(d, 0, n - 1).add_(flux)
            w.narrow(d, 1, n - 1).sub_(flux)
            if case["dirichlet"]:
                w.select(d, 0).sub_(wall[d][0] * th.select(d, 0))
                w.select(d, n - 1).sub_(wall[d][1] * th.select(d, n - 1))
        new = th + coeff * w
        if case["dose"]:
            dose += (rate(new) + rate(th)) * (0.5 * s["dt"] / 60.0)
        th = new
        tm = torch.maximum(tm, th)
    out = {"T": th + T_REF, "T_max": tm + T_REF}
    if case["dose"]:
        out["dose"] = dose
    return out


# --------------------------------------------------------------------- fft --
class _Handle:
    """A handle of the C ABI that is destroyed with its owner."""

    def __init__(self, create, destroy, *args):
        self.h, self._destroy = C.c_void_p(), destroy
        _lib.call(create, *args, C.byref(self.h))

    def __del__(self):
        if self.h:
            getattr(_lib.load(), self._destroy)(self.h)
            self.h = None


def _fft_input(case, seed):
    g = torch.Generator(device=_dev()).manual_seed(int(seed) + 11)
    return torch.randn((case["batch"], case["nx"], case["ny"], case["nz"]), device=_dev(), generator=g)


def _prepare_fft(case, seed):
    n, b = (case["nx"], case["ny"], case["nz"]), case["batch"]
    x = _fft_input(case, seed)
    handle = _Handle("cg_fft3d_create", "cg_fft3d_destroy", *n, b)
    torch.cuda.synchronize()
    return {"kind": "fft", "handle": handle, "x": x, "back": torch.empty_like(x),
            "spec": torch.empty((b, n[0], n[2] // 2 + 1, n[1], 2), dtype=torch.float32, device=x.device)}


def _run_fft(st):
    h = st["handle"].h
    _lib.call("cg_fft3d_forward", h, _ptr(st["x"]), _ptr(st["spec"]))
    _lib.call("cg_fft3d_inverse", h, _ptr(st["spec"]), _ptr(st["back"]))
    return {"spectrum": st["spec"], "back": st["back"]}


# --------------------------------------------------------------- interface --
def prepare(case, seed):
    return {"request": _prepare_request, "cw": _prepare_cw, "heat": _prepare_heat,
            "fft": _prepare_fft}[case["kind"]](case, seed)


def run(state):
    if state["kind"] == "cw":
        return _run_cw(state)
    if state["kind"] == "heat":
        return _run_heat(state)
    if state["kind"] == "fft":
        return _run_fft(state)
    grid, medium, source, spec = state["args"]
    res = state["solver"].run(grid, medium, source, spec, record_region=state["region"],
                              reference_point=state["focus"], harmonics=state["harmonics"])
    return {"phasor": res.phasor, "p_max": res.p_max}


def exact(case, seed):
    if case["kind"] == "cw":
        acc, pm = _solve_exact(case, seed, case["settle"])
        B, H = case["batch"], case["harmonics"]
        return {"phasors": torch.view_as_real(acc.reshape(B, H, -1)).contiguous(), "p_max": pm.reshape(B, -1)}
    if case["kind"] == "request":
        acc, pm = _solve_exact(case, seed, _settle_periods(_acoustic(case, seed), case))
        return {"phasor": acc[0, 0].cpu().numpy(), "p_max": pm[0].cpu().numpy()}
    if case["kind"] == "heat":
        return _heat_exact(case, seed)
    x = _fft_input(case, seed).double()
    X = torch.fft.rfftn(x, dim=(1, 2, 3))
    n = case["nx"] * case["ny"] * case["nz"]
    return {"spectrum": torch.view_as_real(X.transpose(2, 3).contiguous()), "back": x * n}


def work(case):
    if case["kind"] in ("cw", "request"):
        nd, B, pad = case["ndim"], case["batch"], _padded(case)
        cells = float(np.prod(pad)) * B
        settle = case["settle"] if case["kind"] == "cw" else max(case["settle"], 5)
        spp = 13  # steps a period at the water-to-tissue sound speeds of these media
        steps = spp * (settle + case["record"])
        rec = float(np.prod([int(0.4 * n) if case["roi"] else n for n in _shape(case)])) * B
        # a step: p and the velocities read and written, the medium read, each transform's half
        # spectrum across memory once each way (one global transpose)
        per = 8.0 * (1 + nd) + (16.0 if case["storage"] == "dense" else 1.0) + 33.0
        rec_bytes = rec * (spp * case["record"] * 16.0 + 8.0 * case["harmonics"] + 4.0)
        n = float(np.prod(pad))
        flops = steps * B * (2 * (nd + 1) * 2.5 * n * math.log2(n) + (12 + 12 * nd) * n)
        return {"bytes": steps * cells * per + rec_bytes, "flops": flops}
    if case["kind"] == "heat":
        n = float(np.prod(_heat_shape(case)))
        per = 4 * 5 + (16 if case["dose"] else 0) + (1 if case["storage"] == "labels" else 20)
        return {"bytes": case["steps"] * n * per + n * (4 + 4 + 4 + (4 if case["dose"] else 0)),
                "flops": case["steps"] * n * (30 + (12 if case["dose"] else 0))}
    n = float(case["nx"] * case["ny"] * case["nz"]) * case["batch"]
    spec = float(case["nx"] * (case["nz"] // 2 + 1) * case["ny"]) * case["batch"] * 8
    return {"bytes": 2 * (4 * n + spec), "flops": 2 * 2.5 * n * math.log2(n / case["batch"])}
