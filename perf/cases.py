"""The work a user of this framework has it do, as measurable cases.

Every case goes through the public Python entry points (Simulation, Batch, MLP).  Four kinds:

* ``grid``:    one grid advanced by ``Simulation.step`` and its fields and DFT sums read back;
* ``batch``:   uneven grids, or grids with CPML layers, advanced by ``Batch.step``;
* ``design``:  one design of a parameter study, host permittivity in, flux spectrum out;
* ``predict`` / ``train``: the surrogate network's inference and one training epoch.

Grids start from random fields, as a run that is resumed in the middle does, so the whole grid
carries signal from the first step.  ``exact`` evaluates the same update in float64 with plain
torch.
"""
import math

import numpy as np
import torch

import gdiamond_b200 as gd

DX, DT = float(np.float32(0.1)), float(np.float32(0.05))
OMEGA0 = float(np.float32(2) * np.float32(3.14159265359))
FIELDS = ("Ex", "Ey", "Ez", "Hx", "Hy", "Hz")


def listed():
    return [
        # A few steps of a small odd grid at a time: interactive stepping and unit tests, where
        # latency and launches count.
        dict(name="quick_51x37x45", kind="grid", nx=51, ny=37, nz=45, steps=16, storage="f32",
             blt=0, medium="vacuum", boundary="pml", monitors=0, nf=0),
        # The unit-test workload: 100^3 cells with the graded absorbing layer, 100 steps.
        dict(name="unit_100_pml", kind="grid", nx=100, ny=100, nz=100, steps=100, storage="f32",
             blt=0, medium="vacuum", boundary="pml", monitors=0, nf=0),
        # The benchmark grid: 256^3 vacuum with an 8-frequency DFT plane (a tenth of its steps).
        dict(name="vacuum_256", kind="grid", nx=256, ny=256, nz=256, steps=100, storage="f32",
             blt=0, medium="vacuum", boundary="none", monitors=1, nf=8),
        # The largest grid: 200 dielectric spheres, two 16-frequency DFT planes.
        dict(name="spheres_512x512x384", kind="grid", nx=512, ny=512, nz=384, steps=20,
             storage="f32", blt=0, medium="spheres", boundary="none", monitors=2, nf=16),
        # Reduced-precision storage (FP16 E, FP32 H) on an odd grid; the steps per pass are
        # fixed, as a user does who wants the same rounding in every run.
        dict(name="spheres_f16e_251x243x190", kind="grid", nx=251, ny=243, nz=190, steps=40,
             storage="f16e", blt=2, medium="spheres", boundary="none", monitors=2, nf=16),
        # FP64 storage: the error reference of reduced-precision runs.
        dict(name="f64_160", kind="grid", nx=160, ny=160, nz=160, steps=40, storage="f64",
             blt=0, medium="spheres", boundary="none", monitors=1, nf=16),
        # The benchmark grid behind 10-cell CPML layers.
        dict(name="cpml_256", kind="grid", nx=256, ny=256, nz=256, steps=40, storage="f32",
             blt=0, medium="vacuum", boundary="cpml", layer=10, monitors=1, nf=8),
        # Many uneven simulations together: sides from 64 to 192, a slab in each, 32
        # frequencies.
        dict(name="batch_16_uneven", kind="batch", sims=16, lo=64, hi=192, steps=32,
             boundary="pml", layer=10, nf=32),
        # The surrogate's data generation: equal grids behind 8-cell CPML layers, a box in
        # each, a 64-frequency flux monitor.
        dict(name="batch_32_cpml_96", kind="batch", sims=32, lo=96, hi=96, steps=32,
             boundary="cpml", layer=8, nf=64),
        # One design on its own: new permittivity from the host, reset, a run, its spectrum.
        dict(name="design_96", kind="design", n=96, steps=200, nf=64),
        # The surrogate's inference over a large set of designs.
        dict(name="predict_262144", kind="predict", rows=262144, width=256, hidden=3, out=64,
             members=4),
        # One training epoch of the ensemble.
        dict(name="train_epoch_4096", kind="train", rows=4096, batch=64, width=256, hidden=3,
             out=64, members=4),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["grid"] * 6 + ["batch"] * 3 + ["design", "predict", "train"])
    if kind == "grid":
        while True:
            nx, ny, nz = (_log_int(rng, 32, 420) for _ in range(3))
            if nx * ny * nz <= 4e7:
                break
        boundary = rng.choice(["none", "pml", "cpml"])
        storage = "f32" if boundary == "cpml" else \
            rng.choice(["f32"] * 4 + ["f16", "bf16", "f16e", "f64"])
        steps = min(_log_int(rng, 8, 200), max(8, int(6e8 / (nx * ny * nz))))
        if storage in ("f16", "bf16", "f16e"):  # needs a material map: few enough materials
            boundary = "none"
        monitors = rng.choice([0, 1, 2])
        return dict(kind="grid", nx=nx, ny=ny, nz=nz, steps=steps, storage=storage,
                    blt=rng.choice([1, 2, 3]) if storage in ("f16", "bf16", "f16e") else 0,
                    medium=rng.choice(["vacuum", "spheres"]), boundary=boundary,
                    layer=rng.choice([6, 8, 10]), monitors=monitors,
                    nf=rng.choice([1, 8, 16, 33]) if monitors else 0)
    if kind == "batch":
        boundary = rng.choice(["pml", "cpml"])
        lo = _log_int(rng, 48, 110)
        hi = _log_int(rng, lo, 150)
        sims = rng.randint(2, 24)
        return dict(kind="batch", sims=sims, lo=lo, hi=hi, steps=rng.randint(8, 24),
                    boundary=boundary, layer=rng.choice([6, 8, 10]), nf=rng.choice([5, 32, 64]))
    if kind == "design":
        return dict(kind="design", n=rng.randint(48, 128), steps=rng.randint(60, 200),
                    nf=rng.choice([16, 33, 64]))
    net = dict(width=rng.choice([64, 96, 128, 256]), hidden=rng.choice([1, 2, 3]),
               out=rng.choice([32, 64]), members=rng.choice([1, 2, 4]))
    if kind == "predict":
        return dict(kind="predict", rows=_log_int(rng, 500, 250000), **net)
    return dict(kind="train", rows=rng.randint(300, 4000), batch=rng.choice([32, 64, 100]), **net)


# ------------------------------------------------------------------------------- inputs


def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _spheres(shape, count, seed):
    """[z][y][x] float32 permittivity: spheres of radius 4 to 24 cells, eps in 1..12."""
    nx, ny, nz = shape
    rng = np.random.default_rng(seed)
    eps = torch.ones((nz, ny, nx), dtype=torch.float32, device="cuda")
    ax = [torch.arange(n, device="cuda", dtype=torch.float32) for n in (nx, ny, nz)]
    for _ in range(count):
        c = rng.uniform([0, 0, 0], [nx, ny, nz])
        r = rng.uniform(4, 24)
        e = float(rng.uniform(1.0, 12.0))
        lo = [max(int(c[a] - r), 0) for a in range(3)]
        hi = [min(int(c[a] + r) + 1, (nx, ny, nz)[a]) for a in range(3)]
        d = [(ax[a][lo[a]:hi[a]] - float(c[a])) ** 2 for a in range(3)]
        inside = d[2][:, None, None] + d[1][None, :, None] + d[0][None, None, :] <= r * r
        eps[lo[2]:hi[2], lo[1]:hi[1], lo[0]:hi[0]][inside] = e
    return eps


def _slab(shape, rng):
    """One slab: thickness 8..32 cells, eps 2..12, random axis."""
    nx, ny, nz = shape
    eps = torch.ones((nz, ny, nx), dtype=torch.float32, device="cuda")
    axis = int(rng.integers(0, 3))
    n = (nx, ny, nz)[axis]
    th = min(int(rng.integers(8, 33)), n - 2)
    lo = int(rng.integers(1, n - th))
    sl = [slice(None)] * 3
    sl[2 - axis] = slice(lo, lo + th)
    eps[tuple(sl)] = float(rng.uniform(2.0, 12.0))
    return eps


def _box(shape, rng):
    """One box with covered-volume edges, as the designs of a parameter study have."""
    nx, ny, nz = shape
    side, height = rng.uniform(8, max(9, 0.4 * nx)), rng.uniform(8, max(9, 0.4 * nz))
    cov = []
    for n, w in ((nx, side), (ny, side), (nz, height)):
        c = rng.uniform(0.3 * n, 0.7 * n)
        i = np.arange(n, dtype=np.float64)
        cov.append(np.clip(np.minimum(i + 0.5, c + w / 2) - np.maximum(i - 0.5, c - w / 2), 0, 1))
    frac = cov[2][:, None, None] * cov[1][None, :, None] * cov[0][None, None, :]
    return (1.0 + (rng.uniform(2.0, 12.0) - 1.0) * frac).astype(np.float32)


def _stretch(n, layer):
    """Complex per-index stretch of the graded absorbing layer along one axis."""
    i = torch.arange(n, dtype=torch.float64, device="cuda")
    dist = torch.zeros_like(i)
    if layer:
        dist = torch.where(i < layer, 1.0 - i / layer, dist)
        dist = torch.where(i + layer >= n, 1.0 - (n - i - 1) / layer, dist)
        smax = -4.0 * math.log(1e-5) / (2.0 * layer * DX)
    else:
        smax = 0.0
    d3 = dist ** 3
    return torch.complex(1.0 + 2.0 * d3, smax * d3 / OMEGA0)


def _coefficients(shape, eps, layer):
    """The 12 float64 arrays Cax..Dbz ([z][y][x], possibly broadcast) for a permittivity."""
    nx, ny, nz = shape
    s = [_stretch(nx, layer)[None, None, :], _stretch(ny, layer)[None, :, None],
         _stretch(nz, layer)[:, None, None]]
    one = torch.ones((1, 1, 1), dtype=torch.float64, device="cuda")
    e = one if eps is None else eps.to(torch.float64)
    out = [None] * 12
    for c in range(3):
        a, b = [q for q in range(3) if q != c]
        for base, m in ((0, e), (6, one)):
            if layer:
                f = m * (s[a] * s[b] / s[c])
                re, sig = f.real.clamp(min=1.0), (OMEGA0 * f.imag).abs()
            else:
                re, sig = m.clamp(min=1.0), torch.zeros_like(one)
            t = sig * DT / (2.0 * re)
            out[base + c], out[base + 3 + c] = (1.0 - t) / (1.0 + t), DT / re / (1.0 + t) / DX
    return out


def _wave(steps, seed):
    rng = np.random.default_rng(seed)
    n = np.arange(max(steps, 1), dtype=np.float64)
    amp, delay = rng.uniform(20, 60), rng.uniform(5, 40)
    return (amp * np.exp(-((n - delay) ** 2) / 200.0) * np.sin(2 * np.pi * n / 20.0)).astype(np.float32)


def _band(nf):
    f0, sig = 1.0 / (20.0 * DT), 1.0 / (2.0 * math.pi * 10.0 * DT)
    return np.linspace(f0 - 2 * sig, f0 + 2 * sig, nf)


def _types(storage):
    e, h = {"f32": ("float32",) * 2, "f16": ("float16",) * 2, "bf16": ("bfloat16",) * 2,
            "f16e": ("float16", "float32"), "f64": ("float64",) * 2}[storage]
    return [getattr(torch, e)] * 3 + [getattr(torch, h)] * 3


def _grid_inputs(c, seed):
    shape = (c["nx"], c["ny"], c["nz"])
    cells = shape[0] * shape[1] * shape[2]
    count = max(4, min(200, int(round(cells / 500000))))
    eps = _spheres(shape, count, seed) if c["medium"] == "spheres" else None
    g = _gen(seed)
    fields = [torch.randn(shape[::-1], device="cuda", generator=g, dtype=torch.float32).to(t)
              for t in _types(c["storage"])]
    wave = _wave(c["steps"], seed)
    src = dict(component="Jz", wave=wave, i=shape[0] // 2, j=shape[1] // 2, k=shape[2] // 2)
    layer = min(10, min(shape) // 3) if c["boundary"] == "pml" else 0
    planes = [("Ez", shape[2] // 2), ("Hy", shape[2] // 3)][:c["monitors"]]
    return shape, eps, layer, fields, src, planes


def _cpml_layer(c, shape):
    return min(c["layer"], (min(shape) - 2) // 2)


def _set_coefficients(sim, shape, eps, layer):
    full = [a.to(torch.float32).expand(shape[::-1]).contiguous()
            for a in _coefficients(shape, eps, layer)]
    torch.cuda.synchronize()
    sim.set_coefficients(full)
    sim.sync()


def _prepare_grid(c, seed):
    shape, eps, layer, fields, src, planes = _grid_inputs(c, seed)
    sim = gd.Simulation(*shape, storage=c["storage"], blt=c["blt"])
    _set_coefficients(sim, shape, eps, layer)
    if c["boundary"] == "cpml":
        sim.set_cpml(thickness=_cpml_layer(c, shape))
    sim.set_sources([src])
    mons = [sim.add_dft_monitor(name, k, _band(c["nf"])) for name, k in planes]
    torch.cuda.synchronize()
    for q in range(6):
        sim.set_planes_device(q, 0, shape[2], fields[q].data_ptr())
    sim.sync()
    wide = torch.float64 if c["storage"] == "f64" else torch.float32
    out = [torch.empty(shape[::-1], dtype=wide, device="cuda") for _ in range(6)]
    dft = [torch.empty((2, c["nf"], shape[1], shape[0]), dtype=torch.float64, device="cuda")
           for _ in mons]
    torch.cuda.synchronize()
    return dict(case=c, sim=sim, fields=fields if mons or c["boundary"] == "cpml" else None,
                mons=mons, out=out, dft=dft)


def _batch_shapes(c, seed):
    rng = np.random.default_rng(1000 + c["sims"])  # the sizes are the case's, not the seed's
    return [tuple(int(v) for v in rng.integers(c["lo"], c["hi"] + 1, 3)) for _ in range(c["sims"])]


def _batch_inputs(c, seed, n, shape):
    rng = np.random.default_rng([seed, n])
    cpml = c["boundary"] == "cpml"
    eps = torch.from_numpy(_box(shape, rng)).cuda() if cpml else _slab(shape, rng)
    wave = _wave(c["steps"], [seed, n, 1])
    if cpml:
        src = dict(component="Jx", kind=gd.SRC_PLANE_Z, k=10, wave=wave)
    else:
        src = dict(component="Jz", wave=wave, i=shape[0] // 2, j=shape[1] // 2, k=shape[2] // 2)
    return eps, src


def _prepare_batch(c, seed):
    shapes = _batch_shapes(c, seed)
    cpml = c["boundary"] == "cpml"
    sims, mons, init, out, res = [], [], [], [], []
    for n, shape in enumerate(shapes):
        eps, src = _batch_inputs(c, seed, n, shape)
        sim = gd.Simulation(*shape)
        _set_coefficients(sim, shape, eps, 0 if cpml else c["layer"])
        if cpml:
            sim.set_cpml(thickness=_cpml_layer(c, shape))
        sim.set_sources([src])
        if cpml:
            mons.append(sim.add_flux_monitor(shape[2] - c["layer"] - 2, _band(c["nf"])))
        else:
            mons.append(sim.add_dft_monitor("Ez", shape[2] // 2, _band(c["nf"])))
        g = _gen(seed * 1000 + n)
        init.append(torch.randn((6,) + shape[::-1], device="cuda", generator=g))
        out.append(torch.empty((6,) + shape[::-1], device="cuda"))
        res.append(torch.empty(c["nf"] if cpml else (2, c["nf"], shape[1], shape[0]),
                               dtype=torch.float64, device="cuda"))
        sims.append(sim)
    torch.cuda.synchronize()
    return dict(case=c, sims=sims, batch=gd.Batch(sims), mons=mons, init=init, out=out, res=res)


def _prepare_design(c, seed):
    n = c["n"]
    rng = np.random.default_rng(seed)
    sim = gd.Simulation(n, n, n)
    sim.set_sources([dict(component="Jx", kind=gd.SRC_PLANE_Z, k=10, wave=_wave(c["steps"], seed))])
    fid = sim.add_flux_monitor(n - 10, _band(c["nf"]))
    return dict(case=c, sim=sim, fid=fid, eps=_box((n, n, n), rng).reshape(-1))


def _net_inputs(c, seed):
    """He-initialised weights of every member and the designs (and targets) of a data set."""
    dims = (6,) + (c["width"],) * c["hidden"] + (c["out"],)
    g = _gen(seed)
    ws = [[(torch.randn((o, i), device="cuda", generator=g) * math.sqrt(2.0 / i),
            torch.randn(o, device="cuda", generator=g) * 0.1)
           for i, o in zip(dims[:-1], dims[1:])] for _ in range(c["members"])]
    x = torch.rand((c["rows"], 6), device="cuda", generator=g) * 2 - 1
    y = torch.sin(3.0 * x @ torch.randn((6, c["out"]), device="cuda", generator=g))
    return dims, ws, x, y


def _prepare_net(c, seed):
    dims, ws, x, y = _net_inputs(c, seed)
    net = gd.MLP(dims, members=c["members"], seed=int(seed) & 0xFFFF)
    flat = np.zeros((c["members"], net.n_params), np.float32)
    for e in range(c["members"]):
        for (w_off, (o, i), b_off), (w, b) in zip(net.layout(), ws[e]):
            flat[e, w_off:w_off + o * i] = w.reshape(-1).cpu().numpy()
            flat[e, b_off:b_off + o] = b.cpu().numpy()
    net.set_params(flat)
    state = dict(case=c, net=net, x=x)
    if c["kind"] == "train":
        net.set_data(x.cpu().numpy(), y.cpu().numpy())
    else:
        state["mean"] = torch.empty((c["rows"], c["out"]), device="cuda")
        state["sd"] = torch.empty_like(state["mean"])
    torch.cuda.synchronize()
    return state


def prepare(case, seed):
    return {"grid": _prepare_grid, "batch": _prepare_batch, "design": _prepare_design,
            "predict": _prepare_net, "train": _prepare_net}[case["kind"]](case, seed)


# ------------------------------------------------------------------------------- one pass


def run(state):
    c = state["case"]
    if c["kind"] == "grid":
        sim, nz = state["sim"], c["nz"]
        if state["fields"] is not None:  # a run of its own: fresh sums, resumed fields
            sim.reset()
            for q in range(6):
                sim.set_planes_device(q, 0, nz, state["fields"][q].data_ptr())
        sim.step(c["steps"])
        for q, o in enumerate(state["out"]):
            if c["storage"] == "f64":  # the raw planes keep the 64 bits
                sim.get_planes_device(q, 0, nz, o.data_ptr())
            else:
                sim.get_field_device(q, o.data_ptr())
        for m, d in zip(state["mons"], state["dft"]):
            sim.get_dft_device(m, d[0].data_ptr(), d[1].data_ptr())
        return {"fields": state["out"], "dft": state["dft"]}
    if c["kind"] == "batch":
        for sim, f in zip(state["sims"], state["init"]):
            sim.reset()
            for q in range(6):
                sim.set_planes_device(q, 0, sim.shape[2], f[q].data_ptr())
        state["batch"].step(c["steps"])
        for sim, m, o, r in zip(state["sims"], state["mons"], state["out"], state["res"]):
            for q in range(6):
                sim.get_field_device(q, o[q].data_ptr())
            if c["boundary"] == "cpml":
                sim.get_flux_device(m, r.data_ptr())
            else:
                sim.get_dft_device(m, r[0].data_ptr(), r[1].data_ptr())
        return {"fields": state["out"], "result": state["res"]}
    if c["kind"] == "design":
        sim = state["sim"]
        sim.set_permittivity(state["eps"])
        sim.reset()
        sim.step(c["steps"])
        return {"flux": sim.get_flux(state["fid"]), "ex": sim.get_field("Ex")}
    if c["kind"] == "predict":
        state["net"].predict_device(state["x"].data_ptr(), c["rows"], state["mean"].data_ptr(),
                                    state["sd"].data_ptr())
        return {"mean": state["mean"], "sd": state["sd"]}
    loss = state["net"].train(1, batch=c["batch"], lr=1e-3, seed=7)
    return {"loss": loss, "params": state["net"].get_params()}


def _update_flops(cells, steps):
    return 36.0 * cells * steps  # six components, three differences, two products, one sum


def work(case):
    """Fields in and out once (and their read-out), ids, DFT sums; 36 operations a cell-update,
    6 a frequency of a monitored cell."""
    c = case
    if c["kind"] in ("predict", "train"):
        dims = (6,) + (c["width"],) * c["hidden"] + (c["out"],)
        macs = sum(i * o for i, o in zip(dims[:-1], dims[1:]))
        par = c["members"] * (macs + sum(dims[1:]))
        rows = c["rows"]
        if c["kind"] == "predict":
            return {"bytes": 4.0 * (rows * (6 + 2 * c["out"]) + par),
                    "flops": 2.0 * macs * c["members"] * rows}
        return {"bytes": 4.0 * (rows * (6 + c["out"]) + 2 * 3 * par),
                "flops": 6.0 * macs * c["members"] * rows}
    if c["kind"] == "grid":
        shapes, esz = [(c["nx"], c["ny"], c["nz"])], sum(t.itemsize for t in _types(c["storage"]))
        mons, read = c["monitors"], 48 if c["storage"] == "f64" else 24
    elif c["kind"] == "batch":
        shapes, esz, read = _batch_shapes(c, 0), 24, 24
        mons = 6 if c["boundary"] == "cpml" else 1
    else:
        shapes, esz, mons, read = [(c["n"],) * 3], 24, 6, 4 + 4  # Ex out, permittivity in
    cells = sum(x * y * z for x, y, z in shapes)
    mon_cells = sum(x * y for x, y, _ in shapes) * mons
    return {"bytes": float(cells * (2 * esz + 2 + read) + mon_cells * c["nf"] * 32),
            "flops": _update_flops(cells, c["steps"]) + 6.0 * mon_cells * c["nf"] * c["steps"]}


# ------------------------------------------------------------------------------- float64


def _cpml_axis(n, layer, half, axis):
    """(b, a, 1/kappa) along an axis of the CPML layers on both its faces."""
    p = torch.arange(n, dtype=torch.float64, device="cuda") + (0.5 if half else 0.0)
    rho = torch.zeros_like(p)
    rho = torch.where(p < layer, (layer - p) / layer, rho)
    rho = torch.where(p > n - 1 - layer, (p - (n - 1 - layer)) / layer, rho).clamp(max=1.0)
    inside = rho > 0
    sigma = -4.0 * math.log(float(np.float32(1e-6))) / (2.0 * layer * DX) * rho ** 3
    alpha = float(np.float32(0.05)) * (1.0 - rho)
    b = torch.exp(-(sigma + alpha) * DT)
    a = torch.where(inside, sigma / (sigma + alpha).clamp(min=1e-300) * (b - 1.0), 0 * b)
    b = torch.where(inside, b, torch.ones_like(b))
    view = [(None, None, slice(None)), (None, slice(None), None), (slice(None), None, None)][axis]
    return b[view], a[view]


def _steps64(shape, coef, fields, src, steps, layer=0, record=()):
    """Advances float64 fields in place; record: (component, plane, half step, freqs) -> sums."""
    c, m, p = slice(1, -1), slice(0, -2), slice(2, None)

    def mid(a):  # a coefficient over the interior
        return a[tuple(c if n > 1 else slice(None) for n in a.shape)]

    K = [mid(a) for a in coef]
    ex, ey, ez, hx, hy, hz = fields
    n = shape
    psi = {}
    prof = {(ax, h): _cpml_axis(n[ax], layer, h, ax) for ax in range(3) for h in (0, 1)} if layer else {}

    def diff(a, b, axis, half, key):
        d = a - b
        if not layer:
            return d
        bb, aa = (mid(v) for v in prof[axis, half])
        q = psi.get(key)
        q = aa * d if q is None else bb * q + aa * d
        psi[key] = q
        return d + q

    def source(comp, curl, t):
        if src["component"] != comp:
            return
        v = float(src["wave"][t]) * DX if t < len(src["wave"]) else 0.0
        if src.get("kind", gd.SRC_POINT) == gd.SRC_PLANE_Z:
            curl[src["k"] - 1] -= v
        else:
            curl[src["k"] - 1, src["j"] - 1, src["i"] - 1] -= v

    sums = [torch.zeros((2, len(f),) + (shape[1], shape[0]), dtype=torch.float64, device="cuda")
            for _, _, _, f in record]
    for t in range(steps):
        cu = [diff(hz[c, c, c], hz[c, m, c], 1, 0, 0) - diff(hy[c, c, c], hy[m, c, c], 2, 0, 1),
              diff(hx[c, c, c], hx[m, c, c], 2, 0, 2) - diff(hz[c, c, c], hz[c, c, m], 0, 0, 3),
              diff(hy[c, c, c], hy[c, c, m], 0, 0, 4) - diff(hx[c, c, c], hx[c, m, c], 1, 0, 5)]
        for q, f in enumerate((ex, ey, ez)):
            source(("Jx", "Jy", "Jz")[q], cu[q], t)
            f[c, c, c] = K[q] * f[c, c, c] + K[3 + q] * cu[q]
        cu = [diff(ey[p, c, c], ey[c, c, c], 2, 1, 6) - diff(ez[c, p, c], ez[c, c, c], 1, 1, 7),
              diff(ez[c, c, p], ez[c, c, c], 0, 1, 8) - diff(ex[p, c, c], ex[c, c, c], 2, 1, 9),
              diff(ex[c, p, c], ex[c, c, c], 1, 1, 10) - diff(ey[c, c, p], ey[c, c, c], 0, 1, 11)]
        for q, f in enumerate((hx, hy, hz)):
            f[c, c, c] = K[6 + q] * f[c, c, c] + K[9 + q] * cu[q]
        del cu
        for s, (comp, k, off, freqs) in zip(sums, record):
            ph = torch.from_numpy(2.0 * math.pi * freqs * ((t + off) * DT)).cuda()
            v = fields[comp][k][None]
            s[0] += v * torch.cos(ph)[:, None, None]
            s[1] -= v * torch.sin(ph)[:, None, None]
    return sums


def _flux_records(k, nf):
    f = _band(nf)
    return [(0, k, 0.0, f), (1, k, 0.0, f), (3, k - 1, 0.5, f), (3, k, 0.5, f),
            (4, k - 1, 0.5, f), (4, k, 0.5, f)]


def _flux(s):
    ex, ey = s[0], s[1]
    hx, hy = 0.5 * (s[2] + s[3]), 0.5 * (s[4] + s[5])
    v = (ex[0] * hy[0] + ex[1] * hy[1]) - (ey[0] * hx[0] + ey[1] * hx[1])
    return DX * DX * v.sum(dim=(1, 2))


def _round32(coef):
    return [a.to(torch.float32).to(torch.float64) for a in coef]


def exact(case, seed):
    c = case
    if c["kind"] == "grid":
        shape, eps, layer, fields, src, planes = _grid_inputs(c, seed)
        coef = _round32(_coefficients(shape, eps, layer))
        del eps
        f = [fields.pop(0).to(torch.float64) for _ in range(6)]
        cp = _cpml_layer(c, shape) if c["boundary"] == "cpml" else 0
        rec = [(FIELDS.index(name), k, 0.0, _band(c["nf"])) for name, k in planes]
        sums = _steps64(shape, coef, f, src, c["steps"], cp, rec)
        return {"fields": f, "dft": sums}
    if c["kind"] == "batch":
        cpml = c["boundary"] == "cpml"
        res, out = [], []
        for n, shape in enumerate(_batch_shapes(c, seed)):
            eps, src = _batch_inputs(c, seed, n, shape)
            coef = _round32(_coefficients(shape, eps, 0 if cpml else c["layer"]))
            g = _gen(seed * 1000 + n)
            f = torch.randn((6,) + shape[::-1], device="cuda", generator=g).to(torch.float64)
            if cpml:
                rec = _flux_records(shape[2] - c["layer"] - 2, c["nf"])
            else:
                rec = [(2, shape[2] // 2, 0.0, _band(c["nf"]))]
            s = _steps64(shape, coef, list(f), src, c["steps"],
                         _cpml_layer(c, shape) if cpml else 0, rec)
            res.append(_flux(s) if cpml else s[0])
            out.append(f)
        return {"fields": out, "result": res}
    if c["kind"] == "design":
        n = c["n"]
        eps = torch.from_numpy(_box((n, n, n), np.random.default_rng(seed))).cuda()
        coef = _coefficients((n, n, n), eps, 10)
        f = [torch.zeros((n, n, n), dtype=torch.float64, device="cuda") for _ in range(6)]
        src = dict(component="Jx", kind=gd.SRC_PLANE_Z, k=10, wave=_wave(c["steps"], seed))
        s = _steps64((n, n, n), coef, f, src, c["steps"], 0, _flux_records(n - 10, c["nf"]))
        return {"flux": _flux(s), "ex": f[0].reshape(-1)}
    if c["kind"] == "predict":
        _, ws, x, _ = _net_inputs(c, seed)
        mean = torch.zeros((c["rows"], c["out"]), dtype=torch.float64, device="cuda")
        sd = torch.zeros_like(mean)
        for r in range(0, c["rows"], 32768):
            ys = []
            for layers in ws:
                a = x[r:r + 32768].to(torch.float64)
                for q, (w, b) in enumerate(layers):
                    a = a @ w.to(torch.float64).T + b.to(torch.float64)
                    if q + 1 < len(layers):
                        a = 0.5 * a * (1.0 + torch.erf(a / math.sqrt(2.0)))
                ys.append(a)
            ys = torch.stack(ys)
            mean[r:r + 32768], sd[r:r + 32768] = ys.mean(0), ys.std(0, correction=0)
        return {"mean": mean, "sd": sd}
    return None  # an epoch's parameters hang on the library's own shuffle of the rows
