"""What the framework is timed on: the void finder's path as its users call it.

Every case is a whole call, or a chain of calls, through the public entry
points: ``sif_gb300.device`` (particles resident on the GPU),
``sif_gb300.autograd`` (the differentiable contrast) and ``sif_gb300.pysif``
(sif's own API on host arrays). Inputs are Zel'dovich-displaced lattices (the
recipe of ``sif_gb300.synth``, made on the GPU from the seed), ladders of
radii from about twice the mean particle separation upwards in steps of 10%,
and density thresholds between -0.5 and -0.8: a simulation's snapshot, a
halo catalogue with masses, a galaxy survey with its randoms.

The catalogues (centres and radii) are compared as they come; only the fields
and gradients are computed numbers that plain torch gives in 64 bits.
"""
import math

import numpy as np
import torch

from sif_gb300 import abi, autograd, device, pysif, synth

_ready = False


def _init():
    global _ready
    if not _ready:
        pysif.system_init(log_level="error")
        _ready = True


# The excursion-peak preset's options (sif_finder_exodus_preset): minima
# seeds, the extended reach, displacement, an overlap fraction of 1.
_PEAK = abi.SIF_FINDER_SEEDS_MINIMA | abi.SIF_FINDER_EXTEND_REACH | abi.SIF_FINDER_DISPLACE


def listed():
    return [
        # The smallest snapshot anyone searches: latency and launches.
        dict(name="box_64", kind="box", n=64, drop=0, box=250.0, rms=4.0, grid=64, r0=7.5, rungs=19,
             threshold=-0.8, overlap=0.0, variant="set", dtype="float32"),
        # An ordinary snapshot with sizes that are powers of nothing: a
        # lattice less some particles, a grid finer than it, overlap allowed.
        dict(name="box_201_grid_243", kind="box", n=201, drop=1237, box=700.0, rms=5.0, grid=243,
             r0=6.5, rungs=17, threshold=-0.75, overlap=0.3, variant="set", dtype="float32"),
        # The benchmark's own workload: 512^3 particles, 19 rungs.
        dict(name="box_512", kind="box", n=512, drop=0, box=1000.0, rms=5.0, grid=512, r0=4.0,
             rungs=19, threshold=-0.8, overlap=0.0, variant="set", dtype="float32"),
        # The same path in the double form (SIF_USE_DOUBLE's arithmetic).
        dict(name="box_f64_256", kind="box", n=256, drop=0, box=500.0, rms=4.0, grid=256, r0=5.0,
             rungs=19, threshold=-0.8, overlap=0.0, variant="set", dtype="float64"),
        # The excursion-peak preset: displacement among overlapping peaks.
        dict(name="peak_256", kind="box", n=256, drop=0, box=500.0, rms=4.0, grid=256, r0=5.0,
             rungs=19, threshold=-0.8, overlap=1.0, variant="peak", dtype="float32"),
        # Many realisations at once (mocks, an emulator's design): 64 boxes.
        dict(name="batch_64", kind="batch", boxes=64, lo=64, hi=256, threshold=-0.8),
        # Deposit, contrast and chain mesh alone, ragged sizes: what a caller
        # who brings a finder or a power spectrum of their own runs.
        dict(name="fields_401", kind="fields", n=401, drop=77, box=900.0, rms=5.0, grid=500,
             mesh=117, dtype="float32"),
        # One smoothing of a density contrast, on the benchmark's grid.
        dict(name="smooth_512", kind="smooth", grid=512, box=1000.0, radius=8.0, filter="top-hat",
             window="full", dtype="float32"),
        # Forward and backward through deposit and smoothing: a loss on the
        # smoothed field around void centres (the differentiation workload).
        dict(name="gradient_256", kind="gradient", n=256, drop=0, box=500.0, rms=4.0, grid=256,
             radius=5.0, filter="gaussian", centres=1000, dtype="float32"),
        # Haloes with masses: the weighted deposit, mesh and finder.
        dict(name="weighted_150", kind="weighted", n=150, drop=331, box=600.0, rms=5.0, grid=160,
             r0=8.0, rungs=15, threshold=-0.7, dtype="float32"),
        # A galaxy survey with randoms, weighted, through sif's API on host
        # arrays.
        dict(name="survey_host_96", kind="survey", data=120000, randoms=1200000, grid=96, mesh=26,
             r0=10.0, rungs=12, threshold=-0.5),
        # A snapshot in host memory through sif's API: field, grid, mesh,
        # finder, as a script for the reference's pysif runs it.
        dict(name="host_256", kind="host", n=256, drop=0, box=500.0, rms=4.0, grid=256, mesh=62,
             r0=5.0, rungs=19, threshold=-0.8),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["box", "box", "box", "box64", "peak", "batch", "fields", "smooth", "smooth",
                       "gradient", "weighted", "survey", "host"])
    dtype = rng.choice(["float32", "float32", "float64"])
    if kind in ("box", "box64", "peak", "host", "weighted"):
        n = _log_int(rng, 48, dict(box=400, box64=200, peak=220, host=256, weighted=180)[kind])
        sep = rng.uniform(1.9, 4.0)
        c = dict(kind=kind, n=n, drop=rng.randrange(0, n * n // 8), box=round(n * sep, 2),
                 rms=round(sep * rng.uniform(1.0, 2.2), 3),
                 grid=n if rng.random() < 0.4 else int(round(n * rng.uniform(0.8, 1.25))),
                 r0=round(sep * rng.uniform(2.0, 2.4), 3), rungs=rng.randint(8, 19),
                 threshold=round(rng.uniform(-0.85, -0.65), 3))
        if kind in ("box", "box64", "peak"):
            c.update(kind="box", variant="peak" if kind == "peak" else "set",
                     overlap=1.0 if kind == "peak" else rng.choice([0.0, 0.0, 0.25, 0.5]),
                     dtype="float64" if kind == "box64" else "float32")
        elif kind == "host":
            c.update(mesh=max(10, int(round(n / 4.1))))
        else:
            c.update(dtype=dtype)
        return c
    if kind == "batch":
        return dict(kind="batch", boxes=rng.randint(5, 48), lo=rng.randint(48, 90),
                    hi=rng.randint(110, 230), threshold=round(rng.uniform(-0.85, -0.7), 3))
    if kind == "survey":
        data = _log_int(rng, 20000, 150000)
        return dict(kind="survey", data=data, randoms=data * rng.randint(4, 10),
                    grid=rng.randint(48, 120), mesh=rng.randint(16, 30),
                    r0=round(rng.uniform(10.0, 14.0), 2), rungs=rng.randint(6, 12),
                    threshold=round(rng.uniform(-0.8, -0.5), 3))
    n = _log_int(rng, 48, dict(fields=420, smooth=500, gradient=240)[kind])
    sep = rng.uniform(1.9, 4.0)
    if kind == "fields":
        return dict(kind="fields", n=n, drop=rng.randrange(0, n * n // 8), box=round(n * sep, 2),
                    rms=round(sep * rng.uniform(1.0, 2.2), 3), grid=int(round(n * rng.uniform(0.7, 1.25))),
                    mesh=max(8, int(round(n / rng.uniform(2.5, 5.0)))), dtype=dtype)
    c = dict(kind=kind, grid=n, box=round(n * sep, 2), radius=round(sep * rng.uniform(1.5, 8.0), 3),
             filter=rng.choice(["top-hat", "gaussian"]), dtype=dtype)
    if kind == "smooth":
        c.update(window=rng.choice(["none", "full", "aliasing"]))
    else:
        c.update(n=n, drop=rng.randrange(0, n * n // 8), rms=round(sep * rng.uniform(1.0, 2.2), 3),
                 centres=rng.randint(20, 1000))
    return c


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------

def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed) * 7919 + 13)


def _zeldovich(n, box, rms, seed, dtype=torch.float32, drop=0):
    """n^3 - drop particles of a displaced lattice, in [0, box): spectrum
    P(k) ~ k^-1 exp(-(2k)^2), rms displacement `rms` (sif_gb300.synth's recipe,
    with the GPU's random numbers)."""
    g = _generator(seed)
    white = torch.fft.rfftn(torch.randn((n, n, n), generator=g, device="cuda"))
    kf = 2.0 * math.pi / box
    k1 = torch.fft.fftfreq(n, d=1.0 / n, device="cuda") * kf
    kz = torch.fft.rfftfreq(n, d=1.0 / n, device="cuda") * kf
    k2 = k1[:, None, None] ** 2 + k1[None, :, None] ** 2 + kz[None, None, :] ** 2
    k2[0, 0, 0] = 1.0
    white *= torch.sqrt(k2 ** -0.5 * torch.exp(-4.0 * k2)) / k2
    white[0, 0, 0] = 0.0
    del k2
    psi = []
    for a, k in enumerate((k1[:, None, None], k1[None, :, None], kz[None, None, :])):
        psi.append(torch.fft.irfftn(1j * k * white, s=(n, n, n)))
    del white
    scale = rms / math.sqrt(sum(float((p.double() ** 2).mean()) for p in psi))
    q = (torch.arange(n, device="cuda", dtype=torch.float64) + 0.5) * (box / n)
    keep = torch.randperm(n ** 3, generator=g, device="cuda")[drop:].sort().values if drop else None
    edge = torch.tensor(box, dtype=dtype, device="cuda")
    out = []
    for a in range(3):
        shape = [1, 1, 1]
        shape[a] = n
        v = psi[a].double()
        psi[a] = None
        v = torch.remainder(q.reshape(shape) + scale * v, box).to(dtype).reshape(-1)
        v = torch.where(v >= edge, torch.zeros_like(v), v)
        out.append(v[keep].contiguous() if drop else v)
    return out


def _ladder(case):
    return [case["r0"] * 1.1 ** i for i in range(case["rungs"])]


def _mesh_cells(case):
    """pysif's rule; the benchmark's own workload sets 8 Mpc/h."""
    if case["n"] == 512:
        return int(round(case["box"] / 8.0))
    return pysif.finders.suggest_mesh_cells(case["n"] ** 3 - case["drop"], case["box"],
                                            _ladder(case)[-1])


def _dtype(case):
    return getattr(torch, case.get("dtype", "float32"))


def _batch_sizes(case, seed):
    rng = np.random.default_rng(2000)  # the same sizes whatever the seed: the work is the case's
    out = []
    for _ in range(case["boxes"]):
        n = int(round(math.exp(rng.uniform(math.log(case["lo"]), math.log(case["hi"])))))
        out.append((n + n % 2, float(rng.uniform(200.0, 1000.0))))
    return out


def _contrast_field(case, seed):
    """A density contrast as a deposit gives one: lognormal noise around a
    smooth large-scale mode, mean zero, never below -1."""
    n = case["grid"]
    g = _generator(seed)
    v = torch.randn((n, n, n), generator=g, device="cuda", dtype=torch.float32)
    q = torch.arange(n, device="cuda", dtype=torch.float32) * (2.0 * math.pi / n)
    ph = torch.rand(3, generator=g, device="cuda") * 6.28
    v += torch.sin(3 * q + ph[0])[:, None, None] + torch.sin(5 * q + ph[1])[None, :, None] + \
        torch.sin(2 * q + ph[2])[None, None, :]
    v = torch.exp(0.5 * v)
    v = v / v.double().mean().float() - 1.0
    return v.reshape(-1).to(_dtype(case)).contiguous()


def prepare(case, seed):
    _init()
    kind = case["kind"]
    s = dict(case=case)
    if kind in ("box", "fields", "gradient", "weighted", "host"):
        xs = _zeldovich(case["n"], case["box"], case["rms"], seed, _dtype(case), case["drop"])
    if kind in ("box", "weighted", "host"):
        real = np.float64 if case.get("dtype") == "float64" else np.float32
        s["radii"] = np.array(_ladder(case), real)
    if kind in ("box", "weighted"):
        s["mesh"] = _mesh_cells(case)
    if kind == "batch":
        s["boxes"] = []
        for k, (n, box) in enumerate(_batch_sizes(case, seed)):
            x, y, z = _zeldovich(n, box, 4.0, seed * 1000 + k)
            r0 = 2.0 * box / n
            s["boxes"].append(dict(x=x, y=y, z=z, n_grid=n, box=box, mesh_cells=0,
                                   radii=synth.ladder(r0, 6 * r0, 0.10).astype(np.float32),
                                   threshold=case["threshold"]))
    elif kind == "smooth":
        s["delta"] = _contrast_field(case, seed)
    elif kind == "gradient":
        s["xs"] = [v.requires_grad_(True) for v in xs]
        s["mask"] = _near_centres(case, seed)
    elif kind == "weighted":
        # Masses over a decade and a half, a tenth of the haloes masked out.
        g = _generator(seed + 1)
        w = torch.exp(0.8 * torch.randn(xs[0].numel(), generator=g, device="cuda"))
        w *= torch.rand(xs[0].numel(), generator=g, device="cuda") > 0.1
        s.update(xs=xs, w=w.to(_dtype(case)).contiguous())
    elif kind == "host":
        s["xs"] = [v.cpu().numpy() for v in xs]
    elif kind == "survey":
        data, rand = synth.survey(case["data"], case["randoms"], int(seed) + 7, selection=True)
        rng = np.random.default_rng(int(seed) + 8)
        s.update(data=data, rand=rand, wd=rng.uniform(0.5, 1.5, len(data[0])).astype(np.float32),
                 wr=np.full(len(rand[0]), 1.0, np.float32),
                 radii=np.array(_ladder(case), np.float32))
    else:
        s["xs"] = xs
    torch.cuda.synchronize()
    return s


def _near_centres(case, seed):
    """The cells within two radii of some points: where the loss looks."""
    n, box = case["grid"], case["box"]
    cell, reach = box / n, 2.0 * case["radius"]
    g = _generator(seed + 2)
    c = torch.rand((case["centres"], 3), generator=g, device="cuda", dtype=torch.float64) * box
    span = min(int(reach / cell) + 1, n // 2)
    off = torch.arange(-span, span + 1, device="cuda")
    o = torch.stack([v.reshape(-1) for v in torch.meshgrid(off, off, off, indexing="ij")], 1)
    mask = torch.zeros(n ** 3, dtype=torch.bool, device="cuda")
    for chunk in torch.split(c, max(1, (1 << 24) // len(o))):
        i = torch.floor(chunk / cell).long()[:, None, :] + o[None]
        near = ((i.double() * cell - chunk[:, None, :]) ** 2).sum(2) <= reach * reach
        i = torch.remainder(i[near], n)
        mask[(i[:, 0] * n + i[:, 1]) * n + i[:, 2]] = True
    return mask


# ---------------------------------------------------------------------------
# One pass
# ---------------------------------------------------------------------------

def _table(columns, particles):
    """A catalogue as the rows of one table with room for any catalogue of so
    many particles (a void holds hundreds), the rest zero, and its length."""
    n = len(columns[0])
    out = np.zeros((len(columns), 4096 + particles // 128), columns[0].dtype)
    for row, col in zip(out, columns):
        row[:n] = col
    return dict(voids=out, count=n)


def run(s):
    c = s["case"]
    kind = c["kind"]
    if kind == "box":
        peak = c["variant"] == "peak"
        cat = device.box(*s["xs"], c["grid"], c["box"], s["mesh"], s["radii"], c["threshold"],
                         overlap=c["overlap"], options=_PEAK if peak else 0)
        return _table(cat, s["xs"][0].numel())
    if kind == "batch":
        cats, _ = device.box_batch(s["boxes"], engines=4)
        return _table([np.concatenate([cat[k] for cat in cats]) for k in range(4)],
                      sum(b["x"].numel() for b in s["boxes"]))
    if kind == "fields":
        grid = device.cic(*s["xs"], c["grid"], c["box"])
        mean = device.density_contrast(grid)
        mx, my, mz, offs, orig = device.chain_mesh(*s["xs"], c["mesh"], c["box"])
        return dict(contrast=grid, mean=mean, mx=mx, my=my, mz=mz, offsets=offs, indices=orig)
    if kind == "smooth":
        return device.smooth(s["delta"], c["grid"], c["box"], c["radius"], filter=c["filter"],
                             window=c["window"])
    if kind == "gradient":
        f = autograd.smoothed_contrast(*s["xs"], c["grid"], c["box"], c["radius"],
                                       filter=c["filter"])
        loss = (f[s["mask"]] ** 2).sum()
        gx, gy, gz = torch.autograd.grad(loss, s["xs"])
        return dict(field=f.detach(), gx=gx, gy=gy, gz=gz)
    if kind == "weighted":
        grid = device.cic_weighted(*s["xs"], s["w"], c["grid"], c["box"])
        device.density_contrast(grid)
        mesh = device.chain_mesh(*s["xs"], s["mesh"], c["box"])
        weights = device.mesh_weights(s["w"], mesh, s["mesh"])
        cat = device.exodus(grid, c["grid"], c["box"], mesh, s["mesh"], s["radii"], c["threshold"],
                            weights=weights)
        return dict(contrast=grid, catalogue=_table(cat, s["xs"][0].numel()), total=weights[2])
    if kind == "survey":
        box = synth.SURVEY["box"]
        fd = pysif.Field(*s["data"], weights=s["wd"])
        fr = pysif.Field(*s["rand"], weights=s["wr"])
        gd, gr = pysif.Grid(c["grid"], box), pysif.Grid(c["grid"], box)
        gd.assign_cic(fd)
        gr.assign_cic(fr)
        md, mr = (pysif.ChainMesh(c["mesh"], box, f, drop_indices=True) for f in (fd, fr))
        cat = pysif.finders.exodus_survey_raw(gd, gr, md, mr, s["radii"], c["threshold"])
        return _table([*cat.as_tuple(), cat.footprint, cat.footprint_shell], c["data"])
    # host
    f = pysif.Field(*s["xs"])
    grid = pysif.Grid(c["grid"], c["box"])
    grid.assign_cic(f)
    grid.to_density_contrast()
    mesh = pysif.ChainMesh(c["mesh"], c["box"], f, drop_indices=True)
    cat = pysif.finders.exodus_raw(grid, mesh, s["radii"], c["threshold"])
    s["grid"] = grid  # the contrast below is a view of its values
    return dict(contrast=grid.values, catalogue=_table(cat.as_tuple(), len(s["xs"][0])))


# ---------------------------------------------------------------------------
# What a pass cannot do without
# ---------------------------------------------------------------------------

def _fft_flops(n):
    return 2.5 * n ** 3 * 3.0 * math.log2(n)  # a real transform of n^3 values


def work(case):
    """Bytes: inputs read once, outputs written once (a catalogue's few
    hundred kilobytes left out). Operations: the transforms' (one forward, one
    inverse a rung), 60 a particle for its eight corners, 10 a particle for
    its cell."""
    kind = case["kind"]
    w = 8 if case.get("dtype") == "float64" else 4
    if kind == "batch":
        sizes = _batch_sizes(case, 0)
        return dict(bytes=float(sum(12 * n ** 3 for n, _ in sizes)),
                    flops=float(sum(20 * _fft_flops(n) + 70 * n ** 3 for n, _ in sizes)))
    g3 = case["grid"] ** 3
    if kind == "smooth":
        return dict(bytes=2.0 * w * g3, flops=2 * _fft_flops(case["grid"]) + 2.0 * g3)
    if kind == "survey":
        p = case["data"] + case["randoms"]
        return dict(bytes=16.0 * p, flops=2 * (1 + case["rungs"]) * _fft_flops(case["grid"]) + 70.0 * p)
    p = case["n"] ** 3 - case["drop"]
    if kind == "fields":
        m3 = case["mesh"] ** 3
        return dict(bytes=float(3 * w * p + w * g3 + 3 * w * p + 4 * p + 4 * m3), flops=70.0 * p)
    if kind == "gradient":
        return dict(bytes=float(6 * w * p + w * g3 + g3), flops=4 * _fft_flops(case["grid"]) + 160.0 * p)
    flops = (1 + case["rungs"]) * _fft_flops(case["grid"]) + 70.0 * p
    if kind == "weighted":
        return dict(bytes=float(4 * w * p + w * g3), flops=flops)
    if kind == "host":
        return dict(bytes=float(12 * p + 4 * g3), flops=flops)
    return dict(bytes=float(3 * w * p), flops=flops)


# ---------------------------------------------------------------------------
# 64-bit values
# ---------------------------------------------------------------------------

def _deposit64(xs, n, box, weights=None):
    """CIC in float64: node i at i * box / n, weights (1 - t, t) per axis."""
    axes = []
    for v in xs:
        u = torch.remainder(v, box) * (n / box)
        raw = torch.floor(u).detach()
        t = u - raw
        i0 = torch.remainder(raw, n).long()
        axes.append(((i0, 1.0 - t), (torch.remainder(i0 + 1, n), t)))
    rho = torch.zeros(n ** 3, dtype=torch.float64, device=xs[0].device)
    for ix, wx in axes[0]:
        for iy, wy in axes[1]:
            for iz, wz in axes[2]:
                wt = wx * wy * wz
                rho = rho.index_add(0, (ix * n + iy) * n + iz, wt if weights is None else wt * weights)
    return rho


def _inverse_window(n, k, window):
    """The CIC window's correction along one axis: 1/sinc^2 ("full"); None for
    the others ("none" has none, the aliasing-aware one is not separable)."""
    x = math.pi * k / n
    s = torch.where(x.abs() < 1e-9, torch.ones_like(x), torch.sin(x) / x)
    return 1.0 / (s * s) if window == "full" else torch.ones_like(k)


def _smooth64(delta, n, box, radius, filter, window):
    k1 = torch.fft.fftfreq(n, d=1.0 / n, device=delta.device, dtype=torch.float64)
    kz = torch.fft.rfftfreq(n, d=1.0 / n, device=delta.device, dtype=torch.float64)
    x = torch.sqrt(k1[:, None, None] ** 2 + k1[None, :, None] ** 2 + kz[None, None, :] ** 2)
    x *= radius * 2.0 * math.pi / box
    if filter == "gaussian":
        f = torch.exp(-0.5 * x * x)
    else:
        small = x < 1e-2
        x = torch.where(small, torch.ones_like(x), x)
        f = 3.0 * (torch.sin(x) - x * torch.cos(x)) / x ** 3
        y = torch.sqrt(k1[:, None, None] ** 2 + k1[None, :, None] ** 2 + kz[None, None, :] ** 2)
        y *= radius * 2.0 * math.pi / box
        f = torch.where(small, 1.0 - y * y / 10.0 + y ** 4 / 280.0, f)
        del y
    del x
    a, b = _inverse_window(n, k1, window), _inverse_window(n, kz, window)
    f *= a[:, None, None]
    f *= a[None, :, None]
    f *= b[None, None, :]
    spec = torch.fft.rfftn(delta.reshape(n, n, n))
    return torch.fft.irfftn(spec * f, s=(n, n, n)).reshape(-1)


def exact(case, seed):
    kind = case["kind"]
    if kind not in ("fields", "smooth", "gradient", "weighted"):
        return None  # catalogues: decisions, compared with the start's
    if kind == "smooth" and case["window"] == "aliasing":
        return None
    s = prepare(case, seed)
    n, box = case["grid"], case["box"]
    if kind == "smooth":
        return _smooth64(s["delta"].double(), n, box, case["radius"], case["filter"], case["window"])
    xs = [v.detach().double() for v in s["xs"]]
    if kind == "fields":
        mean = xs[0].numel() / box ** 3
        rho = _deposit64(xs, n, box)
        return dict(contrast=rho / (xs[0].numel() / n ** 3) - 1.0, mean=mean, mx=None, my=None,
                    mz=None, offsets=None, indices=None)
    if kind == "weighted":
        w = s["w"].double()
        total = float(w.sum())
        return dict(contrast=_deposit64(xs, n, box, w) / (total / n ** 3) - 1.0, catalogue=None,
                    total=total)
    xs = [v.requires_grad_(True) for v in xs]
    rho = _deposit64(xs, n, box)
    f = _smooth64(rho / (xs[0].numel() / n ** 3) - 1.0, n, box, case["radius"], case["filter"], "full")
    gx, gy, gz = torch.autograd.grad((f[s["mask"]] ** 2).sum(), xs)
    return dict(field=f.detach(), gx=gx, gy=gy, gz=gz)
