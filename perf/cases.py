"""The work this package is measured by: calls a user's program makes through
the public entry points, from the smallest to the largest, with the inputs
they meet in use.  Lengths are in micrometres.

Every case names a ``kind``:

``fields``    simulation.cuda.simulate_batch, complex64 fields of a few images
              (settings with "single")
``double``    the same call in the default FP64 precision, complex128 fields
``plan``      simulation.batch.BatchPlan: uneven images under a CUDA graph
``fit``       simulation.autograd.intensity and its backward pass
``time``      simulation.cutime.simulate, the arrival-time-sorted variant
``detector``  simulation.common.randomphotons, then chargesharing
``autocorr``  reconstruction.cusimple.corr, FFT autocorrelation
``radial``    reconstruction.cucorrad.corrfunction, q-space correlation
"""

from __future__ import annotations

import math

import numpy as np
import torch

from idi_b200 import _native as nat
from idi_b200.reconstruction import cucorrad, cusimple
from idi_b200.simulation import autograd, common, cutime, simobj
from idi_b200.simulation import cuda as sim
from idi_b200.simulation._core import make_geom
from idi_b200.simulation.batch import BatchPlan


def listed():
    return [
        # two small images of a hundred emitters on a small detector: launches and
        # host work are all there is (unit tests, parameter scans)
        dict(name="fields tiny", kind="fields", images=2, emitters=100, radius=0.01, nx=32, ny=30, energy=6400.0,
             pixel=75.0, detz=1e5, settings="nf single", shape="sphere", amplitudes=False, tilt=0.0),
        # the small configuration: 2,000 emitters in a 10 nm sphere, 256^2, 8 images
        dict(name="fields small", kind="fields", images=8, emitters=2000, radius=0.01, nx=256, ny=256, energy=6400.0,
             pixel=75.0, detz=1e5, settings="single", shape="sphere", amplitudes=False, tilt=0.0),
        # the precision configuration: 50,000 fcc sites in a 12 nm cube, 1024^2, near field
        dict(name="fields large", kind="fields", images=2, emitters=50000, radius=0.006, nx=1024, ny=1024,
             energy=8000.0, pixel=50.0, detz=2e5, settings="nf single", shape="fcc", amplitudes=False, tilt=0.0),
        # a wide object on few pixels, as a foil's focal volume: a micrometre across, so that
        # a pixel step is many radians of phase
        dict(name="fields wide object", kind="fields", images=1, emitters=300000, radius=0.5, nx=128, ny=128,
             energy=8000.0, pixel=50.0, detz=2e5, settings="single", shape="sphere", amplitudes=False, tilt=0.0),
        # ragged: odd detector, tilted, amplitudes and the 1/r factor
        dict(name="fields ragged tilted", kind="fields", images=3, emitters=7777, radius=0.017, nx=301, ny=517,
             energy=6400.0, pixel=75.0, detz=1e5, settings="nf scale single", shape="sphere", amplitudes=True,
             tilt=0.2),
        # the default precision on the small configuration
        dict(name="double small", kind="double", images=4, emitters=2000, radius=0.01, nx=256, ny=256, energy=6400.0,
             pixel=75.0, detz=1e5, settings="double", shape="sphere", amplitudes=False, tilt=0.0),
        # the batched configuration: uneven images, amplitudes, one graph replay per batch
        dict(name="plan uneven", kind="plan", images=24, lo=1000, hi=100000, nx=512, ny=512, energy=6400.0,
             pixel=75.0, detz=1e5),
        # the differentiation configuration: one gradient step of a 10,000-emitter structure
        dict(name="fit", kind="fit", emitters=10000, radius=0.015, nx=512, ny=512, energy=6400.0, pixel=75.0,
             detz=1e5, settings="nf", amplitudes=True),
        # the time-dependent configuration: 20,000 emitters, 256^2
        dict(name="time", kind="time", emitters=20000, radius=0.01, nx=256, ny=256, energy=6400.0, pixel=75.0,
             detz=1e5, tau=2.0, fwhm=5.0),
        # photon counts and charge sharing of simulated intensities
        dict(name="detector", kind="detector", images=8, nx=1024, ny=1024, photons=1e5, spread=0.5),
        # FFT autocorrelation of a stack of detector images whose padded size is no power of two
        dict(name="autocorr", kind="autocorr", images=8, nx=1000, ny=1050, dtype="float64"),
        # radial q-space correlation
        dict(name="radial", kind="radial", images=2, nx=512, ny=512, z=2000.0, bins=256),
    ]


# ---------------------------------------------------------------------------
# more cases of the same ranges
# ---------------------------------------------------------------------------
def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _logint(rng, lo, hi):
    return int(round(_log(rng, lo, hi)))


def _even(n, limit):
    """The nearest size from n on whose padded length is even, as the usual widths are."""
    while _fastlen(2 * n) % 2 or _fastlen(2 * n) > limit:
        n -= 1
    return n


def draw(rng):
    kind = rng.choice(["fields", "fields", "fields", "double", "plan", "fit", "time", "detector", "autocorr",
                       "radial"])
    energy, pixel, detz = rng.choice([(6400.0, 75.0, 1e5), (8000.0, 50.0, 2e5)])
    base = dict(kind=kind, energy=energy, pixel=pixel, detz=detz)
    if kind == "fields":
        nx, ny = _logint(rng, 24, 1024), _logint(rng, 24, 1024)
        images = rng.randint(1, 8)
        n = min(_logint(rng, 100, 50000), int(5e10 / (images * nx * ny)))
        return dict(base, images=images, emitters=max(n, 50), radius=_log(rng, 0.005, 0.2), nx=nx, ny=ny,
                    settings=rng.choice(["nf single", "single", "nf scale single"]), shape="sphere",
                    amplitudes=rng.random() < 0.5, tilt=rng.choice([0.0, rng.uniform(-0.4, 0.4)]))
    if kind == "double":
        nx, ny = _logint(rng, 24, 300), _logint(rng, 24, 300)
        images = rng.randint(1, 4)
        return dict(base, images=images, emitters=_logint(rng, 100, 2000), radius=_log(rng, 0.005, 0.05), nx=nx,
                    ny=ny, settings=rng.choice(["double", "nf double"]), shape="sphere", amplitudes=False, tilt=0.0)
    if kind == "plan":
        n = _logint(rng, 100, 512)
        return dict(base, images=rng.randint(2, 24), lo=_logint(rng, 300, 3000), hi=_logint(rng, 5000, 50000), nx=n,
                    ny=_logint(rng, 100, 512))
    if kind == "fit":
        return dict(base, emitters=_logint(rng, 500, 10000), radius=_log(rng, 0.005, 0.025), nx=_logint(rng, 32, 512),
                    ny=_logint(rng, 32, 512), settings=rng.choice(["nf", ""]), amplitudes=rng.random() < 0.5)
    if kind == "time":
        return dict(base, emitters=_logint(rng, 500, 20000), radius=_log(rng, 0.005, 0.025), nx=_logint(rng, 24, 200),
                    ny=_logint(rng, 24, 200), tau=_log(rng, 1.0, 4.0), fwhm=_log(rng, 3.0, 8.0))
    if kind == "detector":
        return dict(kind=kind, images=rng.randint(1, 8), nx=_logint(rng, 64, 1024), ny=_logint(rng, 64, 1024),
                    photons=_log(rng, 1e3, 1e5), spread=rng.uniform(0.3, 0.9))
    if kind == "autocorr":
        return dict(kind=kind, images=rng.randint(1, 8), nx=_even(_logint(rng, 64, 1100), 4096),
                    ny=_even(_logint(rng, 64, 1100), 4096), dtype=rng.choice(["float64", "float32"]))
    n = _logint(rng, 64, 400)
    return dict(kind=kind, images=rng.randint(1, 3), nx=n, ny=_logint(rng, 64, 400), z=rng.uniform(1000.0, 3000.0),
                bins=rng.randint(32, 256))


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _wavenumber(case):
    return 2 * math.pi / (1.24 / case["energy"])


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed) * 7919 + 17)


def _uniform(g, *shape):
    return torch.rand(*shape, generator=g, device="cuda", dtype=torch.float64)


def _sphere(g, n, radius):
    t = 2 * _uniform(g, n) - 1
    p = 2 * math.pi * _uniform(g, n)
    u = radius * _uniform(g, n) ** (1 / 3)
    s = torch.sqrt(1 - t * t)
    return torch.stack([u * t, u * s * torch.sin(p), u * s * torch.cos(p)], 1)


def _fcc(g, n, half):
    """n sites of an fcc lattice (0.36 nm) filling a cube, with 0.01 nm jitter."""
    a = 3.6e-4
    m = int(math.ceil(2 * half / a))
    c = torch.arange(m, device="cuda", dtype=torch.float64)
    cells = torch.stack(torch.meshgrid(c, c, c, indexing="ij"), -1).reshape(-1, 1, 3)
    base = torch.tensor([[0, 0, 0], [0.5, 0.5, 0], [0.5, 0, 0.5], [0, 0.5, 0.5]], device="cuda", dtype=torch.float64)
    sites = ((cells + base) * a).reshape(-1, 3)
    sites = sites[(sites < 2 * half).all(1)] - half
    pick = torch.randperm(sites.shape[0], generator=g, device="cuda")[:n]
    jitter = torch.randn(n, 3, generator=g, device="cuda", dtype=torch.float64)
    return sites[pick] + 1e-5 * jitter


def _rows(g, case, n, radius):
    """(n, 4) emitter rows [x, y, z, phase]."""
    pos = _fcc(g, n, radius) if case.get("shape") == "fcc" else _sphere(g, n, radius)
    return torch.cat([pos, 2 * math.pi * _uniform(g, n, 1)], 1)


def _images(case, seed):
    g = _generator(seed)
    rows = [_rows(g, case, case["emitters"], case["radius"]) for _ in range(case["images"])]
    amps = None
    if case["amplitudes"]:
        amps = [(0.5 + _uniform(g, case["emitters"])).to(torch.float32).cpu().numpy() for _ in rows]
    return rows, amps


def _plan_images(case, seed):
    """Emitter counts log-uniform, radii 5 to 25 nm, amplitudes 0.5 to 1.5."""
    # the counts belong to the plan, not to its inputs: the same for every seed
    r = np.random.default_rng(case["images"] * 1000 + case["nx"])
    counts = np.exp(r.uniform(np.log(case["lo"]), np.log(case["hi"]), case["images"])).astype(np.int64)
    g = _generator(seed)
    radii = (0.005 + 0.02 * _uniform(g, case["images"])).tolist()
    rows = [_rows(g, case, int(c), rad) for c, rad in zip(counts, radii)]
    amps = (0.5 + _uniform(g, int(counts.sum()))).to(torch.float32)
    return counts, rows, amps


def _fit_inputs(case, seed):
    """float32 parameters, as an optimiser holds them, and the intensities to be
    fitted: those of the structure with every position moved by 0.05 nm."""
    g = _generator(seed)
    n = case["emitters"]
    pos = _sphere(g, n, case["radius"])
    phase = 2 * math.pi * _uniform(g, n)
    amp = (0.5 + _uniform(g, n)).to(torch.float32) if case["amplitudes"] else None
    moved = pos + 5e-5 * torch.randn(n, 3, generator=g, device="cuda", dtype=torch.float64)
    return pos.to(torch.float32), phase.to(torch.float32), amp, moved


def _time_inputs(case, seed):
    g = _generator(seed)
    rows = _rows(g, case, case["emitters"], case["radius"]).cpu().numpy()
    pump = torch.randn(case["emitters"], generator=g, device="cuda", dtype=torch.float64) * (case["fwhm"] / 2.35)
    delay = -case["tau"] * torch.log1p(-_uniform(g, case["emitters"]))
    return rows, (pump + delay).cpu().numpy()


_LIGHT = 0.299792458  # um / fs


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("fields", "double"):
        rows, amps = _images(case, seed)
        return dict(case=case, rows=rows, amps=amps)
    if kind == "plan":
        counts, rows, amps = _plan_images(case, seed)
        geom = make_geom([case["nx"], case["ny"]], case["pixel"], case["detz"], _wavenumber(case), flags=nat.NF)
        plan = BatchPlan(counts, geom, nat.SPLIT, nat.OUT_I32, amplitudes="float32", autotune=False)
        return dict(case=case, plan=plan, rows=torch.cat(rows), amps=amps)
    if kind == "fit":
        pos, phase, amp, moved = _fit_inputs(case, seed)
        with torch.no_grad():
            target = autograd.intensity(moved, phase.to(torch.float64), amp, **_fit_geometry(case))
        leaves = [t.requires_grad_(True) for t in (pos, phase, amp) if t is not None]
        return dict(case=case, leaves=leaves, target=target)
    if kind == "time":
        rows, times = _time_inputs(case, seed)
        return dict(case=case, obj=simobj.fixed(case["energy"], rows[:, :3], rows[:, 3]), times=times)
    g = _generator(seed)
    if kind == "detector":
        # speckle: exponentially distributed intensities
        probs = -torch.log1p(-_uniform(g, case["images"], case["nx"], case["ny"]))
        return dict(case=case, probs=probs, seed=int(seed))
    speckle = -torch.log1p(-_uniform(g, case["images"], case["nx"], case["ny"]))
    if kind == "autocorr":
        return dict(case=case, x=speckle.to(getattr(torch, case["dtype"])))
    ctx = cucorrad.corrfunction((case["nx"], case["ny"]), case["z"], case["bins"], return_gpu=True)
    return dict(case=case, ctx=ctx, corr=ctx.__enter__(), x=speckle.to(torch.float32))


def _fit_geometry(case):
    return dict(Ndet=[case["nx"], case["ny"]], pixelsize=case["pixel"], detz=case["detz"], k=_wavenumber(case),
                settings=case["settings"])


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind in ("fields", "double"):
        return sim.simulate_batch(state["rows"], [case["nx"], case["ny"]], case["pixel"], case["detz"],
                                  _wavenumber(case), settings=case["settings"], detangles=(case["tilt"], 0.0),
                                  amplitudes=state["amps"])
    if kind == "plan":
        return state["plan"].run(state["rows"], state["amps"])
    if kind == "fit":
        for t in state["leaves"]:
            t.grad = None
        pos, phase = state["leaves"][:2]
        amp = state["leaves"][2] if case["amplitudes"] else None
        loss = ((autograd.intensity(pos, phase, amp, **_fit_geometry(case)) - state["target"]) ** 2).sum()
        loss.backward()
        return [t.grad for t in state["leaves"]]
    if kind == "time":
        return cutime.simulate(state["obj"], [case["nx"], case["ny"]], case["pixel"], case["detz"],
                               _wavenumber(case), _LIGHT, case["tau"], case["fwhm"], settings="double",
                               times=state["times"], returngpu=True)
    if kind == "detector":
        counts = common.randomphotons(state["probs"], case["photons"], rng=state["seed"], dtype=np.int32)
        return counts, common.chargesharing(counts, case["spread"], rng=state["seed"])
    if kind == "autocorr":
        return cusimple.corr(state["x"], returngpu=True)
    return state["corr"](state["x"])


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def work(case):
    """Bytes: inputs read once and outputs written once.  Operations: of the sum as it is
    defined (per emitter and pixel: the path difference, a sine and a cosine, the
    multiply-add of the field), of the transforms (5 n log2 n), or of the pixel pairs."""
    kind = case["kind"]
    npix = case["nx"] * case["ny"]
    if kind in ("fields", "double"):
        b = case["images"]
        amp = 4 if case["amplitudes"] else 0
        return {"bytes": b * (case["emitters"] * (32 + amp) + npix * (16 if kind == "double" else 8)),
                "flops": 12.0 * b * case["emitters"] * npix}
    if kind == "plan":
        r = np.random.default_rng(case["images"] * 1000 + case["nx"])
        counts = np.exp(r.uniform(np.log(case["lo"]), np.log(case["hi"]), case["images"])).astype(np.int64)
        n = int(counts.sum())
        return {"bytes": n * 36 + case["images"] * npix * 4, "flops": 12.0 * n * npix}
    if kind == "fit":
        n = case["emitters"]
        return {"bytes": n * 40 + npix * 8, "flops": (12.0 + 22.0) * n * npix}
    if kind == "time":
        n = case["emitters"]
        # per emitter and pixel: the sum's 12, the sort and the decaying scan
        return {"bytes": n * 40 + npix * 8, "flops": (12.0 + 20.0 + math.log2(n)) * n * npix}
    if kind == "detector":
        return {"bytes": case["images"] * npix * (8 + 4 + 8), "flops": 20.0 * case["images"] * npix}
    if kind == "autocorr":
        e = 8 if case["dtype"] == "float64" else 4
        full = 4 * npix
        return {"bytes": case["images"] * 5 * npix * e, "flops": 5.0 * case["images"] * full * math.log2(full)}
    rows = sum(max(0, case["nx"] - d) for d in range(case["bins"]))
    cols = sum(max(0, case["ny"] - abs(d)) for d in range(-case["bins"], case["bins"] + 1))
    return {"bytes": case["images"] * npix * 4, "flops": 8.0 * case["images"] * rows * cols}


# ---------------------------------------------------------------------------
# the same in 64 bits, by plain torch
# ---------------------------------------------------------------------------
def _rotation(alpha):
    """Yaw by 0, pitch by 0, roll by alpha: the detector's tilt about x."""
    c, s = math.cos(alpha), math.sin(alpha)
    return torch.tensor([[1, 0, 0], [0, c, -s], [0, s, c]], device="cuda", dtype=torch.float64)


def _pixels(case):
    """(nx * ny, 3) pixel positions."""
    x = (torch.arange(case["nx"], device="cuda", dtype=torch.float64) - case["nx"] / 2) * case["pixel"]
    y = (torch.arange(case["ny"], device="cuda", dtype=torch.float64) - case["ny"] / 2) * case["pixel"]
    d = torch.stack([x[:, None].expand(-1, case["ny"]), y[None, :].expand(case["nx"], -1),
                     torch.full((case["nx"], case["ny"]), case["detz"], device="cuda", dtype=torch.float64)], -1)
    d = d.reshape(-1, 3)
    tilt = case.get("tilt", 0.0)
    return d @ _rotation(tilt).T if tilt else d


def _q(case, d):
    """|d| and q = k (d / |d| - z), its last part without cancellation."""
    k = _wavenumber(case)
    rho2 = d[:, 0] ** 2 + d[:, 1] ** 2
    D = torch.sqrt(rho2 + d[:, 2] ** 2)
    return D, k * torch.stack([d[:, 0] / D, d[:, 1] / D, -rho2 / (D * (D + d[:, 2]))], 1)


def _blocks(npix, n):
    step = max(1, (1 << 22) // max(n, 1))
    return [(p, min(npix, p + step)) for p in range(0, npix, step)]


def _phase(case, near, rows, d, D, q):
    """Phases (pixels, emitters) and distances |d - r| (None in the far field)."""
    r, psi = rows[:, :3], rows[:, 3]
    if not near:
        return psi[None] - q @ r.T, None
    k = _wavenumber(case)
    rr = (r * r).sum(1)
    dr = d @ r.T
    dist = torch.sqrt((D * D)[:, None] + (rr[None] - 2 * dr))
    delta = (rr[None] - 2 * dr) / (dist + D[:, None])
    c = k * (d[:, 0] ** 2 + d[:, 1] ** 2) / (D + d[:, 2])  # k (|d| - d_z)
    return k * (delta + r[:, 2][None]) + psi[None] + c[:, None], dist


def _exact_field(case, settings, rows, amps):
    near, scale = "nf" in settings, "scale" in settings
    rows = rows.to(torch.float64)
    a = torch.ones_like(rows[:, 0]) if amps is None else torch.as_tensor(amps).to("cuda", torch.float64)
    d = _pixels(case)
    D, q = _q(case, d)
    out = torch.empty(d.shape[0], device="cuda", dtype=torch.complex128)
    for p, e in _blocks(d.shape[0], rows.shape[0]):
        ph, dist = _phase(case, near, rows, d[p:e], D[p:e], q[p:e])
        re, im = torch.cos(ph), torch.sin(ph)
        if scale and near:
            re, im = re / dist, im / dist
        out[p:e] = torch.complex(re @ a, im @ a)
        if scale and not near:
            out[p:e] /= D[p:e]
    return out.reshape(case["nx"], case["ny"])


def _exact_fit(case, seed):
    pos, phase, amp, moved = _fit_inputs(case, seed)
    near = "nf" in case["settings"]
    k = _wavenumber(case)
    n = pos.shape[0]
    a = torch.ones(n, device="cuda", dtype=torch.float64) if amp is None else amp.to(torch.float64)
    phase = phase.to(torch.float64)[:, None]
    rows = torch.cat([pos.to(torch.float64), phase], 1)
    target = _exact_field(case, case["settings"], torch.cat([moved, phase], 1), amp).abs().square().reshape(-1)
    E = _exact_field(case, case["settings"], rows, amp).reshape(-1)
    G = 4 * (E.abs().square() - target) * E.conj()  # 2 dL/dI conj(E)
    d = _pixels(case)
    D, q = _q(case, d)
    r = rows[:, :3]
    gp, gr, ga = (torch.zeros(*s, device="cuda", dtype=torch.float64) for s in ((n,), (n, 3), (n,)))
    for p, e in _blocks(d.shape[0], n):
        ph, dist = _phase(case, near, rows, d[p:e], D[p:e], q[p:e])
        c, s = torch.cos(ph), torch.sin(ph)
        ga += G[p:e].real @ c - G[p:e].imag @ s
        w = -a[None] * (G[p:e].real[:, None] * s + G[p:e].imag[:, None] * c)  # dL/dphase of every pair
        gp += w.sum(0)
        if near:  # grad phase = k (z - (d - r) / |d - r|)
            wl = k * w / dist
            gr += r * wl.sum(0)[:, None] - wl.T @ d[p:e]
            gr[:, 2] += k * w.sum(0)
        else:
            gr -= w.T @ q[p:e]
    return [gr, gp] + ([ga] if amp is not None else [])


def _exact_time(case, seed):
    rows, times = _time_inputs(case, seed)
    rows, times = torch.from_numpy(rows).cuda(), torch.from_numpy(times).cuda()
    tau = case["tau"]
    d = _pixels(case)
    _, q = _q(case, d)
    k = _wavenumber(case)
    out = torch.empty(d.shape[0], device="cuda", dtype=torch.float64)
    for p, e in _blocks(d.shape[0], rows.shape[0]):
        path = q[p:e] @ rows[:, :3].T
        t, order = torch.sort(times[None] - path / (k * _LIGHT), dim=1)
        ph = (rows[:, 3][None] - path).gather(1, order)
        # x after every arrival: sum of the amplitudes, each decayed since its own arrival
        mid = t.mean(1, keepdim=True)
        grow, decay = torch.exp((t - mid) / tau), torch.exp((mid - t) / tau)
        x2 = (decay * torch.cumsum(torch.cos(ph) * grow, 1)) ** 2 + (decay * torch.cumsum(torch.sin(ph) * grow, 1)) ** 2
        rest = -torch.expm1(-2 * torch.diff(t, dim=1) / tau)
        out[p:e] = tau / 2 * ((x2[:, :-1] * rest).sum(1) + x2[:, -1])
    return out.reshape(case["nx"], case["ny"])


def _fastlen(x):
    """The smallest length from x on with no prime factor above 11."""
    while True:
        m = x
        for f in (2, 3, 5, 7, 11):
            while m % f == 0:
                m //= f
        if m == 1:
            return x
        x += 1


def _exact_autocorr(x):
    nx, ny = x.shape[-2:]
    full = torch.fft.irfftn(torch.fft.rfftn(x.to(torch.float64), s=[_fastlen(2 * nx), _fastlen(2 * ny)],
                                            dim=(-2, -1)).abs().square(), dim=(-2, -1))
    i = (torch.arange(2 * nx, device="cuda") - nx) % full.shape[-2]
    j = (torch.arange(2 * ny, device="cuda") - ny) % full.shape[-1]
    return full[:, i][:, :, j]


def exact(case, seed):
    kind = case["kind"]
    if kind in ("fields", "double"):
        rows, amps = _images(case, seed)
        if case["settings"] == "nf double":
            return None  # this mode follows the rounding of |d - r| - d_z, about 5e-7 rad a pair
        return torch.stack([_exact_field(case, case["settings"], r, None if amps is None else amps[i])
                            for i, r in enumerate(rows)])
    if kind == "plan":
        counts, rows, amps = _plan_images(case, seed)
        parts = torch.split(amps, [int(c) for c in counts])
        return torch.stack([_exact_field(case, "nf", r, a).abs().square() for r, a in zip(rows, parts)])
    if kind == "fit":
        return _exact_fit(case, seed)
    if kind == "time":
        return _exact_time(case, seed)
    if kind == "autocorr":
        return _exact_autocorr(prepare(case, seed)["x"])
    return None  # detector: random draws; radial: bins of FP32 arithmetic
