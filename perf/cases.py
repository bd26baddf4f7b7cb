"""What is timed: the calls that a user of the migration path makes, over the sizes it is used at.

A case is a plain dict.  ``kind`` names the call:

  forward   ``run_forward`` with a propagator that the program keeps (modelling a survey on one model)
  migrate   ``RTMImager.migrate`` of one shot record (host record in, host image out)
  batch     ``BatchMigrator.migrate_shots``: the shots of one model in one call
  device    ``migrate_device_items``: records and images stay on the GPU; shots may differ in engine and grid
  serve     ``RTMServer``: a burst of migration jobs, every result waited for
  post      ``postprocess_image``: normalisation, Laplacian, wavenumber low-pass and mask of one image
  record    ``prepare_shot`` (resampling, mute, taper) and the data-domain Q compensation of one record
  stack     ``stack_arrays``: the per-shot-normalised stack of a survey

Sizes are those of ``ertm_b200/workloads.py`` (the benchmark's configurations: 301x201, 401x601, 2001x801, the
uneven grids 501x301 ... 2401x1201, serving grids from 256x256), with shorter time axes where the whole record
would take seconds; a step costs the same at any time.
"""

from __future__ import annotations

import math
import os
import sys

import numpy as np
import torch

_PACKAGE = os.path.join(os.getcwd(), "challenge-cup_b200")
if _PACKAGE not in sys.path:
    sys.path.insert(0, _PACKAGE)

from ertm_b200 import imaging, preprocess, propagation, qcomp, serving, stacking  # noqa: E402
from ertm_b200.batch import BatchMigrator, DeviceShot, migrate_device_items  # noqa: E402
from ertm_b200.config import ImagingConfig, QConfig, SolverConfig  # noqa: E402
from ertm_b200.types import ElasticModel, GridSpec, ReceiverSpec, ShotRecord, SourceSpec  # noqa: E402

C8 = (1225.0 / 1024.0, -245.0 / 3072.0, 49.0 / 5120.0, -5.0 / 7168.0)
UNEVEN = ((501, 301), (1001, 501), (1601, 801), (2401, 1201))
ENGINES = ("acoustic", "elastic", "viscoacoustic")


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def _wave(kind, engine, nx, nz, nt, **more):
    case = {"kind": kind, "engine": engine, "nx": nx, "nz": nz, "nt": nt, "h": 5.0, "shots": 1, "every": 2,
            "boundary": "free" if engine == "elastic" else "cpml", "condition": "normalized",
            "modes": "pp,ps" if engine == "elastic" else "pp", "separation": "divcurl", "accumulation": "fp64",
            "checkpoint_mb": 256.0, "f0": 25.0}
    case.update(more)
    return case


def listed():
    return [
        # modelling one shot of the smallest configuration: latency of a time step, every receiver at every step
        {"name": "forward_acoustic", **_wave("forward", "acoustic", 301, 201, 1500, h=10.0, f0=15.0)},
        # modelling the borehole configuration's four components, free surface
        {"name": "forward_elastic_4c", **_wave("forward", "elastic", 401, 601, 1000, every=4)},
        # one shot of the CPU demo configuration: zero-lag image, 64 MB of checkpoints
        {"name": "migrate_acoustic",
         **_wave("migrate", "acoustic", 301, 201, 1500, h=10.0, f0=15.0, condition="zero_lag", checkpoint_mb=64.0)},
        # one shot of the borehole configuration: PP and PS images from one pass
        {"name": "migrate_elastic_4c", **_wave("migrate", "elastic", 401, 601, 800, every=4)},
        # one Q-compensated shot on an odd mid-size grid, as a serving job brings it
        {"name": "migrate_visco_mid", **_wave("migrate", "viscoacoustic", 777, 413, 700, h=7.0)},
        # the borehole survey's eight shots in one call
        {"name": "batch_elastic_4c", **_wave("batch", "elastic", 401, 601, 500, every=4, shots=8)},
        # shots of mixed engine and grid, float32 compensated sums, on the GPU throughout
        {"name": "device_uneven", **_wave("device", "mixed", 0, 0, 360, h=10.0, shots=6, accumulation="kahan", f0=20.0)},
        # the Q-compensated survey at full grid size, four shots of it
        {"name": "device_visco_large", **_wave("device", "viscoacoustic", 2001, 801, 420, every=5, shots=4, f0=30.0)},
        # a burst of small jobs of every engine through the serving loop
        {"name": "serve_burst", **_wave("serve", "mixed", 400, 330, 600, every=4, shots=6, f0=20.0)},
        # post-processing of one migrated image at the large survey's size
        {"name": "post_image", "kind": "post", "nx": 2001, "nz": 801, "h": 5.0},
        # record preparation ahead of migration: 400 traces at 1 ms to the propagation step, then Q compensation
        {"name": "record_prepare", "kind": "record", "nrec": 400, "nt": 1601, "dt_in": 1.0e-3, "dt_out": 0.34e-3},
        # stacking the images of a survey
        {"name": "stack_survey", "kind": "stack", "nx": 2001, "nz": 801, "shots": 16},
    ]


def _between(rng, lo, hi):
    """A whole number, uniform in its logarithm."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("forward", "forward", "migrate", "migrate", "migrate", "batch", "device", "serve", "post",
                       "record", "stack"))
    if kind == "post":
        return {"kind": kind, "nx": _between(rng, 150, 2001), "nz": _between(rng, 120, 801),
                "h": float(rng.randint(5, 10))}
    if kind == "record":
        return {"kind": kind, "nrec": _between(rng, 50, 400), "nt": _between(rng, 400, 1601), "dt_in": 1.0e-3,
                "dt_out": rng.choice((0.34e-3, 0.5e-3, 0.75e-3))}
    if kind == "stack":
        return {"kind": kind, "nx": _between(rng, 200, 2001), "nz": _between(rng, 150, 801),
                "shots": rng.randint(2, 16)}
    engine = rng.choice(ENGINES)
    more = {"h": float(rng.randint(5, 10)), "f0": rng.uniform(10.0, 30.0), "every": rng.choice((2, 4, 5))}
    if engine == "elastic":
        more["separation"] = rng.choice(("divcurl", "stress"))
        more["modes"] = rng.choice(("pp,ps", "pp"))
    if engine != "viscoacoustic":
        more["boundary"] = rng.choice(("free", "cpml"))
    if kind != "forward":
        more["condition"] = rng.choice(("normalized", "normalized", "zero_lag", "excitation"))
        more["checkpoint_mb"] = rng.choice((64.0, 256.0))
        more["accumulation"] = rng.choice(("fp64", "fp64", "kahan"))
    if kind == "device" and rng.random() < 0.5:
        return _wave("device", "mixed", 0, 0, rng.randint(200, 360), **{**more, "shots": rng.randint(2, 6),
                                                                        "boundary": "cpml", "modes": "pp"})
    if kind == "serve":
        return _wave("serve", "mixed", _between(rng, 256, 400), _between(rng, 256, 330), rng.randint(300, 600),
                     **{**more, "shots": rng.randint(3, 6), "boundary": "cpml", "modes": "pp"})
    nx, nz = _between(rng, 150, 1601), _between(rng, 120, 801)
    shots = {"batch": rng.randint(2, 8), "device": rng.randint(2, 4)}.get(kind, 1)
    # bounded by the largest listed case (4 shots of 2001x801, 420 steps)
    nt = int(min(rng.randint(400, 1500), max(150, 1.2e9 / (nx * nz * shots))))
    return _wave(kind, engine, nx, nz, nt, **{**more, "shots": shots})


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _model(rng, nx, nz, h):
    """Layers with a fast or slow body, Gardner density, layered Q."""
    n = int(rng.integers(4, 9))
    tops = np.sort(rng.uniform(0.08, 0.95, n - 1)) * nz * h
    vps = np.sort(rng.uniform(1800.0, 4200.0, n))
    qs = np.round(np.exp(rng.uniform(np.log(30.0), np.log(200.0), n)))
    layer = np.searchsorted(tops, np.arange(nz) * h)
    vp = vps[layer][:, None].repeat(nx, 1)
    cx, cz = rng.uniform(0.3, 0.7) * nx, rng.uniform(0.4, 0.8) * nz
    ax, az = rng.uniform(0.05, 0.15) * nx + 1, rng.uniform(0.03, 0.08) * nz + 1
    zz, xx = np.mgrid[0:nz, 0:nx]
    body = ((xx - cx) / ax) ** 2 + ((zz - cz) / az) ** 2 <= 1.0
    vp = np.where(body, vp * (1.12 if rng.uniform() < 0.5 else 0.88), vp).astype(np.float32)
    rho = (310.0 * vp.astype(np.float64) ** 0.25).astype(np.float32)
    qp = qs[layer][:, None].repeat(nx, 1).astype(np.float32)
    return ElasticModel(grid=GridSpec(nx=nx, nz=nz, dx=h, dz=h), vp=vp, vs=(vp / 1.8).astype(np.float32), rho=rho,
                        qp=qp, qs=(0.5 * qp).astype(np.float32))


def _dt(model):
    """The time step at half of the stability limit's bound."""
    c = sum(abs(v) for v in C8)
    return float(0.5 / (float(model.vp.max()) * math.hypot(c / model.grid.dx, c / model.grid.dz)))


def _traces(rng, nt, dt, f0, delay, offset):
    """A gather: a direct wave and four reflections with moveout under weak noise."""
    t = np.arange(nt)[:, None] * dt
    out = 1.0e-4 * rng.standard_normal((nt, offset.size))
    for k in range(5):
        t0 = 0.0 if k == 0 else rng.uniform(0.15, 0.9) * nt * dt
        arrival = delay + np.sqrt(t0 * t0 + (offset / rng.uniform(1800.0, 3500.0)) ** 2)
        a = (np.pi * f0 * (t - arrival[None, :])) ** 2
        out += rng.uniform(0.2, 1.0) * rng.choice((-1.0, 1.0)) * 10.0 ** -k * (1.0 - 2.0 * a) * np.exp(-a)
    return (1.0e-2 * out).astype(np.float32)


def _components(engine, kind):
    if engine == "elastic":
        return ("p", "vx", "vz", "sxz") if kind in ("forward", "migrate") else ("vz", "p")
    return ("p",)


def _survey(rng, case, engine, nx, nz, shots):
    """A model and the shots on it: (model, dt, sources, receivers, records)."""
    h, nt, f0 = case["h"], case["nt"], case["f0"]
    model = _model(rng, nx, nz, h)
    dt = _dt(model)
    xr = np.arange(0, nx, case["every"]) * h
    receivers = ReceiverSpec(x=xr, z=np.full_like(xr, 2.0 * h), component="p")
    sources = [SourceSpec(x=float(rng.uniform(0.1, 0.9) * (nx - 1) * h), z=2.0 * h, f0=f0, delay=1.2 / f0)
               for _ in range(shots)]
    records = []
    if case["kind"] != "forward":
        for s in sources:
            data = {c: _traces(rng, nt, dt, f0, s.delay, np.abs(xr - s.x)) for c in _components(engine, case["kind"])}
            records.append(data)
    return model, dt, sources, receivers, records


def _imager(case, engine, dt):
    solver = SolverConfig(nt=case["nt"], dt=dt, order=8, boundary=_boundary(case, engine), engine=engine)
    modes = _modes(case, engine)
    config = ImagingConfig(mode=modes[0], condition=case["condition"], separation=case["separation"],
                           checkpoint_mb=case["checkpoint_mb"])
    q = None
    if engine == "viscoacoustic":
        q = QConfig(enabled=True, model="gsls", alpha_c=1.0, f_ref=case["f0"], gain_budget_db=40.0,
                    f_max=2.0 * case["f0"], amplitude_cap=50.0, lowpass_interval=20, n_mechanisms=3)
    return imaging.RTMImager(config, solver, q, accumulation=case["accumulation"])


def _boundary(case, engine):
    if case["engine"] == "mixed":
        return "free" if engine == "elastic" else "cpml"
    return case["boundary"]


def _modes(case, engine):
    if case["engine"] == "mixed":
        return ("pp", "ps") if engine == "elastic" else ("pp",)
    return tuple(case["modes"].split(","))


def _shot(data, dt, nt, receivers, source):
    first = next(iter(data.values()))
    return ShotRecord(data=first, dt=dt, t=np.arange(nt) * dt, receivers=receivers, source=source, components=data)


def _parts(case, seed):
    """The surveys of a case: (engine, survey) each; a mixed case has several models."""
    rng = np.random.default_rng([7, seed])
    if case["engine"] != "mixed":
        return [(case["engine"], _survey(rng, case, case["engine"], case["nx"], case["nz"], case["shots"]))]
    parts = []
    for k in range(case["shots"]):
        if case["kind"] == "serve":
            engine, shots = ENGINES[k % 3], 1 + k % 2
            nx, nz = case["nx"] - 29 * (k % 5), case["nz"] - 13 * (k % 6)
        else:
            engine, shots = ENGINES[k % 2], 1
            nx, nz = UNEVEN[(0, 0, 1, 1, 2, 3)[k % 6]]
        parts.append((engine, _survey(rng, case, engine, nx, nz, shots)))
    return parts


def _image_terms(case, seed):
    rng = np.random.default_rng([11, seed])
    nz, nx = case["nz"], case["nx"]
    depth = np.arange(nz)[:, None] / nz
    illum = np.exp(-4.0 * depth) * (1.0 + 0.1 * rng.standard_normal((nz, nx)) ** 2) + 1.0e-6
    num = illum * rng.standard_normal((nz, nx)) * 0.1
    return num, illum


def _record_shot(case, seed):
    rng = np.random.default_rng([13, seed])
    xr = np.linspace(0.0, 12.5 * case["nrec"], case["nrec"])
    source = SourceSpec(x=float(rng.uniform(0.1, 0.9) * xr[-1]), z=10.0, f0=30.0, delay=0.06)
    data = _traces(rng, case["nt"], case["dt_in"], 30.0, source.delay, np.abs(xr - source.x))
    receivers = ReceiverSpec(x=xr, z=np.full_like(xr, 2.0), component="p")
    return _shot({"p": data}, case["dt_in"], case["nt"], receivers, source)


def _stack_images(case, seed):
    rng = np.random.default_rng([17, seed])
    return [(rng.standard_normal((case["nz"], case["nx"]), dtype=np.float32) * np.float32(rng.uniform(0.1, 10.0)))
            for _ in range(case["shots"])]


def prepare(case, seed):
    kind = case["kind"]
    if kind == "post":
        return {"case": case, "terms": _image_terms(case, seed)}
    if kind == "record":
        q = qcomp.QCompensator(QConfig(enabled=True, alpha_c=0.8, f_ref=30.0), q_value=80.0)
        return {"case": case, "shot": _record_shot(case, seed), "q": q}
    if kind == "stack":
        return {"case": case, "images": _stack_images(case, seed)}
    parts = _parts(case, seed)
    engine, (model, dt, sources, receivers, records) = parts[0]
    if kind == "forward":
        q = propagation.QOptions(enabled=True, f_ref=case["f0"]) if engine == "viscoacoustic" else None
        spec = propagation.PropagationSpec(dt=dt, nt=case["nt"], npml=20, boundary=case["boundary"])
        prop = propagation.build_propagator(model, spec, engine=engine, q_options=q)
        return {"case": case, "model": model, "source": sources[0], "receivers": receivers, "spec": spec, "prop": prop,
                "names": _components(engine, kind)}
    if kind in ("migrate", "batch"):
        shots = [_shot(d, dt, case["nt"], receivers, s) for d, s in zip(records, sources)]
        imager = _imager(case, engine, dt)
        return {"case": case, "model": model, "shots": shots, "imager": imager, "batch": BatchMigrator(imager),
                "modes": _modes(case, engine)}
    if kind == "device":
        items = []
        for engine, (model, dt, sources, receivers, records) in parts:
            imager = _imager(case, engine, dt)
            for s, d in zip(sources, records):
                rec = torch.from_numpy(np.stack(list(d.values()))).cuda()
                items.append(DeviceShot(imaging.ShotMigrator(imager, model), s, receivers, rec, list(d),
                                        propagation.source_wavelet(s, dt, case["nt"]), _modes(case, engine)))
        return {"case": case, "items": items}
    jobs = []
    for k, (engine, (model, dt, sources, receivers, records)) in enumerate(parts):
        shots = [_shot(d, dt, case["nt"], receivers, s) for d, s in zip(records, sources)]
        jobs.append(serving.ServeJob(shots=shots, model=model, imager=_imager(case, engine, dt),
                                     modes=_modes(case, engine), name=f"job {k}"))
    return {"case": case, "jobs": jobs, "server": serving.RTMServer().start()}


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "forward":
        state["prop"].reset()
        return propagation.run_forward(state["model"], state["source"], state["receivers"], state["spec"],
                                       engine=case["engine"], components=state["names"], propagator=state["prop"])
    if kind == "migrate":
        results = state["imager"].migrate_modes(state["shots"][0], state["model"], modes=state["modes"])
        return [r.image for r in results]
    if kind == "batch":
        results = state["batch"].migrate_shots(state["shots"], state["model"], modes=state["modes"])
        return [[r.image for r in shot] for shot in results]
    if kind == "device":
        return migrate_device_items(state["items"])
    if kind == "serve":
        futures = [state["server"].submit(job) for job in state["jobs"]]
        return [[r.image for r in f.result().images] for f in futures]
    if kind == "post":
        num, illum = state["terms"]
        return imaging.postprocess_image(num, illum, None, dx=case["h"], dz=case["h"], by_illum=True, by_rillum=False,
                                         eps=1.0e-10, laplacian=True, lowpass_fraction=0.85, npml=20, boundary="cpml")
    if kind == "record":
        shot = preprocess.prepare_shot(state["shot"], model=None, record_dt=case["dt_out"], v_reference=1500.0)
        return {"prepared": shot.components["p"], "compensated": state["q"](shot.components["p"], shot.dt)}
    return stacking.stack_arrays(state["images"])


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
# arithmetic of a cell and step: 12 per derivative (8 taps and the division), and the updates
_CELL_FLOPS = {"acoustic": 56, "elastic": 122, "viscoacoustic": 74}
_MATERIALS = {"acoustic": 2, "elastic": 3, "viscoacoustic": 3}


def _fft2_flops(nx, nz):
    return 2 * 5.0 * nx * nz * (math.log2(nx) + math.log2(nz))


def _post_work(nx, nz, bytes_per_pixel):
    return {"bytes": float(bytes_per_pixel * nx * nz), "flops": 20.0 * nx * nz + _fft2_flops(nx, nz)}


def work(case):
    kind = case["kind"]
    if kind == "post":
        return _post_work(case["nx"], case["nz"], 8 + 8 + 4)
    if kind == "record":
        n_out = int((case["nt"] - 1) * case["dt_in"] / case["dt_out"] + 1e-9) + 1
        samples = n_out * case["nrec"]
        return {"bytes": 4.0 * case["nt"] * case["nrec"] + (4.0 + 8.0) * samples,
                "flops": samples * (32.0 + 8.0 + 2 * (2 * 5.0 * 7.0 / 2.0 + 6.0 + 4.0))}
    if kind == "stack":
        return {"bytes": 4.0 * case["nx"] * case["nz"] * (case["shots"] + 1),
                "flops": 3.0 * case["nx"] * case["nz"] * case["shots"]}
    if case["engine"] != "mixed":
        surveys = [(case["engine"], case["nx"], case["nz"], case["shots"])]
    elif kind == "serve":
        surveys = [(ENGINES[k % 3], case["nx"] - 29 * (k % 5), case["nz"] - 13 * (k % 6), 1 + k % 2)
                   for k in range(case["shots"])]
    else:
        surveys = [(ENGINES[k % 2], *UNEVEN[(0, 0, 1, 1, 2, 3)[k % 6]], 1) for k in range(case["shots"])]
    total = {"bytes": 0.0, "flops": 0.0}
    for engine, nx, nz, shots in surveys:
        cells, nt = nx * nz, case["nt"]
        record = 4.0 * nt * math.ceil(nx / case["every"]) * len(_components(engine, kind))
        total["bytes"] += 4.0 * _MATERIALS[engine] * cells
        if kind == "forward":
            total["bytes"] += record
            total["flops"] += float(_CELL_FLOPS[engine]) * cells * nt
            continue
        images = len(_modes(case, engine))
        # forward, recomputed forward and backward propagation; two products and sums per image and step
        flops = (3.0 * _CELL_FLOPS[engine] + 4.0 * images) * cells * nt + images * _post_work(nx, nz, 0)["flops"]
        if engine == "viscoacoustic":
            flops += 2.0 * _fft2_flops(nx, nz) * (nt // 20)
        total["flops"] += shots * flops
        total["bytes"] += shots * record + 4.0 * cells * images * (1 if kind == "serve" else shots)
    return total


# ---------------------------------------------------------------------------
# the same results in 64 bits
# ---------------------------------------------------------------------------
class _Exact:
    """Staggered-grid propagation of ``shots`` sources on one model in float64: acoustic or elastic, 8th order, CFS
    absorbing strips (memory variables over the whole grid), free surface."""

    PAD = 5

    def __init__(self, model, dt, boundary, engine, npml, sources):
        self.engine, self.dt, self.boundary, self.h = engine, dt, boundary, float(model.grid.dx)
        self.nz, self.nx = model.grid.shape
        p = self.PAD

        def pad(a):
            return torch.from_numpy(np.pad(a.astype(np.float64), p, mode="edge")).cuda()

        vp, vs, rho = pad(model.vp), pad(model.vs), pad(model.rho)
        self.shape = tuple(vp.shape)
        inv = 1.0 / rho
        self.irx, self.irz = self._face(inv, 1), self._face(inv, 0)
        mu = rho * vs * vs
        self.lam2mu = rho * vp * vp
        self.lam = self.lam2mu - 2.0 * mu
        self.mu = self._face(self._face(mu, 1), 0)
        names = ("p", "vx", "vz") if engine == "acoustic" else ("vx", "vz", "sxx", "szz", "sxz")
        self.f = {n: torch.zeros((len(sources),) + self.shape, dtype=torch.float64, device="cuda") for n in names}
        self.psi = {}
        vmax = float(model.vp.max())
        self.strip = {1: self._strips(self.shape[1], npml, vmax, (True, True)),
                      0: self._strips(self.shape[0], npml, vmax, (boundary != "free", True))}
        at = [(min(max(round(s.z / self.h), 0), self.nz - 1) + p, min(max(round(s.x / self.h), 0), self.nx - 1) + p)
              for s in sources]
        self.at = (torch.arange(len(at), device="cuda"), torch.tensor([a[0] for a in at], device="cuda"),
                   torch.tensor([a[1] for a in at], device="cuda"))

    @staticmethod
    def _face(a, axis):
        out = a.clone()
        if axis == 1:
            out[:, :-1] = 0.5 * (a[:, :-1] + a[:, 1:])
        else:
            out[:-1] = 0.5 * (a[:-1] + a[1:])
        return out

    def _strips(self, length, npml, vmax, sides):
        n = max(1, min(npml, length // 3))
        sigma, alpha = np.zeros(length), np.zeros(length)
        d = (n - np.arange(n)) / n
        top = 3.0 * vmax * math.log(1.0e5) / (2.0 * n * self.h)
        if sides[0]:
            sigma[:n], alpha[:n] = top * d * d, 50.0 * math.pi * (1.0 - d)
        if sides[1]:
            sigma[length - n:], alpha[length - n:] = (top * d * d)[::-1], (50.0 * math.pi * (1.0 - d))[::-1]
        b = np.exp(-(sigma + alpha) * self.dt)
        s = sigma + alpha
        a = np.where(s > 0, sigma / np.where(s > 0, s, 1.0) * (b - 1.0), 0.0)
        return torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda()

    def _raw(self, f, axis, forward):
        n = f.shape[1 + axis]
        out = torch.zeros_like(f)
        m = n - 8
        acc = 0.0
        for k, c in enumerate(C8, 1):
            hi, lo = (4 + k, 5 - k) if forward else (3 + k, 4 - k)
            acc = acc + c * (f.narrow(1 + axis, hi, m) - f.narrow(1 + axis, lo, m))
        out.narrow(1 + axis, 4, m).copy_(acc / self.h)
        return out

    def _d(self, name, f, axis, forward):
        raw = self._raw(f, axis, forward)
        a, b = self.strip[axis]
        a, b = (a[None, None, :], b[None, None, :]) if axis == 1 else (a[None, :, None], b[None, :, None])
        psi = self.psi.setdefault(name, torch.zeros_like(raw))
        # outside the strips a is zero and the memory with it
        psi.mul_(b).addcmul_(a.expand_as(raw), raw)
        return raw + psi

    def step(self, amp):
        f, dt = self.f, self.dt
        if self.engine == "acoustic":
            f["vx"] += dt * self.irx * self._d("a", f["p"], 1, True)
            f["vz"] += dt * self.irz * self._d("b", f["p"], 0, True)
            f["p"] += dt * self.lam2mu * (self._d("c", f["vx"], 1, False) + self._d("d", f["vz"], 0, False))
            if amp is not None:
                f["p"][self.at] += amp
            if self.boundary == "free":
                f["p"][:, self.PAD] = 0.0
            return
        f["vx"] += dt * self.irx * (self._d("a", f["sxx"], 1, True) + self._d("b", f["sxz"], 0, False))
        f["vz"] += dt * self.irz * (self._d("c", f["sxz"], 1, False) + self._d("d", f["szz"], 0, True))
        exx, ezz = self._d("e", f["vx"], 1, False), self._d("f", f["vz"], 0, False)
        f["sxx"] += dt * (self.lam2mu * exx + self.lam * ezz)
        f["szz"] += dt * (self.lam * exx + self.lam2mu * ezz)
        f["sxz"] += dt * self.mu * (self._d("g", f["vx"], 0, True) + self._d("h", f["vz"], 1, True))
        if amp is not None:
            f["sxx"][self.at] += amp
            f["szz"][self.at] += amp
        if self.boundary == "free":
            f["szz"][:, self.PAD] = 0.0
            f["sxz"][:, self.PAD] = 0.0

    def state(self):
        return {k: v.clone() for k, v in self.f.items()}, {k: v.clone() for k, v in self.psi.items()}

    def load(self, state):
        for mine, kept in zip((self.f, self.psi), state):
            for k, v in kept.items():
                mine[k].copy_(v)

    def corners(self, receivers, name):
        """Bilinear weights of the receivers on a component's grid."""
        xo = -0.5 if name in ("vx", "sxz") else 0.0
        zo = -0.5 if name in ("vz", "sxz") else 0.0
        x = np.asarray(receivers.x) / self.h + self.PAD + xo
        z = np.asarray(receivers.z) / self.h + self.PAD + zo
        x0, z0 = np.floor(x).astype(np.int64), np.floor(z).astype(np.int64)
        tx, tz = x - x0, z - z0
        at, w = [], []
        for dz in (0, 1):
            for dx in (0, 1):
                at.append((z0 + dz) * self.shape[1] + x0 + dx)
                w.append((tz if dz else 1.0 - tz) * (tx if dx else 1.0 - tx))
        return torch.from_numpy(np.stack(at)).cuda(), torch.from_numpy(np.stack(w)).cuda()

    def sample(self, name, corners):
        at, w = corners
        f = 0.5 * (self.f["sxx"] + self.f["szz"]) if self.engine == "elastic" and name == "p" else self.f[name]
        return (f.reshape(f.shape[0], -1)[:, at] * w).sum(1)

    def inject(self, name, corners, values):
        at, w = corners
        for n in (("sxx", "szz") if self.engine == "elastic" and name == "p" else (name,)):
            f = self.f[n].reshape(len(values), -1)
            f.index_add_(1, at.reshape(-1), (values[:, None, :] * w).reshape(len(values), -1))

    def image(self, separation):
        f = self.f
        if self.engine == "acoustic":
            out = {"P": f["p"]}
        elif separation == "stress":
            out = {"P": 0.5 * (f["sxx"] + f["szz"]), "S": f["sxz"]}
        else:
            out = {"P": self._raw(f["vx"], 1, False) + self._raw(f["vz"], 0, False),
                   "S": self._raw(f["vx"], 0, False) - self._raw(f["vz"], 1, False)}
        p = self.PAD
        return {k: v[:, p: p + self.nz, p: p + self.nx] for k, v in out.items()}


def _exact_forward(case, engine, survey):
    model, dt, sources, receivers, _ = survey
    wave = propagation_wavelet(sources[0], dt, case["nt"])
    prop = _Exact(model, dt, case["boundary"], engine, 20, sources)
    names = _components(engine, "forward")
    corners = {n: prop.corners(receivers, n) for n in names}
    out = {n: torch.zeros((case["nt"], len(receivers.x)), dtype=torch.float64, device="cuda") for n in names}
    for t in range(case["nt"]):
        prop.step(wave[t])
        for n in names:
            out[n][t] = prop.sample(n, corners[n])[0]
    return {n: v.cpu().numpy() for n, v in out.items()}


def propagation_wavelet(source, dt, nt):
    """The Ricker wavelet of a source, in float64."""
    a = (math.pi * source.f0 * (torch.arange(nt, dtype=torch.float64, device="cuda") * dt - source.delay)) ** 2
    return (1.0 - 2.0 * a) * torch.exp(-a)


def _exact_post(num, illum, h, by_illum, npml, boundary):
    """Illumination, Laplacian, wavenumber low-pass and mask of an image, float64 on the GPU."""
    nz, nx = num.shape
    v = num / (illum + 1.0e-10) if by_illum else num
    a = torch.nn.functional.pad(v[None, None], (1, 1, 1, 1), mode="replicate")[0, 0]
    c = a[1:-1, 1:-1]
    v = (a[1:-1, 2:] - 2.0 * c + a[1:-1, :-2] + a[2:, 1:-1] - 2.0 * c + a[:-2, 1:-1]) / (h * h)
    kz = torch.fft.fftfreq(nz, d=0.5, dtype=torch.float64, device="cuda")
    kx = torch.fft.fftfreq(nx, d=0.5, dtype=torch.float64, device="cuda")
    taper = (1.0 - (torch.sqrt(kz[:, None] ** 2 + kx[None, :] ** 2) - 0.85) / 0.15).clamp(0.0, 1.0)
    v = torch.fft.ifft2(torch.fft.fft2(v) * taper).real
    v[:, :npml] = 0.0
    v[:, -npml:] = 0.0
    v[-npml:] = 0.0
    if boundary == "cpml":
        v[:npml] = 0.0
    return v


def _exact_images(case, engine, survey):
    """Images of every shot of a survey: tensor (shots, modes, nz, nx)."""
    model, dt, sources, receivers, records = survey
    nt, boundary = case["nt"], _boundary(case, engine)
    nz, nx = model.grid.shape
    npml = min(20, max(8, min(nx, nz) // 8))
    modes = _modes(case, engine)
    wave = propagation_wavelet(sources[0], dt, nt)
    fwd = _Exact(model, dt, boundary, engine, npml, sources)
    back = _Exact(model, dt, boundary, engine, npml, sources)
    per_state = 4 * len(fwd.f) * fwd.shape[0] * fwd.shape[1]
    interval = max(1, math.ceil(nt / max(1, int(case["checkpoint_mb"] * 1024 ** 2 // per_state))))
    kept = {}
    for t in range(nt):
        fwd.step(wave[t])
        if t % interval == 0:
            kept[t] = fwd.state()
    start = int(np.clip(math.floor((sources[0].delay + 1.5 / sources[0].f0) / dt), 0, nt))
    names = list(records[0])
    rec = {n: torch.from_numpy(np.stack([r[n] for r in records]).astype(np.float64)).cuda() for n in names}
    corners = {n: back.corners(receivers, n) for n in names}
    num = torch.zeros((len(sources), len(modes), nz, nx), dtype=torch.float64, device="cuda")
    illum = torch.zeros_like(num)
    for s in sorted(kept, reverse=True):
        # the state after step s runs step s again: the recomputation's own convention
        fwd.load(kept.pop(s))
        end = min(s + interval, nt)
        fields = []
        for t in range(s, end):
            fwd.step(wave[t])
            fields.append(fwd.image(case["separation"])["P"].clone())
        for t in range(end - 1, s - 1, -1):
            for n in names:
                back.inject(n, corners[n], rec[n][:, t])
            back.step(None)
            got = back.image(case["separation"])
            src = fields[t - s]
            for k, m in enumerate(modes):
                illum[:, k] += src * src
                if t >= start:
                    num[:, k] += src * got[m[1].upper()]
    by_illum = case["condition"] == "normalized"
    out = torch.empty_like(num)
    for b in range(len(sources)):
        for k in range(len(modes)):
            out[b, k] = _exact_post(num[b, k], illum[b, k], case["h"], by_illum, npml, boundary)
    return out


def _exact_record(case, shot):
    data = shot.data.astype(np.float64)
    dt_in, dt = case["dt_in"], case["dt_out"]
    n_in = data.shape[0]
    n = int(math.floor((n_in - 1) * dt_in / dt + 1e-9)) + 1
    pos = np.arange(n) * (dt / dt_in)
    at = np.floor(pos).astype(np.int64)[:, None] + np.arange(-7, 9)[None, :]
    w = np.sinc(pos[:, None] - at) * np.kaiser(16, 8.6)[None, :]
    w /= w.sum(1, keepdims=True)
    v = sum(w[:, k:k + 1] * data[np.clip(at[:, k], 0, n_in - 1)] for k in range(16))
    t, f0 = np.arange(n) * dt, shot.source.f0
    mute = shot.source.delay + 1.2 / f0 + 1.05 * np.abs(shot.receivers.x - shot.source.x) / 1500.0
    ramp = np.clip((t[:, None] - (mute - 0.5 / f0)) * f0, 0.0, 1.0)
    v = v * (0.5 - 0.5 * np.cos(np.pi * ramp))
    k = max(int(0.05 * n), 1)
    taper = 0.5 - 0.5 * np.cos(np.pi * (np.arange(k) + 0.5) / k)
    v[:k] *= taper[:, None]
    v[n - k:] *= taper[::-1, None]
    # inverse-Q gain and phase over half-overlapping Hann frames of 128 samples
    x = v.astype(np.float32).astype(np.float64)
    length, hop = 128, 64
    win, f = np.hanning(length), np.fft.rfftfreq(length, d=dt)
    out, norm = np.zeros_like(x), np.zeros(n)
    for s in range(0, n, hop):
        m = min(length, n - s)
        if m < 4:
            continue
        frame = np.zeros((length, x.shape[1]))
        frame[:m] = x[s:s + m]
        travel = max((s + 0.5 * length) * dt, 1e-6)
        g = f * 0.8 * travel / 80.0
        fc = max(0.5 / dt * (0.95 - 0.35 * min(travel / 0.5, 1.0)), 60.0)
        h = np.minimum(np.exp(np.pi * g), 30.0) / (1.0 + (f / fc) ** 4)
        h = h * np.exp(2j * g * np.log(np.maximum(f, 1e-9) / 30.0))
        y = np.fft.irfft(np.fft.rfft(frame * win[:, None], axis=0) * h[:, None], n=length, axis=0)
        out[s:s + m] += y[:m] * win[:m, None]
        norm[s:s + m] += win[:m] ** 2
    return {"prepared": v, "compensated": out / np.where(norm > 1e-12, norm, 1.0)[:, None]}


def exact(case, seed):
    kind = case["kind"]
    if kind == "post":
        num, illum = (torch.from_numpy(a).cuda() for a in _image_terms(case, seed))
        return _exact_post(num, illum, case["h"], True, 20, "cpml").cpu().numpy()
    if kind == "record":
        return _exact_record(case, _record_shot(case, seed))
    if kind == "stack":
        return sum(im.astype(np.float64) / float(np.abs(im).max()) for im in _stack_images(case, seed)) / case["shots"]
    # the relaxation times of the viscoacoustic engine come from a least-squares fit that belongs to the package, and
    # the excitation condition's peak step is decided by rounding: neither has a value of its own in 64 bits
    if case["engine"] == "viscoacoustic" or (kind != "forward" and case["condition"] == "excitation"):
        return None
    # three propagations of every shot in float64 at about 1 ms a step and 0.6 M cells
    parts = _parts(case, seed)
    if kind == "forward":
        return _exact_forward(case, *parts[0])
    cells = sum(s[0].grid.nx * s[0].grid.nz * len(s[2]) for e, s in parts if e != "viscoacoustic")
    if case["nt"] * (0.4e-3 * len(parts) + 1.5e-9 * cells) * 3 > 20.0:
        return None
    out = []
    for engine, survey in parts:
        if engine == "viscoacoustic":
            out.append([None] * len(_modes(case, engine)) if kind == "serve" else None)
            continue
        images = _exact_images(case, engine, survey)
        if kind == "serve":
            if len(images) > 1:
                images = images / images.abs().amax((2, 3), keepdim=True)
            out.append(list(images.mean(0).cpu().numpy()))
        else:
            out.extend(images.cpu().numpy())
    if kind == "migrate":
        return list(out[0])
    return [list(v) if v is not None else None for v in out] if kind == "batch" else out
