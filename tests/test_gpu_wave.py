"""Multi-step launches against one launch pair per step: same records and images, bit for bit.

Grids around the split's edges (fewer rows than CTAs take, one column group, strips wider than a CTA), all engines,
boundaries, source mechanisms, conditions and accumulations; the step-by-step path is held to the oracle elsewhere.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _case(nz, nx, engine, nt, boundary, mechanism="explosive", seed=0):
    from ertm_b200.types import ElasticModel, GridSpec, ReceiverSpec, SourceSpec
    rng = np.random.default_rng(seed)
    h = 10.0
    vp = (2000.0 + 40.0 * (np.arange(nz)[:, None] % 30) + 20.0 * rng.standard_normal((nz, nx))).astype(np.float32)
    qp = np.where(np.arange(nz)[:, None] < nz // 2, 40.0, 90.0).repeat(nx, 1).astype(np.float32)
    model = ElasticModel(grid=GridSpec(nx=nx, nz=nz, dx=h, dz=h), vp=vp, vs=(vp / 1.8).astype(np.float32),
                         rho=(310.0 * vp.astype(np.float64) ** 0.25).astype(np.float32), qp=qp, qs=0.5 * qp)
    src = SourceSpec(x=h * (nx // 2), z=2.0 * h, f0=20.0, delay=0.03, mechanism=mechanism)
    # on and between nodes, doubled, and outside the grid
    x = np.concatenate([rng.uniform(0.0, (nx - 1) * h, 23), [0.0, 0.0, (nx - 1) * h, h * 3.5, h * 3.5, -9e3]])
    z = np.concatenate([rng.uniform(0.0, (nz - 1) * h, 23), [0.0, 0.0, (nz - 1) * h, 2.0, 2.0, 0.0]])
    return model, src, ReceiverSpec(x=x, z=z, component="p"), 8e-4, nt, boundary


def _both(fn):
    """fn() without and with multi-step launches."""
    from ertm_b200 import _lib
    L = _lib.lib()
    out = []
    try:
        for mode in (1, 2):
            _lib.check(L.ertm_set_wave(mode), "set_wave")
            before = L.ertm_launch_count()
            out.append(fn())
            out.append(L.ertm_launch_count() - before)
    finally:
        _lib.check(L.ertm_set_wave(0), "set_wave")
    assert out[3] < out[1], "the multi-step path was not taken"
    return out[0], out[2]


_GRIDS = [(8, 8), (17, 9), (33, 70), (48, 64), (61, 203), (201, 301), (420, 411)]


@pytest.mark.parametrize("shape", _GRIDS)
@pytest.mark.parametrize("engine,boundary,mechanism", [
    ("acoustic", "cpml", "explosive"), ("acoustic", "free", "explosive"), ("acoustic", "none", "explosive"),
    ("elastic", "cpml", "shear"), ("elastic", "free", "force_z"), ("viscoacoustic", "cpml", "explosive")])
def test_forward_equals_single_steps(shape, engine, boundary, mechanism):
    from ertm_b200.propagation import PropagationSpec, QOptions, build_propagator, run_forward
    model, src, rec, dt, nt, boundary = _case(*shape, engine, 61, boundary, mechanism)
    spec = PropagationSpec(dt=dt, nt=nt, npml=12, boundary=boundary)
    names = {"acoustic": ("p", "vx", "sxz", "vz"), "elastic": ("p", "vx", "vz", "sxz", "szz"),
             "viscoacoustic": ("p", "vz")}[engine]

    def run():
        prop = build_propagator(model, spec, engine=engine, q_options=QOptions(enabled=True, f_ref=20.0))
        data = run_forward(model, src, rec, spec, engine=engine, components=names, propagator=prop)
        state = prop.state()
        # a second call goes on from the state
        more = run_forward(model, src, rec, spec, engine=engine, components=names[:1], propagator=prop)
        return data, state, more

    a, b = _both(run)
    for x, y in zip(a, b):
        for k in x:
            assert np.array_equal(x[k], y[k]), k


@pytest.mark.parametrize("shape", [(17, 19), (48, 64), (201, 301), (420, 411)])
@pytest.mark.parametrize("engine,boundary,condition,separation,modes,accum", [
    ("acoustic", "cpml", "zero_lag", "stress", ("pp",), "fp64"),
    ("acoustic", "free", "excitation", "stress", ("pp",), "fp64"),
    ("elastic", "free", "normalized", "divcurl", ("pp", "ps"), "fp64"),
    ("elastic", "cpml", "normalized", "stress", ("sp", "ss"), "kahan"),
    ("elastic", "free", "excitation", "divcurl", ("pp", "ps"), "fp64"),
    ("viscoacoustic", "cpml", "normalized", "stress", ("pp",), "fp64"),
    ("viscoacoustic", "cpml", "excitation", "stress", ("pp",), "fp64")])
def test_migrate_equals_single_steps(shape, engine, boundary, condition, separation, modes, accum):
    from ertm_b200 import ImagingConfig, QConfig, RTMImager, SolverConfig
    from ertm_b200.types import ShotRecord
    model, src, rec, dt, nt, boundary = _case(*shape, engine, 90, boundary)
    rng = np.random.default_rng(5)
    comps = ("p", "vx", "vz", "sxz") if engine == "elastic" else ("p",)
    data = {c: (1e-2 * rng.standard_normal((nt, rec.nrec))).astype(np.float32) for c in comps}
    shot = ShotRecord(data=data[comps[0]], dt=dt, t=np.arange(nt) * dt, receivers=rec, source=src, components=data)
    # the amplitude cap clips and the low-pass runs within these steps; several checkpoints
    q = QConfig(enabled=True, model="gsls", alpha_c=1.0, f_ref=20.0, f_max=40.0, amplitude_cap=1.0,
                lowpass_interval=10, n_mechanisms=3)
    state_mb = 4.0 * 5 * (shape[0] + 10) * (shape[1] + 10) / 2.0**20
    imaging = ImagingConfig(mode=modes[0], condition=condition, separation=separation,
                            checkpoint_mb=max(1.0, 4 * state_mb), receiver_normalization=accum == "kahan")
    solver = SolverConfig(nt=nt, dt=dt, order=8, boundary=boundary, engine=engine)

    def run():
        im = RTMImager(imaging, solver, q, accumulation=accum)
        return [r.image for r in im.migrate_modes(shot, model, modes=modes)]

    a, b = _both(run)
    for x, y in zip(a, b):
        assert np.array_equal(x, y)
