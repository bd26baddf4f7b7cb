"""A kept propagator pair used with one imaging setting after another: the same images as a fresh pair, bit for bit.

The settings differ in what a multi-step launch keeps in shared memory, so its split over the SMs differs between the
calls while the receivers, and with them the injection plan, stay.
"""

import itertools

import numpy as np
import pytest

from test_gpu_wave import _case

pytestmark = pytest.mark.gpu

NT = 90


def _shot(shape, engine, boundary):
    from ertm_b200.types import ReceiverSpec, ShotRecord, SourceSpec
    model, src, rec, dt, nt, _ = _case(*shape, engine, NT, boundary)
    nz, nx = shape
    # deep enough for the image to leave the absorbing strips
    src = SourceSpec(x=src.x, z=10.0 * (nz // 2), f0=src.f0, delay=src.delay, mechanism=src.mechanism)
    # every column near the surface, and a well
    x = np.concatenate([rec.x, np.arange(nx) * 10.0, np.full(nz, 10.0 * (nx // 2))])
    z = np.concatenate([rec.z, np.full(nx, 20.0), np.arange(nz) * 10.0])
    rec = ReceiverSpec(x=x, z=z, component="p")
    rng = np.random.default_rng(8)
    data = {c: (1e-2 * rng.standard_normal((nt, rec.nrec))).astype(np.float32)
            for c in (("vz", "p") if engine == "elastic" else ("p",))}
    first = next(iter(data.values()))
    return model, ShotRecord(data=first, dt=dt, t=np.arange(nt) * dt, receivers=rec, source=src, components=data)


def _imager(engine, boundary, dt, condition="normalized"):
    from ertm_b200 import ImagingConfig, QConfig, RTMImager, SolverConfig
    q = QConfig(enabled=True, model="gsls", alpha_c=1.0, f_ref=20.0, f_max=40.0, amplitude_cap=50.0,
                lowpass_interval=20, n_mechanisms=3) if engine == "viscoacoustic" else None
    return RTMImager(ImagingConfig(mode="pp", condition=condition, separation="divcurl", checkpoint_mb=64.0,
                                     start_periods=0.0),
                     SolverConfig(nt=NT, dt=dt, order=8, boundary=boundary, engine=engine), q)


def _images(results):
    assert all(r.image.any() for r in results)
    return [r.image for r in results]


@pytest.mark.parametrize("order", list(itertools.permutations([("pp",), ("pp", "ps")])))
def test_kept_migrator_with_other_modes(order):
    from ertm_b200.imaging import ShotMigrator
    model, shot = _shot((301, 501), "elastic", "free")
    imager = _imager("elastic", "free", shot.dt)
    kept = ShotMigrator(imager, model)
    for modes in order + order[:1]:
        got = _images(kept.migrate(shot, modes=modes))
        want = _images(ShotMigrator(imager, model).migrate(shot, modes=modes))
        for a, b in zip(got, want, strict=True):
            assert np.array_equal(a, b), modes


@pytest.mark.parametrize("order", list(itertools.permutations(["zero_lag", "normalized"])))
def test_kept_imager_with_another_condition(order):
    model, shot = _shot((413, 777), "viscoacoustic", "cpml")
    kept = _imager("viscoacoustic", "cpml", shot.dt)
    for condition in order + order[:1]:
        fresh = _imager("viscoacoustic", "cpml", shot.dt, condition)
        kept.config = fresh.config
        got = _images(kept.migrate_modes(shot, model))
        assert np.array_equal(got[0], _images(fresh.migrate_modes(shot, model))[0]), condition


@pytest.mark.parametrize("order", list(itertools.permutations([("pp",), ("pp", "ps")])))
def test_kept_batch_with_other_modes(order):
    from ertm_b200.batch import BatchMigrator
    model, shot = _shot((330, 400), "elastic", "cpml")
    imager = _imager("elastic", "cpml", shot.dt)
    kept = BatchMigrator(imager)
    for modes in order + order[:1]:
        got = kept.migrate_shots([shot, shot], model, modes=modes)
        want = BatchMigrator(imager).migrate_shots([shot, shot], model, modes=modes)
        for x, y in zip(got, want, strict=True):
            for a, b in zip(_images(x), _images(y), strict=True):
                assert np.array_equal(a, b), modes


def test_session_of_both_routes_gives_one_shot_images():
    """Few shots of one engine beside many of another, more of them joining: ticks and multi-step launches in one
    session."""
    from ertm_b200.serving import RTMServer, ServeJob
    jobs = []
    for engine, boundary, n in (("elastic", "free", 2), ("viscoacoustic", "cpml", 5), ("acoustic", "free", 4)):
        model, shot = _shot((96, 140), engine, boundary)
        jobs += [(_imager(engine, boundary, shot.dt), model, shot)] * n
    want = {id(model): _images(imager.migrate_modes(shot, model)) for imager, model, shot in jobs}
    with RTMServer(max_shots=7, ticks_per_poll=16) as server:
        futures = [server.submit(ServeJob(shots=[shot], model=model, imager=imager)) for imager, model, shot in jobs]
        for f, (_, model, _) in zip(futures, jobs):
            for r, b in zip(f.result(timeout=120).images, want[id(model)], strict=True):
                assert np.array_equal(r.image, b)
