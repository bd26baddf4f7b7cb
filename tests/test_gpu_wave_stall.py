"""A wait inside a multi-step launch that runs out: the call fails with ERTM_ERR_STATE, the next one is as ever.

The waits are made to run out by dropping the edge values; the kernel then gives up and returns by itself.
"""

import ctypes as C
from contextlib import contextmanager

import numpy as np
import pytest

from test_gpu_wave import _case
from test_gpu_wave_kept import _images, _imager, _shot

pytestmark = pytest.mark.gpu

ERR_STATE = -3


@contextmanager
def _dropped_edges():
    from ertm_b200 import _lib
    L = _lib.lib()
    _lib.check(L.ertm_set_wave_drop(1), "set_wave_drop")
    try:
        yield
    finally:
        _lib.check(L.ertm_set_wave_drop(0), "set_wave_drop")


@pytest.mark.parametrize("engine", ["acoustic", "elastic", "viscoacoustic"])
def test_stalled_forward_fails_until_reset(engine):
    from ertm_b200 import _lib
    from ertm_b200.exceptions import SolverError
    from ertm_b200.propagation import PropagationSpec, QOptions, build_propagator, run_forward
    model, src, rec, dt, nt, _ = _case(96, 140, engine, 60, "cpml")
    spec = PropagationSpec(dt=dt, nt=nt, npml=12, boundary="cpml")
    prop = build_propagator(model, spec, engine=engine, q_options=QOptions(enabled=True, f_ref=20.0))

    def run():
        return run_forward(model, src, rec, spec, engine=engine, components=("p",), propagator=prop)["p"]

    want = run()
    prop.reset()
    with _dropped_edges():
        with pytest.raises(SolverError, match="ran out"):
            run()
        out = np.zeros((1, nt, rec.nrec), np.float32)
        comps = np.zeros(1, np.int32)
        prop.reset()
        assert _lib.lib().ertm_forward(prop.handle, nt, None, 1, comps.ctypes.data_as(C.POINTER(C.c_int32)),
                                       _lib.ptr(out)) == ERR_STATE
    assert prop.status == _lib.STATUS_STALLED and prop.finite
    with pytest.raises(SolverError, match="ran out"):   # the wavefield is not one to go on from
        run()
    prop.reset()
    assert prop.status == 0
    assert np.array_equal(run(), want)


@pytest.mark.parametrize("engine,boundary", [("elastic", "free"), ("viscoacoustic", "cpml")])
def test_stalled_migration_fails_and_the_next_is_as_ever(engine, boundary):
    from ertm_b200.batch import BatchMigrator
    from ertm_b200.exceptions import SolverError
    model, shot = _shot((96, 140), engine, boundary)
    imager = _imager(engine, boundary, shot.dt)
    batch = BatchMigrator(imager)
    want = _images(imager.migrate_modes(shot, model))
    with _dropped_edges():
        with pytest.raises(SolverError, match="ran out"):
            imager.migrate_modes(shot, model)
        with pytest.raises(SolverError, match="ran out"):
            batch.migrate_shots([shot], model)
    assert np.array_equal(_images(imager.migrate_modes(shot, model))[0], want[0])
    assert np.array_equal(_images(batch.migrate_shots([shot], model)[0])[0], want[0])


def test_stalled_shot_fails_its_job_alone():
    from ertm_b200 import _lib
    from ertm_b200.exceptions import NonFiniteWavefieldError, SolverError
    from ertm_b200.serving import RTMServer, ServeJob
    jobs = []
    for engine, boundary in (("acoustic", "free"), ("elastic", "free"), ("viscoacoustic", "cpml")):
        model, shot = _shot((96, 140), engine, boundary)
        jobs.append((_imager(engine, boundary, shot.dt), model, shot))
    want = [_images(imager.migrate_modes(shot, model))[0] for imager, model, shot in jobs]

    def drop_second(what, job, index):   # runs in the serving thread, before the shot joins the session
        if what == "prepare":
            _lib.lib().ertm_set_wave_drop(int(job == 1))

    with RTMServer(fault_hook=drop_second, ticks_per_poll=16) as server:
        futures = [server.submit(ServeJob(shots=[shot], model=model, imager=imager)) for imager, model, shot in jobs]
        with pytest.raises(SolverError, match="ran out") as failed:
            futures[1].result(timeout=120)
        assert not isinstance(failed.value, NonFiniteWavefieldError)
        for k in (0, 2):
            assert np.array_equal(futures[k].result(timeout=120).images[0].image, want[k])
        # the server goes on
        again = server.submit(ServeJob(shots=[jobs[1][2]], model=jobs[1][1], imager=jobs[1][0]))
        assert np.array_equal(again.result(timeout=120).images[0].image, want[1])
    s = server.summary()
    assert s["jobs_failed"] == 1 and s["shots_failed"] == 1 and s["jobs_done"] == 3
