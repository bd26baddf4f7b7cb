"""The imaging sums of multi-step migration equal the step-by-step ones, bit for bit: numerators, source and receiver
illumination before any post-processing, with the source inside the grid and correlation from the first step.

Small grids keep the sums in shared memory.  Grids that leave no room for them keep them in global memory (float64 sums
in pairs, compensated float32 ones); those cases check that the split is of that form.
"""

import numpy as np
import pytest

from test_gpu_wave import _both, _case
from wave_split import split

pytestmark = pytest.mark.gpu

NT = 60


def _sums(shape, engine, boundary, condition, separation, modes, accum, receiver_normalization):
    """A function that migrates one shot with a fresh propagator pair and returns (num, illum, rillum)."""
    from ertm_b200 import ImagingConfig, QConfig, RTMImager, SolverConfig, _lib
    from ertm_b200.imaging import ShotMigrator
    from ertm_b200.types import ReceiverSpec, SourceSpec
    model, src, rec, dt, nt, _ = _case(*shape, engine, NT, boundary)
    src = SourceSpec(x=src.x, z=10.0 * (shape[0] // 2), f0=src.f0, delay=src.delay)
    # a well through the source, so that both wavefields meet within the run
    rec = ReceiverSpec(x=np.concatenate([rec.x, np.full(shape[0], src.x)]),
                       z=np.concatenate([rec.z, 10.0 * np.arange(shape[0])]), component="p")
    rng = np.random.default_rng(11)
    names = ("p", "vz", "vx", "sxz") if engine == "elastic" else ("p",)
    record = (1e-2 * rng.standard_normal((len(names), nt, rec.nrec))).astype(np.float32)
    q = QConfig(enabled=True, model="gsls", alpha_c=1.0, f_ref=20.0, f_max=40.0, amplitude_cap=1.0,
                lowpass_interval=10, n_mechanisms=3) if engine == "viscoacoustic" else None
    state_mb = 4.0 * 5 * (shape[0] + 10) * (shape[1] + 10) / 2.0**20
    imager = RTMImager(ImagingConfig(mode=modes[0], condition=condition, separation=separation,
                                     checkpoint_mb=max(1.0, 4 * state_mb),
                                     receiver_normalization=receiver_normalization, start_periods=0.0),
                       SolverConfig(nt=nt, dt=dt, order=8, boundary=boundary, engine=engine), q, accumulation=accum)

    def run():
        from ertm_b200.propagation import source_wavelet
        mig = ShotMigrator(imager, model)
        w = source_wavelet(src, dt, nt)
        pairs, store, start = mig._prepare(src, rec, modes, nt)
        cfg = mig._config(pairs, names, store, start, nt)
        acc = np.zeros((3, len(modes), *shape))
        _lib.check(_lib.lib().ertm_migrate(mig.prop.handle, mig.back.handle, cfg, _lib.ptr(w), _lib.ptr(record),
                                           _lib.ptr(acc[0]), _lib.ptr(acc[1]), _lib.ptr(acc[2])), "migrate")
        return acc

    return run


def _check(run, condition, receiver_normalization):
    a, b = _both(run)
    assert a[0].any() and (condition != "normalized" or a[1].any()) and (not receiver_normalization or a[2].any())
    assert np.array_equal(a, b)


@pytest.mark.parametrize("shape", [(8, 9), (17, 19), (48, 64), (201, 301), (330, 400), (420, 411)])
@pytest.mark.parametrize("engine,boundary,condition,separation,modes,accum", [
    ("acoustic", "cpml", "zero_lag", "stress", ("pp",), "fp64"),
    ("acoustic", "free", "normalized", "stress", ("pp",), "kahan"),
    ("acoustic", "none", "excitation", "stress", ("pp",), "fp64"),
    ("elastic", "free", "normalized", "divcurl", ("pp", "ps"), "fp64"),
    ("elastic", "cpml", "normalized", "stress", ("sp", "ss"), "kahan"),
    ("elastic", "free", "excitation", "divcurl", ("pp", "ps"), "fp64"),
    ("viscoacoustic", "cpml", "normalized", "stress", ("pp",), "fp64"),
    ("viscoacoustic", "free", "zero_lag", "stress", ("pp",), "kahan"),
    ("viscoacoustic", "cpml", "excitation", "stress", ("pp",), "fp64")])
@pytest.mark.parametrize("receiver_normalization", [False, True])
def test_sums_equal_single_steps(shape, engine, boundary, condition, separation, modes, accum,
                                 receiver_normalization):
    _check(_sums(shape, engine, boundary, condition, separation, modes, accum, receiver_normalization), condition,
           receiver_normalization)


@pytest.mark.parametrize("shape,engine,boundary,separation,modes", [
    ((600, 700), "elastic", "free", "divcurl", ("pp", "ps")), ((620, 641), "elastic", "cpml", "stress", ("sp", "ss")),
    ((600, 1000), "acoustic", "cpml", "stress", ("pp",)), ((500, 900), "viscoacoustic", "cpml", "stress", ("pp",))])
@pytest.mark.parametrize("accum", ["fp64", "kahan"])
@pytest.mark.parametrize("receiver_normalization", [False, True])
def test_sums_in_global_memory_equal_single_steps(shape, engine, boundary, separation, modes, accum,
                                                  receiver_normalization):
    import torch
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    # illumination of one source wave, and of every image its sum and its receiver's
    sums = 1 + len(modes) * (2 if receiver_normalization else 1)
    plan = split(engine, *shape, boundary=boundary, ctas=sms, n_epi=(2 if engine == "elastic" else 0), n_src=1,
                 n_acc=sums)
    assert plan is not None and plan.sums == 0, "the grid is meant to leave no room for the sums"
    _check(_sums(shape, engine, boundary, "normalized", separation, modes, accum, receiver_normalization),
           "normalized", receiver_normalization)
