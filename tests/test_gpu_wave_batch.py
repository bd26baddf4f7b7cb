"""Shots in multi-step launches beside shots in ticks: a batch and a serving session give the one-shot images."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _jobs():
    from ertm_b200.workloads import imager_for, uneven_batch
    from ertm_b200.types import ShotRecord
    rng = np.random.default_rng(3)
    out = []
    # 501x301 shots take multi-step launches, the larger grids ticks
    for wl in [w for w in uneven_batch(seed=2, n_shots=40) if w.model.grid.nx in (501, 1001)][:4]:
        wl.nt = 70
        imager, solver = imager_for(wl)
        data = {c: (1e-2 * rng.standard_normal((wl.nt, wl.receivers.nrec))).astype(np.float32) for c in wl.components}
        shot = ShotRecord(data=data[wl.components[0]], dt=wl.dt, t=np.arange(wl.nt) * wl.dt, receivers=wl.receivers,
                          source=wl.sources[0], components=data)
        out.append((wl, imager, shot))
    assert {w.model.grid.nx for w, _, _ in out} == {501, 1001}
    return out


def test_mixed_batch_and_session_equal_one_shot_images():
    from ertm_b200 import _lib
    from ertm_b200.serving import RTMServer, ServeJob
    jobs = _jobs()
    L = _lib.lib()
    try:
        _lib.check(L.ertm_set_wave(1), "set_wave")
        want = [[r.image for r in im.migrate_modes(shot, wl.model, modes=wl.modes)] for wl, im, shot in jobs]
    finally:
        _lib.check(L.ertm_set_wave(0), "set_wave")
    import torch
    from ertm_b200.batch import DeviceShot, migrate_device_items
    from ertm_b200.imaging import ShotMigrator
    from ertm_b200.propagation import source_wavelet
    items = [DeviceShot(ShotMigrator(im, wl.model), shot.source, shot.receivers,
                        torch.from_numpy(np.stack(list(shot.components.values()))).cuda(), list(shot.components),
                        source_wavelet(shot.source, wl.dt, wl.nt), wl.modes) for wl, im, shot in jobs]
    for images, ref in zip(migrate_device_items(items), want):
        for a, b in zip(images.cpu().numpy(), ref):
            assert np.array_equal(a, b)
    with RTMServer(ticks_per_poll=16) as server:
        futures = [server.submit(ServeJob(shots=[shot], model=wl.model, imager=im, modes=wl.modes))
                   for wl, im, shot in jobs]
        for f, ref in zip(futures, want):
            for r, b in zip(f.result(timeout=120).images, ref):
                assert np.array_equal(r.image, b)
