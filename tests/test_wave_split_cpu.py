"""Splits of multi-step launches on the host: which cells a CTA owns, and when tables of one split serve another."""

from __future__ import annotations

import itertools

import numpy as np
import pytest

from wave_split import few_shots, split, takes

# what a work keeps in shared memory beside the fields: (P/S fields, stored source fields, imaging sums)
_NEEDS = {"acoustic": [(0, 0, 0), (0, 1, 1), (0, 1, 2), (0, 1, 3)],
          "viscoacoustic": [(0, 0, 0), (0, 1, 1), (0, 1, 2), (0, 1, 3)],
          "elastic": [(0, 0, 0), (1, 0, 0), (2, 0, 0), (1, 1, 1), (1, 1, 2), (1, 1, 3), (2, 1, 2), (2, 1, 3), (2, 2, 4),
                      (2, 2, 6)]}
_GRIDS = [(201, 301), (301, 501), (330, 400), (360, 401), (400, 751), (413, 777), (420, 411), (500, 601), (601, 401)]


@pytest.mark.parametrize("engine", sorted(_NEEDS))
@pytest.mark.parametrize("boundary", ["free", "cpml"])
def test_splits_with_equal_keys_own_the_same_cells(engine, boundary):
    """A kept propagator's injection tables are looked up by the split's key: a call with other imaging settings
    must not find the tables of a split with other cuts."""
    for nz, nx in _GRIDS:
        plans = [split(engine, nz, nx, boundary=boundary, ctas=c, n_epi=e, n_src=s, n_acc=a)
                 for c in (148, 74) for e, s, a in _NEEDS[engine]]
        for a, b in itertools.combinations([p for p in plans if p], 2):
            if a.key == b.key:
                assert np.array_equal(a.rows, b.rows) and np.array_equal(a.groups, b.groups), (nz, nx, a, b)


@pytest.mark.parametrize("engine", sorted(_NEEDS))
def test_grouped_points_lie_in_their_tile(engine):
    """Every padded cell belongs to one CTA, and a CTA's points lie in its rows and columns."""
    for (nz, nx), (e, s, a) in itertools.product(_GRIDS[:5] + [(8, 8), (17, 9)], _NEEDS[engine]):
        rows, cols = (p.ravel() for p in np.indices((nz + 10, nx + 10)))
        p = split(engine, nz, nx, boundary="cpml", n_epi=e, n_src=s, n_acc=a, points=(rows, cols))
        if p is None:
            continue
        assert p.rows[0] == 0 and p.rows[-1] == nz + 10 and np.diff(p.rows).min() >= 4
        assert p.groups[0] == 0 and p.groups[-1] == (nx + 13) // 4 and np.diff(p.groups).min() >= 1
        assert np.array_equal(np.sort(p.order), np.arange(rows.size))
        cta = np.repeat(np.arange(p.px * p.pz), np.diff(p.first))
        i, g = rows[p.order], cols[p.order] // 4
        tr, tc = cta // p.px, cta % p.px
        assert (p.rows[tr] <= i).all() and (i < p.rows[tr + 1]).all()
        assert (p.groups[tc] <= g).all() and (g < p.groups[tc + 1]).all()


@pytest.mark.parametrize("engine", sorted(_NEEDS))
def test_many_shots_share_ticks(engine):
    """A batch or a loaded server advances its shots in common ticks; one or two small shots run alone."""
    for nz, nx in ((256, 256), (330, 400)):
        assert all(few_shots(engine, nz, nx, n) for n in (1, 2))
        assert not any(few_shots(engine, nz, nx, n) for n in (4, 8, 45))


def test_short_runs_and_dense_receivers_go_step_by_step():
    """Calls that multi-step launches would slow down keep one launch pair per step."""
    assert takes() and takes(8) and takes(corners=4 * 4 * 151, most=600, injected=12)
    assert not any(takes(nt) for nt in (1, 2, 5))
    assert not takes(corners=4 * 60000) and not takes(corners=100000, most=18000)
    assert takes(injected=40) and not takes(injected=80)
