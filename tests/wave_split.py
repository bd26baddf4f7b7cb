"""The splits of multi-step launches, computed on the host from csrc/wave_plan.h (compiled with g++ on first use)."""

from __future__ import annotations

import ctypes as C
import functools
import subprocess
import tempfile
from dataclasses import dataclass
from pathlib import Path

import numpy as np

CSRC = Path(__file__).resolve().parents[1] / "challenge-cup_b200" / "csrc"

_SHIM = r"""
#include <cstring>
#include <utility>
#include "wave_plan.h"
using namespace ertm;
extern "C" int wave_split(const int* g, int ncta, const int* n, int* out, int16_t* cut, int16_t* key, int n_points,
                          const int* rows, const int* cols, int* first, int* order) {
  const WaveGrid h{g[0] != 0, g[1] != 0, g[2], g[3], g[4], g[5], g[6], g[7], g[8]};
  const WavePlan p = make_wave_plan(h, ncta, {n[0], n[1], n[2]});
  if (!p.ok()) return 0;
  const int vals[] = {p.px, p.pz, p.cells, p.n_acc, p.smem};
  std::memcpy(out, vals, sizeof(vals));
  std::copy(p.cut.begin(), p.cut.end(), cut);
  const WaveKey k = wave_key(p);
  std::copy(k.begin(), k.end(), key);
  const WaveGroups q = wave_groups(h, p, n_points, [&](int i) { return std::make_pair(rows[i], cols[i]); });
  std::copy(q.first.begin(), q.first.end(), first);
  std::copy(q.order.begin(), q.order.end(), order);
  return (int)k.size();
}
extern "C" int wave_takes(int nt, int64_t corners, int64_t most, int injected) {
  return wave_long(nt) && wave_samples(corners, most) && wave_injects(injected);
}
extern "C" int wave_few_shots(int visco, int64_t cells, int together) {
  return wave_small(cells) && wave_few(visco != 0, together);
}
"""


@functools.cache
def _shim() -> C.CDLL:
    with tempfile.TemporaryDirectory() as d:
        src, so = Path(d) / "split.cpp", Path(d) / "split.so"
        src.write_text(_SHIM)
        subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", f"-I{CSRC}", "-o", str(so), str(src)],
                       check=True)
        return C.CDLL(str(so))


@dataclass
class Split:
    px: int
    pz: int
    cells: int
    sums: int            # imaging sums in shared memory
    smem: int
    rows: np.ndarray     # row cuts
    groups: np.ndarray   # column-group cuts
    key: tuple
    first: np.ndarray    # the points grouped by CTA
    order: np.ndarray


def split(engine: str, nz: int, nx: int, *, npml: int = 20, boundary: str = "cpml", mechanisms: int = 3,
          ctas: int = 148, n_epi: int = 0, n_src: int = 0, n_acc: int = 0, points=None) -> Split | None:
    """The split of an nz × nx model over `ctas` SMs; `points`: (rows, columns) of padded cells to group."""
    pad = 5
    nzp, nxp = nz + 2 * pad, nx + 2 * pad
    # strip widths as numerics.cpml_profile and the propagator set them
    wx, wz = (0, 0) if boundary == "none" else (max(1, min(npml, nxp // 3)), max(1, min(npml, nzp // 3)))
    top = 0 if boundary == "free" else wz
    grid = (C.c_int * 9)(engine == "elastic", engine == "viscoacoustic", mechanisms if engine == "viscoacoustic" else 0,
                         nzp, nxp, wx, wx, top, wz)
    rows, cols = (np.zeros(0, np.int32),) * 2 if points is None else (np.ascontiguousarray(p, np.int32) for p in points)
    out, cut, key = (C.c_int * 5)(), (C.c_int16 * 512)(), (C.c_int16 * 512)()
    first, order = np.zeros(257, np.int32), np.zeros(max(1, rows.size), np.int32)
    as_int = lambda a: a.ctypes.data_as(C.POINTER(C.c_int))
    k = _shim().wave_split(grid, ctas, (C.c_int * 3)(n_epi, n_src, n_acc), out, cut, key, int(rows.size), as_int(rows),
                           as_int(cols), as_int(first), as_int(order))
    if k == 0:
        return None
    px, pz = out[0], out[1]
    cuts = np.array(cut[: px + pz + 2])
    return Split(px, pz, out[2], out[3], out[4], cuts[: pz + 1], cuts[pz + 1:], tuple(key[:k]),
                 first[: px * pz + 1], order[: rows.size])


def few_shots(engine: str, nz: int, nx: int, together: int) -> bool:
    """Whether small shots of a batch or session take multi-step launches, so many of their engine in flight."""
    return bool(_shim().wave_few_shots(int(engine == "viscoacoustic"), C.c_int64((nz + 10) * (nx + 10)), together))


def takes(nt: int = 1000, *, corners: int = 0, most: int = 0, injected: int = 0) -> bool:
    """Whether modelling or migration of so many steps, receiver corners and values injected into a cell takes
    multi-step launches."""
    return bool(_shim().wave_takes(nt, C.c_int64(corners), C.c_int64(most), injected))
