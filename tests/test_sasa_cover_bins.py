"""CPU check of the surface term's buried bins (covered_bins in sasa_geom.h): a
bin counts as buried only when it lies inside the interval by the margin on both
sides, the seam of the pseudo-angle included, and every bin that lies inside by
a little more does count."""
from __future__ import annotations

import ctypes as C

import numpy as np

from test_sasa_adjoint import shim  # noqa: F401  (fixture)

BINS = 32


def _covered(lib, ts, te):
    ts, te = (np.ascontiguousarray(v, dtype=np.float32) for v in (ts, te))
    out = np.zeros(len(ts), np.uint32)
    fp = C.POINTER(C.c_float)
    lib.shim_covered_bins(C.c_int(len(ts)), ts.ctypes.data_as(fp), te.ctypes.data_as(fp),
                          out.ctypes.data_as(C.POINTER(C.c_uint32)))
    return (out[:, None] >> np.arange(BINS, dtype=np.uint32)) & 1 == 1


def test_covered_bins_keep_the_margin_on_both_sides(shim):  # noqa: F811
    lib = shim
    lib.shim_cover_margin.restype = C.c_float
    margin = float(lib.shim_cover_margin())
    near = np.array([0.0, 1e-4, 0.25, 0.5, 0.9, 0.99, 1.01, 1.1, 2.0, 3.0]) * margin
    edges = np.concatenate([[0.0], near, BINS - near, 1 + near, 1 - near, 17 + near, 17 - near, [8.5, 25.4],
                            np.random.default_rng(2).uniform(0, BINS, 60)])
    ts, te = (v.ravel().astype(np.float32) for v in np.meshgrid(edges, edges))
    use = np.abs(ts - te) > margin  # what buried_interval lets through
    ts, te = ts[use], te[use]
    got = _covered(lib, ts, te)
    b = np.arange(BINS)[None, :]
    ts, te = ts.astype(np.float64)[:, None], te.astype(np.float64)[:, None]
    length = np.where(te > ts, te - ts, te - ts + BINS)
    ahead = (b - ts) % BINS          # from the interval's start to the bin's
    inside = np.minimum(ahead, length - ahead - 1)
    # FP32 rounding of the sums near 32: 4e-6
    assert (inside[got] >= margin - 1e-5).all(), inside[got].min()
    assert got[inside >= margin + 1e-5].all()
