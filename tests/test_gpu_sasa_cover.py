"""The surface term where most circles are buried all around and dropped
before their transitions are built: compact folds, dense random clusters at
the edges of the mask capacity (56 live circles) and beyond it, a circle
buried by two caps that just meet, and an atom whose circles are all buried.
Forces against the FP64 oracle within 1e-6 kJ/mol/A and areas within 1e-9 of
4 pi R^2, the tolerances of the other surface tests."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import dp, host_golden, oracle
from test_gpu_sasa import cluster_topology

pytestmark = pytest.mark.gpu


def _gpu(origami, x, el):
    """(surface forces, areas) of uncharged atoms without any other term."""
    topo = cluster_topology(origami, el)
    f = {}
    for on in (True, False):
        eng = origami.Engine(origami.Params(include_sasa=on))
        eng.add_system(topo, x, 310.0)
        eng.finalize()
        f[on] = eng.total_force(0)
        area = eng.sasa_areas(0, "powersasa")
        eng.close()
    return f[True] - f[False], area


def _cluster(n, spread, seed):
    """A carbon at the origin among n atoms of random elements within
    `spread` A, at least 0.9 A from each other."""
    rng = np.random.default_rng(seed)
    x = [np.zeros(3)]
    while len(x) < n + 1:
        p = rng.uniform(-spread, spread, 3)
        if np.linalg.norm(p) <= spread and min(np.linalg.norm(p - q) for q in x) > 0.9:
            x.append(p)
    el = rng.choice([0, 0, 0, 1, 1, 2, 3], n + 1)
    el[0] = 1
    return np.array(x), el.astype(np.int32)


def _ring(gap):
    """A carbon whose cap of the carbon at +z is buried by two more carbons
    up to an opening of about `gap` radians (closed when negative)."""
    d = 2.0
    a = 0.62 - gap / 4
    return np.array([[0.0, 0.0, 0.0], [0.0, 0.0, 2.2], [d * np.sin(a), 0.01, d * np.cos(a)],
                     [-d * np.sin(a), -0.02, d * np.cos(a)]]), np.array([1, 1, 1, 1], dtype=np.int32)


CASES = ([("cluster", n, s, k) for k, (n, s) in enumerate([(8, 2.5), (30, 4.0), (60, 4.5), (90, 5.0), (120, 5.5)])]
         + [("ring", g, 0.0, 0) for g in (-0.3, -1e-3, 1e-3, 0.3)] + [("native", "1L2Y", 0, 0), ("native", "2HIU", 0, 0)])


def _system(kind, p, q, seed):
    if kind == "cluster":
        return _cluster(p, q, 40 + seed)
    if kind == "ring":
        return _ring(p)
    case = host_golden()[p]
    x = np.array(case["xyz"], dtype=np.float64)
    return x + np.random.default_rng(3).normal(scale=0.01, size=x.shape), np.asarray(case["elements"], dtype=np.int32)


@pytest.mark.parametrize("kind,p,q,seed", CASES)
def test_buried_circles_leave_forces_and_areas_as_the_oracle(origami, kind, p, q, seed):
    x, el = _system(kind, p, q, seed)
    o = oracle()
    rad = np.array([o.orc_sasa_radius(int(e)) for e in el])
    gam = np.array([o.orc_sasa_gamma(int(e), 1.0) for e in el])
    ref = np.zeros_like(x)
    o.orc_sasa_forces_tangent_one_root(x.shape[0], dp(x), dp(rad), dp(gam), dp(ref))
    force, got = _gpu(origami, x, el)
    assert np.max(np.abs(force - ref)) < 1e-6
    area = np.zeros(x.shape[0])
    o.orc_sasa_areas(x.shape[0], dp(x), dp(rad), dp(area))
    assert np.max(np.abs(got - area) / (4 * np.pi * rad ** 2)) < 1e-9


@pytest.mark.parametrize("apart", [30.0, 2000.0])
def test_neighbours_in_wide_tiles_match_oracle(origami, apart):
    """Two clusters whose atoms alternate, so that every tile spans both and
    its FP32 coordinates are coarse (1e-4 A at 2000 A): the neighbour search
    has to find each atom's own cluster all the same."""
    xa, ea = _cluster(23, 3.5, 7)
    xb, eb = _cluster(23, 3.5, 8)
    x = np.ascontiguousarray(np.stack([xa, xb + np.array([apart, 0.3 * apart, 0.0])], 1).reshape(-1, 3))
    el = np.ascontiguousarray(np.stack([ea, eb], 1).reshape(-1))
    o = oracle()
    rad = np.array([o.orc_sasa_radius(int(e)) for e in el])
    gam = np.array([o.orc_sasa_gamma(int(e), 1.0) for e in el])
    ref = np.zeros_like(x)
    o.orc_sasa_forces_tangent_one_root(x.shape[0], dp(x), dp(rad), dp(gam), dp(ref))
    force, got = _gpu(origami, x, el)
    assert np.max(np.abs(force - ref)) < 1e-6
    area = np.zeros(x.shape[0])
    o.orc_sasa_areas(x.shape[0], dp(x), dp(rad), dp(area))
    assert np.max(np.abs(got - area) / (4 * np.pi * rad ** 2)) < 1e-9
