"""The surface term's edge cases through both of its kernels.  An engine of few
surface atoms gives all of them to the large-capacity kernel; beside 1 300 lone
atoms the same clusters go through the default kernel, which hands what exceeds
its capacities (112 caps, 56 live circles, 64 transitions of a batch, 24 arcs, a
tangent pair) to the large one.  Forces within 1e-6 kJ/mol/A of the FP64 oracle,
areas within 1e-9 of 4 pi R^2, the tolerances of the other surface tests."""
from __future__ import annotations

import math

import numpy as np
import pytest

from conftest import ch2_tangent_cluster, dp, host_golden, oracle
from test_gpu_sasa import cluster_topology, dense_shell_cluster, fibonacci_directions
from test_gpu_sasa_cover import _cluster

pytestmark = pytest.mark.gpu


def _cap_distance(ri, rj, angle):
    """Distance at which an atom of radius rj has a cap of that half angle on one of radius ri."""
    c = math.cos(angle)
    return c * ri + math.sqrt((c * ri) ** 2 - (ri * ri - rj * rj))


def _spread_caps(n, degrees, most_z):
    """A sulfur under hydrogens in n evenly spread directions with z < most_z, caps of `degrees`."""
    o = oracle()
    dirs = fibonacci_directions(n)
    dirs = dirs[dirs[:, 2] < most_z]
    d = _cap_distance(o.orc_sasa_radius(5), o.orc_sasa_radius(0), math.radians(degrees))
    return np.vstack([np.zeros(3), dirs * d]), np.array([5] + [0] * len(dirs), dtype=np.int32)


def _rim(n):
    """A sulfur with a carbon's cap of 60 degrees and n hydrogens' caps of 4 degrees along its rim, all apart from each
    other: 2 n transitions on one circle."""
    o = oracle()
    rs, rc, rh = (o.orc_sasa_radius(k) for k in (5, 1, 0))
    phi = 2 * np.pi * (np.arange(n) + 0.3) / n
    tilt = math.radians(60.0)
    ring = np.stack([np.sin(tilt) * np.cos(phi), np.sin(tilt) * np.sin(phi), np.full(n, np.cos(tilt))], 1)
    x = np.vstack([np.zeros(3), [[0.0, 0.0, _cap_distance(rs, rc, tilt)]], ring * _cap_distance(rs, rh, math.radians(4.0))])
    x[2:] += np.random.default_rng(9).normal(scale=0.01, size=(n, 3))
    return x, np.array([5, 1] + [0] * n, dtype=np.int32)


def _fold(copies):
    """Insulins side by side, each turned: a compact fold whose atoms meet their neighbours'."""
    g = host_golden()["2HIU"]
    x0 = np.asarray(g["xyz"], dtype=np.float64)
    x0 = x0 - x0.mean(0)
    rng = np.random.default_rng(6)
    xs = []
    for k in range(copies):
        q = np.linalg.qr(rng.normal(size=(3, 3)))[0]
        xs.append(x0 @ q + np.array([27.0 * k, 0.0, 0.0]))
    x = np.concatenate(xs)
    return x + rng.normal(scale=0.01, size=x.shape), np.tile(np.asarray(g["elements"], dtype=np.int32), copies)


CASES = {
    "140 caps": lambda: dense_shell_cluster(5, 140),
    "69 live circles": lambda: _spread_caps(75, 20.0, 0.85),
    "57 live circles": lambda: _spread_caps(62, 20.0, 0.85),
    "30 whole circles": lambda: _spread_caps(30, 8.0, 2.0),
    "68 transitions on a circle": lambda: _rim(36),
    "54 transitions on a circle": lambda: _rim(28),
    "tangent pair": lambda: ch2_tangent_cluster(),
    "cluster of 30": lambda: _cluster(30, 4.0, 41),
    "cluster of 60": lambda: _cluster(60, 4.5, 42),
    "cluster of 120": lambda: _cluster(120, 5.5, 44),
    "insulin": lambda: _fold(1),
    "two insulins": lambda: _fold(2),
}


@pytest.mark.parametrize("alone", [True, False])
@pytest.mark.parametrize("case", CASES)
def test_edge_cases_match_oracle_in_either_kernel(origami, case, alone):
    x, el = CASES[case]()
    x, el = np.ascontiguousarray(x, dtype=np.float64), np.asarray(el, dtype=np.int32)
    o = oracle()
    rad = np.array([o.orc_sasa_radius(int(e)) for e in el])
    gam = np.array([o.orc_sasa_gamma(int(e), 1.0) for e in el])
    ref, area = np.zeros_like(x), np.zeros(len(x))
    o.orc_sasa_forces_tangent_one_root(len(x), dp(x), dp(rad), dp(gam), dp(ref))
    o.orc_sasa_areas(len(x), dp(x), dp(rad), dp(area))
    lone = np.zeros((1300, 3))
    lone[:, 0] = 20.0 * np.arange(1300)
    f = {}
    for on in (True, False):
        eng = origami.Engine(origami.Params(include_sasa=on))
        eng.add_system(cluster_topology(origami, el), x, 310.0)
        if not alone:
            eng.add_system(cluster_topology(origami, np.ones(1300, np.int32)), lone, 310.0)
        eng.finalize()
        f[on] = eng.total_force(0)
        got = eng.sasa_areas(0, "powersasa")
        eng.close()
    assert np.max(np.abs(f[True] - f[False] - ref)) < 1e-6
    assert np.max(np.abs(got - area) / (4 * np.pi * rad ** 2)) < 1e-9
