"""The surface term's buried bins where a decision in them is a near tie.

golden/surface_bin_limit.npz holds two neighbourhoods from insulin dynamics in
which a cap and a circle lie at the limit up to which the FP32 interval of
buried_interval (sasa.cu) is used, (1 - c_k^2)(1 - sigma^2) = 0.01 to 3e-8: x0,
x1 the positions, el0, el1 the elements.  Forces within 1e-6 kJ/mol/A of the
FP64 oracle and areas within 1e-9 of 4 pi R^2, the tolerances of the other
surface tests, in the large-capacity kernel (one system) and in the default one
(more surface atoms than go to the large-capacity kernel at once)."""
from __future__ import annotations

import os

import numpy as np
import pytest

from conftest import dp, oracle
from test_gpu_sasa import cluster_topology

pytestmark = pytest.mark.gpu

# (fixture, surface atom, circle, cap): the pair at the limit
PAIRS = [(0, 19, 45, 49), (1, 20, 39, 46)]


def _fixture(k):
    z = np.load(os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden", "surface_bin_limit.npz"))
    return z["x%d" % k], z["el%d" % k].astype(np.int32)


def _radii(el):
    return np.array([oracle().orc_sasa_radius(int(e)) for e in el])


def _limit(x, rad, i, k, m):
    """(1 - c_k^2)(1 - sigma^2) of cap m on the circle of cap k on atom i."""
    d = x[[k, m]] - x[i]
    r = np.linalg.norm(d, axis=1)
    ck = (r[0] ** 2 + rad[i] ** 2 - rad[k] ** 2) / (2 * r[0] * rad[i])
    sigma = (d[0] @ d[1]) / (r[0] * r[1])
    return (1 - ck * ck) * (1 - sigma * sigma)


def _at_limit(fixture, i, k, m, target):
    """The fixture with atom m moved across atom i's view of atom k until the pair is at `target`."""
    x, el = _fixture(fixture)
    rad = _radii(el)
    u = (x[k] - x[i]) / np.linalg.norm(x[k] - x[i])
    side = (x[m] - x[i]) - ((x[m] - x[i]) @ u) * u
    side /= np.linalg.norm(side)

    def moved(t):
        y = x.copy()
        y[m] += t * side
        return y

    lo, hi = -0.05, 0.05
    if _limit(moved(lo), rad, i, k, m) > _limit(moved(hi), rad, i, k, m):
        lo, hi = hi, lo
    for _ in range(60):
        mid = 0.5 * (lo + hi)
        lo, hi = (mid, hi) if _limit(moved(mid), rad, i, k, m) < target else (lo, mid)
    return moved(lo), el


def _check(origami, systems):
    f, area = {}, []
    for on in (True, False):
        eng = origami.Engine(origami.Params(include_sasa=on))
        for x, el in systems:
            eng.add_system(cluster_topology(origami, el), x, 310.0)
        eng.finalize()
        f[on] = [eng.total_force(s) for s in range(len(systems))]
        if not on:
            area = [eng.sasa_areas(s, "powersasa") for s in range(len(systems))]
        eng.close()
    o = oracle()
    for s, (x, el) in enumerate(systems):
        rad = _radii(el)
        gam = np.array([o.orc_sasa_gamma(int(e), 1.0) for e in el])
        ref, a = np.zeros_like(x), np.zeros(len(x))
        o.orc_sasa_forces_tangent_one_root(len(x), dp(x), dp(rad), dp(gam), dp(ref))
        o.orc_sasa_areas(len(x), dp(x), dp(rad), dp(a))
        assert np.max(np.abs(f[True][s] - f[False][s] - ref)) < 1e-6, s
        assert np.max(np.abs(area[s] - a) / (4 * np.pi * rad ** 2)) < 1e-9, s


@pytest.mark.parametrize("fixture", [0, 1])
def test_pair_at_the_interval_limit_as_recorded(origami, fixture):
    _check(origami, [_fixture(fixture)])


@pytest.mark.parametrize("fixture,i,k,m", PAIRS)
def test_pairs_across_the_interval_limit(origami, fixture, i, k, m):
    """96 copies whose pair crosses the limit in steps of 6e-9, an FP32
    rounding or so: together 1 500 C atoms or more, the default kernel."""
    systems = [_at_limit(fixture, i, k, m, 0.01 + t) for t in np.linspace(-3e-7, 3e-7, 96)]
    assert sum(int(((el == 1) | (el == 5)).sum()) for _, el in systems) > 1184
    _check(origami, systems)
