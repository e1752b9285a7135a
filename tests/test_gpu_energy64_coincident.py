"""FP64 energies with two atoms in one place: every term has the value the
oracle has, the infinite and undefined ones among them (1/r is infinite, r^-12 -
2 r^-6 undefined, the GB pair finite)."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import INF, Orc

pytestmark = pytest.mark.gpu

TERMS = ("bond", "angle", "dihedral", "improper", "lj", "coulomb", "gb", "gb_self", "gb_pair", "total")


@pytest.mark.parametrize("cutoff", [False, True])
@pytest.mark.parametrize("seq,a,b", [("AGWGA", -3, 2), ("AG" * 12, 3, -4)])
def test_coincident_atoms(origami, seq, a, b, cutoff):
    ch = origami.Chain.build(seq)
    x = np.array(ch.positions) + np.random.default_rng(1).normal(scale=0.05, size=(ch.n_atoms, 3))
    x[a] = x[b]
    eng = origami.Engine(origami.Params() if cutoff else origami.Params.all_pairs())
    eng.add_system(ch, x)
    eng.finalize()
    e = eng.energies(0)
    eng.close()
    ref = Orc(ch).energy_terms(x, *((10.0, 20.0) if cutoff else (INF, INF)))
    assert np.isnan(ref["lj"]) and np.isinf(ref["coulomb"]) and np.isfinite(ref["gb"])
    for t in TERMS:
        if np.isfinite(ref[t]):
            assert abs(e[t] - ref[t]) <= 1e-10 * max(abs(ref[t]), 1.0), (t, e[t], ref[t])
        else:
            assert str(e[t]) == str(float(ref[t])), (t, e[t], ref[t])
