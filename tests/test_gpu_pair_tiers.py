"""The pair passes' distance tiers and launch shapes: chains long enough for
every series length of the Born pass and for the force pass's distant form,
with tile counts that leave partial blocks, against the FP64 oracle (forces
RMS relative < 1e-5, integrals < 1e-6 of the largest, the tolerances of the
other parity tests); and the same engine's second and third force evaluation
(captured and replayed) against its first."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import INF, Orc

pytestmark = pytest.mark.gpu

SEQ = "ARNDCQEGHILKMFPSTWYV"


def _system(origami, n_res, seed):
    ch = origami.Chain.build((SEQ * 8)[:n_res])
    x = ch.positions + np.random.default_rng(seed).normal(scale=0.03, size=(ch.n_atoms, 3))
    return ch, np.ascontiguousarray(x)


def _engine(origami, systems, cutoff):
    eng = origami.Engine(origami.Params() if cutoff else origami.Params.all_pairs())
    for ch, x in systems:
        eng.add_system(ch, x)
    return eng.finalize()


def rms_rel(a, b):
    return float(np.sqrt(((a - b) ** 2).sum() / (b ** 2).sum()))


# residues: 1, 3, 16, 17 and 33 tiles and what lies around them; the last
# spans 300 A, so that its tile pairs reach the three-term series
@pytest.mark.parametrize("cutoff", [False, True])
@pytest.mark.parametrize("n_res", [2, 6, 32, 34, 66, 85])
def test_tiers_and_shapes_match_oracle(origami, n_res, cutoff):
    systems = [_system(origami, n_res, 1), _system(origami, max(2, n_res // 3), 2)]
    cut = (10.0, 20.0, 10.0) if cutoff else (INF, INF, INF)
    refs = [(Orc(c).total_force(x, *cut), Orc(c).born_integrals(x, cut[1])) for c, x in systems]
    eng = _engine(origami, systems, cutoff)
    for shape in range(7):
        for persistent, chunk in ((False, 16), (False, 1), (True, 3)):
            eng.set_pair_launch("born", min(shape, 2), persistent, chunk)
            eng.set_pair_launch("force", shape, persistent, chunk)
            for k, (f, integral) in enumerate(refs):
                assert rms_rel(eng.total_force(k), f) < 1e-5, (shape, chunk, k)
                assert np.max(np.abs(eng.born_integrals(k) - integral)) < 1e-6 * np.max(np.abs(integral)), (shape, chunk, k)
    eng.close()


@pytest.mark.parametrize("cutoff", [False, True])
def test_replayed_evaluations_equal_the_first(origami, cutoff):
    ch, x = _system(origami, 24, 3)
    y = np.ascontiguousarray(x + np.random.default_rng(4).normal(scale=0.02, size=x.shape))
    first = {}
    for name, pos in (("x", x), ("y", y)):
        eng = _engine(origami, [(ch, pos)], cutoff)
        first[name] = eng.total_force(0)
        eng.close()
    eng = _engine(origami, [(ch, x)], cutoff)
    for name, pos in (("x", x), ("y", y), ("x", x), ("y", y)):
        eng.set_positions(0, pos)
        assert np.array_equal(eng.total_force(0), first[name])
        assert np.array_equal(eng.positions(0), pos)
    # a new launch variant, a tunnel and a grown chain each end the replay
    from origami_b200.cotranslate import CylindricalTunnel
    eng.set_pair_launch("force", 1, False, 4)
    assert rms_rel(eng.total_force(0), first["y"]) < 1e-6
    CylindricalTunnel(tuple(y.mean(0)), (0.0, 0.0, 1.0), 1.0, 500.0, 3.0).apply_to(eng)
    fresh = _engine(origami, [(ch, y)], cutoff)
    fresh.set_pair_launch("force", 1, False, 4)
    CylindricalTunnel(tuple(y.mean(0)), (0.0, 0.0, 1.0), 1.0, 500.0, 3.0).apply_to(fresh)
    want = fresh.total_force(0)
    for _ in range(3):
        assert np.array_equal(eng.total_force(0), want)
    assert rms_rel(want, first["y"]) > 1e-3
    eng.close()
    fresh.close()
