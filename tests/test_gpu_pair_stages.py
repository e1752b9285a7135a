"""The pair passes' pipelines over several stages of four j-tiles: an explicit
chunk is taken as it is, so every launch shape runs work items of 2 to 11 stages
here (refilled buffers, double-buffered j sums, the ring of tile tables, the last
stage partly filled)."""
from __future__ import annotations

import math

import numpy as np
import pytest

from conftest import INF, Orc

pytestmark = pytest.mark.gpu

SEQ = "ARNDCQEGHILKMFPSTWYV" * 5


def _system(origami, n_res, seed):
    ch = origami.Chain.build(SEQ[:n_res], math.radians(-57.0), math.radians(-47.0), math.pi)
    x = ch.positions + np.random.default_rng(seed).normal(scale=0.03, size=ch.positions.shape)
    return ch, np.ascontiguousarray(x)


def _engine(origami, systems, cutoff):
    eng = origami.Engine(origami.Params() if cutoff else origami.Params.all_pairs())
    for ch, x in systems:
        eng.add_system(ch, x, 310.0)
    eng.finalize()
    return eng


def rms_rel(a, b):
    return float(np.sqrt(((a - b) ** 2).sum() / (b ** 2).sum()))


# 50 and 42 tiles: 13 stages of a whole list; chunks of 7 (2 stages, the last
# of three tiles), 16, 21 and 42 (11 stages, the last of two)
@pytest.mark.parametrize("cutoff", [False, True])
@pytest.mark.parametrize("chunk", [7, 16, 21, 42])
def test_items_of_several_stages_match_oracle(origami, cutoff, chunk):
    systems = [_system(origami, 100, 1), _system(origami, 85, 2)]
    cut = (10.0, 20.0, 10.0) if cutoff else (INF, INF, INF)
    refs = [(Orc(c).total_force(x, *cut), Orc(c).born_integrals(x, cut[1])) for c, x in systems]
    eng = _engine(origami, systems, cutoff)
    for shape in range(7):
        got = []
        for persistent in (False, True):
            eng.set_pair_launch("born", min(shape, 2), persistent, chunk)
            eng.set_pair_launch("force", shape, persistent, chunk)
            got.append([eng.total_force(k) for k in range(2)])
            for k, (f, integral) in enumerate(refs):
                assert rms_rel(got[-1][k], f) < 1e-5, (shape, persistent, k)
                off = np.max(np.abs(eng.born_integrals(k) - integral))
                assert off < 1e-6 * np.max(np.abs(integral)), (shape, persistent, k)
        for a, b in zip(*got):
            np.testing.assert_array_equal(a, b)
    eng.close()


@pytest.mark.parametrize("cutoff", [False, True])
@pytest.mark.parametrize("shape", range(7))
def test_an_explicit_chunk_does_not_depend_on_the_engine(origami, shape, cutoff):
    """With a fixed shape and chunk a system's work items, and so its fixed-point
    sums, are its own: the same bits alone and beside 40 more."""
    target = _system(origami, 85, 3)
    f = []
    for others in (0, 40):
        eng = _engine(origami, [target] + [_system(origami, 60, 10 + k) for k in range(others)], cutoff)
        eng.set_pair_launch("born", min(shape, 2), False, 16)
        eng.set_pair_launch("force", shape, False, 16)
        f.append(eng.total_force(0))
        eng.close()
    np.testing.assert_array_equal(f[0], f[1])
