"""Learned radii: the judge's evaluation with plain radii does not take the
replayed evaluation away from the engine's own."""
from __future__ import annotations

import time

import numpy as np
import pytest

from origami_b200 import lgb
from test_gpu_lgb import random_params

pytestmark = pytest.mark.gpu


def _engine(origami, seed=3):
    ch = origami.Chain.build("NLYIQWLKDGGPSSGRPPPS")
    x = ch.positions + np.random.default_rng(seed).normal(scale=0.02, size=ch.positions.shape)
    eng = origami.Engine(origami.Params.all_pairs(born_mode=1))
    eng.add_system(ch, x, 310.0)
    eng.finalize()
    lgb.set_params(eng, random_params(origami, 4))
    lgb.set_judge(eng, 0, 1e6)  # judged by hand, always accepted
    return eng


def _best_us(engines):
    """Best time of 20 evaluations of each engine, the engines taken in turn."""
    best = [1e9] * len(engines)
    for _ in range(30):
        for k, eng in enumerate(engines):
            t = time.perf_counter()
            for _ in range(20):
                eng.total_force(0)
            best[k] = min(best[k], time.perf_counter() - t)
    return [b / 20 * 1e6 for b in best]


def test_evaluations_after_a_judgement_are_replayed(origami):
    plain, judged = _engine(origami), _engine(origami)
    want = plain.total_force(0)
    judged.step(0)     # evaluates the forces once
    lgb.judge(judged)  # before their second evaluation, which is the one captured
    for _ in range(3):
        np.testing.assert_array_equal(judged.total_force(0), want)
    a, b = _best_us([plain, judged])
    assert b < 1.2 * a, (a, b)
    lgb.judge(judged)
    lgb.judge(judged)
    np.testing.assert_array_equal(judged.total_force(0), want)
    plain.close()
    judged.close()
