"""The step without constraints (one kernel for the sub-steps before the forces)
against the oracle's BAOAB with the engine's noise, from one atom more than a tile
to several tiles, alone and beside a system that diverges at once.  Tolerances of
the other trajectory tests (1e-6 A, 1e-5 A/fs over 5 steps); beside the diverging
system the same bits as alone."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import Orc, dp, oracle

pytestmark = pytest.mark.gpu


def _steps(origami, systems, v0, n):
    eng = origami.Engine(origami.Params(dt_fs=1.0, friction_ps_inv=2.0, seed=77))
    for ch, x in systems:
        eng.add_system(ch, x, 310.0)
    eng.finalize()
    eng.set_state({"velocities": np.concatenate(v0)})
    eng.step(n, check=False)
    out = eng.positions(0), eng.velocities(0), [eng.stats(k) for k in range(len(systems))]
    eng.close()
    return out


@pytest.mark.parametrize("seq", ["GG", "AGAG", "ARNDCQEGHILK"])
def test_free_steps_match_oracle(origami, seq):
    from test_gpu_parity import minimized
    ch = minimized(origami, seq, helical=len(seq) > 4)
    x0 = ch.positions
    rng = np.random.default_rng(8)
    v0 = rng.normal(scale=0.004, size=x0.shape)
    x, v, (s,) = _steps(origami, [(ch, x0)], [v0], 5)
    orc = Orc(ch)
    xr, vr = np.ascontiguousarray(x0.copy()), np.ascontiguousarray(v0.copy())
    f = orc.total_force(xr)
    oracle().orc_baoab(orc.tp, dp(xr), dp(vr), dp(f), 5, 1.0, 2.0, 310.0, 0, 77, 0, 0, 10.0, 20.0, 10.0)
    assert np.max(np.abs(x - xr)) < 1e-6 and np.max(np.abs(v - vr)) < 1e-5
    assert s["steps"] == 5 and not s["diverged"]
    bad = v0.copy()
    bad[0, 1] = np.inf
    xb, vb, (sa, sb) = _steps(origami, [(ch, x0), (ch, x0)], [v0, bad], 5)
    np.testing.assert_array_equal(xb, x)
    np.testing.assert_array_equal(vb, v)
    assert sa["steps"] == 5 and not sa["diverged"] and sb["diverged"]
