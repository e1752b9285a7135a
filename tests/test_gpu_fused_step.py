"""The fused sub-steps (one kernel without constraints; clusters in warp lanes
with SHAKE) against the general launches, which an engine takes for all its
systems when one of them has a cluster that does not fit a warp.  Both keep
the reference's arithmetic order, and the forces differ in the fixed-point
rounding only, so five steps agree to 1e-9 A and 1e-9 A/fs; also the SHAKE
failure count when constraints cannot be met."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _star(origami, n):
    """A heavy atom with n hydrogens at 1.1 A: n constraints in one cluster."""
    from test_gpu_sasa import cluster_topology
    t = cluster_topology(origami, [1] + [0] * n)
    k = np.arange(n) + 0.5
    phi, th = np.arccos(1.0 - 2.0 * k / n), np.pi * (1.0 + 5 ** 0.5) * k
    x = np.concatenate([np.zeros((1, 3)), 1.1 * np.stack([np.cos(th) * np.sin(phi), np.sin(th) * np.sin(phi), np.cos(phi)], 1)])
    t.mass[1:] = 1.008
    t.constraints = np.stack([np.zeros(n, np.int32), np.arange(1, n + 1, dtype=np.int32)], 1)
    t.constraint_length = np.full(n, 1.1)
    return t, x


def _run(origami, systems, steps=5, **kw):
    eng = origami.Engine(origami.Params.all_pairs(constrain_h_bonds=True, dt_fs=2.0, friction_ps_inv=2.0, seed=3, **kw))
    for topo, x in systems:
        eng.add_system(topo, x, 310.0)
    eng.finalize()
    for k in range(len(systems)):
        eng.init_velocities(k, 17 + k, remove_com=False)
    eng.step(steps, check=False)
    out = [(eng.positions(k), eng.velocities(k), eng.stats(k)) for k in range(len(systems))]
    eng.close()
    return out


@pytest.mark.parametrize("seqs", [("G",), ("AGAGA",), ("ARNDCQEGHILKMFPSTWYV",), ("MKTAYIAK", "GG", "ARNDCQEGHILKMFPSTWYV" * 2)])
def test_fused_step_equals_the_general_launches(origami, seqs):
    chains = [origami.Chain.build(s) for s in seqs]
    systems = [(c, c.positions) for c in chains]
    fused = _run(origami, systems)
    general = _run(origami, systems + [_star(origami, 33)])  # 34 atoms of one cluster do not fit a warp
    for (xa, va, sa), (xb, vb, sb) in zip(fused, general):
        assert np.max(np.abs(xa - xb)) < 1e-9 and np.max(np.abs(va - vb)) < 1e-9
        assert sa == sb


@pytest.mark.parametrize("n", [1, 4, 31])
def test_clusters_up_to_a_warp_keep_their_lengths(origami, n):
    topo, x = _star(origami, n)
    (xa, _, s), = _run(origami, [(topo, x)], steps=20, shake_max_iters=500)
    assert s["shake_failures"] == 0 and s["steps"] == 20
    # the tolerance is on squared lengths
    assert np.max(np.abs(((xa[1:] - xa[0]) ** 2).sum(1) - 1.21)) < 1e-6


def test_failed_constraints_are_counted_per_half_step(origami):
    ch = origami.Chain.build("AGAGA")
    (_, _, s), (_, _, general), _ = _run(origami, [(ch, ch.positions)] * 2 + [_star(origami, 33)], steps=4, shake_max_iters=1)
    (_, _, fused), = _run(origami, [(ch, ch.positions)], steps=4, shake_max_iters=1)
    assert s["shake_failures"] == fused["shake_failures"] == 8
