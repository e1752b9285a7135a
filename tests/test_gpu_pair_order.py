"""With cutoffs, the pair passes' sums do not depend on what else is in the
engine: an untuned engine of few tiles takes them tile pair by tile pair
(k_born_pair, k_force_pair, k_collect; k_near64 with a block per tile pair), one
of many tiles with eight i-tiles per CTA (k_born, k_force; k_near64 with a warp
per tile pair), in the same order.  Forces and Born radii have to be equal bit
for bit, from one tile to more tiles than a work item holds."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import host_golden
from test_gpu_sasa import cluster_topology

pytestmark = pytest.mark.gpu

SEQ = "NLYIQWLKDGGPSSGRPPPSARNDCQEGHILKMFPSTWYV" * 3


def _target(origami, what):
    """(topology or chain, coordinates)"""
    rng = np.random.default_rng(11)
    if isinstance(what, int):
        chain = origami.Chain.build(SEQ[:what])
        return chain, chain.positions + rng.normal(scale=0.05, size=chain.positions.shape)
    names = what.split("+")
    seq, chains, counts, atoms, el, xyz = "", "", [], [], [], []
    for k, n in enumerate(names):
        g = host_golden()[n]
        seq += str(g["seq"])
        chains += "".join(chr(ord(c) + 2 * k) for c in str(g["chains"]))
        counts += [int(c) for c in g["counts"]]
        atoms += [str(a) for a in g["names"]]
        el.append(g["elements"])
        xyz.append(np.asarray(g["xyz"]) - np.asarray(g["xyz"]).mean(0) + np.array([32.0 * k, 0.0, 0.0]))
    x = np.concatenate(xyz)
    chain = origami.Chain.from_structure(seq, counts, atoms, x, elements=np.concatenate(el), chains=chains)
    return chain, x + rng.normal(scale=0.01, size=x.shape)


def _line(origami, n):
    """n uncharged atoms 3 A apart on a line: many tiles, few pairs."""
    x = np.zeros((n, 3))
    x[:, 0] = 3.0 * np.arange(n)
    return cluster_topology(origami, np.ones(n, np.int32)), x


def _evaluate(origami, systems, params):
    eng = origami.Engine(params)
    for topo, x in systems:
        eng.add_system(topo, x, 310.0)
    eng.finalize()
    f, r = eng.total_force(0), eng.born_radii(0)
    eng.close()
    return f, r


@pytest.mark.parametrize("cut", [(10.0, 20.0, 10.0), (6.0, 9.0, 8.0)])
@pytest.mark.parametrize("what", [1, 2, 4, 20, 60, 120, "1L2Y", "2HIU", "2HIU+2HIU+1L2Y"])
def test_results_do_not_depend_on_the_rest_of_the_engine(origami, what, cut):
    target = _target(origami, what)
    p = origami.Params(nb_cutoff=cut[0], born_cutoff=cut[1], gb_force_cutoff=cut[2])
    alone = _evaluate(origami, [target], p)
    # 2 500 tiles in a row: 3.1 million tile pairs, 2 500 in the near field
    batch = _evaluate(origami, [target, _line(origami, 80000)], p)
    assert np.isfinite(alone[0]).all()
    np.testing.assert_array_equal(alone[0], batch[0])
    np.testing.assert_array_equal(alone[1], batch[1])
