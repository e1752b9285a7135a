"""The FP64 energy path (tile kernels, series descreening, pair halves) at the
edges of its layout: systems inside one tile, at tile boundaries, of many
tiles with more warps per tile than tiles, uneven systems in one engine, with
and without cutoffs (tile pairs skipped).  Every term against the FP64 oracle
to 1e-10 of max(|term|, 1): both sum the same FP64 pair terms in another
order (1e5 terms of magnitude up to ~1e2 at 1e-16 each)."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import INF, Orc, dp, oracle

pytestmark = pytest.mark.gpu

TERMS = ("bond", "angle", "dihedral", "improper", "lj", "coulomb", "gb", "gb_self", "gb_pair", "total")
# 1 residue (10 atoms), 32-, 33- and 64-atom neighbourhoods, several hundred to a few thousand atoms
SEQS = ["A", "GAG", "AGAG", "AGAGA", "MKTAYIAK", "NLYIQWLKDGGPSSGRPPPS", "MKTAYIAKQR" * 7, "ARNDCQEGHILKMFPSTWYV" * 6]


def _check(origami, chains, xs, cutoff):
    params = origami.Params() if cutoff else origami.Params.all_pairs()
    eng = origami.Engine(params)
    for c, x in zip(chains, xs):
        eng.add_system(c, x)
    eng.finalize()
    nb, born = (10.0, 20.0) if cutoff else (INF, INF)
    for k, (c, x) in enumerate(zip(chains, xs)):
        e, o = eng.energies(k), Orc(c)
        ref = o.energy_terms(x, nb, born)
        for t in TERMS:
            assert abs(e[t] - ref[t]) <= 1e-10 * max(abs(ref[t]), 1.0), (k, t, e[t], ref[t])
        out, r = np.zeros(4), np.zeros(x.shape[0])
        assert e["nb_pairs"] == oracle().orc_nonbonded_energy(o.tp, dp(x), nb, dp(out))
        assert e["born_clamped"] == oracle().orc_born_radii(o.tp, dp(x), born, dp(r))
    eng.close()


def _built(origami, seqs, seed):
    rng = np.random.default_rng(seed)
    chains = [origami.Chain.build(s) for s in seqs]
    return chains, [np.ascontiguousarray(c.positions + rng.normal(scale=0.05, size=(c.n_atoms, 3))) for c in chains]


@pytest.mark.parametrize("cutoff", [False, True])
@pytest.mark.parametrize("seq", SEQS, ids=[str(len(s)) for s in SEQS])
def test_energy_terms_of_one_system(origami, seq, cutoff):
    chains, xs = _built(origami, [seq], len(seq))
    _check(origami, chains, xs, cutoff)


@pytest.mark.parametrize("cutoff", [False, True])
def test_energy_terms_of_uneven_systems(origami, cutoff):
    chains, xs = _built(origami, SEQS[::-1] + SEQS[2:6], 7)
    _check(origami, chains, xs, cutoff)
