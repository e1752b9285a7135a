"""A tuning cache written for other kernels is not applied: the launch shapes'
numbers mean something else there."""
from __future__ import annotations

import json

import pytest

pytestmark = pytest.mark.gpu


def _engine(origami):
    ch = origami.Chain.build("NLYIQWLKDGGPSSGRPPPS")
    eng = origami.Engine(origami.Params.all_pairs())
    eng.add_system(ch, ch.positions, 310.0)
    eng.finalize()
    return eng


def test_entries_of_other_kernels_are_ignored(origami, tmp_path):
    cache = tmp_path / "tune.json"
    eng = _engine(origami)
    eng.autotune(str(cache))
    eng.close()
    entries = json.loads(cache.read_text())
    assert len(entries) == 1
    (key, value), = entries.items()
    bucket, version = key.rsplit("|kernels=", 1)
    value["born"], value["force"] = [2, 1, 32], [5, 1, 32]
    for other in (bucket, bucket + "|kernels=%d" % (int(version) - 1)):
        cache.write_text("{\n %s: %s\n}\n" % (json.dumps(other), json.dumps(value)))
        eng = _engine(origami)
        r = eng.autotune(str(cache))
        assert r["from_cache"] == 0
        eng.close()
        assert key in json.loads(cache.read_text())
    # the current entry is applied as it stands
    cache.write_text("{\n %s: %s\n}\n" % (json.dumps(key), json.dumps(value)))
    eng = _engine(origami)
    r = eng.autotune(str(cache))
    assert r["from_cache"] == 1 and r["born_shape"] == 2 and r["force_shape"] == 5
    eng.close()
