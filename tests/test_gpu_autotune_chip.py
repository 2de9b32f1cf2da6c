"""Tuning a context whose solves run on the chip leaves them there."""
import json

import numpy as np
import pytest

from tahoe_gb300 import autotune, lib
from tests.test_gpu_memory_short import _context

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,n", [(lib.FP64, 8), (lib.FP64, 24), (lib.MIXED, 8), (lib.MIXED, 30)])
def test_solve_on_the_chip_stays_there(tmp_path, precision, n):
    c, mesh = _context(n)
    c.tangent(precision)
    assert c.routes(precision)[0] != "streamed"
    before, its = c.pcg(None, rel_tol=1e-6, max_it=4000)[:2]
    shapes = c.tuning()
    path = str(tmp_path / "t.json")
    old = {autotune.signature(c, precision, lib.TOTAL_LAGRANGIAN).split("|chip")[0]:
           {"tile_blocks": 256, "stages": 3, "release": 1, "sym": 2, "sym_tile": 256, "tangent_epb": 2}}
    with open(path, "w") as f:
        json.dump(old, f)  # a table from before such solves
    for cached in (False, True):
        out = autotune.Tuner(cache_path=path, reps=3).tune(c, precision, lib.TOTAL_LAGRANGIAN)
        assert out["cached"] == cached and out["chip"] and out["sym"] == 0
        assert c.tuning() == shapes  # the Simo group's tangent has no shape to choose
        after, its2 = c.pcg(None, rel_tol=1e-6, max_it=4000)[:2]
        assert np.array_equal(before, after) and its == its2


def test_tuning_the_streamed_precision_leaves_the_other_on_the_chip(tmp_path):
    c, mesh = _context(30)
    c.tangent(lib.FP64)
    assert [c.routes(p)[0] for p in (lib.FP64, lib.MIXED)] == ["streamed", "hybrid"]
    out = autotune.Tuner(cache_path=str(tmp_path / "t.json"), reps=3, tiles=(640,), stages=(2,)).tune(
        c, lib.FP64, lib.TOTAL_LAGRANGIAN)
    assert out["sym"] == 0 and c.routes(lib.MIXED)[0] == "hybrid"
