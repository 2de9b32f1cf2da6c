"""Batches on the chip: what a partition into RVEs may be, and that an RVE's
solve does not depend on the batch it shares."""
import numpy as np
import pytest

from tahoe_gb300 import lib, rve

pytestmark = pytest.mark.gpu


def _batch(ns, seed=0):
    rng = np.random.default_rng(seed)
    return rve.RVEBatch(ns, [rve.sample_F(rng) for _ in ns])


@pytest.mark.parametrize("form", [-1, 1, 3])
def test_an_rve_without_nodes_is_refused(form):
    b = _batch([4, 5])
    c = b.setup()
    c.pcg_form(form)
    cut = lambda off: [0, off[1], off[1], off[2]]
    c.set_segments(cut(b.node_off), cut(b.elem_off))
    c.set_u(np.zeros_like(b.X))
    with pytest.raises(lib.TahoeError) as e:
        c.predict_prescribed(b.prescribed_idx, b.prescribed_val)
    assert e.value.code == -1
