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


def _varied():
    """RVEs that share a plan and RVEs that only look alike: 0 and 4 are equal, 1
    has a free dof on its boundary, 3 is numbered in another order."""
    b = _batch([5, 5, 6, 5, 5, 6])
    rng = np.random.default_rng(9)
    b.node_off, b.elem_off = b.node_off.copy(), b.elem_off.copy()
    a, e = b.node_off[3], b.node_off[4]
    p = np.arange(b.nnd)
    p[a:e] = a + rng.permutation(e - a)
    X = np.empty_like(b.X)
    X[p] = b.X
    b.X, b.conn = X, p[b.conn].astype(np.int32)
    b.prescribed_idx = p[b.prescribed_idx // 3] * 3 + b.prescribed_idx % 3
    free = np.searchsorted(b.prescribed_idx, b.node_off[1] * 3)
    assert b.node_off[1] <= b.prescribed_idx[free] // 3 < b.node_off[2]
    b.prescribed_idx = np.delete(b.prescribed_idx, free)
    b.prescribed_val = np.delete(b.prescribed_val, free)
    return b


@pytest.mark.parametrize("precision,rel_tol,bound", [(lib.FP64, 1e-12, 1e-9), (lib.MIXED, 1e-7, 1e-3)])
def test_uploaded_rves_with_and_without_a_common_plan(precision, rel_tol, bound):
    b = _varied()
    c = b.setup()
    c.set_prescribed(b.prescribed_idx, 0.2 * b.prescribed_val)
    c.residual(want_vector=False)
    du = {}
    for form in (3, -1):
        c.pcg_form(form)
        c.tangent(precision)
        du[form] = c.pcg(None, rel_tol=rel_tol, max_it=2000)[0]
    assert np.abs(du[-1] - du[3]).max() < bound * np.abs(du[3]).max()
