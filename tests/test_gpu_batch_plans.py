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


@pytest.mark.parametrize("precision,side", [(lib.FP64, 33), (lib.MIXED, 46)])
@pytest.mark.parametrize("composed", [False, True])
def test_an_rve_beside_one_that_does_not_fit(precision, side, composed):
    """The large one is streamed, the others are solved on the chip: each as it
    is alone, bitwise, updates and iterations."""
    ns = [6, side, 9]
    Fs = [np.eye(3) + 0.01 * rve.sample_F(np.random.default_rng(i)) for i in range(3)]

    def solve(which):
        if composed:
            c = lib.Context(0)
            r = rve.ResidentRVEs(c)
            r.compose([ns[i] for i in which])
            c.set_u(np.zeros((c.nnd, 3)))
            c.set_affine(np.array([Fs[i] for i in which]))
        else:
            b = rve.RVEBatch([ns[i] for i in which], [Fs[i] for i in which])
            c = b.setup()
            c.set_u(np.zeros((c.nnd, 3)))
            c.set_prescribed(b.prescribed_idx, b.prescribed_val)
        c.residual(want_vector=False)
        c.tangent(precision)
        its = c.pcg(None, rel_tol=1e-5, max_it=4000, want_du=False)[1]
        c.apply_update()
        u = c.get_u()
        cut = np.concatenate([[0], np.cumsum([(ns[i] + 1) ** 3 for i in which])])
        return its, [u[a:b] for a, b in zip(cut[:-1], cut[1:])]

    its, u = solve([0, 1, 2])
    alone = [solve([i]) for i in range(3)]
    assert its == max(a[0] for a in alone)
    for i in range(3):
        assert np.abs(u[i]).max() > 0 and np.array_equal(u[i], alone[i][1][0]), ns[i]


def test_failing_rves_beside_ones_that_do_not_fit():
    """One Newton iteration with exact inner solves: RVEs under a tiny
    deformation, which start at round-off, fail and the others converge.  Every
    outcome and every converged stress is the RVE's own, alone (bitwise), for
    the streamed ones and those on the chip."""
    rng = np.random.default_rng(5)
    S = [rve.sample_F(rng) - np.eye(3) for _ in range(4)]
    ns = [4, 33, 5, 33]
    Fs = [np.eye(3) + f * S[i] for i, f in enumerate((2e-5, 2e-5, 1.0, 0.02))]
    kw = dict(precision=lib.FP64, rel_tol=1e-8, lin_rel_tol=1e-12, max_iterations=1)
    alone = []
    for i in range(4):
        b = rve.RVEBatch(ns[i:i + 1], Fs[i:i + 1])
        P = b.solve(**kw)[3]
        alone.append((int(b.status[0]), P[0]))
    b = rve.RVEBatch(ns, Fs)
    rc, rep, rel, P = b.solve(**kw)
    st = [int(v) for v in b.status]
    assert st == [a[0] for a in alone]
    assert 0 in st and rc == next(v for v in st if v != 0)
    for i in range(4):
        if st[i] == 0:
            assert np.array_equal(P[i], alone[i][1]), i
