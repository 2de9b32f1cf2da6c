"""Meshes as generators number and shape them, on the chip against the streamed
solve: shuffled node numbers, an edge that many elements share, a strongly graded
box; and right-hand sides and matrices that no solve has an answer to."""
import numpy as np
import pytest
import scipy.sparse as sp

from tahoe_gb300 import lib
from tahoe_gb300.meshgen import BoxMesh, equations
from tahoe_gb300.model import material_params

pytestmark = pytest.mark.gpu

HOOKE = {"kind": "ss_hookean", "E": 1.0, "nu": 0.3}


def _context(X, conn, bottom, top, mat=HOOKE):
    c = lib.Context(0)
    c.upload(X, conn, equations(len(X), np.concatenate([bottom * 3 + d for d in range(3)])))
    c.set_formulation(lib.SMALL_STRAIN)
    c.set_material(0, *material_params(mat))
    f = np.zeros((len(X), 3))
    f[top, 0] = 1e-3
    f[top, 2] = -2e-3
    c.set_fext(f)
    c.set_load_factor(1.0)
    c.set_u(np.zeros((len(X), 3)))
    c.residual(want_vector=False)
    return c


def _box(n, shuffle=None):
    m = BoxMesh(*n)
    p = np.arange(m.nnd) if shuffle is None else np.random.default_rng(shuffle).permutation(m.nnd)
    X = np.empty_like(m.X)
    X[p] = m.X
    return X, p[m.conn].astype(np.int32), p[m.face_nodes(2, 0)], p[m.face_nodes(2, 1)]


def _star(valence, rings, layers):
    """`valence` hexes around every edge of the axis: its nodes have
    3 (2 valence + 1) blocks a row, the others at most 27."""
    k = 2 * valence
    ang = 2 * np.pi * np.arange(k) / k
    plane = [np.zeros((1, 2))]
    for r in range(1, rings + 1):
        # the first ring's outer corners are further out: its quads are convex
        rad = np.where(np.arange(k) % 2 == 0, r, r + 0.35 / r)
        plane.append(np.stack([rad * np.cos(ang), rad * np.sin(ang)], axis=1))
    plane = np.concatenate(plane)
    at = lambda r, i: 1 + (r - 1) * k + i % k
    quads = [(0, at(1, 2 * i), at(1, 2 * i + 1), at(1, 2 * i + 2)) for i in range(valence)]
    quads += [(at(r, i), at(r + 1, i), at(r + 1, i + 1), at(r, i + 1)) for r in range(1, rings) for i in range(k)]
    n = len(plane)
    X = np.concatenate([np.column_stack([plane / rings, np.full(n, 2.0 * z / layers)]) for z in range(layers + 1)])
    q = np.array(quads)
    conn = np.concatenate([np.concatenate([q + z * n, q + (z + 1) * n], axis=1) for z in range(layers)])
    return X, conn.astype(np.int32), np.arange(n), np.arange(n) + layers * n


def _residual(c, precision, du):
    """||R - K du|| / ||R||, K as assembled."""
    R, _ = c.residual()
    rp, ci, v = c.tangent_csr()
    return np.linalg.norm(R - sp.csr_matrix((v, ci, rp)) @ du) / np.linalg.norm(R)


def _check(c, precision, route, rel_tol, bound):
    assert c.routes(precision)[0] == route
    c.tangent(precision)
    du, its, _, rc = c.pcg(None, rel_tol=rel_tol, max_it=5000)
    assert rc == 0 and its > 0
    assert np.array_equal(c.pcg(None, rel_tol=rel_tol, max_it=5000)[0], du)
    c.pcg_form(1)
    c.tangent(precision)
    ref = c.pcg(None, rel_tol=rel_tol, max_it=5000)[0]
    # as small a residual of the same matrix as the streamed solve's
    assert _residual(c, precision, du) <= 2 * _residual(c, precision, ref) + rel_tol
    assert np.abs(du - ref).max() <= bound * np.abs(ref).max()


@pytest.mark.parametrize("precision,n,route", [
    (lib.FP64, 7, "chip"), (lib.FP64, 13, "chip"), (lib.FP64, 17, "chip"), (lib.FP64, 20, "streamed"),
    (lib.MIXED, 7, "chip"), (lib.MIXED, 14, "chip"), (lib.MIXED, 20, "chip"), (lib.MIXED, 25, "streamed"),
    (lib.MIXED, 28, "hybrid")])
def test_shuffled_node_numbers(precision, n, route):
    c = _context(*_box((n, n, n), shuffle=n))
    fp64 = precision == lib.FP64
    _check(c, precision, route, 1e-11 if fp64 else 1e-5, 1e-7 if fp64 else 5e-3)


@pytest.mark.parametrize("precision,rings,layers", [(lib.FP64, 3, 6), (lib.FP64, 12, 20), (lib.MIXED, 3, 6),
                                                   (lib.MIXED, 12, 30), (lib.MIXED, 20, 44)])
def test_an_edge_of_twelve_elements(precision, rings, layers):
    """75 blocks a row: a second and third group of eight steps on the chip, and
    a row that the hybrid form refuses (the last case has 21,645 nodes)."""
    c = _context(*_star(12, rings, layers))
    fp64 = precision == lib.FP64
    _check(c, precision, "chip", 1e-11 if fp64 else 1e-5, 1e-7 if fp64 else 5e-3)


def test_a_strongly_graded_box():
    """An eighth of the nodes in a corner of 0.0001 of the volume: more than the
    hybrid form's ordering takes in one of its cells."""
    X, conn, bottom, top = _box((28, 28, 28))
    X = np.where(X < 0.5, 0.1 * X, 0.05 + 1.9 * (X - 0.5))
    c = _context(X, conn, bottom, top)
    assert c.routes(lib.MIXED)[0] == "chip"
    _check(c, lib.MIXED, "chip", 1e-4, 5e-2)


@pytest.mark.parametrize("precision,n,route", [(lib.FP64, 6, "chip"), (lib.FP64, 18, "chip"), (lib.MIXED, 6, "chip"),
                                               (lib.MIXED, 18, "chip"), (lib.MIXED, 28, "hybrid"),
                                               (lib.FP64, 30, "streamed")])
def test_breakdowns(precision, n, route):
    c = _context(*_box((n, n, n)))
    assert c.routes(precision)[0] == route
    c.tangent(precision)
    R, _ = c.residual()
    ref = c.pcg(R, rel_tol=1e-5)[0]
    for bad in (np.nan, np.inf):
        b = R.copy()
        b[len(b) // 3] = bad
        with pytest.raises(lib.TahoeError) as e:
            c.pcg(b, rel_tol=1e-5)
        assert e.value.code == -5
    assert c.pcg(np.zeros_like(R), rel_tol=1e-5)[1:] == (0, 0.0, 0)
    assert c.pcg(R, rel_tol=1e-5, max_it=3)[1::2] == (3, -6)
    assert np.array_equal(c.pcg(R, rel_tol=1e-5)[0], ref)
    # a negative definite matrix
    c = _context(*_box((n, n, n)), mat={"kind": "ss_hookean", "C": -np.eye(6)})
    c.tangent(precision)
    with pytest.raises(lib.TahoeError) as e:
        c.pcg(None, rel_tol=1e-5)
    assert e.value.code == -5
