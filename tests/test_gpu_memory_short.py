"""Short device memory: a tangent that finds no room leaves the last one as it
was, and what the solves on the chip find no room for is streamed."""
import numpy as np
import pytest

from tahoe_gb300 import lib, rve
from tahoe_gb300.meshgen import BoxMesh, equations
from tahoe_gb300.model import material_params
from tests.memory import ShortMemory

pytestmark = pytest.mark.gpu

SIMO = {"kind": "fs_simo", "mu": 1.0, "kappa": 10.0}


def _context(n=16):
    mesh = BoxMesh(n, n, n, jitter=0.1, seed=2)
    bottom = mesh.face_nodes(2, 0)
    eq = equations(mesh.nnd, np.concatenate([bottom * 3 + d for d in range(3)]))
    c = lib.Context(0)
    c.upload(mesh.X, mesh.conn, eq)
    c.set_formulation(lib.TOTAL_LAGRANGIAN)
    c.set_material(0, *material_params(SIMO))
    f = np.zeros((mesh.nnd, 3))
    f[mesh.face_nodes(2, 1), 0] = 1e-4
    c.set_fext(f)
    c.set_load_factor(1.0)
    c.set_u(np.zeros((mesh.nnd, 3)))
    c.residual(want_vector=False)
    return c, mesh


def _solve(c):
    return c.pcg(None, rel_tol=1e-6, max_it=2000)[0]


@pytest.mark.parametrize("precision,form,n", [(lib.FP64, 3, 16), (lib.MIXED, 3, 16), (lib.MIXED, 1, 33)])
def test_tangent_without_room_leaves_the_last_one(precision, form, n):
    """The default form solves this mesh without a matrix storage; the streamed
    form's storage then finds no room, at another displacement.  (Form 1's bytes
    are reserved on meshes of up to 32,768 nodes.)"""
    c, mesh = _context(n)
    c.tangent(precision)
    ref = _solve(c)
    c.set_u(0.02 * mesh.X * np.array([1.0, -0.3, 0.2]))
    c.pcg_form(form)
    with ShortMemory():
        with pytest.raises(lib.TahoeError) as e:
            c.tangent(precision)
        assert e.value.code == -3
    c.pcg_form(-1)
    assert np.array_equal(_solve(c), ref)
    # streamed: the same matrix, assembled from the same element blocks
    c.pcg_form(form)
    du = _solve(c)
    assert np.abs(du - ref).max() < 1e-3 * np.abs(ref).max()
    # and the tangent that found no room is the next one's
    c.tangent(precision)
    assert np.abs(_solve(c) - ref).max() > 1e-3 * np.abs(ref).max()


def _rves(composed):
    ns, Fs = [16, 16], [rve.sample_F(np.random.default_rng(i)) for i in range(2)]
    c = lib.Context(0)
    if composed:
        r = rve.ResidentRVEs(c)
        r.compose(ns)
        c.set_affine(np.asarray(Fs).reshape(-1))
    else:
        b = rve.RVEBatch(ns, Fs)
        b.setup(ctx=c)
        c.set_prescribed(b.prescribed_idx, b.prescribed_val)
    c.residual(want_vector=False)
    return c


@pytest.mark.parametrize("precision", [lib.FP64, lib.MIXED])
@pytest.mark.parametrize("case", ["mesh", "uploaded", "composed"])
def test_plans_without_room_are_streamed(precision, case):
    """A mesh whose matrix storage is there and whose plans for the solve on
    the chip find no room: the streamed solve, bitwise."""
    c = _context()[0] if case == "mesh" else _rves(case == "composed")
    c.pcg_form(1 if case == "mesh" else 3)
    if case != "mesh":
        c.set_u(np.zeros((c.nnd, 3)))
    c.tangent(precision)
    ref = _solve(c)
    c.pcg_form(-1)
    with ShortMemory():
        c.tangent(precision)
        assert np.array_equal(_solve(c), ref)


def test_exchange_without_room_is_streamed():
    """The plans fit, the solve's exchange words do not."""
    c, mesh = _context()
    c.pcg_form(1)
    c.tangent(lib.FP64)
    ref = _solve(c)
    c.pcg_form(-1)
    c.tangent(lib.FP64)
    with ShortMemory(left=200 << 10):
        assert np.array_equal(_solve(c), ref)


def test_storages_are_whole_or_not_there():
    """An allocation that fails between the arrays of one storage, at any of
    them: the next use finds none or all of it."""
    def ready(form):
        c = _context()[0]
        c.pcg_form(1)
        c.tangent(lib.FP64)
        ref = _solve(c)
        c.pcg_form(form)
        return c, ref

    failed = 0
    for left in range(1, 9):
        # the push storage: tiles, then push slots
        c, ref = ready(3)
        with ShortMemory(left=left << 20):
            try:
                c.tangent(lib.FP64)
            except lib.TahoeError as e:
                assert e.code == -3
                failed += 1
        c.tangent(lib.FP64)
        du = _solve(c)
        assert np.abs(du - ref).max() < 1e-3 * np.abs(ref).max()
        # the symmetric format: eight planes, then one
        c, ref = ready(1)
        with ShortMemory(left=left << 20):
            try:
                c.spmv_symmetric(1)
            except lib.TahoeError as e:
                assert e.code == -3
                failed += 1
        c.spmv_symmetric(1)
        du = _solve(c)
        assert np.abs(du - ref).max() < 1e-3 * np.abs(ref).max()
    assert failed >= 8


@pytest.mark.parametrize("left", [100, 200, 300, 400, 500, 600])
def test_vectors_are_of_one_precision(left):
    """An allocation that fails between the PCG vectors as they change their
    precision: no update is left, and the next solve has all of them."""
    c = _context()[0]
    c.pcg_form(1)
    c.tangent(lib.MIXED)
    small = _solve(c)
    c.tangent(lib.FP64)
    ref = _solve(c)
    c.tangent(lib.MIXED)
    _solve(c)
    c.tangent(lib.FP64)
    with ShortMemory(left=left << 10):  # of five times 157 KB
        with pytest.raises(lib.TahoeError) as e:
            c.pcg(None, rel_tol=1e-6, max_it=2000, want_du=False)
        assert e.value.code == -3
        with pytest.raises(lib.TahoeError):
            c.apply_update()
    assert np.array_equal(_solve(c), ref)
    c.tangent(lib.MIXED)
    assert np.array_equal(_solve(c), small)
