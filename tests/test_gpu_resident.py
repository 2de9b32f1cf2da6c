"""The resident PCG (respcg.cu): the default form on meshes and RVE batches
that fit the chip's shared memory, against the streamed forms on the same
tangent and right-hand side.

Sizes sit where the split over CTAs changes: one chunk of eight rows, a part
of one CTA, clusters of several CTAs, the grid form, and past the capacity
(where the default streams).  Prescribed dofs are partial on one face, so rows
with one or two free dofs take part.
"""
import numpy as np
import pytest

from tahoe_gb300 import lib, rve
from tahoe_gb300.meshgen import BoxMesh, equations
from tahoe_gb300.model import SolidModel

pytestmark = pytest.mark.gpu

SIMO = {"kind": "fs_simo", "mu": 1.0, "kappa": 10.0}


def _system(dims, precision, scale=1.0):
    mesh = BoxMesh(*dims, jitter=0.15, seed=11)
    m = SolidModel(mesh.X, mesh.conn, "total_lagrangian", dict(SIMO, mu=scale, kappa=10.0 * scale))
    for node in mesh.face_nodes(2, 0):
        for d in range(3):
            m.add_kbc(node, d)
    for node in mesh.face_nodes(2, 1):
        m.add_kbc(node, 2, -0.02 / dims[2], True)
    for node in mesh.face_nodes(0, 0):
        m.add_kbc(node, 0)
    m.set_schedule([(0.0, 1.0)])
    m.setup()
    c = m.ctx
    c.pcg_form(1)
    m.apply_step(1.0, (precision, lib.PRECOND_JACOBI, 1e-6))
    c.set_iteration(-1)
    R, _ = c.residual()
    c.pcg_form(-1)
    c.tangent(precision)
    return m, c, R


DIMS = [(1, 1, 1), (1, 2, 1), (2, 2, 2), (5, 5, 5), (7, 6, 8), (10, 9, 11), (13, 13, 13), (17, 15, 16), (26, 25, 24)]


@pytest.mark.parametrize("dims", DIMS)
@pytest.mark.parametrize("precision", [lib.MIXED, lib.FP64])
@pytest.mark.parametrize("precond", [lib.PRECOND_JACOBI, lib.PRECOND_BLOCK_JACOBI])
def test_resident_solve_equals_the_streamed_solve(dims, precision, precond):
    m, c, R = _system(dims, precision)
    tol = 1e-6 if precision == lib.MIXED else 1e-11
    du, its, rr, rc = c.pcg(R, rel_tol=tol, max_it=5000, precond=precond)
    assert rc == 0 and rr <= tol
    again = c.pcg(R, rel_tol=tol, max_it=5000, precond=precond)
    assert np.array_equal(again[0], du) and again[1] == its  # bitwise repeatable
    c.pcg_form(1)  # the streamed form on the same tangent
    du1, its1, _, rc1 = c.pcg(R, rel_tol=tol, max_it=5000, precond=precond)
    assert rc1 == 0
    # both within the tolerance of the solution: condition numbers here stay
    # below 1e4, so the error is below 1e2 times the residual tolerance (its
    # square root bounds the energy norm), and FP32's rounding
    bound = 2e-4 if precision == lib.MIXED else 1e-8
    assert np.abs(du - du1).max() <= bound * np.abs(du1).max()
    assert abs(its - its1) <= max(3, 0.05 * its1)


@pytest.mark.parametrize("precision", [lib.MIXED, lib.FP64])
@pytest.mark.parametrize("scale", [1e-12, 1e9])
def test_scaling_of_matrix_and_right_hand_side(precision, scale):
    # stiffness and residual far from one: the solve works on a power of two
    # of them, so du of (K, R) scaled together is that of the unscaled system
    tol = 1e-6 if precision == lib.MIXED else 1e-11
    m, c, R = _system((7, 6, 8), precision)
    ref = c.pcg(R, rel_tol=tol, max_it=5000)
    m2, c2, R2 = _system((7, 6, 8), precision, scale)
    c2.set_u(c.get_u())  # the same state: each system's predictor stops at its own 1e-6
    c2.tangent(precision)
    du, its, rr, rc = c2.pcg(R * scale, rel_tol=tol, max_it=5000)
    assert rc == 0 and abs(its - ref[1]) <= max(2, 0.05 * ref[1])
    bound = 2e-4 if precision == lib.MIXED else 1e-8
    assert np.abs(du - ref[0]).max() <= bound * np.abs(ref[0]).max()
    tiny = c.pcg(R * 1e-150, rel_tol=tol, max_it=5000)
    assert tiny[3] == 0
    assert np.abs(tiny[0] * 1e150 - ref[0]).max() <= bound * np.abs(ref[0]).max()


@pytest.mark.parametrize("dims", [(5, 5, 5), (17, 15, 16)])
@pytest.mark.parametrize("precision", [lib.MIXED, lib.FP64])
def test_limits_and_breakdown(dims, precision):
    m, c, R = _system(dims, precision)
    du, its, rr, rc = c.pcg(R, rel_tol=1e-14, max_it=4)
    assert rc == -6 and its == 4 and 0.0 < rr
    du, its, rr, rc = c.pcg(np.zeros_like(R), rel_tol=1e-8)
    assert rc == 0 and its == 0 and not du.any()
    bad = R.copy()
    bad[len(bad) // 2] = np.nan
    with pytest.raises(lib.TahoeError) as ei:
        c.pcg(bad, rel_tol=1e-8)
    assert ei.value.code == -5
    assert c.pcg(R, rel_tol=1e-6)[3] == 0  # the context stays usable
    mesh = BoxMesh(*dims)
    neg = SolidModel(mesh.X, mesh.conn, "small_strain",
                     {"kind": "ss_hookean", "C": -np.diag([3.0, 3, 3, 1, 1, 1]).reshape(36)})
    for node in mesh.face_nodes(2, 0):
        for d in range(3):
            neg.add_kbc(node, d)
    neg.setup()
    neg.ctx.tangent(precision)
    with pytest.raises(lib.TahoeError) as ei:
        neg.ctx.pcg(np.ones(neg.ctx.neq), rel_tol=1e-8)
    assert ei.value.code == -5 and "indefinite" in str(ei.value)


@pytest.mark.parametrize("precision", [lib.MIXED, lib.FP64])
def test_the_tangent_outlives_what_overwrites_its_element_blocks(precision):
    # a dump of element matrices and a timing of the tangent kernel re-form
    # the element blocks at another state: the solve still is the tangent's
    m, c, R = _system((7, 6, 8), precision)
    tol = 1e-6 if precision == lib.MIXED else 1e-11
    ref = c.pcg(R, rel_tol=tol)[0]
    u = c.get_u()
    bound = 2e-4 if precision == lib.MIXED else 1e-8
    for disturb in (lambda: c.element_dump(0, 4), lambda: c.time_kernel(2, 1)):
        c.set_u(u)
        c.tangent(precision)
        c.set_u(1.5 * u)
        disturb()
        du = c.pcg(R, rel_tol=tol)[0]
        assert np.abs(du - ref).max() <= bound * np.abs(ref).max()


@pytest.mark.parametrize("precision", [lib.MIXED, lib.FP64])
def test_uploaded_and_composed_batches_agree_and_repartition(precision):
    """A composed batch solves by its templates' plans, an uploaded one by its
    segments', a composed one with another partition by that partition's."""
    ns = [4, 7, 5, 10, 2]
    rng = np.random.default_rng(5)
    Fs = np.stack([rve.sample_F(rng) for _ in ns])
    res = rve.ResidentRVEs(lib.Context(0))
    c = res.ctx
    rc, rep, rel, P = res.solve(ns, Fs, precision=precision)
    status = res.status
    # the one free node of the side-2 RVE is in equilibrium by symmetry: its
    # first residual is rounding, which no iteration makes smaller
    assert (status[:4] == 0).all()
    c.pcg_form(3)  # the streamed solves
    _, _, _, Ps = res.solve(ns, Fs, precision=precision)
    assert np.array_equal(res.status, status)
    assert np.abs(Ps - P).max() <= 1e-8 * np.abs(P).max()
    c.pcg_form(-1)
    up = rve.RVEBatch(ns, Fs)
    _, _, _, P2 = up.solve(precision=precision, precond=lib.PRECOND_BLOCK_JACOBI)
    # (its boundary values are formed on the host: the inputs differ by rounding)
    assert np.array_equal(up.status, status)
    assert np.abs(P2 - P).max() <= 1e-8 * np.abs(P).max()
    # two RVEs as one segment: another Krylov space, the same solution
    no = [0] + list(np.cumsum([(n + 1) ** 3 for n in ns]))
    eo = [0] + list(np.cumsum([n ** 3 for n in ns]))
    res.compose(ns)
    c.set_segments([no[0], no[2], no[3], no[4], no[5]], [eo[0], eo[2], eo[3], eo[4], eo[5]])
    c.set_u(up.u0 * 0.0)
    idx, val = up.prescribed_idx, up.prescribed_val
    c.predict_prescribed(idx, val, precision=precision, precond=lib.PRECOND_BLOCK_JACOBI, lin_rel_tol=1e-4)
    c.newton_segmented(rel_tol=1e-8, precision=precision, precond=lib.PRECOND_BLOCK_JACOBI, check=False)
    assert (c.seg_status[:3] == 0).all()
    P3 = c.segment_stress(np.array([2.0, 1.0, 1.0, 1.0]))
    want = np.stack([0.5 * (P[0] + P[1]), P[2], P[3], P[4]])
    assert np.abs(P3 - want).max() <= 1e-7 * np.abs(P).max()


def test_rve_with_no_free_dof_is_a_zero_update():
    X = BoxMesh(1, 1, 1)
    c = lib.Context(0)
    c.set_formulation(lib.TOTAL_LAGRANGIAN)
    c.set_material(0, lib.MAT_FS_SIMO, np.array([1.0, 10.0]))
    free = c.template_add(BoxMesh(2, 2, 2).X, BoxMesh(2, 2, 2).conn, equations(27, np.arange(27 * 3)[:39]))
    none = c.template_add(X.X, X.conn, equations(8, np.arange(24)))
    c.compose([none, free, none])
    F = np.stack([np.eye(3) * 1.02] * 3)
    c.predict_affine(F, lin_rel_tol=1e-6)
    rc, rep, rel = c.newton_segmented(rel_tol=1e-8)
    assert rc == 0 and (c.seg_status == 0).all()
