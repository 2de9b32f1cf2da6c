"""The streamed solvers and the general tangent kernel, by name: the default form
solves most meshes and batches on the chip, and forms most tangents with kernels
of their own.  Each test checks the route that it is about."""
import numpy as np
import pytest

from tahoe_gb300 import autotune, lib, rve
from tahoe_gb300.meshgen import BoxMesh, equations
from tahoe_gb300.model import material_params
from tests.helpers import rel_err
from tests.test_gpu_memory_short import _context as simo_box
from tests.test_gpu_tangent_blocks import MATS, OTHER

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def batch():
    return rve.sample_batch(6, sizes=(4, 5, 6), seed=11)


def _set_up(ns, Fs, form):
    b = rve.RVEBatch(ns, Fs)
    b.setup()
    b.ctx.pcg_form(form)
    assert (b.ctx.routes(lib.FP64)[0] == "streamed") == (form >= 0)
    return b


# ---- per-RVE solves and the multi-vector PCG --------------------------------

@pytest.mark.parametrize("form", [1, 3])
@pytest.mark.parametrize("precision", [lib.FP64, lib.MIXED])
def test_streamed_rve_alone_equals_rve_in_batch(batch, form, precision):
    ns, Fs = batch
    kw = dict(precision=precision, rel_tol=1e-8, lin_rel_tol=1e-6)
    b = _set_up(ns, Fs, form)
    rc, rep, rel, P = b.solve(**kw)
    assert rc == 0
    u = b.ctx.get_u()
    for r in range(len(ns)):
        one = _set_up(ns[r:r + 1], Fs[r:r + 1], form)
        assert one.solve(**kw)[0] == 0
        assert np.array_equal(b.rve_displacement(r, u), one.ctx.get_u()), r


@pytest.mark.parametrize("form", [1, 3])
def test_streamed_rve_fails_alone(form):
    """As on the chip (test_gpu_rve.py): one Newton iteration, exact solves; the
    RVEs under a tiny deformation start at round-off and fail."""
    rng = np.random.default_rng(5)
    S = [rve.sample_F(rng) - np.eye(3) for _ in range(4)]
    ns = np.array([4, 5, 4, 6])
    Fs = np.stack([np.eye(3) + 2e-5 * S[0], np.eye(3) + S[1], np.eye(3) + 2e-5 * S[2], np.eye(3) + S[3]])
    kw = dict(precision=lib.FP64, rel_tol=1e-8, lin_rel_tol=1e-12, max_iterations=1)
    alone = []
    for r in range(4):
        one = _set_up(ns[r:r + 1], Fs[r:r + 1], form)
        P = one.solve(**kw)[3]
        alone.append((int(one.status[0]), P[0]))
    b = _set_up(ns, Fs, form)
    rc, rep, rel, P = b.solve(**kw)
    st = [int(v) for v in b.status]
    assert st == [a[0] for a in alone]
    assert 0 in st and rc == next(v for v in st if v != 0)
    for r in range(4):
        if st[r] == 0:
            assert np.array_equal(P[r], alone[r][1]), r


@pytest.mark.parametrize("precision", [lib.FP64, lib.MIXED])
def test_push_and_full_storage_and_chip_agree(batch, precision):
    ns, Fs = batch
    out = {}
    for form in (-1, 1, 3):
        b = _set_up(ns, Fs, form)
        rc, rep, rel, P = b.solve(precision=precision, rel_tol=1e-10,
                                  lin_rel_tol=1e-10 if precision == lib.FP64 else 1e-6)
        assert rc == 0 and np.all(b.status == 0) and rel.max() < 1e-10
        out[form] = (P, b.ctx.get_u())
    for form in (1, 3):
        for got, want in zip(out[form], out[-1]):
            assert rel_err(got, want) < 1e-8


@pytest.mark.parametrize("form", [1, 3])
@pytest.mark.parametrize("precision,lin_rel_tol,bound", [(lib.FP64, 1e-12, 1e-8), (lib.MIXED, 1e-7, 1e-5)])
def test_macro_tangent_of_the_multi_vector_pcg(batch, form, precision, lin_rel_tol, bound):
    """Against nine solves of every RVE on the chip, at the same state."""
    ns, Fs = batch
    b = _set_up(ns, Fs, -1)
    assert b.solve(precision=lib.FP64, rel_tol=1e-10, lin_rel_tol=1e-10)[0] == 0
    ref, its = b.ctx.macro_tangent(b.vol0, precision=lib.FP64, lin_rel_tol=1e-12)
    b.ctx.pcg_form(form)
    C, its = b.ctx.macro_tangent(b.vol0, precision=precision, lin_rel_tol=lin_rel_tol)
    assert its > 0
    for r in range(len(ns)):
        assert rel_err(C[r], ref[r]) < bound, r


@pytest.mark.parametrize("precision", [lib.FP64, lib.MIXED])
def test_macro_tangent_beside_an_rve_that_does_not_fit(precision):
    """The whole batch is one multi-vector PCG: the small RVE's tangent within
    the batch's tolerance of its own alone on the chip."""
    side = 33 if precision == lib.FP64 else 46
    Fs = [np.eye(3) + 0.01 * rve.sample_F(np.random.default_rng(i)) for i in range(2)]
    C = []
    for ns in ([6], [6, side]):
        b = rve.RVEBatch(ns, Fs[:len(ns)])
        b.setup()
        assert b.ctx.routes(precision)[0] == ("chip" if len(ns) == 1 else "some")
        b.ctx.set_u(b.u0)
        C.append(b.ctx.macro_tangent(b.vol0, precision=precision, lin_rel_tol=1e-7)[0][0])
    assert rel_err(C[1], C[0]) < 1e-4


@pytest.mark.parametrize("form", [-1, 1, 3])
def test_macro_tangent_at_the_iteration_limit(batch, form):
    """A limit is not an error of the call: the columns as far as they got."""
    ns, Fs = batch
    b = _set_up(ns, Fs, form)
    b.ctx.set_u(np.zeros_like(b.X))
    ref, _ = b.ctx.macro_tangent(b.vol0, precision=lib.FP64, lin_rel_tol=1e-10)
    C, its = b.ctx.macro_tangent(b.vol0, precision=lib.FP64, lin_rel_tol=1e-10, lin_max_it=5)
    assert its == 5 and rel_err(C, ref) > 1e-9


# ---- single meshes ----------------------------------------------------------

@pytest.mark.parametrize("n", [24, 26, 28])
def test_fp64_meshes_up_to_the_capacity(n):
    """15,625 to 24,389 nodes in FP64 on the chip, against form 1."""
    c, mesh = simo_box(n)
    c.tangent(lib.FP64)
    du = {}
    for form in (-1, 1):
        c.pcg_form(form)
        assert c.routes(lib.FP64)[0] == ("chip" if form < 0 else "streamed")
        du[form] = c.pcg(None, rel_tol=1e-11, max_it=4000)[0]
    assert rel_err(du[-1], du[1]) < 1e-7


def test_release_variants_and_the_tuned_product(tmp_path):
    """Form 1, whose product has shapes to choose: the two stage releases give
    bitwise the same solve, and the tuned one the same to rounding."""
    c, mesh = simo_box(10)
    c.pcg_form(1)
    assert c.routes(lib.MIXED)[0] == "streamed"
    c.tangent(lib.MIXED)
    du0 = c.pcg(None, rel_tol=1e-7)[0]
    out = autotune.Tuner(cache_path=str(tmp_path / "t.json"), reps=3, tiles=(256, 640, 1024), stages=(2, 3)).tune(
        c, lib.MIXED, lib.TOTAL_LAGRANGIAN)
    assert not out["cached"] and len(out["spmv_sweep"]) > 3
    c.spmv_symmetric(0)
    sols = []
    for r in (0, 1):
        c.spmv_release(r)
        c.tangent(lib.MIXED)
        sols.append(c.pcg(None, rel_tol=1e-7)[:2])
    assert np.array_equal(sols[0][0], sols[1][0]) and sols[0][1] == sols[1][1]
    assert rel_err(sols[0][0], du0) < 1e-4


# ---- the general tangent kernel ---------------------------------------------

def _bar(nel, formulation, mats, amplitude, bbar=0, used=None):
    mesh = BoxMesh(nel, 1, 1, lx=nel)
    rng = np.random.default_rng(nel)
    X = mesh.X + rng.uniform(-0.15, 0.15, size=mesh.X.shape)
    c = lib.Context(0)
    c.upload(X, mesh.conn, equations(len(X), []))
    c.set_formulation(formulation)
    c.set_strain_displacement(bbar)
    for b, m in enumerate(mats):
        c.set_material(b, *material_params(m))
    c.set_blocks(np.arange(nel) % (used or len(mats)))
    c.set_u(rng.uniform(-amplitude, amplitude, size=X.shape))
    c.set_iteration(0)
    c.residual(want_vector=False)
    return c


@pytest.mark.parametrize("precision", [lib.FP64, lib.MIXED])
@pytest.mark.parametrize("group", ["bbar", "updated simo", "updated stvenant", "simo", "stvenant", "j2", "hooke"])
@pytest.mark.parametrize("nel", [1, 7, 9, 17])
def test_general_tangent_shapes_bitwise_equal(group, precision, nel):
    if group == "bbar":
        c = _bar(nel, lib.SMALL_STRAIN, MATS["j2"][1], 0.004, bbar=1)
    elif group.startswith("updated"):
        _, mats, amp = MATS[group.split()[1]]
        c = _bar(nel, lib.UPDATED_LAGRANGIAN, mats, amp)
    else:  # an unused block of another material
        form, mats, amp = MATS[group]
        c = _bar(nel, form, mats + [OTHER[group]], amp, used=len(mats))
    assert c.routes(precision)[1]
    values = []
    for epb in (8, 4, 2):
        c.tangent_config(epb)
        c.tangent(precision)
        values.append(c.tangent_csr()[2])
    assert np.abs(values[0]).max() > 0
    assert np.array_equal(values[0], values[1]) and np.array_equal(values[0], values[2])


@pytest.mark.parametrize("nel", [1, 31, 33, 65])
@pytest.mark.parametrize("kind", ["simo", "j2", "hooke"])
def test_isotropic_tangent_equals_the_general_kernel(nel, kind):
    """tangent_iso.cu in mixed precision against tangent_kernel in FP64."""
    form, mats, amp = MATS[kind]
    c = _bar(nel, form, mats, amp)
    g = _bar(nel, form, mats + [OTHER[kind]], amp, used=len(mats))
    assert not c.routes(lib.MIXED)[1] and g.routes(lib.FP64)[1]
    c.tangent(lib.MIXED)
    g.tangent(lib.FP64)
    got, want = c.tangent_csr()[2], g.tangent_csr()[2]
    # FP32 sums of 8 points of products of at most 10 factors of order one: 100
    # roundings of 6e-8 at most, of the largest entry
    assert np.abs(got - want).max() <= 6e-6 * np.abs(want).max()
