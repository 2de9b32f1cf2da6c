"""tg_routes_get: where a solve and a tangent run."""
import numpy as np
import pytest

from tahoe_gb300 import lib, rve
from tahoe_gb300.meshgen import BoxMesh, equations
from tahoe_gb300.model import material_params

pytestmark = pytest.mark.gpu

HOOKE = {"kind": "ss_hookean", "E": 1.0, "nu": 0.3}
SIMO = {"kind": "fs_simo", "mu": 1.0, "kappa": 10.0}
STVENANT = {"kind": "fs_stvenant", "E": 1.0, "nu": 0.3}


def _context(n, formulation=lib.SMALL_STRAIN, mat=HOOKE):
    mesh = BoxMesh(*n)
    bottom = mesh.face_nodes(2, 0)
    c = lib.Context(0)
    c.upload(mesh.X, mesh.conn, equations(mesh.nnd, np.concatenate([bottom * 3 + d for d in range(3)])))
    c.set_formulation(formulation)
    c.set_material(0, *material_params(mat))
    return c


@pytest.mark.parametrize("n,fp64,mixed", [((6, 6, 6), "chip", "chip"), ((24, 24, 24), "chip", "chip"),
                                          ((31, 31, 31), "streamed", "hybrid"),
                                          ((80, 80, 80), "streamed", "streamed")])
def test_of_a_mesh(n, fp64, mixed):
    c = _context(n)
    assert (c.routes(lib.FP64)[0], c.routes(lib.MIXED)[0]) == (fp64, mixed)
    for off, on in ((lambda: c.pcg_form(1), lambda: c.pcg_form(-1)),
                    (lambda: c.spmv_symmetric(1), lambda: c.spmv_symmetric(0))):
        off()
        assert c.routes(lib.FP64)[0] == c.routes(lib.MIXED)[0] == "streamed"
        on()
    assert c.routes(lib.MIXED)[0] == mixed


def test_of_a_batch():
    def route(ns):
        return rve.RVEBatch(ns, [np.eye(3)] * len(ns)).setup().routes(lib.FP64)[0]
    assert [route(ns) for ns in ([4, 9], [4, 33], [33, 33])] == ["chip", "some", "streamed"]


def test_of_a_tangent():
    C = np.diag([3.0, 3.0, 3.0, 1.0, 1.0, 1.5]) + 0.5 * np.pad(np.ones((3, 3)), (0, 3))
    for formulation, mat, bbar, general in (
            (lib.SMALL_STRAIN, HOOKE, 0, False), (lib.SMALL_STRAIN, HOOKE, 1, True),
            (lib.SMALL_STRAIN, {"kind": "ss_hookean", "C": C}, 0, True), (lib.TOTAL_LAGRANGIAN, SIMO, 0, False),
            (lib.TOTAL_LAGRANGIAN, STVENANT, 0, False), (lib.UPDATED_LAGRANGIAN, SIMO, 0, True)):
        c = _context((2, 2, 2), formulation, mat)
        c.set_strain_displacement(bbar)
        assert [c.routes(p)[1] for p in (lib.FP64, lib.MIXED)] == [general] * 2
