"""Device memory of the plans of the solves on the chip: it goes with the
partition or the mesh that it was made for."""
import numpy as np
import pytest

from tahoe_gb300 import lib, rve
from tahoe_gb300.meshgen import BoxMesh, equations
from tahoe_gb300.model import material_params
from tests.memory import pool_used

pytestmark = pytest.mark.gpu


def test_partitions_leave_nothing_behind():
    rng = np.random.default_rng(0)
    b = rve.RVEBatch([6] * 8, [rve.sample_F(rng) for _ in range(8)])
    c = b.setup()
    used = []
    for _ in range(4):
        b.solve(max_iterations=2)
        used.append(pool_used())
        c.set_segments(b.node_off, b.elem_off)
    assert used[1:] == used[:1] * 3


@pytest.mark.parametrize("precision", [lib.FP64, lib.MIXED])
def test_a_mesh_that_does_not_fit_leaves_nothing_behind(precision):
    """Shuffled node numbers: every part's rows reach the whole mesh, and no
    split over the SMs holds that many columns."""
    n = 20 if precision == lib.FP64 else 25
    mesh = BoxMesh(n, n, n)
    p = np.random.default_rng(1).permutation(mesh.nnd)
    X = np.empty_like(mesh.X)
    X[p] = mesh.X
    bottom = p[mesh.face_nodes(2, 0)]
    eq = equations(mesh.nnd, np.concatenate([bottom * 3 + d for d in range(3)]))

    def used(form):
        start = pool_used()
        c = lib.Context(0)
        c.upload(X, p[mesh.conn].astype(np.int32), eq)
        c.set_formulation(lib.SMALL_STRAIN)
        c.set_material(0, *material_params({"kind": "ss_hookean", "E": 1.0, "nu": 0.3}))
        c.pcg_form(form)
        c.tangent(precision)
        out = pool_used() - start
        c.close()
        return out

    assert used(-1) == used(1)
