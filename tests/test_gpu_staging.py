"""Displacements and residuals of meshes on both sides of the size up to which
they pass through pinned memory (128 KB: 5,461 nodes): the round trip is exact,
the residual vector has the norm returned, and errors leave the next call
intact."""
import numpy as np
import pytest

from tahoe_gb300 import lib
from tahoe_gb300.meshgen import BoxMesh
from tahoe_gb300.model import SolidModel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(1, 1, 1), (9, 8, 7), (16, 16, 17), (17, 17, 16), (24, 20, 20)])
@pytest.mark.parametrize("precision", [lib.MIXED, lib.FP64])
def test_small_vectors(dims, precision):
    mesh = BoxMesh(*dims, jitter=0.1, seed=1)
    m = SolidModel(mesh.X, mesh.conn, "total_lagrangian", {"kind": "fs_simo", "mu": 1.0, "kappa": 10.0})
    for node in mesh.face_nodes(2, 0):
        m.add_kbc(node, 2)
    m.set_schedule([(0.0, 1.0)])
    c = m.setup()
    X = np.asarray(mesh.X).reshape(-1, 3)
    rng = np.random.default_rng(3)
    got = []
    for k in range(2):
        u = 0.02 / max(dims) * rng.standard_normal(X.shape)
        c.set_u(u)
        assert np.array_equal(c.get_u(), u)
        R, norm = c.residual(precision=precision)
        assert abs(np.linalg.norm(R) - norm) <= 1e-12 * norm  # two orders of one FP64 sum
        assert c.residual(want_vector=False, precision=precision)[1] == norm
        got.append((u, R))
        c.set_u(-3.0 * X)  # turned inside out
        with pytest.raises(lib.TahoeError):
            c.residual(precision=precision)
    c.set_u(got[0][0])
    assert np.array_equal(c.residual(precision=precision)[0], got[0][1])
