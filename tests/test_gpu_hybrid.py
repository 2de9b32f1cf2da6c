"""The hybrid PCG (hybridpcg.cu): the default FP32 form on meshes of 20,000
nodes and more, against the streamed forms on the same tangent and
right-hand side.

Sizes: parts that fit tensor memory, parts that just do not (the rest kept in
L2), an elongated mesh whose parts are slabs, odd sides, sizes where p, s
and a block preconditioner no longer fit shared memory, and past the largest
(streamed).
"""
import numpy as np
import pytest

from tahoe_gb300 import lib
from tahoe_gb300.meshgen import BoxMesh
from tahoe_gb300.model import SolidModel

pytestmark = pytest.mark.gpu

SIMO = {"kind": "fs_simo", "mu": 1.0, "kappa": 10.0}


def _system(dims):
    mesh = BoxMesh(*dims, jitter=0.15, seed=11)
    m = SolidModel(mesh.X, mesh.conn, "total_lagrangian", SIMO)
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
    m.apply_step(1.0, (lib.MIXED, lib.PRECOND_JACOBI, 1e-6))
    c.set_iteration(-1)
    R, _ = c.residual()
    c.pcg_form(-1)
    c.tangent(lib.MIXED)
    return m, c, R


@pytest.mark.parametrize("dims", [(27, 26, 26), (37, 29, 23), (48, 48, 16), (50, 48, 30), (200, 21, 18), (53, 47, 41), (71, 63, 59), (69, 70, 65), (73, 75, 70)])
def test_hybrid_solve_equals_the_streamed_solve(dims):
    m, c, R = _system(dims)
    # unit material, stiffness ratio of the layers' count squared at most:
    # condition number below 1e6 for the longest side, and the error in the
    # energy norm below sqrt(condition) times the residual tolerance
    tol, bound = 1e-6, 1e-3
    for precond in (lib.PRECOND_JACOBI, lib.PRECOND_BLOCK_JACOBI):
        du, its, rr, rc = c.pcg(R, rel_tol=tol, max_it=5000, precond=precond)
        assert rc == 0 and rr <= tol
        before = c.launches
        again = c.pcg(R, rel_tol=tol, max_it=5000, precond=precond)
        # one launch for the whole solve, or a streamed one past the largest
        assert (c.launches - before < 10) == (dims[0] * dims[1] * dims[2] < 350000)
        assert np.array_equal(again[0], du) and again[1] == its  # bitwise repeatable
        c.pcg_form(1)
        du1, its1, _, rc1 = c.pcg(R, rel_tol=tol, max_it=5000, precond=precond)
        c.pcg_form(-1)
        c.tangent(lib.MIXED)
        assert rc1 == 0
        assert np.abs(du - du1).max() <= bound * np.abs(du1).max()
        assert abs(its - its1) <= max(3, 0.05 * its1)
        # cut short: the iterate of the limit, reported as such
        _, cut, _, rc2 = c.pcg(R, rel_tol=tol, max_it=7, precond=precond)
        assert cut == 7 and rc2 != 0



def test_contexts_on_two_threads():
    # two cooperative launches at a time, each of every SM
    import threading

    systems = [_system((37, 29, 23)), _system((50, 48, 30))]
    alone = [c.pcg(R, rel_tol=1e-6, max_it=5000) for _, c, R in systems]
    got = [[], []]

    def work(i):
        _, c, R = systems[i]
        for _ in range(6):
            got[i].append(c.pcg(R, rel_tol=1e-6, max_it=5000))

    threads = [threading.Thread(target=work, args=(i,)) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for i in range(2):
        assert len(got[i]) == 6
        for du, its, _, rc in got[i]:
            assert rc == 0 and its == alone[i][1] and np.array_equal(du, alone[i][0])
