"""FP64 element forces of total-Lagrangian Simo groups (residual_tl.cu) against
extended precision on the host: one element, partly filled CTAs (8 elements
each), odd sides, several material blocks, large and vanishing deformation, and
the points that are refused."""
import numpy as np
import pytest

from tahoe_gb300 import lib
from tahoe_gb300.meshgen import BoxMesh
from tahoe_gb300.model import SolidModel

pytestmark = pytest.mark.gpu

S = np.array([[-1, -1, -1], [1, -1, -1], [1, 1, -1], [-1, 1, -1],
              [-1, -1, 1], [1, -1, 1], [1, 1, 1], [-1, 1, 1]], dtype=np.longdouble)


def _forces(X, conn, u, mu, kappa):
    """Nodal internal forces and the sum of their terms' magnitudes."""
    L = np.longdouble
    f, scale = np.zeros(X.shape, L), np.zeros(X.shape, L)
    Xe, Ue = X.astype(L)[conn], u.astype(L)[conn]
    g = 1 / np.sqrt(L(3))
    for p in range(8):
        n = 1 + g * S[p] * S                             # [8, 3]
        dN = np.stack([S[:, 0] * n[:, 1] * n[:, 2], S[:, 1] * n[:, 0] * n[:, 2], S[:, 2] * n[:, 0] * n[:, 1]], 1) / 8
        J0 = np.einsum("eai,ak->eik", Xe, dN)
        cof = lambda A: np.stack([np.cross(A[:, 1], A[:, 2]), np.cross(A[:, 2], A[:, 0]), np.cross(A[:, 0], A[:, 1])], 1)
        C0 = cof(J0)
        det0 = (J0[:, 0] * C0[:, 0]).sum(1)
        grad = np.einsum("ak,eik->eai", dN, C0 / det0[:, None, None])  # dN/dX = dN/dxi J0^-1
        F = np.eye(3, dtype=L) + np.einsum("eai,eal->eil", Ue, grad)
        C = cof(F)
        J = (F[:, 0] * C[:, 0]).sum(1)
        b = np.einsum("eil,ejl->eij", F, F)
        dev = b - np.eye(3) * (np.trace(b, axis1=1, axis2=2) / 3)[:, None, None]
        sig = (mu / J * J ** (-L(2) / 3))[:, None, None] * dev + np.eye(3) * (kappa / 2 * (J - 1 / J))[:, None, None]
        Q = np.einsum("eij,ejl->eil", sig, C) * det0[:, None, None]
        fe = np.einsum("eil,eal->eai", Q, grad)
        size = ((mu + kappa) * (1 + np.abs(F).max((1, 2)) ** 3 / J) * det0)[:, None, None] * np.abs(grad).sum(2)[:, :, None]
        np.add.at(f, conn, fe)
        np.add.at(scale, conn, np.broadcast_to(size, fe.shape))
    return f, scale


def _model(dims, nblocks=1):
    mesh = BoxMesh(*dims, jitter=0.2, seed=3)
    kinds = [{"kind": "fs_simo", "mu": 1.0 + b, "kappa": 10.0 / (1 + b)} for b in range(nblocks)]
    blk = np.arange(len(mesh.conn), dtype=np.int32) % nblocks
    m = SolidModel(mesh.X, mesh.conn, "total_lagrangian", kinds, blocks=blk if nblocks > 1 else None)
    m.set_schedule([(0.0, 1.0)])
    m.setup()
    mu = np.array([k["mu"] for k in kinds], dtype=np.longdouble)[blk]
    kappa = np.array([k["kappa"] for k in kinds], dtype=np.longdouble)[blk]
    return mesh, m, mu, kappa


@pytest.mark.parametrize("dims", [(1, 1, 1), (3, 1, 1), (2, 2, 2), (3, 3, 1), (7, 5, 3), (13, 9, 8)])
@pytest.mark.parametrize("size", [1e-7, 0.05, 0.15])
@pytest.mark.parametrize("nblocks", [1, 3])
def test_forces_against_extended_precision(dims, size, nblocks):
    mesh, m, mu, kappa = _model(dims, nblocks)
    X = np.asarray(mesh.X).reshape(-1, 3)
    u = size / max(dims) * np.random.default_rng(5).standard_normal(X.shape) * 0.5
    m.ctx.set_u(u)
    R, _ = m.ctx.residual(precision=lib.FP64)
    f, scale = _forces(X, np.asarray(mesh.conn), u, mu, kappa)
    # about 200 roundings of 2^-53 on terms no larger than the scale
    assert (np.abs(-R.reshape(-1, 3) - f) <= 200 * 2.0**-53 * scale).all()


def test_rigid_motion_and_refused_points():
    mesh, m, _, _ = _model((5, 4, 3))
    X = np.asarray(mesh.X).reshape(-1, 3)
    m.ctx.set_u(np.full(X.shape, 3.5))
    R, _ = m.ctx.residual(precision=lib.FP64)
    assert np.abs(R).max() <= 200 * 2.0**-53 * 11.0
    u = np.zeros(X.shape)
    u[:, 0] = -2.0 * X[:, 0]  # mirrored: det F = -1 everywhere
    m.ctx.set_u(u)
    with pytest.raises(lib.TahoeError):
        m.ctx.residual(precision=lib.FP64)
    u[:, 0] = np.nan
    m.ctx.set_u(u)
    with pytest.raises(lib.TahoeError):
        m.ctx.residual(precision=lib.FP64)
    m.ctx.set_u(np.zeros(X.shape))
    R, _ = m.ctx.residual(precision=lib.FP64)
    assert np.abs(R).max() <= 200 * 2.0**-53 * 11.0
