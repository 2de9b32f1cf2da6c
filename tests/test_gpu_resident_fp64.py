"""FP64 resident solves whose CTAs keep a chunk of every warp in tensor memory:
batches of RVEs around the sizes where a second chunk a warp begins and where a
cluster grows to the largest the chip holds as many of, against one solve of
each RVE alone, and single meshes up to the capacity."""
import numpy as np
import pytest

from tahoe_gb300 import lib, rve

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sides", [(5, 6, 7), (8, 9), (10, 11), (12, 13, 4), (16,)])
def test_batch_equals_solves_alone(sides):
    rng = np.random.default_rng(2)
    Fs = np.eye(3) + 0.02 * rng.standard_normal((len(sides), 3, 3))
    ctx = lib.Context(0)
    res = rve.ResidentRVEs(ctx)
    kw = dict(precision=lib.FP64, precond=lib.PRECOND_BLOCK_JACOBI, rel_tol=1e-10)
    P = res.solve(np.array(sides), Fs, **kw)[3]
    C = ctx.macro_tangent(precision=lib.FP64, precond=lib.PRECOND_BLOCK_JACOBI, lin_rel_tol=1e-11)[0]
    for i, n in enumerate(sides):
        one = rve.ResidentRVEs(lib.Context(0))
        P1 = one.solve(np.array([n]), Fs[i:i + 1], **kw)[3]
        C1 = one.ctx.macro_tangent(precision=lib.FP64, precond=lib.PRECOND_BLOCK_JACOBI, lin_rel_tol=1e-11)[0]
        # both within 1e-10 of the equilibrium, and 1e-11 of the columns
        assert np.abs(P[i] - P1[0]).max() <= 1e-8 * np.abs(P1).max()
        assert np.abs(C[i] - C1[0]).max() <= 1e-8 * np.abs(C1).max()
