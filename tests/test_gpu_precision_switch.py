"""Solves of one context in FP64 and mixed precision in turn: every form's
captured iterations go with the vectors that they name."""
import numpy as np
import pytest

from tahoe_gb300 import lib, rve

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("side", [8, 31])
def test_streamed_batch_after_a_solve_on_the_chip(side):
    """A batch whose FP64 solves are streamed (side 31: too large for the chip;
    side 8: the one-system solver's turn between two per-RVE ones): the FP64
    update after a mixed-precision solve is bitwise the one before it."""
    b = rve.RVEBatch([side, 5], [rve.sample_F(np.random.default_rng(i)) for i in range(2)])
    c = b.setup()
    if side == 8:
        c.pcg_form(3)
    c.set_prescribed(b.prescribed_idx, 0.1 * b.prescribed_val)
    c.residual(want_vector=False)

    def solve(precision):
        c.tangent(precision)
        return c.pcg(None, rel_tol=1e-6, max_it=4000)[0]

    ref = solve(lib.FP64)
    for _ in range(2):
        if side == 8:
            c.segment_solver(False)
        other = solve(lib.MIXED)
        c.segment_solver(True)
        assert np.abs(other - ref).max() < 1e-2 * np.abs(ref).max()
        assert np.array_equal(solve(lib.FP64), ref)
