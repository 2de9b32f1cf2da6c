"""Waits of the solves on the chip that run out: a part's sums are not sent, and
the solve ends with an error that the host reads; the context solves on."""
import ctypes
import time

import numpy as np
import pytest

from tahoe_gb300 import lib
from tests.test_gpu_memory_short import _context

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,n,route", [(lib.FP64, 20, "chip"), (lib.MIXED, 20, "chip"),
                                               (lib.MIXED, 30, "hybrid")])
def test_a_wait_that_runs_out_ends_the_solve(precision, n, route):
    c, mesh = _context(n)
    assert c.routes(precision)[0] == route
    c.tangent(precision)
    ref = c.pcg(None, rel_tol=1e-6, max_it=4000)[0]
    limits = lib.load().tgx_wait_limits
    limits.argtypes = [ctypes.c_void_p, ctypes.c_int, ctypes.c_int]
    # 2^16 polls are 50 ms; the CTAs' other waits of the solve end with the first
    assert limits(c.h, 1 << 16, 3) == 0
    t = time.perf_counter()
    with pytest.raises(lib.TahoeError) as e:
        c.pcg(None, rel_tol=1e-6, max_it=4000)
    assert e.value.code == -5 and "wait timed out" in str(e.value)
    assert time.perf_counter() - t < 2.0
    assert limits(c.h, 1 << 21, -1) == 0
    assert np.array_equal(c.pcg(None, rel_tol=1e-6, max_it=4000)[0], ref)
