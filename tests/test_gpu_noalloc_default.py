"""tg_pcg_solve_noalloc after a tangent of the default form, which needs no matrix
storage itself: the call finds its bytes reserved."""
import numpy as np
import pytest

from tahoe_gb300 import lib
from tests.memory import ShortMemory
from tests.test_gpu_memory_short import _context

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [lib.FP64, lib.MIXED])
@pytest.mark.parametrize("n", [8, 30])
def test_first_call_allocates_nothing(precision, n):
    torch = pytest.importorskip("torch")
    c, mesh = _context(n)
    R, _ = c.residual()
    d_rhs = torch.tensor(R, device="cuda:0")
    d_du = torch.zeros_like(d_rhs)
    torch.cuda.synchronize()
    c.tangent(precision)
    with ShortMemory(left=1):
        its, _, rc = c.pcg_noalloc(d_rhs.data_ptr(), d_du.data_ptr(), rel_tol=1e-6, max_it=4000)
    assert rc == 0 and its > 0
    c.pcg_form(0)
    ref = c.pcg(R, rel_tol=1e-6, max_it=4000)[0]
    assert np.abs(d_du.cpu().numpy() - ref).max() <= 1e-12 * np.abs(ref).max()
