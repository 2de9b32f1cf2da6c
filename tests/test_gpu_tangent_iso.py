"""The tangent kernel of the isotropic moduli (tangent_iso.cu) against the FP64
element matrices of the general kernel, at element counts around its 32
elements per CTA, for every material it takes and for groups that mix them.
"""
import numpy as np
import pytest

from tahoe_gb300 import lib
from tahoe_gb300.meshgen import BoxMesh, equations
from tahoe_gb300.model import material_params

pytestmark = pytest.mark.gpu

SIMO = [{"kind": "fs_simo", "mu": 1.0, "kappa": 10.0}, {"kind": "fs_simo", "mu": 10.0, "kappa": 3.0}]
SMALL = [{"kind": "ss_j2", "E": 200e3, "nu": 0.3, "a": 1000.0, "b": 250.0}, {"kind": "ss_hookean", "E": 70e3, "nu": 0.25}]


def _context(nel, formulation, mats, amplitude):
    mesh = BoxMesh(nel, 1, 1, lx=nel, jitter=0.0)
    rng = np.random.default_rng(nel)
    X = mesh.X + rng.uniform(-0.15, 0.15, size=mesh.X.shape)
    c = lib.Context(0)
    c.upload(X, mesh.conn, equations(len(X), []))
    c.set_formulation(formulation)
    for b, m in enumerate(mats):
        c.set_material(b, *material_params(m))
    c.set_blocks(np.arange(nel) % len(mats))
    c.set_u(rng.uniform(-amplitude, amplitude, size=X.shape))
    c.set_iteration(0)
    c.residual(want_vector=False)  # J2: the yielding points of this state
    return c


@pytest.mark.parametrize("nel", [1, 31, 32, 33, 65])
@pytest.mark.parametrize("kind", ["simo", "j2", "hooke"])
def test_mixed_tangent_equals_fp64_element_matrices(nel, kind):
    form, mats, amp = {"simo": (lib.TOTAL_LAGRANGIAN, SIMO, 0.08), "j2": (lib.SMALL_STRAIN, SMALL, 0.004),
                       "hooke": (lib.SMALL_STRAIN, SMALL[1:], 0.004)}[kind]
    c = _context(nel, form, mats, amp)
    if kind == "j2" and nel > 1:
        flags = c.active_set()
        assert (flags == lib.J2_PLASTIC).any()  # the plastic branch takes part
    c.tangent(lib.MIXED)
    _, _, v32 = c.tangent_csr()
    c.tangent(lib.FP64)  # the general kernel
    _, _, v64 = c.tangent_csr()
    # FP32 sums of 8 points of products of at most 10 factors of order one:
    # 100 roundings of 6e-8 at most, of the largest entry
    assert np.abs(v32 - v64).max() <= 6e-6 * np.abs(v64).max()


def test_inverted_element_is_reported():
    c = _context(40, lib.TOTAL_LAGRANGIAN, SIMO, 0.05)
    u = np.zeros((c.nnd, 3))
    u[20, 0] = 3.0
    c.set_u(u)
    with pytest.raises(lib.TahoeError) as ei:
        c.tangent(lib.MIXED)
    assert ei.value.code == -4
    c.set_u(0.0 * u)
    c.tangent(lib.MIXED)  # the context stays usable


def test_other_groups_keep_the_general_kernel():
    # an anisotropic Hookean block in the group, and B-bar
    C = np.diag([3.0, 4.0, 5.0, 1.0, 1.5, 2.0])
    for mats, bbar in (([SMALL[1], {"kind": "ss_hookean", "C": C.reshape(36)}], 0), ([SMALL[1]], 1)):
        c = _context(35, lib.SMALL_STRAIN, mats, 0.004)
        c.set_strain_displacement(bbar)
        c.tangent(lib.MIXED)
        _, _, v32 = c.tangent_csr()
        c.tangent(lib.FP64)
        _, _, v64 = c.tangent_csr()
        assert np.abs(v32 - v64).max() <= 6e-6 * np.abs(v64).max()
