"""The tangent by node-pair blocks (tangent_blocks.cu) against the general
kernel, at element counts around its 8 elements per CTA: FP64 of every material
it takes, St.Venant groups in both precisions, groups of several blocks."""
import numpy as np
import pytest

from tahoe_gb300 import lib
from tahoe_gb300.meshgen import BoxMesh, equations
from tahoe_gb300.model import material_params

pytestmark = pytest.mark.gpu

MATS = {
    "simo": (lib.TOTAL_LAGRANGIAN, [{"kind": "fs_simo", "mu": 1.0, "kappa": 10.0},
                                    {"kind": "fs_simo", "mu": 10.0, "kappa": 3.0}], 0.08),
    "stvenant": (lib.TOTAL_LAGRANGIAN, [{"kind": "fs_stvenant", "E": 100.0, "nu": 0.3},
                                        {"kind": "fs_stvenant", "E": 30.0, "nu": 0.1}], 0.08),
    "j2": (lib.SMALL_STRAIN, [{"kind": "ss_j2", "E": 200e3, "nu": 0.3, "a": 1000.0, "b": 250.0},
                              {"kind": "ss_hookean", "E": 70e3, "nu": 0.25}], 0.004),
    "hooke": (lib.SMALL_STRAIN, [{"kind": "ss_hookean", "E": 70e3, "nu": 0.25}], 0.004),
}


# an unused block of a material that the kernel does not take sends a group to
# the general one
OTHER = {
    "simo": {"kind": "fs_stvenant", "E": 1.0, "nu": 0.2},
    "stvenant": {"kind": "fs_simo", "mu": 1.0, "kappa": 1.0},
    "j2": {"kind": "ss_hookean", "C": np.diag([3.0, 4.0, 5.0, 1.0, 1.5, 2.0]).reshape(36)},
}
OTHER["hooke"] = OTHER["j2"]


def _context(nel, kind, general):
    formulation, mats, amplitude = MATS[kind]
    mesh = BoxMesh(nel, 1, 1, lx=nel, jitter=0.0)
    rng = np.random.default_rng(nel)
    X = mesh.X + rng.uniform(-0.15, 0.15, size=mesh.X.shape)
    c = lib.Context(0)
    c.upload(X, mesh.conn, equations(len(X), []))
    c.set_formulation(formulation)
    for b, m in enumerate(mats + [OTHER[kind]] * general):
        c.set_material(b, *material_params(m))
    c.set_blocks(np.arange(nel) % len(mats))
    c.set_u(rng.uniform(-amplitude, amplitude, size=X.shape))
    c.set_iteration(0)
    c.residual(want_vector=False)  # J2: the yielding points of this state
    return c, X


@pytest.mark.parametrize("nel", [1, 7, 8, 9, 33])
@pytest.mark.parametrize("kind,precision", [("simo", lib.FP64), ("stvenant", lib.FP64), ("stvenant", lib.MIXED),
                                            ("j2", lib.FP64), ("hooke", lib.FP64)])
def test_equals_the_general_kernel(nel, kind, precision):
    c, X = _context(nel, kind, 0)
    c.tangent(precision)
    v = c.tangent_csr()[2]
    g, _ = _context(nel, kind, 1)
    g.tangent(lib.FP64)
    ref = g.tangent_csr()[2]
    # sums of 8 points of products of at most 20 factors of order one: 200
    # roundings of 2^-53 (2^-24) of the largest entry
    eps = 2.0**-53 if precision == lib.FP64 else 2.0**-24
    assert np.abs(v - ref).max() <= 200 * eps * np.abs(ref).max()
    for epb in (2, 4):  # bitwise the same for every launch shape
        c.tangent_config(epb)
        c.tangent(precision)
        assert np.array_equal(c.tangent_csr()[2], v)
    if MATS[kind][0] == lib.TOTAL_LAGRANGIAN:  # turned inside out
        u = np.zeros(X.shape)
        u[:, 0] = -2.0 * X[:, 0]
        c.set_u(u)
        with pytest.raises(lib.TahoeError):
            c.tangent(precision)
