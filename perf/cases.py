"""Performance cases of the hex8 solid path: the work a user has it do.

Each case is one call sequence of a user's program through the public entry
points (``tahoe_gb300.model``, ``rve``, ``serve``, ``lib.Context``):

  rve     a batch of FE^2 microscale RVEs composed from resident templates,
          affine predictor and Newton per RVE, averaged stresses (and the
          consistent macro tangent): one macroscopic iteration's worth of
          points.  Mixed precision is the production form, FP64 the plain one.
  serve   a burst of RVE requests through the library's request loop.
  step    one finite-strain load step of a jittered block (prescribed
          compression through the predictor, then full Newton), displacements
          back on the host.
  static  one small-strain step under a surface traction (Newton with tight
          CG, as a deck asks for).
  j2      one load step of a small-strain J2 plate and its nodal output
          (stresses, equivalent plastic strain) as a ``.run`` file holds it.
  force   a residual evaluation for a host-driven solver: displacements in,
          residual vector out.

``exact`` solves the same problems in FP64 with plain torch (element matrices
from forward-mode derivatives of the stress, conjugate gradients), without
this repository's code.
"""
import numpy as np
import torch

FP64, MIXED = 0, 1
JACOBI, BLOCK_JACOBI = 0, 1

HOOKE = {"kind": "ss_hookean", "E": 200e3, "nu": 0.3}
SIMO = {"kind": "fs_simo", "mu": 1.0, "kappa": 10.0}
STVENANT = {"kind": "fs_stvenant", "E": 100.0, "nu": 0.25}
J2 = {"kind": "ss_j2", "E": 200e3, "nu": 0.3, "a": 1000.0, "b": 250.0}
RVE_MATRIX = {"kind": "fs_simo", "mu": 1.0, "kappa": 10.0}
RVE_INCLUSION = {"kind": "fs_simo", "mu": 10.0, "kappa": 100.0}
MATERIAL = {"simo": SIMO, "stvenant": STVENANT, "hooke": HOOKE, "j2": J2}


def listed():
    return [
        # one macroscopic Gauss point's RVE (or one lone request): launches and latency
        dict(name="rve_1_n8", kind="rve", count=1, nmin=8, nmax=8, mix=0, precision=MIXED, precond=BLOCK_JACOBI,
             macro=False),
        # a served batch: the sides of the request stream, log-uniform 4..24
        dict(name="rve_64_served", kind="rve", count=64, nmin=4, nmax=24, mix=1, precision=MIXED,
             precond=BLOCK_JACOBI, macro=False),
        # the FE^2 batch at full size: every macroscopic point of an iteration at once
        dict(name="rve_4096", kind="rve", count=4096, nmin=4, nmax=16, mix=2, precision=MIXED, precond=JACOBI,
             macro=False),
        # plain FP64 with the consistent tangent a macroscopic Newton iteration needs
        dict(name="rve_48_fp64_macro", kind="rve", count=48, nmin=4, nmax=12, mix=3, precision=FP64,
             precond=BLOCK_JACOBI, macro=True),
        # requests arriving together at the request loop (four lanes)
        dict(name="serve_192", kind="serve", count=192, nmin=4, nmax=24, mix=4, lanes=4),
        # the flagship load step: 64^3 block, 823,875 dofs
        dict(name="step_64", kind="step", nx=64, ny=64, nz=64, material="simo", precision=MIXED, precond=JACOBI),
        # an ordinary component-sized mesh with odd sides
        dict(name="step_37x29x23", kind="step", nx=37, ny=29, nz=23, material="simo", precision=MIXED,
             precond=BLOCK_JACOBI),
        # a plain FP64 deck: St.Venant, tight linear solves
        dict(name="step_fp64_19x14x11", kind="step", nx=19, ny=14, nz=11, material="stvenant", precision=FP64,
             precond=JACOBI),
        # the small linear deck: 16^3 cube under traction, FP64 CG
        dict(name="static_16", kind="static", nx=16, ny=16, nz=16, precision=FP64),
        # a plate load step with history and nodal output
        dict(name="j2_48x48x24", kind="j2", nx=48, ny=48, nz=24),
        # residuals for a solver on the host side of the boundary
        dict(name="force_fp64_45x40x33", kind="force", nx=45, ny=40, nz=33, material="simo", precision=FP64),
        dict(name="force_mixed_9x8x7", kind="force", nx=9, ny=8, nz=7, material="simo", precision=MIXED),
    ]


def _log_int(rng, lo, hi):
    return int(round(np.exp(rng.uniform(np.log(lo), np.log(hi)))))


def draw(rng):
    kind = rng.choice(["rve", "rve", "rve", "serve", "step", "step", "step", "static", "j2", "force"])
    if kind == "rve":
        nmin = rng.choice([4, 4, 5, 6])
        nmax = max(nmin, rng.choice([7, 9, 12, 16, 24]))
        precision = rng.choice([MIXED, MIXED, MIXED, FP64])
        macro = precision == FP64 and rng.random() < 0.5
        count = _log_int(rng, 1, (2500 if nmax <= 16 else 600) if precision == MIXED else 90)
        return dict(kind=kind, count=count, nmin=nmin, nmax=nmax, mix=rng.randrange(1, 10000), precision=precision,
                    precond=rng.choice([JACOBI, BLOCK_JACOBI]), macro=macro)
    if kind == "serve":
        return dict(kind=kind, count=_log_int(rng, 2, 400), nmin=4, nmax=rng.choice([12, 16, 24]),
                    mix=rng.randrange(1, 10000), lanes=rng.choice([2, 4]))
    if kind == "step":
        precision = rng.choice([MIXED, MIXED, FP64])
        top = 64 if precision == MIXED else 28
        n = _log_int(rng, 4, top)
        material = "simo" if precision == MIXED else rng.choice(["simo", "stvenant"])
        side = lambda: max(3, min(top, int(round(n * rng.uniform(0.75, 1.25)))))  # noqa: E731
        return dict(kind=kind, nx=side(), ny=side(), nz=side(), material=material, precision=precision,
                    precond=rng.choice([JACOBI, BLOCK_JACOBI]))
    n = _log_int(rng, 4, {"static": 28, "j2": 40, "force": 56}[kind])
    side = lambda: max(3, int(round(n * rng.uniform(0.75, 1.25))))  # noqa: E731
    if kind == "static":
        return dict(kind=kind, nx=side(), ny=side(), nz=side(), precision=rng.choice([FP64, FP64, MIXED]))
    if kind == "j2":
        return dict(kind=kind, nx=max(6, side()), ny=max(6, side()), nz=max(3, side() // 2))
    return dict(kind=kind, nx=side(), ny=side(), nz=side(), material=rng.choice(["simo", "simo", "stvenant"]),
                precision=rng.choice([FP64, MIXED]))


# ---- inputs (shared by prepare and exact) ---------------------------------

def _sides(case):
    """RVE sides of a batch: fixed by the case (uniform for the FE^2 batch,
    log-uniform where the range reaches the request stream's 24)."""
    rng = np.random.default_rng(case["mix"])
    lo, hi, k = case["nmin"], case["nmax"], case["count"]
    if hi > 16:
        ns = np.floor(np.exp(rng.uniform(np.log(lo), np.log(hi + 1), size=k))).astype(np.int64)
        return np.clip(ns, lo, hi)
    return rng.integers(lo, hi + 1, size=k)


def _defgrads(count, seed):
    """F = I + 0.05 S, S symmetric with entries U(-1, 1)."""
    rng = np.random.default_rng(seed)
    A = rng.uniform(-1.0, 1.0, size=(count, 3, 3))
    S = np.triu(A) + np.transpose(np.triu(A, 1), (0, 2, 1))
    return np.eye(3) + 0.05 * S


def _box(nx, ny, nz, lx, ly, lz, jitter, seed):
    """Structured hex8 box, nodes x-fastest; interior nodes jittered."""
    xs, ys, zs = (np.linspace(0.0, l, n + 1) for l, n in ((lx, nx), (ly, ny), (lz, nz)))
    Z, Y, Xg = np.meshgrid(zs, ys, xs, indexing="ij")
    X = np.stack([Xg.ravel(), Y.ravel(), Z.ravel()], axis=1)
    K, J, I = np.meshgrid(np.arange(nz + 1), np.arange(ny + 1), np.arange(nx + 1), indexing="ij")
    ijk = np.stack([I.ravel(), J.ravel(), K.ravel()], axis=1)
    if jitter:
        inner = ((ijk > 0) & (ijk < np.array([nx, ny, nz]))).all(axis=1)
        d = np.random.default_rng(seed).uniform(-jitter, jitter, size=X.shape)
        X = X + d * np.array([lx / nx, ly / ny, lz / nz]) * inner[:, None]
    k, j, i = np.meshgrid(np.arange(nz), np.arange(ny), np.arange(nx), indexing="ij")
    i, j, k = i.ravel(), j.ravel(), k.ravel()
    nid = lambda a, b, c: a + (nx + 1) * (b + (ny + 1) * c)  # noqa: E731
    conn = np.stack([nid(i, j, k), nid(i + 1, j, k), nid(i + 1, j + 1, k), nid(i, j + 1, k), nid(i, j, k + 1),
                     nid(i + 1, j, k + 1), nid(i + 1, j + 1, k + 1), nid(i, j + 1, k + 1)], axis=1).astype(np.int32)
    return X, conn, ijk


def _block(case, seed):
    """Mesh, prescribed dofs (node, dof, value) and nodal loads of a single-mesh case."""
    n = (case["nx"], case["ny"], case["nz"])
    kind = case["kind"]
    h = 1.0 / max(n)
    lx, ly, lz = (v * h for v in n)
    X, conn, ijk = _box(*n, lx, ly, lz, 0.0 if kind == "j2" else 0.2, seed)
    rng = np.random.default_rng(seed + 1)
    kbc, tractions = [], []
    if kind == "j2":
        # one side clamped, the other gripped and pulled in x
        pull = 0.001 * lx * rng.uniform(0.9, 1.05)
        for a in np.nonzero(ijk[:, 0] == 0)[0]:
            kbc += [(a, 0, 0.0), (a, 1, 0.0), (a, 2, 0.0)]
        for a in np.nonzero(ijk[:, 0] == n[0])[0]:
            kbc += [(a, 0, pull), (a, 1, 0.0), (a, 2, 0.0)]
        return X, conn, kbc, tractions
    for a in np.nonzero(ijk[:, 2] == 0)[0]:
        kbc += [(a, 0, 0.0), (a, 1, 0.0), (a, 2, 0.0)]
    if kind == "static":
        e = np.arange(conn.shape[0])[-n[0] * n[1]:]  # the top layer, facet z+
        t = np.array([0.0, 0.0, 1.0]) + 0.2 * rng.uniform(-1.0, 1.0, size=3)
        tractions = [(int(k), 1, list(t)) for k in e]
    elif kind == "step":
        for a in np.nonzero(ijk[:, 2] == n[2])[0]:
            kbc.append((a, 2, -0.01 * lz))
    return X, conn, kbc, tractions


def _field(X, seed):
    """A smooth displacement of a few percent strain."""
    rng = np.random.default_rng(seed + 2)
    u = np.zeros_like(X)
    for _ in range(3):
        k, a, ph = rng.uniform(-3, 3, size=3), rng.uniform(-0.01, 0.01, size=3), rng.uniform(0, 6)
        u += np.sin(X @ k + ph)[:, None] * a
    return u


# ---- the user's program -----------------------------------------------------

def prepare(case, seed):
    from tahoe_gb300 import lib, rve, serve
    from tahoe_gb300.model import SolidModel
    kind = case["kind"]
    if kind == "rve":
        ctx = lib.Context(0)
        res = rve.ResidentRVEs(ctx)
        ns = _sides(case)
        for n in np.unique(ns):
            res.template_id(int(n))
        return dict(case=case, res=res, ns=ns, Fs=_defgrads(len(ns), seed))
    if kind == "serve":
        server = serve.NativeServer(lanes=case["lanes"], max_batch=64)
        ns = _sides(case)
        return dict(case=case, server=server, ns=ns, Fs=_defgrads(len(ns), seed), at=np.zeros(len(ns)))
    X, conn, kbc, tractions = _block(case, seed)
    form = "small_strain" if kind in ("static", "j2") else "total_lagrangian"
    material = MATERIAL[case.get("material", "hooke" if kind == "static" else "j2")]
    m = SolidModel(X, conn, form, material)
    m.set_schedule([(0.0, 0.0), (1.0, 1.0)])
    for a, d, v in kbc:
        m.add_kbc(a, d, v, v != 0.0)
    for e, f, t in tractions:
        m.add_traction(e, f, t)
    ctx = m.setup()
    if kind == "force":
        return dict(case=case, ctx=ctx, model=m, u=_field(X, seed))
    ctx.checkpoint()
    return dict(case=case, ctx=ctx, model=m)


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "rve":
        res = state["res"]
        rc, rep, rel, P = res.solve(state["ns"], state["Fs"], precision=case["precision"], precond=case["precond"],
                                    rel_tol=1e-9)
        out = dict(P=P, status=res.status)
        if case["macro"]:
            out["C"], _ = res.ctx.macro_tangent(precision=case["precision"], precond=case["precond"],
                                                lin_rel_tol=1e-11)
        return out
    if kind == "serve":
        r = state["server"].run(state["at"], state["ns"], state["Fs"])
        return dict(P=r["P"], status=r["status"])
    ctx = state["ctx"]
    if kind == "force":
        ctx.set_u(state["u"])
        R, norm = ctx.residual(precision=case["precision"])
        return dict(R=R, norm=norm)
    m = state["model"]
    ctx.rollback()
    if kind == "step":
        lin = 1e-4 if case["precision"] == MIXED else 1e-8
        m.apply_step(1.0, (case["precision"], case["precond"], lin))
        ctx.newton(rel_tol=1e-8, abs_tol=0.0, div_tol=10.0, max_iterations=20, precision=case["precision"],
                   precond=case["precond"], lin_rel_tol=lin)
        return dict(u=ctx.get_u())
    if kind == "static":
        m.apply_step(1.0)
        ctx.newton(rel_tol=1e-10, abs_tol=0.0, max_iterations=10, precision=case["precision"],
                   lin_rel_tol=1e-11 if case["precision"] == FP64 else 1e-4)
        return dict(u=ctx.get_u(), stress=ctx.nodal_stress())
    # j2
    ctx.reset_step()
    m.apply_step(1.0, (MIXED, JACOBI, 1e-4))
    ctx.newton(rel_tol=1e-10, abs_tol=0.0, div_tol=1e3, max_iterations=30, precision=MIXED, lin_rel_tol=1e-4)
    return dict(u=ctx.get_u(), stress=ctx.nodal_stress(), material=ctx.nodal_material_output())


# ---- the work no implementation can do without ------------------------------

def work(case):
    """Bytes and operations of one pass: the mesh in, the results out, and per
    Newton iteration the element matrices (25 kflop each with the stress) and
    a conjugate-gradient solve whose iterations read the upper half of the
    block matrix once.  CG iterations by side: about 9 per element across for
    1e-4 (3 times that for the tight FP64 solves)."""
    kind = case["kind"]
    if kind in ("rve", "serve"):
        ns = _sides(case).astype(float)
        size = 8 if case.get("precision") == FP64 else 4
        nel, nnd = ns ** 3, (ns + 1) ** 3
        passes, its = 4, 30 + 3 * ns
        flops = (passes * (nel * 25e3 + its * nnd * 27 * 18)).sum()
        byts = (passes * its * nnd * 14 * 9 * size + nnd * 24 + nel * 32).sum() + len(ns) * 144
        if case.get("macro"):
            flops += (9 * 3 * its * nnd * 27 * 18).sum()
            byts += (3 * its * nnd * 14 * 9 * size).sum() + len(ns) * 648
        return dict(bytes=float(byts), flops=float(flops))
    n = (case["nx"], case["ny"], case["nz"])
    nel, nnd = n[0] * n[1] * n[2], (n[0] + 1) * (n[1] + 1) * (n[2] + 1)
    mesh = nnd * 24 + nel * 32
    if kind == "force":
        return dict(bytes=float(mesh + nnd * 48), flops=float(nel * 8 * 400))
    passes, tight = {"step": (4, 1), "static": (1, 3), "j2": (8, 1)}[kind]
    if case.get("precision") == FP64:
        tight = 3
    size = 8 if case.get("precision") == FP64 else 4
    its = 9 * max(n) * tight
    return dict(bytes=float(mesh + nnd * 24 + passes * its * nnd * 14 * 9 * size),
                flops=float(passes * (nel * 25e3 + its * nnd * 27 * 18)))


# ---- the same in FP64 with plain torch --------------------------------------

_G = 1.0 / np.sqrt(3.0)
_S = np.array([[-1, -1, -1], [1, -1, -1], [1, 1, -1], [-1, 1, -1], [-1, -1, 1], [1, -1, 1], [1, 1, 1], [-1, 1, 1]],
              dtype=float)


def _gradients(X, conn):
    """dN/dX (nel, 8 points, 8 nodes, 3) and det J (nel, 8)."""
    dN = np.zeros((8, 8, 3))
    for p in range(8):
        f = 1.0 + _G * _S[p] * _S  # (8, 3)
        for d in range(3):
            o = [k for k in range(3) if k != d]
            dN[p, :, d] = 0.125 * _S[:, d] * f[:, o[0]] * f[:, o[1]]
    dN = torch.from_numpy(dN).to(X)
    J = torch.einsum("eai,pak->epik", X[conn], dN)
    return torch.einsum("pak,epkl->epal", dN, torch.linalg.inv(J)), torch.linalg.det(J)


def _cofactor(F):
    a, b, c = F[..., 0, :], F[..., 1, :], F[..., 2, :]
    return torch.stack([torch.linalg.cross(b, c), torch.linalg.cross(c, a), torch.linalg.cross(a, b)], dim=-2)


def _stress(kind, H, p):
    """First Piola-Kirchhoff stress (Cauchy for small strain) of one point from
    the displacement gradient, and the equivalent plastic strain."""
    eye = torch.eye(3, dtype=H.dtype, device=H.device)
    zero = H.sum() * 0.0
    if kind in ("ss_hookean", "ss_j2"):
        eps = 0.5 * (H + H.transpose(-1, -2))
        E, nu = p[0], p[1]
        mu, lam = 0.5 * E / (1 + nu), E * nu / ((1 + nu) * (1 - 2 * nu))
        tr = eps.diagonal().sum()
        s = 2 * mu * eps + lam * tr * eye
        if kind == "ss_hookean":
            return s, zero
        rel = 2 * mu * (eps - tr / 3 * eye)
        nr = torch.sqrt((rel * rel).sum() + 1e-60)
        f = nr - (2.0 / 3.0) ** 0.5 * p[3]
        dg = torch.where(f > 1e-10, 0.5 * f / (mu + p[2] / 3), zero)
        return s - 2 * mu * dg * rel / nr, (2.0 / 3.0) ** 0.5 * dg
    F = H + eye
    cof = _cofactor(F)
    J = (F[0] * cof[0]).sum()
    if kind == "fs_stvenant":
        E, nu = p[0], p[1]
        mu, lam = 0.5 * E / (1 + nu), E * nu / ((1 + nu) * (1 - 2 * nu))
        C = 0.5 * (F.transpose(-1, -2) @ F - eye)
        return F @ (2 * mu * C + lam * C.diagonal().sum() * eye), zero
    b = F @ F.transpose(-1, -2)
    bb = J ** (-2.0 / 3.0) * b
    s = p[0] / J * (bb - bb.diagonal().sum() / 3 * eye) + 0.5 * p[1] * (J - 1 / J) * eye
    return s @ cof, zero  # J sigma F^-T


class _Exact:
    """Newton with conjugate gradients on one (possibly disconnected) mesh."""

    def __init__(self, X, conn, materials, blocks, fixed):
        self.dev = "cuda" if torch.cuda.is_available() else "cpu"
        t = lambda a, d=torch.float64: torch.as_tensor(np.asarray(a), dtype=d, device=self.dev)  # noqa: E731
        self.X, self.conn = t(X), t(conn, torch.int64)
        self.free = torch.ones_like(self.X)
        self.free.view(-1)[t(fixed, torch.int64)] = 0.0
        self.materials = materials
        self.block = t(np.zeros(len(conn)) if blocks is None else blocks, torch.int64)
        self.g, self.w = _gradients(self.X, self.conn)
        self.u = torch.zeros_like(self.X)
        self.fext = torch.zeros_like(self.X)

    def _params(self, m):
        return {"ss_hookean": ("E", "nu"), "fs_stvenant": ("E", "nu"), "fs_simo": ("mu", "kappa"),
                "ss_j2": ("E", "nu", "a", "b")}[m["kind"]]

    def points(self, tangent):
        """Stress (and moduli) of every point at the current displacements."""
        H = torch.einsum("eai,epal->epil", self.u[self.conn], self.g)
        P = torch.empty_like(H)
        al = torch.empty_like(self.w)
        A = torch.empty(H.shape + (3, 3), dtype=H.dtype, device=H.device) if tangent else None
        for b, m in enumerate(self.materials):
            sel = torch.nonzero(self.block == b)[:, 0]
            p = [float(m[k]) for k in self._params(m)]
            f = lambda h: _stress(m["kind"], h, p)  # noqa: E731, B023
            for part in sel.split(1 << 15):
                h = H[part].reshape(-1, 3, 3)
                s, a = torch.func.vmap(f)(h)
                P[part], al[part] = s.reshape(-1, 8, 3, 3), a.reshape(-1, 8)
                if tangent:
                    d = torch.func.vmap(torch.func.jacfwd(lambda h: f(h)[0]))(h)  # noqa: B023
                    A[part] = d.reshape(-1, 8, 3, 3, 3, 3)
        return H, P, al, A

    def forces(self, P):
        return torch.einsum("ep,epij,epaj->eai", self.w, P, self.g)

    def gather(self, fe):
        return torch.zeros_like(self.X).index_add_(0, self.conn.reshape(-1), fe.reshape(-1, 3))

    def residual(self):
        return self.fext - self.gather(self.forces(self.points(False)[1]))

    def set_matrix(self):
        A = self.points(True)[3]
        K = torch.empty(len(self.conn), 24, 24, dtype=self.X.dtype, device=self.dev)
        for part in torch.arange(len(self.conn), device=self.dev).split(1 << 14):
            # (i, k, J, L) moduli: half contracted, then a product over points and L
            h = torch.einsum("ep,epiJkL,epaJ->eaikpL", self.w[part], A[part], self.g[part])
            K[part] = torch.einsum("eaikpL,epbL->eaibk", h, self.g[part]).reshape(-1, 24, 24)
        self.K = K
        D = torch.zeros(len(self.X), 3, 3, dtype=self.X.dtype, device=self.dev)
        Kd = torch.diagonal(K.reshape(-1, 8, 3, 8, 3), dim1=1, dim2=3).permute(0, 3, 1, 2)
        D.index_add_(0, self.conn.reshape(-1), Kd.reshape(-1, 3, 3))
        D = D * self.free[:, :, None] * self.free[:, None, :] + torch.diag_embed(1.0 - self.free)
        self.M = torch.linalg.inv(D)

    def times(self, v):
        return self.gather(torch.bmm(self.K, v[self.conn].reshape(-1, 24, 1)))

    def solve(self, b, tol, most=20000):
        b = b * self.free
        x, r = torch.zeros_like(b), b.clone()
        z = torch.einsum("nij,nj->ni", self.M, r)
        p, rz, top = z.clone(), (r * z).sum(), float(r.norm())
        for it in range(most):
            q = self.times(p) * self.free
            a = rz / (p * q).sum()
            x += a * p
            r -= a * q
            if it % 16 == 15 and float(r.norm()) <= tol * top:
                break
            z = torch.einsum("nij,nj->ni", self.M, r)
            rz, old = (r * z).sum(), rz
            p = z + (rz / old) * p
        return x

    def step(self, v):
        """The prescribed increment through the linear response, then Newton."""
        r = self.residual()
        self.set_matrix()
        du = self.solve(r - self.times(v), 1e-6)
        self.u = self.u + v + du * self.free
        first = None
        for _ in range(40):
            r = self.residual() * self.free
            now = float(r.norm())
            first = first or max(now, float(self.forces(self.points(False)[1]).norm()))
            if now <= 2e-14 * first:
                break
            if _:
                if now > 0.5 * last:  # noqa: F821
                    break
            last = now  # noqa: F841
            self.set_matrix()
            self.u = self.u + self.solve(r, 1e-6) * self.free

    def nodal(self):
        """Cauchy stress [11, 22, 33, 23, 13, 12] and (equivalent plastic
        strain, von Mises stress, pressure) extrapolated to the element nodes
        and averaged (small strain)."""
        _, s, al, _ = self.points(False)
        tr = s.diagonal(dim1=-2, dim2=-1).sum(-1)
        dev = s - (tr / 3)[..., None, None] * torch.eye(3, dtype=s.dtype, device=self.dev)
        vm = torch.sqrt(1.5 * (dev * dev).sum((-1, -2)))
        vals = torch.stack([s[..., 0, 0], s[..., 1, 1], s[..., 2, 2], s[..., 1, 2], s[..., 0, 2], s[..., 0, 1], al, vm,
                            tr / 3], dim=-1)
        # the smoothing matrix of the element: the linear fit through the points, at the nodes
        E = torch.from_numpy((1.0 + 3.0 ** 0.5 * _S @ _S.T) / 8.0).to(vals)
        at = torch.einsum("ap,epk->eak", E, vals)
        out = torch.zeros(len(self.X), 9, dtype=vals.dtype, device=self.dev)
        out.index_add_(0, self.conn.reshape(-1), at.reshape(-1, 9))
        n = torch.zeros(len(self.X), dtype=vals.dtype, device=self.dev)
        n.index_add_(0, self.conn.reshape(-1), torch.ones(self.conn.numel(), dtype=vals.dtype, device=self.dev))
        return out / n[:, None]


def _exact_rve(case, seed):
    ns, Fs = _sides(case), _defgrads(case["count"], seed)
    Xs, conns, blocks, fixed, vs, seg, off = [], [], [], [], [], [], 0
    for s, n in enumerate(ns):
        n = int(n)
        X, conn, ijk = _box(n, n, n, 1.0, 1.0, 1.0, 0.0, 0)
        edge = ((ijk == 0) | (ijk == n)).any(axis=1)
        blocks.append((np.linalg.norm(X[conn].mean(axis=1) - 0.5, axis=1) < 0.3).astype(np.int64))
        v = X @ (Fs[s] - np.eye(3)).T * edge[:, None]
        fixed.append(((np.nonzero(edge)[0] + off)[:, None] * 3 + np.arange(3)).ravel())
        Xs.append(X)
        conns.append(conn.astype(np.int64) + off)
        vs.append(v)
        seg.append(np.full(len(conn), s))
        off += len(X)
    m = _Exact(np.concatenate(Xs), np.concatenate(conns), (RVE_MATRIX, RVE_INCLUSION), np.concatenate(blocks),
               np.concatenate(fixed))
    seg = torch.as_tensor(np.concatenate(seg), device=m.dev)
    k = len(ns)
    m.step(torch.as_tensor(np.concatenate(vs), device=m.dev))
    Xe = m.X[m.conn]

    def average(fe):
        return torch.zeros(k, 3, 3, dtype=fe.dtype, device=m.dev).index_add_(0, seg, torch.einsum("eai,eaJ->eiJ", fe, Xe))

    out = dict(P=average(m.forces(m.points(False)[1])).cpu().numpy(), status=None)
    if case.get("macro"):
        m.set_matrix()
        C = torch.zeros(k, 9, 9, dtype=m.X.dtype, device=m.dev)
        for c in range(9):
            v = torch.zeros_like(m.X)
            v[:, c // 3] = m.X[:, c % 3]
            v = v * (1.0 - m.free)
            w = v + m.solve(-m.times(v), 1e-13)
            fe = torch.bmm(m.K, w[m.conn].reshape(-1, 24, 1)).reshape(-1, 8, 3)
            C[:, :, c] = average(fe).reshape(k, 9)
        out["C"] = C.cpu().numpy()
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind in ("rve", "serve"):
        if (_sides(case).astype(float) ** 3).sum() > 8e5:
            return None
        return _exact_rve(case, seed)
    X, conn, kbc, tractions = _block(case, seed)
    if kind == "step" and len(X) > 120000 or case.get("precision") == FP64 and len(X) > 250000:
        return None
    material = MATERIAL[case.get("material", "hooke" if kind == "static" else "j2")]
    idx = np.array([a * 3 + d for a, d, _ in kbc], dtype=np.int64)
    m = _Exact(X, conn, (material,), None, idx)
    if kind == "force":
        m.u = torch.as_tensor(_field(X, seed), device=m.dev)
        r = m.residual().reshape(-1)[m.free.reshape(-1) > 0]
        return dict(R=r.cpu().numpy(), norm=float(r.norm()))
    v = np.zeros(X.size)
    v[idx] = [a[2] for a in kbc]
    if kind == "static":
        # uniform traction on undistorted boundary facets: a quarter each per node
        area = (X[:, 0].max() / case["nx"]) * (X[:, 1].max() / case["ny"])
        f = np.zeros_like(X)
        for e, _, t in tractions:
            f[conn[e, 4:]] += 0.25 * area * np.array(t)
        m.fext = torch.as_tensor(f, device=m.dev)
    m.step(torch.as_tensor(v.reshape(-1, 3), device=m.dev))
    out = dict(u=m.u.cpu().numpy())
    if kind != "step":
        n = m.nodal().cpu().numpy()
        out["stress"] = n[:, :6]
        if kind == "j2":
            out["material"] = n[:, 6:]
    return out
