"""Plates of thin solid elements (1 : 100 to 1 : 10^5, in each direction) that rotate as a whole and strain little: the
components of dN/dX and of the increment differ by the aspect ratio, and the membrane strains are what matters.  Every
entry of the strains, the residual, the tangent and the adjoints against the same sums in extended precision, from the
device's own dN/dX and weights, relative to the products that the entry itself is summed of.

Tolerances.  A strain G_d . u_i is a sum of n nodes' products with u relative to the first node; FP64 rounds u - u_0,
every product and every sum, 2^-53 each: n 2^-53 max|G_d| max|u_i - u_0| for the differences and as much for the sums.
The integers' operands are rounded at 2^-58 of the element's largest, a point's own being up to 2^3 smaller: 2 n 2^-58
2^5 of the same.  Together below n 2^-51; a shear has two such sums.  The other outputs go through a few products more,
each 2^-53 of the same kind of bound, up to 27 points: 2^-46.  FP32 tangents: 8 roundings of the operands and products and
one for each point added, 2^-24 each."""

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

ld = np.longdouble
VM = [210e3, 0.3, 250.0, 1000.0, 0.0, 0.0]
LE = [210e3, 0.3]
VOIGT = [(0, 0), (1, 1), (2, 2), (0, 1), (0, 2), (1, 2)]


def _plate(nn, axis, aspect, rng):
    """2 x 2 x 1 elements of in-plane edge 1, the thin direction along `axis`; Hexa8's nodes are moved in the plane (Hexa20's
    Jacobian, as the reference's, does not reproduce linear fields on curved elements: the plate would flow)."""
    from edelweissfe_gb300 import meshes

    coords, conn, nodeDof, nDof = meshes.box(2, 2, 1, 2.0, 2.0, 1.0, nNodes=nn)
    if nn == 8:
        coords = coords + rng.uniform(-0.03, 0.03, coords.shape) * [1, 1, 0]
    coords[:, 2] /= aspect
    return np.roll(coords, axis - 2, axis=1), conn, nodeDof, nDof


def _increment(X, axis, strain, rotation, rng):
    """Rigid rotation about an axis of the plane (which moves it across) and in-plane strains."""
    p, q = (axis + 1) % 3, (axis + 2) % 3
    u = np.zeros_like(X)
    u[:, p] = strain * (X[:, p] + 0.3 * X[:, q]) + rotation * X[:, axis]
    u[:, q] = -0.4 * strain * X[:, q]
    u[:, axis] = -rotation * X[:, p] - 0.3 * strain * X[:, axis]
    return u + rng.uniform(-0.05, 0.05, X.shape) * strain * np.ptp(X[:, axis])  # noise of the thin edges' size


def _geometry(asm, E):
    """dN/dX [E, Q, 3, n] and weights [E, Q] of the device's set-up."""
    d = asm.groups[0]._dev
    G = d["geomG"].cpu().numpy().astype(ld)
    s = d["geomS"].cpu().numpy().astype(ld).reshape(E, -1)
    return G.reshape(3, -1, E, s.shape[1]).transpose(2, 3, 0, 1), s


def _gradient(G, u):
    """u_i dN/dX_d sums H [E, Q, i, d] and the bound of their rounding (u: [E, n, 3])."""
    v = u.astype(ld) - u.astype(ld)[:, :1]
    H = np.einsum("eqda,eai->eqid", G, v)
    du = np.abs(v).max(1)
    return H, G.shape[3] * np.abs(G).max(3)[:, :, None, :] * du[:, None, :, None]


def _voigt(H):
    return np.stack([H[..., i, j] + (H[..., j, i] if i != j else 0) for i, j in VOIGT], -1)


def _matrix(v):
    """Voigt stresses [..., 6] as [..., 3, 3]."""
    m = np.zeros(v.shape[:-1] + (3, 3), v.dtype)
    for f, (i, j) in enumerate(VOIGT):
        m[..., i, j] = m[..., j, i] = v[..., f]
    return m


def _below(got, ref, bound, what):
    err = np.abs(got.astype(ld) - ref)
    worst = np.unravel_index(np.argmax(err / bound), err.shape)
    assert (err <= bound).all(), f"{what}: {err[worst]} at {worst} of {ref[worst]}, {err[worst] / bound[worst]} of the bound"


def _nodal(shape, idx, values):
    out = np.zeros(shape, ld)
    np.add.at(out, idx, values)
    return out


CASES = [(el, axis, aspect) for el in ("C3D8", "C3D20", "C3D8E", "C3D20R") for axis, aspect in ((0, 1e2), (1, 1e4), (2, 1e4), (2, 1e5))
         if el[-1] in "80" or axis != 1]  # fmt: skip


def _pass(elType, axis, aspect, precision, kind, props):
    """One pass of a plate: an elastic one that rotates, or one that flows in its plane."""
    from edelweissfe_gb300 import ElementGroup, GPUAssembler

    rng = np.random.default_rng(11)
    coords, conn, nodeDof, nDof = _plate(20 if "20" in elType else 8, axis, aspect, rng)
    elastic = kind == "linearelastic"
    u = _increment(coords, axis, 1e-4 if elastic else 4e-3, 0.05 if elastic else 0.0, rng)
    E = len(conn)
    asm = GPUAssembler(coords, nodeDof, nDof, [ElementGroup(elType, kind, np.tile(props, (E, 1)), conn)], precision=precision)
    dU = np.zeros(nDof)
    dU[nodeDof[:, None] + np.arange(3)] = u
    t = torch.tensor(dU, device=asm.device)
    P, F, K = asm.constructDofVector(), asm.constructDofVector(), asm.constructSystemMatrix()
    asm.computeElements(None, t, t, P, K, F)
    G, s = _geometry(asm, E)
    state = asm.group_state(0, "temp")
    if not elastic:
        assert (state[..., 12] > 0).all()
    return asm, conn, u, nodeDof[conn][:, :, None] + np.arange(3), P.cpu().numpy(), K, G, s, state, _matrix(state[..., :6].astype(ld))


def _tangent(asm, dof, K, G, s, state, sig, props):
    """The assembled K, the exact one and the bound of its products: C = C_iso(c12 + beta / 3, c44 - beta / 2) - a n (x) n
    with n along the device's stress deviator."""
    E, NQ = s.shape
    nDof = asm.nDof
    Gm = np.abs(G).max(3)
    Em, nu = ld(props[0]), ld(props[1])
    lam, mu = Em * nu / ((1 + nu) * (1 - 2 * nu)), Em / (2 * (1 + nu))
    c12, c44, a = np.full((E, NQ), lam), np.full((E, NQ), mu), np.zeros((E, NQ), ld)
    n = np.zeros((E, NQ, 3, 3), ld)
    if len(props) > 2:
        dev = sig - np.trace(sig, axis1=2, axis2=3)[..., None, None] / 3 * np.eye(3)
        q = np.sqrt((dev**2).sum((2, 3)))
        n = dev / q[..., None, None]
        g2 = 2 * mu * np.sqrt(ld(1.5)) * state[..., 12].astype(ld)
        qt = q + g2  # of the trial stress
        beta = 2 * mu * g2 / qt
        c12, c44, a = lam + beta / 3, mu - beta / 2, 2 * mu * (1 / (1 + ld(props[3]) / (3 * mu)) - g2 / qt)
    nG, nGm = np.einsum("eqjd,eqda->eqja", n, G), np.einsum("eqjd,eqd->eqj", np.abs(n), Gm)
    # K_ab[j][k], symmetric: row and column order does not matter
    Ke = np.einsum("eq,eqja,eqkb->eajbk", s * c12, G, G) + np.einsum("eq,eqka,eqjb->eajbk", s * c44, G, G)
    Ke -= np.einsum("eq,eqja,eqkb->eajbk", s * a, nG, nG)
    dot = np.einsum("eq,eqda,eqdb->eab", s * c44, G, G)
    Kb = np.einsum("eq,eqj,eqk->ejk", np.abs(s) * (np.abs(c12) + np.abs(c44)), Gm, Gm)
    Kb += np.einsum("eq,eqj,eqk->ejk", np.abs(s * a), nGm, nGm)
    dotb = np.einsum("eq,eqd,eqd->e", np.abs(s * c44), Gm, Gm)
    for j in range(3):
        Ke[:, :, j, :, j] += dot
        Kb[:, j, j] += dotb
    full = np.zeros((nDof, nDof))
    rows = np.repeat(np.arange(nDof), np.diff(asm.indptr_host))
    full[rows, asm.indices_host] = K.double().cpu().numpy()
    i, j = np.broadcast_arrays(dof[:, :, :, None, None], dof[:, None, None, :, :])
    ref = _nodal((nDof, nDof), (i, j), Ke)
    bound = _nodal((nDof, nDof), (i, j), np.broadcast_to(Kb[:, None, :, None, :], Ke.shape))
    return full, ref, bound + (bound == 0)


MATERIALS = pytest.mark.parametrize("kind,props", [("linearelastic", LE), ("vonmises", VM)])


@MATERIALS
@pytest.mark.parametrize("precision", ["fp64", "mixed", "mixed-ff"])
@pytest.mark.parametrize("elType,axis,aspect", CASES)
def test_small_strain_pass(elType, axis, aspect, precision, kind, props):
    asm, conn, u, dof, P, K, G, s, state, sig = _pass(elType, axis, aspect, precision, kind, props)
    H, Hb = _gradient(G, u[conn])
    _below(state[..., 6:12], _voigt(H), 2.0**-51 * _voigt(Hb), "strain")
    # the residual from the device's stresses
    ref = _nodal(asm.nDof, dof, -np.einsum("eq,eqcd,eqda->eac", s, sig, G))
    bound = np.einsum("eq,eqcd,eqd->ec", np.abs(s), np.abs(sig), np.abs(G).max(3))
    _below(P, ref, 2.0**-46 * _nodal(asm.nDof, dof, np.broadcast_to(bound[:, None, :], dof.shape)), "P")
    if precision == "fp64":
        full, ref, bound = _tangent(asm, dof, K, G, s, state, sig, props)
        _below(full, ref, 2.0**-46 * bound, "K")


@MATERIALS
@pytest.mark.parametrize("precision", ["mixed", "mixed-ff"])
@pytest.mark.parametrize("elType,axis,aspect", CASES)
def test_fp32_tangent(elType, axis, aspect, precision, kind, props):
    asm, _, _, dof, _, K, G, s, state, sig = _pass(elType, axis, aspect, precision, kind, props)
    full, ref, bound = _tangent(asm, dof, K, G, s, state, sig, props)
    _below(full, ref, (8 + s.shape[1]) * 2.0**-24 * bound, "K")

def _neo_hooke(H, mu, K):
    """F, F^-1 and sB, sI, dsI/dJ J of variant a: tau = mu B + sI I."""
    F = H + np.eye(3, dtype=ld)
    C = np.stack([np.cross(F[..., 1, :], F[..., 2, :]), np.cross(F[..., 2, :], F[..., 0, :]), np.cross(F[..., 0, :], F[..., 1, :])], -2)
    J = (F[..., 0, :] * C[..., 0, :]).sum(-1)
    iF = np.swapaxes(C, -1, -2) / J[..., None, None]
    return F, iF, mu, (K - 2 * mu / 3) * (J * J - J) - mu, (K - 2 * mu / 3) * (2 * J * J - J)


@pytest.mark.parametrize("precision", ["mixed", "mixed-ff"])
@pytest.mark.parametrize("axis,aspect", [(0, 1e2), (1, 1e4), (2, 1e5)])
def test_total_lagrangian_hexa20_pass(axis, aspect, precision):
    from edelweissfe_gb300 import ElementGroup, GPUAssembler

    rng = np.random.default_rng(12)
    coords, conn, nodeDof, nDof = _plate(20, axis, aspect, rng)
    u = _increment(coords, axis, 1e-4, 0.05, rng)
    mu, Kb = 400.0, 2500.0
    E = len(conn)
    asm = GPUAssembler(coords, nodeDof, nDof, [ElementGroup("C3D20TL", "neohookewa", np.tile([mu, Kb], (E, 1)), conn)],
                       precision=precision)  # fmt: skip
    U = np.zeros(nDof)
    U[nodeDof[:, None] + np.arange(3)] = u
    t = torch.tensor(U, device=asm.device)
    P, F, K = asm.constructDofVector(), asm.constructDofVector(), asm.constructSystemMatrix()
    asm.computeElements(None, t, t, P, K, F)
    G, s = _geometry(asm, E)
    H, Hb = _gradient(G, u[conn])
    eps, epsb = _voigt(H), _voigt(Hb)
    quad, quadb = np.einsum("eqki,eqkj->eqij", H, H), np.einsum("eqki,eqkj->eqij", Hb, np.abs(H))
    for f, (i, j) in enumerate(VOIGT):
        eps[..., f] += quad[..., i, j] * (0.5 if i == j else 1.0)
        epsb[..., f] += quadb[..., i, j] + quadb[..., j, i]
    order = [0, 1, 2, 3, 5, 4]  # 11, 22, 33, 12, 23, 13
    _below(asm.group_state(0, "temp")[..., 6:12][..., order], eps, 2.0**-50 * epsb, "strain")
    Fd, iF, sB, sI, _ = _neo_hooke(H, ld(mu), ld(Kb))
    sP = s[..., None, None] * (sB * Fd + sI[..., None, None] * np.swapaxes(iF, 2, 3))
    # the stress is a difference of near equal terms; H's own rounding enters through the stiffness
    sPb = np.abs(s)[..., None, None] * (mu * np.abs(Fd) + np.abs(sI)[..., None, None] * np.abs(np.swapaxes(iF, 2, 3)))
    sPb = sPb + np.abs(s)[..., None, None] * Kb * (Hb + np.swapaxes(Hb, 2, 3) + np.trace(Hb, axis1=2, axis2=3)[..., None, None] * np.abs(Fd)) * 2.0**-3
    dof = nodeDof[conn][:, :, None] + np.arange(3)
    ref = _nodal(nDof, dof, -np.einsum("eqcd,eqda->eac", sP, G))
    bound = _nodal(nDof, dof, np.broadcast_to(np.einsum("eqcd,eqd->ec", sPb, np.abs(G).max(3))[:, None, :], dof.shape))
    _below(P.cpu().numpy(), ref, 2.0**-46 * bound, "P")


@pytest.mark.parametrize("elType,axis,aspect", CASES)
def test_small_strain_adjoint(elType, axis, aspect):
    """Linear elastic: sigma0Bar = -s B PBar, dUbar = -sum s B^T C B PBar and the coordinates' adjoint sum_l Q[l][c] dN/dX_l with Q = -s (sigma :
    B PBar) I - deBar Hu + s sigma Hp (Hexa8; Hexa20's has a term more)."""
    from edelweissfe_gb300 import ElementGroup, GPUAssembler

    rng = np.random.default_rng(13)
    coords, conn, nodeDof, nDof = _plate(20 if "20" in elType else 8, axis, aspect, rng)
    u, p = _increment(coords, axis, 1e-4, 0.05, rng), _increment(coords, axis, 0.03, -1.0, rng)
    E = len(conn)
    asm = GPUAssembler(coords, nodeDof, nDof, [ElementGroup(elType, "linearelastic", np.tile(LE, (E, 1)), conn)])
    v = [torch.zeros(nDof, dtype=torch.float64, device=asm.device) for _ in range(2)]
    for x, y in zip(v, (u, p)):
        x[torch.as_tensor((nodeDof[:, None] + np.arange(3)).ravel(), device=asm.device).long()] = torch.tensor(y.ravel(), device=asm.device)
    hexa8 = "20" not in elType
    G, s = _geometry(asm, E)
    Gm = np.abs(G).max(3)
    Em, nu = ld(LE[0]), ld(LE[1])
    lam, mu = Em * nu / ((1 + nu) * (1 - 2 * nu)), Em / (2 * (1 + nu))

    def stress(H):
        return lam * np.trace(H, axis1=2, axis2=3)[..., None, None] * np.eye(3) + mu * (H + np.swapaxes(H, 2, 3))

    (Hu, Hub), (Hp, Hpb) = _gradient(G, u[conn]), _gradient(G, p[conn])
    sq = s[..., None, None]
    deBar, deBarb = -sq * stress(Hp), np.abs(sq) * stress(Hpb)
    dof = nodeDof[conn][:, :, None] + np.arange(3)
    for withX in (False, True):
        dUbar = torch.zeros(nDof, dtype=torch.float64, device=asm.device)
        gX = torch.zeros((len(coords), 3), dtype=torch.float64, device=asm.device) if withX else None
        before = asm.groups[0]._dev["stateRef"]
        barOut = torch.zeros_like(before)
        asm.adjointSmallStrain(0, before, v[0], dUbar, Pbar=v[1], stateBarOut=barOut, gX=gX)
        sigBar = barOut[:6].T.reshape(E, -1, 6).cpu().numpy()
        _below(sigBar, -s[..., None] * _voigt(Hp), 2.0**-50 * np.abs(s)[..., None] * _voigt(Hpb), "sigma0Bar")
        ref = _nodal(nDof, dof, np.einsum("eqcd,eqda->eac", deBar, G))
        bound = _nodal(nDof, dof, np.broadcast_to(np.einsum("eqcd,eqd->ec", deBarb, Gm)[:, None, :], dof.shape))
        _below(dUbar.cpu().numpy(), ref, 2.0**-46 * bound, "dUbar")
        if not (withX and hexa8):
            continue
        sig, sigb = stress(Hu), stress(Hub)
        sBar, sBarb = -(sig * Hp).sum((2, 3)), (sigb * Hpb).sum((2, 3))
        Q = sq * sBar[..., None, None] * np.eye(3) - deBar @ Hu + sq * (sig @ Hp)
        Qb = np.abs(sq) * sBarb[..., None, None] * np.eye(3) + deBarb @ Hub + np.abs(sq) * (sigb @ Hpb)
        idx = (conn[:, :, None], np.arange(3))
        ref = _nodal(coords.shape, idx, np.einsum("eqlc,eqla->eac", Q, G))
        bound = _nodal(coords.shape, idx, np.broadcast_to(np.einsum("eqlc,eql->ec", Qb, Gm)[:, None, :], conn.shape + (3,)))
        _below(gX.cpu().numpy(), ref, 2.0**-46 * bound, "gX")


def _coordinate_adjoint(coords, conn, u, l, mu, K, ty):
    """gX of C3D8TL, Neo-Hooke a, in the number type ty: sum dL/dJ[r][c] dN/dxi_r with dL/dJ = s J^-T (dphi/dF^T H + P^T
    Lambda - phi I) (an order of the axes of xi makes no difference to the sum over the points), and the sum of its products'
    magnitudes."""
    nat = np.array([(-1, -1, -1), (-1, -1, 1), (1, -1, 1), (1, -1, -1), (-1, 1, -1), (-1, 1, 1), (1, 1, 1), (1, 1, -1)], ty)
    f = 1 + (nat / np.sqrt(ty(3)))[:, None, :] * nat[None]  # [q, a, d]
    D = np.stack([nat[:, r] * f[..., (r + 1) % 3] * f[..., (r + 2) % 3] / 8 for r in range(3)], 1)  # [q, r, a]
    rel = [(x[conn] - x[conn][:, :1]).astype(ty) for x in (coords, u, l)]
    J = np.einsum("qra,eac->eqrc", D, rel[0])
    C = np.stack([np.cross(J[..., 1, :], J[..., 2, :]), np.cross(J[..., 2, :], J[..., 0, :]), np.cross(J[..., 0, :], J[..., 1, :])], -2)
    s = (J[..., 0, :] * C[..., 0, :]).sum(-1)
    iJ = np.swapaxes(C, 2, 3) / s[..., None, None]  # [c][r]
    H, Lam = (np.einsum("qra,eai,eqjr->eqij", D, x, iJ) for x in rel[1:])
    F, iF, sB, sI, dI = _neo_hooke(H, ty(mu), ty(K))
    iFT = np.swapaxes(iF, 2, 3)
    trM = (iFT * Lam).sum((2, 3))[..., None, None]
    sI, dI = sI[..., None, None], dI[..., None, None]
    P = sB * F + sI * iFT
    phi = (P * Lam).sum((2, 3))[..., None, None]
    dphi = sB * Lam + dI * trM * iFT - sI * (iFT @ np.swapaxes(Lam, 2, 3) @ iFT)
    E = np.swapaxes(dphi, 2, 3) @ H + np.swapaxes(P, 2, 3) @ Lam - phi * np.eye(3, dtype=ty)
    size = np.swapaxes(np.abs(dphi) + mu * np.abs(Lam), 2, 3) @ np.abs(H) + mu * (np.abs(F) + np.abs(iFT)) @ np.abs(Lam)
    size = size + np.trace(size, axis1=2, axis2=3)[..., None, None] * np.eye(3)
    gX, sizeX = np.zeros(coords.shape, ty), np.zeros(coords.shape, ty)
    idx = (conn[:, :, None], np.arange(3))
    np.add.at(gX, idx, np.einsum("eq,eqkr,eqkc,qra->eac", s, iJ, E, D))
    size = np.einsum("eq,eqkr,eqkc->ec", np.abs(s), np.abs(iJ), size)
    np.add.at(sizeX, idx, np.broadcast_to(size[:, None, :], conn.shape + (3,)))
    return gX, sizeX


@pytest.mark.parametrize("axis,aspect", [(2, 1.0), (0, 1e2), (1, 1e4), (2, 1e5)])
def test_total_lagrangian_adjoint(axis, aspect):
    """The rounding of H and Lambda (2^-53 of dN/dX across the plate) enters gX through the stiffness; its measure is the
    same formula in FP64, and four times its distance from the exact values is allowed beside eight roundings of the
    products that gX is summed of."""
    from edelweissfe_gb300 import ElementGroup, GPUAssembler

    rng = np.random.default_rng(14)
    coords, conn, nodeDof, nDof = _plate(8, axis, aspect, rng)
    u, l = _increment(coords, axis, 1e-2, 0.05, rng), _increment(coords, axis, 0.03, -1.0, rng)
    mu, K = 400.0, 2500.0
    asm = GPUAssembler(coords, nodeDof, nDof, [ElementGroup("C3D8TL", "neohookewa", np.tile([mu, K], (len(conn), 1)), conn)])
    v = [np.zeros(nDof) for _ in range(2)]
    for x, y in zip(v, (u, l)):
        x[nodeDof[:, None] + np.arange(3)] = y
    gX, _ = asm.adjointTL(torch.tensor(v[0], device=asm.device), torch.tensor(v[1], device=asm.device))
    (ref, size), (plain, _) = (_coordinate_adjoint(coords, conn, u, l, mu, K, ty) for ty in (ld, np.float64))
    err, err64 = (np.abs(x.astype(ld) - ref).max(0) for x in (gX.cpu().numpy(), plain))
    assert (err <= 4 * err64 + 2.0**-50 * size.max(0)).all(), (err, err64, size.max(0))
