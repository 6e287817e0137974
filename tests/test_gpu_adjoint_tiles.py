"""The total-Lagrangian adjoint kernel (csrc/efe_adjoint.cuh) on every element type at the edges of its tiles (one element,
a tile partly filled, one element past a tile) and with lengths of 2^-20 and 2^20, which move the scales of its integer
sums, against fourth-order central differences of lambda . P of the oracle along random directions.

Tolerance: with a step of 2^-9 of the edge length the differences' truncation error is h^4 / 30 of the fifth derivative,
below 1e-9 of the derivative here, and rounding 2^-52 / h, below 1e-12; both with a factor of 10: 1e-8."""

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("elType,material,n,length",
                         [("C3D8TL", "neohookewa", 1, 1.0), ("C3D8TL", "neohookewb", 17, 2.0**20),
                          ("C3D8TL", "neohookewc", 16, 2.0**-20), ("C3D8RTL", "neohookewa", 33, 1.0),
                          ("C3D8ETL", "neohookewb", 5, 1.0), ("C3D20TL", "neohookewb", 5, 1.0),
                          ("C3D20RTL", "neohookewa", 17, 1.0), ("CPE4TL", "neohookewc", 33, 1.0),
                          ("CPE8TL", "neohookewa", 15, 2.0**-20), ("CPE8RTL", "neohookewb", 1, 1.0)])  # fmt: skip
def test_adjoint_matches_differences_of_the_oracle(elType, material, n, length):
    from edelweissfe_gb300 import ElementGroup, GPUAssembler, meshes
    from oracle.assembly import Model

    dim = 3 if elType.startswith("C3D") else 2
    nn = int(elType[3:].rstrip("RETL"))
    coords, conn, nodeDof, nDof = (meshes.box(n, 1, 1, nNodes=nn) if dim == 3 else meshes.rect(n, 1, nNodes=nn))
    rng = np.random.default_rng(3)
    coords = coords / np.abs(coords).max(0) * [n, 1.0, 1.0][:dim] + rng.uniform(-0.03, 0.03, coords.shape)
    coords = coords * length
    U = rng.normal(0.0, 1e-2, nDof) * length
    lam = rng.normal(0.0, 1.0, nDof)
    props = np.tile([400.0, 2500.0], (n, 1)) * (1.0 + rng.uniform(0.0, 0.2, (n, 2)))
    thick = np.full(n, 0.7)

    def value(X, p):
        g = dict(elType=elType, kind=material, props=p, conn=conn.astype(np.int64), thickness=thick, order=np.arange(n))
        m = Model(X, nodeDof, nDof, [g])
        return lam @ m.compute_elements(U, U, m.initial_state())["P"]

    def slope(f):
        h = 2.0**-9
        return (8.0 * (f(h) - f(-h)) - (f(2 * h) - f(-2 * h))) / (12.0 * h)

    asm = GPUAssembler(coords, nodeDof, nDof, [ElementGroup(elType, material, props, conn, 0.7)])
    gX, gP = asm.adjointTL(torch.as_tensor(U, device=asm.device), torch.as_tensor(lam, device=asm.device))
    gX = gX.cpu().numpy()
    gP = (gP[0] if isinstance(gP, (list, tuple)) else gP).cpu().numpy()
    dX = rng.uniform(-0.1, 0.1, coords.shape) * length
    ref = slope(lambda h: value(coords + h * dX, props))
    assert abs((gX * dX).sum() - ref) <= 1e-8 * np.abs(gX * dX).sum()
    dp = props * rng.uniform(0.5, 1.0, props.shape)
    ref = slope(lambda h: value(coords, props + h * dp))
    assert abs((gP * dp).sum() - ref) <= 1e-8 * np.abs(gP * dp).sum()


@pytest.mark.parametrize("elType,props,n,length",
                         [("C3D8", [210e3, 0.3, 250.0, 1000.0, 0.0, 0.0], 1, 1.0),
                          ("C3D8", [210e3, 0.3, 250.0, 1000.0, 100.0, 20.0], 17, 2.0**20),
                          ("C3D8R", [210e3, 0.3, 250.0, 1000.0, 0.0, 0.0], 33, 1.0),
                          ("C3D8E", [210e3, 0.3, 250.0, 1000.0, 0.0, 0.0], 5, 2.0**-20),
                          ("C3D20", [210e3, 0.3, 250.0, 1000.0, 0.0, 0.0], 5, 1.0),
                          ("C3D20R", [210e3, 0.3, 250.0, 1000.0, 0.0, 0.0], 16, 1.0),
                          ("CPE4", [210e3, 0.3, 250.0, 1000.0, 0.0, 0.0], 33, 1.0),
                          ("CPE8", [210e3, 0.3], 15, 2.0**20)])  # fmt: skip
def test_small_strain_adjoint_matches_differences_of_the_oracle(elType, props, n, length):
    from edelweissfe_gb300 import ElementGroup, GPUAssembler, meshes
    from oracle.assembly import Model

    kind = "linearelastic" if len(props) == 2 else "vonmises"
    dim = 3 if elType.startswith("C3D") else 2
    nn = int(elType[3:].rstrip("RE"))
    coords, conn, nodeDof, nDof = (meshes.box(n, 1, 1, nNodes=nn) if dim == 3 else meshes.rect(n, 1, nNodes=nn))
    rng = np.random.default_rng(5)
    X = coords / np.abs(coords).max(0) * [n, 1.0, 1.0][:dim] + rng.uniform(-0.03, 0.03, coords.shape)
    coords = X * length
    # a field far beyond yield at every point, so that no difference crosses the yield surface
    u = np.stack([6e-3 * X[:, 0] + 1e-3 * X[:, 1], -3e-3 * X[:, 1], -1e-3 * X[:, -1]], 1)[:, :dim] * length
    dofs = (nodeDof[:, None] + np.arange(dim)).ravel()
    d = [np.empty(nDof) for _ in range(2)]
    for k, f in enumerate((1.0, 0.5)):
        d[k][dofs] = (f * u + rng.normal(0.0, 1e-5, u.shape) * length).ravel()
    p0 = np.tile(props, (n, 1)) * (1.0 + rng.uniform(0.0, 0.05, (n, 1)))
    p0[:, 1] = 0.3
    lam = rng.normal(0.0, 1.0, nDof) / length**(dim - 1)

    def model(x, p):
        g = dict(elType=elType, kind=kind, props=p, conn=conn.astype(np.int64), thickness=np.full(n, 0.7), order=np.arange(n))
        return Model(x, nodeDof, nDof, [g])

    m0 = model(coords, p0)
    st = m0.accept_state(m0.compute_elements(d[0], d[0], m0.initial_state())["stateTemp"])
    s0 = st[0]["state"]
    # seeds of stress, strain and hardening of like weight
    seed = rng.normal(0.0, 1.0, s0.shape) / np.array(([1.0] * 6 + [1e-5] * 6 + [1e-5])[: s0.shape[-1]]) * 1e-2

    def value(du, p, x):
        r = model(x, p).compute_elements(d[0] + du, du, st)
        return lam @ r["P"] + (seed * r["stateTemp"][0]["state"]).sum()

    def slope(f):
        h = 2.0**-9
        return (8.0 * (f(h) - f(-h)) - (f(2 * h) - f(-2 * h))) / (12.0 * h)

    asm = GPUAssembler(coords, nodeDof, nDof, [ElementGroup(elType, kind, p0, conn, 0.7)])
    dev = asm.device
    pts = lambda v: torch.as_tensor(np.ascontiguousarray(v.reshape(-1, v.shape[-1]).T), device=dev)
    dUbar = torch.zeros(nDof, dtype=torch.float64, device=dev)
    out = torch.zeros_like(pts(s0))
    gP = torch.zeros(p0.shape, dtype=torch.float64, device=dev)
    gX = torch.zeros(coords.shape, dtype=torch.float64, device=dev)
    asm.adjointSmallStrain(0, pts(s0), torch.as_tensor(d[1], device=dev), dUbar, Pbar=torch.as_tensor(lam, device=dev),
                           stateBarIn=pts(seed), stateBarOut=out, gProps=gP, gX=gX)  # fmt: skip
    dirs = [d[1] * rng.uniform(-0.2, 0.2, nDof), p0 * rng.uniform(0.05, 0.1, p0.shape), rng.uniform(-0.02, 0.02, X.shape) * length]
    at = [d[1], p0, coords]
    for k, g in enumerate((dUbar, gP, gX)):
        ref = slope(lambda h: value(*[v + (h * dirs[k] if i == k else 0.0) for i, v in enumerate(at)]))
        terms = g.cpu().numpy() * dirs[k]
        assert abs(terms.sum() - ref) <= 1e-8 * np.abs(terms).sum(), (k, terms.sum(), ref)
