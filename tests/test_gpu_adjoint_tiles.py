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
