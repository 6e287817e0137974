"""Small-strain solids with their B-products in integers (csrc/efe_fixed.cuh): every element type, precision and tile
shape at the edges of the tiles (one element, the last group of a tile partly filled, one past a tile) against the
oracle, with lengths of 2^-20, 1 and 2^20 so that the common scales of the integer sums move, and on a mesh whose edges
differ by 2^12, where the entries of one scale differ most.

Tolerances as in the parity tests: 1e-12 of the largest entry for P, F, the state and an FP64 tangent.  An FP32 tangent
sums at most 27 points of 12 products with operands rounded at most three times: 6 x 2^-24 each and the sums' own
roundings, which average out, stay below 2e-6."""

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

VM = [210e3, 0.3, 250.0, 1000.0, 0.0, 0.0]
SAT = [210e3, 0.3, 250.0, 1000.0, 100.0, 20.0]  # saturation hardening: a Newton iteration per point
LE = [2.1e11, 0.25]


def _rel(a, b):
    return np.abs(a - b).max() / max(np.abs(b).max(), 1e-300)


@pytest.mark.parametrize("precision", ["fp64", "mixed", "mixed-ff"])
@pytest.mark.parametrize("elType,kind,props,n,length,stretch",
                         [("C3D8", "vonmises", VM, 1, 1.0, 1.0), ("C3D8", "vonmises", SAT, 5, 2.0**20, 1.0),
                          ("C3D8", "vonmises", VM, 16, 1.0, 2.0**12), ("C3D8", "linearelastic", LE, 17, 2.0**-20, 1.0),
                          ("C3D8R", "vonmises", VM, 33, 1.0, 1.0), ("C3D8E", "vonmises", VM, 5, 2.0**-20, 1.0),
                          ("C3D20R", "vonmises", VM, 17, 1.0, 2.0**12), ("C3D20", "vonmises", SAT, 1, 1.0, 1.0),
                          ("C3D20", "vonmises", VM, 10, 2.0**20, 1.0), ("C3D20", "linearelastic", LE, 4, 1.0, 2.0**12)])  # fmt: skip
def test_tiles_match_the_oracle(elType, kind, props, n, length, stretch, precision):
    from edelweissfe_gb300 import ElementGroup, GPUAssembler, meshes
    from oracle.assembly import Model

    coords, conn, nodeDof, nDof = meshes.box(n, 1, 1, nNodes=20 if "20" in elType else 8)
    rng = np.random.default_rng(7)
    coords = (coords / np.abs(coords).max(0) * [n, 1.0, 1.0] + rng.uniform(-0.04, 0.04, coords.shape)) * length
    coords[:, 2] *= stretch
    conn = conn[rng.permutation(n)]
    # a smooth field far beyond yield on top of noise
    X = coords / length / [1.0, 1.0, stretch]
    u = np.stack([4e-3 * X[:, 0] + 1e-3 * X[:, 1], -2e-3 * X[:, 1] + 1e-3 * X[:, 2], -1e-3 * X[:, 2]], 1)
    scale = length  # displacements of the short edges' size: with the long edges' the shear strains would be 2^12 times these
    d = [np.empty(nDof) for _ in range(2)]
    for k, f in enumerate((1.0, 0.3)):
        v = (f * u + rng.normal(0, 1e-4, u.shape)) * scale
        for c in range(3):
            d[k][nodeDof + c] = v[:, c]
    p = np.tile(props, (n, 1)) * (1.0 + rng.uniform(0.0, 0.1, (n, 1)))
    p[:, 1] = props[1]
    g = dict(elType=elType, kind=kind, props=p, conn=conn.astype(np.int64), thickness=np.ones(n), order=np.arange(n))
    m = Model(coords, nodeDof, nDof, [g])
    st = m.accept_state(m.compute_elements(d[0], d[0], m.initial_state())["stateTemp"])
    r = m.compute_elements(d[0] + d[1], d[1], st)
    assert r["first_failed_element"] is None
    asm = GPUAssembler(coords, nodeDof, nDof, [ElementGroup(elType, kind, p, conn, 1.0)], precision=precision)
    dev = asm.device
    d0, d1 = (torch.as_tensor(x, device=dev) for x in d)
    P, F, K = asm.constructDofVector(), asm.constructDofVector(), asm.constructSystemMatrix()
    asm.computeElements(None, d0, d0, P, K, F)
    asm.acceptLastState()
    for variant in (0, 1, 2):
        asm._groups_c[0].tileVariant = variant
        for t in (P, F, K):
            t.zero_()
        asm.computeElements(None, d0 + d1, d1, P, K, F)
        assert _rel(P.cpu().numpy(), r["P"]) <= 1e-12
        assert _rel(F.cpu().numpy(), r["F"]) <= 1e-12
        assert _rel(K.double().cpu().numpy(), r["Kdata"]) <= (1e-12 if precision == "fp64" else 2e-6)
        assert _rel(asm.group_state(0, "temp"), r["stateTemp"][0]["state"]) <= 1e-12


@pytest.mark.parametrize("elType", ["C3D8", "C3D20"])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_non_finite_increment_reaches_all_outputs_of_its_element_only(elType, precision, bad):
    from edelweissfe_gb300 import ElementGroup, GPUAssembler, meshes
    from edelweissfe_gb300 import _lib as L

    coords, conn, nodeDof, nDof = meshes.box(3, 1, 1, nNodes=20 if "20" in elType else 8)
    asm = GPUAssembler(coords, nodeDof, nDof, [ElementGroup(elType, "vonmises", VM, conn)], precision=precision)
    asm._groups_c[0].tileVariant = 0
    dU = np.zeros(nDof)
    node = int(np.setdiff1d(conn[2], conn[1])[0])  # of the last element alone
    dU[nodeDof[node] + 1] = bad
    P, F, K = asm.constructDofVector(), asm.constructDofVector(), asm.constructSystemMatrix()
    asm.status.zero_()
    t = torch.tensor(dU, device=asm.device)
    asm.launch(t, t, P, K, F)
    assert asm.status.cpu().numpy()[0] & L.EFE_STATUS_NONFINITE
    P = P.cpu().numpy()
    d2, d01 = nodeDof[conn[2]], nodeDof[np.setdiff1d(conn[:2], conn[2])]
    assert not np.isfinite(P[d2]).any() and (P[d01] == 0).all()
