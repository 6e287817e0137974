"""Both sides of the rule that gives small groups small tiles (csrc/efe_launch.cuh: up to two tiles per SM): the largest
group with small tiles and one element more, each with a last tile that is partly filled, against the oracle.
Tolerances as in the parity tests: 1e-12 of the largest entry, 2e-6 for an FP32 tangent."""

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _rel(a, b):
    return np.abs(a - b).max() / max(np.abs(b).max(), 1e-300)


@pytest.mark.parametrize("side", [-1, 1])
@pytest.mark.parametrize("elType,kind,props,precision,epb",
                         [("C3D8", "vonmises", [210e3, 0.3, 250.0, 1000.0, 0.0, 0.0], "fp64", 2),
                          ("C3D8", "vonmises", [210e3, 0.3, 250.0, 1000.0, 0.0, 0.0], "mixed", 4),
                          ("C3D20R", "linearelastic", [210e3, 0.3], "fp64", 2),
                          ("CPE4", "vonmises", [210e3, 0.3, 250.0, 1000.0, 0.0, 0.0], "fp64", 4),
                          ("CPS8R", "linearelastic", [210e3, 0.3], "mixed", 4),
                          ("C3D8TL", "neohookewa", [400.0, 2500.0], "mixed", 2),
                          ("C3D8TL", "neohookewb", [400.0, 2500.0], "mixed-ff", 2),
                          ("CPE8RTL", "neohookewc", [400.0, 2500.0], "fp64", 4)])  # fmt: skip
def test_both_sides_match_the_oracle(elType, kind, props, precision, epb, side):
    from edelweissfe_gb300 import ElementGroup, GPUAssembler, meshes
    from oracle.assembly import Model

    n = 2 * torch.cuda.get_device_properties(0).multi_processor_count * epb + side
    dim = 3 if elType.startswith("C3D") else 2
    nn = int(elType[3:].rstrip("RETL"))
    coords, conn, nodeDof, nDof = (meshes.box(n, 1, 1, nNodes=nn) if dim == 3 else meshes.rect(n, 1, nNodes=nn))
    rng = np.random.default_rng(11)
    X = coords / np.abs(coords).max(0) * [n, 1.0, 1.0][:dim] + rng.uniform(-0.03, 0.03, coords.shape)
    # strains of about 0.4 % with the gradient of a bent bar: a displacement of the bar's length would lose digits
    u = np.stack([4e-3 * np.sin(X[:, 0]) * X[:, 1], -2e-3 * X[:, 1], 1e-3 * X[:, -1]], 1)[:, :dim]
    U = np.empty(nDof)
    U[(nodeDof[:, None] + np.arange(dim)).ravel()] = (u + rng.normal(0.0, 1e-4, u.shape)).ravel()
    p = np.tile(props, (n, 1)) * (1.0 + rng.uniform(0.0, 0.05, (n, 1)))
    p[:, 1] = props[1]
    g = dict(elType=elType, kind=kind, props=p, conn=conn.astype(np.int64), thickness=np.full(n, 0.8), order=np.arange(n))
    m = Model(X, nodeDof, nDof, [g])
    r = m.compute_elements(U, U, m.initial_state())
    assert r["first_failed_element"] is None
    asm = GPUAssembler(X, nodeDof, nDof, [ElementGroup(elType, kind, p, conn, 0.8)], precision=precision)
    t = torch.as_tensor(U, device=asm.device)
    P, F, K = asm.constructDofVector(), asm.constructDofVector(), asm.constructSystemMatrix()
    asm.computeElements(None, t, t, P, K, F)
    assert _rel(P.cpu().numpy(), r["P"]) <= 1e-12
    assert _rel(F.cpu().numpy(), r["F"]) <= 1e-12
    assert _rel(K.double().cpu().numpy(), r["Kdata"]) <= (1e-12 if precision == "fp64" else 2e-6)
    assert _rel(asm.group_state(0, "temp"), r["stateTemp"][0]["state"]) <= 1e-12
