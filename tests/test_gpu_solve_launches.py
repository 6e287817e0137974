"""Device solves that take several launches of CG iterations (50 each here, as in a system whose iterations are long)
against the same solves in one launch: same bits, same iteration counts; the end of a solve in an earlier launch than the
last queued one; the exact stop at pcgMaxIter; and the multigrid CG, whose batches pcgGraphs replays as a graph, against
directly launched ones."""

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _system(precision, elType="C3D8", size=(9, 8, 7)):
    from edelweissfe_gb300 import ElementGroup, GPUAssembler, meshes
    from edelweissfe_gb300.solver import NISTGPU

    coords, conn, nodeDof, nDof = meshes.box(*size, nNodes=20 if "20" in elType else 8)
    # moduli over three decades: more iterations
    rng = np.random.default_rng(5)
    props = np.stack([210e3 * 10.0 ** rng.uniform(-1.5, 1.5, len(conn)), np.full(len(conn), 0.3)], 1)
    asm = GPUAssembler(coords, nodeDof, nDof, [ElementGroup(elType, "linearelastic", props, conn)], precision=precision)
    K = NISTGPU(asm).tangentAt(torch.zeros(nDof, dtype=torch.float64, device=asm.device))
    fixed = torch.as_tensor(nodeDof[coords[:, 2] < 1e-9][:, None] + np.arange(3), device=asm.device).ravel()
    R = torch.tensor(rng.normal(0, 1, nDof), device=asm.device)
    return asm, K, R, fixed


def _solve(asm, K, R, fixed, **kw):
    from edelweissfe_gb300.solver import NISTGPU

    s = NISTGPU(asm, **kw)
    x = s._solve_pcg(K, R, fixed)
    return x, s


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("pre", ["jacobi", "block"])
def test_several_launches_match_one(precision, pre, monkeypatch):
    import scipy.sparse as sp
    import scipy.sparse.linalg as sla

    from edelweissfe_gb300 import solver

    asm, K, R, fixed = _system(precision)
    one, s1 = _solve(asm, K, R, fixed, pcgTolerance=1e-12, pcgPreconditioner=pre)
    assert s1.linearIterations[-1] > 150 and s1.linearIterations[-1] % 10 == 0  # four launches or more below
    monkeypatch.setattr(solver, "LAUNCH_SECONDS", 0.0)
    many, s2 = _solve(asm, K, R, fixed, pcgTolerance=1e-12, pcgPreconditioner=pre)
    assert torch.equal(one, many)
    assert s1.linearIterations == s2.linearIterations and s2.linearConverged[-1]
    # |r| <= 1e-12 |b|, so the error against a direct solve is below cond(K) 1e-12
    A = sp.csr_matrix((K.double().cpu().numpy(), asm.indices_host, asm.indptr_host))
    f = fixed.cpu().numpy()
    free = np.setdiff1d(np.arange(asm.nDof), f)
    b = R.cpu().numpy()
    res = b[free] - (A @ many.cpu().numpy())[free]
    # the recursive residual's 1e-12 and the rounding of the products with x, |A| |x| 2^-47 (float pairs) or better
    x = many.cpu().numpy()
    assert np.linalg.norm(res) <= 2e-12 * np.linalg.norm(b) + 2.0**-44 * np.linalg.norm(abs(A) @ abs(x))
    assert np.array_equal(x[f], b[f])


@pytest.mark.parametrize("limit", [0, 7, 50, 63, 100, 117])
def test_stop_at_the_iteration_limit(limit, monkeypatch):
    from edelweissfe_gb300 import solver

    asm, K, R, fixed = _system("fp64")
    one, s1 = _solve(asm, K, R, fixed, pcgTolerance=1e-14, pcgMaxIter=limit)
    monkeypatch.setattr(solver, "LAUNCH_SECONDS", 0.0)
    many, s2 = _solve(asm, K, R, fixed, pcgTolerance=1e-14, pcgMaxIter=limit)
    assert s1.linearIterations[-1] == s2.linearIterations[-1] == limit and not s2.linearConverged[-1]
    assert torch.equal(one, many)
    if limit == 0:
        free = torch.ones_like(R, dtype=torch.bool)
        free[fixed] = False
        assert (many[free] == 0).all() and torch.equal(many[fixed], R[fixed])


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_multigrid_graph_replay_matches_direct_launches(precision):
    asm, K, R, fixed = _system(precision, size=(14, 12, 10))
    xg, g = _solve(asm, K, R, fixed, pcgTolerance=1e-13, pcgPreconditioner="amg")
    xd, d = _solve(asm, K, R, fixed, pcgTolerance=1e-13, pcgPreconditioner="amg", pcgGraphs=False)
    assert g.linearIterations == d.linearIterations and g.linearIterations[-1] >= 40  # two graph replays or more
    assert torch.equal(xg, xd)
