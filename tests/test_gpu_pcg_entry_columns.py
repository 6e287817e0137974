"""CG products with one column index per entry (efe_pcg_iterate, whose caller gives no block columns and no entry count;
efe_pcg_solve without block columns) around the size from which four lanes instead of eight work on a row (more rows
than four to every warp of the grid), with rows that fit a warp's copy, rows that do not, and one very long row, with
every preconditioner block.  Against the host's CG in FP64 on the same values: after `steps` iterations from the same
start the two differ by rounding only, amplified by at most the condition number (below 100, from the diagonal's
dominance) in each of the few steps taken: 1e-10 of the largest entry."""

import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _host_cg(A, Minv, b, steps):
    x, r = np.zeros_like(b), b.copy()
    z = Minv(r)
    p, rz = z.copy(), r @ z
    for _ in range(steps):
        q = A @ p
        alpha = rz / (p @ q)
        x += alpha * p
        r -= alpha * q
        z = Minv(r)
        rz, old = r @ z, rz
        p = z + rz / old * p
    return x


@pytest.mark.parametrize("nodes,bs,reach,hub", [(3242, 3, 13, 0), (3243, 3, 13, 0), (5001, 2, 45, 0), (4000, 3, 13, 3900),
                                                (9729, 1, 40, 0)])  # fmt: skip
@pytest.mark.parametrize("precision,pFF", [("fp64", False), ("mixed", True), ("mixed", False)])
def test_iterations_match_the_host(nodes, bs, reach, hub, precision, pFF):
    from edelweissfe_gb300 import _lib as L
    from test_gpu_pcg import _matrix, _setup

    lib = L.load()
    A = _matrix(nodes, bs, reach, nodes, hub)
    n = A.shape[0]
    b = np.random.default_rng(1).normal(size=n)
    bd = torch.tensor(b, device="cuda")
    st = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    steps = 12
    for blockSize in sorted({1, bs}):
        s, _, vec, work, Ah, keep = _setup(A, bs, blockSize, precision, pFF, blocks=False)
        D = keep[3].cpu().numpy()
        Minv = (lambda r: D * r) if blockSize == 1 else (lambda r: np.einsum("kij,kj->ki", D, r.reshape(-1, blockSize)).ravel())
        ref = _host_cg(Ah, Minv, b, steps)
        for nnz in (None, 0, A.nnz):  # efe_pcg_iterate; efe_pcg_solve
            L.check(lib.efe_pcg_start(ctypes.byref(s), ctypes.c_void_p(bd.data_ptr()), st), "efe_pcg_start")
            if nnz is None:
                L.check(lib.efe_pcg_iterate(ctypes.byref(s), 0, steps, st), "efe_pcg_iterate")
            else:
                L.check(lib.efe_pcg_solve(ctypes.byref(s), None, nnz, 0, steps, steps, 0.0, st), "efe_pcg_solve")
            x = vec[0].cpu().numpy()
            assert work[5].item() == 0.0
            assert np.abs(x - ref).max() <= 1e-10 * np.abs(ref).max(), (blockSize, nnz)
