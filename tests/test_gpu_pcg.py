"""The persistent CG kernel (efe_pcg_solve, efe_pcg_iterate) at the edges of its dispatch: one cluster, a few CTAs and a
full grid; node blocks of 2 and 3 and per-entry columns; FP64, float-float and FP64-on-float products; point and block
Jacobi, also with blocks that the product's rows do not follow; values and columns that are not 16-byte aligned, and
rows longer than a copy holds.  Against SciPy's direct solve at a relative tolerance of 1e-14: the error is bounded by
the condition number (below 1e5 here) times that, so 1e-9 as in the other solver tests."""

import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _matrix(nodes, bs, reach, seed, hub=0):
    """SPD CSR matrix of `nodes` node blocks of bs DOFs, each coupled to the next `reach` nodes; node 0 to the first
    `hub` nodes."""
    import scipy.sparse as sp

    rng = np.random.default_rng(seed)
    i = np.repeat(np.arange(nodes), reach)
    j = i + np.tile(np.arange(1, reach + 1), nodes)
    keep = j < nodes
    i, j = np.concatenate([i[keep], np.zeros(max(hub - 1, 0), int)]), np.concatenate([j[keep], np.arange(1, max(hub, 1))])
    pairs = np.unique(i * nodes + j)
    i, j = pairs // nodes, pairs % nodes
    ii = (bs * i[:, None, None] + np.arange(bs)[None, :, None]).repeat(bs, 2).ravel()
    jj = (bs * j[:, None, None] + np.arange(bs)[None, None, :]).repeat(bs, 1).ravel()
    v = rng.uniform(-1, 1, len(ii))
    A = sp.coo_matrix((v, (ii, jj)), shape=(nodes * bs,) * 2).tocsr()
    d = sp.kron(sp.identity(nodes), np.ones((bs, bs)))  # full diagonal blocks
    A = A + A.T
    D = sp.diags(np.asarray(abs(A).sum(1)).ravel() + rng.uniform(bs, 2 * bs, nodes * bs))
    A = (A + 0.1 * d + D).tocsr()
    A.sort_indices()
    return A


def _setup(A, bs, blockSize, precision, pFF=True, blocks=True, offset=0):
    from edelweissfe_gb300 import _lib as L

    dev = torch.device("cuda", 0)
    n = A.shape[0]
    kdt = torch.float64 if precision == "fp64" else torch.float32
    vals = torch.empty(A.nnz + offset, dtype=kdt, device=dev)[offset:]
    vals.copy_(torch.tensor(A.data))
    Ah = A.copy()
    Ah.data = vals.double().cpu().numpy()
    ip = torch.tensor(A.indptr, dtype=torch.int32, device=dev)
    ix = torch.tensor(A.indices, dtype=torch.int32, device=dev)
    cols = None
    if blocks and bs > 1:
        cols = torch.tensor(np.concatenate([A.indices[A.indptr[r] : A.indptr[r + 1]][::bs] for r in range(0, n, bs)]),
                            dtype=torch.int32, device=dev)  # fmt: skip
    if blockSize == 1:
        dinv = torch.tensor(1.0 / Ah.diagonal(), device=dev)
    else:
        dense = np.stack([Ah[k : k + blockSize, k : k + blockSize].toarray() for k in range(0, n, blockSize)])
        dinv = torch.tensor(np.linalg.inv(0.5 * (dense + dense.transpose(0, 2, 1))), device=dev)
    vec = torch.zeros((5, n), dtype=torch.float64, device=dev)
    work = torch.full((L.EFE_PCG_WORK_DOUBLES,), 3.25, dtype=torch.float64, device=dev)
    pf = torch.empty((n, 2), dtype=torch.float32, device=dev) if precision != "fp64" and pFF else None
    kp = L.EFE_K_FP64 if precision == "fp64" else L.EFE_K_FP32
    s = L.EfePcg(n, ip.data_ptr(), ix.data_ptr(), vals.data_ptr(), kp, None, dinv.data_ptr(),
                 *[vec[i].data_ptr() for i in range(5)], work.data_ptr(), pf.data_ptr() if pf is not None else None,
                 blockSize, bs if blocks else 0)  # fmt: skip
    return s, cols, vec, work, Ah, (ip, ix, vals, dinv, pf)


def _solve(s, cols, work, A, b, tol=1e-14, steps=400):
    from edelweissfe_gb300 import _lib as L

    lib = L.load()
    st = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    L.check(lib.efe_pcg_start(ctypes.byref(s), ctypes.c_void_p(b.data_ptr()), st), "efe_pcg_start")
    c = ctypes.c_void_p(cols.data_ptr() if cols is not None else None)
    tol2 = (tol * float(b.norm())) ** 2
    for k in range(0, 4 * steps, steps):
        L.check(lib.efe_pcg_solve(ctypes.byref(s), c, A.nnz, k, steps, 10, tol2, st), "efe_pcg_solve")
    return work[:8].cpu().numpy()


# (nodes, DOFs per node, neighbours ahead, hub): a single group; one cluster; a few CTAs; more chunks than warps;
# Hexa20-like long rows; one row group far longer than a copy
SHAPES = [(1, 3, 1, 0), (40, 2, 4, 0), (211, 3, 13, 0), (1000, 3, 13, 0), (3001, 2, 4, 0), (21000, 3, 13, 0), (700, 3, 40, 0),
          (2500, 3, 13, 2400), (257, 1, 13, 0)]  # fmt: skip


@pytest.mark.parametrize("nodes,bs,reach,hub", SHAPES)
@pytest.mark.parametrize("precision,pFF", [("fp64", False), ("mixed", True), ("mixed", False)])
def test_solve_matches_direct(nodes, bs, reach, hub, precision, pFF):
    import scipy.sparse.linalg as sla

    A = _matrix(nodes, bs, reach, nodes, hub)
    rng = np.random.default_rng(2)
    b = rng.normal(size=A.shape[0])
    bd = torch.tensor(b, device="cuda")
    variants = [(1, True, 0), (1, False, 0), (1, True, 1)] + ([(bs, True, 0), (bs, False, 0)] if bs > 1 else [])
    for blockSize, blocks, offset in variants:
        s, cols, vec, work, Ah, keep = _setup(A, bs, blockSize, precision, pFF, blocks, offset)
        w = _solve(s, cols, work, A, bd)
        assert w[5] == 1.0 and 0 < w[6] <= 400 and w[6] % 10 == 0, (blockSize, blocks, offset, w)
        x = vec[0].cpu().numpy()
        ref = sla.spsolve(Ah.tocsc(), b)
        assert np.abs(x - ref).max() <= 1e-9 * np.abs(ref).max(), (blockSize, blocks, offset)
        first = vec[0].clone()
        _solve(s, cols, work, A, bd)
        assert torch.equal(first, vec[0])  # fixed-order sums


@pytest.mark.parametrize("nodes", [100, 4000])
def test_iterations_in_pieces_and_in_a_graph(nodes):
    """efe_pcg_iterate: 12 iterations as 12, as 5 + 7 and as a captured graph give the same bits."""
    from edelweissfe_gb300 import _lib as L

    lib = L.load()
    A = _matrix(nodes, 3, 13, 5)
    b = torch.tensor(np.random.default_rng(3).normal(size=A.shape[0]), device="cuda")
    s, _, vec, work, _, keep = _setup(A, 3, 1, "fp64")

    def start():
        st = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
        L.check(lib.efe_pcg_start(ctypes.byref(s), ctypes.c_void_p(b.data_ptr()), st), "efe_pcg_start")

    def iterate(k, n):
        st = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
        L.check(lib.efe_pcg_iterate(ctypes.byref(s), k, n, st), "efe_pcg_iterate")

    start()
    iterate(0, 12)
    whole, rr = vec[0].clone(), work[2].clone()
    start()
    iterate(0, 5)
    iterate(5, 7)
    assert torch.equal(whole, vec[0]) and torch.equal(rr, work[2])
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        start()
        iterate(0, 12)
    for _ in range(2):
        vec.zero_()
        g.replay()
        assert torch.equal(whole, vec[0])


def test_two_streams():
    """Solves in flight on two streams at once give the answers of solves one after the other."""
    A = _matrix(30000, 3, 13, 7)
    b = torch.tensor(np.random.default_rng(4).normal(size=A.shape[0]), device="cuda")
    a = [_setup(A, 3, 1, "mixed") for _ in range(2)]
    _solve(a[0][0], a[0][1], a[0][3], A, b)
    ref = a[0][2][0].clone()
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in range(2)]
    for s, st in zip(a, streams):
        with torch.cuda.stream(st):
            s[2].zero_()
            _launch(s, A, b)
    torch.cuda.synchronize()
    for s in a:
        assert s[3][5].item() == 1.0
        assert torch.equal(ref, s[2][0])


def _launch(s, A, b):
    from edelweissfe_gb300 import _lib as L

    lib = L.load()
    st = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    L.check(lib.efe_pcg_start(ctypes.byref(s[0]), ctypes.c_void_p(b.data_ptr()), st), "efe_pcg_start")
    tol2 = 1e-28 * A.shape[0]  # no host read between the launches
    L.check(lib.efe_pcg_solve(ctypes.byref(s[0]), ctypes.c_void_p(s[1].data_ptr()), A.nnz, 0, 400, 10, tol2, st),
            "efe_pcg_solve")  # fmt: skip
