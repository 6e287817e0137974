"""The work that a user of this framework has it do, as cases that can be timed and compared.

One Newton iteration of an implicit static simulation is an element pass (`GPUAssembler.computeElements`:
material update, residual, tangent, CSR assembly) and a linear solve (`NISTGPU.linearSolve`, device CG);
gradients add one reverse element pass (`GPUAssembler.adjointTL`, `GPUAssembler.adjointSmallStrain`).
Every case is one such call through the public entry points, on the element types, materials, precisions
and sizes of this repository's configurations, tests and benchmark:

* "pass": one element pass on a structured mesh with jittered nodes.  Small strain: the second increment of
  a uniaxial strain path, the first accepted (so that von Mises points are plastic); total Lagrangian: an
  affine deformation I + 0.05 N(0, 1) plus 0.2 % of the element size of noise.
* "batch": one persistent pass over a batch of uneven 2D and 3D meshes, replayed as a CUDA graph.
* "solve": one Newton system: a clamped block whose opposite face is moved, elements with log-normal moduli.
* "adjoint_tl", "adjoint_ss": the reverse pass of the total-Lagrangian / small-strain element residual.

Meshes are numbered like the structured generators' (x outer, z inner).
"""

import math

import numpy as np
import torch

# natural coordinates of the nodes in the element's node order
_QUAD = [(-1, -1), (1, -1), (1, 1), (-1, 1), (0, -1), (1, 0), (0, 1), (-1, 0)]
_HEXA = [(-1, -1, -1), (-1, -1, 1), (1, -1, 1), (1, -1, -1), (-1, 1, -1), (-1, 1, 1), (1, 1, 1), (1, 1, -1),
         (-1, -1, 0), (0, -1, 1), (1, -1, 0), (0, -1, -1), (-1, 1, 0), (0, 1, 1), (1, 1, 0), (0, 1, -1),
         (-1, 0, -1), (-1, 0, 1), (1, 0, 1), (1, 0, -1)]  # fmt: skip
# element type -> (dimension, nodes, quadrature points)
_TYPES = {
    "CPE4": (2, 4, 4), "CPS4": (2, 4, 4), "CPE8": (2, 8, 9), "CPE8R": (2, 8, 4), "CPE8RTL": (2, 8, 4),
    "C3D8": (3, 8, 8), "C3D8TL": (3, 8, 8), "C3D20": (3, 20, 27), "C3D20R": (3, 20, 8), "C3D20TL": (3, 20, 27),
}  # fmt: skip


def listed():
    return [
        # smallest call: the 40 x 8 linear-elastic plate, latency of one element pass in a small simulation
        dict(name="pass_cpe4_plate_fp64", kind="pass", elType="CPE4", material="linearelastic", precision="fp64",
             nx=40, ny=8, nz=0),
        # the default precision on an ordinary solid block
        dict(name="pass_c3d8_j2_fp64", kind="pass", elType="C3D8", material="vonmises", precision="fp64",
             nx=33, ny=31, nz=29),
        # the headline: a 64^3 von Mises block, FP32 tangent with FP64 residual
        dict(name="pass_c3d8_j2_mixed_64", kind="pass", elType="C3D8", material="vonmises", precision="mixed",
             nx=64, ny=64, nz=64),
        # the same pass with the float-float residual, ragged sizes
        dict(name="pass_c3d8_j2_ff", kind="pass", elType="C3D8", material="vonmises", precision="mixed-ff",
             nx=41, ny=37, nz=43),
        # the element pass of the plastic path adjoint's forward run
        dict(name="pass_c3d20_j2_mixed", kind="pass", elType="C3D20", material="vonmises", precision="mixed",
             nx=48, ny=48, nz=24),
        # quadratic solids in the default precision
        dict(name="pass_c3d20_j2_fp64", kind="pass", elType="C3D20", material="vonmises", precision="fp64",
             nx=17, ny=16, nz=9),
        # uneven meshes (parameter studies): one persistent launch over 2D and 3D meshes in a CUDA graph
        dict(name="batch_neohooke_mixed", kind="batch", precision="mixed", meshes=24, scale=0.1),
        # Newton's linear systems: the headline block with an FP32 tangent, an FP64 tangent, and a small plate
        dict(name="solve_c3d8_mixed_64", kind="solve", elType="C3D8", precision="mixed", nx=64, ny=64, nz=64),
        dict(name="solve_c3d8_fp64_32", kind="solve", elType="C3D8", precision="fp64", nx=32, ny=32, nz=32),
        dict(name="solve_cpe4_plate_fp64", kind="solve", elType="CPE4", precision="fp64", nx=40, ny=8, nz=0),
        # gradients: Neo-Hooke coordinates and moduli at 32^3; one reverse pass of a plastic increment
        dict(name="adjoint_tl_c3d8_32", kind="adjoint_tl", elType="C3D8TL", material="neohookewa", precision="fp64",
             nx=32, ny=32, nz=32),
        dict(name="adjoint_ss_c3d20", kind="adjoint_ss", elType="C3D20", precision="mixed", nx=24, ny=24, nz=12,
             coordinates=False),
    ]  # fmt: skip


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _sizes(rng, dim, elements):
    """Edge counts of an uneven block of about `elements` elements."""
    n = elements ** (1.0 / dim)
    a = max(1, round(n * rng.uniform(0.7, 1.4)))
    if dim == 2:
        return dict(nx=a, ny=max(1, round(elements / a)), nz=0)
    b = max(1, round(n * rng.uniform(0.7, 1.4)))
    return dict(nx=a, ny=b, nz=max(1, round(elements / (a * b))))


# element passes in use: (element type, materials, largest mesh in FP64, with an FP32 tangent)
_PASSES = [
    ("CPE4", ["linearelastic", "vonmises"], 60000, 200000), ("CPS4", ["linearelastic"], 60000, 200000),
    ("CPE8", ["linearelastic", "vonmises"], 20000, 60000), ("CPE8R", ["vonmises"], 20000, 80000),
    ("CPE8RTL", ["neohookewa", "neohookewb"], 20000, 80000), ("C3D8", ["linearelastic", "vonmises"], 50000, 250000),
    ("C3D8TL", ["neohookewa", "neohookewb", "neohookewc"], 30000, 120000),
    ("C3D20", ["linearelastic", "vonmises"], 4000, 50000), ("C3D20R", ["vonmises"], 6000, 30000),
    ("C3D20TL", ["neohookewa", "neohookewb"], 4000, 50000),
]  # fmt: skip


def draw(rng):
    kind = rng.choice(["pass"] * 10 + ["solve"] * 5 + ["adjoint_tl", "adjoint_ss", "adjoint_ss", "batch"])
    precision = rng.choice(["fp64", "mixed", "mixed-ff"])
    if kind == "pass":
        elType, materials, most64, most32 = rng.choice(_PASSES)
        size = _log_int(rng, 250, most64 if precision == "fp64" else most32)
        return dict(kind=kind, elType=elType, material=rng.choice(materials), precision=precision,
                    **_sizes(rng, _TYPES[elType][0], size))  # fmt: skip
    if kind == "solve":
        elType, most = rng.choice([("CPE4", 4000), ("C3D8", 100000), ("C3D8", 100000), ("C3D20", 5000)])
        size = _log_int(rng, 100, most // 2 if precision == "fp64" else most)
        return dict(kind=kind, elType=elType, precision=precision, **_sizes(rng, _TYPES[elType][0], size))
    if kind == "batch":
        return dict(kind=kind, precision=precision if precision != "fp64" else "mixed", meshes=2 * rng.randint(2, 16),
                    scale=round(math.exp(rng.uniform(math.log(0.02), math.log(0.12))), 4))  # fmt: skip
    if kind == "adjoint_tl":
        elType = rng.choice(["C3D8TL", "C3D8TL", "C3D20TL", "CPE8RTL"])
        most = {"C3D8TL": 60000, "C3D20TL": 6000, "CPE8RTL": 60000}[elType]
        return dict(kind=kind, elType=elType, material=rng.choice(["neohookewa", "neohookewb", "neohookewc"]),
                    precision="fp64", **_sizes(rng, _TYPES[elType][0], _log_int(rng, 250, most)))  # fmt: skip
    elType = rng.choice(["C3D20", "C3D8", "CPE8"])
    most = {"C3D20": 7000, "C3D8": 60000, "CPE8": 40000}[elType]
    return dict(kind=kind, elType=elType, precision=precision, coordinates=rng.random() < 0.3,
                **_sizes(rng, _TYPES[elType][0], _log_int(rng, 250, most)))  # fmt: skip


# ------------------------------------------------------------------ meshes and inputs (host, from the seed)
def _mesh(elType, n, rng, jitter=0.05, lengths=None):
    """coords [n, d], conn [E, nn] (int32) of a structured block, inner nodes moved by up to `jitter` of an
    element edge."""
    d, nn, _ = _TYPES[elType]
    n = np.array(n[:d])
    nat = np.array((_QUAD if d == 2 else _HEXA)[:nn])
    f = 2 if nn > 2**d else 1
    cells = np.stack(np.meshgrid(*[np.arange(k) for k in n], indexing="ij"), -1).reshape(-1, d)
    grid = f * n + 1
    flat = np.zeros((len(cells), nn), np.int64)
    for c in range(d):
        flat = flat * grid[c] + f * cells[:, None, c] + (nat[None, :, c] + 1) * f // 2
    used = np.zeros(int(grid.prod()), bool)
    used[flat.ravel()] = True
    conn = (np.cumsum(used) - 1)[flat].astype(np.int32)
    ijk = np.stack(np.unravel_index(np.nonzero(used)[0], grid), 1)
    lengths = np.ones(d) if lengths is None else np.asarray(lengths, float)
    coords = ijk / (f * n) * lengths
    inside = np.all((ijk > 0) & (ijk < f * n), axis=1)
    coords[inside] += rng.uniform(-jitter, jitter, (int(inside.sum()), d)) * lengths / n
    return coords, conn


def _edges(case):
    return (case["nx"], case["ny"]) if _TYPES[case["elType"]][0] == 2 else (case["nx"], case["ny"], case["nz"])


def _props(case, E, rng):
    if case["material"] == "linearelastic":
        return np.tile([210e3, 0.3], (E, 1))
    if case["material"] == "vonmises":  # per-element yield stress and hardening, as in the plastic path adjoint
        p = np.tile([210e3, 0.3, 250.0, 1000.0, 0.0, 0.0], (E, 1))
        p[:, 2] = rng.uniform(200, 300, E)
        p[:, 3] = rng.uniform(800, 1200, E)
        return p
    mod = 1000.0 * np.exp(0.3 * rng.normal(size=E))  # log-normal Young's moduli, nu = 0.3
    return np.stack([mod / 2.6, mod / 1.2], 1)


def _inputs(case, seed):
    """coords, conn, props and displacements of a pass or of an adjoint: small strain (first increment,
    second increment), total Lagrangian (total displacement)."""
    rng = np.random.default_rng(seed)
    n = _edges(case)
    coords, conn = _mesh(case["elType"], n, rng)
    case = dict(case, material=case.get("material", "vonmises"))
    props = _props(case, len(conn), rng)
    h = 1.0 / max(n)
    d = coords.shape[1]
    if case["elType"].endswith("TL"):
        F = np.eye(d) + 0.05 * rng.normal(size=(d, d))
        U = coords @ (F - np.eye(d)).T + 0.002 * h * rng.normal(size=coords.shape)
        return coords, conn, props, U.ravel(), None
    dU1, dU2 = np.zeros_like(coords), np.zeros_like(coords)
    dU1[:, 1] = 0.0025 * (1 + 0.1 * rng.uniform(-1, 1)) * coords[:, 1]
    dU2[:, 1] = 0.00025 * coords[:, 1]
    dU2 += 6e-5 * h * rng.uniform(-1, 1, coords.shape)
    return coords, conn, props, dU1.ravel(), dU2.ravel()


def _batch_inputs(case, seed):
    """(element type, coords, conn, props, U) of every mesh: even index Quad8 plane strain, odd Hexa20; element
    counts log-uniform in [1e3, 5e4] times `scale` (the same for every seed)."""
    sizes, rng = np.random.default_rng(3), np.random.default_rng(seed)
    out = []
    for i in range(case["meshes"]):
        n = max(2, int(round(np.exp(sizes.uniform(np.log(1e3), np.log(5e4))) * case["scale"])))
        mu = float(np.exp(rng.uniform(np.log(1e2), np.log(1e4))))
        elType = "C3D20TL" if i % 2 else "CPE8RTL"
        d = _TYPES[elType][0]
        nx = max(1, int(round(n ** (1.0 / d))))
        last = int(np.ceil(n / nx ** (d - 1)))
        coords, conn = _mesh(elType, [nx] * (d - 1) + [last], rng, lengths=[1.0] * (d - 1) + [last / nx])
        F = np.eye(d) + 0.05 * rng.normal(size=(d, d))
        U = coords @ (F - np.eye(d)).T + 0.002 / nx * rng.normal(size=coords.shape)
        out.append((elType, coords, conn, np.array([mu, 10.0 * mu]), U.ravel()))
    return out


def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _solve_inputs(case, seed):
    """coords, conn, the CSR values of the tangent (canonical order), the right-hand side (prescribed values on
    prescribed DOFs, loads elsewhere) and the prescribed DOFs.  The element stiffnesses are rounded to a
    common grid, so that their sums are the same in any order."""
    rng = np.random.default_rng(seed)
    n = _edges(case)
    d, nn, _ = _TYPES[case["elType"]]
    coords, conn = _mesh(case["elType"], n, rng)
    E = torch.as_tensor(np.exp(0.3 * rng.normal(size=len(conn))), device=_device())
    lam, mu = 0.3 / 1.3 / 0.4 * 210e3, 210e3 / 2.6
    cn = torch.as_tensor(conn, device=_device(), dtype=torch.int64)
    Ke = []
    for X, e in zip(torch.as_tensor(coords, device=_device())[cn].split(20000), E.split(20000)):
        G, s = _geometry(case["elType"], X)
        s = s * e[:, None]
        GG = torch.einsum("eq,eqja,eqkb->eajbk", s, G, G)
        dot = torch.einsum("eajbj->eab", GG)
        k = lam * GG + mu * GG.permute(0, 1, 4, 3, 2)
        k += mu * torch.einsum("eab,jk->eajbk", dot, torch.eye(d, dtype=torch.float64, device=e.device))
        Ke.append(k.reshape(len(e), nn * d, nn * d))
    Ke = torch.cat(Ke)
    unit = 2.0 ** (math.floor(math.log2(1e6 / min(n))) - 44)
    _, values = _assemble(torch.round(Ke / unit) * unit, cn, d, len(coords))
    if case["precision"] != "fp64":
        values = values.to(torch.float32)
    c1 = coords[:, 1]
    nodes = np.arange(len(coords))
    bottom, top = nodes[c1 < 1e-9], nodes[c1 > 1 - 1e-9]
    fixed = np.unique(np.concatenate([(d * bottom[:, None] + np.arange(d)).ravel(), d * top + 1]))
    R = 1.0 * rng.normal(size=d * len(coords))
    R[fixed] = 0.0
    R[d * top + 1] = 1e-3
    return coords, conn, values, R, fixed


# ------------------------------------------------------------------ the calls
def _assembler(case, coords, conn, props):
    from edelweissfe_gb300 import ElementGroup, GPUAssembler

    d = coords.shape[1]
    nodeDof = (d * np.arange(len(coords))).astype(np.int32)
    return GPUAssembler(coords, nodeDof, coords.size, [ElementGroup(case["elType"], case["material"], props, conn)],
                        precision=case["precision"])  # fmt: skip


def prepare(case, seed):
    if case["kind"] == "batch":
        from edelweissfe_gb300.batch import BatchedPass, MeshBatch

        meshes = _batch_inputs(case, seed)
        batches = []
        for elType in ("C3D20TL", "CPE8RTL"):
            mine = [m for m in meshes if m[0] == elType]
            b = MeshBatch([dict(coords=x, conn=c, nodeDof=x.shape[1] * np.arange(len(x)), nDof=x.size, props=p)
                           for _, x, c, p, _ in mine], elType, "neohookewa", case["precision"])  # fmt: skip
            b.U.copy_(torch.as_tensor(np.concatenate([m[4] for m in mine])))
            batches.append(b)
        bp = BatchedPass(batches, persistent=True)
        bp.capture()
        return dict(kind="batch", bp=bp)
    if case["kind"] == "solve":
        from edelweissfe_gb300.solver import NISTGPU

        coords, conn, values, R, fixed = _solve_inputs(case, seed)
        asm = _assembler(dict(case, material="linearelastic"), coords, conn, np.array([210e3, 0.3]))
        return dict(kind="solve", solver=NISTGPU(asm), K=values, R=torch.as_tensor(R, device=asm.device),
                    fixed=torch.as_tensor(fixed, device=asm.device))  # fmt: skip
    coords, conn, props, U1, U2 = _inputs(case, seed)
    case = dict(case, material=case.get("material", "vonmises"))
    asm = _assembler(case, coords, conn, props)
    dev = asm.device
    P, F, K = asm.constructDofVector(), asm.constructDofVector(), asm.constructSystemMatrix()
    U = torch.as_tensor(U1, device=dev)
    dU = U
    if U2 is not None:
        asm.computeElements(None, U, U, P, K, F)
        asm.acceptLastState()
        dU = torch.as_tensor(U2, device=dev)
        U = U + dU
    st = dict(kind=case["kind"], asm=asm, U=U, dU=dU, P=P, F=F, K=K)
    if case["kind"] == "adjoint_tl":
        lam, _ = _seeds(case, seed, coords, props)
        st["lam"] = torch.as_tensor(lam, device=dev)
    elif case["kind"] == "adjoint_ss":
        Pbar, sbar = _seeds(case, seed, coords, props, asm.groups[0]._dev["stateRef"].shape)
        new = lambda *s: torch.zeros(s, dtype=torch.float64, device=dev)  # noqa: E731
        st.update(Pbar=torch.as_tensor(Pbar, device=dev), sbar=torch.as_tensor(sbar, device=dev),
                  before=asm.groups[0]._dev["stateRef"], dUbar=new(coords.size), sout=new(*sbar.shape),
                  gProps=new(*props.shape), gX=new(*coords.shape) if case["coordinates"] else None)  # fmt: skip
    return st


def _seeds(case, seed, coords, props, stateShape=None):
    """Adjoint of the residual (zero on the fixed face) and of the new state."""
    rng = np.random.default_rng(seed + 1000003)
    lam = rng.normal(size=coords.shape) * 1e-3
    lam[coords[:, 1] < 1e-9] = 0.0
    sbar = None
    if stateShape is not None:
        scale = np.array([1e-5] * 6 + [1.0] * 6 + [1.0] * (stateShape[0] - 12))
        sbar = rng.normal(size=stateShape) * scale[:, None]
    return lam.ravel(), sbar


def run(st):
    if st["kind"] == "batch":
        bp = st["bp"]
        bp.replay()
        return [dict(P=b.P, F=b.F, K=b.K, state=b.asm.groups[0]._dev["stateTemp"]) for b in bp.batches]
    if st["kind"] == "solve":
        return st["solver"].linearSolve(st["K"], st["R"], st["fixed"])
    asm = st["asm"]
    if st["kind"] == "adjoint_tl":
        gX, gP = asm.adjointTL(st["U"], st["lam"])
        return dict(gX=gX, gP=gP[0])
    if st["kind"] == "adjoint_ss":
        for k in ("dUbar", "sout", "gProps", "gX"):
            if st[k] is not None:
                st[k].zero_()
        asm.adjointSmallStrain(0, st["before"], st["dU"], st["dUbar"], Pbar=st["Pbar"], stateBarIn=st["sbar"],
                               stateBarOut=st["sout"], gProps=st["gProps"], gX=st["gX"])  # fmt: skip
        return {k: st[k] for k in ("dUbar", "sout", "gProps", "gX") if st[k] is not None}
    st["P"].zero_()
    st["F"].zero_()
    st["K"].zero_()
    asm.computeElements(None, st["U"], st["dU"], st["P"], st["K"], st["F"])
    return dict(P=st["P"], F=st["F"], K=st["K"], state=asm.groups[0]._dev["stateTemp"])


# ------------------------------------------------------------------ what a pass cannot do without
def _counts(elType, n):
    """(elements, nodes, stored entries) of a structured block: nodes and node pairs by inclusion and exclusion
    over the elements' shared faces, edges and corners."""
    d, nn, _ = _TYPES[elType]
    shared = {(2, 4): [2, 1], (2, 8): [3, 1], (3, 8): [4, 2, 1], (3, 20): [8, 3, 1]}[(d, nn)]
    n = list(n)[:d]
    sub = [0] * (d + 1)  # shared entities of codimension k
    for m in range(2**d):
        v = 1
        for c in range(d):
            v *= n[c] - 1 if m >> c & 1 else n[c]
        sub[bin(m).count("1")] += v
    per = [nn] + shared
    nodes = sum((-1) ** k * sub[k] * per[k] for k in range(d + 1))
    pairs = sum((-1) ** k * sub[k] * per[k] ** 2 for k in range(d + 1))
    return sub[0], nodes, pairs * d * d


def _pass_work(elType, n, nState, kBytes, tl):
    d, nn, nq = _TYPES[elType]
    E, nodes, nnz = _counts(elType, n)
    history = E * nq * 8 * (nState if tl else 2 * nState)  # hyperelastic points only write theirs
    bytes_ = history + E * nn * 4 + nodes * d * 8 * 4 + nnz * kBytes + E * 2 * 8
    # gradient, residual, the blocks of the node pairs (symmetric) and about 150 operations of the material
    flops = E * nq * (4 * nn * d * d + nn * (nn + 1) // 2 * d**3 * 2 + 150)
    return dict(bytes=bytes_, flops=flops)


def work(case):
    if case["kind"] == "batch":
        sizes, tot = np.random.default_rng(3), dict(bytes=0, flops=0)
        for i in range(case["meshes"]):
            n = max(2, int(round(np.exp(sizes.uniform(np.log(1e3), np.log(5e4))) * case["scale"])))
            elType = "C3D20TL" if i % 2 else "CPE8RTL"
            d = _TYPES[elType][0]
            nx = max(1, int(round(n ** (1.0 / d))))
            w = _pass_work(elType, [nx] * (d - 1) + [int(np.ceil(n / nx ** (d - 1)))], 13, 4, True)
            tot = {k: tot[k] + w[k] for k in tot}
        return tot
    kBytes = 8 if case["precision"] == "fp64" else 4
    n = _edges(case)
    d, nn, nq = _TYPES[case["elType"]]
    E, nodes, nnz = _counts(case["elType"], n)
    if case["kind"] == "pass":
        return _pass_work(case["elType"], n, 12 if case["material"] == "linearelastic" else 13, kBytes,
                          case["elType"].endswith("TL"))  # fmt: skip
    if case["kind"] == "solve":
        # a Krylov solve carries the prescribed values through every element of the longest edge at least once and
        # back: two products per element edge, each reading the matrix (one column index per node block)
        its = 2 * max(n) * (2 if nn > 2**d else 1)
        return dict(bytes=its * (nnz * kBytes + nnz // (d * d) * 4 + nodes * d * 8 * 2), flops=its * 2 * nnz)
    if case["kind"] == "adjoint_tl":
        return dict(bytes=E * nn * 4 + nodes * d * 8 * 4 + E * 32, flops=E * nq * (12 * nn * d * d + 500))
    return dict(bytes=E * nq * 13 * 8 * 4 + E * nn * 4 + nodes * d * 8 * 4 + E * 6 * 8 * 2,
                flops=E * nq * (6 * nn * d * d + 400))  # fmt: skip


# ------------------------------------------------------------------ the same in plain 64-bit torch
def _shape(p, nn):
    """N_a at natural point p."""
    d = len(p)
    c = torch.as_tensor((_QUAD if d == 2 else _HEXA)[:nn], dtype=torch.float64)
    lin = 1.0 + c * p
    corner = lin.prod(1) / 2**d
    if nn == 2**d:
        return corner
    corner = corner * ((c * p).sum(1) - (d - 1))
    mid = torch.where(c == 0, 1.0 - p * p, lin).prod(1) / 2 ** (d - 1)
    return torch.where((c == 0).any(1), mid, corner)


def _rule(d, nq):
    """Quadrature points (xi, eta, zeta) and weights in the element types' order."""
    g, s = 1.0 / math.sqrt(3.0), math.sqrt(0.6)
    if d == 2 and nq == 4:
        return [(g, g), (g, -g), (-g, -g), (-g, g)], [1.0] * 4
    if d == 2:
        x, y = [0, -1, -1, 1, 1, -1, 0, 1, 0], [0, -1, 1, 1, -1, 0, 1, 0, -1]
        w = [64 / 81] + [25 / 81] * 4 + [40 / 81] * 4
        return [(s * a, s * b) for a, b in zip(x, y)], w
    if nq == 8:
        return [(g * x, g * y, g * z) for x in (-1, 1) for y, z in ((-1, -1), (-1, 1), (1, 1), (1, -1))], [1.0] * 8
    W = [5 / 9, 8 / 9, 5 / 9]
    ijk = [(i, j, k) for i in range(3) for j in range(3) for k in range(3)]
    return [(s * (i - 1), s * (j - 1), s * (k - 1)) for i, j, k in ijk], [W[i] * W[j] * W[k] for i, j, k in ijk]


def _tables(elType, dev):
    """dN/dxi at every point (taken at (eta, xi, zeta)), the table the Jacobian is formed with (Hexa20: the third
    row differentiates the t u monomial of the polynomial fit to zeta instead of xi) and the weights."""
    d, nn, nq = _TYPES[elType]
    pts, w = _rule(d, nq)
    D, M = [], []
    for p in pts:
        q = torch.tensor([p[1], p[0]] + list(p[2:]), dtype=torch.float64)
        dN = torch.func.jacrev(lambda x: _shape(x, nn))(q).T
        D.append(dN)
        m = dN.clone()
        if nn == 20:
            c = np.array(_HEXA, float)
            s, t, u = c.T
            A = np.stack([s**0, s, t, u, s * t, t * u, s * u, s * s, t * t, u * u, s * s * t, s * t * t, t * t * u,
                          t * u * u, s * u * u, s * s * u, s * t * u, s * s * t * u, s * t * t * u, s * t * u * u],
                         1)  # fmt: skip
            m[2] += (p[2] - p[0]) * torch.as_tensor(np.linalg.inv(A)[5])
        M.append(m)
    return torch.stack(D).to(dev), torch.stack(M).to(dev), torch.tensor(w, dtype=torch.float64, device=dev)


def _geometry(elType, X):
    """dN/dX [E, q, d, nn] and det J w [E, q] of elements with node coordinates X [E, nn, d]."""
    D, M, w = _tables(elType, X.device)
    J = torch.einsum("qra,eac->eqrc", M, X)
    return torch.einsum("eqcr,qra->eqca", torch.linalg.inv(J), D), torch.linalg.det(J) * w


_VOIGT = {False: [(0, 0), (1, 1), (2, 2), (0, 1), (0, 2), (1, 2)], True: [(0, 0), (1, 1), (2, 2), (0, 1), (1, 2), (0, 2)]}


def _strain(H):
    """Engineering strain (11, 22, 33, 12, 13, 23) of displacement gradients H [..., d, d]."""
    H = torch.nn.functional.pad(H, (0, 3 - H.shape[-1], 0, 3 - H.shape[-1]))
    return torch.stack([H[..., i, j] if i == j else H[..., i, j] + H[..., j, i] for i, j in _VOIGT[False]], -1)


def _von_mises(sig0, k0, de, props, tangent=False):
    """Radial return of one increment: new stress, kappa and (optionally) the consistent tangent [..., 6, 6].
    props broadcasts against the points: [..., nProps]; two properties: linear elasticity."""
    E, nu = props[..., 0], props[..., 1]
    f = E / ((1 + nu) * (1 - 2 * nu))
    lam, G = f * nu, E / (2 * (1 + nu))
    tr3 = de[..., :3].sum(-1)
    tr = sig0 + torch.cat([(lam * tr3)[..., None] + 2 * G[..., None] * de[..., :3], G[..., None] * de[..., 3:]], -1)
    I6 = torch.diag(torch.tensor([2.0, 2, 2, 1, 1, 1], dtype=de.dtype, device=de.device))
    one = torch.tensor([1.0, 1, 1, 0, 0, 0], dtype=de.dtype, device=de.device)
    C = (lam[..., None, None] * torch.outer(one, one) + G[..., None, None] * I6) if tangent else None
    if props.shape[-1] == 2:
        return tr, k0, None if C is None else C.expand(*de.shape, 6)
    fy0, Hl, dfy, delta = (props[..., i] for i in range(2, 6))
    dev = tr - tr[..., :3].sum(-1, keepdim=True) / 3 * one
    q = torch.sqrt((dev * dev * torch.tensor([1.0, 1, 1, 2, 2, 2], dtype=de.dtype, device=de.device)).sum(-1))
    s23, s6 = math.sqrt(2 / 3), math.sqrt(6.0)
    fy = lambda k: fy0 + Hl * k + dfy * (1 - torch.exp(-delta * k))  # noqa: E731
    dfyk = lambda k: Hl + dfy * delta * torch.exp(-delta * k)  # noqa: E731
    plastic = q - s23 * fy(k0) > 0
    with torch.no_grad():
        dK = torch.zeros_like(q)
        for _ in range(20):
            dK = dK + (q - s6 * G * dK - s23 * fy(k0 + dK)) / (s6 * G + s23 * dfyk(k0 + dK))
        slope = s6 * G + s23 * dfyk(k0 + dK)
    dK = dK + (q - s6 * G * dK - s23 * fy(k0 + dK)) / slope  # carries the derivatives of the converged step
    dK = torch.where(plastic, dK, torch.zeros_like(dK))
    g2 = 2 * G * math.sqrt(1.5) * dK
    n = dev / q[..., None]
    sig, k = tr - g2[..., None] * n, k0 + dK
    if tangent:
        Idev = 0.5 * I6 - torch.outer(one, one) / 3
        a = 2 * G * (1 / (1 + dfyk(k) / (3 * G)) - g2 / q)
        Cp = C - (2 * G * g2 / q)[..., None, None] * Idev - a[..., None, None] * n[..., :, None] * n[..., None, :]
        C = torch.where(plastic[..., None, None], Cp, C)
    return sig, k, C


def _plane_stress_elastic(sig0, de, props):
    E, nu = props[..., 0], props[..., 1]
    f = E / (1 - nu * nu)
    C = torch.zeros((*de.shape, 6), dtype=de.dtype, device=de.device)
    C[..., 0, 0] = C[..., 1, 1] = f
    C[..., 0, 1] = C[..., 1, 0] = f * nu
    C[..., 3, 3] = f * (1 - nu) / 2
    sig = sig0 + torch.einsum("...ij,...j->...i", C, de)
    de = de.clone()
    de[..., 2] = -nu / (1 - nu) * (de[..., 0] + de[..., 1])
    return sig, de, C


def _neo_hooke(material, F, mu, K):
    """Kirchhoff stress [3, 3] and energy at F [3, 3]."""
    J, B = torch.linalg.det(F), F @ F.T
    I1, I = B.diagonal().sum(), torch.eye(3, dtype=F.dtype, device=F.device)
    if material == "neohookewa":
        tau = mu * B + ((K - 2 / 3 * mu) * (J * J - J) - mu) * I
        return tau, mu / 2 * (I1 - 3) + (K / 2 - mu / 3) * (J - 1) ** 2 - mu * torch.log(J)
    if material == "neohookewb":
        m = mu * J ** (-2 / 3)
        tau = m * B + (K / 4 * (J * J - J**-2) - m / 3 * I1) * I
        return tau, mu / 2 * (I1 * J ** (-2 / 3) - 3) + K / 8 * (J * J + J**-2 - 2)
    p = J ** (2 / 3 - K / mu)
    return mu * B - mu * p * I, mu / 2 * (F.diagonal().sum() - 3) + 3 * mu * mu / (3 * K - 2 * mu) * (p - 1)


def _embed(Fd):
    """3 x 3 deformation gradients of plane ones (plane strain)."""
    d = Fd.shape[-1]
    return Fd if d == 3 else torch.nn.functional.pad(Fd, (0, 1, 0, 1)) + torch.diag(
        torch.tensor([0.0, 0, 1], dtype=Fd.dtype, device=Fd.device))  # fmt: skip


def _assemble(Ke, conn, d, nNodes):
    """(keys row * n + column, values) of the canonical CSR matrix of element matrices Ke [E, nd, nd]."""
    n = nNodes * d
    dof = (d * conn[:, :, None] + torch.arange(d, device=conn.device)).reshape(len(conn), -1)
    key, at = torch.unique((dof[:, :, None] * n + dof[:, None, :]).reshape(-1), return_inverse=True)
    return key, torch.zeros(len(key), dtype=Ke.dtype, device=Ke.device).index_add_(0, at, Ke.reshape(-1))


def _exact_pass(elType, material, coords, conn, props, U1, U2):
    dev = _device()
    d, nn, nq = _TYPES[elType]
    cn = torch.as_tensor(conn, device=dev, dtype=torch.int64)
    X = torch.as_tensor(coords, device=dev)
    pr = torch.as_tensor(np.broadcast_to(props, (len(conn), props.shape[-1])).copy(), device=dev)
    u = [torch.as_tensor(v, device=dev).reshape(-1, d) for v in (U1, U2) if v is not None]
    tl = elType.endswith("TL")
    Pe, Ke, states = [], [], []
    step = max(1, 40000000 // (nq * nn * nn * d * d))
    for e0 in range(0, len(conn), step):
        c, p = cn[e0 : e0 + step], pr[e0 : e0 + step, None, :]
        G, s = _geometry(elType, X[c])
        if tl:
            F = _embed(torch.einsum("eai,eqja->eqij", u[0][c], G) + torch.eye(d, dtype=G.dtype, device=dev))

            def first_pk(F, mu, K):
                return (_neo_hooke(material, F, mu, K)[0] @ torch.linalg.inv(F).T)[:d, :d]

            flat = F.reshape(-1, 3, 3)
            mu, K = (p[..., i].expand(F.shape[:2]).reshape(-1) for i in (0, 1))
            tau, W = torch.func.vmap(lambda f, m, k: _neo_hooke(material, f, m, k))(flat, mu, K)
            pk = torch.func.vmap(first_pk)(flat, mu, K).reshape(*s.shape, d, d)
            A = torch.func.vmap(torch.func.jacrev(first_pk))(flat, mu, K)[..., :d, :d].reshape(*s.shape, d, d, d, d)
            pe = -torch.einsum("eq,eqij,eqja->eai", s, pk, G)
            T = torch.einsum("eq,eqiJkL,eqJa->eqaikL", s, A, G)
            ke = torch.einsum("eqaikL,eqLb->eaibk", T, G)
            H = F - torch.eye(3, dtype=F.dtype, device=dev)
            Eg = 0.5 * (H + H.mT + H.mT @ H)
            st = [tau.reshape(*s.shape, 3, 3)[..., i, j] for i, j in _VOIGT[True]]
            st += [Eg[..., i, j] * (1 if i == j else 2) for i, j in _VOIGT[True]] + [W.reshape(s.shape)]
        else:
            sig = torch.zeros((*s.shape, 6), dtype=torch.float64, device=dev)
            eps, k = sig.clone(), sig[..., 0].clone()
            for v in u:
                de = _strain(torch.einsum("eai,eqja->eqij", v[c], G))
                if elType.startswith("CPS"):
                    sig, de, C = _plane_stress_elastic(sig, de, p)
                else:
                    sig, k, C = _von_mises(sig, k, de, p, tangent=True)
                eps = eps + de
            rows = [(v, i, j) for v, (i, j) in enumerate(_VOIGT[False]) if max(i, j) < d]
            B = torch.zeros((*s.shape, len(rows), nn, d), dtype=torch.float64, device=dev)
            for r, (_, i, j) in enumerate(rows):
                B[:, :, r, :, i] += G[:, :, j]
                if i != j:
                    B[:, :, r, :, j] += G[:, :, i]
            B = B.reshape(*s.shape, len(rows), nn * d)
            act = [v for v, _, _ in rows]
            pe = -torch.einsum("eq,eqr,eqrn->en", s, sig[..., act], B)
            CB = torch.einsum("eq,eqrt,eqtn->eqrn", s, C[..., act, :][..., act], B)
            ke = torch.einsum("eqrm,eqrn->emn", B, CB)
            st = list(sig.unbind(-1)) + list(eps.unbind(-1)) + ([k] if pr.shape[1] > 2 else [])
        Pe.append(pe.reshape(len(c), -1))
        Ke.append(ke.reshape(len(c), nn * d, nn * d))
        states.append(torch.stack(st).reshape(len(st), -1))
    dof = (d * cn[:, :, None] + torch.arange(d, device=dev)).reshape(-1)
    Pe, Ke = torch.cat(Pe), torch.cat(Ke)
    zero = torch.zeros(X.numel(), dtype=torch.float64, device=dev)
    _, K = _assemble(Ke, cn, d, len(coords))
    return dict(P=zero.clone().index_add_(0, dof, Pe.reshape(-1)), F=zero.index_add_(0, dof, Pe.abs().reshape(-1)), K=K,
                state=torch.cat(states, 1))  # fmt: skip


def _exact_solve(case, seed):
    """Conjugate gradients in 64 bits far beyond the tolerance asked for, on the free DOFs."""
    coords, conn, values, R, fixed = _solve_inputs(case, seed)
    dev, d, n = _device(), coords.shape[1], coords.size
    cn = torch.as_tensor(conn, device=dev, dtype=torch.int64)
    dof = (d * cn[:, :, None] + torch.arange(d, device=dev)).reshape(len(conn), -1)
    key = torch.unique((dof[:, :, None] * n + dof[:, None, :]).reshape(-1))
    row, col = key // n, key % n
    crow = torch.searchsorted(row, torch.arange(n + 1, device=dev))
    A = torch.sparse_csr_tensor(crow, col, values.double(), size=(n, n))
    free = torch.ones(n, dtype=torch.float64, device=dev)
    free[torch.as_tensor(fixed, device=dev)] = 0.0
    dinv = free / values.double()[row == col]
    R = torch.as_tensor(R, device=dev)
    xd = R * (1 - free)
    x = torch.zeros_like(R)
    b = free * (R - A @ xd)
    for _ in range(3):  # the residual is formed anew, so that its drift does not limit the solution
        r = free * (b - A @ x)
        z = dinv * r
        p, rz = z.clone(), torch.dot(r, z)
        stop = 1e-15 * float(b.norm())
        for it in range(20000):
            Ap = free * (A @ p)
            alpha = rz / torch.dot(p, Ap)
            x += alpha * p
            r -= alpha * Ap
            z = dinv * r
            rz, old = torch.dot(r, z), rz
            p = z + rz / old * p
            if it % 25 == 24 and float(r.norm()) <= stop:
                break
    return x + xd


def _exact_adjoint(case, seed):
    dev = _device()
    coords, conn, props, U1, U2 = _inputs(case, seed)
    d = coords.shape[1]
    cn = torch.as_tensor(conn, device=dev, dtype=torch.int64)
    X = torch.as_tensor(coords, device=dev).requires_grad_()
    pr = torch.as_tensor(props, device=dev).requires_grad_()
    U1 = torch.as_tensor(U1, device=dev).reshape(-1, d)
    if case["kind"] == "adjoint_tl":
        lam = torch.as_tensor(_seeds(case, seed, coords, props)[0], device=dev).reshape(-1, d)
        G, s = _geometry(case["elType"], X[cn])
        F = _embed(torch.einsum("eai,eqja->eqij", U1[cn], G) + torch.eye(d, dtype=G.dtype, device=dev))
        mu, K = (pr[:, i, None].expand(s.shape).reshape(-1) for i in (0, 1))
        tau = torch.func.vmap(lambda f, m, k: _neo_hooke(case["material"], f, m, k)[0])(F.reshape(-1, 3, 3), mu, K)
        pk = (tau @ torch.linalg.inv(F.reshape(-1, 3, 3)).mT).reshape(*s.shape, 3, 3)[..., :d, :d]
        L = -torch.einsum("eq,eqij,eqja,eai->", s, pk, G, lam[cn])
        gX, gP = torch.autograd.grad(L, (X, pr))
        return dict(gX=gX, gP=gP)
    shape = (13, len(conn) * _TYPES[case["elType"]][2])
    Pbar, sbar = (torch.as_tensor(v, device=dev) for v in _seeds(case, seed, coords, props, shape))
    before = _exact_pass(case["elType"], "vonmises", coords, conn, props, U1.reshape(-1), None)["state"]
    before.requires_grad_()
    dU = torch.as_tensor(U2, device=dev).requires_grad_()
    G, s = _geometry(case["elType"], X[cn])
    st0 = before.T.reshape(*s.shape, 13)
    de = _strain(torch.einsum("eai,eqja->eqij", dU.reshape(-1, d)[cn], G))
    sig, k, _ = _von_mises(st0[..., :6], st0[..., 12], de, pr[:, None, :])
    new = torch.cat([sig, st0[..., 6:12] + de, k[..., None]], -1)
    bp = _strain(torch.einsum("eai,eqja->eqij", Pbar.reshape(-1, d)[cn], G))
    L = (new * sbar.T.reshape(*s.shape, 13)).sum() - (s[..., None] * sig * bp).sum()
    gU, gS, gP, gX = torch.autograd.grad(L, (dU, before, pr, X))
    out = dict(dUbar=gU, sout=gS, gProps=gP)
    return dict(out, gX=gX) if case["coordinates"] else out


def exact(case, seed):
    if case["kind"] == "batch":
        meshes = _batch_inputs(case, seed)
        out = []
        for elType in ("C3D20TL", "CPE8RTL"):
            parts = [_exact_pass(t, "neohookewa", x, c, p, U, None) for t, x, c, p, U in meshes if t == elType]
            out.append({k: torch.cat([m[k] for m in parts], -1) for k in parts[0]})
        return out
    if case["kind"] == "solve":
        return _exact_solve(case, seed)
    if case["kind"] == "pass":
        return _exact_pass(case["elType"], case["material"], *_inputs(case, seed))
    return _exact_adjoint(case, seed)
