"""Performance cases of the block-sparse DG solver library, through its public entry points.

The cases are the work a program that solves DG systems has the library do: operator products on their own, single
smoother applications, whole Krylov solves with and without the p-multigrid preconditioner, the set-up of a new
system, and a batch of independent systems.  ``listed`` names the cases that are always timed, ``draw`` gives others
of the same ranges.

Two kinds of systems are used.  ``product`` and ``smoother`` cases take a symmetric block system on a Cartesian
grid whose blocks are seeded random numbers (diagonally dominant), handed over as block-CSR arrays; their results
are restated in ``exact`` with plain torch in FP64.  The solves take the SIP operator of a diffusion problem,
assembled by the library, or its two-species sphere problem; the right-hand side is the operator times a seeded
smooth solution, so that solution is the exact result.
"""
import math

import numpy as np
import torch

from bosss_b200 import assembly, xdg
from bosss_b200.solvers import (BlockJacobiConfig, BlockMsrMatrix, CellILUConfig, FGMRESConfig, GpuBatch,
                                MultigridOperator, PmgConfig, SchwarzConfig, SoftPCGConfig)

DEV = "cuda"
# the p-multigrid settings of the benchmark (bench.py SOLVER_PARAMS)
PMG = dict(NoOfPostSmootherSweeps=10, BlockJacobiIterations=1, CoarseSolver="pcg", CoarseTolerance=0.05,
           CoarseMaxIterations=120, SubLevelReduction=0.1, SubLevelMaxIterations=100, RecalcResiPeriod=40)
TOL = 1e-13  # relative residual of the solves: the solution to about ten digits


def listed():
    return [
        # one product of the small 2-D configuration (64 x 64 quads, p = 2): the latency of a single call
        dict(name="product 2d p2 64x64", kind="product", nx=64, ny=64, nz=0, p=2, dtype="f64", form="product",
             radius=0.0),
        # one product of the largest configuration (64^3 hexes, p = 3): 5.8 GB of blocks from memory
        dict(name="product 3d p3 64^3", kind="product", nx=64, ny=64, nz=64, p=3, dtype="f64", form="product",
             radius=0.0),
        # residual b - A x on a ragged 2-D grid of degree 4, the residual evaluation of a non-linear iteration
        dict(name="residual 2d p4 333x251", kind="product", nx=333, ny=251, nz=0, p=4, dtype="f64", form="residual",
             radius=0.0),
        # FP32 product with one- and two-species blocks around a sphere (cut-cell discretisation)
        dict(name="product f32 two species 40^3", kind="product", nx=40, ny=40, nz=40, p=2, dtype="f32",
             form="product", radius=0.3),
        # block-Jacobi relaxation as a stand-alone smoother (five updates)
        dict(name="block jacobi 3d p2 48^3", kind="smoother", nx=48, ny=48, nz=48, p=2, smoother="blockjacobi",
             updates=5),
        # one application of the natural-order block ILU(0)
        dict(name="ilu natural 3d p2 28^3", kind="smoother", nx=28, ny=28, nz=28, p=2, smoother="ilu", updates=1),
        # the 2-D Poisson configuration: block-Jacobi preconditioned CG, 24,576 unknowns
        dict(name="pcg 2d p2 64x64", kind="pcg", nx=64, ny=64, nz=0, p=2, variance=0.0),
        # the benchmark's system and fast settings: FP32 p-multigrid recorded as a graph inside FP64 FlexGMRES
        dict(name="pmg mixed 3d p3 64^3", kind="pmg", nx=64, ny=64, nz=64, p=3, variance=0.0, mixed=True,
             graph="vcycle", smoother="blockjacobi", sweeps=10),
        # the default settings (FP64, driven from the host) with a variable diffusivity
        dict(name="pmg f64 3d p2 24^3", kind="pmg", nx=24, ny=24, nz=24, p=2, variance=1.0, mixed=False,
             graph="off", smoother="blockjacobi", sweeps=10),
        # a two-species sphere problem with the cut-cell settings (FP32 Schwarz smoothing, recorded V-cycle)
        dict(name="xdg mixed p2 24^3", kind="xdg", n=24, p=2, radius=0.28, jump=10.0, smoother="schwarz", sweeps=4),
        # a new operator every call: assembly, change of basis, solver set-up, solve (changing coefficients)
        dict(name="new system 3d p2 32^3", kind="new", nx=32, ny=32, nz=32, p=2, variance=0.5),
        # independent systems solved from one graph launch
        dict(name="batch of 6 16^3 p2", kind="batch", count=6, n=16, p=2, variance=0.5),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _dims(rng, D, cells):
    """Grid extents near ``cells`` cells in total, each its own size (odd and ragged ones among them)."""
    e = [max(3, int(round(cells ** (1.0 / D) * rng.uniform(0.8, 1.25)))) for _ in range(D)]
    return dict(nx=e[0], ny=e[1], nz=e[2] if D == 3 else 0)


def draw(rng):
    kind = rng.choice(["product", "product", "product", "smoother", "smoother", "pcg", "pmg", "pmg", "xdg", "new",
                       "batch"])
    D = rng.choice([2, 3])
    if kind == "product":
        p = rng.choice([1, 2, 3, 4])
        Np = _np(D, p)
        two = rng.random() < 0.3
        values = _log(rng, 1e5, 3e8)  # block entries: 0.8 MB to 2.4 GB of FP64
        c = _dims(rng, D, max(16.0, values / ((2 * D + 1) * Np * Np)))
        return dict(kind=kind, **c, p=p, dtype=rng.choice(["f64", "f64", "f32"]),
                    form=rng.choice(["product", "residual"]), radius=rng.uniform(0.2, 0.4) if two else 0.0)
    if kind == "smoother":
        sm = rng.choice(["blockjacobi", "schwarz", "ilu"])
        p = rng.choice([1, 2, 3] if D == 3 else [2, 3]) if sm != "ilu" else rng.choice([1, 2, 3]) if D == 3 else 2
        c = _dims(rng, D, _log(rng, 100, 8e4) if sm != "schwarz" else _log(rng, 100, 2e4))
        return dict(kind=kind, **c, p=p, smoother=sm, updates=1 if sm == "ilu" else rng.randint(1, 8))
    if kind == "pcg":
        return dict(kind=kind, **_dims(rng, D, _log(rng, 100, 3e4)), p=rng.choice([1, 2, 3]),
                    variance=rng.choice([0.0, 0.5]))
    if kind == "pmg":
        mixed = rng.random() < 0.6
        return dict(kind=kind, **_dims(rng, 3, _log(rng, 400, 3.2e4)), p=rng.choice([2, 3]),
                    variance=rng.choice([0.0, 0.5]), mixed=mixed,
                    graph=rng.choice(["vcycle", "solve"]) if mixed else "off",
                    smoother="blockjacobi", sweeps=10)
    if kind == "xdg":
        return dict(kind=kind, n=rng.randint(10, 24), p=2, radius=rng.uniform(0.2, 0.35), jump=10.0,
                    smoother=rng.choice(["schwarz", "blockjacobi"]), sweeps=rng.choice([4, 6]))
    if kind == "new":
        return dict(kind=kind, **_dims(rng, 3, _log(rng, 400, 3.2e4)), p=2, variance=0.5)
    return dict(kind="batch", count=rng.randint(2, 8), n=rng.randint(8, 18), p=2, variance=0.5)


# ---- grids and seeded data -------------------------------------------------------------------------------------


def _np(D, p):
    return math.comb(D + p, D)


def _shape(case):
    return [case["nx"], case["ny"]] + ([case["nz"]] if case["nz"] else [])


def _generator(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    return g


def _randn(g, *shape):
    return torch.randn(*shape, generator=g, dtype=torch.float64, device=DEV)


def _stencil(shape):
    """Block columns per cell in ascending order (-z, -y, -x, self, +x, +y, +z), -1 where outside; x fastest."""
    nc = math.prod(shape)
    ids = torch.arange(nc, device=DEV)
    cols, stride, strides, idx = [], 1, [], []
    for n in shape:
        idx.append((ids // stride) % n)
        strides.append(stride)
        stride *= n
    for d in reversed(range(len(shape))):
        cols.append(torch.where(idx[d] > 0, ids - strides[d], -1))
    cols.append(ids)
    for d in range(len(shape)):
        cols.append(torch.where(idx[d] < shape[d] - 1, ids + strides[d], -1))
    return torch.stack(cols, 1), strides


def _csr(cols):
    keep = cols >= 0
    rp = torch.zeros(cols.shape[0] + 1, dtype=torch.int64, device=DEV)
    rp[1:] = torch.cumsum(keep.sum(1), 0)
    return rp, cols[keep].to(torch.int32), keep


def _centres(shape):
    nc = math.prod(shape)
    ids = torch.arange(nc, device=DEV)
    out, stride = [], 1
    for n in shape:
        out.append((((ids // stride) % n).double() + 0.5) / n)
        stride *= n
    return torch.stack(out, 1)


def _degrees(D, p):
    """Total degree of each mode, in the order of total degree."""
    return [q for q in range(p + 1) for _ in range(_np(D, q) - (_np(D, q - 1) if q else 0))]


def _smooth(shape, p, seed, repeat=None):
    """Coefficients of a smooth DG function: waves over the cells, decaying with the degree of the mode."""
    g = _generator(seed)
    D = len(shape)
    deg = torch.tensor(_degrees(D, p), dtype=torch.float64, device=DEV)
    k = torch.randint(1, 5, (6, D), generator=g, device=DEV).double()
    amp, phase = _randn(g, 6, len(deg)), 2 * math.pi * torch.rand(6, len(deg), generator=g, dtype=torch.float64,
                                                                  device=DEV)
    arg = math.pi * (_centres(shape) @ k.T)
    u = torch.zeros(math.prod(shape), len(deg), dtype=torch.float64, device=DEV)
    for m in range(6):
        u += amp[m] * torch.sin(arg[:, m, None] + phase[m])
    u *= 0.2 ** deg
    return u if repeat is None else u.repeat_interleave(repeat, 0)


def _diffusivity(shape, variance, seed):
    if variance == 0.0:
        return None
    n = max(shape)
    f = assembly.gaussian_random_field(shape, 1.0 / n, length=0.15, variance=variance, seed=int(seed))
    return torch.from_numpy(np.exp(np.ascontiguousarray(f).reshape(-1))).to(DEV)


# ---- random block systems --------------------------------------------------------------------------------------


def _blocks(case, seed):
    """(Np, row_ptr, col_idx, values [blocks, Np, Np]) of the seeded symmetric block system of a grid."""
    shape = _shape(case)
    D, Np, nc = len(shape), _np(len(shape), case["p"]), math.prod(shape)
    g = _generator(seed)
    cols, strides = _stencil(shape)
    rp, ci, keep = _csr(cols)
    pos = torch.cumsum(keep.reshape(-1), 0).reshape(keep.shape) - 1
    v = torch.empty(int(rp[-1]), Np, Np, dtype=torch.float64, device=DEV)
    d0 = _randn(g, nc, Np, Np) * (0.05 / math.sqrt(Np))
    v[pos[:, D]] = d0 + d0.transpose(1, 2) + torch.eye(Np, dtype=torch.float64, device=DEV)
    for d in range(D):
        up = keep[:, D + 1 + d]
        f = _randn(g, int(up.sum()), Np, Np) * (0.2 / (D * math.sqrt(Np)))
        v[pos[up, D + 1 + d]] = f
        down = keep[:, D - 1 - d]  # the same faces from their upper cells, in the same order
        v[pos[down, D - 1 - d]] = f.transpose(1, 2)
    return Np, rp, ci, v


def _species(case):
    """Species per cell: two where the sphere cuts the cell."""
    shape = _shape(case)
    if not case["radius"]:
        return None
    r = torch.linalg.norm(_centres(shape) - 0.5, dim=1)
    return 1 + ((r - case["radius"]).abs() < 0.6 / max(shape)).to(torch.int32)


def _species_blocks(case, seed):
    """(Np, row_ptr, col_idx, flat values, nspc) of a seeded system with blocks of one or two species."""
    shape = _shape(case)
    Np = _np(len(shape), case["p"])
    nspc = _species(case)
    rp, ci, keep = _csr(_stencil(shape)[0])
    rows = torch.repeat_interleave(torch.arange(len(nspc), device=DEV), torch.diff(rp))
    size = nspc[rows].long() * nspc[ci.long()].long() * Np * Np
    v = _randn(_generator(seed), int(size.sum())) / math.sqrt(Np)
    return Np, rp, ci, v, nspc, rows, size


def _vector(n, seed):
    return _randn(_generator(seed * 2 + 1), n)


# ---- the interface ---------------------------------------------------------------------------------------------


def _pmg(case, op):
    shape_p = case["p"]
    levels = (20, 10, 4) if shape_p == 3 else (10, 4, 1)
    pmg = dict(PMG, NoOfPostSmootherSweeps=case["sweeps"], Smoother=case["smoother"])
    return FGMRESConfig(ConvergenceCriterion=TOL, termination="relative", MaxKrylovDim=30,
                        Preconditioners=[PmgConfig(DegreeHierarchy=levels, **pmg)],
                        MixedPrecision=case["mixed"], Graph=case["graph"]).CreateInstance(op)


def _system(shape, p, coeff):
    return BlockMsrMatrix.AssembleSIP(shape, p, penalty=(p + 1) * (p + 2), coeff=coeff)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "product":
        if case["radius"]:
            Np, rp, ci, v, nspc = _species_blocks(case, seed)[:5]
            M = BlockMsrMatrix.from_bsr(Np, rp, ci, v, nspc)
        else:
            Np, rp, ci, v = _blocks(case, seed)
            M = BlockMsrMatrix.from_bsr(Np, rp, ci, v.reshape(-1))
        del v
        x, b = _vector(M.N, seed), _vector(M.N, seed + 1)
        if case["dtype"] == "f32":
            M, x, b = M.ToSingle(), x.float(), b.float()
        torch.cuda.synchronize()
        return dict(case=case, M=M, x=x, b=b, y=torch.empty_like(x))
    if kind == "smoother":
        Np, rp, ci, v = _blocks(case, seed)
        op = MultigridOperator(BlockMsrMatrix.from_bsr(Np, rp, ci, v.reshape(-1)))
        if case["smoother"] == "blockjacobi":
            cfg = BlockJacobiConfig(NoOfIterations=case["updates"] - 1)
        elif case["smoother"] == "schwarz":
            cfg = SchwarzConfig(FixedNoOfIterations=case["updates"], Blocking="cell")
        else:
            cfg = CellILUConfig()
        B = _vector(op.BaseMatrix.N, seed)
        return dict(case=case, op=op, slv=cfg.CreateInstance(op), B=B, X=torch.zeros_like(B))
    if kind in ("pcg", "pmg", "xdg"):
        if kind == "xdg":
            s = _sphere(case)
            M = BlockMsrMatrix.from_system(s)
            u = _solution(case, seed, s.nspc)
        else:
            shape = _shape(case)
            M = _system(shape, case["p"], _diffusivity(shape, case["variance"], seed))
            u = _solution(case, seed)
        B = torch.zeros_like(u)
        M.SpMV(1.0, u, 0.0, B)
        op = MultigridOperator(M)
        if kind == "pcg":
            slv = SoftPCGConfig(ConvergenceCriterion=TOL, termination="relative",
                                MaxSolverIterations=20000).CreateInstance(op)
        else:
            slv = _pmg(case if kind == "pmg" else dict(case, mixed=True, graph="vcycle"), op)
        return dict(case=case, op=op, slv=slv, B=B, X=torch.zeros_like(B))
    if kind == "new":
        shape = _shape(case)
        coeff = _diffusivity(shape, case["variance"], seed)
        M = _system(shape, case["p"], coeff)
        u = _solution(case, seed)
        B = torch.zeros_like(u)
        M.SpMV(1.0, u, 0.0, B)
        torch.cuda.synchronize()
        M.Dispose()
        return dict(case=case, shape=shape, coeff=coeff, B=B, X=torch.zeros_like(B))
    ops, slvs, Bs = [], [], []
    for i in range(case["count"]):
        shape = [case["n"]] * 3
        M = _system(shape, case["p"], _diffusivity(shape, case["variance"], seed * 16 + i))
        u = _smooth(shape, case["p"], seed * 16 + i).reshape(-1)
        B = torch.zeros_like(u)
        M.SpMV(1.0, u, 0.0, B)
        ops.append(MultigridOperator(M))
        slvs.append(_pmg(dict(case, mixed=True, graph="solve", smoother="blockjacobi", sweeps=10), ops[-1]))
        Bs.append(B)
    return dict(case=case, ops=ops, batch=GpuBatch(slvs), Bs=Bs, Xs=[torch.zeros_like(B) for B in Bs])


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "product":
        M, y = state["M"], state["y"]
        if case["form"] == "residual":
            y.copy_(state["b"])
            return M.SpMV(-1.0, state["x"], 1.0, y)
        return M.SpMV(1.0, state["x"], 0.0, y)
    if kind == "batch":
        for X in state["Xs"]:
            X.zero_()
        torch.cuda.current_stream().synchronize()  # the solver works on its own stream
        return state["batch"].Solve(state["Xs"], state["Bs"])
    X = state["X"]
    X.zero_()
    torch.cuda.current_stream().synchronize()  # the solver works on its own stream
    if kind != "new":
        return state["slv"].Solve(X, state["B"])
    M = _system(state["shape"], case["p"], state["coeff"])
    op = MultigridOperator(M)
    slv = _pmg(dict(case, mixed=True, graph="vcycle", smoother="blockjacobi", sweeps=10), op)
    slv.Solve(X, state["B"])
    slv.Dispose()
    op.Dispose()
    M.Dispose()
    return X


def _unknowns(case):
    """(block rows, blocks, block entries, unknowns) of one system of a case."""
    if case["kind"] in ("xdg", "batch"):
        shape, p = [case["n"]] * 3, case["p"]
    else:
        shape, p = _shape(case), case["p"]
    D, Np, nc = len(shape), _np(len(shape), p), math.prod(shape)
    nnzb = nc + 2 * sum(nc // n * (n - 1) for n in shape)
    cut = 1.0
    if case["kind"] == "xdg":  # cells cut by the sphere carry a second species
        cut += 1.5 * 4 * math.pi * case["radius"] ** 2 * case["n"] ** 2 / nc
    elif case.get("radius"):
        cut += float((_species(case) == 2).double().mean())
    return nc, nnzb, nnzb * Np * Np * cut, nc * Np * cut


def work(case):
    nc, nnzb, entries, n = _unknowns(case)
    size = 4 if case.get("dtype") == "f32" else 8
    structure = 4 * nnzb + 8 * (nc + 1)
    matrix = size * entries + structure
    kind = case["kind"]
    if kind == "product":
        vectors = 3 if case["form"] == "residual" else 2
        return {"bytes": matrix + vectors * size * n, "flops": 2 * entries}
    if kind == "smoother":  # every update needs one product with the operator and the block inverses
        return {"bytes": matrix + 2 * size * n, "flops": 2 * entries * case["updates"]}
    if kind == "new":  # the coefficients and the right-hand side in, the solution out
        return {"bytes": 8 * nc + 16 * n, "flops": 2 * entries}
    count = case.get("count", 1)
    return {"bytes": count * (matrix + 2 * size * n), "flops": count * 2 * entries}


def _sphere(case):
    return xdg.xdg_sphere(n=case["n"], p=case["p"], mu=(1.0, case["jump"]), radius=case["radius"],
                          centre=(0.5, 0.5, 0.5), rhs_f=lambda X: X[0])


def _solution(case, seed, nspc=None):
    """The seeded solution of a solve's system (nspc: species per cell of a sphere problem)."""
    if case["kind"] != "xdg":
        return _smooth(_shape(case), case["p"], seed).reshape(-1)
    nspc = _sphere(case).nspc if nspc is None else nspc
    return _smooth([case["n"]] * 3, case["p"], seed, torch.from_numpy(nspc.astype(np.int64)).to(DEV)).reshape(-1)


# ---- FP64 restatements -----------------------------------------------------------------------------------------


def _rows(rp):
    return torch.repeat_interleave(torch.arange(len(rp) - 1, device=DEV), torch.diff(rp))


def _product(rp, ci, v, x, rows=None):
    """A x for uniform blocks v [blocks, Np, Np], x [cells, Np]."""
    rows = _rows(rp) if rows is None else rows
    y = torch.zeros_like(x)
    for k in range(0, len(ci), 1 << 18):
        y.index_add_(0, rows[k:k + (1 << 18)], torch.bmm(v[k:k + (1 << 18)],
                                                         x[ci[k:k + (1 << 18)].long()].unsqueeze(2)).squeeze(2))
    return y


def _exact_product(case, seed):
    if not case["radius"]:
        Np, rp, ci, v = _blocks(case, seed)
        n = (len(rp) - 1) * Np
    else:
        Np, rp, ci, v, nspc, rows, size = _species_blocks(case, seed)
        n = int(nspc.sum()) * Np
    x, b = _vector(n, seed), _vector(n, seed + 1)
    if case["dtype"] == "f32":
        x, b, v = x.float().double(), b.float().double(), v.float().double()
    if not case["radius"]:
        y = _product(rp, ci, v, x.reshape(-1, Np)).reshape(-1)
    else:
        L = nspc.long() * Np
        start, off = torch.cumsum(L, 0) - L, torch.cumsum(size, 0) - size
        y = torch.zeros_like(x)
        for a in (1, 2):
            for c in (1, 2):
                I, J = a * Np, c * Np
                k = ((nspc[rows] == a) & (nspc[ci.long()] == c)).nonzero().squeeze(1)
                for q in k.split(1 << 16):
                    B = v[off[q, None] + torch.arange(I * J, device=DEV)].reshape(-1, I, J)
                    xs = x[start[ci[q].long(), None] + torch.arange(J, device=DEV)]
                    t = start[rows[q], None] + torch.arange(I, device=DEV)
                    y.index_add_(0, t.reshape(-1), torch.bmm(B, xs.unsqueeze(2)).reshape(-1))
    return b - y if case["form"] == "residual" else y


def _diagonal(rp, ci, rows):
    return (ci.long() == rows).nonzero().squeeze(1)


def _exact_jacobi(case, rp, ci, v, b):
    rows = _rows(rp)
    D = v[_diagonal(rp, ci, rows)]
    x = torch.zeros_like(b)
    for _ in range(case["updates"]):
        x = x + torch.linalg.solve(D, (b - _product(rp, ci, v, x, rows)).unsqueeze(2)).squeeze(2)
    return x


def _exact_schwarz(case, rp, ci, v, b):
    """Restricted additive Schwarz with one patch per cell: the cell and its neighbours."""
    cols = _stencil(_shape(case))[0]
    nc, S = cols.shape
    Np = v.shape[1]
    pos = torch.cumsum((cols >= 0).reshape(-1), 0).reshape(cols.shape) - 1
    own = S // 2
    W = torch.zeros(nc, S * Np, Np, dtype=torch.float64, device=DEV)  # columns of the centre rows of the inverses
    for c0 in range(0, nc, 2048):
        cell = cols[c0:c0 + 2048]
        n = len(cell)
        P = torch.zeros(n, S, Np, S, Np, dtype=torch.float64, device=DEV)
        for a in range(S):
            there = (cell[:, a] >= 0).nonzero().squeeze(1)
            gone = (cell[:, a] < 0).nonzero().squeeze(1)
            P[gone, a, :, a, :] = torch.eye(Np, dtype=torch.float64, device=DEV)
            nbr = cols[cell[there, a]]
            for t in range(S):  # block (neighbour a, its neighbour t) where that lies in the patch
                for c in range(S):
                    hit = ((nbr[:, t] >= 0) & (nbr[:, t] == cell[there, c])).nonzero().squeeze(1)
                    if len(hit):
                        P[there[hit], a, :, c, :] = v[pos[cell[there[hit], a], t]]
        P = P.reshape(n, S * Np, S * Np)
        E = torch.zeros(n, S * Np, Np, dtype=torch.float64, device=DEV)
        E[:, own * Np:(own + 1) * Np] = torch.eye(Np, dtype=torch.float64, device=DEV)
        W[c0:c0 + 2048] = torch.linalg.solve(P.transpose(1, 2), E)
    x, rows = torch.zeros_like(b), _rows(rp)
    for _ in range(case["updates"]):
        r = b - _product(rp, ci, v, x, rows)
        g = torch.where((cols >= 0)[:, :, None], r[cols.clamp(min=0)], torch.zeros_like(r[:1, None]))
        x = x + torch.bmm(W.transpose(1, 2), g.reshape(nc, S * Np, 1)).squeeze(2)
    return x


def _exact_ilu(case, rp, ci, v, b):
    """Block ILU(0) in the cell order.  Two neighbours of a cell of a Cartesian grid are never neighbours of each
    other, so only the diagonal blocks change: L_ik = A_ik U_kk^-1, U_ii = A_ii - sum_k<i L_ik A_ki."""
    shape = _shape(case)
    D, Np = len(shape), v.shape[1]
    cols, _ = _stencil(shape)
    pos = torch.cumsum((cols >= 0).reshape(-1), 0).reshape(cols.shape) - 1
    level, stride = torch.zeros(len(cols), dtype=torch.int64, device=DEV), 1
    for n in shape:
        level += (torch.arange(len(cols), device=DEV) // stride) % n
        stride *= n
    order = [(level == l).nonzero().squeeze(1) for l in range(int(level.max()) + 1)]
    Uinv = torch.empty(len(cols), Np, Np, dtype=torch.float64, device=DEV)
    y, x = b.clone(), torch.zeros_like(b)
    for i in order:
        U = v[pos[i, D]].clone()
        for s in range(D):  # lower neighbours, ascending
            has = (cols[i, s] >= 0).nonzero().squeeze(1)
            k = cols[i[has], s]
            L = v[pos[i[has], s]] @ Uinv[k]
            U[has] -= L @ v[pos[k, 2 * D - s]]
            y[i[has]] -= torch.bmm(L, y[k].unsqueeze(2)).squeeze(2)
        Uinv[i] = torch.linalg.inv(U)
    for i in reversed(order):
        r = y[i].clone()
        for s in range(D + 1, 2 * D + 1):
            has = (cols[i, s] >= 0).nonzero().squeeze(1)
            r[has] -= torch.bmm(v[pos[i[has], s]], x[cols[i[has], s]].unsqueeze(2)).squeeze(2)
        x[i] = torch.bmm(Uinv[i], r.unsqueeze(2)).squeeze(2)
    return x


def exact(case, seed):
    kind = case["kind"]
    if kind == "product":
        return _exact_product(case, seed)
    if kind == "smoother":
        Np, rp, ci, v = _blocks(case, seed)
        b = _vector((len(rp) - 1) * Np, seed).reshape(-1, Np)
        f = {"blockjacobi": _exact_jacobi, "schwarz": _exact_schwarz, "ilu": _exact_ilu}[case["smoother"]]
        return f(case, rp, ci, v, b).reshape(-1)
    if kind == "batch":
        return [_smooth([case["n"]] * 3, case["p"], seed * 16 + i).reshape(-1) for i in range(case["count"])]
    return _solution(case, seed)
