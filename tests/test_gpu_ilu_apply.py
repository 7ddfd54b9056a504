"""Application of the natural-order block ILU(0) (CellILU.Solve, CellILU.cs:182-250) in one launch: against the oracle's
ILU(0) with all four block sizes, with fewer and with many more rows than the launch has warps, and on patterns without
upper or without lower blocks, where ILU(0) is the exact factorisation."""
import numpy as np
import pytest
import scipy.sparse as sp
import scipy.sparse.linalg as spla

import oracle as O
from bosss_b200 import assembly as A
from bosss_b200.solvers import BlockMsrMatrix, CellILUConfig, FGMRESConfig, MultigridOperator, PmgConfig

pytestmark = pytest.mark.gpu


def _solve(s, order="natural", reps=1):
    op = MultigridOperator(BlockMsrMatrix.from_system(s), MultigridOperator.Eye)
    slv = CellILUConfig(Order=order).CreateInstance(op)
    for _ in range(reps):
        x = np.random.default_rng(1).standard_normal(s.N)
        slv.Solve(x, s.rhs)
    return x


@pytest.mark.parametrize("D,n,p", [(2, 1, 2), (2, 3, 2), (2, 90, 2), (3, 2, 1), (3, 17, 1), (3, 9, 2), (3, 6, 3)])
def test_ilu_apply(cuda, D, n, p):
    s = A.poisson_2d_c1(seed=2, n=n, p=p) if D == 2 else A.poisson_3d(n, p, seed=4)
    Bo = O.Bsr.of(s)
    ref = O.ilu0_solve(Bo, O.ilu0_factor(Bo, None), s.rhs, None)
    for reps in (1, 3):  # a handle's later applications
        x = _solve(s, reps=reps)
        assert np.abs(x - ref).max() <= 1e-11 * np.abs(ref).max()


@pytest.mark.parametrize("Np", [4, 6, 10, 20])
@pytest.mark.parametrize("upper", [False, True])
def test_ilu_triangular_pattern(cuda, Np, upper):
    rng = np.random.default_rng(Np)
    nb = 700
    rows, cols = [], []
    for i in range(nb):
        for j in sorted({i, *(int(q) for q in rng.integers(0, i + 1, 5))}):
            rows.append(nb - 1 - i if upper else i)
            cols.append(nb - 1 - j if upper else j)
    o = np.lexsort((cols, rows))
    r, c = np.array(rows)[o], np.array(cols)[o]
    v = rng.standard_normal((len(r), Np, Np)) * (0.1 / Np)
    v[r == c] += np.eye(Np)
    rp = np.concatenate([[0], np.cumsum(np.bincount(r, minlength=nb))])

    class S:
        N, row_ptr, col_idx, values, rhs = nb * Np, rp, c.astype(np.int32), v.ravel(), rng.standard_normal(nb * Np)
    S.Np = Np
    ref = spla.spsolve(sp.bsr_matrix((v, c, rp), shape=(S.N, S.N)).tocsc(), S.rhs)
    # exact factorisation: rounding only, amplified by the system's condition (below 10)
    assert np.abs(_solve(S) - ref).max() <= 1e-12 * np.abs(ref).max()


def test_ilu_recorded_fp32(cuda):
    """FP32 application inside the recorded V-cycle: the solve of the recorded and of the host-driven form."""
    s = A.poisson_3d(9, 2, seed=6)
    op = MultigridOperator(BlockMsrMatrix.from_system(s))
    xd = O.direct_solve(s)
    for graph in (False, "vcycle", "solve"):
        pmg = PmgConfig(DegreeHierarchy=(10, 4, 1), UseILU=True, NoOfPostSmootherSweeps=3, CoarseTolerance=1e-1,
                        CoarseMaxIterations=60)
        slv = FGMRESConfig(ConvergenceCriterion=1e-11, termination="relative", Preconditioners=[pmg],
                           MixedPrecision=True, Graph=graph).CreateInstance(op)
        x = np.zeros(s.N)
        slv.Solve(x, s.rhs)
        assert slv.Converged
        assert np.linalg.norm(x - xd) <= 1e-9 * np.linalg.norm(xd)
