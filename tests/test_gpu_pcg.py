"""Block-preconditioned CG (SoftPCG.cs:113-194) against a plain FP64 CG on the same block system, step by step, at the
sizes where the persistent kernels change: one block, full and overfull tiles, the widths of the row split, one tile
per CTA and several, block sizes with and without kernels of their own, one and two species."""
import numpy as np
import pytest
import scipy.sparse as sp

pytestmark = pytest.mark.gpu


def _system(Np, nb, two, seed, far=()):
    """Symmetric diagonally dominant block system on a ring with two further neighbours per row and those at `far`."""
    rng = np.random.default_rng(seed)
    nspc = 1 + (rng.random(nb) < 0.3).astype(np.int32) if two else np.ones(nb, np.int32)
    L = nspc.astype(np.int64) * Np
    hop = max(2, int(round(nb ** 0.5)))
    pairs = {(min(i, j), max(i, j)) for i in range(nb) for j in {(i + d) % nb for d in (1, hop, *far)}
             if i != j}
    blocks = {}
    for i, j in pairs:
        v = rng.standard_normal((L[i], L[j])) * (0.1 / np.sqrt(Np))
        blocks[i, j], blocks[j, i] = v, v.T
    for i in range(nb):
        d = rng.standard_normal((L[i], L[i])) * (0.05 / np.sqrt(Np))
        blocks[i, i] = d + d.T + np.diag(1.0 + rng.random(L[i]))
    keys = sorted(blocks)
    rp = np.zeros(nb + 1, np.int64)
    np.add.at(rp, np.array([k[0] for k in keys]) + 1, 1)
    rp = np.cumsum(rp)
    ci = np.array([k[1] for k in keys], np.int32)
    values = np.concatenate([blocks[k].ravel() for k in keys])
    i0 = np.concatenate([[0], np.cumsum(L)])
    rows = np.concatenate([np.repeat(np.arange(i0[i], i0[i + 1]), L[j]) for i, j in keys])
    cols = np.concatenate([np.tile(np.arange(i0[j], i0[j + 1]), L[i]) for i, j in keys])
    A = sp.csr_matrix((values, (rows, cols)), shape=(i0[-1], i0[-1]))
    diag = [np.linalg.inv(blocks[i, i]) for i in range(nb)]
    return rp, ci, values, nspc if two else None, A, sp.block_diag([sp.csr_matrix(d) for d in diag], format="csr")


def _cg(A, D, x, b, steps):
    r = b - A @ x
    z = D @ r
    p = z.copy()
    rz = r @ z
    hist = [np.sqrt(r @ r)]
    for k in range(1, steps + 1):
        q = A @ p
        alpha = rz / (p @ q)
        x = x + alpha * p
        r = r - alpha * q
        z = D @ r
        rz, old = r @ z, rz
        p = z + (rz / old) * p
        if k % 8 == 0 or k == steps:
            hist.append(np.sqrt(r @ r))
    return x, hist


@pytest.mark.parametrize("Np,nb,two,precond", [
    (20, 1, False, False), (1, 127, False, True), (1, 128, False, True), (1, 129, False, True), (1, 60000, False, True),
    (3, 43, False, True), (3, 9000, False, True), (4, 33, False, False), (4, 30000, False, True), (6, 21, False, True),
    (6, 4096, False, True), (10, 13, False, True), (10, 9001, False, True), (15, 9, False, True),
    (15, 6000, False, True), (20, 7, False, True), (20, 4500, False, True), (7, 300, False, True),
    (9, 12000, False, True), (1, 700, True, True), (10, 300, True, True), (4, 30000, True, False)])
def test_cg_steps(cuda, Np, nb, two, precond):
    _check_steps(Np, nb, two, precond)


# the operand gathered once per CTA: rows of 8 blocks at most (7 and 9 here), four or two threads per DOF row
@pytest.mark.parametrize("Np,nb,far", [
    (1, 900, (7,)), (1, 900, (7, 11)), (6, 300, (7,)), (6, 300, (7, 11)), (3, 8000, (7,)), (10, 3000, (7,)),
    (10, 3000, (7, 11)), (15, 2000, (7,)), (20, 1500, (7,)), (20, 200, (7,)), (4, 18000, (7,))])
def test_cg_row_lengths(cuda, Np, nb, far):
    _check_steps(Np, nb, False, True, far)


def _check_steps(Np, nb, two, precond, far=()):
    from bosss_b200.solvers import BlockMsrMatrix, MultigridOperator, SoftPCGConfig
    rp, ci, values, nspc, A, D = _system(Np, nb, two, 100 * Np + nb, far)
    rng = np.random.default_rng(5)
    N = A.shape[0]
    b, x0 = rng.standard_normal(N), rng.standard_normal(N)
    steps = 13
    op = MultigridOperator(BlockMsrMatrix.from_bsr(Np, rp, ci, values, nspc), mode=MultigridOperator.Eye)
    slv = SoftPCGConfig(ConvergenceCriterion=1e-300, termination="relative", MaxSolverIterations=steps - 1,
                        BlockJacobiPrecond=precond).CreateInstance(op)
    for zero in (False, True):
        x = np.zeros(N) if zero else x0.copy()
        ref, hist = _cg(A, D if precond else sp.identity(N, format="csr"), x.copy(), b, steps)
        slv.Solve(x, b)
        assert slv.ThisLevelIterations == steps
        # rounding differs by the order of the sums; the recurrence of 13 steps on a system of condition < 10
        # amplifies it by far less than 1e4
        assert np.linalg.norm(x - ref) <= 1e-11 * np.linalg.norm(ref)
        got = slv.History()
        assert len(got) == len(hist)
        assert np.allclose(got, hist, rtol=1e-8, atol=1e-12 * hist[0])


@pytest.mark.parametrize("Np,n", [(1, 1500), (3, 45000)])
def test_cg_continues_over_launches(cuda, Np, n):
    """More iterations than one launch runs (1,024): the 1-D Laplacian without preconditioner (one block row per cell,
    Np decoupled copies), stopped by its iteration limit; the history has one entry per eight iterations."""
    from bosss_b200.solvers import BlockMsrMatrix, MultigridOperator, SoftPCGConfig
    limit = 2100
    cols = np.stack([np.arange(n) - 1, np.arange(n), np.arange(n) + 1], 1)
    keep = (cols >= 0) & (cols < n)
    rp = np.concatenate([[0], np.cumsum(keep.sum(1))])
    vals = np.tile(np.array([-1.0, 2.0, -1.0]), (n, 1))[keep]
    values = (vals[:, None, None] * np.eye(Np)).ravel()
    op = MultigridOperator(BlockMsrMatrix.from_bsr(Np, rp, cols[keep].astype(np.int32), values),
                           mode=MultigridOperator.Eye)
    slv = SoftPCGConfig(ConvergenceCriterion=1e-300, termination="relative", MaxSolverIterations=limit,
                        BlockJacobiPrecond=False).CreateInstance(op)
    b = np.random.default_rng(2).standard_normal(n * Np)
    x = np.zeros(n * Np)
    slv.Solve(x, b)
    it = slv.ThisLevelIterations
    assert it == limit + 1 or (n == 1500 and it > 1024)
    assert len(slv.History()) == 1 + -(-it // 8)
    T = sp.diags([-1.0, 2.0, -1.0], [-1, 0, 1], shape=(n, n))
    r = b - sp.kron(T, sp.identity(Np)).tocsr() @ x
    # the true residual against the recurrence's last entry: FP64 rounding of n-sized sums, amplified by |x|
    assert abs(np.linalg.norm(r) - slv.History()[-1]) <= 1e-9 * (np.linalg.norm(b) + 4 * np.linalg.norm(x))
