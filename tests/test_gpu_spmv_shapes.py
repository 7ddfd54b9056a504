"""Block products and block-Jacobi updates (BlockMsrMatrix.cs:2970, BlockJacobi.cs:68-266) where the kernel changes: the
block sizes of degree 1 to 4 in two and three dimensions (even ones in pairs of values, odd ones singly, others in the
general kernel), four threads per DOF row up to 49,152 rows and one above, blocks of one or two species in FP32."""
import numpy as np
import pytest
import scipy.sparse as sp

pytestmark = pytest.mark.gpu


def _system(Np, nb, two, seed):
    """Blocks on a ring of random width with some empty off-diagonals; rows of 1 to 6 blocks."""
    rng = np.random.default_rng(seed)
    L = (1 + (rng.random(nb) < 0.4).astype(np.int64) if two else np.ones(nb, np.int64)) * Np
    hops = (1, max(2, nb // 7), max(3, nb // 3))
    i = np.arange(nb)
    pairs = [np.stack([i, (i + d) % nb], 1)[rng.random(nb) < 0.8] for h in hops for d in (h, -h)]
    rc = np.unique(np.concatenate([np.stack([i, i], 1)] + pairs), axis=0)
    r, c = rc[:, 0], rc[:, 1]
    size = L[r] * L[c]
    off = np.concatenate([[0], np.cumsum(size)])
    values = rng.standard_normal(off[-1]) * (0.1 / np.sqrt(Np))
    for k in np.nonzero(r == c)[0]:
        n = L[r[k]]
        values[off[k]:off[k + 1]] += np.eye(n).ravel() * 2.0
    i0 = np.concatenate([[0], np.cumsum(L)])
    # entry e of block k: row e // L[c], column e % L[c]
    k = np.repeat(np.arange(len(r)), size)
    e = np.arange(off[-1]) - off[k]
    A = sp.csr_matrix((values, (i0[r[k]] + e // L[c[k]], i0[c[k]] + e % L[c[k]])), shape=(i0[-1], i0[-1]))
    rp = np.concatenate([[0], np.cumsum(np.bincount(r, minlength=nb))])
    return rp, c.astype(np.int32), values, (L // Np).astype(np.int32) if two else None, A, i0


CASES = [(Np, nb, False) for Np in (1, 3, 4, 6, 10, 15, 20, 35, 7)
         for nb in sorted({1, 2, 49152 // Np, 49152 // Np + 1} if Np != 35 else {1, 7, 8, 1500})]
CASES += [(Np, nb, True) for Np in (1, 4, 10, 20) for nb in (1, 37, 3000)]


@pytest.mark.parametrize("Np,nb,two", CASES)
def test_product(cuda, Np, nb, two):
    import torch
    from bosss_b200.solvers import BlockMsrMatrix
    rp, ci, values, nspc, A, _ = _system(Np, nb, two, 7 * Np + nb)
    M = BlockMsrMatrix.from_bsr(Np, rp, ci, values, nspc)
    rng = np.random.default_rng(3)
    x, y = rng.standard_normal(A.shape[0]), rng.standard_normal(A.shape[0])
    # a row sums at most n products: rounding of n eps |A||x| (FP32: and of the rounded values and vectors)
    n = int(np.diff(A.indptr).max()) + 4
    size = abs(A) @ abs(x) * 1.5 + abs(y)
    for M_, dt, eps in ((M, torch.float64, 2.0 ** -53), (M.ToSingle(), torch.float32, 2.0 ** -24)):
        xd, yd = torch.from_numpy(x).to(cuda, dt), torch.from_numpy(y).to(cuda, dt)
        torch.cuda.synchronize()
        M_.SpMV(1.5, xd, -1.0, yd)
        assert np.all(np.abs(yd.double().cpu().numpy() - (1.5 * (A @ x) - y)) <= n * eps * size)
        M_.SpMV(1.5, xd, 0.0, yd)
        assert np.all(np.abs(yd.double().cpu().numpy() - 1.5 * (A @ x)) <= n * eps * size)


@pytest.mark.parametrize("Np,nb,two", [
    (1, 130, False), (3, 16384, False), (3, 16385, False), (6, 100, False), (15, 60, False), (15, 3277, False),
    (20, 2458, False), (35, 40, False), (1, 1, True), (1, 300, True), (4, 37, True), (10, 1000, True), (20, 500, True),
    (20, 3000, True)])
def test_block_jacobi(cuda, Np, nb, two):
    from bosss_b200.solvers import BlockJacobiConfig, BlockMsrMatrix, MultigridOperator
    rp, ci, values, nspc, A, i0 = _system(Np, nb, two, Np + nb)
    op = MultigridOperator(BlockMsrMatrix.from_bsr(Np, rp, ci, values, nspc), MultigridOperator.Eye)
    D = sp.block_diag([sp.csr_matrix(np.linalg.inv(A[a:b, a:b].toarray())) for a, b in zip(i0, i0[1:])], format="csr")
    rng = np.random.default_rng(9)
    b = rng.standard_normal(A.shape[0])
    x0 = rng.standard_normal(A.shape[0])
    x, ref = x0.copy(), x0.copy()
    BlockJacobiConfig(NoOfIterations=2, omega=0.8).CreateInstance(op).Solve(x, b)
    for _ in range(3):
        ref = ref + 0.8 * (D @ (b - A @ ref))
    # three updates of a diagonally dominant system (factors of condition < 10): sums of some hundred products each
    assert np.abs(x - ref).max() <= 1e-12 * np.abs(ref).max()
