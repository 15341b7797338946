"""The dense inverse of the coarsest level at the edges of its panels and tiles.

A hierarchy whose stop rule holds on the fine matrix itself is one dense
level, so one V-cycle from zero is x = A^-1 b.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS = np.finfo(np.float64).eps


def _csr(A):
    n = A.shape[0]
    rp, ci, va = [0], [], []
    for i in range(n):
        js = [i] + [j for j in np.nonzero(A[i])[0] if j != i]
        ci += js
        va += list(A[i, js])
        rp.append(len(ci))
    return np.array(rp, np.int32), np.array(ci, np.int32), np.array(va)


def _matrix(n, kind, seed):
    """Symmetric, diagonally dominant by a factor of two in scaled form (condition number of the scaled matrix at
    most 3), rows scaled over four decades; `nonsym` perturbs one triangle, `indef` flips half the signs."""
    rng = np.random.default_rng(seed)
    A = np.zeros((n, n))
    for off in (1, 2, 7, 60, 255, 256):
        if off < n:
            v = rng.uniform(-1.0, 1.0, n - off)
            A[np.arange(n - off), np.arange(off, n)] = v
    A = A + A.T
    if kind == "nonsym":
        A = np.triu(A) + 0.5 * np.tril(A, -1)
    d = 2.0 * np.maximum(np.abs(A).sum(1), np.abs(A).sum(0)) + 1.0
    if kind == "indef":
        d *= np.where(np.arange(n) % 2 == 0, 1.0, -1.0)
    A = A + np.diag(d)
    s = 10.0 ** rng.uniform(-2.0, 2.0, n)
    return A * s[:, None] * s[None, :], s


@pytest.mark.parametrize("n,kind", [(1, "spd"), (15, "spd"), (16, "spd"), (17, "spd"), (128, "spd"), (255, "spd"),
                                    (256, "spd"), (257, "spd"), (385, "spd"), (512, "spd"), (513, "spd"),
                                    (1000, "spd"), (2049, "spd"), (40, "nonsym"), (40, "indef"), (600, "nonsym"),
                                    (600, "indef")])
def test_dense_inverse(ctx, n, kind):
    from afepack_gb300.amg import AMGSolver
    from afepack_gb300.fem import SparseMatrix
    A, s = _matrix(n, kind, n)
    K = SparseMatrix.from_csr(ctx, *_csr(A))
    amg = AMGSolver(K, nmpo=n + 1, nmpsd=0.0)
    assert amg.solve_levels() == 1
    b = np.random.default_rng(n + 1).uniform(-1.0, 1.0, n) * s
    x = np.zeros(n)
    amg.solve(x, b, step=0)
    # in the scaled variables both solves are backward stable for a matrix of condition number <= 3
    want = np.linalg.solve(A, b)
    assert np.linalg.norm((x - want) * s) <= 8 * 3 * (n + 10) * EPS * np.linalg.norm(want * s)
