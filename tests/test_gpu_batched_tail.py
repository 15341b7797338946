"""The dense tail of the batched V-cycle at the edges of its tiles, chunks and column paddings.

A hierarchy whose stop rule holds on the fine matrix itself is one dense level, so the preconditioner is A^-1 and CG
stops after as many steps as the product needs to be accurate: one in FP64; in mixed precision the result of a V-cycle
is rounded to FP32, a factor of about 2^-24 times the condition number (at most 3 here) per step.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _spd(n, seed):
    rng = np.random.default_rng(seed)
    A = np.zeros((n, n))
    for off in (1, 3, 50, 127, 511):
        if off < n:
            A[np.arange(n - off), np.arange(off, n)] = rng.uniform(-1.0, 1.0, n - off)
    A = A + A.T
    return A + np.diag(2.0 * np.abs(A).sum(1) + 1.0)


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("n,ks", [(100, (3,)), (127, (5, 64)), (128, (1, 16, 17)), (129, (33,)), (511, (2, 64)),
                                  (512, (32, 31)), (513, (64, 7)), (1000, (15,)), (1023, (8, 9)), (1024, (8, 9)),
                                  (1153, (64, 48))])
def test_batched_tail(ctx, n, ks, precision):
    import scipy.sparse as sp
    from afepack_gb300.amg import AMGSolver
    from afepack_gb300.fem import SparseMatrix
    A = _spd(n, n)
    S = sp.csr_matrix(A)
    rp, ci, va = [0], [], []
    for i in range(n):
        js = [i] + [j for j in S.indices[S.indptr[i]:S.indptr[i + 1]] if j != i]
        ci += js
        va += list(A[i, js])
        rp.append(len(ci))
    K = SparseMatrix.from_csr(ctx, np.array(rp, np.int32), np.array(ci, np.int32), np.array(va))
    amg = AMGSolver(K, nmpo=n + 1, nmpsd=0.0, precision=precision)
    assert amg.solve_levels() == 1
    for k in ks:
        # columns of very different size, and rows within a column over six decades
        rng = np.random.default_rng(k)
        B = rng.standard_normal((n, k)) * 10.0 ** rng.uniform(-3, 3, (n, 1)) * 10.0 ** rng.uniform(-9, 9, (1, k))
        X, info = amg.pcg_multi(B, 1e-12, 20)
        want = np.linalg.solve(A, B)
        err = np.linalg.norm(X - want, axis=0) / np.linalg.norm(want, axis=0)
        assert err.max() <= 1e-11, (k, err.max())
        assert max(i["iterations"] for i in info) <= (1 if precision == 0 else 3), (k, info)
