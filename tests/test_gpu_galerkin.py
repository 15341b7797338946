"""The Galerkin product against the oracle's getPMPt over the forms its passes choose between: column windows (bitmaps)
and unordered numberings (hash sets), short and long rows of P^T, level by level and bit for bit; the dense-tail
product to rounding."""
import numpy as np
import oracle as O
import pytest

pytestmark = pytest.mark.gpu


def _shuffled_grid(nx, seed):
    """Five-point matrix of an nx x nx grid, rows and columns in a random order."""
    import scipy.sparse as sp
    n = nx * nx
    d = sp.diags([np.ones(n - 1), np.ones(n - nx)], [1, nx]).tolil()
    A = d.tocsr()
    A.setdiag(0)
    A = -(A + A.T)
    p = np.random.default_rng(seed).permutation(n)
    A = A.tocsr()[p][:, p].tocsr()
    A.sort_indices()
    rng = np.random.default_rng(seed + 1)
    vals = A.data * 1.0
    deg = np.asarray(-A.sum(1)).ravel() + rng.uniform(0.0, 0.1, n)
    rp = A.indptr + np.arange(n + 1)
    ci = np.empty(rp[-1], np.int32)
    va = np.empty(rp[-1])
    ci[rp[:-1]], va[rp[:-1]] = np.arange(n), deg
    off = np.ones(rp[-1], bool)
    off[rp[:-1]] = False
    ci[off], va[off] = A.indices, vals
    return rp.astype(np.int32), ci, va


def _random_spd(n, per_row, seed):
    rng = np.random.default_rng(seed)
    A = np.zeros((n, n))
    for i in range(n):
        j = rng.integers(0, n, per_row)
        A[i, j] = -rng.uniform(0.1, 1.0, per_row)
    A = A + A.T
    np.fill_diagonal(A, 0.0)
    np.fill_diagonal(A, -A.sum(1) + 0.1)
    rp, ci, va = [0], [], []
    for i in range(n):
        js = [i] + [j for j in np.nonzero(A[i])[0] if j != i]
        ci += js
        va += list(A[i, js])
        rp.append(len(ci))
    return np.array(rp, np.int32), np.array(ci, np.int32), np.array(va)


CASES = {
    "shuffled_grid_wide": (lambda: _shuffled_grid(540, 3), dict(dense_tail=0)),
    "shuffled_grid": (lambda: _shuffled_grid(70, 5), dict(dense_tail=0)),
    "random": (lambda: _random_spd(500, 5, 7), dict(dense_tail=0)),
    "small": (lambda: _random_spd(70, 2, 9), dict(nmpo=20, dense_tail=0)),
    "random_tail": (lambda: _random_spd(501, 5, 11), dict()),
}


@pytest.mark.parametrize("name", list(CASES))
def test_galerkin_levels(ctx, name):
    from afepack_gb300.amg import AMGSolver
    from afepack_gb300.fem import SparseMatrix
    make, opts = CASES[name]
    rp, ci, va = make()
    n = rp.shape[0] - 1
    amg = AMGSolver(SparseMatrix.from_csr(ctx, rp, ci, va), **opts)
    levels = amg.n_project()
    assert levels >= 1
    A = O.CSR(rp, ci, va, (n, n))
    if name == "shuffled_grid_wide":
        assert amg.level_info(1)[0] > 128 * 1024
    for l in range(min(levels, 2) if name == "shuffled_grid_wide" else levels):
        prp, pci, pva = amg.projection(l)
        n_c = prp.shape[0] - 1
        want = O.rap(O.CSR(prp, pci, pva, (n_c, n)), A)
        rp, ci, va = amg.level_matrix(l + 1)
        if opts.get("dense_tail", 1) == 0:
            assert np.array_equal(rp, want.rowptr) and np.array_equal(ci, want.cols) and np.array_equal(va, want.vals)
        else:  # formed in another order; exact zeros dropped
            D = np.abs(want.to_scipy() - O.CSR(rp, ci, va, (n_c, n_c)).to_scipy()).max()
            assert D <= 1e-13 * np.abs(want.vals).max()
        A, n = O.CSR(rp, ci, va, (n_c, n_c)), n_c
