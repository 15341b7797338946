"""C/F flags and P of the GPU's waves against the host routine's sequential sweeps: short and long rows (a thread or a
warp per row of weights), rows with more strong C neighbours than a warp's set holds, P^T rows longer than the
shared-memory list, a pattern that is not symmetric, one-row and zero-row-coupling matrices."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _rows(n, pick, seed, symmetric=True):
    """[diag, ascending others] rows of an M-matrix whose off-diagonal pattern is pick(i) for row i."""
    rng = np.random.default_rng(seed)
    A = np.zeros((n, n))
    for i in range(n):
        j = np.unique(pick(i, rng))
        A[i, j] = -rng.uniform(0.1, 1.0, j.size)
    if symmetric:
        A = np.minimum(A, A.T)
    np.fill_diagonal(A, 0.0)
    np.fill_diagonal(A, np.abs(A).sum(1) + 0.5)
    rp, ci, va = [0], [], []
    for i in range(n):
        js = [i] + [j for j in np.nonzero(A[i])[0] if j != i]
        ci += js
        va += list(A[i, js])
        rp.append(len(ci))
    return np.array(rp, np.int32), np.array(ci, np.int32), np.array(va)


def _band(w):
    return lambda n: lambda i, rng: np.clip(i + rng.integers(-w, w + 1, 2 * w), 0, n - 1)


def _star(hubs):
    """Every row coupled to all of the last `hubs` rows and two neighbours: P^T rows and hub rows are long."""
    return lambda n: lambda i, rng: np.concatenate([[(i + 1) % n, (i + 7) % n], np.arange(n - hubs, n)])


CASES = {
    "path": (300, _band(1), True), "band8": (1000, _band(8), True), "band30": (900, _band(30), True),
    "random": (700, lambda n: lambda i, rng: rng.integers(0, n, 12), True),
    "dense": (1100, lambda n: lambda i, rng: rng.integers(0, n, 700), True),
    "star": (800, _star(5), True), "one": (1, lambda n: lambda i, rng: np.array([0]), True),
    "diagonal": (65, lambda n: lambda i, rng: np.array([i]), True),
    "nonsymmetric": (600, lambda n: lambda i, rng: rng.integers(0, n, 9), False),
}


@pytest.mark.parametrize("alpha", [0.25, 0.02])
@pytest.mark.parametrize("name", list(CASES))
def test_cf_matches_host(ctx, name, alpha):
    from afepack_gb300.amg import AMGSolver, host_coarsen
    from afepack_gb300.fem import SparseMatrix
    n, pick, symmetric = CASES[name]
    rp, ci, va = _rows(n, pick(n), 5, symmetric)
    cf, prp, pci, pva = host_coarsen(rp, ci, va, alpha)
    nc = prp.shape[0] - 1
    if nc == n:  # nothing to coarsen: the hierarchy keeps no projection
        assert (cf == -1).all()
        return
    # one projection: the stop rule holds on the coarse matrix
    amg = AMGSolver(SparseMatrix.from_csr(ctx, rp, ci, va), nmpo=n - 1, nmpsd=0.0, alp=alpha, dense_tail=0)
    assert amg.n_project() == 1
    grp, gci, gva = amg.projection(0)
    assert np.array_equal(grp, prp) and np.array_equal(gci, pci) and np.array_equal(gva, pva)
