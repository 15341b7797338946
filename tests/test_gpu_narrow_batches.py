"""Batched CG at every way of splitting a row over lanes: one lane, groups of 2 to 32, scalar and vector gathers, short
and long rows, one group a row and many."""
import types

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

WIDTHS = [1, 2, 3, 4, 5, 8, 12, 16, 21, 32, 33, 48, 64]


@pytest.fixture(scope="module", params=[(2, 1, 23), (2, 2, 14), (3, 1, 9), (3, 2, 5)], ids=str)
def system(request, ctx):
    import scipy.sparse as sp
    from afepack_gb300.fem import BoundaryConditionAdmin, Space, assemble
    from afepack_gb300.mesh import cube_mesh, square_mesh
    from afepack_gb300.workloads import ACC
    dim, degree, n = request.param
    mesh = square_mesh(n, 0.2, 1) if dim == 2 else cube_mesh(n, 0.15, 1)
    space = Space.numbered(ctx, mesh, degree)
    _, mark, _ = space.dofs()
    K, M = assemble(space, *ACC[(dim, degree)])
    rng = np.random.default_rng(2)
    B = np.stack([M.vmult(rng.uniform(-1.0, 1.0, space.n_dof)) for _ in range(max(WIDTHS))], axis=1)
    bca = BoundaryConditionAdmin(types.SimpleNamespace(n_dof=mark.shape[0], dof_bmark=mark, dof_point=None))
    bca.add(1, 0.0)
    for c in range(B.shape[1]):
        b = B[:, c].copy()
        bca.apply(K, b)
        B[:, c] = b
    rowptr, cols, vals = K.download()
    return K, sp.csr_matrix((vals, cols, rowptr), shape=(len(rowptr) - 1,) * 2), B


@pytest.mark.parametrize("precision,dense_tail", [(0, 0), (1, 0), (0, 200), (1, 200)])
def test_every_width(system, precision, dense_tail):
    """Residuals by scipy are within the tolerance (CG's own recurrence drifts by rounding only), every width takes as
    many iterations as the widest, up to one, and a second solve gives the same bits."""
    from afepack_gb300.amg import AMGSolver
    K, A, B = system
    amg = AMGSolver(K, precision=precision, dense_tail=dense_tail)
    _, widest = amg.pcg_multi(B, 1e-9, 300)
    for k in WIDTHS:
        Bk = np.ascontiguousarray(B[:, :k])
        X, info = amg.pcg_multi(Bk, 1e-9, 300)
        res = np.linalg.norm(Bk - A @ X, axis=0) / np.linalg.norm(Bk, axis=0)
        assert res.max() <= 1.01e-9, (k, res.max())
        assert max(abs(i["iterations"] - w["iterations"]) for i, w in zip(info, widest)) <= 1
        again, _ = amg.pcg_multi(Bk, 1e-9, 300)
        assert np.array_equal(X, again)
