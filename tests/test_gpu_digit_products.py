"""The tensor-core digit products, entry by entry, on matrices whose entries and inverses span many decades.

The matrices are 7-point operators with a random coefficient a cell, of a given contrast: M-matrices, whose inverse
has positive entries only.  A hierarchy whose stop rule holds on the fine matrix itself is one dense level, so a V-cycle
from zero is x = T b with T the inverse as the library holds it (for a unit vector b: a column of T, exactly in FP64),
and one step of batched CG from zero gives alpha_c T B per column.
"""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS = np.finfo(np.float64).eps
M = 9
N_ROWS = M ** 3  # 729: three panels of the inverse, two chunks of the batched product


def cells(contrast, seed, m=M):
    """Dense 7-point matrix of m^3 unknowns with a coefficient 10^U(0, log10 contrast) in every cell."""
    rng = np.random.default_rng(seed)
    k = 10.0 ** rng.uniform(0.0, np.log10(contrast), (m + 2,) * 3)
    idx = np.arange(m ** 3).reshape(m, m, m)
    A = np.zeros((m ** 3, m ** 3))
    diag = np.zeros((m, m, m))
    inner = (slice(1, -1),) * 3
    for axis in range(3):
        for step in (-1, 1):
            near = np.roll(k, -step, axis)[inner]
            w = 2.0 * k[inner] * near / (k[inner] + near)
            diag += w
            here = [slice(None)] * 3
            there = [slice(None)] * 3
            here[axis] = slice(1, None) if step < 0 else slice(None, -1)
            there[axis] = slice(None, -1) if step < 0 else slice(1, None)
            A[idx[tuple(here)].ravel(), idx[tuple(there)].ravel()] = -w[tuple(here)].ravel()
    A[np.arange(m ** 3), np.arange(m ** 3)] = diag.ravel()
    return (A + A.T) / 2


def hierarchy(ctx, A, precision=0):
    from afepack_gb300.amg import AMGSolver
    from afepack_gb300.fem import SparseMatrix
    n = len(A)
    rp, ci, va = [0], [], []
    for i in range(n):
        js = [i] + [j for j in np.nonzero(A[i])[0] if j != i]
        ci += js
        va += list(A[i, js])
        rp.append(len(ci))
    K = SparseMatrix.from_csr(ctx, np.array(rp, np.int32), np.array(ci, np.int32), np.array(va))
    amg = AMGSolver(K, nmpo=n + 1, nmpsd=0.0, precision=precision)
    assert amg.solve_levels() == 1
    return amg


def held_inverse(amg, n, columns=None):
    """Columns of the FP64 inverse that the hierarchy holds."""
    columns = range(n) if columns is None else columns
    out = []
    for j in columns:
        b, x = np.zeros(n), np.zeros(n)
        b[j] = 1.0
        amg.solve(x, b, step=0)
        out.append(x)
    return np.stack(out, axis=1)


def one_step(native, amg, B):
    """alpha_c T B_c: the iterate after one CG step from zero (whether it converged or not)."""
    from afepack_gb300 import _native as N
    X = np.zeros_like(B)
    infos = (N.SolveInfo * B.shape[1])()
    st = native.afp_pcg_solve_multi(amg.handle, N.ptr(X), N.ptr(B), B.shape[1], 1e-300, 1, infos)
    assert st in (0, 5), native.afp_last_error()  # converged, or out of steps
    return X


def long_product(T, B):
    return T.astype(np.longdouble) @ B.astype(np.longdouble)


def right_hand_sides(A, k, seed):
    """Half of the columns A x (graded as the matrix is), half of one size."""
    rng = np.random.default_rng(seed)
    B = rng.standard_normal((len(A), k))
    B[:, ::2] = A @ B[:, ::2]
    return B


@pytest.mark.parametrize("contrast", [1e4, 1e8])
@pytest.mark.parametrize("k", [5, 16, 24, 64])
def test_fp64_tail_is_as_good_as_fp64_sums(native, ctx, k, contrast):
    """The batched product against the held inverse times B, per entry, within the classical bound of FP64 sums of
    n terms, n eps sum |T||B|."""
    A = cells(contrast, 11)
    amg = hierarchy(ctx, A)
    T = held_inverse(amg, N_ROWS)
    B = right_hand_sides(A, k, 12)
    X = one_step(native, amg, B)
    want = long_product(T, B)
    size = np.abs(T) @ np.abs(B)
    for c in range(k):
        alpha = np.median(X[:, c] / want[:, c])  # the step length, 1 to rounding
        assert abs(alpha - 1) < 1e-9
        err = np.abs(X[:, c] / alpha - want[:, c])
        assert (err <= N_ROWS * EPS * size[:, c]).all(), (c, float((err / size[:, c]).max()))


def pair(T):
    """T as the mixed-precision hierarchy holds it."""
    hi = T.astype(np.float32)
    lo = (T - hi).astype(np.float32)
    return hi.astype(np.float64) + lo.astype(np.float64)


def assert_mixed_product(X, T, B, k):
    """Z is rounded to FP32 and so is, in effect, the step length taken from it (two roundings, 2^-22.5 with the
    division); the sums themselves are good to 2^-40 of sum |T||R|: 729 terms of a double-float sum, whose low part
    rounds at 2^-48 of the sum each."""
    R = B.astype(np.float32).astype(np.float64)
    want = long_product(T, R)
    size = np.abs(T) @ np.abs(R)
    for c in range(k):
        alpha = np.median(X[:, c] / want[:, c])
        err = np.abs(X[:, c] / alpha - want[:, c])
        bound = 2.0 ** -22.5 * np.abs(want[:, c]) + 2.0 ** -40 * size[:, c]
        assert (err <= bound).all(), (c, float((err / bound).max()))


@pytest.mark.parametrize("contrast", [1e4, 1e8])
@pytest.mark.parametrize("k", [5, 9, 33, 64])
def test_mixed_tail_is_as_good_as_double_float_sums(native, ctx, k, contrast):
    A = cells(contrast, 11)
    T = pair(held_inverse(hierarchy(ctx, A), N_ROWS))
    B = right_hand_sides(A, k, 13)
    assert_mixed_product(one_step(native, hierarchy(ctx, A, 1), B), T, B, k)


@pytest.mark.parametrize("kind", ["nonsymmetric", "indefinite"])
@pytest.mark.parametrize("k", [16, 40])
def test_mixed_tail_of_other_matrices(native, ctx, k, kind):
    """Tails that are not symmetric positive definite, whose diagonal says nothing about their entries."""
    A = cells(1e4, 14)
    if kind == "nonsymmetric":
        A = np.triu(A) + 0.5 * np.tril(A, -1)
    else:
        A[np.arange(0, N_ROWS, 2), np.arange(0, N_ROWS, 2)] *= -1
    T = pair(held_inverse(hierarchy(ctx, A), N_ROWS))
    B = right_hand_sides(A, k, 15)
    assert_mixed_product(one_step(native, hierarchy(ctx, A, 1), B), T, B, k)


def refined_columns(A, columns):
    """Columns of the inverse to beyond FP64: iterative refinement with residuals in long double."""
    inv = np.linalg.inv(A)
    rows, cols = np.nonzero(A)
    vals = A[rows, cols].astype(np.longdouble)[:, None]
    X = inv[:, columns].astype(np.longdouble)
    for _ in range(4):
        R = np.zeros(X.shape, np.longdouble)
        R[columns, range(len(columns))] = 1
        np.subtract.at(R, rows, vals * X[cols])
        X = X + (inv @ R.astype(np.float64)).astype(np.longdouble)
    return X


def worst_of_median_row(T, want):
    return float(np.median((np.abs(T - want) / np.abs(want)).max(axis=1)))


@pytest.mark.parametrize("contrast", [1e2, 1e4])
def test_inverse_entry_by_entry(ctx, contrast):
    """The inverse of an M-matrix by elimination has small relative errors in every entry; entries span six decades a
    row at contrast 1e4.  The worst entry of the median row is within n eps, a rounding per pivot."""
    A = cells(contrast, 11)
    amg = hierarchy(ctx, A)
    cols = list(range(0, N_ROWS, 4))
    T = held_inverse(amg, N_ROWS, cols)
    assert worst_of_median_row(T, refined_columns(A, cols)) <= N_ROWS * EPS


def test_inverse_of_a_graded_matrix(ctx):
    """At contrast 1e8 the scaled matrix is ill-conditioned, and FP64 elimination itself loses digits: the median
    row's worst entry stays within four times that of LAPACK's inverse."""
    A = cells(1e8, 11)
    amg = hierarchy(ctx, A)
    cols = list(range(0, N_ROWS, 4))
    T = held_inverse(amg, N_ROWS, cols)
    want = refined_columns(A, cols)
    assert worst_of_median_row(T, want) <= 4 * worst_of_median_row(np.linalg.inv(A)[:, cols], want)


BREAKDOWN, TIMEOUT = 6, 8


def solve_status(native, amg, B):
    from afepack_gb300 import _native as N
    X = np.zeros_like(B)
    infos = (N.SolveInfo * B.shape[1])()
    return native.afp_pcg_solve_multi(amg.handle, N.ptr(X), N.ptr(B), B.shape[1], 1e-8, 200, infos)


def test_infinity_in_the_tail_is_a_breakdown(native, ctx):
    """An entry that FP32 cannot hold is an infinity in the V-cycle: the solve breaks down, as it does where the
    product is summed entry by entry, and does not go on with a number made of it."""
    A = cells(1e2, 16)
    amg = hierarchy(ctx, A, 1)
    B = right_hand_sides(A, 48, 17)
    bad = B.copy()
    bad[5, 3] = 1e39
    assert solve_status(native, amg, bad) == BREAKDOWN, native.afp_last_error()
    assert solve_status(native, amg, B) == 0


@pytest.mark.parametrize("entry", [0.0, 1e39])
def test_a_failed_tail_product_is_reported_once(native, ctx, entry):
    """The first product of the width reports a wait that ran out (set from the host).  The call fails for that and
    not for what the residual looks like then, and the next one on the same hierarchy is not blamed for it."""
    A = cells(1e2, 16)
    amg = hierarchy(ctx, A, 1)
    amg.opts.inject_barrier_stall = 2
    amg.reinit(amg.matrix)
    B = right_hand_sides(A, 48, 17)
    first = B.copy()
    first[5, 3] += entry
    assert solve_status(native, amg, first) == TIMEOUT, native.afp_last_error()
    assert solve_status(native, amg, B) == 0, native.afp_last_error()


def test_a_failed_tail_product_ends_the_server_and_nothing_after_it(native, ctx):
    from afepack_gb300.serve import BatchServer
    A = cells(1e2, 16)
    amg = hierarchy(ctx, A, 1)
    amg.opts.inject_barrier_stall = 2
    amg.reinit(amg.matrix)
    B = right_hand_sides(A, 48, 17)
    with BatchServer(amg, width=48) as srv:
        _, res = srv.wait(srv.submit(np.ascontiguousarray(B[:, 0])))
    assert res["status"] == TIMEOUT
    assert solve_status(native, amg, B) == 0, native.afp_last_error()


def test_inverse_of_a_diagonal_matrix_is_its_reciprocal(ctx):
    """Pivots alone: every entry within an ulp of the quotient, over the range of scales that the sweep takes."""
    rng = np.random.default_rng(18)
    d = rng.uniform(1.0, 2.0, 300) * 2.0 ** rng.integers(-390, 390, 300)
    amg = hierarchy(ctx, np.diag(d))
    x = np.zeros(300)
    amg.solve(x, np.ones(300), step=0)
    assert (np.abs(x - 1.0 / d) <= np.spacing(1.0 / d)).all()


@pytest.mark.parametrize("precision", [0, 1])
def test_bytes_of_a_batched_vcycle(ctx, precision):
    """The reported bytes are those of the code that runs: a tail product reads the digits, two bytes each."""
    k = 48
    A = cells(1e2, 16)
    amg = hierarchy(ctx, A, precision)
    amg.pcg_multi(right_hand_sides(A, k, 17), 1e-6, 50)
    _, nbytes = amg.time_kernel(4, 0, 1)
    assert nbytes == N_ROWS ** 2 * 2 * 10 + 2 * N_ROWS * k * (4 if precision else 8)


@pytest.mark.parametrize("n_side,k,precision,digits", [(5, 64, 0, False), (6, 2, 0, False), (7, 3, 0, True),
                                                       (9, 2, 0, True), (6, 64, 1, False), (7, 64, 1, True),
                                                       (7, 16, 1, False), (8, 32, 1, False), (9, 32, 1, True),
                                                       (11, 16, 1, True), (11, 8, 1, False)])
def test_route_of_the_batched_tail(ctx, n_side, k, precision, digits):
    """Small and narrow tails are summed row by row, the others by digits (by the bytes that a V-cycle reports)."""
    A = cells(1e2, 19, n_side)
    n = len(A)
    amg = hierarchy(ctx, A, precision)
    amg.pcg_multi(right_hand_sides(A, k, 20), 1e-6, 50)
    _, nbytes = amg.time_kernel(4, 0, 1)
    assert nbytes == n * n * (20 if digits else 8) + 2 * n * k * (4 if precision else 8)


@pytest.mark.parametrize("first_bad", [0, 250, 300, 520])
def test_pivot_that_turns_out_not_positive(ctx, first_bad):
    """Symmetric, unit diagonal, no entry above it, yet indefinite from row first_bad on (in the first panel of the
    symmetric sweep, across its edge, in the second and in the third): the pivoted sweep takes over from the start."""
    n = 600
    A = np.eye(n)
    i = np.arange(n - 1)
    A[i, i + 1] = A[i + 1, i] = np.where(i >= first_bad, -0.6, -0.3)
    amg = hierarchy(ctx, A)
    b = np.random.default_rng(21).uniform(-1.0, 1.0, n)
    x = np.zeros(n)
    amg.solve(x, b, step=0)
    want = np.linalg.solve(A, b)
    assert np.linalg.eigvalsh(A)[0] < -0.1
    # two sweeps without pivoting across panels, each with growth of a few units
    assert np.linalg.norm(x - want) <= 100 * n * EPS * np.linalg.cond(A) * np.linalg.norm(want)


@pytest.mark.parametrize("exponent,digits", [(-390, False), (-240, False), (-9, False), (-8, True), (0, True),
                                             (8, True), (9, False), (240, False), (390, False)])
def test_tail_with_rows_of_two_sizes(native, ctx, exponent, digits):
    """Rows of size 2^(2 exponent) and of 2^(-2 exponent), coupled by 2^-905 of their diagonals alone: for a solution
    of one size their residuals' scaled entries are 2^(2 exponent) apart, and a chunk that holds nothing but such a
    coupling has a scale far from its row's.  Digits up to a spread of 2^34, row by row beyond; in either case the
    product is good to rounding in both kinds of rows."""
    n, k = 1100, 5
    i = np.arange(400)
    e = 2 * exponent if abs(exponent) < 100 else exponent
    d = np.where(np.arange(n) < 550, 2.0 ** e, 2.0 ** -e)
    A = np.diag(8.0 * d)
    A[i, i + 600] = A[i + 600, i] = -(2.0 ** -905)
    amg = hierarchy(ctx, A)
    want = np.random.default_rng(22).uniform(-1.0, 1.0, (n, k))
    X = one_step(native, amg, want * 8.0 * d[:, None])  # the coupling is far below rounding
    assert np.abs(X - want).max() <= 8 * n * EPS
    _, nbytes = amg.time_kernel(4, 0, 1)
    assert nbytes == n * n * (20 if digits else 8) + 2 * n * k * 8
