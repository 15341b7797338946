"""SparseMatrix::vmult with the arrays a caller may pass: host, device, in place, overlapping, at an odd offset of an
allocation; every form gives the same product."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _call(K, x, y):
    from afepack_gb300 import _native as N
    import ctypes as C
    N.call("afp_matrix_vmult", K.handle, C.c_void_p(x), C.c_void_p(y))


@pytest.mark.parametrize("n", [1, 31, 1000])
def test_vmult_array_forms(ctx, n):
    torch = pytest.importorskip("torch")
    from afepack_gb300.fem import SparseMatrix
    rng = np.random.default_rng(n)
    rp, ci, va = [0], [], []
    for i in range(n):
        js = [i] + sorted({int(j) for j in rng.integers(0, n, 6)} - {i})
        ci += js
        va += list(rng.standard_normal(len(js)))
        rp.append(len(ci))
    K = SparseMatrix.from_csr(ctx, np.array(rp, np.int32), np.array(ci, np.int32), np.array(va))
    x = rng.standard_normal(n)
    want = K.vmult(x)
    buf = torch.zeros(3 * n + 8, dtype=torch.float64, device="cuda")
    bytes_ = torch.zeros(16 * n + 64, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    at = lambda t, i: t.data_ptr() + i * t.element_size()

    def run(xi, yi, t):
        """x at element xi and y at element yi of one allocation"""
        raw = torch.from_numpy(x.view(np.uint8).copy()).cuda()
        t.view(torch.uint8)[xi * t.element_size():xi * t.element_size() + 8 * n] = raw
        torch.cuda.synchronize()
        _call(K, at(t, xi), at(t, yi))
        got = t.view(torch.uint8)[yi * t.element_size():yi * t.element_size() + 8 * n].cpu().numpy().copy()
        return got.view(np.float64)

    assert np.array_equal(run(0, n, buf), want)          # one after the other
    assert np.array_equal(run(n + 3, 1, buf), want)      # the other way round, odd elements
    assert np.array_equal(run(2, 2, buf), want)          # in place
    assert np.array_equal(run(0, max(1, n // 2), buf), want)  # overlapping
    assert np.array_equal(run(3, 8 * n + 13, bytes_), want)   # not aligned to a double
    y = np.empty(n)
    d = torch.from_numpy(x).cuda()
    torch.cuda.synchronize()
    _call(K, d.data_ptr(), y.ctypes.data)                # device in, host out
    assert np.array_equal(y, want)
    out = torch.empty(n, dtype=torch.float64, device="cuda")
    _call(K, x.ctypes.data, out.data_ptr())              # host in, device out
    assert np.array_equal(out.cpu().numpy(), want)
