"""A X and A^T Y (k_spmm_lean, csrc/spmm.cu) at every width class: the edges of
its lane groups (4 columns FP32, 2 FP64, times 4 / 8 / 16 / 32 lanes and up to
three vectors), widths whose rows are not whole 16-byte vectors (copied), an
unaligned X, several 128-column blocks, rows of every remainder of a chunk,
rows cut into segments, empty rows, an X above 4 GB.

Tolerances, per entry, of sum |a| |x|: FP64 7000 terms x 1.1e-16 < 1e-12; FP32
at most 32 terms in FP32 (1.9e-6), the FP64 sum of the chunks and one rounding:
2.1e-6."""
import ctypes as C

import numpy as np
import pytest
import scipy.sparse as sp
import torch

import matrices as M
from gpu_util import upload
from single_svdlib import _abi
from single_svdlib._core import check

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def rows_of_every_length():
    rng = np.random.default_rng(31)
    m, n = 700, 7500
    lens = np.concatenate([np.arange(0, 200), rng.integers(0, 90, m - 200)])
    lens[[0, 50, 300, 301]] = [0, 0, 7000, 2100]
    rows = np.repeat(np.arange(m), lens)
    cols = np.concatenate([rng.choice(n, k, replace=False) for k in lens])
    S = sp.csr_matrix((rng.standard_normal(len(rows)), (rows, cols)), shape=(m, n))
    S.sort_indices()
    return M.from_scipy(S)


@pytest.fixture(scope="module")
def handle(rows_of_every_length):
    return upload("csr", rows_of_every_length)


def product(h, X, rows, l, transposed, precision, shift=0):
    """Device product of X (numpy), X and the result `shift` elements past an aligned address."""
    dt = torch.float32 if precision else torch.float64
    x = torch.empty(X.size + shift, dtype=dt, device="cuda")
    x[shift:] = torch.from_numpy(X.ravel()).to(dt)
    y = torch.full((rows * l + shift,), float("nan"), dtype=dt, device="cuda")
    torch.cuda.synchronize()
    check(_abi.lib().svdb_multiply_with_dense_device(h.handle, x[shift:].data_ptr(), l, y[shift:].data_ptr(),
                                                     transposed, precision, None))
    torch.cuda.synchronize()
    return y[shift:].double().cpu().numpy().reshape(rows, l)


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("l", [1, 2, 3, 7, 8, 9, 15, 16, 17, 20, 31, 32, 33, 37, 40, 48, 49, 60, 63, 64, 65, 100, 127,
                               128, 129, 200])
def test_widths(rows_of_every_length, handle, l, precision):
    A = rows_of_every_length
    S = M.to_scipy(A)
    if precision:
        S = S.astype(np.float32).astype(np.float64)
    rng = np.random.default_rng(l)
    tol = 2.1e-6 if precision else 1e-12
    for transposed, T in ((0, S), (1, S.T.tocsr())):
        X = rng.standard_normal((T.shape[1], l))
        if precision:
            X = X.astype(np.float32).astype(np.float64)
        got = product(handle, X, T.shape[0], l, transposed, precision)
        bound = abs(T) @ np.abs(X)
        assert np.all(np.abs(got - T @ X) <= tol * bound), (transposed, np.max(np.abs(got - T @ X) / (bound + 1e-300)))
        assert np.all(got[np.diff(T.indptr) == 0] == 0.0)


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("l", [8, 37, 64])
def test_unaligned_operands_give_the_same_bits(rows_of_every_length, handle, l, precision):
    A = rows_of_every_length
    X = np.random.default_rng(3).standard_normal((A["ncols"], l))
    a = product(handle, X, A["nrows"], l, 0, precision)
    np.testing.assert_array_equal(a, product(handle, X, A["nrows"], l, 0, precision, shift=1))


def test_operand_above_4_gb():
    m, n, l, per = 40, 9_000_000, 60, 50
    if torch.cuda.mem_get_info()[0] < 20 << 30:
        pytest.skip("needs 20 GB of free device memory")
    rng = np.random.default_rng(4)
    cols = np.sort(rng.choice(n, (m, per), replace=False), axis=1)
    cols[:, -1] = n - 1 - np.arange(m)  # the far end of X
    vals = torch.from_numpy(rng.standard_normal((m, per))).cuda()
    ip = torch.arange(0, m * per + 1, per, dtype=torch.int64, device="cuda")
    ci = torch.from_numpy(cols.astype(np.int32)).cuda()
    x = torch.randn(n, l, dtype=torch.float64, device="cuda")
    y = torch.empty(m, l, dtype=torch.float64, device="cuda")
    h = C.c_void_p()
    torch.cuda.synchronize()
    check(_abi.lib().svdb_matrix_create_csr_device(m, n, m * per, ip.data_ptr(), ci.data_ptr(), vals.data_ptr(),
                                                   C.byref(h)))
    try:
        check(_abi.lib().svdb_multiply_with_dense_device(h, x.data_ptr(), l, y.data_ptr(), 0, 0, None))
        torch.cuda.synchronize()
    finally:
        _abi.lib().svdb_matrix_destroy(h)
    g = x[ci.long().reshape(-1)].reshape(m, per, l)
    ref, bound = (vals[:, :, None] * g).sum(1), (vals[:, :, None] * g).abs().sum(1)
    assert bool(((y - ref).abs() <= 1e-13 * bound).all())
