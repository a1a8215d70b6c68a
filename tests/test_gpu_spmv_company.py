"""A row's product does not depend on the rows beside it: 2,048 entries are one
warp's, 2,049 a block's, whatever else the operator holds (the length classes of
k_spmv_keys, csrc/spmm.cu, end at the bounds)."""
import numpy as np
import pytest

import matrices as M
from gpu_util import upload
from test_gpu_spmv_order import operator, product

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["f64", "mixed"])
@pytest.mark.parametrize("length", [64, 65, 80, 81, 2047, 2048, 2049, 2050])
def test_same_bits_in_any_company(length, precision):
    n = 5000
    row = operator([length], n, 3)
    x = np.random.default_rng(4).standard_normal(n)
    alone = product(upload("csr", M.from_scipy(row)), x, 1, False, precision)[0]
    import scipy.sparse as sp

    for others in ([2048] * 3, [2049, 2300, 2559], [2560] * 3, [64, 65, 80, 81], [1]):
        a = sp.vstack([operator(others, n, 5), row, operator(others, n, 6)]).tocsr()
        got = product(upload("csr", M.from_scipy(a)), x, a.shape[0], False, precision)
        assert got[len(others)] == alone
