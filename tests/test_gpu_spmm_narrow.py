"""Products whose operand rows are no whole 16-byte vectors (lean_operand,
csrc/spmm.cu): read element by element in small products, copied in larger ones,
either way the bits of the same columns inside an operand of whole vectors; and a
small product is one launch."""
import numpy as np
import pytest
import scipy.sparse as sp

import matrices as M
from gpu_util import upload
from single_svdlib import _abi
from test_gpu_spmm_widths import product

pytestmark = pytest.mark.gpu


def handle(per, seed):
    """900 x 3000, `per` entries a row, a row of 1500 and an empty one."""
    rng = np.random.default_rng(seed)
    lens = np.full(900, per)
    lens[[3, 400]] = [1500, 0]
    rows = np.repeat(np.arange(900), lens)
    cols = np.concatenate([rng.choice(3000, k, replace=False) for k in lens])
    S = sp.csr_matrix((rng.standard_normal(len(rows)), (rows, cols)), shape=(900, 3000))
    S.sort_indices()
    return upload("csr", M.from_scipy(S))


@pytest.fixture(scope="module")
def handles():
    return {"small": handle(30, 1), "larger": handle(400, 2)}  # 27,000 and 360,000 entries


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("transposed", [0, 1])
@pytest.mark.parametrize("l", [1, 3, 7, 9, 15, 17, 31, 33, 47, 49, 63, 65, 101, 127, 129])
@pytest.mark.parametrize("size", ["small", "larger"])
def test_same_bits_as_whole_vectors(handles, size, l, transposed, precision):
    h = handles[size]
    rows, n = (3000, 900) if transposed else (900, 3000)
    X = np.random.default_rng(l).standard_normal((n, l))
    wide = np.zeros((n, l + 3 & ~3))  # no class of widths ends between
    wide[:, :l] = X
    a = product(h, X, rows, l, transposed, precision)
    np.testing.assert_array_equal(a, product(h, wide, rows, wide.shape[1], transposed, precision)[:, :l])


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("l", [1, 7, 37, 63, 101, 127])
def test_small_products_are_one_launch(handles, l, precision):
    X = np.zeros((3000, l))
    product(handles["small"], X, 900, l, 0, precision)
    before = _abi.lib().svdb_kernel_launches()
    product(handles["small"], X, 900, l, 0, precision)
    assert _abi.lib().svdb_kernel_launches() - before == 1
