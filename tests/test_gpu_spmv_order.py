"""SpMV over rows whose lengths sit at the edges of the length classes.

The product deals the rows, longest class first, forwards and backwards over
the warps (and the rows of more than 2,048 entries over the blocks), so the
cases are lengths on both sides of every class edge, counts that end inside a
round, and operators with one class only.  The reference is the row sums in
extended precision; FP64 sums of at most 20,000 products in some order are
within 20,000 x 2^-53 < 3e-12 of sum |a||x|, and a tree of lanes is far closer:
1e-13 is taken, as for the other SpMV tests.
"""

import numpy as np
import pytest
import scipy.sparse as sp

import matrices as M
from gpu_util import upload
from single_svdlib import _abi

pytestmark = pytest.mark.gpu

EDGES = [0, 1, 2, 7, 8, 9, 15, 16, 17, 31, 32, 33, 63, 64, 65, 127, 128, 129, 255, 256, 511, 512, 1023, 1024, 2047,
         2048, 2049, 2303, 2304, 2559, 2560, 4095, 4096, 4097, 8191, 8192]


def operator(lengths, n, seed):
    rng = np.random.default_rng(seed)
    lengths = np.asarray(lengths)
    indptr = np.concatenate([[0], np.cumsum(lengths)])
    idx = np.concatenate([np.sort(rng.choice(n, k, replace=False)) for k in lengths] or [np.zeros(0)])
    return sp.csr_matrix((rng.standard_normal(indptr[-1]), idx.astype(np.int64), indptr), shape=(len(lengths), n))


def lengths_of(kind):
    rng = np.random.default_rng(7)
    if kind == "edges":  # every edge, in no order
        return rng.permutation(np.repeat(EDGES, 3))
    if kind == "rounds":  # short rows for several rounds of every warp, and a few long ones
        return rng.permutation(np.concatenate([rng.integers(0, 70, 150_001), [2049, 5000, 8192, 300, 900]]))
    if kind == "long":  # only rows taken by a block, more than one round of them
        return 2049 + rng.integers(0, 40, 1501)
    return np.full(1, {"one": 3, "one_long": 8000, "empty": 0}[kind])


def product(h, x, rows, transposed, precision):
    import torch

    dx = torch.from_numpy(x).cuda()
    dy = torch.full((rows,), float("nan"), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    rc = _abi.lib().svdb_opa_device(h.handle, dx.data_ptr(), dy.data_ptr(), int(transposed), int(precision == "mixed"),
                                    None)
    assert rc == 0, _abi.last_error()
    torch.cuda.synchronize()
    return dy.cpu().numpy()


@pytest.mark.parametrize("precision", ["f64", "mixed"])
@pytest.mark.parametrize("kind", ["edges", "rounds", "long", "one", "one_long", "empty"])
def test_length_classes(kind, precision):
    a = operator(lengths_of(kind), 9001, 11)
    rng = np.random.default_rng(5)
    h = upload("csr", M.from_scipy(a))
    stored = a if precision == "f64" else a.astype(np.float32).astype(np.float64)
    for op, transposed in ((stored, False), (stored.T.tocsr(), True)):
        x = rng.standard_normal(op.shape[1])
        got = product(h, x, op.shape[0], transposed, precision)
        terms = op.data.astype(np.longdouble) * x[op.indices]
        want, scale = np.zeros((2, op.shape[0]), dtype=np.longdouble)
        rows = np.diff(op.indptr) > 0
        if op.nnz:
            want[rows] = np.add.reduceat(terms, op.indptr[:-1][rows])
            scale[rows] = np.add.reduceat(abs(terms), op.indptr[:-1][rows])
        assert np.all(abs(got - want) <= 1e-13 * scale)
