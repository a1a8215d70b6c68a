"""Rows cut into segments as one block's work (k_spmm_cut, csrc/spmm.cu): lengths
on both sides of every class bound (128 entries a segment; 2, 4 and 8 warps a
row; several rounds of a block; 16,384, above which partials are merged), class
sizes that leave a block's slots empty, every width class, both types.

Tolerances, per entry, of sum |a| |x|: as in test_gpu_spmm_widths.py with up to
17,000 terms, 17,000 x 1.1e-16 < 2e-12 at FP64, 2.1e-6 at FP32."""
import numpy as np
import pytest
import scipy.sparse as sp

import matrices as M
from gpu_util import upload
from single_svdlib import _abi
from test_gpu_spmm_widths import product

pytestmark = pytest.mark.gpu

N = 17_000
LENS = {
    "classes": [127, 128, 129, 130, 255, 256, 257, 257, 300, 383, 384, 385, 511, 512, 513, 640, 1023, 1024, 1025, 1026,
                2047, 2048, 2049, 8191, 8193, 16383, 16384],
    "one_of_each": [129, 257, 513],
    "many": [129 + k % 390 for k in range(401)],
    "merged": [16385, 17000, 16384, 700, 200, 130],
}


def operator(kind):
    rng = np.random.default_rng(len(kind))
    lens = rng.permutation(np.concatenate([LENS[kind], rng.integers(0, 40, 4000)]))
    rows = np.repeat(np.arange(len(lens)), lens)
    cols = np.concatenate([rng.choice(N, k, replace=False) for k in lens])
    S = sp.csr_matrix((rng.standard_normal(len(rows)), (rows, cols)), shape=(len(lens), N))
    S.sort_indices()
    return S


@pytest.fixture(scope="module")
def made():
    return {k: (S := operator(k), upload("csr", M.from_scipy(S))) for k in LENS}


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("l", [1, 8, 9, 16, 17, 32, 37, 48, 64, 65, 128, 129, 200])
@pytest.mark.parametrize("kind", sorted(LENS))
def test_cut_rows(made, kind, l, precision):
    S, h = made[kind]
    if precision:
        S = S.astype(np.float32).astype(np.float64)
    X = np.random.default_rng(l).standard_normal((N, l))
    if precision:
        X = X.astype(np.float32).astype(np.float64)
    got = product(h, X, S.shape[0], l, 0, precision)
    assert np.all(np.abs(got - S @ X) <= (2.1e-6 if precision else 2e-12) * (abs(S) @ np.abs(X)))


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("kind", sorted(LENS))
def test_same_bits_as_merged_partials(made, kind, precision, monkeypatch):
    S, h = made[kind]
    X = np.random.default_rng(2).standard_normal((N, 60))
    a = product(h, X, S.shape[0], 60, 0, precision)
    monkeypatch.setenv("SVDB_SPMM", "seg")
    np.testing.assert_array_equal(a, product(h, X, S.shape[0], 60, 0, precision))


@pytest.mark.parametrize("kind,launches", [("classes", 1), ("one_of_each", 1), ("many", 1), ("merged", 2)])
def test_launches(made, kind, launches):
    S, h = made[kind]
    X = np.zeros((N, 20))
    product(h, X, S.shape[0], 20, 0, 0)
    before = _abi.lib().svdb_kernel_launches()
    product(h, X, S.shape[0], 20, 0, 0)
    assert _abi.lib().svdb_kernel_launches() - before == launches
