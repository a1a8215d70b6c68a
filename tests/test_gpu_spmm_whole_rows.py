"""Rows of several segments without partials (k_spmm_cut, csrc/spmm.cu) in structures
of more than 10^6 entries: the longest row ends at, or one entry past, the length
from which rows are cut (below it one warp takes a row whole) and four times that,
on both sides of 2^21 and 2^22 entries and of 64 columns.

Tolerances, per entry, of sum |a| |x|: as in test_gpu_spmm_cut.py."""
import numpy as np
import pytest
import scipy.sparse as sp

import matrices as M
from gpu_util import upload
from single_svdlib import _abi
from test_gpu_spmm_widths import product

pytestmark = pytest.mark.gpu

N = 6000
# rows, shortest, longest but five, the five (148 SMs: cut from 257, 513 and 1,025 entries)
SHAPES = {
    "small": (5000, 230, 256, 256),    # 1.2 M entries, segments of 128
    "large": (6000, 300, 512, 512),    # 2.4 M, segments of 256
    "one_past": (6000, 300, 512, 513),
    "four": (6000, 300, 512, 2048),    # four times the length from which rows are cut
    "above": (6000, 300, 512, 2049),   # merged from partials
    "longer": (6000, 600, 1024, 1024),  # 4.9 M, segments of 512
    "cut": (6000, 600, 1024, 1025),    # merged from partials
}


def operator(kind):
    rows, lo, hi, longest = SHAPES[kind]
    rng = np.random.default_rng(rows + longest)
    lens = rng.integers(lo, hi + 1, rows)
    lens[rng.integers(0, rows, 5)] = longest
    r = np.repeat(np.arange(rows), lens)
    c = np.concatenate([rng.choice(N, k, replace=False) for k in lens])
    S = sp.csr_matrix((rng.standard_normal(len(r)), (r, c)), shape=(rows, N))
    S.sort_indices()
    return S


@pytest.fixture(scope="module")
def made():
    return {k: (S := operator(k), upload("csr", M.from_scipy(S))) for k in SHAPES}


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("l", [8, 37, 48, 64, 65, 130])
@pytest.mark.parametrize("kind", sorted(SHAPES))
def test_products(made, kind, l, precision):
    S, h = made[kind]
    X = np.random.default_rng(l).standard_normal((N, l))
    if precision:
        S = S.astype(np.float32).astype(np.float64)
        X = X.astype(np.float32).astype(np.float64)
    got = product(h, X, S.shape[0], l, 0, precision)
    assert np.all(np.abs(got - S @ X) <= (2.1e-6 if precision else 2e-12) * (abs(S) @ np.abs(X)))


@pytest.mark.parametrize("kind,l,launches", [
    ("small", 64, 1), ("small", 128, 1), ("large", 64, 1), ("large", 128, 1), ("one_past", 64, 1), ("one_past", 66, 2),
    ("four", 64, 1), ("above", 64, 2), ("longer", 64, 1), ("longer", 66, 2), ("cut", 64, 2)])
def test_launches(made, kind, l, launches):
    S, h = made[kind]
    X = np.zeros((N, l))
    product(h, X, S.shape[0], l, 0, 0)
    before = _abi.lib().svdb_kernel_launches()
    product(h, X, S.shape[0], l, 0, 0)
    assert _abi.lib().svdb_kernel_launches() - before == launches
