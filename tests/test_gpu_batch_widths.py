"""Batches of column subsets at the width classes of their kernels (csrc/batch.cu):
FP64 products in lane groups of 4 / 8 / 16 lanes with one to three vectors on
rows padded to 16 bytes, Gram and X R^-1 tiles of 8 columns, subsets as small
as the sample, rows that are no multiple of a tile.  Each subset against
randomized_svd on the same masked view and seed: singular values within 1e-10
(the suite's bound for FP64 batches), 1e-6 for mixed ones."""
import numpy as np
import pytest

import matrices as M
from gpu_util import upload
from single_svdlib import MaskedCSRMatrix, randomized
from single_svdlib.randomized import PowerIterationNormalizer as PIN

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def case():
    A = M.lowrank_plus_noise(777, 301, 40, 1e-2, 8, density=0.4)
    return A, upload("csr", A)


@pytest.mark.parametrize("norm", [PIN.QR, PIN.LU])
@pytest.mark.parametrize("l", [2, 7, 8, 9, 15, 16, 17, 31, 32, 33, 47, 48, 49, 63, 64])
def test_f64_widths(case, l, norm):
    A, h = case
    rng = np.random.default_rng(l)
    subs = [rng.choice(301, k, replace=False) for k in (l, 64, 301, 150)]
    rank = max(1, l - 3)
    got = randomized.randomized_svd_batch(h, subs, rank, l - rank, 2, norm, 9, precision="f64")
    for cols, g in zip(subs, got):
        r = randomized.randomized_svd(MaskedCSRMatrix.with_columns(h, cols), rank, l - rank, 2, norm, False, 9)
        np.testing.assert_allclose(g.s, r.s, rtol=1e-10)
        assert g.u.shape == (777, rank) and g.vt.shape == (rank, len(cols))
        assert np.abs(g.u.T @ g.u - np.eye(rank)).max() < 1e-10 and np.abs(g.vt @ g.vt.T - np.eye(rank)).max() < 1e-10


@pytest.mark.parametrize("l", [17, 20, 40, 63, 64])
def test_mixed_widths(case, l):
    A, h = case
    rng = np.random.default_rng(l)
    subs = [rng.choice(301, k, replace=False) for k in (70, 301, 150)]
    rank = l - 4
    a = randomized.randomized_svd_batch(h, subs, rank, 4, 2, PIN.QR, 9, precision="mixed")
    b = randomized.randomized_svd_batch(h, subs, rank, 4, 2, PIN.QR, 9, precision="f64")
    for x, y in zip(a, b):
        assert np.max(np.abs(x.s - y.s) / y.s[0]) < 1e-6
