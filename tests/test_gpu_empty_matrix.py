"""randomized_svd of a matrix without rows or columns raises, as it always did
(zero columns once reached a division by the number of tiles on the host)."""
import numpy as np
import pytest

from single_svdlib import CsrMatrix, MaskedCSRMatrix, SvdLibError, randomized

pytestmark = pytest.mark.gpu
PIN = randomized.PowerIterationNormalizer


@pytest.mark.parametrize("precision", ["f64", "mixed"])
@pytest.mark.parametrize("norm", ["QR", "LU", "None_"])
@pytest.mark.parametrize("shape", [(5, 0), (0, 5), (0, 0), "masked"])
def test_no_rows_or_columns(shape, norm, precision):
    if shape == "masked":
        parent = CsrMatrix(6, 4, np.arange(0, 13, 2), np.tile([0, 3], 6), np.ones(12))
        A = MaskedCSRMatrix(parent, np.zeros(4, dtype=bool))
    else:
        m, n = shape
        A = CsrMatrix(m, n, np.zeros(m + 1, dtype=np.int64), np.zeros(0, dtype=np.int64), np.zeros(0))
    for q in (0, 2):
        with pytest.raises(SvdLibError, match="no rows or no columns"):
            randomized.randomized_svd(A, 3, 4, q, getattr(PIN, norm), False, 7, precision=precision)
