"""The factorisation after the last power iteration is left out only where the
one before it was harmless (csrc/qr_loose.h): Y with one weak direction, spread
over all columns by Omega, from one that the first CholeskyQR pass resolves to
one lost in rounding.  The one-cluster form (900 rows) and the launch-per-step
one (6,000)."""
import numpy as np
import pytest

import matrices as M
from gpu_util import upload
from single_svdlib import randomized

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("c", [40, 60])
@pytest.mark.parametrize("m", [900, 6000])
@pytest.mark.parametrize("seed", [1, 2, 3])
def test_one_weak_spread_direction(m, c, seed):
    """U = Q U_B with all c columns kept, so U^T U - I shows Q's.  Gram, Cholesky,
    X R^-1 and the back product leave c u each of an orthonormal Q; 20 c u asked."""
    n = 120
    rng = np.random.default_rng(seed)
    U, _ = np.linalg.qr(rng.standard_normal((m, c)))
    V, _ = np.linalg.qr(rng.standard_normal((n, c)))
    off = {}
    for weak in 10.0 ** np.linspace(-6.0, -13.0, 15):
        A = M.dense((U * np.r_[np.ones(c - 1), weak]) @ V.T)
        g = randomized.randomized_svd(upload("csr", A), c, 0, 1, randomized.PowerIterationNormalizer.QR, False, seed)
        off[f"{weak:.0e}"] = np.abs(g.u.T @ g.u - np.eye(c)).max()
    assert max(off.values()) <= 20 * c * 2.0 ** -53, off
