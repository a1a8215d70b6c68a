"""The tall-skinny FP64 products (csrc/dense_tall.cuh) at the edges of their
8-column fragments, 32-column tile blocks and 64-column CTAs."""
import numpy as np
import pytest

import matrices as M
from gpu_util import upload
from single_svdlib import adjoint
from test_gpu_adjoint import at_pattern, dense_reference

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [1, 7, 8, 9, 32, 33, 40, 65, 100, 128])
def test_adjoint_widths(k):
    """X^T Y and X C of every width through the adjoint, against torch's dense
    backward.  Singular values 10 .. 1 in equal steps (0.065): the systems'
    condition is at most 100 / 0.13, CG stops at 1e-12, so 1e-8 of the largest
    entry leaves a factor of ten."""
    m, n = 150, 140
    rng = np.random.default_rng(k)
    Q, _ = np.linalg.qr(rng.standard_normal((m, n)))
    W, _ = np.linalg.qr(rng.standard_normal((n, n)))
    A = M.dense((Q * np.linspace(10.0, 1.0, n)) @ W.T)
    gU, gs, gV = rng.standard_normal((m, k)), rng.standard_normal(k), rng.standard_normal((n, k))
    U, S, V, D = dense_reference(A, k, gU, gs, gV)
    got = adjoint.svd_adjoint(upload("csr", A), U, S, V, gU, gs, gV)
    ref = at_pattern(A, D)
    assert np.abs(got - ref).max() <= 1e-8 * np.abs(ref).max()
