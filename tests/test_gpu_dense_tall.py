"""The tall-skinny FP64 products (csrc/dense_tall.cuh) at the edges of their
8-column fragments, 32-column tile blocks and 64-column CTAs."""
import numpy as np
import pytest

import matrices as M
from gpu_util import upload
import oracle as O
import torch
from single_svdlib import _abi, adjoint, randomized
from single_svdlib._core import check
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


@pytest.mark.parametrize("c", [1, 7, 8, 9, 24, 25, 32, 33, 40, 60, 64, 65, 96, 100, 128])
@pytest.mark.parametrize("rows", [1, 3, 64, 65, 1000, 20011])
def test_gram(rows, c):
    """X^T X: rows terms of one rounding each, u sum |x_a| |x_b|, and symmetric."""
    x = torch.from_numpy(np.random.default_rng(rows + c).standard_normal((rows, c))).cuda()
    g = torch.full((c, c), float("nan"), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    check(_abi.lib().svdb_gram_device(x.data_ptr(), rows, c, g.data_ptr(), 0, None))
    torch.cuda.synchronize()
    bound = (rows + 2) * 2.0 ** -53 * (x.abs().T @ x.abs())
    assert bool(((g - x.T @ x).abs() <= 2 * bound).all())  # the reference rounds as often
    assert bool((g == g.T).all())


@pytest.mark.parametrize("l", [1, 2, 7, 8, 9, 15, 16, 17, 33, 40, 59, 64, 65, 100, 117])
@pytest.mark.parametrize("shape", [(260, 200), (1500, 130), (120, 700)])
def test_solve_widths(l, shape):
    """CholeskyQR2 (panels of eight pivots, one tile row per panel), X R^-1 and
    the back products at every width class against the checker on the same
    Omega.  Singular values within 1e-10, the suite's bound for FP64."""
    m, n = shape
    A = M.uniform(m, n, 0.3, 40 + m, -1.0, 1.0)
    om = M.omega(n, l, l)
    g = randomized.randomized_svd(upload("csr", A), l, 0, 1, randomized.PowerIterationNormalizer.QR, False, 3, False,
                                  omega=om)
    r = O.randomized(A, l, 0, 1, "QR", omega=om)
    np.testing.assert_allclose(g.s, r["s"], rtol=1e-10)
    k = len(g.s)
    assert np.abs(g.u.T @ g.u - np.eye(k)).max() < 1e-12 and np.abs(g.vt @ g.vt.T - np.eye(k)).max() < 1e-12


@pytest.mark.parametrize("q", [0, 1, 3])
@pytest.mark.parametrize("m", [900, 6000])
@pytest.mark.parametrize("kind", ["deficient", "graded"])
def test_difficult_factorisations(kind, m, q):
    """Shifted passes and nearly dependent columns, in the one-cluster form
    (900 x 64) and the launch-per-step one (6,000 x 64), with the factorisation
    after the last power iteration skipped only where it may be: the leading
    singular values against numpy's, and orthonormal leading vectors.  A has 30
    singular values, equal-sized or spread over 1e-9: with 64 sample columns its
    range is captured to rounding, u ||A|| sqrt(n) = 2e-15 ||A||, 1e-12 asked."""
    n, k = 200, 30
    rng = np.random.default_rng(m + q)
    U, _ = np.linalg.qr(rng.standard_normal((m, k)))
    V, _ = np.linalg.qr(rng.standard_normal((n, k)))
    s = np.linspace(5.0, 3.0, k) if kind == "deficient" else 10.0 ** np.linspace(0, -9, k)
    A = M.dense((U * s) @ V.T)
    g = randomized.randomized_svd(upload("csr", A), 40, 24, q, randomized.PowerIterationNormalizer.QR, False, 3)
    ref = np.linalg.svd(M.to_scipy(A).toarray(), compute_uv=False)
    assert np.abs(g.s[:k] - ref[:k]).max() <= 1e-12 * ref[0]
    lead = k if kind == "deficient" else 20  # those above 1e-6: the others' directions are rounding at 1e-9
    u, vt = g.u[:, :lead], g.vt[:lead]
    assert np.abs(u.T @ u - np.eye(lead)).max() < 1e-10 and np.abs(vt @ vt.T - np.eye(lead)).max() < 1e-10
