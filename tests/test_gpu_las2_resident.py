"""LAS2 with both operands in the cluster's shared memory (k_lanczos_block RES,
csrc/lanczos_kernel.cu) against the same cluster with the operands in global
memory (SVDB_LZ_CLUSTER=2) and the cooperative grid (0): fewer rows than CTAs,
row slices that are not whole, odd sizes, transposed shapes, rows longer than
32 lanes' share, empty rows and columns, FP32 values, purges and restarts.
Steps and purges equal; alpha, beta and sigma within 1e-10, the suite's bound
between implementations."""
import numpy as np
import pytest
import scipy.sparse as sp

import matrices as M
from gpu_util import upload
from single_svdlib import lanczos

pytestmark = pytest.mark.gpu


def dense_lines(m, n, seed):
    """Short rows, one full row, one full column, empty rows and columns."""
    rng = np.random.default_rng(seed)
    D = (rng.random((m, n)) < 0.02) * rng.random((m, n))
    D[m // 3, :] = rng.random(n)
    D[:, n // 2] = rng.random(m)
    D[5:9, :] = 0.0
    D[:, 3:5] = 0.0
    return M.from_scipy(sp.csr_matrix(D))


CASES = {
    "tiny": M.uniform(17, 9, 0.6, 1, 0.1, 1.0),
    "one_row_per_cta": M.uniform(40, 16, 0.5, 2, 0.1, 1.0),
    "odd": M.poisson_rows(1213, 515, 9, 3),
    "wide": M.poisson_rows(301, 1100, 14, 4),
    "square": M.poisson_rows(700, 700, 11, 5),
    "lines": dense_lines(900, 431, 6),
    "lowrank": M.lowrank_plus_noise(120, 90, 6, 0.0, 7),
}


@pytest.mark.parametrize("precision", ["f64", "mixed"])
@pytest.mark.parametrize("name", sorted(CASES))
def test_resident_cluster_follows_the_other_forms(name, precision, monkeypatch):
    A = CASES[name]
    out = {}
    for mode in ("1", "2", "0"):
        monkeypatch.setenv("SVDB_LZ_CLUSTER", mode)
        out[mode] = lanczos.las2_traced(upload("csr", A), 5, 0, random_seed=5, algorithm="legacy", precision=precision)
    r = out["1"]
    assert r["lanczos_blocks"] in (8, 16)
    for mode in ("2", "0"):
        o = out[mode]
        assert type(r["error"]) is type(o["error"]), (mode, r["error"], o["error"])
        assert r["steps"] == o["steps"] and r["purges"] == o["purges"], mode
        for k in ("alf", "bet"):
            np.testing.assert_allclose(r[k], o[k], rtol=0, atol=1e-10 * np.abs(o[k]).max(), err_msg=mode)
        if o["error"] is None:
            assert r["rec"].d == o["rec"].d
            np.testing.assert_allclose(r["rec"].s, o["rec"].s, rtol=0, atol=1e-10 * o["rec"].s.max())
