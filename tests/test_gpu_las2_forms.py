"""Which form LAS2's Lanczos blocks take (svdb_lanczos_form) at the limits of
the resident cluster: n = 8192 / 8193, operands below and above its shared
memory, a layout that leaves no room for the coefficients, 2^20 nonzeros and
one more or less, with the cluster forced.  Steps and purges as the
cooperative grid's; alpha, beta within 1e-10 of the largest, the suite's bound
between implementations."""
import numpy as np
import pytest
import scipy.sparse as sp

import matrices as M
from gpu_util import upload
from single_svdlib import lanczos
from test_gpu_las2_resident import CASES

pytestmark = pytest.mark.gpu

SMEM = 232448 - 1024 - 8192  # dynamic shared memory of a resident CTA


def circulant(m, n, p, seed, extra=0):
    """p entries a row, m p / n a column: the 16 row ranges hold equal counts."""
    rng = np.random.default_rng(seed)
    r = np.repeat(np.arange(m), p)
    c = (r + 3 * np.tile(np.arange(p), m)) % n
    D = sp.csr_matrix((rng.uniform(0.1, 1.0, m * p), (r, c)), shape=(m, n))
    if extra:
        D = sp.csr_matrix(D)
        D[0, n - 1] = 0.5
    return M.from_scipy(sp.csr_matrix(D))


def layout(m, n, p):
    """Bytes of the resident layout of circulant(m, n, p) at FP64, without the coefficients."""
    rows = [((k + 15) // 16 + 1) // 2 * 2 for k in (m, n)]
    nnz = [rows[0] * p, rows[1] * (m * p // n)]
    b = (n + 1) // 2 * 16 + (m + 1) // 2 * 16 + 8 * max(rows)
    return b + 8 * sum(nnz) + sum((k + 2) // 2 * 8 for k in rows) + \
        sum((2 * k + 7) // 8 * 8 for k in nnz)


def tight():
    """A shape whose layout leaves less than 512 bytes: the coefficients of 14 steps do not fit."""
    for m in range(2048, 4096, 32):
        for n in (m, m // 2):
            for p in range(20, 80, 2):
                if 0 <= SMEM - layout(m, n, p) < 512:
                    return m, n, p
    raise AssertionError("no tight shape")


FORMS = {
    "n8192": (lambda: circulant(9000, 8192, 3, 1), None, "resident"),
    "n8193": (lambda: circulant(9000, 8193, 3, 2), None, "cluster"),
    "smem_below": (lambda: circulant(3072, 2048, 38, 3), None, "resident"),
    "smem_above": (lambda: circulant(3072, 2048, 56, 4), None, "cluster"),
    "tight": (lambda: circulant(*tight(), 5), None, "resident"),
    "nnz_2^20-1": (lambda: circulant(1025, 1025, 1023, 6), None, "cluster"),
    "nnz_2^20": (lambda: circulant(4096, 4096, 256, 7), None, "cluster"),
    "nnz_2^20_rows16384": (lambda: circulant(16384, 4096, 64, 8), None, "cluster"),
    "nnz_2^20_forced": (lambda: circulant(4096, 4096, 256, 7), "1", "cluster"),
    "nnz_2^20+1": (lambda: circulant(4096, 4096, 256, 9, 1), None, "grid"),
    "nnz_2^20+1_forced": (lambda: circulant(4096, 4096, 256, 9, 1), "1", "cluster"),
}


@pytest.mark.parametrize("name", sorted(FORMS))
def test_form_at_the_limits(name, monkeypatch):
    make, mode, form = FORMS[name]
    A = make()
    if "2^20" in name:
        want = (1 << 20) + (1 if "+1" in name else -1 if "-1" in name else 0)
        assert len(A["data"]) == want
    out = {}
    for env in (mode, "0"):
        if env is None:
            monkeypatch.delenv("SVDB_LZ_CLUSTER", raising=False)
        else:
            monkeypatch.setenv("SVDB_LZ_CLUSTER", env)
        out[env] = lanczos.las2_traced(upload("csr", A), 4, 24, random_seed=5, algorithm="legacy")
    r, o = out[mode], out["0"]
    assert r["lanczos_form"] == form and o["lanczos_form"] == "grid"
    assert type(r["error"]) is type(o["error"]), (r["error"], o["error"])
    assert r["steps"] == o["steps"] and r["purges"] == o["purges"]
    for k in ("alf", "bet"):
        np.testing.assert_allclose(r[k], o[k], rtol=0, atol=1e-10 * np.abs(o[k]).max())


@pytest.mark.parametrize("name", sorted(CASES))
def test_form_of_small_operators(name, monkeypatch):
    for env, form in (("1", "resident"), ("2", "cluster"), ("0", "grid")):
        monkeypatch.setenv("SVDB_LZ_CLUSTER", env)
        assert lanczos.las2_traced(upload("csr", CASES[name]), 5, 0, random_seed=5)["lanczos_form"] == form
