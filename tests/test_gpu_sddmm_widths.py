"""svdb_sddmm_device (k_sddmm, csrc/adjoint.cu) at the edges of its lane groups
and vectors, ranks whose rows are not whole 16-byte vectors, unaligned
factors, rows of every remainder of a 32-entry chunk and rows cut into
segments, CSR and CSC entry order.

Tolerance per entry: rank products and sums of sum |l| |r|, each rounded once:
(rank + 1) u, u = 2^-53 or 2^-24."""
import numpy as np
import pytest
import scipy.sparse as sp
import torch

import matrices as M
from gpu_util import upload
from single_svdlib import adjoint

pytestmark = pytest.mark.gpu
m, n = 300, 6000


@pytest.fixture(scope="module")
def A():
    rng = np.random.default_rng(12)
    lens = np.concatenate([np.arange(100), rng.integers(0, 150, m - 100)])
    lens[[0, 7, 200]] = [0, 0, 5000]
    rows = np.repeat(np.arange(m), lens)
    cols = np.concatenate([rng.choice(n, k, replace=False) for k in lens])
    S = sp.csr_matrix((rng.standard_normal(len(rows)), (rows, cols)), shape=(m, n))
    S.sort_indices()
    return M.from_scipy(S)


@pytest.mark.parametrize("precision", ["f64", "mixed"])
@pytest.mark.parametrize("rank", [1, 2, 3, 4, 8, 9, 16, 17, 31, 32, 33, 48, 63, 64, 65, 96, 97, 128, 129, 200, 256])
def test_ranks(A, rank, precision):
    dt, u = (torch.float64, 2.0 ** -53) if precision == "f64" else (torch.float32, 2.0 ** -24)
    rng = np.random.default_rng(rank)
    L, R = (torch.from_numpy(rng.standard_normal((k, rank))).to(dt).cuda() for k in (m, n))
    for kind in ("csr", "csc"):
        h = upload(kind, A)
        D = A if kind == "csr" else M.to_csc(A)
        major = np.repeat(np.arange(m if kind == "csr" else n), np.diff(D["indptr"]))
        r, c = (major, D["indices"]) if kind == "csr" else (D["indices"], major)
        l, x = L.double().cpu().numpy()[r], R.double().cpu().numpy()[c]
        ref, bound = (l * x).sum(1), np.abs(l * x).sum(1)
        for shift in (0, 1):  # factors one element past an aligned address
            ls, rs = (torch.empty(t.numel() + shift, dtype=dt, device="cuda") for t in (L, R))
            ls[shift:], rs[shift:] = L.ravel(), R.ravel()
            out = torch.full((len(ref) + shift,), float("nan"), dtype=dt, device="cuda")
            torch.cuda.synchronize()
            adjoint.sddmm_device(h, ls[shift:].data_ptr(), rs[shift:].data_ptr(), rank, out[shift:].data_ptr(),
                                 precision)
            torch.cuda.synchronize()
            got = out[shift:].double().cpu().numpy()
            assert np.all(np.abs(got - ref) <= (rank + 1) * u * bound), (kind, shift)
