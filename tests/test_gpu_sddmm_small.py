"""SDDMM of small products at ranks that are no whole 16-byte vectors
(sddmm_launch, csrc/adjoint.cu): read element by element, one launch, no copy;
copied in one launch more where enough is gathered.  Every width class of both
forms, unaligned factors, rows on both sides of a 32-entry chunk and of a segment.

Tolerances: rank terms, rank x 2^-53 (2^-24 at FP32) of sum |l| |r|, twice for the
reference's own."""
import numpy as np
import pytest
import scipy.sparse as sp
import torch

import matrices as M
from gpu_util import upload
from single_svdlib import _abi
from single_svdlib._core import check

pytestmark = pytest.mark.gpu


def pattern(m, n, per, seed):
    rng = np.random.default_rng(seed)
    lens = rng.integers(max(0, per - 20), per + 20, m)
    lens[:12] = [0, 1, 31, 32, 33, 63, 64, 65, 127, 128, 129, min(n, 600)]
    rows = np.repeat(np.arange(m), lens)
    cols = np.concatenate([np.sort(rng.choice(n, k, replace=False)) for k in lens])
    return rows, cols, sp.csr_matrix((np.ones(len(rows)), (rows, cols)), shape=(m, n))


@pytest.fixture(scope="module")
def made():
    out = {}
    for name, (m, n, per) in {"small": (700, 800, 25), "larger": (3000, 1500, 220)}.items():
        rows, cols, S = pattern(m, n, per, m)
        S.sort_indices()
        out[name] = (torch.from_numpy(rows).cuda(), torch.from_numpy(cols).cuda(), upload("csr", M.from_scipy(S)), m, n)
    return out


def sddmm(h, left, right, rank, nnz, dt, shift):
    def at(x):
        b = torch.empty(x.numel() + shift, dtype=dt, device="cuda")
        b[shift:] = x.reshape(-1)
        return b[shift:]

    l, r = at(left), at(right)
    y = torch.full((nnz,), float("nan"), dtype=dt, device="cuda")
    torch.cuda.synchronize()
    before = _abi.lib().svdb_kernel_launches()
    check(_abi.lib().svdb_sddmm_device(h.handle, l.data_ptr(), r.data_ptr(), rank, y.data_ptr(),
                                       1 if dt == torch.float32 else 0, None))
    torch.cuda.synchronize()
    return y, _abi.lib().svdb_kernel_launches() - before


@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("dt", [torch.float32, torch.float64])
@pytest.mark.parametrize("rank", [1, 3, 4, 5, 7, 8, 9, 15, 17, 31, 33, 37, 63, 64, 65, 96, 97, 127, 129, 192, 193, 255])
@pytest.mark.parametrize("size", ["small", "larger"])
def test_ranks(made, size, rank, dt, shift):
    rows, cols, h, m, n = made[size]
    g = torch.Generator(device="cuda")
    g.manual_seed(rank)
    left = torch.randn(m, rank, dtype=dt, device="cuda", generator=g)
    right = torch.randn(n, rank, dtype=dt, device="cuda", generator=g)
    got, launches = sddmm(h, left, right, rank, len(rows), dt, shift)
    prod = left.double()[rows] * right.double()[cols]
    bound = 2 * rank * 2.0 ** (-24 if dt == torch.float32 else -53) * prod.abs().sum(1)
    assert bool(((got.double() - prod.sum(1)).abs() <= bound).all())
    whole = rank * left.element_size() % 16 == 0 and shift == 0
    copied = len(rows) * rank > 1 << 25
    assert launches == (1 if whole or not copied else 2)
