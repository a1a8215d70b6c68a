"""FP32 SDDMM is no further from 64 bits than a lane per column and a tree over
the lanes (chains of rank / 32 products, five levels), the order it had first.
Rounding variances, in units of one product's: rank 64 416 in both orders, rank 96
688 against 672, rank 128 960 in both; so 1.3 % further off at most, and 3 % asked
(the sample's own spread is below 0.5 %)."""
import numpy as np
import pytest
import scipy.sparse as sp
import torch

import matrices as M
from gpu_util import upload
from single_svdlib import adjoint

pytestmark = pytest.mark.gpu


def lanes_and_tree(prod, rank):
    """prod: exact FP64 products (entries x rank), summed as the 32 lanes did."""
    slots = -(-rank // 32)
    p = np.zeros((prod.shape[0], slots * 32))
    p[:, :rank] = prod
    p = p.reshape(-1, slots, 32)
    acc = np.zeros((prod.shape[0], 32), dtype=np.float32)
    for j in range(slots):  # fused: one rounding each
        acc = (acc.astype(np.float64) + p[:, j]).astype(np.float32)
    w = 16
    while w:
        acc = acc[:, :w] + acc[:, w:2 * w]
        w //= 2
    return acc[:, 0]


@pytest.mark.parametrize("rank", [16, 32, 48, 64, 80, 96, 112, 128, 256])
def test_error_against_64_bits(rank):
    m, n, per = 2000, 1500, 40
    rng = np.random.default_rng(rank)
    cols = np.concatenate([np.sort(rng.choice(n, per, replace=False)) for _ in range(m)])
    S = sp.csr_matrix((np.ones(m * per), cols, np.arange(0, m * per + 1, per)), shape=(m, n))
    h = upload("csr", M.from_scipy(S))
    left, right = (rng.standard_normal((k, rank)).astype(np.float32) for k in (m, n))
    tl, tr = torch.from_numpy(left).cuda(), torch.from_numpy(right).cuda()
    out = torch.full((m * per,), float("nan"), dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()
    adjoint.sddmm_device(h, tl.data_ptr(), tr.data_ptr(), rank, out.data_ptr(), "mixed")
    torch.cuda.synchronize()
    prod = left.astype(np.float64)[np.repeat(np.arange(m), per)] * right.astype(np.float64)[cols]
    exact = prod.sum(1)
    got = np.linalg.norm(out.cpu().numpy().astype(np.float64) - exact)
    tree = np.linalg.norm(lanes_and_tree(prod, rank).astype(np.float64) - exact)
    assert got <= 1.03 * tree, got / tree
