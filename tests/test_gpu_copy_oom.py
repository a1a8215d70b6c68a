"""A product whose operand copy cannot be allocated is done without it, as before
there was one (lean_operand in csrc/spmm.cu, sddmm_launch in csrc/adjoint.cu):
the copies' bits for SpMM, one launch less."""
import ctypes as C

import pytest
import torch

from single_svdlib import _abi
from single_svdlib._core import check

pytestmark = pytest.mark.gpu
MB = 1 << 20


class Filled:
    """All device memory but `left` bytes taken, the library's cached blocks included."""

    def __init__(self, left):
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        check(_abi.lib().svdb_release_cached_memory())
        free = torch.cuda.mem_get_info()[0]
        self.buf = torch.empty(max(free - left, 0), dtype=torch.uint8, device="cuda")

    def __enter__(self):
        return self

    def __exit__(self, *exc):
        del self.buf
        torch.cuda.empty_cache()


def handle(m, n, per):
    g = torch.Generator(device="cuda")
    g.manual_seed(m)
    ip = torch.arange(0, m * per + 1, per, dtype=torch.int64, device="cuda")
    ci = torch.randint(n // per, (m, per), device="cuda", generator=g, dtype=torch.int32)
    ci += torch.arange(0, n // per * per, n // per, device="cuda", dtype=torch.int32)  # ascending, distinct
    v = torch.randn(m * per, dtype=torch.float64, device="cuda", generator=g)
    h = C.c_void_p()
    torch.cuda.synchronize()
    check(_abi.lib().svdb_matrix_create_csr_device(m, n, m * per, ip.data_ptr(), ci.data_ptr(), v.data_ptr(), C.byref(h)))
    return h


def run(call):
    before = _abi.lib().svdb_kernel_launches()
    check(call())
    torch.cuda.synchronize()
    return _abi.lib().svdb_kernel_launches() - before


@pytest.mark.parametrize("m", [20_000, 60_000])  # below and above 2^21 entries: k_spmm_cut, k_spmm_seg
def test_spmm(m):
    n, per, l = 1_000_000, 50, 51
    h = handle(m, n, per)
    try:
        x = torch.randn(n, l, dtype=torch.float64, device="cuda")  # 408 MB, its copy 416 MB
        y, z = (torch.full((m, l), float("nan"), dtype=torch.float64, device="cuda") for _ in range(2))
        L = _abi.lib()
        assert run(lambda: L.svdb_multiply_with_dense_device(h, x.data_ptr(), l, y.data_ptr(), 0, 0, None)) == 2
        with Filled(200 * MB):
            assert run(lambda: L.svdb_multiply_with_dense_device(h, x.data_ptr(), l, z.data_ptr(), 0, 0, None)) == 1
        assert bool((y == z).all())
    finally:
        _abi.lib().svdb_matrix_destroy(h)


def test_sddmm():
    m, n, per, rank = 80_000, 500_000, 50, 63
    h = handle(m, n, per)
    try:
        a = torch.randn(m, rank, dtype=torch.float64, device="cuda")
        b = torch.randn(n, rank, dtype=torch.float64, device="cuda")  # 252 MB, both copies 297 MB
        y, z = (torch.full((m * per,), float("nan"), dtype=torch.float64, device="cuda") for _ in range(2))
        L = _abi.lib()
        assert run(lambda: L.svdb_sddmm_device(h, a.data_ptr(), b.data_ptr(), rank, y.data_ptr(), 0, None)) == 2
        with Filled(200 * MB):
            assert run(lambda: L.svdb_sddmm_device(h, a.data_ptr(), b.data_ptr(), rank, z.data_ptr(), 0, None)) == 1
        # sums of 63 products in two orders: 63 x 2^-53 of sum |a||b| <= |a| |b|, twice
        bound = 2 * 63 * 2.0 ** -53 * a.norm(dim=1).max() * b.norm(dim=1).max()
        assert float((y - z).abs().max()) <= float(bound)
    finally:
        _abi.lib().svdb_matrix_destroy(h)
