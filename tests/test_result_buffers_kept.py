"""Results lent to numpy (single_svdlib._core) where the caller keeps them or
forks, against a fake of the library: what stays out, and whose memory it is."""
import ctypes as C
import gc
import mmap
import os

import numpy as np
import pytest

from single_svdlib import _abi, _core
from test_result_buffers import FakeLib, record


@pytest.fixture()
def fake(monkeypatch):
    f = FakeLib()
    monkeypatch.setattr(_abi, "lib", lambda: f)
    for name, value in (("_lent", 0), ("_lent_cap", 0), ("_out", {}), ("_calls", {})):
        monkeypatch.setattr(_core, name, value)
    yield f
    gc.collect()
    assert not f.live and _core._lent == 0 and _core._lent_cap == 0 and not _core._out and not _core._calls


def solve(f, m, call=None):
    r = record(f, m, 4, 10)
    rec = _core.rec_from_c(r, call)
    f.svdb_rec_free(C.byref(r))
    return rec


@pytest.mark.parametrize("kb", [64, 200, 1000, 4096])
def test_kept_results_are_copied_after_a_few(fake, kb):
    """No fresh page-locked buffer per call: a few are out, the others are copies."""
    m = kb * 1024 // 32
    kept = [solve(fake, m) for _ in range(40)]
    assert len(_core._out) <= _core._KEPT_CALLS + 2
    cap = max(2 * kb << 10, 2 << 20)
    assert _core._lent_cap == cap * len(_core._out) and _core._lent_cap <= _core._LENT_CAP
    for k in kept:
        np.testing.assert_array_equal(k.u.ravel(), np.arange(m * 4.0))
    del k, kept


def test_dropped_results_are_always_lent(fake):
    first, last = solve(fake, 20000), None
    for _ in range(30):  # the previous result lives while the next one is made, and so does the first
        last = solve(fake, 20000)
        assert last.u.ctypes.data in _core._out
    del first, last


def test_results_of_one_call_count_once(fake):
    for _ in range(6):
        call = _core.next_call()
        batch = [solve(fake, 3000, call) for _ in range(16)]
        assert all(b.u.ctypes.data in _core._out for b in batch)
    del batch


def test_page_locked_bytes_are_bounded(fake, monkeypatch):
    monkeypatch.setattr(_core, "_KEPT_CALLS", 10 ** 6)
    kept = [solve(fake, 2048) for _ in range(600)]  # 64 KB each, 2 MB behind each
    assert _core._lent_cap <= _core._LENT_CAP and len(_core._out) == _core._LENT_CAP >> 21
    del kept


@pytest.mark.skipif(not hasattr(os, "fork"), reason="needs fork")
@pytest.mark.filterwarnings("ignore::DeprecationWarning")
def test_a_forked_child_has_its_own_results(fake):
    shared = mmap.mmap(-1, 1 << 20)  # shared with a child, page-aligned: as page-locked memory is
    a = np.frombuffer(shared, dtype=np.float64)
    a[:20000 * 4] = np.arange(80000.0)
    r = record(fake, 20000, 4, 10)
    del fake.live[C.cast(r.u, C.c_void_p).value]
    fake.live[a.ctypes.data] = a
    r.u = C.cast(a.ctypes.data, C.POINTER(C.c_double))
    rec = _core.rec_from_c(r)
    fake.svdb_rec_free(C.byref(r))
    assert rec.u.ctypes.data == a.ctypes.data
    to_child, go = os.pipe()
    pid = os.fork()
    if pid == 0:
        ok = 1
        try:
            os.read(to_child, 1)
            ok = 0 if np.array_equal(rec.u.ravel(), np.arange(80000.0)) else 2
            rec.u[:] = -1.0
            freed = len(fake.freed)
            del rec
            gc.collect()
            ok = ok or (0 if len(fake.freed) == freed and not _core._out else 3)
        finally:
            os._exit(ok)
    rec.u[0, 0] = 5.0  # the parent goes on: the child must not see it
    os.write(go, b"x")
    _, status = os.waitpid(pid, 0)
    assert os.waitstatus_to_exitcode(status) == 0
    assert rec.u[0, 0] == 5.0 and rec.u[-1, -1] == 79999.0
    del rec, a
