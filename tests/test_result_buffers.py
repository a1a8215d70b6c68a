"""Result buffers lent to numpy arrays (single_svdlib._core._take), against a
fake of the library: who frees what, and when."""
import ctypes as C
import gc

import numpy as np
import pytest

from single_svdlib import _abi, _core


class FakeLib:
    """svdb_rec_free on buffers of this process."""

    def __init__(self):
        self.live, self.freed = {}, []

    def buffer(self, values):
        a = np.array(values)
        self.live[a.ctypes.data] = a
        return a.ctypes.data

    def svdb_rec_free(self, ref):
        r = ref._obj
        for f in ("u", "s", "vt"):
            if getattr(r, f):
                addr = C.cast(getattr(r, f), C.c_void_p).value
                self.freed.append(addr)
                del self.live[addr]


@pytest.fixture()
def fake(monkeypatch):
    f = FakeLib()
    monkeypatch.setattr(_abi, "lib", lambda: f)
    monkeypatch.setattr(_core, "_lent", 0)
    return f


def record(f, m, d, n, f32=False):
    r = _abi.svdb_rec_f32() if f32 else _abi.svdb_rec()
    t, ct = (np.float32, C.c_float) if f32 else (np.float64, C.c_double)
    r.d, r.u_rows, r.u_cols, r.vt_rows, r.vt_cols = d, m, d, d, n
    for name, count in (("u", m * d), ("s", d), ("vt", d * n)):
        setattr(r, name, C.cast(f.buffer(np.arange(count, dtype=t)), C.POINTER(ct)))
    return r


@pytest.mark.parametrize("f32", [False, True])
def test_large_buffers_move_and_come_back_with_the_last_view(fake, f32):
    r = record(fake, 20000, 3, 10, f32)
    addr = C.cast(r.u, C.c_void_p).value
    rec = _core.rec_from_c(r)
    fake.svdb_rec_free(C.byref(r))  # as the callers do: s and vt, not the lent u
    assert len(fake.freed) == 2 and addr in fake.live and not r.u
    assert rec.u.ctypes.data == addr and rec.u.flags.writeable and rec.u.flags.c_contiguous
    assert rec.u.dtype == (np.float32 if f32 else np.float64) and rec.u[-1, -1] == 20000 * 3 - 1
    assert rec.vt.shape == (3, 10)
    view = rec.u[5:7]
    del rec
    gc.collect()
    assert addr in fake.live and view[0, 0] == 15
    del view
    gc.collect()
    assert addr not in fake.live and fake.freed[-1] == addr and _core._lent == 0


def test_limit_falls_back_to_copies(fake, monkeypatch):
    monkeypatch.setattr(_core, "_LENT_MAX", 20000 * 3 * 8)
    kept, lent = [], []
    for _ in range(3):
        r = record(fake, 20000, 3, 10)
        lent.append(C.cast(r.u, C.c_void_p).value)
        kept.append(_core.rec_from_c(r))
        fake.svdb_rec_free(C.byref(r))
    assert lent[0] in fake.live and lent[1] not in fake.live and lent[2] not in fake.live
    for k in kept:
        np.testing.assert_array_equal(k.u.ravel(), np.arange(60000.0))
    kept.clear()
    gc.collect()
    assert not fake.live and _core._lent == 0


def test_empty_results(fake):
    r = _abi.svdb_rec()
    r.d, r.u_rows, r.u_cols, r.vt_rows, r.vt_cols = 0, 5, 0, 0, 7
    rec = _core.rec_from_c(r)
    assert rec.u.shape == (5, 0) and rec.vt.shape == (0, 7) and rec.s.shape == (0,)
