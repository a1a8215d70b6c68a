"""Timing cases over the library's public entry points.

Each case is a plain dict: `kind` names the entry point, the rest its sizes
and options.  Matrices are generated on the GPU from the seed; a program that
uses the library keeps the matrix handle (and the batch) between calls, so
`prepare` makes them and `run` makes one call.
"""
import ctypes as C
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "single-svdlib_b200"))

from single_svdlib import _abi, legacy, randomized  # noqa: E402
from single_svdlib._core import BorrowedMatrix, CsrMatrix, MaskedCSRMatrix, check, options  # noqa: E402

DEV = "cuda"
SEED = 7  # the solvers' own seed; the inputs' seed is prepare()'s


# ------------------------------------------------------------------ cases --
def listed():
    return [
        # one product on a small operator: an outer Krylov loop in the caller's program
        {"name": "spmv_5000x2000", "kind": "spmv", "m": 5000, "n": 2000, "per_row": 20, "data": "uniform",
         "transposed": False, "precision": "f64"},
        # A X of the 100k x 30k count matrix, 60 columns: the product every randomized solve repeats
        {"name": "spmm_f64_100kx30k_l60", "kind": "spmm", "m": 100000, "n": 30000, "per_row": 600, "l": 60,
         "data": "counts", "groups": 50, "transposed": False, "precision": "f64"},
        # A^T X with an odd number of columns and odd sizes, FP32
        {"name": "spmm_mixed_t_50021x20011_l37", "kind": "spmm", "m": 50021, "n": 20011, "per_row": 200, "l": 37,
         "data": "counts", "groups": 20, "transposed": True, "precision": "mixed"},
        # gradient of a low-rank model at a sparsity pattern: FP32 SDDMM
        {"name": "sddmm_f32_50kx20k_r64", "kind": "sddmm", "m": 50000, "n": 20000, "per_row": 100, "l": 64,
         "data": "counts", "groups": 20, "precision": "mixed"},
        # the smallest solve, where launches and latency count, with its signs fixed on the host
        {"name": "randomized_f64_1000x250", "kind": "randomized", "m": 1000, "n": 250, "per_row": 25, "rank": 10,
         "over": 10, "q": 2, "norm": "QR", "center": False, "kept": 1.0, "data": "counts", "groups": 10,
         "precision": "f64", "host": True},
        # principal components of a count matrix on a subset of its columns (centred, odd sizes)
        {"name": "pca_f64_30011x8009", "kind": "randomized", "m": 30011, "n": 8009, "per_row": 150, "rank": 30,
         "over": 10, "q": 2, "norm": "QR", "center": True, "kept": 0.7, "data": "counts", "groups": 30,
         "precision": "f64", "host": False},
        # the large solve at T = f32: 100k x 30k, rank 50, three power iterations
        {"name": "randomized_f32_100kx30k", "kind": "randomized", "m": 100000, "n": 30000, "per_row": 600, "rank": 50,
         "over": 10, "q": 3, "norm": "QR", "center": False, "kept": 1.0, "data": "counts", "groups": 50,
         "precision": "f32", "host": False},
        # resampled column subsets of one matrix at the batch's default precision
        {"name": "batch_mixed_20000x6000", "kind": "batch", "m": 20000, "n": 6000, "per_row": 150, "count": 16,
         "smin": 500, "smax": 4000, "rank": 30, "over": 10, "q": 2, "data": "counts", "groups": 30,
         "precision": "mixed"},
        # the same in f64 with odd sizes
        {"name": "batch_f64_10007x3001", "kind": "batch", "m": 10007, "n": 3001, "per_row": 100, "count": 12,
         "smin": 300, "smax": 2500, "rank": 10, "over": 7, "q": 2, "data": "counts", "groups": 10,
         "precision": "f64"},
        # backward of the truncated SVD: dL/dvalues of 32 triplets
        {"name": "adjoint_f64_50kx20k_k32", "kind": "adjoint", "m": 50000, "n": 20000, "per_row": 100, "k": 32,
         "data": "counts", "groups": 32, "precision": "f64"},
        # LAS2 on the small matrix (k = 10): latency of the Lanczos step
        {"name": "las2_5000x2000_k10", "kind": "las2", "m": 5000, "n": 2000, "per_row": 20, "k": 10,
         "data": "uniform"},
        # LAS2 on a large matrix with Zipf row lengths: sparse products
        {"name": "las2_200kx40k_k10", "kind": "las2", "m": 200000, "n": 40000, "per_row": 200, "k": 10,
         "data": "zipf"},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["spmv", "spmm", "spmm", "sddmm", "randomized", "randomized", "randomized", "batch", "batch",
                       "adjoint", "las2"])
    groups = rng.randint(8, 40)
    if kind == "spmv":
        per_row = _log(rng, 8, 200)
        m = _log(rng, 2000, min(400000, 40_000_000 // per_row))
        return {"kind": kind, "m": m, "n": max(per_row * 4, _log(rng, m // 10 + 64, m)), "per_row": per_row,
                "data": rng.choice(["uniform", "zipf" if per_row > 50 else "uniform"]),
                "transposed": rng.random() < 0.5, "precision": rng.choice(["f64", "mixed"])}
    if kind in ("spmm", "sddmm"):
        per_row = _log(rng, 20, 400)
        m = _log(rng, 2000, min(100000, 30_000_000 // per_row))
        c = {"kind": kind, "m": m, "n": max(per_row * 4, 64, _log(rng, m // 5 + 64, m)), "per_row": per_row,
             "l": rng.choice([rng.randint(1, 128), 4 * rng.randint(2, 16), 4 * rng.randint(2, 32)]),
             "data": "counts", "groups": groups, "precision": rng.choice(["f64", "mixed"])}
        if kind == "spmm":
            c["transposed"] = rng.random() < 0.5
        return c
    if kind == "randomized":
        per_row = _log(rng, 20, 300)
        m = _log(rng, 800, min(100000, 15_000_000 // per_row))
        rank = min(_log(rng, 5, 100), groups)
        return {"kind": kind, "m": m, "n": max(per_row * 4, 256, _log(rng, m // 5 + 64, m)), "per_row": per_row,
                "rank": rank, "over": rng.randint(5, 20), "q": rng.randint(1, 3),
                "norm": rng.choice(["QR", "QR", "LU"]), "center": rng.random() < 0.3,
                "kept": rng.choice([1.0, 0.6]), "data": "counts", "groups": groups,
                "precision": rng.choice(["f64", "f64", "f32"]), "host": m < 4000}
    if kind == "batch":
        per_row = _log(rng, 30, 150)
        m = _log(rng, 2000, 20000)
        n = max(per_row * 6, 800, m // rng.randint(2, 5))
        return {"kind": kind, "m": m, "n": n, "per_row": per_row, "count": rng.randint(4, 20), "smin": n // 4,
                "smax": 3 * n // 4, "rank": rng.randint(5, 30), "over": rng.randint(5, 20), "q": rng.randint(1, 2),
                "data": "counts", "groups": 40, "precision": rng.choice(["f64", "mixed"])}
    if kind == "adjoint":
        per_row = _log(rng, 30, 120)
        m = _log(rng, 2000, 40000)
        k = rng.randint(4, 32)
        return {"kind": kind, "m": m, "n": max(per_row * 4, 512, _log(rng, m // 4 + 64, m)), "per_row": per_row,
                "k": k, "data": "counts", "groups": k, "precision": "f64"}
    m = _log(rng, 2000, 150000)
    data = rng.choice(["uniform", "zipf"]) if m > 20000 else "uniform"
    return {"kind": kind, "m": m, "n": max(512, _log(rng, m // 5, m)), "per_row": 200 if data == "zipf" else 20,
            "k": rng.randint(4, 20), "data": data}


# --------------------------------------------------------------- matrices --
def _matrix(c, seed):
    """(indptr int64, cols int32, vals f64) of the case's matrix, on the GPU.

    The SDDMM and the adjoint write one value per stored entry: their pattern
    is the same for every seed, so that the outputs have one length."""
    g = torch.Generator(device=DEV)
    g.manual_seed(11 if c["kind"] in ("sddmm", "adjoint") else seed)
    m, n, per = c["m"], c["n"], c["per_row"]

    def rand(k):
        return torch.rand(k, dtype=torch.float64, device=DEV, generator=g)

    lam = torch.randn(n, dtype=torch.float64, device=DEV, generator=g).square()  # Gamma(1/2, scale 2)
    if c["data"] == "counts":  # log-normal row lengths, Gamma column rates, row groups with a column program each
        k = torch.randn(m, dtype=torch.float64, device=DEV, generator=g).mul(0.5).add(math.log(per)).exp()
    elif c["data"] == "zipf":  # row lengths Zipf(1.85) on [per/10, 100 per]
        ks = torch.arange(max(per // 10, 1), min(100 * per, n // 2) + 1, dtype=torch.float64, device=DEV)
        cdf = torch.cumsum(ks ** -1.85, 0)
        k = ks[torch.searchsorted(cdf / cdf[-1], rand(m)).clamp_(max=len(ks) - 1)]
    else:  # Poisson row lengths, uniform columns
        k = torch.poisson(torch.full((m,), float(per), dtype=torch.float64, device=DEV), generator=g)
    k = k.round().clamp_(0 if c["data"] == "uniform" else 1, n).long()
    rows = torch.repeat_interleave(torch.arange(m, device=DEV), k)
    u = rand(rows.numel())
    if c["data"] == "counts":
        cdf = torch.cumsum(lam, 0)
        cols = torch.searchsorted(cdf / cdf[-1], u).clamp_(max=n - 1)
        w = 0.96 ** torch.arange(c["groups"], dtype=torch.float64, device=DEV)
        gid = torch.searchsorted(torch.cumsum(w, 0) / w.sum(), rand(m)).clamp_(max=c["groups"] - 1)
        width = max(8, n // (2 * c["groups"]))
        perm = torch.randperm(n, device=DEV, generator=g)
        prog = perm[(gid[rows] * width + (u * width).long()) % n]
        cols = torch.where(rand(rows.numel()) < 0.5, prog, cols)
        del prog
    else:
        cols = (u * n).long().clamp_(max=n - 1)
    keys = torch.unique_consecutive(torch.sort(rows * n + cols).values)
    del rows, cols, u
    rows = keys // n
    cols = keys - rows * n
    indptr = torch.zeros(m + 1, dtype=torch.int64, device=DEV)
    indptr[1:] = torch.cumsum(torch.bincount(rows, minlength=m), 0)
    g.manual_seed(seed + 500_009)
    if c["data"] == "counts":
        vals = torch.log1p(torch.poisson(lam[cols], generator=g) + 1.0)
    elif c["data"] == "uniform":
        vals = rand(cols.numel())
    else:  # N(0, 1) and a planted signal
        r = 12
        uu = torch.randn(m, r, dtype=torch.float64, device=DEV, generator=g)
        vv = torch.randn(n, r, dtype=torch.float64, device=DEV, generator=g)
        s = torch.logspace(0.8, 0, r, dtype=torch.float64, device=DEV)
        vals = torch.randn(cols.numel(), dtype=torch.float64, device=DEV, generator=g)
        for a in range(0, cols.numel(), 1 << 23):
            b = a + (1 << 23)
            vals[a:b] += (uu[rows[a:b]] * vv[cols[a:b]] * s).sum(1)
    return indptr, cols.to(torch.int32), vals


class _DeviceCsr(BorrowedMatrix):
    """A CSR handle made from device arrays, destroyed with this object."""

    def __init__(self, m, n, indptr, cols, vals):
        h = C.c_void_p()
        torch.cuda.synchronize()
        check(_abi.lib().svdb_matrix_create_csr_device(m, n, vals.numel(), indptr.data_ptr(), cols.data_ptr(),
                                                       vals.data_ptr(), C.byref(h)))
        super().__init__(h)

    def close(self):
        if self._h:
            _abi.lib().svdb_matrix_destroy(self._h)
            self._h = None


def _handle(c, arrays):
    indptr, cols, vals = arrays
    if c.get("precision") == "f32":  # a T = f32 matrix
        return CsrMatrix(c["m"], c["n"], indptr.cpu().numpy(), cols.cpu().numpy(), vals.float().cpu().numpy())
    return _DeviceCsr(c["m"], c["n"], indptr, cols, vals)


def _kept(c, seed):
    """Column mask of the case, None for all columns."""
    if c.get("kept", 1.0) >= 1.0:
        return None
    mask = np.zeros(c["n"], dtype=bool)
    mask[np.random.default_rng(seed).permutation(c["n"])[:int(c["n"] * c["kept"])]] = True
    return mask


def _subsets(c, seed):
    sizes = np.random.default_rng(11).integers(c["smin"], c["smax"] + 1, c["count"])
    r = np.random.default_rng(seed)
    return [r.choice(c["n"], int(k), replace=False) for k in sizes]


def _randn(seed, *shape, dtype=torch.float64):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed + 1_000_003)
    return torch.randn(*shape, dtype=dtype, device=DEV, generator=g)


def _spmm64(arrays, m, n):
    """(X -> A X, Y -> A^T Y) in 64 bits."""
    indptr, cols, vals = arrays
    a = torch.sparse_csr_tensor(indptr, cols.long(), vals, (m, n))
    rows = torch.repeat_interleave(torch.arange(m, device=DEV), indptr[1:] - indptr[:-1])
    order = torch.sort(cols.long() * m + rows).indices
    tp = torch.zeros(n + 1, dtype=torch.int64, device=DEV)
    tp[1:] = torch.cumsum(torch.bincount(cols, minlength=n), 0)
    at = torch.sparse_csr_tensor(tp, rows[order], vals[order], (n, m))
    return (lambda x: a @ x), (lambda y: at @ y)


def _triplets(arrays, m, n, k, seed):
    """The k leading singular triplets by subspace iteration in 64 bits."""
    ax, aty = _spmm64(arrays, m, n)
    q = torch.linalg.qr(aty(ax(_randn(seed, n, k + 16)))).Q
    for _ in range(12):
        q = torch.linalg.qr(aty(ax(q))).Q
    y, r = torch.linalg.qr(ax(q))
    ur, s, vh = torch.linalg.svd(r)
    return (y @ ur[:, :k]).contiguous(), s[:k].contiguous(), (q @ vh[:k].T).contiguous()


# ---------------------------------------------------------------- prepare --
def prepare(case, seed):
    c = dict(case)
    arrays = _matrix(c, seed)
    m, n, nnz = c["m"], c["n"], arrays[2].numel()
    st = {"c": c, "a": _handle(c, arrays), "stream": torch.cuda.Stream()}
    f32 = c.get("precision") == "mixed"
    dt = torch.float32 if f32 else torch.float64
    if c["kind"] == "spmv":
        rin, rout = (m, n) if c["transposed"] else (n, m)
        st["x"], st["y"] = _randn(seed, rin), torch.empty(rout, dtype=torch.float64, device=DEV)
    elif c["kind"] == "spmm":
        rin, rout = (m, n) if c["transposed"] else (n, m)
        st["x"] = _randn(seed, rin, c["l"], dtype=dt)
        st["y"] = torch.empty(rout, c["l"], dtype=dt, device=DEV)
    elif c["kind"] == "sddmm":
        st["x"], st["z"] = _randn(seed, m, c["l"], dtype=dt), _randn(seed + 1, n, c["l"], dtype=dt)
        st["y"] = torch.empty(nnz, dtype=dt, device=DEV)
    elif c["kind"] == "randomized":
        mask = _kept(c, seed)
        if mask is not None:
            st["a"] = MaskedCSRMatrix(st["a"], mask)
            st["a"].dtype = np.float32 if c["precision"] == "f32" else np.float64
    elif c["kind"] == "batch":
        st["b"] = randomized.RandomizedBatch(st["a"], _subsets(c, seed), c["rank"], c["over"], c["q"], seed=SEED,
                                             precision=c["precision"])
    elif c["kind"] == "adjoint":
        st["u"], st["s"], st["v"] = _triplets(arrays, m, n, c["k"], seed)
        st["gu"], st["gs"], st["gv"] = (_randn(seed + 2, m, c["k"]), _randn(seed + 3, c["k"]),
                                        _randn(seed + 4, n, c["k"]))
        st["y"] = torch.empty(nnz, dtype=torch.float64, device=DEV)
        o = _abi.svdb_adjoint_options()
        _abi.lib().svdb_adjoint_options_default(C.byref(o))
        o.precision = _abi.PRECISION[c["precision"]]
        o.inputs_on_device = 1
        st["o"] = o
    torch.cuda.synchronize()
    return st


class _View:
    """A library-owned device buffer as torch sees it."""

    def __init__(self, ptr, shape, typestr):
        self.__cuda_array_interface__ = {"data": (C.cast(ptr, C.c_void_p).value, False), "shape": shape,
                                         "typestr": typestr, "version": 3}


def _tensors(r, typestr):
    """u, s, vt of a device-resident record, copied into tensors."""
    shapes = ((r.u, (int(r.u_rows), int(r.u_cols))), (r.s, (int(r.d),)), (r.vt, (int(r.vt_rows), int(r.vt_cols))))
    return tuple(torch.as_tensor(_View(p, s, typestr), device=DEV).clone() for p, s in shapes)


def _flip(u, vt):
    """The sign convention of svd_flip on float32 tensors."""
    sign = torch.where(u.gather(0, u.abs().argmax(0, keepdim=True)) < 0, -1.0, 1.0).to(u.dtype)
    return u * sign, vt * sign.T


# -------------------------------------------------------------------- run --
def run(st):
    c, L, s = st["c"], _abi.lib(), st["stream"].cuda_stream
    kind = c["kind"]
    prec = _abi.PRECISION["mixed" if c.get("precision") == "mixed" else "f64"]
    h = st["a"].handle
    if kind == "spmv":
        check(L.svdb_opa_device(h, st["x"].data_ptr(), st["y"].data_ptr(), int(c["transposed"]), prec, s))
        return st["y"]
    if kind == "spmm":
        check(L.svdb_multiply_with_dense_device(h, st["x"].data_ptr(), c["l"], st["y"].data_ptr(),
                                                int(c["transposed"]), prec, s))
        return st["y"]
    if kind == "sddmm":
        check(L.svdb_sddmm_device(h, st["x"].data_ptr(), st["z"].data_ptr(), c["l"], st["y"].data_ptr(), prec, s))
        return st["y"]
    if kind == "batch":
        return [(r.u, r.s, r.vt) for r in st["b"].run()]
    if kind == "las2":
        r = legacy.svdLAS2(st["a"], c["k"], 0, (-1e-30, 1e-30), 1e-6, 42)
        return r.ut, r.s, r.vt
    if kind == "adjoint":
        check(L.svdb_svd_adjoint(h, c["k"], *(st[x].data_ptr() for x in ("u", "s", "v", "gu", "gs", "gv")),
                                 C.byref(st["o"]), st["y"].data_ptr()))
        return st["y"]
    if c["host"]:
        norm = randomized.PowerIterationNormalizer(c["norm"])
        r = randomized.randomized_svd(st["a"], c["rank"], c["over"], c["q"], norm, c["center"], SEED)
        if c["precision"] == "f32":
            u, vt = _flip(torch.from_numpy(r.u), torch.from_numpy(r.vt))
            return u, r.s, vt
        u, vt = randomized.svd_flip(r.u, r.vt)
        return u, r.s, vt
    o = options(result_on_device=True)
    f32 = c["precision"] == "f32"
    r = _abi.svdb_rec_f32() if f32 else _abi.svdb_rec()
    check((L.svdb_randomized_svd_f32 if f32 else L.svdb_randomized_svd)(
        h, c["rank"], c["over"], c["q"], _abi.NORMALIZER[c["norm"]], int(c["center"]), 1, SEED, 0, C.byref(o),
        C.byref(r)))
    if f32:
        u, sv, vt = _tensors(r, "<f4")
        L.svdb_rec_f32_free(C.byref(r))
        u, vt = _flip(u, vt)
        return u, sv, vt
    check(L.svdb_svd_flip(r.u, r.u_rows, r.u_cols, r.vt, r.vt_rows, r.vt_cols, 1, 1))
    out = _tensors(r, "<f8")
    L.svdb_rec_free(C.byref(r))
    return out


# ------------------------------------------------------------------- work --
def work(case):
    """Bytes: the matrix, the operands and the results once.  Operations: the products' and the dense steps'."""
    c = case
    m, n = c["m"], c["n"]
    nnz = m * c["per_row"] * (0.85 if c["data"] == "counts" else 1.0)
    vs = 4 if c.get("precision") in ("mixed", "f32") else 8
    kind = c["kind"]
    if kind == "spmv":
        return {"bytes": nnz * (vs + 4) + 8 * (m + n), "flops": 2 * nnz}
    if kind == "spmm":
        return {"bytes": nnz * (vs + 4) + vs * c["l"] * (m + n), "flops": 2 * nnz * c["l"]}
    if kind == "sddmm":
        return {"bytes": nnz * (vs + 4) + vs * c["l"] * (m + n), "flops": 2 * nnz * c["l"]}
    if kind == "las2":  # at least 2 k steps of two products each
        return {"bytes": nnz * 12 + 8 * c["k"] * (m + n), "flops": 4 * nnz * 2 * c["k"]}
    if kind == "adjoint":  # two products per solver step, about 20 steps
        return {"bytes": nnz * 20 + 32 * c["k"] * (m + n), "flops": 20 * 4 * nnz * c["k"]}
    l = c["rank"] + c["over"]
    passes = 2 * c["q"] + 2

    def solve(nz, cols):
        return 2 * nz * l * passes + (c["q"] + 1) * 4 * (m + cols) * l * l

    if kind == "batch":
        cols = (c["smin"] + c["smax"]) / 2
        out = 8 * c["rank"] * (m + cols) * c["count"]
        return {"bytes": nnz * 8 + out, "flops": c["count"] * solve(nnz * cols / n, cols)}
    cols = n * c["kept"]
    return {"bytes": nnz * c["kept"] * (vs + 4) + vs * c["rank"] * (m + cols),
            "flops": solve(nnz * c["kept"], cols)}


# ------------------------------------------------------------------ exact --
def _omega(n, l, f32):
    """The library's Omega stream for SEED: splitmix64 of (seed, index), Box-Muller."""
    def i64(x):
        return x - (1 << 64) if x >= 1 << 63 else x

    def shr(x, k):
        return (x >> k) & ((1 << (64 - k)) - 1)

    def mix(x):
        x = x + i64(0x9E3779B97F4A7C15)
        x = (x ^ shr(x, 30)) * i64(0xBF58476D1CE4E5B9)
        x = (x ^ shr(x, 27)) * i64(0x94D049BB133111EB)
        return x ^ shr(x, 31)

    key = mix(torch.tensor(SEED ^ 0x5DEECE66D, dtype=torch.int64, device=DEV))
    i = torch.arange(n * l, dtype=torch.int64, device=DEV)
    a, b = mix(key + 2 * i), mix(key + 2 * i + 1)
    u1 = (shr(a, 11).double() + 0.5) / 9007199254740992.0
    u2 = shr(b, 11).double() / 9007199254740992.0
    w = (torch.sqrt(-2.0 * torch.log(u1)) * torch.cos(2.0 * math.pi * u2)).reshape(n, l)
    return w.float().double() if f32 else w


def _randomized64(arrays, m, n, c, f32=False):
    """randomized_svd in 64 bits with the signs of svd_flip."""
    ax, aty = _spmm64(arrays, m, n)
    rank = min(c["rank"], m, n)
    l = rank + c["over"]
    if c.get("center"):
        mu = aty(torch.ones(m, 1, dtype=torch.float64, device=DEV)) / m
        fwd, bwd = (lambda x: ax(x) - mu.T @ x), (lambda y: aty(y) - mu * y.sum(0))
    else:
        fwd, bwd = ax, aty

    def normalise(x):
        if c.get("norm", "QR") == "QR":
            return torch.linalg.qr(x).Q
        if c["norm"] == "LU":
            nr = x.norm(dim=0)
            return x / torch.where(nr > 1e-10, nr, torch.ones_like(nr))
        return x

    y = fwd(_omega(n, l, f32))
    for _ in range(c["q"]):
        y = normalise(fwd(normalise(bwd(y))))
    q = torch.linalg.qr(y).Q
    qb, r = torch.linalg.qr(bwd(q))
    ur, s, vh = torch.linalg.svd(r.T)
    u, vt = (q @ ur)[:, :rank], (vh @ qb.T)[:rank]
    u, vt = _flip(u, vt)
    return u, s[:rank], vt


def _columns(arrays, keep, m):
    """The arrays of A[:, keep] (keep: ascending column ids)."""
    indptr, cols, vals = arrays
    n = int(keep.max()) + 1
    o2m = torch.full((max(n, int(cols.max()) + 1),), -1, dtype=torch.int64, device=DEV)
    o2m[keep] = torch.arange(len(keep), device=DEV)
    rows = torch.repeat_interleave(torch.arange(m, device=DEV), indptr[1:] - indptr[:-1])
    new = o2m[cols.long()]
    ok = new >= 0
    ip = torch.zeros(m + 1, dtype=torch.int64, device=DEV)
    ip[1:] = torch.cumsum(torch.bincount(rows[ok], minlength=m), 0)
    return ip, new[ok].to(torch.int32), vals[ok]


def _adjoint64(arrays, c, seed):
    m, n, k = c["m"], c["n"], c["k"]
    u, s, v = _triplets(arrays, m, n, k, seed)
    gu, gs, gv = _randn(seed + 2, m, k), _randn(seed + 3, k), _randn(seed + 4, n, k)
    ax, aty = _spmm64(arrays, m, n)
    fwd = lambda x: ax(x) - u @ (s[:, None] * (v.T @ x))  # noqa: E731
    bwd = lambda y: aty(y) - v @ (s[:, None] * (u.T @ y))  # noqa: E731
    a, b = gu - u @ (u.T @ gu), gv - v @ (v.T @ gv)
    rhs = b * s + (lambda z: z - v @ (v.T @ z))(aty(a))
    x, r = torch.zeros_like(rhs), rhs.clone()
    p, rr = r.clone(), (r * r).sum(0)
    rr0 = rr.clone()
    for _ in range(400):
        w = p * s * s - bwd(fwd(p))
        live = rr > 1e-29 * rr0
        al = torch.where(live, rr / (p * w).sum(0), torch.zeros_like(rr))
        x += p * al
        r -= w * al
        r -= v @ (v.T @ r)
        new = (r * r).sum(0)
        p = r + p * torch.where(live, new / rr, torch.zeros_like(rr))
        rr = new
        if not bool((rr > 1e-28 * rr0).any()):
            break
    t = fwd(x)
    gamma = (a + t - u @ (u.T @ t)) / s
    ju, jv = u.T @ gu, v.T @ gv
    f = 1.0 / (s[None, :] ** 2 - s[:, None] ** 2 + torch.eye(k, dtype=torch.float64, device=DEV))
    f.fill_diagonal_(0.0)
    mm = torch.diag(gs) + f * (ju - ju.T) * s[None, :] + s[:, None] * f * (jv - jv.T)
    left, right = torch.cat([u @ mm + gamma, u], 1), torch.cat([v, x], 1)
    return _dots(arrays, left, right)


def _dots(arrays, left, right):
    indptr, cols, _ = arrays
    rows = torch.repeat_interleave(torch.arange(left.shape[0], device=DEV), indptr[1:] - indptr[:-1])
    out = torch.empty(cols.numel(), dtype=torch.float64, device=DEV)
    for a in range(0, out.numel(), 1 << 21):
        b = a + (1 << 21)
        out[a:b] = (left[rows[a:b]] * right[cols[a:b].long()]).sum(1)
    return out


def exact(case, seed):
    c = dict(case)
    m, n, kind = c["m"], c["n"], c["kind"]
    arrays = _matrix(c, seed)
    f32 = c.get("precision") == "mixed"
    dt = torch.float32 if f32 else torch.float64
    if kind in ("spmv", "spmm"):
        rin = m if c["transposed"] else n
        x = _randn(seed, rin)[:, None] if kind == "spmv" else _randn(seed, rin, c["l"], dtype=dt).double()
        y = _spmm64(arrays, m, n)[1 if c["transposed"] else 0](x)
        return y[:, 0] if kind == "spmv" else y
    if kind == "sddmm":
        return _dots(arrays, _randn(seed, m, c["l"], dtype=dt).double(), _randn(seed + 1, n, c["l"], dtype=dt).double())
    if kind == "randomized":
        if c["precision"] == "f32":
            arrays = arrays[:2] + (arrays[2].float().double(),)
        mask = _kept(c, seed)
        if mask is not None:
            arrays = _columns(arrays, torch.from_numpy(np.nonzero(mask)[0]).to(DEV), m)
            n = int(mask.sum())
        return _randomized64(arrays, m, n, c, c["precision"] == "f32")
    if kind == "batch":  # u and vt carry the solver's own signs
        out = []
        for cols in _subsets(c, seed):
            keep = torch.from_numpy(np.sort(cols)).to(DEV)
            out.append((None, _randomized64(_columns(arrays, keep, m), m, len(keep), c)[1], None))
        return out
    if kind == "adjoint":
        return _adjoint64(arrays, c, seed)
    return None, _triplets(arrays, m, n, c["k"], seed)[1] if c["data"] == "zipf" else \
        _dense_sigma(arrays, m, n, c["k"]), None  # las2: u and vt carry the solver's own signs


def _dense_sigma(arrays, m, n, k):
    """Singular values of a small matrix from its dense Gram matrix's side, by a dense SVD."""
    if m * n > 40_000_000:
        return None
    indptr, cols, vals = arrays
    return torch.linalg.svdvals(torch.sparse_csr_tensor(indptr, cols.long(), vals, (m, n)).to_dense())[:k]
