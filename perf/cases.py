"""The calls whose speed this library answers for, with their inputs and their 64-bit results.

Every case is a call of the C ABI as a program makes it: the handle, the matrices and (where the
entry point takes them) the inverted diagonal blocks or the batch descriptors stay in device
memory, the right-hand sides of a pass are copied to the buffer that the solve overwrites, and
the solution is what comes back.  Matrices are column-major with the leading dimension ``ld``,
held as ``(columns, ld)`` tensors.  A's other triangle holds other numbers, as it does after an
LU factorisation.
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

import rocblas_b200 as rb
from rocblas_b200 import devmem as dm
from rocblas_b200 import workloads

DTYPES = {"s": torch.float32, "d": torch.float64, "c": torch.complex64, "z": torch.complex128}
BYTES = {"s": 4, "d": 8, "c": 8, "z": 16}
WIDE = {"s": torch.float64, "d": torch.float64, "c": torch.complex128, "z": torch.complex128}
NP = {"s": np.float32, "d": np.float64, "c": np.complex64, "z": np.complex128}

# one descriptor of the variable-size batch (rocblas_b200_trsm_problem)
DESCRIPTOR = np.dtype([("A", "<u8"), ("B", "<u8"), ("m", "<i4"), ("n", "<i4"), ("lda", "<i4"), ("ldb", "<i4"),
                       ("side", "<i4"), ("uplo", "<i4"), ("trans", "<i4"), ("diag", "<i4")])


def _trsm(name, kind, dtype, combo, m, n, pad=0, **more):
    side, uplo, trans, diag = combo
    return {"name": name, "kind": kind, "dtype": dtype, "side": side, "uplo": uplo, "trans": trans, "diag": diag,
            "m": m, "n": n, "pad": pad, **more}


def listed():
    return [
        # the smallest calls: one small triangle, bound by the launch and one block's substitution
        _trsm("dtrsm 96x24", "trsm", "d", "RUNN", 24, 96),
        # an ordinary small solve (one panel of a blocked factorisation)
        _trsm("dtrsm 512x256", "trsm", "d", "LLNN", 512, 256),
        # a tall triangle and few right-hand sides, transposed: the second half of an LU or
        # Cholesky solve
        _trsm("dtrsm 8192x512", "trsm", "d", "LUTN", 8192, 512),
        # the large square solve from the right with a unit triangle: the trailing panel of an LU
        _trsm("dtrsm 8192x8192", "trsm", "d", "RLNU", 8192, 8192),
        # the large square solve in single precision
        _trsm("strsm 8192x8192", "trsm", "s", "LLNN", 8192, 8192),
        # a small triangle and many right-hand sides in single precision: the block row of a
        # blocked factorisation
        _trsm("strsm 512x8192", "trsm", "s", "LUNN", 512, 8192),
        # a server's request: odd sizes and few right-hand sides against a matrix that stays
        # resident with its inverted diagonal blocks
        _trsm("dtrsm_ex 3001x77", "ex", "d", "LLNN", 3001, 77),
        # the precision form (solve and test) at the size it is made for
        {"name": "refined 16384x4096", "kind": "refined", "m": 16384, "n": 4096},
        # thousands of equal small systems
        _trsm("dtrsm 4096 of 128x32", "strided", "d", "LLNN", 128, 32, batch=4096),
        # thousands of uneven small systems in one call
        {"name": "vbatched 20000", "kind": "vbatched", "dtype": "d", "count": 20000, "max_m": 512, "max_n": 64},
        # one right-hand side
        {"name": "dtrsv 16384", "kind": "trsv", "dtype": "d", "uplo": "L", "trans": "N", "diag": "N", "n": 16384,
         "incx": 1, "pad": 0},
        # complex, conjugate-transposed
        _trsm("ztrsm 2048x1000", "trsm", "z", "LLCN", 2048, 1000),
    ]


def _log_uniform(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.49)))))))


def draw(rng):
    kind = rng.choice(["trsm", "trsm", "trsm", "trsm", "ex", "ex", "refined", "strided", "strided", "vbatched",
                       "trsv", "complex"])
    combo = rng.choice("LR") + rng.choice("LU") + rng.choice("NT") + rng.choice("NNU")
    pad = rng.choice([0, 0, 0, 1, 8, rng.randint(1, 100)])
    if kind in ("trsm", "ex"):
        least = 16 if kind == "trsm" else 200
        k, cols = _log_uniform(rng, least, 8192), _log_uniform(rng, 1, 8192)
        m, n = (k, cols) if combo[0] == "L" else (cols, k)
        case = _trsm("", kind, rng.choice("sd"), combo, m, n, pad)
    elif kind == "complex":
        k, cols = _log_uniform(rng, 32, 2048), _log_uniform(rng, 8, 2048)
        combo = combo[:2] + rng.choice("NTC") + combo[3]
        m, n = (k, cols) if combo[0] == "L" else (cols, k)
        case = _trsm("", "trsm", rng.choice("cz"), combo, m, n, pad)
    elif kind == "refined":
        return {"kind": kind, "m": _log_uniform(rng, 4096, 16384), "n": _log_uniform(rng, 512, 4096)}
    elif kind == "strided":
        k, cols = _log_uniform(rng, 8, 512), _log_uniform(rng, 1, 64)
        batch = min(_log_uniform(rng, 64, 4096), (1 << 27) // (k * k))
        m, n = (k, cols) if combo[0] == "L" else (cols, k)
        case = _trsm("", kind, rng.choice("sd"), combo, m, n, pad, batch=batch)
    elif kind == "vbatched":
        return {"kind": kind, "dtype": rng.choice("sd"), "count": _log_uniform(rng, 500, 20000), "max_m": 512,
                "max_n": 64}
    else:
        return {"kind": kind, "dtype": rng.choice("sd"), "uplo": combo[1], "trans": combo[2], "diag": combo[3],
                "n": _log_uniform(rng, 256, 32768), "incx": rng.choice([1, 1, 1, 3]), "pad": pad}
    del case["name"]
    return case


# ---- inputs ------------------------------------------------------------------------------------
def _uniform(shape, dtype, g):
    """Entries (real and imaginary parts) from U(-1, 1)."""
    if dtype.is_complex:
        real = torch.float32 if dtype == torch.complex64 else torch.float64
        return torch.view_as_complex(torch.rand(*shape, 2, generator=g, device="cuda", dtype=real).mul_(2).sub_(1))
    return torch.rand(*shape, generator=g, device="cuda", dtype=dtype).mul_(2).sub_(1)


def _triangle(k, ld, dtype, g, batch=None):
    """A well-conditioned triangular matrix: off-diagonal U(-1, 1) / k, diagonal 1 + U(0, 1)."""
    lead = () if batch is None else (batch,)
    A = _uniform(lead + (k, ld), dtype, g).div_(k)
    d = torch.rand(*lead, k, generator=g, device="cuda", dtype=torch.float64).add_(1)
    A.diagonal(dim1=-2, dim2=-1).copy_(d.to(dtype))
    return A


_handles = []


def _handle():
    """The program's one handle."""
    if not _handles:
        _handles.append(rb.Handle())
    return _handles[0]


def _scalar(dtype, value):
    a = np.array([value], dtype=NP[dtype])
    return a, ctypes.c_void_p(a.ctypes.data)


def _ptr(t):
    return ctypes.c_void_p(t.data_ptr())


def _codes(case):
    return rb.SIDE[case["side"]], rb.UPLO[case["uplo"]], rb.TRANS[case["trans"]], rb.DIAG[case["diag"]]


def _order(case):
    return case["m"] if case["side"] == "L" else case["n"]


def _system(case, seed):
    """(A, B, alpha) of one system or a uniform batch."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    dtype, batch = DTYPES[case["dtype"]], case.get("batch")
    k = _order(case)
    A = _triangle(k, k + case["pad"], dtype, g, batch)
    lead = () if batch is None else (batch,)
    B = _uniform(lead + (case["n"], case["m"] + case["pad"]), dtype, g)
    return A, B, (0.5 - 1.0j) if dtype.is_complex else 1.0


def _vector(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    dtype = DTYPES[case["dtype"]]
    return _triangle(case["n"], case["n"] + case["pad"], dtype, g), _uniform((case["n"] * case["incx"],), dtype, g)


def _refined_system(case, seed):
    return workloads.condition_band_lower_torch(case["m"], case["n"], 0, seed)


def _batch_sizes(case):
    """(m, n, k, left, lower) of the batch's systems; they belong to the case, not to the seed."""
    r = np.random.default_rng(case["count"])
    count = case["count"]
    m = np.minimum(np.exp(r.uniform(math.log(16), math.log(case["max_m"] + 1), count)).astype(np.int64), case["max_m"])
    n = r.integers(1, case["max_n"] + 1, count)
    left, lower = r.random(count) < 0.5, r.random(count) < 0.5
    return m, n, np.where(left, m, n), left, lower


def _batch(case, seed):
    """The systems' A and B back to back in two arrays."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    dtype = DTYPES[case["dtype"]]
    m, n, k, left, lower = _batch_sizes(case)
    a0, b0 = np.cumsum(k * k) - k * k, np.cumsum(m * n) - m * n
    A = _uniform((int((k * k).sum()),), dtype, g)
    kt = torch.from_numpy(k).cuda()
    at = torch.from_numpy(a0).cuda()
    A.div_(torch.repeat_interleave(kt, kt * kt))
    first = torch.cumsum(kt, 0) - kt
    i = torch.arange(int(k.sum()), device="cuda") - torch.repeat_interleave(first, kt)  # row of each diagonal entry
    diagonal = torch.rand(i.numel(), generator=g, device="cuda", dtype=torch.float64).add_(1).to(dtype)
    A[torch.repeat_interleave(at, kt) + i * (torch.repeat_interleave(kt, kt) + 1)] = diagonal
    return A, _uniform((int((m * n).sum()),), dtype, g), a0, b0


def prepare(case, seed):
    L, h, kind = rb.lib(), _handle(), case["kind"]
    if kind == "refined":
        A, B = _refined_system(case, seed)
        X = torch.empty_like(B)
        keep, alpha = _scalar("d", 1.0)
        opts = rb.RefineOptions(0, -1, 0, 1, 0.0)
        info = rb.RefineInfo()
        m, n = case["m"], case["n"]
        args = (h.value, rb.side_left, rb.fill_lower, rb.operation_none, rb.diagonal_non_unit, m, n, alpha, _ptr(A),
                m, _ptr(X), m, ctypes.cast(ctypes.byref(opts), ctypes.c_void_p),
                ctypes.cast(ctypes.byref(info), ctypes.c_void_p))
        return {"call": L.rocblas_b200_dtrsm_refined, "args": args, "B": B, "X": X, "keep": (A, keep, opts, info)}
    dtype = case["dtype"]
    if kind == "trsv":
        A, b = _vector(case, seed)
        x = torch.empty_like(b)
        args = (h.value, rb.UPLO[case["uplo"]], rb.TRANS[case["trans"]], rb.DIAG[case["diag"]], case["n"], _ptr(A),
                A.shape[-1], _ptr(x), case["incx"])
        return {"call": getattr(L, "rocblas_%strsv" % dtype), "args": args, "B": b, "X": x, "keep": A}
    if kind == "vbatched":
        A, B, a0, b0 = _batch(case, seed)
        X = torch.empty_like(B)
        m, n, k, left, lower = _batch_sizes(case)
        d = np.zeros(case["count"], dtype=DESCRIPTOR)
        d["A"], d["B"] = A.data_ptr() + a0 * BYTES[dtype], X.data_ptr() + b0 * BYTES[dtype]
        d["m"], d["n"], d["lda"], d["ldb"] = m, n, k, m
        d["side"] = np.where(left, rb.side_left, rb.side_right)
        d["uplo"] = np.where(lower, rb.fill_lower, rb.fill_upper)
        d["trans"], d["diag"] = rb.operation_none, rb.diagonal_non_unit
        desc = torch.from_numpy(d.view(np.uint8)).cuda()
        keep, alpha = _scalar(dtype, 1.0)
        args = (h.value, alpha, _ptr(desc), case["count"], case["max_m"], None)
        return {"call": getattr(L, "rocblas_b200_%strsm_vbatched" % dtype), "args": args, "B": B, "X": X,
                "keep": (A, desc, keep)}
    A, B, value = _system(case, seed)
    X = torch.empty_like(B)
    keep, alpha = _scalar(dtype, value)
    m, n, lda, ldb = case["m"], case["n"], A.shape[-1], B.shape[-1]
    args = (h.value, *_codes(case), m, n, alpha, _ptr(A), lda)
    if kind == "strided":
        args += (A.shape[-2] * lda, _ptr(X), ldb, n * ldb, case["batch"])
        call = getattr(L, "rocblas_%strsm_strided_batched" % dtype)
    elif kind == "ex":
        k = _order(case)
        invA = dm.build_invA(h, case["uplo"], case["diag"], A, lda, k)
        keep = (keep, invA)
        args += (_ptr(X), ldb, _ptr(invA), invA.numel(), rb.datatype_f32_r if dtype == "s" else rb.datatype_f64_r)
        call = L.rocblas_trsm_ex
    else:
        args += (_ptr(X), ldb)
        call = getattr(L, "rocblas_%strsm" % dtype)
    return {"call": call, "args": args, "B": B, "X": X, "keep": (A, keep)}


def run(state):
    """The right-hand sides into the buffer that the solve overwrites, and the solve."""
    state["X"].copy_(state["B"])
    rb.check("solve", state["call"](*state["args"]))
    return state["X"]


# ---- what a pass cannot do without ---------------------------------------------------------------
def work(case):
    """A's triangle and B read once, X written once; k * k * columns flops (complex: 4 times)."""
    kind = case["kind"]
    if kind == "vbatched":
        m, n, k, _, _ = _batch_sizes(case)
        return {"bytes": BYTES[case["dtype"]] * float((k * (k + 1) // 2 + 2 * m * n).sum()),
                "flops": float((m * n * k).sum())}
    if kind == "refined":
        m, n = case["m"], case["n"]
        return {"bytes": 8.0 * (m * (m + 1) // 2 + 2 * m * n), "flops": float(m) * m * n}
    if kind == "trsv":
        n = case["n"]
        return {"bytes": BYTES[case["dtype"]] * (n * (n + 1) // 2 + 2.0 * n), "flops": float(n) * n}
    m, n, k, batch = case["m"], case["n"], _order(case), case.get("batch", 1)
    each = 4.0 if case["dtype"] in "cz" else 1.0
    return {"bytes": BYTES[case["dtype"]] * batch * (k * (k + 1) // 2 + 2.0 * m * n),
            "flops": each * batch * m * n * k}


def tolerance(case):
    """About four times the error against 64-bit (FP64: another order's) results: up to 1.1e-7 in
    single precision; in double up to 4e-16, and 1.9e-15 for the precision form and for long
    single right-hand sides, whose sums of thousands of terms are rounded in another order."""
    if case["kind"] in ("refined", "trsv") and case.get("dtype") != "s":
        return {"rel": 1e-14}
    return {"rel": 5e-7 if case["dtype"] in ("s", "c") else 2e-15}


# ---- 64-bit results ------------------------------------------------------------------------------
def _solve(A, B, side, uplo, trans, diag, alpha):
    """op(A)^-1 alpha B or alpha B op(A)^-1 for matrices as written (rows, columns)."""
    upper = uplo == "U"
    if trans != "N":
        A, upper = A.mT, not upper
    if trans == "C":
        A = A.conj().resolve_conj()
    return torch.linalg.solve_triangular(A, alpha * B, upper=upper, left=side == "L", unitriangular=diag == "U")


def exact(case, seed):
    kind = case["kind"]
    if kind == "refined":
        A, B = _refined_system(case, seed)
        return _solve(A.mT, B.mT, "L", "L", "N", "N", 1.0).mT.contiguous()
    wide = WIDE[case["dtype"]]
    if kind == "trsv":
        A, b = _vector(case, seed)
        n = case["n"]
        out = b.to(wide)
        x = out.view(n, case["incx"])[:, :1]
        x.copy_(_solve(A[:, :n].mT.to(wide), x.clone(), "L", case["uplo"], case["trans"], case["diag"], 1.0))
        return out
    if kind == "vbatched":
        A, B, a0, b0 = _batch(case, seed)
        m, n, k, left, lower = (v.tolist() for v in _batch_sizes(case))
        A, out = A.to(wide), B.to(wide)
        for i, (p, q) in enumerate(zip(a0.tolist(), b0.tolist())):
            a = A[p : p + k[i] * k[i]].view(k[i], k[i]).mT
            x = out[q : q + m[i] * n[i]].view(n[i], m[i]).mT
            x.copy_(torch.linalg.solve_triangular(a, x.clone(), upper=not lower[i], left=left[i]))
        return out
    A, B, alpha = _system(case, seed)
    m, k = case["m"], _order(case)
    out = B.to(wide)
    x = out[..., :m].mT
    x.copy_(_solve(A[..., :k].mT.to(wide), x.clone(), *(case[w] for w in ("side", "uplo", "trans", "diag")), alpha))
    return out
