"""The streaming TRSV (trsv_stream.cuh) at the edges of its 128-row blocks, all combinations, both
element types, increments and leading dimensions, against the oracle; the flag solve in a workspace
that holds only its flags gives the same answer, also under capture; a wait that runs out is
reported."""
import ctypes
import itertools

import numpy as np
import pytest

torch = pytest.importorskip("torch")

import oracle  # noqa: E402
import rocblas_b200 as rb  # noqa: E402
from rocblas_b200 import devmem as dm  # noqa: E402

pytestmark = pytest.mark.gpu


def _trsv(h, dtype, uplo, trans, diag, n, A, lda, b, incx):
    L = rb.lib()
    fn = L.rocblas_dtrsv if dtype == np.float64 else L.rocblas_strsv
    dA = dm.to_device(A)
    x = torch.full((1 + (n - 1) * incx,), float("nan"), dtype=dA.dtype, device="cuda")
    x[::incx] = torch.from_numpy(b).cuda()
    assert fn(h.value, rb.UPLO[uplo], rb.TRANS[trans], rb.DIAG[diag], n, ctypes.c_void_p(dA.data_ptr()), lda,
              ctypes.c_void_p(x.data_ptr()), incx) == 0
    torch.cuda.synchronize()
    if incx > 1:
        gaps = x.clone()
        gaps[::incx] = float("nan")
        assert torch.isnan(gaps).all()
    return x[::incx].cpu().numpy()


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("n", [256, 257, 383, 384, 385, 1000])
def test_block_edges(n, dtype):
    with rb.Handle() as h, rb.Handle() as flags_only:
        assert rb.lib().rocblas_set_device_memory_size(flags_only.value, 64) == 0
        for i, (uplo, trans, diag) in enumerate(itertools.product("UL", "NT", "NU")):
            lda, incx = n + i % 3, 1 + i % 2
            A, B = oracle.nan_triangle_problem(i, "L", uplo, trans, diag, n, 1, lda, n, dtype)
            b = np.ascontiguousarray(B[:, 0])
            X = oracle.trsm("L", uplo, trans, diag, 1.0, A, B)[:, 0]
            tol = oracle.trsm_tolerance(dtype, n) * max(1.0, np.abs(X).max())
            for handle in (h, flags_only):
                out = _trsv(handle, dtype, uplo, trans, diag, n, A, lda, b, incx)
                assert np.abs(out - X).max() <= tol, (uplo, trans, diag)


@pytest.mark.parametrize("trans", "NT")
def test_more_blocks_than_ctas(trans):
    n = 20000  # 157 blocks
    g = torch.Generator(device="cuda").manual_seed(1)
    A = (torch.rand(n, n, generator=g, device="cuda", dtype=torch.float64) * 2 - 1) / n
    A.diagonal().copy_(1 + torch.rand(n, generator=g, device="cuda", dtype=torch.float64))
    b = torch.rand(n, generator=g, device="cuda", dtype=torch.float64)
    x = b.clone()
    with rb.Handle() as h:
        assert rb.lib().rocblas_dtrsv(h.value, rb.fill_lower, rb.TRANS[trans], rb.diagonal_non_unit, n,
                                      ctypes.c_void_p(A.data_ptr()), n, ctypes.c_void_p(x.data_ptr()), 1) == 0
        torch.cuda.synchronize()
    M = torch.tril(A.mT)  # the stored lower triangle, as written
    M = M if trans == "N" else M.mT
    # residual of a backward stable solve: n eps of |M| |x|
    assert ((M @ x - b).abs() <= 2.3e-16 * n * (M.abs() @ x.abs())).all()


def test_non_finite_entry_reaches_only_its_own_and_later_rows():
    n, row = 700, 300
    A, B = oracle.nan_triangle_problem(3, "L", "L", "N", "N", n, 1, n, n, np.float64)
    b = np.ascontiguousarray(B[:, 0])
    b[row] = np.inf
    with rb.Handle() as h:
        out = _trsv(h, np.float64, "L", "N", "N", n, A, n, b, 1)
    assert np.isfinite(out[:row]).all() and not np.isfinite(out[row:]).any()


@pytest.mark.parametrize("trans", "NT")
@pytest.mark.parametrize("what", ["nan", "inf", "zero", "overflow"])
@pytest.mark.parametrize("pos,before", [(20, 3), (50, 20), (300, 260), (383, 256), (500, 30)])
def test_rows_solved_before_a_bad_entry_of_a_stay_finite(pos, before, what, trans):
    """An infinity, a NaN or a zero pivot of A reaches the row that holds it and those solved after it
    (position = row for a lower triangle, from the end for its transpose); a pivot whose inverse row
    overflows leaves the others finite."""
    n = 700
    A, B = oracle.nan_triangle_problem(9, "L", "L", trans, "N", n, 1, n, n, np.float64)
    b = np.ascontiguousarray(B[:, 0])
    order = np.arange(n) if trans == "N" else np.arange(n)[::-1]
    r, c = order[pos], order[before]
    M = A if trans == "N" else A.T
    if what == "zero":
        M[r, r] = 0
    elif what == "overflow":
        M[r, r], M[r, c] = 1e-300, 1e10
    else:
        M[r, c] = float(what)
    with rb.Handle() as h:
        out = _trsv(h, np.float64, "L", trans, "N", n, A, n, b, 1)[order]
    assert np.isfinite(out[:pos]).all()
    sub = order[:pos]
    X = oracle.trsm("L", "L" if trans == "N" else "U", "N", "N", 1.0, np.asfortranarray(M[np.ix_(np.sort(sub), np.sort(sub))]),
                    np.asfortranarray(b[np.sort(sub), None]))[:, 0]
    X = X if trans == "N" else X[::-1]
    assert np.abs(out[:pos] - X).max() <= oracle.trsm_tolerance(np.float64, n) * max(1.0, np.abs(X).max())
    if what != "overflow":
        assert not np.isfinite(out[pos:]).any()


@pytest.mark.parametrize("trans", "NT")
@pytest.mark.parametrize("first_block", [1, 5])
def test_wait_that_runs_out_is_reported(first_block, trans):
    """The failure is made on the host: the claims start past the first blocks, whose x nothing then
    publishes, and the waits are short.  The call returns, error 5 is reported once, and the handle
    solves afterwards."""
    n = 2048
    A, B = oracle.nan_triangle_problem(2, "L", "L", trans, "N", n, 1, n, n, np.float64)
    b = np.ascontiguousarray(B[:, 0])
    L, code = rb.lib(), ctypes.c_int(-1)

    def error(h):
        assert L.rocblas_b200_get_device_error(h.value, ctypes.byref(code)) == 0
        return code.value

    keys = {b"wait_cycles_log2": 16, b"chain_first_item": first_block}
    with rb.Handle() as h:
        assert error(h) == 0
        old = {}
        try:
            for key, value in keys.items():
                assert L.rocblas_b200_get_tuning(key, ctypes.byref(code)) == 0
                old[key] = code.value
                assert L.rocblas_b200_set_tuning(key, value) == 0
            _trsv(h, np.float64, "L", trans, "N", n, A, n, b, 1)
        finally:
            for key, value in old.items():
                L.rocblas_b200_set_tuning(key, value)
        assert error(h) == 5 and error(h) == 0
        out = _trsv(h, np.float64, "L", trans, "N", n, A, n, b, 1)
        X = oracle.trsm("L", "L", trans, "N", 1.0, A, B)[:, 0]
        assert np.abs(out - X).max() <= oracle.trsm_tolerance(np.float64, n) * max(1.0, np.abs(X).max())
        assert error(h) == 0


def test_capture_with_a_workspace_of_flags():
    """Under capture the workspace does not grow: a handle whose workspace is that of a short solve
    captures a longer one as the flag solve."""
    small, n = 256, 2048
    A, B = oracle.nan_triangle_problem(4, "L", "L", "N", "N", n, 1, n, n, np.float64)
    X = oracle.trsm("L", "L", "N", "N", 1.0, A, B)[:, 0]
    s = torch.cuda.Stream()
    with rb.Handle() as h, torch.cuda.stream(s):
        h.set_stream(ctypes.c_void_p(s.cuda_stream))
        _trsv(h, np.float64, "L", "N", "N", small, np.asfortranarray(A[:small, :small]), small,
              np.ascontiguousarray(B[:small, 0]), 1)
        dA, x = dm.to_device(A), torch.from_numpy(np.ascontiguousarray(B[:, 0])).cuda()
        s.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=s):
            assert rb.lib().rocblas_dtrsv(h.value, rb.fill_lower, rb.operation_none, rb.diagonal_non_unit, n,
                                          ctypes.c_void_p(dA.data_ptr()), n, ctypes.c_void_p(x.data_ptr()), 1) == 0
        graph.replay()
        s.synchronize()
        out = x.cpu().numpy()
    assert np.abs(out - X).max() <= oracle.trsm_tolerance(np.float64, n) * max(1.0, np.abs(X).max())
