"""The chain solve (trsm_chain.cuh) at every strip width and at ragged strips, blocks and leading
dimensions, forward and backward, both element types; the workspace does
not depend on the width; and the inverse-block kernel (trtri_block.cuh) at its tile edges."""
import ctypes
import itertools

import numpy as np
import pytest

torch = pytest.importorskip("torch")

import oracle  # noqa: E402
import rocblas_b200 as rb  # noqa: E402
from rocblas_b200 import devmem as dm  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.fixture()
def width():
    L, old = rb.lib(), ctypes.c_int(-1)
    assert L.rocblas_b200_get_tuning(b"chain_w", ctypes.byref(old)) == 0
    yield lambda w: L.rocblas_b200_set_tuning(b"chain_w", w)
    L.rocblas_b200_set_tuning(b"chain_w", old.value)


def _solve(h, side, uplo, trans, diag, m, n, A, B):
    dA, dB = dm.to_device(A), dm.to_device(B)
    dm.trsm(h, side, uplo, trans, diag, m, n, 1.25, dA, A.shape[0], dB, B.shape[0])
    torch.cuda.synchronize()
    return dm.to_host(dB)


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("w", [8, 16, 32, 64])
def test_widths(width, w, dtype):
    assert width(w) == 0
    with rb.Handle() as h:
        for i, (side, uplo, trans, diag) in enumerate(itertools.product("LR", "UL", "NT", "NU")):
            k, cols = [(129, 1), (257, w), (384, w + 1), (513, 2 * w - 1), (640, 9)][i % 5]
            m, n = (k, cols) if side == "L" else (cols, k)
            A, B = oracle.nan_triangle_problem(i, side, uplo, trans, diag, m, n, k + i % 3, m + i % 2, dtype)
            out = _solve(h, side, uplo, trans, diag, m, n, A, B)
            X = oracle.trsm(side, uplo, trans, diag, 1.25, A, np.asfortranarray(B[:m]))
            assert oracle.matrix_norm_1(X, out[:m]) <= oracle.trsm_tolerance(dtype, max(m, n)), (side, uplo, trans, diag)
            assert np.isnan(out[m:]).all()
        code = ctypes.c_int(-1)
        assert rb.lib().rocblas_b200_get_device_error(h.value, ctypes.byref(code)) == 0 and code.value == 0


@pytest.mark.parametrize("k,cols", [(1000, 48), (200, 300), (140, 8)])
def test_workspace_does_not_depend_on_the_width(width, k, cols):
    """The strips' counts share the space of one word per block and 64-column strip, as words or
    (few blocks, narrow strips) as bytes; a fixed workspace of the queried size is enough."""
    L = rb.lib()

    def query(h, w):
        assert width(w) == 0
        size, a = ctypes.c_size_t(0), ctypes.c_double(1.0)
        assert L.rocblas_start_device_memory_size_query(h.value) == 0
        L.rocblas_dtrsm(h.value, rb.side_left, rb.fill_lower, rb.operation_none, rb.diagonal_non_unit, k, cols,
                        ctypes.cast(ctypes.byref(a), ctypes.c_void_p), None, k, None, k)
        assert L.rocblas_stop_device_memory_size_query(h.value, ctypes.byref(size)) == 0
        return size.value

    A, B = oracle.nan_triangle_problem(5, "L", "L", "N", "N", k, cols, k, k, np.float64)
    X = oracle.trsm("L", "L", "N", "N", 1.25, A, B)
    with rb.Handle() as h:
        sizes = [query(h, w) for w in (8, 16, 32, 64)]
        assert len(set(sizes)) == 1
        assert L.rocblas_set_device_memory_size(h.value, sizes[0]) == 0
        for w in (8, 16, 32, 64):
            assert width(w) == 0
            out = _solve(h, "L", "L", "N", "N", k, cols, A, B)
            assert oracle.matrix_norm_1(X, out) <= oracle.trsm_tolerance(np.float64, k)


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("n", [1, 15, 16, 17, 32, 33, 64, 65, 127, 128, 200])
def test_inverse_blocks(n, dtype):
    rng = np.random.default_rng(n)
    with rb.Handle() as h:
        for uplo, diag in itertools.product("UL", "NU"):
            A = rng.uniform(-1, 1, (n, n)) / n
            A = np.tril(A, -1) if uplo == "L" else np.triu(A, 1)
            T = A + (np.eye(n) if diag == "U" else np.diag(rng.uniform(1, 2, n)))
            stored = np.where(np.eye(n, dtype=bool) & (diag == "U"), np.nan, T)
            other = np.triu(np.ones((n, n), bool), 1) if uplo == "L" else np.tril(np.ones((n, n), bool), -1)
            stored[other] = np.nan
            dA = dm.to_device(np.asfortranarray(stored, dtype=dtype))
            dX = dm.empty(n + 1, n, dA.dtype, fill=0.0)
            dm.trtri(h, uplo, diag, n, dA, n, dX, n + 1)
            torch.cuda.synchronize()
            X = dm.to_host(dX)[:n]
            eps = np.finfo(dtype).eps
            # the inverse's entries are at most about 1; n terms per product
            assert np.abs(X - np.linalg.inv(T.astype(dtype).astype(np.float64))).max() <= 4 * n * eps
            assert (X[other] == 0).all()


@pytest.mark.parametrize("k,cols,fixed", [(600, 700, False), (600, 700, True), (1900, 600, False), (2304, 520, False),
                                          (2400, 530, False)])
def test_fp32_with_many_columns(k, cols, fixed):
    """FP32 with more right-hand sides than chain_max_cols_f32: on the chain, or sliced updates
    between chain sub-solves; in a workspace of the inverse blocks alone, the recursive solve."""
    A, B = oracle.nan_triangle_problem(k, "L", "L", "N", "N", k, cols, k, k, np.float32)
    with rb.Handle() as h:
        if fixed:
            assert rb.lib().rocblas_set_device_memory_size(h.value, 128 * k * 4) == 0
        out = _solve(h, "L", "L", "N", "N", k, cols, A, B)  # status success
    X = oracle.trsm("L", "L", "N", "N", 1.25, A, B)
    assert oracle.matrix_norm_1(X, out) <= oracle.trsm_tolerance(np.float32, k)


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("k,cols", [(257, 2000), (512, 1300), (256, 2000)])
@pytest.mark.parametrize("fixed", [False, True])
def test_small_orders_with_many_columns(k, cols, dtype, fixed):
    """Orders above 256 go to the chain; in a workspace that holds nothing, to the strip solver,
    with the same status."""
    for side, uplo in ("LL", "RU"):
        m, n = (k, cols) if side == "L" else (cols, k)
        A, B = oracle.nan_triangle_problem(k, side, uplo, "N", "N", m, n, k, m, dtype)
        with rb.Handle() as h:
            if fixed:
                assert rb.lib().rocblas_set_device_memory_size(h.value, 64) == 0
            out = _solve(h, side, uplo, "N", "N", m, n, A, B)
        X = oracle.trsm(side, uplo, "N", "N", 1.25, A, B)
        assert oracle.matrix_norm_1(X, out) <= oracle.trsm_tolerance(dtype, max(m, n))


@pytest.mark.parametrize("dtype", [np.complex128, np.complex64])
@pytest.mark.parametrize("w", [0, 8, 16, 32, 64])
def test_complex_widths(width, w, dtype):
    """Complex systems as real ones of twice the order: blocks of 64, every side / uplo / trans."""
    assert width(w) == 0
    alpha = 0.5 - 1.25j
    with rb.Handle() as h:
        for i, (side, uplo, trans, diag) in enumerate(itertools.product("LR", "UL", "NTC", "NU")):
            k, cols = [(129, 1), (191, w + 1), (256, 9), (257, 2 * w + 3), (320, 33)][i % 5]
            m, n = (k, cols) if side == "L" else (cols, k)
            A, B = oracle.nan_triangle_problem(i, side, uplo, trans, diag, m, n, k + i % 3, m + i % 2, dtype)
            dA, dB = dm.to_device(A), dm.to_device(B)
            dm.trsm(h, side, uplo, trans, diag, m, n, alpha, dA, A.shape[0], dB, B.shape[0], alpha_on_device=i % 2 == 1)
            torch.cuda.synchronize()
            out = dm.to_host(dB)
            X = oracle.trsm(side, uplo, trans, diag, alpha, A, np.asfortranarray(B[:m]))
            assert oracle.matrix_norm_1(X, out[:m]) <= oracle.trsm_tolerance(dtype, max(m, n)), (side, uplo, trans, diag)
            assert np.isnan(out[m:]).all()


def test_capture_of_a_call_whose_workspace_was_never_grown():
    """Paths that want more workspace than their fallback must not allocate under capture: a fresh
    handle's complex solve and an order of the strip solver are captured."""
    for dtype, k, cols in ((np.complex128, 200, 20), (np.float64, 400, 2000)):
        A, B = oracle.nan_triangle_problem(k, "L", "L", "N", "N", k, cols, k, k, dtype)
        X = oracle.trsm("L", "L", "N", "N", 1.0, A, B)
        s = torch.cuda.Stream()
        with rb.Handle() as h, torch.cuda.stream(s):
            h.set_stream(ctypes.c_void_p(s.cuda_stream))
            dA, dB0 = dm.to_device(A), dm.to_device(B)
            dB = dB0.clone()
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph, stream=s):
                dm.trsm(h, "L", "L", "N", "N", k, cols, 1.0, dA, k, dB, k)
            graph.replay()
            s.synchronize()
            assert oracle.matrix_norm_1(X, dm.to_host(dB)) <= oracle.trsm_tolerance(dtype, max(k, cols))


def _substitution_80_bit(A, B, upper):
    X = B.astype(np.clongdouble if np.iscomplexobj(B) else np.longdouble)
    k = len(A)
    for i in range(k - 1, -1, -1) if upper else range(k):
        X[i] /= A[i, i]
        rest = slice(0, i) if upper else slice(i + 1, k)
        X[rest] -= np.outer(A[rest, i].astype(X.dtype), X[i])
    return X


@pytest.mark.parametrize("dtype", [np.float64, np.complex128])
@pytest.mark.parametrize("w", [8, 16, 32, 64])
@pytest.mark.parametrize("uplo", "LU")
@pytest.mark.parametrize("side,k,cols", [("L", 500, 150), ("R", 300, 1300)])
def test_rounding_error(width, side, k, cols, uplo, w, dtype):
    """With a dominant diagonal a row's result is rounded three times: its right-hand side less the sum
    over the finished blocks, the reciprocal of its diagonal entry and their product plus the rest of
    the sum.  A rounding to nearest has a relative error of u / sqrt(3 m^2) in the mean square over
    mantissas m in [1, 2), 0.41 u; three give 0.71 u, and the bound leaves no room for a fourth
    (0.82 u).  Complex: the reciprocal and the product have one more each, 0.91 u.  (A block that is
    substituted has one rounding per row before it; order 300 with 1300 rows from the right is checked
    for blocks to substitute, and its last one is short.)"""
    assert width(w) == 0
    m, n = (k, cols) if side == "L" else (cols, k)
    A, B = oracle.nan_triangle_problem(3, side, uplo, "N", "N", m, n, k, m, dtype)
    with rb.Handle() as h:
        dA, dB = dm.to_device(A), dm.to_device(B)
        dm.trsm(h, side, uplo, "N", "N", m, n, 1.0, dA, k, dB, m)
        torch.cuda.synchronize()
    out = dm.to_host(dB)
    X = _substitution_80_bit(A, B, uplo == "U") if side == "L" else _substitution_80_bit(A.T, B.T, uplo == "L").T
    d = out - X
    error = np.sqrt((abs(d) ** 2).sum() / (abs(X) ** 2).sum())
    assert error <= (0.8 if dtype == np.float64 else 0.95) * 2.0**-53, error / 2.0**-53


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("bad", [np.nan, np.inf])
@pytest.mark.parametrize("i,j", [(5, 2), (20, 3), (27, 17), (50, 3), (120, 60), (127, 0)])
def test_inverse_block_of_a_non_finite_entry(i, j, bad, dtype):
    """Rows of the inverse before the entry's do not depend on it, nor do the columns after its own;
    a substitution leaves them finite."""
    n = 128
    rng = np.random.default_rng(i)
    T = np.tril(rng.uniform(-1, 1, (n, n)) / n, -1) + np.diag(rng.uniform(1, 2, n))
    T[i, j] = bad
    with rb.Handle() as h:
        for uplo in "LU":
            M = T if uplo == "L" else T[::-1, ::-1]
            dA = dm.to_device(np.asfortranarray(M, dtype=dtype))
            dX = dm.empty(n, n, dA.dtype, fill=0.0)
            dm.trtri(h, uplo, "N", n, dA, n, dX, n)
            torch.cuda.synchronize()
            X = dm.to_host(dX)
            X = X if uplo == "L" else X[::-1, ::-1]
            assert np.isfinite(X[:i]).all() and np.isfinite(X[:, j + 1:]).all()
            assert not np.isfinite(X[i, j]) and (np.triu(X, 1) == 0).all()
            Y = np.linalg.inv(T[:i, :i].astype(dtype).astype(np.float64))
            assert np.abs(X[:i, :i] - Y).max() <= 4 * n * np.finfo(dtype).eps


@pytest.mark.parametrize("dtype,lines", [
    (np.float64, [(257, 2), (320, 2), (321, 0.75), (352, 0.75), (353, 0.75)]),
    (np.float32, [(320, 2), (352, 0.75)]),
    (np.complex128, [(129, 2), (160, 1), (161, 2)]),
    (np.complex64, [(129, 4), (192, 4), (193, 1.5), (224, 1.5), (225, 1.5)])])
def test_both_sides_of_the_line_between_chain_and_one_cta_solvers(dtype, lines):
    """(order, d): the line is at SMs / d strips of 32 columns."""
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    u = np.finfo(dtype).eps / 2
    with rb.Handle() as h:
        for k, d in lines:
            for cols in (int(sms / d) * 32, int(sms / d) * 32 + 1):
                for side in "LR":
                    m, n = (k, cols) if side == "L" else (cols, k)
                    A, B = oracle.nan_triangle_problem(k, side, "L", "N", "N", m, n, k, m, dtype)
                    dA, dB = dm.to_device(A), dm.to_device(B)
                    dm.trsm(h, side, "L", "N", "N", m, n, 1.0, dA, k, dB, m)
                    M = torch.tril(dA.mT)
                    # residual of a backward stable solve: 2 k u of |M| |X| (complex: twice as many products)
                    if side == "L":
                        R, bound = (M @ dB.mT - dm.to_device(B).mT).abs(), M.abs() @ dB.mT.abs()
                    else:
                        R, bound = (dB.mT @ M - dm.to_device(B).mT).abs(), dB.mT.abs() @ M.abs()
                    assert (R <= (4 if np.iscomplexobj(A) else 2) * k * u * bound).all(), (k, cols, side)
