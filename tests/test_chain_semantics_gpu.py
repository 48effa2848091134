"""What one system of order 257 to 512 with many right-hand sides, or a complex one above 128, must
answer on the chain (trsm_chain.cuh) as in the solvers that substitute (strip_solve.cuh,
block_solve.cuh), which take it where the workspace is small."""
import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")

import oracle  # noqa: E402
import rocblas_b200 as rb  # noqa: E402
from rocblas_b200 import devmem as dm  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,k,cols", [(np.float64, 300, 1300), (np.float32, 400, 2000), (np.float64, 700, 40),
                                          (np.complex128, 200, 20), (np.complex64, 300, 20)])
def test_alpha_zero_on_the_device_leaves_a_unread(dtype, k, cols):
    """A NULL A is accepted with device-mode alpha.  Whether A was read shows in the workspace, where
    a NaN triangle's inverse blocks would be NaN."""
    A = np.full((k, k), np.nan, dtype=dtype, order="F")
    B = np.full((k, cols), np.nan, dtype=dtype, order="F")
    dA, dB = dm.to_device(A), dm.to_device(B)
    ws = torch.zeros(1 << 18, dtype=torch.float64, device="cuda")
    with rb.Handle() as h:
        assert rb.lib().rocblas_set_workspace(h.value, ctypes.c_void_p(ws.data_ptr()), ws.numel() * 8) == 0
        dm.trsm(h, "L", "L", "N", "N", k, cols, 0.0, dA, k, dB, k, alpha_on_device=True)
        torch.cuda.synchronize()
    assert (dB == 0).all()
    assert not torch.isnan(ws.view(torch.float32 if dtype in (np.float32, np.complex64) else torch.float64)).any()


SYSTEMS = [("L", "L", "N"), ("L", "U", "N"), ("R", "L", "T"), ("R", "U", "C")]
SIZES = [(np.float64, 300, 1300), (np.float32, 400, 2000), (np.complex128, 200, 20), (np.complex64, 300, 20)]


def _system(side, uplo, trans, k, cols, dtype, seed=7):
    """A well-conditioned triangle, the right-hand sides, and the positions of A's rows in the order
    in which the solve reaches them."""
    m, n = (k, cols) if side == "L" else (cols, k)
    A, B = oracle.nan_triangle_problem(seed, side, uplo, trans, "N", m, n, k, m, dtype)
    forward = ((uplo == "L") != (trans != "N")) == (side == "L")
    return A, B, np.arange(k) if forward else np.arange(k)[::-1]


def _entry(B, side, r, c):
    return (r, c) if side == "L" else (c, r)


def _solve_both(side, uplo, trans, A, B):
    """On the chain, and in a workspace too small for it."""
    m, n = B.shape
    out = []
    for small in (False, True):
        with rb.Handle() as h:
            if small:
                assert rb.lib().rocblas_set_device_memory_size(h.value, 64) == 0
            dA, dB = dm.to_device(A), dm.to_device(B)
            dm.trsm(h, side, uplo, trans, "N", m, n, 1.0, dA, A.shape[0], dB, m)
            torch.cuda.synchronize()
            out.append(dm.to_host(dB))
    return out


def _same_where_finite(chain, other, dtype, k):
    fin = np.isfinite(chain)
    assert (fin == np.isfinite(other)).all()
    a, b = np.where(fin, chain, 0), np.where(fin, other, 0)
    assert np.abs(a - b).max() <= oracle.trsm_tolerance(dtype, k) * max(1.0, np.abs(b).max())


@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
@pytest.mark.parametrize("dtype,k,cols", SIZES)
@pytest.mark.parametrize("side,uplo,trans", SYSTEMS)
def test_non_finite_right_hand_side(side, uplo, trans, dtype, k, cols, bad):
    """It reaches its own row and the ones solved after it, in its own column."""
    A, B, order = _system(side, uplo, trans, k, cols, dtype)
    at = [(0, 0), (13, 2), (31, 9), (127, 3), (128, 11), (150, 4), (k - 1, 5)]  # (position in the solve, column)
    for pos, col in at:
        B[_entry(B, side, order[pos], col)] = bad
    chain, other = _solve_both(side, uplo, trans, A, B)
    _same_where_finite(chain, other, dtype, k)
    X = chain if side == "L" else chain.T
    expect = np.ones(X.shape, bool)
    for pos, col in at:
        expect[order[pos:], col] = False
    assert (np.isfinite(X) == expect).all()


@pytest.mark.parametrize("dtype,k,cols", SIZES)
@pytest.mark.parametrize("side,uplo,trans", SYSTEMS)
@pytest.mark.parametrize("pos", [0, 20, 63, 130, -1])
def test_zero_on_the_diagonal(side, uplo, trans, dtype, k, cols, pos):
    """The substitution divides by it: nothing finite from its row on."""
    A, B, order = _system(side, uplo, trans, k, cols, dtype)
    r = order[pos]
    A[r, r] = 0
    chain, other = _solve_both(side, uplo, trans, A, B)
    _same_where_finite(chain, other, dtype, k)
    X = chain if side == "L" else chain.T
    assert np.isfinite(X[order[: pos % k]]).all() and not np.isfinite(X[order[pos % k:]]).any()


@pytest.mark.parametrize("bad", [np.nan, np.inf])
@pytest.mark.parametrize("dtype,k,cols", SIZES)
@pytest.mark.parametrize("side,uplo,trans", SYSTEMS)
@pytest.mark.parametrize("pos,before", [(20, 3), (60, 20), (120, 100), (190, 10)])
def test_non_finite_entry_of_a(side, uplo, trans, dtype, k, cols, bad, pos, before):
    """In the row solved at `pos`, beside the row solved at `before`: as a right-hand side's."""
    A, B, order = _system(side, uplo, trans, k, cols, dtype)
    i, j = order[pos], order[before]
    M = A if (trans == "N") == (side == "L") else A.T  # the matrix whose rows are solved
    M[i, j] = bad
    chain, other = _solve_both(side, uplo, trans, A, B)
    _same_where_finite(chain, other, dtype, k)
    X = chain if side == "L" else chain.T
    assert np.isfinite(X[order[:pos]]).all() and not np.isfinite(X[order[pos:]]).any()


@pytest.mark.parametrize("dtype,k,cols", [s for s in SIZES if s[0] in (np.float64, np.complex128)])
def test_inverse_that_overflows(dtype, k, cols):
    """Row 50 of [[1, 0], [1, 1e-300]] has the solution 0; an inverse would subtract infinities."""
    A, B, _ = _system("L", "L", "N", k, cols, dtype)
    A[50, :50] = A[51:, 50] = 0
    A[50, 3] = 1
    A[50, 50] = 1e-300
    A[3, :3] = 0
    A[3, 3] = 1
    B[3] = B[50] = 1e10
    chain, other = _solve_both("L", "L", "N", A, B)
    assert (chain[50] == 0).all() and (other[50] == 0).all()
    _same_where_finite(chain, other, dtype, k)


def test_supplied_inverse_blocks():
    """trsm_ex with the inverse blocks, whose builder reads a zero as 1."""
    k, cols, r = 300, 1300, 140
    A, B, _ = _system("L", "L", "N", k, cols, np.float64)
    A[r, r] = 0
    with rb.Handle() as h:
        dA, dB = dm.to_device(A), dm.to_device(B)
        inv = dm.build_invA(h, "L", "N", dA, k, k)
        dm.trsm_ex(h, "L", "L", "N", "N", k, cols, 1.0, dA, k, dB, k, inv, inv.numel())
        torch.cuda.synchronize()
    out = dm.to_host(dB)
    assert np.isfinite(out[:r]).all() and np.isinf(out[r]).all() and not np.isfinite(out[r:]).any()


@pytest.mark.parametrize("dtype,k,cols", SIZES + [(np.float32, 600, 700)])
def test_workspace_that_starts_anywhere(dtype, k, cols):
    """The caller's buffer has no alignment that the API asks for; what the chain cannot use goes to a
    solver that can, with the same status."""
    A, B, _ = _system("L", "L", "N", k, cols, dtype)
    ws = torch.zeros(1 << 20, dtype=torch.float32, device="cuda")
    with rb.Handle() as h:
        assert rb.lib().rocblas_set_workspace(h.value, ctypes.c_void_p(ws.data_ptr() + 4), ws.numel() * 4 - 64) == 0
        dA, dB = dm.to_device(A), dm.to_device(B)
        dm.trsm(h, "L", "L", "N", "N", k, cols, 1.0, dA, k, dB, k)
        torch.cuda.synchronize()
    X = oracle.trsm("L", "L", "N", "N", 1.0, A, B)
    assert oracle.matrix_norm_1(X, dm.to_host(dB)) <= oracle.trsm_tolerance(dtype, max(k, cols))
