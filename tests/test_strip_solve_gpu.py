"""The one-CTA strip solver (strip_solve.cuh) at the edges of its 8-row tiles, 32-column panels and
64- and 128-row super-blocks, against the oracle, and its treatment of infinities and NaNs, which
must reach exactly the entries that they reach in a row-by-row substitution."""
import itertools

import numpy as np
import pytest

torch = pytest.importorskip("torch")

import oracle  # noqa: E402
import rocblas_b200 as rb  # noqa: E402
from rocblas_b200 import devmem as dm  # noqa: E402

pytestmark = pytest.mark.gpu
ORDERS = [1, 7, 8, 9, 31, 33, 63, 64, 65, 96, 127, 128]


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("k", ORDERS)
def test_tile_edges(k, dtype):
    with rb.Handle() as h:
        for i, (side, uplo, trans, diag) in enumerate(itertools.product("LR", "UL", "NT", "NU")):
            cols = [1, 7, 8, 9, 32, 33][i % 6]
            m, n = (k, cols) if side == "L" else (cols, k)
            A, B = oracle.nan_triangle_problem(i, side, uplo, trans, diag, m, n, k + i % 3, m + i % 2, dtype)
            dA, dB = dm.to_device(A), dm.to_device(B)
            dm.trsm(h, side, uplo, trans, diag, m, n, -0.75, dA, A.shape[0], dB, B.shape[0])
            torch.cuda.synchronize()
            out = dm.to_host(dB)
            X = oracle.trsm(side, uplo, trans, diag, -0.75, A, np.asfortranarray(B[:m]))
            assert oracle.matrix_norm_1(X, out[:m]) <= oracle.trsm_tolerance(dtype, max(m, n)), (side, uplo, trans, diag)
            assert np.isnan(out[m:]).all()


@pytest.mark.parametrize("k", [129, 200, 256, 257, 511, 512])
def test_super_blocks(k):
    # enough strips that the strip solver takes orders above 128; a strided batch of a few systems
    batch, cols = 64, 40
    g = torch.Generator().manual_seed(k)
    A = torch.rand(batch, k, k, generator=g, dtype=torch.float64) * 2 - 1
    A = torch.tril(A / k) + torch.eye(k, dtype=torch.float64) * 1.5
    B = torch.rand(batch, k, cols, generator=g, dtype=torch.float64)
    X = torch.linalg.solve_triangular(A, B, upper=False)
    with rb.Handle() as h:
        dA, dB = A.mT.contiguous().cuda(), B.mT.contiguous().cuda()
        dm.trsm_strided_batched(h, "L", "L", "N", "N", k, cols, 1.0, dA, k, k * k, dB, k, k * cols, batch)
        torch.cuda.synchronize()
    # 40 eps k of the largest entry, the gate of the single solves
    assert (dB.mT.cpu() - X).abs().max() <= 40 * 2.3e-16 * k * X.abs().max()


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
def test_non_finite_right_hand_sides(bad, dtype):
    k, cols = 77, 5
    rng = np.random.default_rng(0)
    A = np.asfortranarray(np.tril(rng.uniform(-1, 1, (k, k)) / k) + 1.5 * np.eye(k), dtype=dtype)
    B = np.asfortranarray(rng.uniform(-1, 1, (k, cols)), dtype=dtype)
    for row, col in [(0, 0), (13, 2), (38, 3), (76, 4)]:
        Bb = B.copy(order="F")
        Bb[row, col] = bad
        with rb.Handle() as h:
            dA, dB = dm.to_device(A), dm.to_device(Bb)
            dm.trsm(h, "L", "L", "N", "N", k, cols, 1.0, dA, k, dB, k)
            torch.cuda.synchronize()
        out = dm.to_host(dB)
        # rows above the entry and the other columns do not depend on it; the entry's row does
        assert np.isfinite(out[:row, col]).all() and np.isfinite(np.delete(out, col, 1)).all()
        assert not np.isfinite(out[row, col])
        if row + 1 < k:
            assert not np.isfinite(out[row + 1:, col]).any()


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
def test_zero_diagonal(dtype):
    # the reference's substitution divides by it: infinite or NaN from that row on, finite above
    k, cols, row = 60, 9, 29
    rng = np.random.default_rng(1)
    A = np.asfortranarray(np.tril(rng.uniform(0.1, 1, (k, k)) / k) + 1.5 * np.eye(k), dtype=dtype)
    A[row, row] = 0
    B = np.asfortranarray(rng.uniform(0.5, 1, (k, cols)), dtype=dtype)
    with rb.Handle() as h:
        dA, dB = dm.to_device(A), dm.to_device(B)
        dm.trsm(h, "L", "L", "N", "N", k, cols, 1.0, dA, k, dB, k)
        torch.cuda.synchronize()
    out = dm.to_host(dB)
    X = oracle.trsm("L", "L", "N", "N", 1.0, np.asfortranarray(A[:row, :row]), np.asfortranarray(B[:row]))
    assert oracle.matrix_norm_1(X, out[:row]) <= oracle.trsm_tolerance(dtype, k)
    assert np.isinf(out[row]).all() and not np.isfinite(out[row:]).any()


@pytest.mark.parametrize("k", [2, 60, 100])
def test_terms_that_overflow_and_cancel(k):
    """The last row of [[1, 0], [1, 1e-300]] X = 1e10 has the solution 0; the product with the inverse
    of the 2 x 2 block would subtract two infinities."""
    A = np.asfortranarray(np.eye(k))
    A[-1, -2], A[-1, -1] = 1, 1e-300
    B = np.asfortranarray(np.full((k, 9), 1e10))
    with rb.Handle() as h:
        dA, dB = dm.to_device(A), dm.to_device(B)
        dm.trsm(h, "L", "L", "N", "N", k, 9, 1.0, dA, k, dB, k)
        torch.cuda.synchronize()
    out = dm.to_host(dB)
    assert (out[:-1] == 1e10).all() and (out[-1] == 0).all()
