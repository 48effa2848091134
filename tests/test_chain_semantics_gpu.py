"""What one system of order 257 to 512 with many right-hand sides, or a complex one above 128, must
answer on the chain (trsm_chain.cuh) as in the solvers that substitute (strip_solve.cuh,
block_solve.cuh), which take it where the workspace is small."""
import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")

import oracle  # noqa: E402,F401
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
