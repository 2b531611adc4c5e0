"""FP64 Gaussian-erf U/J of device arrays that hold NaNs of any bits: NaN comes out."""
import ctypes

import numpy as np
import pytest

from flowunsteady_gb300 import _lib as L

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bits", [0x7ff8000000000000, 0xfff8000000000000, 0xfff8000012345678,
                                  0xffffffffffffffff, 0x7ff80000ffffffff])
def test_nan_position_gives_nan(bits):
    n = 200
    rng = np.random.default_rng(3)
    X = rng.uniform(-1, 1, (3, n))
    X.view(np.uint64)[1, 17] = bits
    X, G, S = (torch.tensor(a, device="cuda:0") for a in
               (X, rng.normal(0, 0.1, (3, n)), np.full(n, 0.1)))
    U = torch.zeros((3, n), dtype=torch.float64, device="cuda:0")
    J = torch.zeros((9, n), dtype=torch.float64, device="cuda:0")
    L.check(L.lib().vpm_uj_device_async(
        L.KERNEL_GAUSSIANERF, L.PREC_FP64, n, X.data_ptr(), G.data_ptr(), S.data_ptr(), n, n, None,
        n, U.data_ptr(), J.data_ptr(), n, ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
    torch.cuda.synchronize()
    assert torch.isnan(J).all()
    assert torch.isnan(U).all()
