"""The FP64 exponential far below its range (csrc/pair_f64.cuh): 2^(n/2048) where the
32-bit words of n wrap, n = -2^31 and -2^32.  ζ and its derivatives are zero there."""
import ctypes

import numpy as np
import pytest

from flowunsteady_gb300 import _lib as L
from tests.helpers import Ctx, scheme

pytestmark = pytest.mark.gpu

# n = -r²/(2σ²)·log2(e)·2048, rounded: r of the middle of n's interval, which is 1e-7
# wide in r at n = -2^32 and 2e-7 at -2^31, 10^9 times the rounding of r.
N = [-(1 << 31) + d for d in (-1, 0, 1)] + [-(1 << 32) + d for d in (-2, -1, 0, 1, 2)] + [-(1 << 33)]
FLAGS = {"zeta": (L.SFS_CONSTANT, 0), "analytic": (L.SFS_DYNAMIC, L.SFS_ANALYTIC_DSIGMA),
         "difference": (L.SFS_DYNAMIC, 0)}


@pytest.mark.parametrize("form", sorted(FLAGS))
@pytest.mark.parametrize("n", N)
def test_zeta_is_zero_where_the_words_of_its_exponent_wrap(form, n):
    # Exact: every ζ, Dζ, Dq and Dp is below 2^-1000000, so E_str and both averages of
    # C_d are sums of zeros.  The finite difference has n at the cores ασ, α = 1/2.
    r = np.sqrt(-n / (1024.0 * np.log2(np.e))) * (0.5 if form == "difference" else 1.0)
    X = np.array([[0.0, 0.0, 0.0], [r, 0.0, 0.0]])
    G = np.array([[0.3, -0.5, 0.2], [-0.1, 0.4, 0.7]])
    sfs, flags = FLAGS[form]
    s = scheme(kernel=L.KERNEL_GAUSSIANERF, prec=L.PREC_FP64, sfs=sfs, flags=flags,
               alpha=0.5 if form == "difference" else 0.999)
    with Ctx(2) as c:
        c.set(X, G, np.ones(2))
        c.rc(c.lib.vpm_eval_sfs(c.p, ctypes.byref(s)))
        C, E = c.sfs()
    assert np.all(E == 0.0)
    if sfs == L.SFS_DYNAMIC:
        assert np.all(C[:, 1:] == 0.0)
