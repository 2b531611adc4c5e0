"""Fields at the edges of what the direct passes choose by size: steps whose chunks lie
below a tile, whose slots are summed in runs and whose updates run in the reduction, and
the ζ passes' staging per warp."""
import ctypes

import numpy as np
import pytest

from flowunsteady_gb300 import _lib as L
from flowunsteady_gb300.workloads import uniform_box
from tests.helpers import Ctx, rel_l2, scheme

pytestmark = pytest.mark.gpu

KERNELS = [L.KERNEL_WINCKELMANS, L.KERNEL_GAUSSIANERF]


def field(n):
    X, G, S = uniform_box(n, seed_index=300 + n % 97)
    return X * 0.5, G * 200.0, S * 3.0


@pytest.mark.parametrize("k", KERNELS)
@pytest.mark.parametrize("n,static", [(1, 0), (2, 1), (31, 0), (33, 4), (129, 0), (513, 100),
                                      (1201, 0), (4097, 1000), (8192, 0), (8193, 500)])
def test_step_at_the_edges_of_small_fields(oracle, k, n, static):
    # One RK3 step from U and J that are within 1e-5 in the 2-norm: what moves is a
    # mean of the stages' rates (weights 1/6, 3/10, 8/15), so ΔX is within 1e-5 of its
    # own norm, and ΔΓ and Δσ within 1e-5 of dt·|J| times the largest |Γ| and σ
    # (1 + 3/5 and 3/5 of the stretching: factor 2).
    X, G, S = field(n)
    dt, nm = 1e-3, n - static
    sc = scheme(kernel=k, prec=L.PREC_FP32C, uinf=(0.1, 0, 0))
    Xo, Go, So, _, _ = oracle.step(sc, X, G, S, None, dt, n_static=static)
    _, J = oracle.uj_direct(k, X, G, S, Xt=X[:nm])
    with Ctx(n) as c:
        c.set(X[:nm], G[:nm], S[:nm])
        if static:
            c.append(X[nm:], G[nm:], S[nm:], static=True)
        c.step(sc, dt)
        Xg, Gg, Sg = c.state()
    nj = dt * np.linalg.norm(J)
    assert np.array_equal(Xg[nm:], X[nm:]) and np.array_equal(Gg[nm:], G[nm:])
    assert np.linalg.norm(Xg - Xo) <= 1e-5 * np.linalg.norm(Xo - X) + 1e-15
    assert np.linalg.norm(Gg - Go) <= 2e-5 * nj * np.linalg.norm(G, axis=1).max() + 1e-15
    assert np.linalg.norm(Sg - So) <= 2e-5 * nj * S.max() + 1e-15


@pytest.mark.parametrize("k", KERNELS)
@pytest.mark.parametrize("n", [1, 31, 32, 33, 127, 257, 1025, 4096])
def test_zeta_pass_at_the_edges_of_its_tiles(oracle, k, n):
    X, G, S = field(n)
    _, J = oracle.uj_direct(k, X, G, S)
    E0, _ = oracle.estr_direct(k, X, G, S, J)
    sc = scheme(kernel=k, prec=L.PREC_FP32C, sfs=L.SFS_CONSTANT)
    with Ctx(n) as c:
        c.set(X, G, S)
        c.uj(k, L.PREC_FP32C)
        c.rc(c.lib.vpm_eval_sfs(c.p, ctypes.byref(sc)))
        _, E = c.sfs()
    if n == 1:
        assert np.all(E == 0)
    else:
        assert rel_l2(E, E0) <= 2e-5   # 1e-5 each from J and from the sum
