"""FP64 pair routines (csrc/pair_f64.cuh) over the range of ρ = r/σ: table nodes and
the middles between them, the switch to the far form at ρ² = 90, coincident and nearly
coincident particles, and the exponential down to its subnormal results."""
import ctypes

import numpy as np
import pytest

from flowunsteady_gb300 import _lib as L
from tests.helpers import Ctx, rel_l2, scheme

pytestmark = pytest.mark.gpu

# Nodes of the core expansions lie at ρ² = k/8, their limits at odd multiples of 1/16.
RHO = [1e-9, 1e-3, 0.25, 0.125 ** 0.5, (1 / 16) ** 0.5, 0.5, 1.0, 3.0, (719.5 / 8) ** 0.5,
       90 ** 0.5 * (1 - 1e-15), 90 ** 0.5 * (1 + 1e-15), 12.0, 25.0, 37.0]
FAR = [37.3, 37.9, 38.2, 38.55, 38.7, 60.0, 1e4]    # ζ below 2^-1000: subnormal, then zero


def pair(rho, sigma=0.7):
    d = np.array([0.6, -0.48, 0.64])
    X = np.stack([np.array([0.3, -0.2, 0.5]), np.array([0.3, -0.2, 0.5]) + rho * sigma * d])
    G = np.array([[0.3, -0.5, 0.2], [-0.1, 0.4, 0.7]])
    return X, G, np.full(2, sigma)


@pytest.mark.parametrize("k", [L.KERNEL_WINCKELMANS, L.KERNEL_GAUSSIANERF])
@pytest.mark.parametrize("rho", RHO + FAR)
def test_pairs_over_the_range_of_rho(oracle, k, rho):
    # 1e-12 and 1e-11 as for every FP64 sum: both sides form q and p to a few units of
    # 2^-53, the oracle with the cancellation of erf - ρe^{-ρ²/2} above its series.
    X, G, S = pair(rho)
    U0, J0 = oracle.uj_direct(k, X, G, S)
    E0, _ = oracle.estr_direct(k, X, G, S, J0)
    s = scheme(kernel=k, prec=L.PREC_FP64, sfs=L.SFS_CONSTANT)
    with Ctx(2) as c:
        c.set(X, G, S)
        U, J = c.uj(k, L.PREC_FP64)
        c.rc(c.lib.vpm_eval_sfs(c.p, ctypes.byref(s)))
        _, E = c.sfs()
    assert rel_l2(U, U0) <= 1e-12 and rel_l2(J, J0) <= 1e-12
    if rho in RHO:
        assert rel_l2(E, E0) <= 1e-11
    else:   # the argument's own rounding, ρ²/2·2^-53, or results at the end of the range
        assert np.all(np.abs(E - E0) <= 1e-11 * np.abs(E0).max() + 1e-320)


@pytest.mark.parametrize("k", [L.KERNEL_WINCKELMANS, L.KERNEL_GAUSSIANERF])
@pytest.mark.parametrize("nb,nf", [(1, 1), (31, 63), (33, 65), (129, 2000), (5, 40000)])
def test_bound_forces_at_the_edges_of_chunks(oracle, k, nb, nf):
    # One bound particle to more than a block, one chunk to several hundred, particles
    # in common between the two sets (dropped); FP64 sums as above.
    rng = np.random.default_rng(nb + nf)
    X, G, S = rng.uniform(-1, 1, (nf, 3)), rng.normal(0, 0.1, (nf, 3)), np.full(nf, 0.05)
    Xb, Gb = rng.uniform(-1, 1, (nb, 3)), rng.normal(0, 0.1, (nb, 3))
    Sb = rng.uniform(0.02, 0.3, nb)
    Xb[0] = X[nf // 2]
    M0 = oracle.ffv_direct(k, Xb, Gb, Sb, X, G)
    M = np.empty((nb, 6))
    with Ctx(nf) as c:
        c.set(X, G, S)
        c.rc(c.lib.vpm_ffv_direct(c.p, k, nb, L.dptr(Xb), 3, L.dptr(Gb), 3, L.dptr(Sb), 1,
                                  L.dptr(M), 6))
    assert rel_l2(M, M0) <= 1e-12


@pytest.mark.parametrize("alpha", [0.999, 0.6, 1.3])
@pytest.mark.parametrize("n", [1, 127, 129, 700])
def test_finite_difference_cd_in_one_pass(oracle, alpha, n):
    # The dynamic C_d of the finite-difference form, whose differences the FP64
    # Gaussian-erf passes sum directly.  Both sides carry the rounding of q, p and ζ
    # (a few 2^-53 of each) over the difference, |1 - α| of them: 1e-11/|1 - α|.
    rng = np.random.default_rng(n)
    X, G = rng.uniform(-1, 1, (n, 3)), rng.normal(0, 0.1, (n, 3))
    S = rng.uniform(0.1, 0.3, n)
    s = scheme(kernel=L.KERNEL_GAUSSIANERF, prec=L.PREC_FP64, sfs=L.SFS_DYNAMIC, alpha=alpha,
               flags=L.SFS_FORCE_POSITIVE, maxC=0.0)
    Xo, Go, So, Co, Eo = oracle.step(s, X, G, S, None, 1e-3)
    with Ctx(n) as c:
        c.set(X, G, S)
        c.step(s, 1e-3)
        Xg, Gg, Sg = c.state()
        C, E = c.sfs()
    tol = 1e-11 / abs(1 - alpha)
    assert rel_l2(C[:, 1:], Co[:, 1:]) <= tol
    assert rel_l2(Xg, Xo) <= 1e-12 and rel_l2(E, Eo) <= max(tol, 1e-9)
    assert rel_l2(Gg, Go) <= max(tol, 1e-9)
