"""∂w/∂z of the FP64 passes is a sum of its own: next to the two other diagonal elements
of J it may be as small as the plane of the particles makes it."""
import ctypes

import numpy as np
import pytest

from flowunsteady_gb300 import _lib as L
from tests.helpers import Ctx, scheme

pytestmark = pytest.mark.gpu

W, G = L.KERNEL_WINCKELMANS, L.KERNEL_GAUSSIANERF
INV4PI = 1.0 / (4.0 * np.pi)


def p_of(k, r2, s):
    """q'/r of a pair."""
    if k == W:
        return -3.0 * (r2 + 3.5 * s * s) * (r2 + s * s) ** -3.5
    from math import erf, exp, pi, sqrt
    rho = sqrt(r2) / s
    g = erf(rho / sqrt(2.0)) - sqrt(2.0 / pi) * rho * exp(-0.5 * rho * rho)
    return (sqrt(2.0 / pi) * rho ** 3 * exp(-0.5 * rho * rho) - 3.0 * g) / (rho * s) ** 5


def dp_of(k, r2, s):
    """Its derivative by a common scale of the cores."""
    if k == W:
        return 52.5 * s ** 4 * (r2 + s * s) ** -4.5
    return np.sqrt(2.0 / np.pi) / s ** 5 * np.exp(-0.5 * r2 / (s * s))


def pair(rho, sigma=0.7):
    d = np.array([0.6, -0.8, 1e-9]) * rho * sigma
    X = np.stack([d, np.zeros(3)])
    Ga = np.array([[0.0, 0.0, 0.7], [0.3, 0.5, 0.2]])
    c2 = d[0] * Ga[1, 1] - d[1] * Ga[1, 0]
    return X, Ga, np.full(2, sigma), d, c2


@pytest.mark.parametrize("k", [W, G])
@pytest.mark.parametrize("rho", [1.7, 4.0, 20.0])
def test_j22_of_a_nearly_planar_pair(k, rho):
    # J22 = -p c2 dz/(4π), 1e-9 of the rest of J, from the one product of that sum: 1e-12
    # covers the closed form's cancellation at ρ = 1.7 (a factor of ten on 2^-53 for every
    # operation), where J00 + J11 would leave 1e-7.
    X, Ga, S, d, c2 = pair(rho)
    exact = -INV4PI * p_of(k, d @ d, S[1]) * c2 * d[2]
    with Ctx(2) as c:
        c.set(X, Ga, S)
        _, J = c.uj(k, L.PREC_FP64)
    assert abs(J[0, 2, 2] - exact) <= 1e-12 * abs(exact)


@pytest.mark.parametrize("k,form,alpha", [(W, "analytic", 0.999), (G, "analytic", 0.999),
                                          (G, "difference", 0.5), (W, "difference", 0.5)])
def test_j22_of_the_test_filter(k, form, alpha):
    # The target's strength along z: <Γ·L> = (3α-2) Γz² times (α-1) dJ22/dα or the
    # difference of J22 at the cores ασ and σ.  As above; differences at α = 1/2 cancel
    # less than one digit.
    X, Ga, S, d, c2 = pair(1.7)
    r2, sg = d @ d, S[1]
    dp = ((alpha - 1.0) * dp_of(k, r2, sg) if form == "analytic"
          else p_of(k, r2, alpha * sg) - p_of(k, r2, sg))
    exact = (3.0 * alpha - 2.0) * -INV4PI * dp * c2 * d[2] * Ga[0, 2] ** 2
    s = scheme(kernel=k, prec=L.PREC_FP64, sfs=L.SFS_DYNAMIC, alpha=alpha,
               flags=L.SFS_ANALYTIC_DSIGMA if form == "analytic" else 0)
    with Ctx(2) as c:
        c.set(X, Ga, S)
        c.rc(c.lib.vpm_eval_sfs(c.p, ctypes.byref(s)))
        C, _ = c.sfs()
    assert abs(C[0, 1] - exact) <= 1e-11 * abs(exact)
