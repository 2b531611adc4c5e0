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


def line(n):
    # Particles in order along a line 200 cores long: warps whose targets are close to each
    # other, most 32 sources beyond the 13.3 cores where ζ vanishes, some cut by that limit.
    rng = np.random.default_rng(n)
    X = rng.uniform(-0.1, 0.1, (n, 3))
    X[:, 0] = np.sort(rng.uniform(0.0, 20.0, n))
    return X, rng.normal(0.0, 0.2, (n, 3)), rng.uniform(0.08, 0.12, n)


def stretch(J, v):
    return np.einsum("iba,ib->ia", J, v)   # the transposed scheme


@pytest.mark.parametrize("chunk", [128, 1 << 20])
@pytest.mark.parametrize("prec", [L.PREC_FP32, L.PREC_FP32C])
@pytest.mark.parametrize("layout", ["box", "line"])
@pytest.mark.parametrize("n", [1, 33, 127, 513, 700, 1057])
def test_zeta_passes_staged_per_warp(oracle, n, layout, prec, chunk):
    # The form of four targets a thread (Gaussian-erf ζ and ζ with its derivative), pinned
    # on fields whose last 32 sources, last warps and last chunks are cut short.  Terms of
    # E_str and dE_str/dα within 1e-5 from J or dJ/dα and 1e-5 from their sums, each of its
    # own 2-norm; two coincident particles are dropped from each other's sums.
    X, Ga, S = field(n) if layout == "box" else line(n)
    if n > 1:
        X[n // 2] = X[0]
    k, alpha = L.KERNEL_GAUSSIANERF, 0.999
    _, J = oracle.uj_direct(k, X, Ga, S)
    DJ = oracle.uj_dsigma(k, X, Ga, S)
    r2 = ((X[:, None] - X[None]) ** 2).sum(2)
    x = r2 / S ** 2
    z = np.where(r2 > 0, (2 * np.pi) ** -1.5 * np.exp(-0.5 * x) / S ** 3, 0.0)
    dz = z * (x - 3.0)
    V, W = stretch(J, Ga), stretch(DJ, Ga)
    terms = stretch(J, z @ Ga), z @ V
    dterms = stretch(DJ, z @ Ga), stretch(J, dz @ Ga), dz @ V + z @ W
    E0, DE0 = terms[0] - terms[1], dterms[0] + dterms[1] - dterms[2]
    den = (alpha - 1.0) * S ** 3 * (2 * np.pi) ** 1.5   # <Γ·m> = den Γ·dE_str/dα
    tile = L.Tile(128, 4, chunk, 0)
    with Ctx(n) as c:
        c.set(X, Ga, S)
        c.rc(c.lib.vpm_set_tile(c.p, k, prec, ctypes.byref(tile)))
        for sfs, flags in ((L.SFS_CONSTANT, 0), (L.SFS_DYNAMIC, L.SFS_ANALYTIC_DSIGMA)):
            s = scheme(kernel=k, prec=prec, sfs=sfs, flags=flags, alpha=alpha, maxC=0.0)
            c.rc(c.lib.vpm_eval_sfs(c.p, ctypes.byref(s)))
            C, E = c.sfs()
            norms = sum(np.linalg.norm(t) for t in terms)
            assert np.linalg.norm(E - E0) <= 2e-5 * norms
    bound = [np.linalg.norm(den * np.linalg.norm(Ga, axis=1) * np.linalg.norm(t, axis=1))
             for t in dterms]
    assert np.linalg.norm(C[:, 2] - den * (Ga * DE0).sum(1)) <= 2e-5 * sum(bound)
