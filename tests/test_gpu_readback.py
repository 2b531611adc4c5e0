"""Readbacks of some of the arrays of a state or an evaluation: what is asked for, at its
stride, and nothing else."""
import itertools

import numpy as np
import pytest

from flowunsteady_gb300 import _lib as L
from flowunsteady_gb300.workloads import uniform_box
from tests.helpers import Ctx

pytestmark = pytest.mark.gpu


def take(c, call, args, widths, n, want):
    out = [np.full((n, w + 2), 7.0) if q else None for w, q in zip(widths, want)]
    ptrs = []
    for w, o in zip(widths, out):
        ptrs += [None if o is None else L.dptr(o), w + 2 if o is not None else 0]
    c.rc(call(c.p, *args, *ptrs))
    for w, o in zip(widths, out):
        assert o is None or np.all(o[:, w:] == 7.0)
    return [None if o is None else o[:, :w] for w, o in zip(widths, out)]


@pytest.mark.parametrize("n", [1, 33, 50000])
def test_any_of_the_arrays(n):
    X, G, S = uniform_box(n, seed_index=5)
    with Ctx(n + 40) as c:   # rows further apart than the particles
        c.set(X, G, S)
        for want in itertools.product((False, True), repeat=3):
            got = take(c, c.lib.vpm_get_state, (n,), (3, 3, 1), n, want)
            for g, a in zip(got, (X, G, S[:, None])):
                assert g is None or np.array_equal(g, a)
        U, J = c.uj(L.KERNEL_GAUSSIANERF, L.PREC_FP32C)
        lo, m = n // 3, n - n // 3
        for want in itertools.product((False, True), repeat=2):
            got = take(c, c.lib.vpm_get_UJ, (lo, m), (3, 9), m, want)
            for g, a in zip(got, (U[lo:], J[lo:].reshape(m, 9))):
                assert g is None or np.array_equal(g, a)
