"""Rounding of the panel step's pivots: L_jj and 1 / L_jj over random mantissas, the
exponents on both sides of the fast reciprocal root's window and the ends of it.

The matrix is [[D, .], [B, 8 I]] with D diagonal and B diagonal of powers of two, so
L_jj is the root of one input and L_64+j,j = b_j / L_jj shows the reciprocal without
a rounding of its own.

Tolerance: the root is the correctly rounded one (numpy's).  The reciprocal may be off by
the rounding of the result and that of one more value it is made from, 2^-53 each."""
import numpy as np
import pytest

import exageostatcpp_b200 as egs

pytestmark = pytest.mark.gpu


def _pivots(kind):
    rng = np.random.default_rng(7)
    m = rng.uniform(1.0, 2.0, 64)
    if kind == "mantissas":
        e = rng.integers(-2, 2, 64)
    elif kind == "exponents":  # the whole window of the fast root, ends included
        e = rng.integers(-930, 926, 64)
        e[:2], e[-2:] = -930, 925
    else:  # outside it, subnormal and huge, alone and beside ordinary pivots
        e = np.where(rng.uniform(size=64) < 0.5, rng.integers(-1040, -931, 64), rng.integers(927, 1023, 64))
        e[::3] = 0
    return np.ldexp(m, e)


@pytest.mark.parametrize("kind", ["mantissas", "exponents", "outside"])
def test_pivot_roots_and_reciprocals(kind):
    d = _pivots(kind)
    assert np.all(d > 0)
    b = np.ldexp(1.0, np.frexp(np.sqrt(d))[1])
    a = np.eye(128)
    j = np.arange(64)
    a[j, j], a[64 + j, 64 + j], a[64 + j, j] = d, 8.0, b
    p = egs.Problem(128, 128)
    p.set_locations(*egs.generate_locations(128, 3))
    egs._check(p._lib.egs_set_tile(p._h, 0, 0, np.asfortranarray(a).ctypes.data_as(egs._D)), "set_tile")
    p.potrf()
    L = p.lower_matrix()
    p.close()
    assert np.array_equal(L[j, j], np.sqrt(d))
    exact = 1.0 / np.sqrt(d.astype(np.longdouble))
    got = L[64 + j, j].astype(np.longdouble) / b.astype(np.longdouble)
    assert np.abs(got / exact - 1.0).max() <= 2.0 ** -52
