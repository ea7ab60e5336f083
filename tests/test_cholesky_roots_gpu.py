"""Pivot roots of the Cholesky factorization over the whole range of FP64:
diagonal matrices with every binary exponent from the smallest subnormal number to
the largest finite one, so that L(j, j) is the root of one pivot and L^-1 1 its
reciprocal.

Bounds. The reciprocal root is CUDA's rsqrt: within 1 unit in the last place
(documented maximum error of the double precision function), and the products
with an identity that follow are exact. The roots are CUDA's sqrt: 1 unit in the
last place at most. The reference values are roots in 80-bit numbers."""

import numpy as np
import pytest

from pysisyphus_addons import _native as nat

pytestmark = pytest.mark.gpu


def pivots():
    m = np.concatenate([[1.0, np.nextafter(1.0, 2.0), np.nextafter(2.0, 1.0)], np.random.default_rng(1).uniform(1.0, 2.0, 3)])
    e = np.arange(-1074, 1024)
    x = np.ldexp(m[:, None], e[None, :]).ravel()
    return x[np.isfinite(x) & (x > 0.0)]


def ulps(x, ref):
    return np.abs((x.astype(np.longdouble) - ref) / np.spacing(ref.astype(float)))


def test_roots_of_all_exponents():
    assert np.finfo(np.longdouble).nmant >= 63
    x = pivots()
    assert x.min() == 5e-324 and x.max() == np.finfo(float).max
    for k in range(0, len(x), 512):
        d = x[k : k + 512]
        L, y = nat.cholesky_solve(np.diag(d), np.ones((len(d), 1)))
        root = np.sqrt(d.astype(np.longdouble))
        assert np.array_equal(L, np.diag(np.diag(L)))
        assert ulps(np.diag(L), root).max() <= 1.0 + 1e-3
        assert ulps(y[:, 0], 1.0 / root).max() <= 1.0 + 1e-3


def test_infinite_pivot():
    d = np.array([4.0, np.inf, 9.0])
    L, y = nat.cholesky_solve(np.diag(d), np.ones((3, 1)))
    assert np.array_equal(np.diag(L), [2.0, np.inf, 3.0])
    assert y[1, 0] == 0.0 and np.isfinite(y).all()
