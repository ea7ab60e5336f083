"""Explicit three-center blocks and half-transformation of the std tensors where
their tiles can go wrong: contracted shells of every L (several primitive pairs
per block), MO counts around the 16-wide orbital tiles and the 64-wide chunks,
more than one group of 256 partner shells, and more than one batch of auxiliary
columns.

Tolerance against the oracle: integrals agree to rounding (1e-13 of the largest
element); an integral or half-transformed value within rounding of the
reference's 1e-10 skips may be kept on one side and dropped on the other, which
moves an element by at most 1e-10 times two orbital coefficients: 2e-11.
"""

import numpy as np
import pytest

import oracle
from pysisyphus_addons import _native as nat
from pysisyphus_addons.common.shells import Shell, Shells
from pysisyphus_addons.common.synthetic import make_workload
from pysisyphus_addons.std import intor as std

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def raw():
    nat.set_boys_mode("exact")
    oracle.set_boys_mode("exact")
    nat.set_skip_metric(1)
    oracle.set_skip_metric(1)
    yield
    nat.set_skip_metric(0)
    oracle.set_skip_metric(0)
    nat.set_boys_mode("reference")
    oracle.set_boys_mode("reference")


def check(x, ref):
    assert np.abs(x - ref).max() <= 2e-11 + 1e-13 * np.abs(ref).max()


def contracted(centers, lmax, seed):
    """Shells of every L up to lmax on each center, with 1, 2 or 3 primitives."""
    rng = np.random.default_rng(seed)
    out = []
    for i, c in enumerate(centers):
        for L in range(lmax + 1):
            n = 1 + (L + i) % 3
            out.append(Shell(L, c, rng.uniform(0.2, 1.0, n), np.exp(rng.uniform(-1.5, 1.5, n)), i, 6))
    return Shells(out)


@pytest.mark.parametrize("nmos", [1, 15, 16, 17, 33, 48, 49])
def test_contracted_shells(nmos):
    X = np.random.default_rng(1).uniform(-2.0, 2.0, (2, 3))
    orb, aux = contracted(X, 4, 2), contracted(X, 5, 3)
    C = np.linalg.qr(np.random.default_rng(4).normal(size=(orb.sph_size, nmos)))[0]
    check(std.int_df2c_mo(orb, aux, C), oracle.int_df2c_mo(orb, aux, C))
    check(std.int_df1c(orb, aux), oracle.int_df1c(orb, aux))


@pytest.mark.parametrize("nshells,nmos", [(256, 64), (257, 65), (300, 130)])
def test_many_partner_shells(nshells, nmos):
    """s and p shells spread over a long line: most pairs are screened."""
    rng = np.random.default_rng(5)
    X = np.stack([np.linspace(0, 200, nshells), rng.normal(size=nshells), rng.normal(size=nshells)], axis=1)
    orb = Shells([Shell(i % 2, X[i], [1.0], [0.4 + (i % 5)], i, 1) for i in range(nshells)])
    aux = Shells([Shell(L, X[k], [1.0], [0.5 + L], k, 1) for k in (0, 150, nshells - 1) for L in range(3)])
    C = np.linalg.qr(rng.normal(size=(orb.sph_size, nmos)))[0]
    check(std.int_df2c_mo(orb, aux, C), oracle.int_df2c_mo(orb, aux, C))


def test_auxiliary_batches():
    """130 orbitals take two batches of auxiliary columns, their first 40 one:
    the pairs of those are the same bit for bit."""
    w = make_workload(60, 2, 2, 1, seed=3)
    C = np.linalg.qr(np.random.default_rng(6).normal(size=(w.shells.sph_size, 130)))[0]
    assert C.shape[1] * w.shells.sph_size * w.shells_aux.sph_size > 2**27
    many = std.int_df2c_mo(w.shells, w.shells_aux, C)
    few = std.int_df2c_mo(w.shells, w.shells_aux, C[:, :40])
    assert np.array_equal(many[: few.shape[0]], few)
