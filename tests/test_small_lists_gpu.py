"""Sorted lists of small systems (one block per list, up to 4096 entries) against
the general sorts: basis sets just below and above the limit, with ties, in both
screenings. 90 s shells of one primitive have 4095 primitive pairs, 91 have 4186.

The same molecule takes the general path with shells added far away that have no
density. Tolerance: 1e-13 of the largest element; the added shells change the
tiles and the order of the sums, but no term."""

import numpy as np
import pytest

from pysisyphus_addons import _native as nat
from pysisyphus_addons.common.shells import Shell, Shells
from pysisyphus_addons.diabatization import intor

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def raw():
    nat.set_skip_metric(1)
    yield
    nat.set_skip_metric(0)
    nat.set_screening("schwarz")


def basis(n):
    """Every third shell repeats the one before it: equal Schwarz values."""
    rng = np.random.default_rng(1)
    X, e = rng.uniform(0.0, 12.0, (n, 3)), np.exp(rng.uniform(-1.0, 3.0, n))
    k = [i - 1 if i % 3 == 2 else i for i in range(n)]
    return Shells([Shell(0, X[j], [1.0], [e[j]], i, 1) for i, j in enumerate(k)])


@pytest.mark.parametrize("screening", ["schwarz", "qvl"])
@pytest.mark.parametrize("n", [1, 2, 3, 32, 89, 90])
def test_small_lists(n, screening):
    nat.set_screening(screening)
    rng = np.random.default_rng(2)
    orb = basis(n)
    aux = Shells([Shell(L, rng.uniform(0.0, 12.0, 3), [1.0], [0.4 * 2.0**L], i, 1) for i, L in enumerate([0, 1, 2, 3] * 5)])
    D = rng.normal(size=(3, n, n))
    got = intor.contract_coulomb_densities_2d(orb, aux, D)
    # the general path: 91 shells, the added ones without density
    big = basis(n).shells + [Shell(0, [500.0 + 40.0 * i, 0.0, 0.0], [1.0], [1.0], n + i, 1) for i in range(91 - n)]
    E = np.zeros((3, 91, 91))
    E[:, :n, :n] = D
    wide = intor.contract_coulomb_densities_2d(Shells(big), aux, E)
    assert np.abs(wide - got).max() <= 1e-13 * np.abs(got).max()
