"""The one-launch lists and density folding of small systems (up to 4096 primitive
pairs) with several classes, against the general path: shells of mixed L with one
to three primitives, classes that are empty, and more densities than one chunk of
the folded product (40).

As in test_small_lists_gpu.py the same molecule takes the general path with shells
added far away that have no density; the added shells change the order of the sums,
but no term. Tolerance: an element sums some 1e4 products of random sign, whose
rounding in another order is about 1e2 eps = 2e-14 of its size; 1e-12 of the
largest element."""

import numpy as np
import pytest

from pysisyphus_addons import _native as nat
from pysisyphus_addons.common.shells import Shell, Shells
from pysisyphus_addons.diabatization import intor

pytestmark = pytest.mark.gpu

LIMIT = 4096


@pytest.fixture(autouse=True)
def raw():
    nat.set_skip_metric(1)
    yield
    nat.set_skip_metric(0)
    nat.set_screening("schwarz")


def prim_pairs(shells):
    k = np.array([s.nprims for s in shells])
    return int((k.sum() ** 2 + (k**2).sum()) // 2)


def basis(Ls):
    """As many shells as stay within the limit; the last ones have one primitive."""
    rng = np.random.default_rng(1)
    out = []
    while True:
        i = len(out)
        n = 1 + i % 3 if i < 30 else 1
        sh = Shell(Ls[i % len(Ls)], rng.uniform(0.0, 9.0, 3), rng.uniform(0.2, 1.0, n), np.exp(rng.uniform(-1.0, 2.0, n)), i, 1)
        if prim_pairs(out + [sh]) > LIMIT:
            return out
        out.append(sh)


@pytest.mark.parametrize("screening", ["schwarz", "qvl"])
@pytest.mark.parametrize("Ls", [(0, 1, 2, 3), (3, 0), (4, 1), (2,)])
def test_several_classes(Ls, screening):
    nat.set_screening(screening)
    small = basis(Ls)
    assert LIMIT - 100 < prim_pairs(small) <= LIMIT
    far = [Shell(0, [500.0 + 40.0 * i, 0.0, 0.0], [1.0], [1.0], len(small) + i, 1) for i in range(3)]
    assert prim_pairs(small + far) > LIMIT
    orb, big = Shells(small), Shells(small + far)
    n, m = orb.sph_size, big.sph_size
    rng = np.random.default_rng(2)
    aux = Shells([Shell(L, rng.uniform(0.0, 9.0, 3), [1.0], [0.4 * 2.0**L], i, 1) for i, L in enumerate([0, 1, 2, 3, 4] * 4)])
    D = rng.normal(size=(45, n, n))
    E = np.zeros((45, m, m))
    E[:, :n, :n] = D
    got = intor.contract_coulomb_densities_2d(orb, aux, D)
    wide = intor.contract_coulomb_densities_2d(big, aux, E)
    assert np.abs(wide - got).max() <= 1e-12 * np.abs(got).max()
