"""Grid and primitive densities as products on tiles of 64 x 32 functions and 32,
64 or 128 points: point counts around the tiles, function lists that straddle
them inside one shell, unsymmetric density matrices in both layouts, points and
densities that are not finite. Tolerance as in test_grid_gpu.py (1e-13 of the
largest value: sums over pairs in another order).

The primitive density is compared with the sum of all pairs that pass the
reference's two tests of a pair, without its cutoff of single terms at exponents
of 36 (gdma/prim_dens.f90:13), which moves g shells far from their centers by
1e-11 and which the product form does not apply."""

import numpy as np
import pytest

import oracle
from grid_common import box_grid, cart_size, prim_data
from pysisyphus_addons.common.synthetic import make_workload
from pysisyphus_addons.gdma import prim_dens
from pysisyphus_addons.grid import grid

pytestmark = pytest.mark.gpu


def shells_of(natoms, lmax):
    return make_workload(natoms, lmax=lmax, lauxmax=0, nstates=1, seed=3).shells


def prim(sh, g, P, switch):
    li, pd = prim_data(sh)
    got, ref = np.full(len(g), np.nan), np.zeros(len(g))
    prim_dens.eval_prim_density(li, pd, g, P, switch, got)
    oracle.eval_prim_density(li, pd, g, P, switch, ref)
    return got, ref


def prim_pairs(sh, g, P, switch):
    li, pd = prim_data(sh)
    comps = {L: [(i, j, L - i - j) for i in range(L, -1, -1) for j in range(L - i, -1, -1)] for L in range(5)}
    dfact = [1.0, 1.0, 3.0, 15.0, 105.0]
    phi = []
    for (L, _), (c, e, *A) in zip(li, pd):
        d = g - np.array(A)
        poly = np.array([d[:, 0] ** i * d[:, 1] ** j * d[:, 2] ** k / np.sqrt(dfact[i] * dfact[j] * dfact[k])
                         for i, j, k in comps[L]])
        phi.append(c * np.exp(-e * (d**2).sum(1)) * poly)
    rho = np.zeros(len(g))
    for a in range(len(pd)):
        for b in range(a, len(pd)):
            ea, eb = pd[a][1], pd[b][1]
            dsum = (pd[a][2:] - pd[b][2:]).sum()
            if ea + eb >= switch or ea * eb / (ea + eb) * dsum**2 >= 36.0:
                continue
            ia, ib = li[a][1], li[b][1]
            blk = P[ia : ia + len(phi[a]), ib : ib + len(phi[b])]
            rho += (1.0 if a == b else 2.0) * np.einsum("ip,ij,jp->p", phi[a], blk, phi[b])
    return rho


@pytest.mark.parametrize("npoints", [1, 31, 32, 33, 64, 65, 9471, 9472, 9473])
def test_prim_point_tiles(npoints):
    sh = shells_of(6, 4)
    P = np.random.default_rng(1).normal(size=(cart_size(sh),) * 2)  # not symmetric
    g = box_grid(sh, n=npoints)
    got, ref = prim(sh, g, P, 4.0)[0], prim_pairs(sh, g, P, 4.0)
    assert np.abs(got - ref).max() <= 1e-13 * np.abs(ref).max()
    assert np.array_equal(got, prim(sh, g, np.asfortranarray(P), 4.0)[0])


@pytest.mark.parametrize("npoints,blk", [(1, 100), (127, 127), (129, 129), (1000, 128), (1000, 257)])
def test_grid_point_tiles(npoints, blk):
    sh = shells_of(6, 4)
    D = np.random.default_rng(2).normal(size=(2,) + (cart_size(sh),) * 2)  # the triangle mu >= nu is read
    g = box_grid(sh, n=npoints)
    got = grid.eval_densities(sh, g, D, blk_size=blk)
    ref = oracle.eval_densities(sh, g, D, blk_size=blk)
    assert np.abs(got - ref).max() <= 1e-13 * np.abs(ref).max()
    assert np.array_equal(got, grid.eval_densities(sh, g, np.asfortranarray(D), blk_size=blk))


def test_not_finite():
    """A point at infinity has no density, one that is not a number none other
    than itself, and a density element that is not finite only points its pair
    reaches."""
    sh = shells_of(6, 2)
    n = cart_size(sh)
    P = np.random.default_rng(3).normal(size=(n, n))
    g = box_grid(sh, n=70)
    ref = prim(sh, g, P, 4.0)[0]
    h = g.copy()
    h[5] = np.inf
    h[40, 1] = np.nan
    got, want = prim(sh, h, P, 4.0)
    keep = np.ones(70, bool)
    keep[[5, 40]] = False
    assert np.array_equal(got[keep], ref[keep]) and got[5] == 0.0 and np.isnan(got[40])
    assert np.array_equal(np.isnan(got), np.isnan(want))
    P[n - 1, n - 1] = np.nan
    far = np.concatenate([g, [[1e3, 0.0, 0.0]]])
    got, want = prim(sh, far, P, 4.0)
    assert np.array_equal(np.isnan(got), np.isnan(want)) and got[-1] == 0.0
