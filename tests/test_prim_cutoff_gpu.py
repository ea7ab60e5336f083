"""The two kernels of the primitive density and the reference's cutoff of single
terms (gdma/prim_dens.f90:13: a pair is left out at points with p |r - P|^2 >= 36).

Finite input with positive exponents takes the product form, which sums those
terms: its values minus the terms are the oracle's. Other input takes the
pair-by-pair kernel, which leaves them out as the oracle does. Tolerance as in
test_grid_gpu.py: 1e-13 of the largest value (sums over pairs in another order)."""

import numpy as np
import pytest

import oracle
from grid_common import box_grid, cart_size, prim_data
from pysisyphus_addons.common.synthetic import make_workload
from pysisyphus_addons.gdma import prim_dens

pytestmark = pytest.mark.gpu

SWITCH = 4.0
DFACT = [1.0, 1.0, 3.0, 15.0, 105.0]


def values(sh, g, P):
    li, pd = prim_data(sh)
    got, ref = np.full(len(g), np.nan), np.zeros(len(g))
    prim_dens.eval_prim_density(li, pd, g, P, SWITCH, got)
    oracle.eval_prim_density(li, pd, g, P, SWITCH, ref)
    return got, ref


def terms_beyond_cutoff(sh, g, P):
    """Sum of the terms with p |r - P|^2 >= 36 of the pairs that pass the
    reference's two tests."""
    li, pd = prim_data(sh)
    phi = []
    for (L, _), (c, e, *A) in zip(li, pd):
        d = g - np.array(A)
        poly = np.array([d[:, 0] ** i * d[:, 1] ** j * d[:, 2] ** (L - i - j) / np.sqrt(DFACT[i] * DFACT[j] * DFACT[L - i - j])
                         for i in range(L, -1, -1) for j in range(L - i, -1, -1)])
        phi.append(c * np.exp(-e * (d**2).sum(1)) * poly)
    rho = np.zeros(len(g))
    for a in range(len(pd)):
        for b in range(a, len(pd)):
            ea, eb, A, B = pd[a][1], pd[b][1], pd[a][2:], pd[b][2:]
            p = ea + eb
            if p >= SWITCH or ea * eb / p * (A - B).sum() ** 2 >= 36.0:
                continue
            out = p * ((g - (ea * A + eb * B) / p) ** 2).sum(1) >= 36.0
            if not out.any():
                continue
            ia, ib = li[a][1], li[b][1]
            blk = P[ia : ia + len(phi[a]), ib : ib + len(phi[b])]
            rho[out] += (1.0 if a == b else 2.0) * np.einsum("ip,ij,jp->p", phi[a][:, out], blk, phi[b][:, out])
    return rho


@pytest.mark.parametrize("lmax", [2, 4])
def test_product_form_sums_the_terms_beyond_the_cutoff(lmax):
    sh = make_workload(6, lmax=lmax, lauxmax=0, nstates=1, seed=3).shells
    P = np.random.default_rng(1).normal(size=(cart_size(sh),) * 2)
    g = box_grid(sh, n=400, margin=6.0)
    got, ref = values(sh, g, P)
    beyond = terms_beyond_cutoff(sh, g, P)
    top = np.abs(ref).max()
    assert np.abs(got - beyond - ref).max() <= 1e-13 * top
    assert np.abs(beyond).max() <= 1e-10 * top  # what the cutoff moves


@pytest.mark.parametrize("lmax", [2, 4])
def test_pair_kernel_keeps_the_cutoff(lmax):
    """One element of P is not a number: points that its pair does not reach agree
    with the oracle, which has the same cutoff, and the others are the oracle's too."""
    sh = make_workload(6, lmax=lmax, lauxmax=0, nstates=1, seed=3).shells
    n = cart_size(sh)
    P = np.random.default_rng(1).normal(size=(n, n))
    P[n - 1, n - 1] = np.nan
    g = np.concatenate([box_grid(sh, n=400, margin=6.0), [[1e3, 0.0, 0.0]]])
    got, ref = values(sh, g, P)
    assert np.array_equal(np.isnan(got), np.isnan(ref))
    ok = ~np.isnan(ref)
    assert ok.sum() >= 20
    assert np.abs(got[ok] - ref[ok]).max() <= 1e-13 * np.abs(ref[ok]).max()


def test_unused_element_that_is_not_a_number():
    """An element that no primitive pair reads changes the kernel, not the values
    beyond the terms of the cutoff."""
    sh = make_workload(6, lmax=4, lauxmax=0, nstates=1, seed=3).shells
    n = cart_size(sh)
    P = np.zeros((n + 1, n + 1))
    P[:n, :n] = np.random.default_rng(1).normal(size=(n, n))
    g = box_grid(sh, n=400, margin=6.0)
    got, ref = values(sh, g, P)
    P[n, n] = np.nan
    pairwise, _ = values(sh, g, P)
    top = np.abs(ref).max()
    assert np.abs(pairwise - ref).max() <= 1e-13 * top
    assert np.abs(got - terms_beyond_cutoff(sh, g, P[:n, :n]) - pairwise).max() <= 1e-13 * top
