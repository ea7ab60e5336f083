"""int_df2c_mo where the block matrix, not the half-transformed tensor, limits a
batch of auxiliary columns (few orbitals, many shell pairs).

Every auxiliary column is computed by itself, so the tensor of all auxiliary
shells (two batches) is that of its halves (one batch each), bit for bit."""

import numpy as np
import pytest

from pysisyphus_addons import _native as nat
from pysisyphus_addons.common.shells import Shells
from pysisyphus_addons.common.synthetic import make_workload
from pysisyphus_addons.intor import intor
from pysisyphus_addons.std import intor as std

pytestmark = pytest.mark.gpu

BLOCK_DOUBLES = 1 << 28  # of the block matrix of one batch


def test_block_matrix_limits_the_batch():
    nat.set_boys_mode("exact")
    nat.set_skip_metric(1)
    try:
        w = make_workload(50, 3, 4, 1, seed=3)
        aux = list(w.shells_aux.shells)
        halves = [Shells(aux[0::2]), Shells(aux[1::2])]
        # rows of the pairs that meet the largest auxiliary Schwarz value
        q = intor.int_schwarz_bra(w.shells) * intor.int_schwarz_aux(w.shells_aux).max()
        n = np.array([s.sph_size for s in w.shells.shells])
        a, b = np.tril_indices(len(n))
        rows = int((n[a] * n[b])[q >= np.float32(1e-10)].sum())
        assert BLOCK_DOUBLES < rows * w.shells_aux.sph_size < 1.9 * BLOCK_DOUBLES
        C = np.linalg.qr(np.random.default_rng(6).normal(size=(w.shells.sph_size, 5)))[0]
        whole = std.int_df2c_mo(w.shells, w.shells_aux, C)
        size = np.array([s.sph_size for s in aux])
        first = np.concatenate([[0], np.cumsum(size)])
        for k, half in enumerate(halves):
            cols = np.concatenate([np.arange(first[i], first[i + 1]) for i in range(k, len(aux), 2)])
            part = std.int_df2c_mo(w.shells, half, C)
            assert np.array_equal(whole[:, cols], part)
    finally:
        nat.set_skip_metric(0)
        nat.set_boys_mode("reference")
