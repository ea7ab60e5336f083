"""Order of the Cholesky factorization's launches on its two streams.

Step c (the panel of block column c and the next diagonal block) takes the
contribution of column c - 1 itself, so it needs the trailing updates up to that
of column c - 2 and must not wait for that of column c - 1, which runs beside it.
The order is read from a captured graph that is never launched; the factor itself
is compared bit for bit with the one-stream form, repeatedly, since an order that
is not enough would show in some runs only.
"""

import ctypes

import numpy as np
import pytest

from pysisyphus_addons import _native as nat

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 64, 65, 128, 129, 192, 193, 256, 257, 320, 449, 960, 2240])
def test_updates_run_beside_the_next_step(n):
    missing, apart, pairs = ctypes.c_int(-1), ctypes.c_int(-1), ctypes.c_int(-1)
    nat.check(nat.load().pa_cholesky_order_check(n, ctypes.byref(missing), ctypes.byref(apart), ctypes.byref(pairs)))
    nblk = (n + 63) // 64
    assert missing.value == 0
    assert pairs.value == max(0, nblk - 3)  # an update has more to do than the next diagonal tile up to column nblk - 4
    assert apart.value == pairs.value


@pytest.mark.parametrize("n", [129, 193, 256, 257, 320, 384, 700, 1500])
def test_two_streams_give_the_factor_of_one(n):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(n)
    X = rng.normal(size=(n, n))
    A = X @ X.T + n * np.eye(n)
    d = torch.from_numpy(A.copy()).cuda()  # symmetric: either order
    b, x = torch.ones(n, dtype=torch.float64, device="cuda"), torch.empty(n, dtype=torch.float64, device="cuda")
    nat.check(nat.load().pa_cholesky_solve_noalloc(n, d.data_ptr(), 1, b.data_ptr(), x.data_ptr(),
                                                   torch.cuda.current_stream().cuda_stream))
    L = np.tril(d.cpu().numpy().T)  # column-major
    for _ in range(5):
        M, y = nat.cholesky_solve(A, np.ones((n, 1)))
        np.testing.assert_array_equal(np.tril(M), L)
        np.testing.assert_array_equal(y[:, 0], x.cpu().numpy())
