"""The Cholesky factor and the forward substitution at the sizes where their
64-column steps and column tiles begin and end: block edges of n, one step with
and without a trailing update, and the column counts around the tiles of 8, 32
and 40 and the switch between two and four blocks per step.

Bounds: Cholesky's backward error ||A - L L^T||_F <= (n + 1) eps ||A||_F (Higham,
"Accuracy and Stability of Numerical Algorithms", theorem 10.3, in norm), and for
the well conditioned matrices here (condition number below 10) forward errors of
L^-1 B below 8 n eps of its norm.
"""

import numpy as np
import pytest

from pysisyphus_addons import _native as nat

pytestmark = pytest.mark.gpu
EPS = np.finfo(float).eps


def spd(n, seed):
    """Eigenvalues in [1, 9], elements of every size."""
    rng = np.random.default_rng(seed)
    Q = np.linalg.qr(rng.normal(size=(n, n)))[0]
    A = (Q * rng.uniform(1.0, 9.0, n)) @ Q.T
    return 0.5 * (A + A.T)


@pytest.mark.parametrize("n", [1, 2, 15, 16, 17, 63, 64, 65, 127, 128, 129, 191, 193, 256, 257, 449, 641])
def test_factor_and_solve_block_edges(n):
    A = spd(n, n)
    B = np.random.default_rng(n + 1).normal(size=(n, 5))
    L, Y = nat.cholesky_solve(A, B)
    L = np.tril(L)
    assert np.linalg.norm(A - L @ L.T) <= (n + 1) * EPS * np.linalg.norm(A)
    ref = np.linalg.solve(np.linalg.cholesky(A.astype(np.longdouble).astype(float)), B)
    assert np.linalg.norm(Y - ref) <= 8 * n * EPS * np.linalg.norm(ref)


@pytest.mark.parametrize("n", [130, 400])
@pytest.mark.parametrize("nrhs", [1, 7, 8, 9, 40, 41, 64, 128, 129, 192, 193, 300])
def test_solve_column_counts(n, nrhs):
    A = spd(n, 7)
    B = np.random.default_rng(nrhs).normal(size=(n, nrhs))
    L, Y = nat.cholesky_solve(A, B)
    assert np.linalg.norm(np.tril(L) @ Y - B) <= 8 * n * EPS * np.linalg.norm(Y) * 3.0


@pytest.mark.parametrize("scale", [1e-140, 1e140])
def test_factor_scaled(scale):
    """Squares of the pivots are out of range; the factor is not."""
    A = spd(100, 3)
    L, _ = nat.cholesky_solve(A * scale, np.ones((100, 1)))
    ref = np.linalg.cholesky(A)
    assert np.linalg.norm(np.tril(L) / np.sqrt(scale) - ref) <= 8 * 100 * EPS * np.linalg.norm(ref)


@pytest.mark.parametrize("col", [0, 1, 15, 16, 63, 64, 127, 130, 199])
def test_pivot_reported(col):
    A = spd(200, 5)
    L = np.linalg.cholesky(A)
    A[col, col] -= L[col, col] ** 2 + 0.5  # the Schur complement of this column is -0.5
    with pytest.raises(nat.PaError) as e:
        nat.cholesky_solve(A, np.ones((200, 1)))
    assert e.value.code == nat.PA_ERR_NOT_SPD and f"pivot {col + 1})" in str(e.value)
