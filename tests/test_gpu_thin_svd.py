"""The exact thin SVD by QR and Jacobi on the triangle: singular vectors of small values, and a column that is
not a number."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
EPS = np.finfo(np.float64).eps


# one block of rows, several, and a last block of fewer rows than columns; columns per lane 1, 2 and 3; wide
@pytest.mark.parametrize("rows,cols", [(30, 8), (375, 22), (8, 8), (515, 3), (22, 375), (70, 64), (2000, 90), (1000, 96), (2048, 2), (2049, 2), (512, 4),
                                       (4, 4), (3, 513), (8193, 1)])
@pytest.mark.parametrize("decay", [0.8, 0.5, 0.1])
def test_vectors_of_small_values_are_orthogonal(lib, rows, cols, decay):
    rng = np.random.default_rng(rows + cols)
    c = min(rows, cols)
    k = min(c, int(np.log(1e-12) / np.log(decay)))   # values from 1 down to 1e-12
    q, r = (np.linalg.qr(rng.standard_normal((d, c)))[0] for d in (rows, cols))
    A = (q * decay ** np.arange(c)) @ r.T
    got = lib.truncated_svd(A, k, svd_method=3)
    # a level of c reflectors, each off by a few eps in norm, three levels at most
    tol = 12 * c * EPS
    assert np.max(np.abs(got["u"].T @ got["u"] - np.eye(k))) < tol
    assert np.max(np.abs(got["vt"] @ got["vt"].T - np.eye(k))) < tol
    assert np.max(np.abs(got["d"] - np.linalg.svd(A, compute_uv=False)[:k])) < tol
    left = A @ got["vt"].T - got["u"] * got["d"]
    assert np.max(np.abs(left)) < tol


def test_a_nan_stays_in_its_column(lib):
    rng = np.random.default_rng(3)
    A = np.linalg.qr(rng.standard_normal((700, 12)))[0] * 10.0 ** -np.arange(12)
    A = A @ (np.eye(12) + 0.1 * np.triu(rng.standard_normal((12, 12)), 1))
    want = np.linalg.svd(np.delete(A, 4, axis=1), compute_uv=False)
    A[123, 4] = np.nan
    got = lib.truncated_svd(A, 12, svd_method=3)
    assert np.isfinite(got["u"]).all() and np.max(np.abs(got["u"].T @ got["u"] - np.eye(12))) < 144 * EPS
    assert np.max(np.abs(got["d"][:11] - want)) < 144 * EPS * want[0]
    assert np.isnan(got["d"][11])


@pytest.mark.parametrize("n", [2, 4, 5, 16])   # one launch, and QR first
def test_null_direction_with_equal_entries(lib, n):
    """The direction left over keeps 1 / n of every unit vector's squared length."""
    P = np.eye(n) - np.full((n, n), 1.0 / n)
    got = lib.truncated_svd(P, n, svd_method=3)
    assert np.max(np.abs(got["u"].T @ got["u"] - np.eye(n))) < 12 * n * EPS
    assert np.max(np.abs(got["d"] - np.r_[np.ones(n - 1), 0.0])) < 12 * n * EPS
