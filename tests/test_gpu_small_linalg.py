"""Small dense FP64 kernels behind the randomized and exact SVDs, at the sizes
where their tiles, lane groups and shared-memory limits begin and end."""
import numpy as np
import pytest

from oracle import svd as osvd

pytestmark = pytest.mark.gpu
EPS = np.finfo(np.float64).eps


def _matrix(rows, cols, seed, decay):
    rng = np.random.default_rng(seed)
    r = min(rows, cols)
    u = np.linalg.qr(rng.standard_normal((rows, r)))[0]
    v = np.linalg.qr(rng.standard_normal((cols, r)))[0]
    return (u * (5.0 * decay ** np.arange(r))) @ v.T


# l = k + 10 eigenvalues of the projected Gram: odd and even, one pair per lane
# (l <= 64), two (65 ..), the largest that fits in shared memory and the first
# that does not
@pytest.mark.parametrize("k", [1, 2, 21, 22, 53, 54, 55, 80, 101, 102, 103])
def test_randomized_svd_core_sizes(lib, k):
    rows, cols = 150, 131
    A = _matrix(rows, cols, k, 0.97)
    got = lib.truncated_svd(A, k, svd_method=4, oversample=10, power_iters=2, seed=3)
    ref = osvd.truncated_svd(A, k, svd_method=4, oversample=10, power_iters=2, seed=3)
    # singular values: sqrt of eigenvalues of B B^T, each off by at most a few
    # hundred eps of the largest one; vectors by that over the smallest gap
    # (decay 0.97: neighbours 3 % apart, the smallest value 0.97^k of the first)
    tol = 1000 * EPS / 0.97 ** (2 * k)
    assert np.max(np.abs(got["d"] - ref.s)) <= tol * ref.s[0]
    assert np.linalg.norm(got["u"].T @ got["u"] - np.eye(k)) < 1000 * EPS * k
    proj = np.linalg.norm(ref.U @ (ref.U.T @ got["u"]) - got["u"])
    assert proj < 1000 * tol
    approx = (got["u"] * got["d"]) @ got["vt"]
    want = (ref.U * ref.s) @ ref.Vt
    assert np.linalg.norm(approx - want) <= 1000 * tol * np.linalg.norm(want)
