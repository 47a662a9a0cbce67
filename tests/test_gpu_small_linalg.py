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


# Cholesky solves: the lane groups' register counts change at 32, 64, 104, 128
# and 160 unknowns (161: the global-memory kernel); 64 right-hand sides a CTA pass
@pytest.mark.parametrize("d,q", [(1, 5), (7, 63), (8, 64), (16, 65), (17, 66), (32, 129), (33, 129), (64, 200), (65, 200),
                                 (104, 300), (105, 300), (128, 330), (129, 330), (160, 400), (161, 400)])
def test_spd_solve_sizes(lib, d, q):
    from oracle import gaussian_y as ogy
    rng = np.random.default_rng(d)
    Y = rng.standard_normal((450, q))
    G = rng.standard_normal((q, d)) / np.sqrt(d)
    got = lib.gaussian_y_encode(Y, G)
    ref = ogy.prepare_regression(Y, G)
    # condition of Z^T Z below 1e5 at every size: rounding 1e-16 stays below 1e-9
    assert np.linalg.norm(got["Z"] - ref["Z"]) < 1e-9 * np.linalg.norm(ref["Z"])
    assert np.linalg.norm(got["decoder"] - ref["decoder"]) < 1e-9 * np.linalg.norm(ref["decoder"])


# CholeskyQR2 at the same register counts (l = k + 10 columns; 161: Gram-Schmidt)
# and around whole groups of 64 rows
@pytest.mark.parametrize("rows,l", [(90, 16), (91, 17), (127, 22), (128, 32), (129, 33), (300, 64), (301, 65), (320, 104), (321, 105),
                                    (400, 128), (401, 129), (449, 160), (450, 161)])
def test_cholesky_qr_sizes(lib, rows, l):
    k, cols = l - 10, min(rows, l + 40)
    A = _matrix(rows, cols, l, 0.98)
    got = lib.truncated_svd(A, k, svd_method=4, oversample=10, power_iters=1, seed=5)
    assert np.linalg.norm(got["u"].T @ got["u"] - np.eye(k)) < 1000 * EPS * k
    ref = osvd.truncated_svd(A, k, svd_method=4, oversample=10, power_iters=1, seed=5)
    # one power iteration cubes the decay: the sample's smallest direction is
    # 0.98^(3 l) of the largest, which is how far rounding is amplified
    tol = 1000 * EPS / 0.98 ** (3 * l)
    assert np.max(np.abs(got["d"] - ref.s)) <= tol * ref.s[0]


# Exact thin SVD through QR: one block of rows, several, a ragged last one shorter
# than the columns, two levels, wide inputs, one / two / three registers a lane,
# the largest column count of this route, the first of the whole-GPU one
@pytest.mark.parametrize("rows,cols", [(5, 1), (8, 5), (32, 32), (375, 22), (512, 22), (513, 22), (522, 22), (5000, 22),
                                       (40, 4000), (400, 33), (300, 64), (700, 65), (260, 96), (2000, 96), (200, 97)])
@pytest.mark.parametrize("deficient", [False, True])
def test_exact_svd_shapes(lib, rows, cols, deficient):
    r = min(rows, cols)
    A = _matrix(rows, cols, rows + cols, 0.95)
    if deficient and r > 1:     # a centred class response: one exact null direction
        A = A - A.mean(axis=1 if cols <= rows else 0, keepdims=True)
    got = lib.truncated_svd(A, r, svd_method=3)
    s = np.linalg.svd(A, compute_uv=False)
    # backward stable: eps times the size, of the largest singular value
    tol = 20 * EPS * max(rows, cols) * s[0]
    assert np.max(np.abs(got["d"] - s)) < tol
    assert np.linalg.norm((got["u"] * got["d"]) @ got["vt"] - A) < 10 * r * tol
    assert np.linalg.norm(got["vt"] @ got["vt"].T - np.eye(r)) < 1e3 * EPS * r
    # U = A V / s amplifies rounding by up to 1e4, weaker columns are made orthogonal
    assert np.linalg.norm(got["u"].T @ got["u"] - np.eye(r)) < 1e4 * EPS * max(rows, cols)
