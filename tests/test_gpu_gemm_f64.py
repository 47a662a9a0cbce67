"""FP64 tensor-core GEMM at the edges of its tiles: every tile width and the
counts next to it, rows around 64, contractions around the 4- and 16-step
blocks, split ranges, odd leading dimensions (8-byte copies) and even ones."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
EPS = np.finfo(np.float64).eps


def _check(C, A, B):
    # every product and sum rounds once: K eps of the absolute products
    bound = 2 * A.shape[1] * EPS * (np.abs(A) @ np.abs(B)) + 1e-300
    assert np.all(np.abs(C - A @ B) <= bound)


@pytest.mark.parametrize("n", [1, 7, 8, 9, 16, 17, 32, 33, 40, 41, 56, 57, 64, 65, 80, 81, 104, 105, 208, 300])
@pytest.mark.parametrize("m,k", [(1, 1), (63, 3), (64, 16), (65, 17), (130, 100), (127, 515)])
def test_product_shapes(lib, m, n, k):
    rng = np.random.default_rng(m * 1000 + n + k)
    A, B = rng.standard_normal((m, k)), rng.standard_normal((k, n))
    _check(lib.matrix_multiply(A, B), A, B)


# 2^28 multiply-adds and more: ranges by modelled time
@pytest.mark.parametrize("m,n,k", [(768, 100, 4001), (2049, 1000, 133), (20000, 50, 300), (130, 31, 70000)])
def test_large_products(lib, m, n, k):
    rng = np.random.default_rng(n)
    A, B = rng.standard_normal((m, k)), rng.standard_normal((k, n))
    _check(lib.matrix_multiply(A, B), A, B)


# the transposed operands, through calls that use them: Z^T Z and Z^T Y (A^T B) and
# scores T L^T (A B^T) with a row vector added
@pytest.mark.parametrize("n,d,q", [(65, 5, 33), (257, 40, 81), (1000, 64, 104), (513, 31, 211)])
def test_transposed_operands(lib, n, d, q):
    from oracle import gaussian_y as ogy
    rng = np.random.default_rng(n)
    Y, G = rng.standard_normal((n, q)), rng.standard_normal((q, d))
    got, ref = lib.gaussian_y_encode(Y, G), ogy.prepare_regression(Y, G)
    assert np.linalg.norm(got["decoder"] - ref["decoder"]) < 1e-9 * np.linalg.norm(ref["decoder"])
    dec, mu = rng.standard_normal((d, q)), rng.standard_normal(q)
    Z = rng.standard_normal((n, d))
    _check(lib.gaussian_y_decode(Z, dec, mu), np.hstack([Z, np.ones((n, 1))]), np.vstack([dec, mu]))
    lin, const = rng.standard_normal((q, d)), rng.standard_normal(q)
    sc = lib.lda_predict(Z, dict(linear=lin, constants=const), return_scores=True)["scores"]
    _check(sc, np.hstack([Z, np.ones((n, 1))]), np.vstack([lin.T, const]))
