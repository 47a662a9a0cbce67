"""FP64 products whose operands allow 8-byte copies only (odd leading dimensions): the staged 64 x 64 tiles and the
asynchronous ones, full and ragged tiles, contractions that end inside a step."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# A B: staged tiles (33 to 64 columns, one and several ranges), widths of 5, 7 and 13 eights, one column
@pytest.mark.parametrize("m,n,k", [(20001, 61, 101), (5001, 60, 2001), (20000, 64, 777), (129, 50, 333), (20001, 101, 333),
                                   (2001, 101, 3001), (65, 39, 17), (63, 1, 5), (4097, 127, 1023), (20001, 47, 301)])
def test_products(lib, m, n, k):
    rng = np.random.default_rng(m + n + k)
    # integers up to 8: every sum is exact, so the order does not matter
    A = rng.integers(-8, 9, (m, k)).astype(np.float64)
    B = rng.integers(-8, 9, (k, n)).astype(np.float64)
    assert np.array_equal(lib.matrix_multiply(A, B), A @ B)


# A^T B and A B^T inside: Z^T Z and Z^T Y over an odd number of rows, and the scores' product with the weights
@pytest.mark.parametrize("n,q,d", [(777, 61, 9), (20001, 130, 33), (3001, 500, 7), (301, 64, 60)])
def test_products_of_transposes(lib, n, q, d):
    from oracle import gaussian_y as ogy
    rng = np.random.default_rng(n)
    Y = rng.standard_normal((n, q))
    G = rng.standard_normal((q, d)) / np.sqrt(d)
    got, ref = lib.gaussian_y_encode(Y, G), ogy.prepare_regression(Y, G)
    # condition of Z^T Z below 1e5: rounding 1e-16 stays below 1e-9
    assert np.linalg.norm(got["Z"] - ref["Z"]) < 1e-9 * np.linalg.norm(ref["Z"])
    assert np.linalg.norm(got["decoder"] - ref["decoder"]) < 1e-9 * np.linalg.norm(ref["decoder"])
