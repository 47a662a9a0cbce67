"""The phases between a component's products in one launch: chunks in a cluster, chunks of a cooperative
launch, and the separate launches past what shared memory holds, against the oracle."""
import numpy as np
import pytest

from oracle import pls as opls

pytestmark = pytest.mark.gpu


# (p, m): 3 and 10 chunks of predictors; response counts whose chunk of S just fits shared memory (102) and
# does not (105), fewer than eight, and one; more than 32 columns take larger blocks.  n p is above the
# one-launch loop's limit.
@pytest.mark.parametrize("p,m", [(601, 3), (601, 33), (601, 102), (601, 105), (2311, 1), (2311, 9), (2311, 102),
                                 (2311, 105)])
def test_update_matches_oracle(lib, p, m):
    rng = np.random.default_rng(p + m)
    n, k = (4 << 20) // p + 77, 6
    L = rng.standard_normal((n, 8)) * np.arange(8, 0, -1)
    X = L @ rng.standard_normal((8, p)) + 0.3 * rng.standard_normal((n, p))
    Y = L @ rng.standard_normal((8, m)) + 0.1 * rng.standard_normal((n, m))
    got = lib.pls_model2_fast(X, Y, [2, k], seed=3)
    ref = opls.pls_model2_fast(X, Y, [2, k], seed=3)
    assert got["n_components"] == k
    # sums of 2^22 products in another order, amplified by the deflations' cancellation
    for key in ("R", "Q", "B"):
        assert np.linalg.norm(got[key] - ref[key]) <= 1e-9 * np.linalg.norm(ref[key]), key


# X^T t of a tall matrix in row ranges: two, and four of unequal length; a row-sharded fit on one rank adds
# the same ranges before its all-reduce
@pytest.mark.parametrize("n,p,m", [(16385, 300, 2), (33001, 259, 9)])
def test_row_ranges(lib, n, p, m):
    rng = np.random.default_rng(n)
    L = rng.standard_normal((n, 4))
    X = L @ rng.standard_normal((4, p)) + 0.3 * rng.standard_normal((n, p))
    Y = L @ rng.standard_normal((4, m)) + 0.1 * rng.standard_normal((n, m))
    got = lib.pls_model2_fast(X, Y, [4], seed=1)
    ref = opls.pls_model2_fast(X, Y, [4], seed=1)
    one = lib.pls_model2_fast(X, Y, [4], seed=1, allreduce=lambda buf, count, stream: None)
    for key in ("R", "Q", "B"):
        assert np.linalg.norm(got[key] - ref[key]) <= 1e-9 * np.linalg.norm(ref[key]), key
        assert np.array_equal(one[key], got[key]), key
