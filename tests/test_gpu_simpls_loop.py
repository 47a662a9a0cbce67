"""The one-launch SIMPLS loop of small fits against the loop of launches: a
row-sharded fit on one rank (its all-reduce is the identity) always takes the
launches, with the same sums in the same order, so the results are equal."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _data(n, p, m, seed):
    rng = np.random.default_rng(seed)
    L = rng.standard_normal((n, 6))
    X = L @ rng.standard_normal((6, p)) + 0.5 * rng.standard_normal((n, p))
    return X, L @ rng.standard_normal((6, m)) + 0.3 * rng.standard_normal((n, m))


# chunks of the predictors (256 rows), rows of an X tile (32) and of a score chunk
# (256), response counts around the eight warps, one response, column ranges
# longer than a tile (few rows allow many ranges, many rows few)
@pytest.mark.parametrize("n,p,m,k", [(31, 6, 2, 2), (33, 255, 1, 4), (64, 256, 7, 5), (65, 257, 8, 5), (257, 300, 9, 6),
                                     (400, 2000, 5, 10), (500, 3001, 33, 7), (4000, 1000, 3, 5), (30000, 130, 4, 4),
                                     (300, 500, 100, 12)])
@pytest.mark.parametrize("fit", [False, True])
def test_loop_equals_launches(lib, n, p, m, k, fit):
    X, Y = _data(n, p, m, n + p)
    one = lib.pls_model2_fast(X, Y, [1, k], fit=fit, allreduce=lambda buf, count, stream: None)
    got = lib.pls_model2_fast(X, Y, [1, k], fit=fit)
    for key in ("R", "Q", "B", "mX", "mY", "R2Y") + (("Yfit",) if fit else ()):
        assert np.array_equal(one[key], got[key]), key
    assert one["n_components"] == got["n_components"] == k


def test_loop_stops_with_the_launches(lib):
    """A rank-two predictor block: the third component is degenerate in both."""
    rng = np.random.default_rng(0)
    X = np.zeros((60, 40))
    X[:, 0], X[:, 1] = rng.integers(-2, 3, 60), rng.integers(-2, 3, 60)
    Y = np.stack([X[:, 0], X[:, 1]], axis=1)
    one = lib.pls_model2_fast(X, Y, [6], scaling=3, allreduce=lambda buf, count, stream: None)
    got = lib.pls_model2_fast(X, Y, [6], scaling=3)
    assert one["n_components"] == got["n_components"]
    k = got["n_components"]
    assert np.array_equal(one["R"][:, :k], got["R"][:, :k]) and np.array_equal(one["Q"][:, :k], got["Q"][:, :k])
    zero = lib.pls_model2_fast(np.zeros((50, 30)), Y[:50], [3], scaling=3)
    assert zero["n_components"] == 0
