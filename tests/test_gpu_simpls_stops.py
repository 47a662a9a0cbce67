"""A fit that stops in the launch of the phases between the products: in the loading (||t|| overflows), in the
deflation (||v|| overflows), and in the next refresh (nothing is left to fit), on chunks that form a cluster and
on chunks that count their arrivals in memory."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _rows(p):
    return (4 << 20) // p + 50   # above the one-launch loop's n p


def _overflowing_scores(p):
    rng = np.random.default_rng(p)
    return 1e200 * rng.standard_normal((_rows(p), p)), 1e-200 * rng.standard_normal((_rows(p), 2))


def _overflowing_loading(p):
    """One column of +-1e200 on two rows with equal responses: no weight on it, but a loading."""
    rng = np.random.default_rng(p)
    X, Y = rng.standard_normal((_rows(p), p)), rng.standard_normal((_rows(p), 2))
    X[:, p // 2] = 0.0
    X[0, p // 2], X[1, p // 2] = 1e200, -1e200
    Y[1] = Y[0]
    return X, Y


def _one_direction(p):
    X = np.zeros((_rows(p), p))
    X[:, p - 1] = np.random.default_rng(p).integers(-2, 3, _rows(p))
    return X, X[:, [p - 1, p - 1]] * np.array([1.0, 2.0])


# the component count is known beforehand: none, none and one
@pytest.mark.parametrize("make,count", [(_overflowing_scores, 0), (_overflowing_loading, 0), (_one_direction, 1)])
@pytest.mark.parametrize("p", [259, 2048, 2049, 5003])   # 2 and 8 chunks (clusters), 9 and 20
def test_stopped_fit(lib, make, count, p):
    X, Y = make(p)
    for _ in range(3):   # launch by launch, then as a graph
        got = lib.pls_model2_fast(X, Y, [1, 5], scaling=3, seed=4, store_B=False)
        assert got["n_components"] == count
        assert not got["R"][:, count:].any() and not got["Q"][:, count:].any()
    if count:
        assert np.flatnonzero(got["R"][:, 0]).tolist() == [p - 1]
    # the fit after it is not affected
    rng = np.random.default_rng(1)
    X, Y = rng.standard_normal(X.shape), rng.standard_normal(Y.shape)
    assert lib.pls_model2_fast(X, Y, [1, 5], scaling=3, seed=4, store_B=False)["n_components"] == 5
