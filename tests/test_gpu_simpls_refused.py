"""Fits whose resident or cluster launches the driver refuses, from the first one or in mid-loop, go on with the
separate launches: the same sums in the same order."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# the one-launch loop; the phases as a cluster and on counted arrivals, with fewer responses than warps and more
@pytest.mark.parametrize("n,p,m", [(300, 500, 3), (300, 700, 9), (6000, 750, 2), (6000, 750, 40), (1900, 2311, 5),
                                   (1900, 2311, 12)])
def test_refused_launches(lib, monkeypatch, n, p, m):
    rng = np.random.default_rng(n + m)
    L = rng.standard_normal((n, 6))
    X = L @ rng.standard_normal((6, p)) + 0.3 * rng.standard_normal((n, p))
    Y = L @ rng.standard_normal((6, m)) + 0.1 * rng.standard_normal((n, m))
    fit = lambda: lib.pls_model2_fast(X, Y, [2, 6], seed=3, store_B=False)
    want = fit()
    assert want["n_components"] == 6
    for first in (0, 1, 3):
        monkeypatch.setenv("FASTPLS_TEST_REFUSE_FROM", str(first))
        got = [fit() for _ in range(2)]   # launch by launch, and as a graph
        monkeypatch.delenv("FASTPLS_TEST_REFUSE_FROM")
        for g in got:
            for key in ("R", "Q", "n_components"):
                assert np.array_equal(g[key], want[key]), (first, key)
    assert np.array_equal(fit()["R"], want["R"])
