"""Wide three-plane products whose segments are dealt out by chunk of the contraction."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# 2048 x 512 is the smallest product of 128 x 128 tiles; contractions of one short segment, of a whole number
# of them and with a remainder
@pytest.mark.parametrize("n,p,m", [(700, 2048, 512), (2048, 2049, 640), (2500, 2300, 513)])
def test_wide_product(lib, n, p, m):
    rng = np.random.default_rng(n)
    t = rng.standard_normal((n, 1))
    X = t @ rng.standard_normal((1, p)) + 0.1 * rng.standard_normal((n, p))
    Y = t @ rng.standard_normal((1, m)) + 0.1 * rng.standard_normal((n, m))
    ref = lib.pls_model2_fast(X, Y, [1], seed=1)
    lib.set_precision("bf16x6")
    try:
        got = lib.pls_model2_fast(X, Y, [1], seed=1)
    finally:
        lib.set_precision("fp64")
    # S = X^T Y loses at most (6 x 1024) 2^-24 |x||y| in a segment's FP32 sums: 3.7e-4 of a rank-one S, and
    # the leading pair of vectors moves by that times 1 / (1 - 0.1)
    for key in ("R", "Q"):
        assert np.linalg.norm(got[key] - ref[key]) <= 4.1e-4 * np.linalg.norm(ref[key]), key
